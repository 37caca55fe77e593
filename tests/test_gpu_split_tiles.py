"""Sub-tiles whose parts go to CTAs of their own (8x and 16x) against the oracle:
coarse tiles with a few primitives less and more than it takes, several of them,
at the frame's corners and across tile borders, single-sampled ones among them,
and tiles whose counts serve blend demotion too; and instances small enough that
all of them are split.  Which CTA shades a part changes no result: every plane and
the covered-sample count must be equal."""
import numpy as np
import pytest

import gsgen
from test_gpu_parity import assert_same, run_both

pytestmark = pytest.mark.gpu

W, H, ZBP = 320, 224, 64


def cluster(s, rng, n, x0, y0, size, prim=gsgen.PRIM_TRI, **flags):
    k = 3 if prim == gsgen.PRIM_TRI else 2
    x = np.clip(rng.integers(x0 * 16, (x0 + size) * 16 + 1, size=(n, k)), 0, W * 16 - 1)
    y = np.clip(rng.integers(y0 * 16, (y0 + size) * 16 + 1, size=(n, k)), 0, H * 16 - 1)
    q = np.zeros((n * k, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(n * k, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), rng.integers(0, 1 << 24, size=n * k))
    s.packed(gsgen.prim_reg(prim, iip=1, **flags), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))


def flat_sprites(s, rng, n, x0, y0):
    """Opaque, on pixel boundaries, one depth: tiles that need one sample."""
    q = np.zeros((n * 2, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(n * 2, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(np.tile([x0 * 16, (x0 + 8) * 16], n), np.tile([y0 * 16, (y0 + 8) * 16], n), np.full(n * 2, 77))
    s.packed(gsgen.prim_reg(gsgen.PRIM_SPRITE), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))


def frame(ss, n, aa1, blended=False, hacks=None):
    rng = np.random.default_rng(ss * 10000 + n)
    s = gsgen.GifStream()
    gsgen._frame_setup(s, 0, W // 64, gsgen.PSMCT32, ZBP, gsgen.PSMZ24, W, H, gsgen.test_reg(zte=1, ztst=2),
                       alpha=gsgen.alpha_reg(0, 1, 0, 1), extra=[(gsgen.COLCLAMP, 1)])
    if blended:
        s.ad([(gsgen.ZBUF_1, gsgen.zbuf_reg(ZBP, gsgen.PSMZ24, 1)), (gsgen.TEST_1, gsgen.test_reg(zte=1, ztst=1))])
    cluster(s, rng, 40, 0, 0, W)
    for x0, y0, size in ((0, 0, 8), (W - 8, H - 8, 8), (60, 36, 9), (128, 96, 16)):
        cluster(s, rng, n - n // 4, x0, y0, size, aa1=aa1, abe=int(blended))
        cluster(s, rng, n // 4, x0, y0, size, abe=1)
    flat_sprites(s, rng, n, 200, 104)
    cluster(s, rng, 20, 0, 0, W, prim=gsgen.PRIM_SPRITE, abe=1)
    meta = {"width": W, "height": H}
    if hacks:
        meta["hacks"] = hacks
    return gsgen.Frame("split", s.tobytes(), ss, ss == 16, 5 * n + 60, meta)


@pytest.mark.parametrize("ss", [8, 16])
@pytest.mark.parametrize("n,aa1", [(1000, 0), (1100, 0), (2500, 0), (240, 1), (300, 1), (9000, 1)])
def test_clusters(ss, n, aa1):
    assert_same(*run_both(frame(ss, n, aa1)))


@pytest.mark.parametrize("ss", [8, 16])
def test_clusters_with_blend_demotion(ss):
    assert_same(*run_both(frame(ss, 1100, 0, blended=True, hacks={"allow_blend_demote": True})))


@pytest.mark.parametrize("ss", [8, 16])
@pytest.mark.parametrize("w,h", [(8, 8), (33, 17), (96, 96), (104, 96), (152, 128), (160, 128)])
@pytest.mark.parametrize("n,aa1", [(5, 0), (28, 0), (29, 0), (300, 0), (60, 1)])
def test_small_instances(ss, w, h, n, aa1):
    """Up to 152 sub-tiles at 16x, and 304 at 8x from 32 primitives on, are all split."""
    rng = np.random.default_rng(ss * w + n)
    s = gsgen.GifStream()
    gsgen._frame_setup(s, 0, W // 64, gsgen.PSMCT32, ZBP, gsgen.PSMZ24, W, H, gsgen.test_reg(zte=1, ztst=2),
                       alpha=gsgen.alpha_reg(0, 1, 0, 1), extra=[(gsgen.COLCLAMP, 1)])
    s.ad([(gsgen.SCISSOR_1, gsgen.scissor_reg(24, 24 + w - 1, 40, 40 + h - 1))])
    flat_sprites(s, rng, 1, 24, 40)
    cluster(s, rng, n, 20, 36, max(w, h) + 8, aa1=aa1)
    cluster(s, rng, 2, 20, 36, max(w, h) + 8, abe=1)
    assert_same(*run_both(gsgen.Frame("small", s.tobytes(), ss, ss == 16, n + 3, {"width": W, "height": H})))


@pytest.mark.parametrize("ss", [8, 16])
def test_many_coarse_tiles(ss):
    """1120 coarse tiles of 16x16 pixels: the split ones are found 1024 at a time."""
    w, h = 640, 448
    rng = np.random.default_rng(ss)
    s = gsgen.GifStream()
    gsgen._frame_setup(s, 0, w // 64, gsgen.PSMCT32, 140, gsgen.PSMZ24, w, h, gsgen.test_reg(zte=1, ztst=2),
                       alpha=gsgen.alpha_reg(0, 1, 0, 1), extra=[(gsgen.COLCLAMP, 1)])
    n, spots = 1100, ((0, 0), (632, 96), (320, 104), (8, 328), (632, 440))
    x0, y0 = (np.repeat(np.array(spots)[:, k], n) for k in (0, 1))
    x = x0[:, None] * 16 + rng.integers(0, 128, size=(n * len(spots), 3))
    y = y0[:, None] * 16 + rng.integers(0, 128, size=(n * len(spots), 3))
    q = np.zeros((x.size, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(x.size, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), rng.integers(0, 1 << 24, size=x.size))
    for k in range(len(spots)):
        s.packed(gsgen.prim_reg(gsgen.PRIM_TRI, iip=1, abe=k & 1), [gsgen.D_RGBAQ, gsgen.D_XYZ2],
                 q[k * 3 * n:(k + 1) * 3 * n].reshape(-1, 2))
    assert_same(*run_both(gsgen.Frame("spots", s.tobytes(), ss, True, n * len(spots), {"width": w, "height": h})))
