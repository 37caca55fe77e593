"""The shading walk of passes with AA1 primitives, mip-mapped or super-sampled
textures against the oracle, at list lengths around its capacities: more than a
batch of 32, than the 2048 indices held at a time and than the 1024 mask words
of a chunk, at every rate, so also where a CTA runs a sub-tile's parts one after
the other (8x and 16x) and in the batched kernel's groups.  The primitives are a
few pixels large: a warp that culls by another warp's rectangle, or by one that
is not written yet, loses some.  Every plane and the covered-sample count must
be equal."""
import numpy as np
import pytest

import gsgen
import pgs
import pgs_oracle
from test_gpu_parity import assert_same, run_both

pytestmark = pytest.mark.gpu

W, H, ZBP, TEX_PAGE = 128, 96, 64, 96


def setup(s):
    gsgen._frame_setup(s, 0, W // 64, gsgen.PSMCT32, ZBP, gsgen.PSMZ24, W, H, gsgen.test_reg(zte=1, ztst=2),
                       alpha=gsgen.alpha_reg(0, 1, 0, 1), extra=[(gsgen.COLCLAMP, 1)])


def positions(rng, n, k):
    """Vertices of n primitives: up to some thousand in one sub-tile and every
    seventh over its neighbours, more of them 5 pixels large all over the frame."""
    if n > 4096:
        x = rng.integers(0, W * 16, size=(n, 1)) + rng.integers(-40, 41, size=(n, k))
        y = rng.integers(0, H * 16, size=(n, 1)) + rng.integers(-40, 41, size=(n, k))
    else:
        size = np.where(np.arange(n) % 7 == 6, 24, 8)[:, None] * 16
        x = 8 * 16 + (rng.uniform(size=(n, k)) * size).astype(np.int64)
        y = 8 * 16 + (rng.uniform(size=(n, k)) * size).astype(np.int64)
    return np.clip(x, 0, W * 16 - 1), np.clip(y, 0, H * 16 - 1)


def draw(s, rng, n, prim, **flags):
    k = 3 if prim == gsgen.PRIM_TRI else 2
    x, y = positions(rng, n, k)
    words = [gsgen.q_rgbaq(rng.integers(0, 256, size=(n * k, 4), dtype=np.int64))]
    desc = [gsgen.D_RGBAQ]
    if flags.get("tme"):
        q = rng.uniform(0.25, 4.0, size=n * k).astype(np.float32)
        st = rng.uniform(-1.0, 2.0, size=(2, n * k)).astype(np.float32)
        words.insert(0, gsgen.q_st(st[0] * q, st[1] * q, q))
        desc.insert(0, gsgen.D_ST)
    words.append(gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), rng.integers(0, 1 << 24, size=n * k)))
    desc.append(gsgen.D_XYZ2)
    s.packed(gsgen.prim_reg(prim, iip=1, **flags), desc, np.stack(words, axis=1).reshape(-1, 2))


def aa1_frame(ss, ordered, n, seed):
    rng = np.random.default_rng(seed)
    s = gsgen.GifStream()
    setup(s)
    draw(s, rng, n - n // 3 - n // 4, gsgen.PRIM_TRI, aa1=1)
    draw(s, rng, n // 3, gsgen.PRIM_LINE, aa1=1, abe=1)
    draw(s, rng, n // 4, gsgen.PRIM_TRI, abe=1)
    draw(s, rng, 3, gsgen.PRIM_SPRITE)
    return gsgen.Frame("aa1_walk", s.tobytes(), ss, ordered, n + 3, {"width": W, "height": H})


def mip_frame(ss, ordered, n, seed):
    rng = np.random.default_rng(seed)
    s = gsgen.GifStream()
    levels = []
    for lv in range(4):
        size = 64 >> lv
        levels.append(((TEX_PAGE + 2 * lv) * gsgen.BLOCKS_PER_PAGE, 1))
        s.upload(*levels[lv], gsgen.PSMCT32, 0, 0, size, size, rng.integers(0, 256, size=size * size * 4, dtype=np.uint8).tobytes())
    setup(s)
    s.ad([(gsgen.TEX0_1, gsgen.tex0_reg(*levels[0], gsgen.PSMCT32, 6, 6)),
          (gsgen.TEX1_1, gsgen.tex1_reg(mxl=3, mmag=1, mmin=5, l=0, k=0)),
          (gsgen.MIPTBP1_1, gsgen.miptbp_reg(levels[1:4])), (gsgen.CLAMP_1, gsgen.clamp_reg(0, 1))])
    draw(s, rng, n - n // 3, gsgen.PRIM_TRI, tme=1)
    draw(s, rng, n // 3, gsgen.PRIM_SPRITE, tme=1, abe=1)
    return gsgen.Frame("mip_walk", s.tobytes(), ss, ordered, n, {"width": W, "height": H})


def layered_frame(ss, ordered, n, seed):
    """Sprites that sample, sample by sample, what a super-sampled pass drew."""
    rng = np.random.default_rng(seed)
    s = gsgen.GifStream()
    setup(s)
    m = 200
    x, y = gsgen.random_triangles(rng, m, W, H, 8.0, 1500.0)
    q = np.zeros((m * 3, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(m * 3, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), rng.integers(0, 1 << 24, size=m * 3))
    s.packed(gsgen.prim_reg(gsgen.PRIM_TRI, iip=1), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
    s.ad([(gsgen.FRAME_1, gsgen.frame_reg(TEX_PAGE, W // 64, gsgen.PSMCT32)),
          (gsgen.ZBUF_1, gsgen.zbuf_reg(ZBP, gsgen.PSMZ24, 1)), (gsgen.TEST_1, gsgen.test_reg(zte=1, ztst=1)),
          (gsgen.TEX0_1, gsgen.tex0_reg(0, W // 64, gsgen.PSMCT32, 7, 7, tcc=1, tfx=1)),
          (gsgen.TEX1_1, gsgen.tex1_reg(mmag=0)), (gsgen.CLAMP_1, gsgen.clamp_reg(1, 1))])
    x, y = positions(rng, n, 2)
    x, y = np.sort(x, axis=1), np.sort(y, axis=1)
    q = np.zeros((n * 2, 3, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(np.full((n * 2, 4), 0x80, dtype=np.int64))
    q[:, 1] = gsgen.q_uv(x.reshape(-1), y.reshape(-1))
    q[:, 2] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), np.zeros(n * 2, dtype=np.int64))
    s.packed(gsgen.prim_reg(gsgen.PRIM_SPRITE, tme=1, fst=1, abe=1), [gsgen.D_RGBAQ, gsgen.D_UV, gsgen.D_XYZ2], q.reshape(-1, 2))
    return gsgen.Frame("layered_walk", s.tobytes(), ss, ordered, m + n, {"width": W, "height": H, "ssaa_textures": True})


@pytest.mark.parametrize("n", [33, 2300, 36000])
@pytest.mark.parametrize("ss,ordered", [(1, True), (2, True), (4, True), (8, False), (16, True)])
@pytest.mark.parametrize("scene", [aa1_frame, mip_frame], ids=["aa1", "mip"])
def test_culled_walk(scene, ss, ordered, n):
    assert_same(*run_both(scene(ss, ordered, n, ss + n)))


@pytest.mark.parametrize("n", [70, 2300, 36000])
@pytest.mark.parametrize("ss,ordered", [(4, True), (8, False), (16, True)])
def test_culled_walk_layered(ss, ordered, n):
    assert_same(*run_both(layered_frame(ss, ordered, n, ss + n)))


@pytest.mark.parametrize("cta_threads", [128, 256, 512])
def test_batched_rounds_aa1(cta_threads):
    """The batched kernel's groups hold 512 indices and chunks of 256 mask words
    per 64 threads."""
    frames = [aa1_frame(ss, True, n, cta_threads + ss) for ss, n in ((1, 8300), (2, 2000), (4, 2000), (4, 36000))]
    backends, batch = [], pgs.Batch(0)
    try:
        for f in frames:
            be = pgs.CudaBackend(0, max_samples_log2=2)
            backends.append(be)
            gs = pgs.GSInterface(be, super_sampling=f.super_sampling, ordered=f.ordered)
            be.begin_record()
            gs.gif_transfer(0, f.data)
            gs.flush()
            be.end_record()
            gs.close()
            batch.add(be)
        batch.set_tuning(cta_threads, 1024 // cta_threads, True, 0)
        batch.replay(1)
        batch.synchronize()
        for be, f in zip(backends, frames):
            ref = pgs_oracle.render(f, planes=True)
            assert_same(ref, np.stack([be.read_plane(p) for p in range(ref.shape[0])]))
    finally:
        batch.close()
        for be in backends:
            be.close()
