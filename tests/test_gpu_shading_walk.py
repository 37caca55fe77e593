"""Shading walk against the oracle where it can go wrong: list lengths around
the shared-lane, batch and list-capacity edges, depths one step apart under
every depth test and format, untested depth writes between tested ones,
SCANMSK, edges longer than the depth bound accepts, and every alpha test, blend
operand and wrap mode of the sampling and blending code.  All results are
integers: every VRAM plane and the covered-sample count must be equal."""
import numpy as np
import pytest

import gsgen
import pgs
import pgs_oracle
from test_gpu_parity import assert_same, run_both

pytestmark = pytest.mark.gpu

W, H, ZBP = 128, 96, 64
ZMAX = {gsgen.PSMZ32: (1 << 32) - 1, gsgen.PSMZ24: (1 << 24) - 1, gsgen.PSMZ16: (1 << 16) - 1}


def setup(s, fpsm, zpsm, extra=()):
    gsgen._frame_setup(s, 0, W // 64, fpsm, ZBP, zpsm, W, H, gsgen.test_reg(zte=1, ztst=2),
                       alpha=gsgen.alpha_reg(0, 1, 0, 1), extra=[(gsgen.COLCLAMP, 1), *extra])


def triangles(s, rng, n, x0, y0, size, z, prim=gsgen.PRIM_TRI, abe=0):
    """n primitives inside the square at (x0, y0) with the given vertex depths."""
    k = 3 if prim == gsgen.PRIM_TRI else 2
    x = rng.integers(x0 * 16, (x0 + size) * 16 + 1, size=(n, k))
    y = rng.integers(y0 * 16, (y0 + size) * 16 + 1, size=(n, k))
    q = np.zeros((n * k, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(n * k, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), np.asarray(z, dtype=np.int64)[:, :k].reshape(-1))
    s.packed(gsgen.prim_reg(prim, iip=1, abe=abe), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))


def frame(s, ss, ordered=True, n=0):
    return gsgen.Frame("walk", s.tobytes(), ss, ordered, n, {"width": W, "height": H})


@pytest.mark.parametrize("ss,ordered", [(1, True), (2, True), (4, True), (4, False), (8, False), (16, True), (16, False)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 31, 33, 2049])
def test_list_lengths(ss, ordered, n):
    """One 8x8 sub-tile's list of n primitives, larger neighbours around it."""
    rng = np.random.default_rng(n)
    s = gsgen.GifStream()
    setup(s, gsgen.PSMCT32, gsgen.PSMZ24)
    triangles(s, rng, n, 8, 8, 8, rng.integers(0, 1 << 24, size=(n, 3)))
    triangles(s, rng, 5, 0, 0, 96, rng.integers(0, 1 << 24, size=(5, 3)), abe=1)
    triangles(s, rng, 3, 4, 4, 30, rng.integers(0, 1 << 24, size=(3, 3)), prim=gsgen.PRIM_SPRITE)
    assert_same(*run_both(frame(s, ss, ordered, n + 8)))


@pytest.mark.parametrize("ss", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("zpsm", sorted(ZMAX))
def test_depths_one_step_apart(ss, zpsm):
    """Near-coplanar stacks at the bottom, middle and top of the depth range,
    with untested depth writes and blended primitives in between."""
    rng = np.random.default_rng(ss)
    zmax = ZMAX[zpsm]
    fpsm = gsgen.PSMCT16 if zpsm == gsgen.PSMZ16 else gsgen.PSMCT32
    s = gsgen.GifStream()
    setup(s, fpsm, zpsm)
    total = 0
    for base in (0, zmax // 2, zmax - 8):
        for ztst in (2, 3, 1, 2):
            for zmsk in (0, 1):
                s.ad([(gsgen.TEST_1, gsgen.test_reg(zte=1, ztst=ztst)),
                      (gsgen.ZBUF_1, gsgen.zbuf_reg(ZBP, zpsm, zmsk))])
                n = 70 if ztst != 1 else 3
                flat = base + rng.integers(0, 8, size=(n, 1)) + np.zeros((n, 3), dtype=np.int64)
                tilted = base + rng.integers(0, 8, size=(n, 3))
                steep = np.stack([np.full(n, base), rng.integers(0, zmax + 1, size=n), np.full(n, zmax)], 1)
                for k, z in enumerate((flat, tilted, steep)):
                    triangles(s, rng, n, 3, 5, 40, z, abe=k & 1)
                    total += n
    assert_same(*run_both(frame(s, ss, ss != 8, total)))


@pytest.mark.parametrize("ss", [1, 4, 16])
def test_scanmsk_and_long_edges(ss):
    rng = np.random.default_rng(3)
    s = gsgen.GifStream()
    setup(s, gsgen.PSMCT32, gsgen.PSMZ32)
    for mask in (0, 2, 3):
        s.ad([(gsgen.SCANMSK, mask)])
        triangles(s, rng, 40, 0, 0, 90, rng.integers(0, 1 << 32, size=(40, 3)))
        triangles(s, rng, 10, 0, 0, 90, rng.integers(0, 1 << 32, size=(10, 3)), prim=gsgen.PRIM_SPRITE)
        # Edges up to 4095 pixels: past what the depth bound takes.
        triangles(s, rng, 40, 0, 0, 4095, rng.integers(0, 1 << 32, size=(40, 3)))
        # Slivers: a huge change of the barycentrics across the block.
        z = rng.integers(0, 1 << 32, size=(40, 3))
        x = rng.integers(0, 90 * 16, size=(40, 1)) + np.array([[0, 1, 700]])
        y = rng.integers(0, 90 * 16, size=(40, 1)) + np.array([[0, 1, 690]])
        q = np.zeros((120, 2, 2), dtype=np.uint64)
        q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(120, 4), dtype=np.int64))
        q[:, 1] = gsgen.q_xyz2(x.reshape(-1), y.reshape(-1), z.reshape(-1))
        s.packed(gsgen.prim_reg(gsgen.PRIM_TRI, iip=1), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
    assert_same(*run_both(frame(s, ss, True, 390)))


@pytest.mark.parametrize("fpsm", [gsgen.PSMCT32, gsgen.PSMCT24, gsgen.PSMCT16])
@pytest.mark.parametrize("ss", [1, 4])
def test_blend_alpha_and_wrap_states(fpsm, ss):
    rng = np.random.default_rng(fpsm)
    s = gsgen.GifStream()
    zpsm = gsgen.PSMZ16 if fpsm == gsgen.PSMCT16 else gsgen.PSMZ24
    setup(s, fpsm, zpsm, extra=[(gsgen.DTHE, 1), (gsgen.DIMX, gsgen.dimx_reg(gsgen.DEFAULT_DIMX))])
    tex0s, _ = gsgen._texture_set(rng, s, 128, 2, 6, 6, gsgen.PSMT8)
    total = 0
    for i in range(160):
        s.ad([(gsgen.TEX0_1, tex0s[i & 1] ^ (int(rng.integers(0, 4)) << 35)),
              (gsgen.TEST_1, gsgen.test_reg(ate=int(i % 3 != 0), atst=i & 7, aref=int(rng.integers(0, 256)),
                                            afail=(i >> 3) & 3, date=int(i % 5 == 0), datm=i & 1, zte=1, ztst=2)),
              (gsgen.ALPHA_1, gsgen.alpha_reg(*(int(v) for v in rng.integers(0, 3, size=4)), int(rng.integers(0, 256)))
               if i % 4 else gsgen.alpha_reg(0, 1, 0, 1)),
              (gsgen.COLCLAMP, int(i % 7 != 0)), (gsgen.PABE, int(i % 11 == 0)), (gsgen.FBA_1, i & 1),
              (gsgen.FRAME_1, gsgen.frame_reg(0, W // 64, fpsm, int(rng.integers(0, 1 << 32)) if i % 9 == 0 else 0)),
              (gsgen.TEX1_1, gsgen.tex1_reg(mmag=(i >> 1) & 1)),
              (gsgen.CLAMP_1, gsgen.clamp_reg(i & 3, (i >> 2) & 3, int(rng.integers(0, 64)), int(rng.integers(0, 64)),
                                              int(rng.integers(0, 64)), int(rng.integers(0, 64))))])
        n = 4
        x = rng.integers(0, W * 16, size=(n * 3,))
        y = rng.integers(0, H * 16, size=(n * 3,))
        qv = rng.uniform(0.25, 4.0, size=n * 3).astype(np.float32)
        st = rng.uniform(-2.0, 3.0, size=(2, n * 3)).astype(np.float32)
        q = np.zeros((n * 3, 3, 2), dtype=np.uint64)
        fst = (i >> 4) & 1
        q[:, 0] = gsgen.q_uv(rng.integers(0, 1 << 14, size=n * 3), rng.integers(0, 1 << 14, size=n * 3)) if fst else \
            gsgen.q_st(st[0] * qv, st[1] * qv, qv)
        q[:, 1] = gsgen.q_rgbaq(rng.integers(0, 256, size=(n * 3, 4), dtype=np.int64))
        q[:, 2] = gsgen.q_xyz2(x, y, rng.integers(0, 1 << 16, size=n * 3))
        s.packed(gsgen.prim_reg(gsgen.PRIM_TRI, iip=i & 1, tme=1, abe=int(i % 6 != 0), fst=fst),
                 [gsgen.D_UV if fst else gsgen.D_ST, gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
        total += n
    assert_same(*run_both(frame(s, ss, True, total)))


@pytest.mark.parametrize("cta_threads", [128, 256, 512])
def test_batched_rounds(cta_threads):
    """Streams of every rate share the rounds: single-sampled tiles inside a
    super-sampled stream, a sub-tile's list past the batched kernel's 512 and the
    mask words past one chunk of 64 threads (8192 primitives)."""
    rng = np.random.default_rng(cta_threads)
    frames = []
    for ss, ordered, n in ((1, True, 8300), (2, True, 700), (4, False, 600), (4, True, 40)):
        s = gsgen.GifStream()
        setup(s, gsgen.PSMCT32, gsgen.PSMZ24)
        triangles(s, rng, n, 8, 8, 8, rng.integers(0, 1 << 24, size=(n, 3)))
        triangles(s, rng, 9, 0, 0, 96, rng.integers(0, 1 << 24, size=(9, 3)), abe=1)
        # Flat sprites on pixel boundaries, away from the rest: tiles that need one sample.
        x = np.array([[100, 126]] * 3) * 16
        q = np.zeros((6, 2, 2), dtype=np.uint64)
        q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(6, 4), dtype=np.int64))
        q[:, 1] = gsgen.q_xyz2(x.reshape(-1), x.reshape(-1) - 40 * 16, np.full(6, 77))
        s.packed(gsgen.prim_reg(gsgen.PRIM_SPRITE), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
        frames.append(frame(s, ss, ordered, n + 12))
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


@pytest.mark.parametrize("ss", [1, 8, 16])
def test_lists_of_several_chunks(ss):
    """33,000 primitives: more than 1024 mask words, so lists come in chunks, also
    where a CTA runs several parts of a sub-tile."""
    rng = np.random.default_rng(ss)
    s = gsgen.GifStream()
    setup(s, gsgen.PSMCT32, gsgen.PSMZ24)
    n = 33000
    x = rng.integers(0, W * 16, size=(n, 1)) + rng.integers(-40, 41, size=(n, 3))
    y = rng.integers(0, H * 16, size=(n, 1)) + rng.integers(-40, 41, size=(n, 3))
    q = np.zeros((n * 3, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(rng.integers(0, 256, size=(n * 3, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(np.clip(x, 0, W * 16).reshape(-1), np.clip(y, 0, H * 16).reshape(-1), rng.integers(0, 1 << 24, size=n * 3))
    s.packed(gsgen.prim_reg(gsgen.PRIM_TRI, iip=1), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
    assert_same(*run_both(frame(s, ss, True, n)))
