"""Transfers and texture decode at every alignment of their four-pixel groups."""
import numpy as np
import pytest

import gsgen
import pgs
import pgs_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["CT32", "CT24", "CT16", "CT16S", "Z16", "T8", "T4", "T8H", "T4HL"])
@pytest.mark.parametrize("sx,dx,w,h", [(0, 0, 1, 1), (3, 2, 5, 3), (4, 8, 33, 33), (2, 1, 31, 40), (1, 2046, 7, 2)])
def test_quads_at_every_alignment(name, sx, dx, w, h):
    """Upload, local copy and decode work on four pixels of a row at a time:
    rectangles that start and end inside a quad, wrap at 2048, and textures
    whose rows are no multiple of four texels, against the oracle."""
    psm = {"Z16": gsgen.PSMZ16, "CT32": gsgen.PSMCT32, "CT24": gsgen.PSMCT24, "CT16": gsgen.PSMCT16, "CT16S": gsgen.PSMCT16S,
           "T8": gsgen.PSMT8, "T4": gsgen.PSMT4, "T8H": gsgen.PSMT8H, "T4HL": 0x24}[name]
    bpp = {"CT32": 32, "CT24": 24, "T8": 8, "T8H": 8, "T4": 4, "T4HL": 4}.get(name, 16)
    rng = np.random.default_rng(w * 64 + dx)
    s = gsgen.GifStream()
    s.upload(0, 32, psm, dx, 1, w, h, rng.integers(0, 256, size=(w * h * bpp + 7) // 8, dtype=np.uint8).tobytes())
    s.upload(1024, 4, psm, 0, 0, 64, 48, rng.integers(0, 256, size=64 * 48 * bpp // 8, dtype=np.uint8).tobytes())
    s.ad([(gsgen.BITBLTBUF, gsgen.bitbltbuf_reg(1024, 4, psm, 2048, 32, psm)),
          (gsgen.TRXPOS, gsgen.trxpos_reg(sx, 2, dx, 3)), (gsgen.TRXREG, gsgen.trxreg_reg(w, h)), (gsgen.TRXDIR, 2)])
    # Draw with the second upload as a texture whose decoded rows are ext wide.
    gsgen._frame_setup(s, 256, 2, gsgen.PSMCT32, 300, gsgen.PSMZ24, 128, 64, gsgen.test_reg(zte=1, ztst=1))
    s.ad([(gsgen.TEX0_1, gsgen.tex0_reg(1024, 4, psm, 1, 5, tfx=1)), (gsgen.TEX1_1, gsgen.tex1_reg(mmag=1)),
          (gsgen.CLAMP_1, gsgen.clamp_reg(2, 2, 0, w % 62 + 1, 0, 31))])
    q = np.zeros((2, 3, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_uv(np.array([0, 63 * 16]), np.array([0, 40 * 16]))
    q[:, 1] = gsgen.q_rgbaq(np.full((2, 4), 128, dtype=np.int64))
    q[:, 2] = gsgen.q_xyz2(np.array([0, 100 * 16]), np.array([0, 60 * 16]), np.zeros(2, dtype=np.int64))
    s.packed(gsgen.prim_reg(gsgen.PRIM_SPRITE, tme=1, fst=1), [gsgen.D_UV, gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
    f = gsgen.Frame("quads", s.tobytes(), 1, True, 1, {"width": 128, "height": 64})
    be = pgs.CudaBackend(0, max_samples_log2=0)
    try:
        out = pgs_oracle.render(f, be)
    finally:
        be.close()
    assert np.array_equal(out, pgs_oracle.render(f))
