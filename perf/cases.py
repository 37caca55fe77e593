"""What a program does with this framework, as cases that can be timed.

Every case is one pass through the public entry points of pgs.py:

  live     a GIF packet stream of one frame handed to GSInterface, then the
           vsync image or the GS memory read back: an emulator's frame
  replay   a frame recorded once into the backend and replayed as a CUDA graph
           from its starting VRAM, then the picture read out on the device
  batch    several recorded streams of uneven size replayed together
  stream   textures streamed in through HWREG transfers, copied inside GS
           memory and one of them downloaded again
  upscale  the learned upscaler on RGBA8 frames
  train    loss and gradient of the upscaler's training on image crops

The scenes are gsgen's: `plain` (Gouraud triangles, Z test), `textured`
(perspective-textured, alpha-blended, alpha-tested triangles and sprites over
PSMT8 textures), `feedback` (ten passes of mostly tiny triangles that sample
the previous pass's framebuffer).  Heights need not be multiples of a tile;
widths are multiples of 64 because FRAME.FBW is.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "parallel-gs_gb300"))

import gsgen  # noqa: E402
import pgs  # noqa: E402

SAMPLES_LOG2 = {1: 0, 2: 1, 4: 2, 8: 3, 16: 4}
# Pixels covered by a triangle whose area is log-uniform in [4, 4000], and by
# one of the feedback scene (80 % in [1, 16], 20 % in [16, 4000]).
MEAN_AREA = 3996 / math.log(1000)
MEAN_AREA_FEEDBACK = 0.8 * 15 / math.log(16) + 0.2 * 3984 / math.log(250)
# Operations one covered sample cannot do without: three edge values and their
# signs, two barycentrics, the depth and its comparison.
OPS_PER_SAMPLE = 16
UPSCALER_MACS = 9 * (4 * 32 + 4 * 32 * 32 + 32 * 4)


def listed():
    return [
        # A menu or a loading screen at the size of a small game: what counts
        # is the fixed cost of a frame through the whole stack.
        {"name": "live_menu_1x", "kind": "live", "scene": "plain", "prims": 60, "sprites": 0, "width": 320,
         "height": 224, "ss": 1, "out": "vsync"},
        # An emulator's frame at the headline configuration, from host packets
        # to the GS memory in host memory.
        {"name": "live_textured_4x", "kind": "live", "scene": "textured", "prims": 50000, "sprites": 2000,
         "width": 640, "height": 448, "ss": 4, "out": "vram"},
        # A light frame replayed from its recording.
        {"name": "replay_light_1x", "kind": "replay", "scene": "textured", "prims": 500, "sprites": 37, "width": 320,
         "height": 221, "ss": 1},
        # The plain configuration at native rate.
        {"name": "replay_plain_1x", "kind": "replay", "scene": "plain", "prims": 10000, "sprites": 0, "width": 640,
         "height": 448, "ss": 1},
        # An ordinary textured frame at the smallest super-sampling rate and
        # ragged sizes.
        {"name": "replay_textured_2x", "kind": "replay", "scene": "textured", "prims": 12501, "sprites": 499,
         "width": 512, "height": 445, "ss": 2},
        # The headline configuration.
        {"name": "replay_textured_4x", "kind": "replay", "scene": "textured", "prims": 50000, "sprites": 2000,
         "width": 640, "height": 448, "ss": 4},
        # Render-to-texture feedback over many small triangles at high rates.
        {"name": "replay_feedback_8x", "kind": "replay", "scene": "feedback", "prims": 100000, "sprites": 0,
         "width": 640, "height": 448, "ss": 8},
        {"name": "replay_feedback_16x", "kind": "replay", "scene": "feedback", "prims": 100000, "sprites": 0,
         "width": 640, "height": 448, "ss": 16},
        # A server replaying streams of several clients: formats, sizes and
        # rates differ, the small ones share the batched shading kernel.
        {"name": "batch_mixed", "kind": "batch", "streams": 12, "prims_lo": 400, "prims_hi": 20000, "solo": 2000},
        # A loading phase: textures in, moved, and one out again.
        {"name": "stream_textures", "kind": "stream", "psm": "T8", "size_log2": 8, "count": 6},
        # The learned path on one frame.
        {"name": "upscale_frame", "kind": "upscale", "n": 1, "width": 640, "height": 448},
        # A step's gradient as upscaler_train computes it.
        {"name": "train_crops", "kind": "train", "n": 16, "size": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _height(rng, width):
    """A height whose framebuffer's pages gsgen counts exactly: up to 32 * 64 / width
    rows below a multiple of the page height."""
    return 32 * rng.randrange(7, 15) - rng.randrange(0, 32 * 64 // width)


def draw(rng):
    kind = rng.choice(["live", "replay", "replay", "replay", "replay", "batch", "stream", "upscale", "train"])
    if kind in ("live", "replay"):
        scene = rng.choice(["plain", "textured", "textured", "feedback"])
        width = 64 * rng.randrange(5, 11)
        case = {"kind": kind, "scene": scene, "prims": _log_int(rng, 60, 100000 if scene == "feedback" else 50000),
                "sprites": 0, "width": width, "height": _height(rng, width),
                "ss": rng.choice([1, 2, 4, 8, 16] if scene == "feedback" else [1, 2, 4])}
        if scene == "textured":
            case["sprites"] = case["prims"] // rng.randrange(10, 40)
        if kind == "live":
            case["out"] = rng.choice(["vram", "vsync"])
        return case
    if kind == "batch":
        hi = _log_int(rng, 1000, 20000)
        return {"kind": kind, "streams": rng.randrange(2, 13), "prims_lo": _log_int(rng, 60, 400), "prims_hi": hi,
                "solo": rng.choice([0, 1, 2000])}
    if kind == "stream":
        return {"kind": kind, "psm": rng.choice(["CT32", "CT16", "T8", "T4"]), "size_log2": rng.randrange(6, 9),
                "count": rng.randrange(1, 7)}
    if kind == "upscale":
        return {"kind": kind, "n": rng.randrange(1, 4), "width": rng.randrange(64, 641), "height": rng.randrange(64, 449)}
    return {"kind": kind, "n": rng.randrange(1, 17), "size": rng.randrange(48, 129)}


# ---------------------------------------------------------------------------
class State:
    """Handles a program keeps between passes, closed with the state."""

    def __init__(self, case):
        self.case = case
        self.handles = []  # closed in reverse order

    def keep(self, handle):
        self.handles.append(handle)
        return handle

    def __del__(self):
        for h in reversed(self.handles):
            h.close()


def _scene(case, seed):
    size = {"width": case["width"], "height": case["height"]}
    if case["scene"] == "plain":
        return gsgen.frame_c1(seed=seed, num_triangles=case["prims"], **size)
    if case["scene"] == "textured":
        return gsgen.frame_c2(seed=seed, num_triangles=case["prims"], num_sprites=case["sprites"],
                              super_sampling=case["ss"], **size)
    return gsgen.frame_c4(seed=seed, super_sampling=case["ss"], num_triangles=case["prims"], **size)


def _clear(frame):
    """The clear a program draws at the start of a frame: one sprite over the
    framebuffer that writes colour and depth."""
    w, h = frame.meta["width"], frame.meta["height"]
    s = gsgen.GifStream()
    s.ad([(gsgen.PRMODECONT, 1), (gsgen.FRAME_1, gsgen.frame_reg(0, w // 64, gsgen.PSMCT32)),
          (gsgen.ZBUF_1, gsgen.zbuf_reg(frame.meta["zbp"], gsgen.PSMZ24)),
          (gsgen.SCISSOR_1, gsgen.scissor_reg(0, w - 1, 0, h - 1)), (gsgen.XYOFFSET_1, 0),
          (gsgen.TEST_1, gsgen.test_reg(zte=1, ztst=1)), (gsgen.FBA_1, 0), (gsgen.DTHE, 0)])
    q = np.zeros((2, 2, 2), dtype=np.uint64)
    q[:, 0] = gsgen.q_rgbaq(np.zeros((2, 4), dtype=np.int64))
    q[:, 1] = gsgen.q_xyz2(np.array([0, w * 16]), np.array([0, h * 16]), np.zeros(2, dtype=np.int64))
    s.packed(gsgen.prim_reg(gsgen.PRIM_SPRITE), [gsgen.D_RGBAQ, gsgen.D_XYZ2], q.reshape(-1, 2))
    return s.tobytes()


def _prepare_live(case, seed):
    st = State(case)
    frame = _scene(case, seed)
    # The feedback scene at 8x uses the 2x4 sparse grid, everything else ordered grids.
    ordered = frame.ordered if case["scene"] == "feedback" else True
    be = st.keep(pgs.CudaBackend(0, max_samples_log2=SAMPLES_LOG2[case["ss"]], arena_mib=64))
    st.gs = st.keep(pgs.GSInterface(be, super_sampling=case["ss"], ordered=ordered))
    st.data = _clear(frame) + frame.data
    if case["out"] == "vsync":
        st.gs.write_priv_register("PMODE", gsgen.pmode_reg(en1=1, en2=0))
        st.gs.write_priv_register("SMODE1", gsgen.smode1_reg(cmod=2))
        st.gs.write_priv_register("SMODE2", gsgen.smode2_reg(interlace=1, ffmd=0))
        st.gs.write_priv_register("DISPFB1", gsgen.dispfb_reg(0, case["width"] // 64, gsgen.PSMCT32))
        st.gs.write_priv_register("DISPLAY1", gsgen.display_reg(636, 50, 3, 0, case["width"] * 4 - 1,
                                                                case["height"] - 1))
    else:
        st.vram = torch.empty(pgs.VRAM_SIZE, dtype=torch.uint8, pin_memory=True).numpy()
    return st


def _run_live(st):
    st.gs.gif_transfer(0, st.data)
    if st.case["out"] == "vsync":
        image, _ = st.gs.vsync(0, 0)
        return image
    return st.gs.read_vram(out=st.vram)


def _record(st, frame, arena_mib):
    be = st.keep(pgs.CudaBackend(0, max_samples_log2=SAMPLES_LOG2[frame.super_sampling], arena_mib=arena_mib))
    gs = pgs.GSInterface(be, super_sampling=frame.super_sampling, ordered=frame.ordered)
    be.begin_record()
    gs.gif_transfer(0, frame.data)
    gs.flush()
    be.end_record()
    gs.close()
    return be


def _prepare_replay(case, seed):
    st = State(case)
    frame = _scene(case, seed)
    frame.super_sampling = case["ss"]
    st.be = _record(st, frame, 64)
    st.image = torch.empty((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
    return st


def _run_replay(st):
    c = st.case
    st.be.replay(1)
    st.be.sample_circuit(st.image.data_ptr(), 0, c["width"] // 64, gsgen.PSMCT32, c["width"], c["height"])
    return st.image


def _batch_prims(case):
    n, lo, hi = case["streams"], case["prims_lo"], case["prims_hi"]
    return [int(round(lo * (hi / lo) ** (i / max(1, n - 1)))) for i in range(n)]


def _prepare_batch(case, seed):
    st = State(case)
    st.streams = []
    for i, prims in enumerate(_batch_prims(case)):
        frame = gsgen.stream_c3((seed * 16 + i) % (1 << 40), num_primitives=prims)
        # Every client's picture goes to a display of one size, 640x512, the largest frame there is.
        image = torch.empty((512, 640, 4), dtype=torch.uint8, device="cuda")
        st.streams.append((_record(st, frame, 8), image, frame.meta))
    st.batch = st.keep(pgs.Batch(0))
    for be, _, _ in st.streams:
        st.batch.add(be)
    # Streams of `solo` primitives and more are branches of the graph, the others share the rounds.
    st.batch.set_tuning(256, 4, True, case["solo"])
    return st


def _run_batch(st):
    st.batch.replay(1)
    st.batch.synchronize()
    for be, image, m in st.streams:
        be.sample_circuit(image.data_ptr(), m["fbp"], m["width"] // 64, m["fpsm"], 640, 512)
    return [image for _, image, _ in st.streams]


STREAM_PSM = {"CT32": (gsgen.PSMCT32, 32), "CT16": (gsgen.PSMCT16, 16), "T8": (gsgen.PSMT8, 8), "T4": (gsgen.PSMT4, 4)}


def _prepare_stream(case, seed):
    st = State(case)
    be = st.keep(pgs.CudaBackend(0, max_samples_log2=0, arena_mib=64))
    st.gs = st.keep(pgs.GSInterface(be, super_sampling=1))
    psm, bpp = STREAM_PSM[case["psm"]]
    rng = np.random.Generator(np.random.PCG64(seed))
    w = h = 1 << case["size_log2"]
    tbw = max(1, w // 64) if bpp > 8 else max(2, w // 64)
    pages = max(1, w * h * bpp // 8 // gsgen.PAGE_BYTES) * (2 if bpp <= 8 and w < 128 else 1)
    s = gsgen.GifStream()
    for i in range(case["count"]):
        data = rng.integers(0, 256, size=w * h * bpp // 8, dtype=np.uint8).tobytes()
        s.upload(i * pages * gsgen.BLOCKS_PER_PAGE, tbw, psm, 0, 0, w, h, data)
    # The last one, less its first 16 columns and 8 rows, is copied to a place behind all of them.
    src, dst = (case["count"] - 1) * pages, case["count"] * pages
    st.last = dict(sbp=dst * gsgen.BLOCKS_PER_PAGE, sbw=tbw, spsm=psm)
    s.ad([(gsgen.BITBLTBUF, gsgen.bitbltbuf_reg(sbp=src * gsgen.BLOCKS_PER_PAGE, sbw=tbw, spsm=psm,
                                                dbp=dst * gsgen.BLOCKS_PER_PAGE, dbw=tbw, dpsm=psm)),
          (gsgen.TRXPOS, gsgen.trxpos_reg(ssax=16, ssay=8, dsax=0, dsay=0)),
          (gsgen.TRXREG, gsgen.trxreg_reg(w - 16, h - 8)), (gsgen.TRXDIR, 2)])
    # Download: PSMT4 cannot be transferred out, as on the hardware, so the
    # same bytes are read as PSMT8.
    down = gsgen.PSMT8 if psm == gsgen.PSMT4 else psm
    down_h = h // 2 if psm == gsgen.PSMT4 else h
    s.ad([(gsgen.BITBLTBUF, gsgen.bitbltbuf_reg(sbp=dst * gsgen.BLOCKS_PER_PAGE, sbw=tbw, spsm=down)),
          (gsgen.TRXPOS, gsgen.trxpos_reg()), (gsgen.TRXREG, gsgen.trxreg_reg(w, down_h)), (gsgen.TRXDIR, 1)])
    st.qwords = w * h * bpp // 8 // 16
    st.data = s.tobytes()
    st.vram = torch.empty(pgs.VRAM_SIZE, dtype=torch.uint8, pin_memory=True).numpy()
    return st


def _run_stream(st):
    st.gs.gif_transfer(0, st.data)
    texture = st.gs.read_transfer_fifo(st.qwords)
    return [np.frombuffer(texture, dtype=np.uint8), st.gs.read_vram(out=st.vram)]


def _images(gen, n, h, w):
    """RGBA8 frames with flat areas, gradients and hard edges, as renders have."""
    y = torch.arange(h, device="cuda", dtype=torch.float32).view(1, h, 1, 1)
    x = torch.arange(w, device="cuda", dtype=torch.float32).view(1, 1, w, 1)
    f = torch.rand((n, 8, 4), generator=gen, device="cuda")
    img = torch.zeros((n, h, w, 4), device="cuda")
    for k in range(8):
        a = f[:, k]
        ramp = torch.sin((x * (a[:, 0] - 0.5).view(n, 1, 1, 1) + y * (a[:, 1] - 0.5).view(n, 1, 1, 1)) * 0.4)
        img = torch.where(ramp > (a[:, 2] * 2 - 1).view(n, 1, 1, 1), a.view(n, 1, 1, 4) * 0.7 + ramp * 0.3, img)
    noise = torch.rand((n, h, w, 4), generator=gen, device="cuda")
    return ((img * 0.8 + noise * 0.2).clamp(0, 1) * 255).to(torch.uint8)


def _params(seed, train):
    if not train:
        return np.load(Path(pgs.__file__).resolve().parent / "upscaler_weights.npy")
    return pgs.upscaler_init_params(seed)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _train_images(case, seed):
    gen = _generator(seed)
    return (_images(gen, case["n"], case["size"], case["size"]), _images(gen, case["n"], case["size"], case["size"]))


def _prepare_upscale(case, seed):
    st = State(case)
    st.up = st.keep(pgs.Upscaler(0))
    st.up.set_params(_params(seed, False))
    st.images = _images(_generator(seed), case["n"], case["height"], case["width"])
    st.out = torch.empty_like(st.images)
    torch.cuda.synchronize()
    return st


def _run_upscale(st):
    st.up.forward(st.images, st.out)
    return st.out


def _prepare_train(case, seed):
    st = State(case)
    st.up = st.keep(pgs.Upscaler(0))
    st.up.set_params(_params(seed, True))
    st.images, st.targets = _train_images(case, seed)
    torch.cuda.synchronize()
    return st


def _run_train(st):
    loss = st.up.backward(st.images, st.targets)
    return {"loss": loss, "gradient": st.up.gradient()}


KINDS = {"live": (_prepare_live, _run_live), "replay": (_prepare_replay, _run_replay),
         "batch": (_prepare_batch, _run_batch), "stream": (_prepare_stream, _run_stream),
         "upscale": (_prepare_upscale, _run_upscale), "train": (_prepare_train, _run_train)}


def prepare(case, seed):
    return KINDS[case["kind"]][0](case, seed)


def run(state):
    return KINDS[state.case["kind"]][1](state)


def work(case):
    kind = case["kind"]
    if kind in ("live", "replay"):
        px, prims, ss = case["width"] * case["height"], case["prims"] + case["sprites"], case["ss"]
        feedback = case["scene"] == "feedback"
        # Colour and depth of every sample out (and, with samples, the resolved
        # and the reference plane), 152 bytes per primitive record and the
        # textures in, the read-out.
        planes = ss + (2 if ss > 1 else 0)
        passes = 10 if feedback else 1
        textures = {"plain": 0, "textured": 8 * (65536 + 1024), "feedback": 4 * (16384 + 1024)}[case["scene"]]
        out = pgs.VRAM_SIZE if case.get("out") == "vram" else 4 * px
        return {"bytes": passes * 8 * px * planes + 152 * prims + textures + out,
                "flops": OPS_PER_SAMPLE * ss * prims * (MEAN_AREA_FEEDBACK if feedback else MEAN_AREA)}
    if kind == "batch":
        # The streams' mean size and rate: 480x384 at 16 or 32 bits, 1x to 4x.
        prims, px = sum(_batch_prims(case)), 480 * 384
        return {"bytes": 152 * prims + case["streams"] * (px * 6 * 3 + 4 * 640 * 512),
                "flops": OPS_PER_SAMPLE * 7 / 3 * prims * MEAN_AREA * px / (640 * 448)}
    if kind == "stream":
        size = STREAM_PSM[case["psm"]][1] << (2 * case["size_log2"])
        return {"bytes": (2 * case["count"] + 4) * size // 8 + pgs.VRAM_SIZE, "flops": 0}
    px = case["n"] * (case["width"] * case["height"] if kind == "upscale" else case["size"] ** 2)
    if kind == "upscale":
        return {"bytes": 8 * px, "flops": 2 * UPSCALER_MACS * px}
    # Forward, weight gradients, and data gradients of all layers but the first.
    return {"bytes": 8 * px + 4 * sum(9 * a * b + b for a, b in pgs.UPSCALER_SHAPES),
            "flops": 2 * px * (3 * UPSCALER_MACS - 9 * 4 * 32)}


def exact(case, seed):
    """Loss and gradient of the training case in 64 bits; everything else
    returns whole numbers."""
    if case["kind"] != "train":
        return None
    images, targets = _train_images(case, seed)
    flat = torch.from_numpy(_params(seed, True)).cuda().double()
    layers, at = [], 0
    for cin, cout in pgs.UPSCALER_SHAPES:
        w = flat[at:at + 9 * cin * cout].view(9, cout, cin).detach().requires_grad_()
        at += 9 * cin * cout
        b = flat[at:at + cout].detach().requires_grad_()
        at += cout
        layers.append((w, b))
    x = images.permute(0, 3, 1, 2).double() / 255
    a = x
    for k, (w, b) in enumerate(layers):
        a = torch.nn.functional.conv2d(a, w.view(3, 3, *w.shape[1:]).permute(2, 3, 0, 1), b, padding=1)
        if k + 1 < len(layers):
            a = torch.relu(a)
    loss = ((a + x - targets.permute(0, 3, 1, 2).double() / 255) ** 2).mean()
    grads = torch.autograd.grad(loss, [p for layer in layers for p in layer])
    return {"loss": loss.item(), "gradient": torch.cat([g.reshape(-1) for g in grads]).cpu().numpy()}
