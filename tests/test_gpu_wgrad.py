"""Weight and bias gradients at the edges of the tiling: images smaller than a
tile, ragged ones, and more tiles than CTAs."""
import numpy as np
import pytest

import pgs
import upscaler_ref as U

pytestmark = pytest.mark.gpu


def images(seed, n, h, w):
    rng = np.random.default_rng(seed)
    return (rng.integers(0, 256, size=(n, h, w, 4), dtype=np.uint8), rng.integers(0, 256, size=(n, h, w, 4), dtype=np.uint8))


def gradient(img, tgt, params):
    import torch
    up = pgs.Upscaler(0)
    try:
        up.set_params(params)
        loss = up.backward(torch.from_numpy(img).cuda(), torch.from_numpy(tgt).cuda())
        return loss, up.gradient().astype(np.float64)
    finally:
        up.close()


def layers(flat):
    at = 0
    for cin, cout in U.SHAPES:
        for n in (9 * cin * cout, cout):
            yield flat[at:at + n]
            at += n


@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 15, 17), (2, 16, 16), (3, 33, 50), (1, 97, 31)])
def test_ragged_images_match_the_oracle(n, h, w):
    """The two sides differ by BF16 roundings that fall the other way after sums
    in another order: 2^-8 of single activations and gradients, 3 % of a norm."""
    img, tgt = images(n * 1000 + h, n, h, w)
    p = pgs.upscaler_init_params(h)
    loss, g = gradient(img, tgt, p)
    ref_loss, ref = U.backward(img, tgt, p)
    assert abs(loss - ref_loss) < 1e-3 * ref_loss
    for a, b in zip(layers(g), layers(ref.astype(np.float64))):
        assert np.linalg.norm(a - b) < 3e-2 * max(np.linalg.norm(b), 1e-12)


def test_repeated_images_sum_over_all_tiles():
    """32 copies of an image: the output gradient is scaled by exactly 2^-5 and
    the 512 tiles go round the CTAs, so the gradient is the single image's up to
    the order of some 500 FP32 additions (6e-8 each, times 22 for their random
    sum, times 100 for cancellation in an element: 1e-3 of the norm at most)."""
    img, tgt = images(7, 1, 64, 64)
    p = pgs.upscaler_init_params(7)
    _, one = gradient(img, tgt, p)
    _, many = gradient(np.repeat(img, 32, 0), np.repeat(tgt, 32, 0), p)
    for a, b in zip(layers(many), layers(one)):
        assert np.linalg.norm(a - b) < 1e-3 * np.linalg.norm(b)


def test_targets_and_outputs_at_any_byte():
    """Target and output images need no alignment (the input's is four bytes)."""
    import torch
    img, tgt = images(9, 2, 21, 19)
    p = pgs.upscaler_init_params(9)
    loss, g = gradient(img, tgt, p)
    up = pgs.Upscaler(0)
    try:
        up.set_params(p)
        di = torch.from_numpy(img).cuda()
        odd = torch.empty(img.size + 1, dtype=torch.uint8, device="cuda")[1:]
        odd.copy_(torch.from_numpy(tgt.reshape(-1)).cuda())
        assert abs(up.backward(di, odd.view(img.shape)) - loss) <= 1e-12 * loss
        even = torch.empty_like(di)
        up.forward(di, even)
        up.forward(di, odd.view(img.shape))
        up.synchronize()
        assert torch.equal(even.view(-1), odd)
    finally:
        up.close()
