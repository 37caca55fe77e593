"""32 -> 32 layers with three stages of input and with five, at the tile count
where one takes over from the other.  A frame's result does not depend on the
frames beside it, so a batch one tile larger must give the same bytes."""
import numpy as np
import pytest

import pgs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas_per_sm", [1, 2])
@pytest.mark.parametrize("h,w", [(16, 8), (13, 7)])
def test_few_and_many_tiles(ctas_per_sm, h, w):
    import torch
    few = 6 * torch.cuda.get_device_properties(0).multi_processor_count  # one tile per image
    rng = np.random.default_rng(few + h)
    img = torch.from_numpy(rng.integers(0, 256, size=(few + 1, h, w, 4), dtype=np.uint8)).cuda()
    up = pgs.Upscaler(0)
    try:
        up.set_params(pgs.upscaler_init_params(7))
        up.set_tensor_path(ctas_per_sm)
        outs = []
        for part in (img, img[:few], img[few:]):
            outs.append(torch.empty_like(part))
            up.forward(part, outs[-1])
        up.synchronize()
        assert up.error_flags() == 0
    finally:
        up.close()
    assert torch.equal(outs[0][:few], outs[1]) and torch.equal(outs[0][few:], outs[2])
