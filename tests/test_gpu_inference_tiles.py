"""The fused inference kernel's split: one or two tiles of 128 points in flight per SM give the same
bits (each point's sums have one order), at point counts around a tile, one tile per SM, an odd tile
and several turns."""
import numpy as np
import pytest

from tests.test_gpu_surrogate import INPUTS, _inputs, _net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1, 128, 129])
@pytest.mark.parametrize("tiles_per_sm", [0, 1, 2, 5])
def test_tiles_in_flight_give_the_same_bits(tiles_per_sm, extra):
    import torch

    from oracle import surrogate_oracle as O
    from pacuda_b200 import surrogate as S

    count = 128 * tiles_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    if count < 1:
        pytest.skip("no points")
    net, p = _net(4)
    x = _inputs(count, 6)
    xt, got = torch.tensor(x, device="cuda"), []
    for tiles in (2, 1):
        S.set_inference_blocks(tiles)
        try:
            got.append(net.forward(xt).cpu().numpy())
        finally:
            S.set_inference_blocks(2)
    assert net.error() == 0 and x.shape[1] == INPUTS
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    # the last points (the ragged tile) against the oracle, to the few BF16 ulps of the device's tanh
    want = O.forward(p, x[-300:])
    assert np.max(np.abs(got[0][-300:] - want) / (np.abs(want) + np.sqrt(np.mean(want ** 2)))) < 2e-2
