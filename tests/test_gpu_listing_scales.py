"""The listing's f32 first look at energies whose products leave f32's range, on either side of where the look
stops deciding: the list is that of the f64 restatement."""
import numpy as np
import pytest

from oracle import unweight_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sqrt_s", [1e-26, 1e-23, 3e-22, 1e-21, 1e-20, 1e-19, 1e-16, 0.9e-15, 1.1e-15, 1e-12, 0.9e-9, 1.1e-9,
                                    1e-6, 1e6, 0.9e12, 1.1e12, 1e13, 1e14, 0.9e15, 1.1e15, 1e18, 3e18, 1e19, 1e20])
@pytest.mark.parametrize("family,final_state", [("gg>ggg", 3), ("gg>gggg", 4)])
def test_list_is_the_f64_decision(family, final_state, sqrt_s):
    from pacuda_b200 import unweight

    first, n, cuts = 1 << 33, 30001, (0.02 * sqrt_s, 4.0, 0.4)
    pl = unweight.Pipeline(families=[family], sqrt_s=sqrt_s, cuts=cuts, capacity=n)
    got = pl.passing(0, first, n).cpu().numpy().astype(np.uint64)
    idx = np.arange(first, first + n, dtype=np.uint64)
    p, _ = U.momenta(U.uniforms(pl.family_seed(0), idx, final_state), sqrt_s, final_state)
    want = idx[U.passes(p, *cuts)]
    assert 100 < len(want) < n
    assert np.array_equal(got, want), (len(got), len(want))
