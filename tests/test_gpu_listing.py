"""The listing's f32 first look, which drops what surely fails and lists what surely passes: at energies
and cuts where its margins are wide, narrow, or cover everything, and where its arithmetic overflows,
the list is that of the f64 restatement (a candidate within 1e-9 of a cut, where the restatement's
rounding decides, would be a difference; none of these samples has one)."""
import numpy as np
import pytest

from oracle import unweight_oracle as U

pytestmark = pytest.mark.gpu

CASES = [  # sqrt(s), (pt_min, eta_max, dr_min)
    (13000.0, (20.0, 5.0, 0.4)),
    (13000.0, (0.3, 8.0, 0.001)),     # cuts within the look's error
    (13000.0, (0.0, 5.0, 0.0)),
    (13000.0, (-20.0, 5.0, -0.4)),    # cut like their sizes
    (13000.0, (20.0, 200.0, 0.4)),    # sinh(eta_max) overflows f32
    (13000.0, (20.0, -1.0, 0.4)),     # nothing passes
    (13000.0, (6000.0, 2.0, 1.5)),
    (91.2, (5.0, 3.0, 0.7)),
    (1e-3, (1e-5, 4.0, 0.4)),
    (1e22, (1e19, 4.0, 0.4)),         # squares overflow f32
]


@pytest.mark.parametrize("sqrt_s,cuts", CASES)
@pytest.mark.parametrize("family,final_state", [("gg>ggg", 3), ("gg>gggg", 4)])
def test_list_is_the_f64_decision(family, final_state, sqrt_s, cuts):
    from pacuda_b200 import unweight

    first, n = 1 << 33, 30001
    pl = unweight.Pipeline(families=[family], sqrt_s=sqrt_s, cuts=cuts, capacity=n)
    got = pl.passing(0, first, n).cpu().numpy().astype(np.uint64)
    idx = np.arange(first, first + n, dtype=np.uint64)
    with np.errstate(all="ignore"):
        p, _ = U.momenta(U.uniforms(pl.family_seed(0), idx, final_state), sqrt_s, final_state)
        want = idx[U.passes(p, *cuts)]
    assert np.array_equal(got, want), (len(got), len(want), np.setdiff1d(want, got)[:5], np.setdiff1d(got, want)[:5])
