"""Points that share a block with one that is not finite: it alone is computed again with the plain
formulas, and the others' outputs have the bits that they have without it, in every kernel kind (with
contracted multiply-adds the two forms round differently), in blocks of eight points and of other
counts. The point itself has the plain formulas' infinities and NaNs."""
import numpy as np
import pytest

from oracle import oracle as O
from pacuda_b200 import abi, phase_space, processes

from tests.test_gpu_folds import run, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["f64fma", "f64", "mixed", "mixed64"])
@pytest.mark.parametrize("lanes", [64, 32, 80])  # eight, sixteen and six points per block
@pytest.mark.parametrize("name", ["gg>gg", "qg>qgg"])
def test_finite_points_keep_their_bits(name, lanes, kind):
    t = processes.template(name)
    p = phase_space.sample(len(processes.PROCESSES[name]), 41, 12)
    alone = run(t, p, kind, lanes)
    assert np.isfinite(alone).all()
    beside = p.copy()
    bad = [0, 13, 40]  # in three blocks: the first, one in the middle, the last, which is not full
    beside[0, 2, 1] = np.nan
    beside[13] *= 1e200
    beside[40, 3, 2] = np.inf
    got = run(t, beside, kind, lanes)
    with np.errstate(all="ignore"):
        _, want = O.evaluate(t, beside, kernel=abi.KERNELS["f64" if kind == "f64fma" else kind])
    assert not np.isfinite(want[bad]).all(axis=1).any()
    rest = np.setdiff1d(np.arange(len(p)), bad)
    same(got[rest], alone[rest])
    if kind != "f64fma":
        same(got, want)
    else:
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
