"""The items of the on-chip executor's blocks: fewer than the blocks, a few rounds of them and one over,
for two plans in one launch, with points that are computed twice (not finite) among them; each
output equals the oracle's bit for bit, run after run."""
import numpy as np
import pytest

from oracle import oracle as O
from pacuda_b200 import abi, phase_space, processes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["f64", "df64", "mixed", "mixed64"])
@pytest.mark.parametrize("counts", [(1, 1), (3, 140), (148, 445)])
def test_every_item_once(counts, kind):
    import torch

    from pacuda_b200 import batch as B

    plans, inputs, outs, want = [], [], [], []
    for name, n in zip(("gg>gg", "qq~>gg"), counts):
        t = processes.template(name)
        p = phase_space.sample(4, n, 11)
        p[n // 2] *= 1e200  # overflows: not finite on the folded constants, computed again
        plans.append(B.Plan(t, kind))
        plans[-1].lanes_per_point = 512  # one point per block
        inputs.append(torch.tensor(phase_space.source_major(p), device="cuda"))
        outs.append(torch.full((n * t.outputs,), -1.0, dtype=torch.float64, device="cuda"))
        with np.errstate(all="ignore"):
            want.append(O.evaluate(t, p, kernel=abi.KERNELS[kind])[1])
    b = B.Batch(plans, inputs, outs)
    for _ in range(2):
        for o in outs:
            o.fill_(-1.0)
        b.run()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            got = o.cpu().numpy().reshape(w.shape)
            nan = np.isnan(w)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.uint64), w[~nan].view(np.uint64))
