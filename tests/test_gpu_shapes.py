"""Plans at the limit of a block's shared memory: the lanes per point and blocks per SM that fit a plan's
points without their reciprocals and without its table of folded entries are accepted (here the points
are padded with unused forms, 32 bytes each, up to the limit), and the outputs have the oracle's bits."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from pacuda_b200 import abi, phase_space, processes

from tests.test_gpu_folds import same

pytestmark = pytest.mark.gpu
ROOM = 232448 - 64  # a block's shared memory, less the kernel's own


def padded(t, forms):
    return dataclasses.replace(t, momentum_planes=t.momentum_planes + 4 * forms,
                               form_terms=np.concatenate([t.form_terms, np.zeros(2 * forms, np.uint32)]).astype(np.uint32))


def batch(t, p, kind):
    import torch

    from pacuda_b200 import batch as B

    plan = B.Plan(t, kind)
    out = torch.full((len(p) * t.outputs,), -1.0, dtype=torch.float64, device="cuda")
    return plan, torch.tensor(phase_space.source_major(p), device="cuda"), out


@pytest.mark.parametrize("kind,bare", [("f64", 11360), ("df64", 11360), ("mixed", 6304)])
@pytest.mark.parametrize("points,lanes", [(16, 32), (5, 96), (1, 512)])
def test_lanes_per_point_at_the_limit(points, lanes, kind, bare):
    import torch

    from pacuda_b200 import batch as B

    base = processes.template("qg>qgg")
    t = padded(base, (ROOM // points - bare) // 32)
    p = phase_space.sample(5, 23, 4)
    _, want = O.evaluate(base, p, kernel=abi.KERNELS[kind])
    plan, ext, out = batch(t, p, kind)
    plan.lanes_per_point = lanes
    assert plan.lanes_per_point == lanes
    b = B.Batch([plan], [ext], [out])
    assert b.lanes_per_point(0) == lanes
    b.run()
    torch.cuda.synchronize()
    same(out.cpu().numpy().reshape(want.shape), want)


@pytest.mark.parametrize("blocks", [2, 4])
def test_blocks_per_sm_at_the_limit(blocks):
    import torch

    from pacuda_b200 import batch as B

    base = processes.template("qg>qgg")
    room = (233472 - 1024 * blocks) // blocks - 64
    t = padded(base, (room - 11360) // 32)
    p = phase_space.sample(5, 23, 4)
    _, want = O.evaluate(base, p, kernel=abi.KERNELS["f64"])
    plan, ext, out = batch(t, p, "f64")
    b = B.Batch([plan], [ext], [out])
    b.blocks_per_sm = blocks
    assert b.plan_blocks_per_sm(0) == blocks
    b.run()
    torch.cuda.synchronize()
    same(out.cpu().numpy().reshape(want.shape), want)


@pytest.mark.parametrize("points,lanes", [(16, 32), (1, 512)])
def test_the_runner_at_the_limit(points, lanes, tmp_path):
    """The runner's on-chip executor at configured lanes per point (a process of its own: it is configured once)."""
    import os
    import subprocess
    import sys

    base = processes.template("qg>qgg")
    forms = (ROOM // points - (16 * 632 + 16 * 96 + 32 * 15)) // 32  # its slots, amplitudes and forms in f64
    code = f"""
import numpy as np
from pacuda_b200 import phase_space, processes, runner
from tests.test_gpu_shapes import padded
r = runner.Runner()
assert r.configure("f64", executor="onchip", lanes_per_point={lanes}) == 0
_, outs = r.evaluate(padded(processes.template("qg>qgg"), {forms}), phase_space.sample(5, 23, 4))
np.save(r"{tmp_path / 'out.npy'}", outs)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    _, want = O.evaluate(base, phase_space.sample(5, 23, 4), kernel=abi.KERNELS["f64"])
    same(np.load(tmp_path / "out.npy").reshape(want.shape), want)
