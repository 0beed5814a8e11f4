"""Runner calls without a words key compile their program anew each time: what one call's program holds on the
device is given back by the next. (A process of its own: the runner is configured once per process.)"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import numpy as np, torch
from pacuda_b200 import phase_space, processes, runner
t = processes.template("gg>ggg")
call = t.call(phase_space.source_major(phase_space.sample(5, 8, 3)), 8, words_key=0)
r = runner.Runner(kernel="f64", executor="onchip")
def free(calls):
    for _ in range(calls):
        assert r.run(call) == 0
    return torch.cuda.mem_get_info()[0]
torch.zeros(1, device="cuda")
before = free(4)
print("lost", before - free(120))
"""


def test_programs_without_a_key_are_given_back():
    p = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert int(p.stdout.split("lost")[1]) <= 4 << 20, p.stdout
