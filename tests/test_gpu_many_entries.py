"""A plan with more distinct pairs of scale and factor than 16 bits index: accepted as each index fits, by the
batch and by the runner's on-chip executor, with the oracle's bits."""
import dataclasses
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as O
from pacuda_b200 import abi, phase_space, plan as P, processes

from tests.test_gpu_folds import factors_of, run, same

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
POINTS = 5


def many(scales=270, factors=250):
    """gg>gg with a run of scales x factors more contributions, each with its own pair of constants, and the
    rows after it on the last entries of the factors."""
    t = processes.template("gg>gg")
    rng = np.random.default_rng(2)
    rows, n_f = P.decode(t.words, t.width), len(t.factor_re)
    n_s = len(t.scale_re)
    at = max(n for n, r in enumerate(rows) if r[0] == 6)
    run = [(6, 0, n_s + s, *rows[at][3:8], n_f + f) for s in range(scales) for f in range(factors)]
    table = np.concatenate([factors_of(t), 1e-3 * (rng.normal(size=factors) + 1j * rng.normal(size=factors)), factors_of(t)])
    late = []
    for r in rows[at + 1:]:
        if r[0] == 11:
            r = (*r[:4], n_f + factors + r[4], n_f + factors + r[5], r[6])
        elif r[0] in (7, 8, 9):
            r = (*r[:3], n_f + factors + r[3])
        late.append(r)
    rows = rows[:at + 1] + run + late
    sre = np.concatenate([t.scale_re, 1e-3 * rng.normal(size=scales)])
    sim = np.concatenate([t.scale_im, 1e-3 * rng.normal(size=scales)])
    width = P.widths_for(rows, t.current_planes, t.amplitude_planes, t.momentum_planes // 4, len(table), len(sre), k_max=4)
    return dataclasses.replace(t, words=P.encode(rows, width), width=width, factor_re=table.real.copy(),
                               factor_im=table.imag.copy(), scale_re=sre, scale_im=sim)


def points():
    return phase_space.sample(4, POINTS, 9)


def test_the_plan_needs_more_than_16_bits():
    from tests.test_folds import folds

    t = many()
    entries = folds(t, t.scale_re + 1j * t.scale_im, t.factor_re + 1j * t.factor_im)[2]
    assert len(entries) > 0x10000 and max(len(t.scale_re), len(t.factor_re)) < 1000


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["f64", "df64", "mixed", "mixed64", "f64fma"])
def test_a_batch(kind):
    t, p = many(), points()
    _, want = O.evaluate(t, p, kernel=abi.KERNELS["f64" if kind == "f64fma" else kind])
    for lanes in (None, 512):
        got = run(t, p, kind, lanes)
        if kind == "f64fma":
            assert np.all(np.abs(got - want) <= 1e-10 * np.abs(want).max(axis=1, keepdims=True))
        else:
            same(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["f64", "df64", "mixed"])
def test_the_runner(kind, tmp_path):
    code = f"""
import numpy as np
from pacuda_b200 import phase_space, runner
from tests.test_gpu_many_entries import many, points
r = runner.Runner(kernel="{kind}", executor="onchip")
amps, outs = r.evaluate(many(), points())
np.save(r"{tmp_path / 'out.npy'}", outs)
"""
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    got = np.load(tmp_path / "out.npy")
    _, want = O.evaluate(many(), points(), kernel=abi.KERNELS[kind])
    same(got.reshape(want.shape), want)
