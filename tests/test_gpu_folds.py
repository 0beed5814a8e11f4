"""Folded constants in the on-chip executor: every class of constant (real, imaginary, one, general)
in every kernel kind, tables too large for shared memory, runs that add to their destination's
value, and points whose values overflow or are not numbers, each equal to the oracle's values (the
plain formulas) bit for bit."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from pacuda_b200 import abi, phase_space, plan as P, processes

pytestmark = pytest.mark.gpu
POINTS = 37


def with_rows(t, rows, factors):
    """The template with other rows and factor table (the first factors unchanged)."""
    width = P.widths_for(rows, t.current_planes, t.amplitude_planes, t.momentum_planes // 4, len(factors), len(t.scale_re),
                         k_max=6)
    return dataclasses.replace(t, words=P.encode(rows, width), width=width, factor_re=np.real(factors).copy(),
                               factor_im=np.imag(factors).copy())


def factors_of(t):
    return np.asarray(t.factor_re) + 1j * np.asarray(t.factor_im)


def refactored(t, pick):
    """Every contribution, propagator and closure row with its own factor: pick(row number) times its
    old one (a closure's row factor alone)."""
    rows, table = P.decode(t.words, t.width), list(factors_of(t))
    at = {2: 8, 3: 8, 4: 8, 5: 8, 6: 8, 7: 3, 8: 3, 9: 3, 11: 5}  # the row factor's place in a row
    out = []
    for n, row in enumerate(rows):
        if row[0] in at:
            row = list(row)
            k = at[row[0]] if row[0] != 11 else 4
            table.append(table[row[k]] * pick(n))
            row[k] = len(table) - 1
            row = tuple(row)
        out.append(row)
    return with_rows(t, out, np.array(table))


def run(t, p, kind, lanes=None):
    import torch

    from pacuda_b200 import batch as B

    plan = B.Plan(t, kind)
    if lanes:
        plan.lanes_per_point = lanes
    out = torch.full((len(p) * t.outputs,), -1.0, dtype=torch.float64, device="cuda")
    b = B.Batch([plan], [torch.tensor(phase_space.source_major(p), device="cuda")], [out])
    b.run()
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(len(p), t.outputs)


def same(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


CLASSES = {
    "one": lambda n: 1.0,
    "real": lambda n: (1.5, -0.75, 2.0)[n % 3],
    "imaginary": lambda n: (1j, -0.5j)[n % 2],
    "general": lambda n: (0.6 + 0.8j, -0.8 + 0.6j, 1.0, 1j)[n % 4],
}


@pytest.mark.parametrize("kind", ["f64", "df64", "mixed", "mixed64"])
@pytest.mark.parametrize("cls", list(CLASSES))
@pytest.mark.parametrize("name", ["gg>gg", "qq~>gg"])
def test_classes(name, cls, kind):
    t = refactored(processes.template(name), CLASSES[cls])
    p = phase_space.sample(4, POINTS, 5)
    _, want = O.evaluate(t, p, kernel=abi.KERNELS[kind])
    for lanes in (None, 64, 512):  # several, eight and one point per block
        same(run(t, p, kind, lanes), want)


def test_a_table_beyond_shared_memory():
    t = refactored(processes.template("gg>ggg"), CLASSES["general"])
    assert len(t.factor_re) > 256
    p = phase_space.sample(5, POINTS, 6)
    _, want = O.evaluate(t, p, kernel=abi.KERNEL_F64)
    same(run(t, p, "f64"), want)
    same(run(t, p, "f64", 512), want)


def test_runs_that_add_to_their_destination():
    base = processes.template("gg>ggg")
    rows, out, cleared = P.decode(base.words, base.width), [], set()
    for row in rows:
        if row[0] in (5, 6) and row[1] == 1:  # (op, init, scale, parent, parent, destination, ...)
            row = (row[0], 0, *row[2:])
            if row[5] not in cleared:
                cleared.add(row[5])
                out.append((1, row[5], 4 if row[0] == 6 else 6))
        out.append(row)
    t = with_rows(base, out, factors_of(base))
    p = phase_space.sample(5, POINTS, 7)
    _, want = O.evaluate(t, p, kernel=abi.KERNEL_F64)
    same(run(t, p, "f64"), want)


@pytest.mark.parametrize("kind", ["f64", "mixed"])
def test_points_that_are_not_finite(kind):
    """Overflowing and not-a-number points among ordinary ones, in blocks of several points and of
    one: the ordinary points' bits, and the plain formulas' infinities and NaNs in the others."""
    t = processes.template("gg>ggg")
    p = phase_space.sample(5, POINTS, 8)
    p[3] *= 1e160
    p[10, 2, 1] = np.nan
    p[11, 4, 3] = np.inf
    p[20] = 0.0
    p[21] *= 1e-160
    _, want = O.evaluate(t, p, kernel=abi.KERNELS[kind])
    assert not np.isfinite(want[[10, 11]]).all()
    for lanes in (None, 512):
        same(run(t, p, kind, lanes), want)
