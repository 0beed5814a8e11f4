"""The folded constants of a schedule on the CPU (the product's fold_constants, tests/harness): each
instruction's entry is the product its plain form computes, and its class only leaves out products
with an exactly zero part."""
import ctypes as C

import numpy as np
import pytest

from pacuda_b200 import processes
from tests import schedule_emulator as E

K_CONTRIB, K_PROP, K_CLOSURE, K_IDENTITY = 1, 2, 5, 3
REAL, IMAG, ONE, GENERAL = 0, 1, 2, 3
HOT = {0: (4, IMAG), 1: (6, IMAG), 2: (5, ONE), 3: (11, REAL), 4: (2, REAL), 5: (3, REAL), 6: (9, IMAG), 7: (11, REAL)}


def folds(t, scales, factors, known=True):
    keep, args = E._args(t.words, t.width, t.current_planes, t.amplitude_planes, t.momentum_planes // 4, len(scales),
                         len(factors))
    parts = [np.ascontiguousarray(x, dtype=np.float64) for x in (scales.real, scales.imag, factors.real, factors.imag)]
    ptr = [x.ctypes.data if known else None for x in parts]
    sizes = np.zeros(3, np.uint32)
    f = E.lib().fold_export
    f.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p] + [C.c_uint32] * 5 + [C.c_void_p] * 9
    assert f(*args, *ptr, sizes.ctypes.data, None, None, None, None) == 0
    ins, codes = np.zeros((sizes[0], 8), np.uint32), np.zeros(sizes[0], np.uint32)
    entries, recips = np.zeros((sizes[1], 2), np.uint32), np.zeros(sizes[2] + 1, np.uint32)
    assert f(*args, *ptr, sizes.ctypes.data, ins.ctypes.data, codes.ctypes.data, entries.ctypes.data,
             recips.ctypes.data) == 0
    return ins, codes, entries, recips[:-1]


def value(entry, scales, factors):
    kind, a, b = entry[0] >> 28, entry[0] & 0xFFFFFFF, entry[1]
    return scales[a] * factors[b] if kind == 0 else factors[a] * (factors[b] if kind == 1 else 1.0 if kind == 2 else -1j)


@pytest.mark.parametrize("table", ["plan", "mixed", "unknown"])
@pytest.mark.parametrize("name", ["gg>ggg", "qg>qgg"])
def test_entries_and_classes(name, table):
    t = processes.template(name)
    scales, factors = t.scale_re + 1j * t.scale_im, t.factor_re + 1j * t.factor_im
    if table == "mixed":  # zeros, ones and general values in every place
        rng = np.random.default_rng(3)
        pool = np.array([0, 1, -1, 1j, 2.5, -0.5j, 0.3 + 0.4j, complex(np.inf, 0)])
        scales, factors = rng.choice(pool, len(scales)), rng.choice(pool, len(factors))
    ins, codes, entries, recips = folds(t, scales, factors, table != "unknown")
    used = set()
    for i, code in zip(ins, codes):
        kind, op, flags, cls = i[0] & 15, i[0] >> 4 & 15, i[0] >> 8 & 255, i[0] >> 16
        if kind == K_CONTRIB and op:
            which = [i[5]]
        elif kind in (K_PROP, K_IDENTITY):
            which = [i[6]]
        elif kind == K_CLOSURE:
            which = list(range(i[7], i[7] + i[5]))
        else:
            assert code == 15
            continue
        if kind == K_PROP:
            assert recips[i[5]] == i[4]
        used |= set(which)
        with np.errstate(invalid="ignore"):
            v = [value(entries[e], scales, factors) for e in which]
        if table == "unknown":
            assert cls == GENERAL
        elif cls == REAL:
            assert all(x.imag == 0 for x in v)
        elif cls == IMAG:
            assert all(x.real == 0 for x in v)
        elif cls == ONE:
            assert all(x == 1 for x in v)
        if code != 15:
            assert HOT[code] == (op, cls) and (kind != K_CLOSURE or (i[5] == (4 if code == 3 else 2) and flags & 64))
        if table == "plan":
            assert cls != GENERAL
    assert used == set(range(len(entries)))
