"""Performance cases of the framework's public entry points on one GPU.

What a program does with this framework falls into seven paths, each with cases over its real range:

* batch: matrix elements of points that are already on the device (a generator's integrand or a
  labelling run): plans compiled once, tuned and captured, one replay per call;
* stable: mixed precision with the rotated-momentum check, failing points again in f64;
* abi: the runner's C ABI on host buffers, one run and one resolved reduction per tile (how a
  RustiCol host drives it);
* umami: umami_matrix_element of the p p -> 3 jets library on host events (how MadGraph drives it);
* forward: the surrogate's inference on given points;
* train: Adam steps of the surrogate on one epoch's batches, the weights read at the end;
* unweight: one step of (two-stage or plain) unweighting: the weight of every candidate.
"""
import ctypes
import functools
import math
import os
import tempfile

import numpy as np
import torch

from pacuda_b200 import abi, batch, pacuda_file, processes, runner, stability, surrogate, unweight
from pacuda_b200.umami import build as umami_build

ECM = 13000.0
MIX = {"pp3j": processes.PP3J, "pp4j": processes.PP4J}
# how a mix's points fall on its families: uneven, as subprocess cross sections are
SHARES = (0.43, 0.31, 0.17, 0.09)
NETWORK_FLOPS = 2 * (64 * 256 + 3 * 256 * 256 + 256)  # one point through the surrogate


def listed():
    return [
        # the latency of one small integrand call
        {"name": "gg>ggg 64", "path": "batch", "process": "gg>ggg", "kernel": "f64", "points": 64},
        # the small configuration: one process, 4096 points
        {"name": "gg>ggg 4096", "path": "batch", "process": "gg>ggg", "kernel": "f64", "points": 4096},
        # the benchmark's workload: every 3-jet family, 2^20 points
        {"name": "pp3j 1048576", "path": "batch", "process": "pp3j", "kernel": "f64", "points": 1 << 20},
        # a quark family with contracted multiply-adds, an odd number of points
        {"name": "qg>qgg fma 50021", "path": "batch", "process": "qg>qgg", "kernel": "f64fma", "points": 50021},
        # the reference's default precision (double floats) on the 3-jet mix
        {"name": "pp3j df64 65537", "path": "batch", "process": "pp3j", "kernel": "df64", "points": 65537},
        # the six-gluon process: the largest plans (three parts)
        {"name": "gg>gggg 10007", "path": "batch", "process": "gg>gggg", "kernel": "f64", "points": 10007},
        # mixed precision with the stability check at the soft cuts it was made for
        {"name": "gg>gggg stable 6000", "path": "stable", "process": "gg>gggg", "points": 6000},
        # a RustiCol tile
        {"name": "abi gg>ggg 65536", "path": "abi", "process": "gg>ggg", "points": 1 << 16},
        # a generator's call over a quarter of a million events
        {"name": "umami 262144", "path": "umami", "points": 1 << 18},
        # labelled or proposed points through the trained network
        {"name": "forward 300007", "path": "forward", "inputs": 9, "points": 300007},
        # sixteen steps of the training configuration
        {"name": "train 16x16384", "path": "train", "inputs": 9, "batch": 16384, "steps": 16},
        # one step of the learned configuration: 2^22 candidates of the 3-jet families
        {"name": "two-stage 4194304", "path": "unweight", "process": "pp3j", "stages": 2, "points": 1 << 22},
    ]


# points per second of a batch (f64), by process, and each kernel kind's rate against f64: only to
# keep a drawn case no dearer than the largest listed one
RATES = {"gg>gg": 4e8, "qq~>gg": 8e8, "gg>ggg": 2.4e7, "qg>qgg": 1e8, "qq~>ggg": 1e8, "gg>qq~g": 1e8, "gg>gggg": 1.1e6,
         "qg>qggg": 5e6, "qq~>gggg": 5e6, "gg>qq~gg": 5e6, "pp3j": 4e7, "pp4j": 2.2e6}
KINDS = {"f64": 1.0, "f64fma": 1.0, "mixed": 1.0, "mixed64": 1.0, "df64": 0.12}


def _between(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    path = rng.choice(["batch", "batch", "batch", "stable", "abi", "umami", "forward", "train", "unweight"])
    if path == "batch":
        process, kernel = rng.choice(sorted(RATES)), rng.choice(["f64", "f64"] + sorted(KINDS))
        most = int(0.012 * RATES[process] * KINDS[kernel])
        return {"path": path, "process": process, "kernel": kernel,
                "points": _between(rng, 4 if process in MIX else 1, min(most, 1 << 20))}
    if path == "stable":
        return {"path": path, "process": rng.choice(["gg>ggg", "gg>gggg"]), "points": _between(rng, 64, 6000)}
    if path == "abi":
        return {"path": path, "process": rng.choice(["gg>gg", "gg>ggg", "qg>qgg", "gg>qq~g"]),
                "points": _between(rng, 1, 1 << 16)}
    if path == "umami":
        return {"path": path, "points": _between(rng, 4, 1 << 18)}
    if path == "forward":
        return {"path": path, "inputs": rng.choice([9, 12]), "points": _between(rng, 1, 1 << 21)}
    if path == "train":
        return {"path": path, "inputs": rng.choice([9, 12]), "batch": 128 * _between(rng, 1, 128),
                "steps": rng.randint(4, 16)}
    return {"path": path, "process": rng.choice(["pp3j", "pp4j"]), "stages": rng.choice([2, 2, 1]),
            "points": _between(rng, 1 << 12, 1 << 18)}


# ---- plans, points --------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _templates(process):
    return processes.parts(process)


@functools.lru_cache(maxsize=None)
def _plans(process, kernel):
    """A program compiles its plans once."""
    return [batch.Plan(t, kernel) for t in _templates(process)]


def _split(case):
    """[(process, points)] of a case: a mix's families in their shares, each with a point at least."""
    if case.get("process", "pp3j") not in MIX:
        return [(case["process"], case["points"])]
    names = MIX[case.get("process", "pp3j")]
    n = [max(1, int(s * case["points"])) for s in SHARES]
    n[0] += case["points"] - sum(n)
    return list(zip(names, n))


def _rambo(legs, n, gen):
    """n massless RAMBO points [leg][E, px, py, pz][point] at sqrt(s) = ECM, the beams first."""
    u = torch.rand(legs - 2, 4, n, dtype=torch.float64, device="cuda", generator=gen).clamp_min_(1e-16)
    c, f = 2 * u[:, 0] - 1, 2 * math.pi * u[:, 1]
    e, s = -(u[:, 2] * u[:, 3]).log(), (1 - c * c).sqrt()
    q = torch.stack([e, e * s * f.cos(), e * s * f.sin(), e * c], 1)
    t = q.sum(0)
    m = (t[0] ** 2 - (t[1:] ** 2).sum(0)).sqrt()
    b, g, x = -t[1:] / m, t[0] / m, ECM / m
    bq = (b * q[:, 1:]).sum(1)
    p = torch.empty(legs, 4, n, dtype=torch.float64, device="cuda")
    p[:2] = 0
    p[:2, 0] = p[0, 3] = ECM / 2
    p[1, 3] = -ECM / 2
    p[2:, 0] = x * (g * q[:, 0] + bq)
    p[2:, 1:] = x * (q[:, 1:] + b * (q[:, :1] + (bq / (1 + g)).unsqueeze(1)))
    return p


def _inside(p, pt_min, eta_max, dr_min):
    fin = p[2:]
    pt = torch.hypot(fin[:, 1], fin[:, 2])
    eta, phi = torch.asinh(fin[:, 3] / pt), torch.atan2(fin[:, 2], fin[:, 1])
    ok = (pt > pt_min).all(0) & (eta.abs() < eta_max).all(0)
    for i in range(len(fin)):
        for j in range(i):
            d = (phi[i] - phi[j]).abs()
            ok &= torch.hypot(eta[i] - eta[j], torch.minimum(d, 2 * math.pi - d)) > dr_min
    return ok


def _points(legs, n, gen, soft=False):
    """n points inside the jet cuts, [leg][component][point]."""
    got, have = [], 0
    while have < n:
        p = _rambo(legs, 2 * (n - have) + 256, gen)
        p = p[:, :, _inside(p, 5.0 if soft else 20.0, 5.0, 0.1 if soft else 0.4)]
        got.append(p[:, :, :n - have])
        have += got[-1].shape[2]
    return torch.cat(got, 2).contiguous()


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mix_points(case, seed):
    gen = _generator(seed)
    return [(name, _points(len(processes.PROCESSES[name]), n, gen, case["path"] == "stable"))
            for name, n in _split(case)]


def _features(case, seed, n):
    """n points of the network's inputs: the phase-space numbers and a subprocess one-hot."""
    gen, k = _generator(seed), case["inputs"] - 4
    x = torch.zeros(n, case["inputs"], device="cuda")
    x[:, :k] = torch.rand(n, k, device="cuda", generator=gen)
    x[torch.arange(n, device="cuda"), k + torch.randint(4, (n,), device="cuda", generator=gen)] = 1.0
    return x


def _targets(x):
    """A standardized smooth function of the inputs, in the place of the log weight."""
    y = torch.sin(3 * x[:, 0]) + x[:, 1] * x[:, 2] - torch.cos(2 * x[:, 3] + x[:, 4]) + x[:, -1]
    return ((y - y.mean()) / y.std()).contiguous()


# ---- the paths ------------------------------------------------------------------------------------


def _prepare_batch(case, seed):
    plans, ext, out = [], [], []
    for name, p in _mix_points(case, seed):
        for t, plan in zip(_templates(name), _plans(name, case["kernel"])):
            plans.append(plan)
            ext.append(p.view(-1))
            out.append(torch.empty(p.shape[2] * t.outputs, dtype=torch.float64, device="cuda"))
    b = batch.Batch(plans, ext, out)
    b.tune()
    b.capture()
    return {"batch": b, "out": out}


def _prepare_stable(case, seed):
    p = _mix_points(case, seed)[0][1]
    return {"stable": stability.StableMixed(_templates(case["process"]), case["points"], 1e-6), "ext": p.view(-1)}


@functools.lru_cache(maxsize=None)
def _runner():
    """The C ABI's runner takes its kernel kind once per process."""
    r = runner.Runner()
    if r.configure("f64") != 0:
        raise RuntimeError("the runner is configured otherwise")
    return r


def _pinned(n, dtype):
    return torch.zeros(n, dtype=dtype, pin_memory=True).numpy()


def _prepare_abi(case, seed):
    (name, p), t, n = _mix_points(case, seed)[0], _templates(case["process"])[0], case["points"]
    ext, out = _pinned(p.numel(), torch.float64), _pinned(n * t.outputs, torch.float64)
    ext[:] = p.view(-1).cpu().numpy()
    red, keep = abi.reduce_resolved_args(t.planes, t.weights, t.offsets, out, n, 1, t.outputs, abi.OUTPUT_ZERO)
    return {"runner": _runner(), "call": t.call(ext, n), "reduce": red, "keep": keep, "out": out}


@functools.lru_cache(maxsize=None)
def _umami():
    """(library, handle) of the p p -> 3 jets subprocess, initialised from its artifact."""
    ctypes.CDLL(runner.DEFAULT_LIB, mode=ctypes.RTLD_GLOBAL)  # this tree's runner, wherever the library was linked
    d = tempfile.mkdtemp(prefix="umami_pp3j_")
    path = os.path.join(os.path.dirname(umami_build.__file__), "_build", "libumami_pp3j.so")
    try:
        lib = ctypes.CDLL(path)
    except OSError:
        from pacuda_b200.umami import provider

        with open(os.path.join(d, "provider_pp3j.h"), "w") as f:
            f.write(provider.header(umami_build.pp3j_spec()))
        lib = ctypes.CDLL(umami_build.build(f.name, os.path.join(d, "libumami_pp3j.so")))
    size, vp, ip = ctypes.c_size_t, ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_int)
    lib.umami_initialize.argtypes = [vp, ctypes.c_char_p]
    lib.umami_matrix_element.argtypes = [ctypes.c_void_p, size, size, size, size, ip, vp, size, ip, vp]
    os.mkdir(os.path.join(d, "artifact"))
    pacuda_file.write(pacuda_file.from_processes(umami_build.PP3J, kernel=1, reference_points=0),
                      os.path.join(d, "artifact.pacuda"))
    handle = ctypes.c_void_p()
    if lib.umami_initialize(ctypes.byref(handle), os.path.join(d, "artifact").encode()) != 0:
        raise RuntimeError("umami_initialize failed")
    return lib, handle


def _prepare_umami(case, seed):
    lib, handle = _umami()
    n, at = case["points"], 0
    mom, flavour = _pinned(20 * n, torch.float64), _pinned(n, torch.int32)
    me = _pinned(n, torch.float64)
    rows = mom.reshape(4, 5, n)  # UMAMI's order: component, particle, event
    for name, p in _mix_points(case, seed):
        m = p.shape[2]
        rows[:, :, at:at + m] = p.transpose(0, 1).cpu().numpy()
        flavour[at:at + m] = umami_build.PP3J.index(name)
        at += m
    keys_in, ptr_in = (ctypes.c_int * 2)(0, 2), (ctypes.c_void_p * 2)(mom.ctypes.data, flavour.ctypes.data)
    keys_out, ptr_out = (ctypes.c_int * 1)(0), (ctypes.c_void_p * 1)(me.ctypes.data)
    return {"call": lib.umami_matrix_element, "args": (handle, n, n, 0, 2, keys_in, ptr_in, 1, keys_out, ptr_out),
            "keep": (mom, flavour), "me": me}


def _prepare_forward(case, seed):
    return {"net": surrogate.Network(case["inputs"], max_batch=128, seed=seed + 1),
            "x": _features(case, seed, case["points"])}


def _prepare_train(case, seed):
    x = _features(case, seed, case["batch"] * case["steps"])
    return {"net": surrogate.Network(case["inputs"], max_batch=case["batch"], seed=seed + 1), "x": x, "y": _targets(x),
            "batch": case["batch"], "steps": case["steps"]}


def _fitted(net, x, y):
    """Gives the network's output layer the least-squares fit of y on its random hidden features: a
    network whose values follow the weights, from torch alone."""
    p = torch.tensor(net.params(), dtype=torch.float64, device="cuda")
    h = torch.cat([_network64(p, x, hidden=True), torch.ones(len(x), 1, dtype=torch.float64, device="cuda")], 1)
    eye = torch.eye(257, dtype=torch.float64, device="cuda")
    p[-257:] = torch.linalg.solve(h.T @ h + 1e-3 * len(x) * eye, h.T @ y)
    net.set_params(p.float().cpu().numpy())


def _prepare_unweight(case, seed):
    names, counts = zip(*_split(case))
    pilot_n, inside = (1 << 14, 0.4) if case["process"] == "pp3j" else (1 << 16, 0.1)
    pl = unweight.Pipeline(families=names, seed=seed + 1, capacity=int(inside * max(pilot_n, *counts)) + 4096)
    # a pilot sample of each family gives the network, its scale and the reduced maxima
    pilot = [pl.labelled(k, 1 << 40, pilot_n) for k in range(len(names))]
    logw = torch.cat([me * jac for _, me, jac, _ in pilot]).log()
    mu, sigma = float(logw.mean()), float(logw.std())
    net, w_max, s_max, r_max = surrogate.Network(pl.inputs, max_batch=128, seed=seed + 1), [], [], []
    _fitted(net, torch.cat([x for x, _, _, _ in pilot]), (logw - mu) / sigma)
    for x, me, jac, _ in pilot:
        w, s = me * jac, pl.surrogate_values(net, x, mu, sigma)
        w_max.append(unweight.maxima(w))
        s_max.append(unweight.maxima(s))
        r_max.append(unweight.maxima(w / s, s))
    return {"pipeline": pl, "net": net, "counts": counts, "scale": (mu, sigma), "w_max": w_max, "s_max": s_max,
            "r_max": r_max, "stages": case["stages"]}


def prepare(case, seed):
    state = globals()["_prepare_" + case["path"]](case, seed)
    state["path"] = case["path"]
    return state


def _run_batch(s):
    s["batch"].run()
    return s["out"]


def _run_stable(s):
    out, redone = s["stable"].run(s["ext"])
    return {"out": out, "redone": redone}


def _run_abi(s):
    if s["runner"].run(s["call"]) != 0 or s["runner"].reduce_resolved(s["reduce"]) != 0:
        raise RuntimeError("a runner call failed")
    return s["out"]


def _run_umami(s):
    if s["call"](*s["args"]) != 0:
        raise RuntimeError("umami_matrix_element failed")
    return s["me"]


def _run_forward(s):
    return s["net"].forward(s["x"])


RATE = 1e-5  # the learning rate that training ends with


def _run_train(s):
    loss, b = torch.zeros(1, device="cuda"), s["batch"]
    for k in range(s["steps"]):
        s["net"].train_step(s["x"][k * b:(k + 1) * b], s["y"][k * b:(k + 1) * b], RATE, loss)
    return {"params": s["net"].params(), "loss": loss}


def _run_unweight(s):
    pl = s["pipeline"]
    if s["stages"] == 2:
        events, exact = pl.two_stage(s["net"], 0, s["counts"], *s["scale"], s["s_max"], s["r_max"])
    else:
        events, exact = pl.plain(0, s["counts"], s["w_max"])
    weights = []  # every candidate's weight, 0 where it is not kept
    for n, e in zip(s["counts"], events):
        index, weight = e.compact()
        weights.append(torch.zeros(n, dtype=torch.float64, device="cuda").scatter_(0, index, weight))
    return {"weights": weights, "exact": exact}


def run(state):
    return globals()["_run_" + state["path"]](state)


# ---- work -----------------------------------------------------------------------------------------

# floating-point operations of a row (the runner's fixed counts), by op; 10 and 11 by component
ROW_FLOPS = {2: 82, 3: 82, 4: 126, 5: 138, 6: 180, 7: 50, 8: 50, 9: 40, 12: 30}


@functools.lru_cache(maxsize=None)
def _point_work(process):
    """(bytes, flops) of one point: its momenta in, its helicity outputs out, the rows of all parts."""
    parts = _templates(process)
    flops = 0
    for t in parts:
        for op, *f in _rows(t):
            flops += 20 * f[5] if op == 11 else 6 * f[1] if op == 10 else ROW_FLOPS.get(op, 0)
    return 32 * parts[0].external_count + sum(8 * t.outputs for t in parts), flops


def work(case):
    if case["path"] == "forward":
        return {"bytes": case["points"] * 4 * (case["inputs"] + 1) + NETWORK_FLOPS, "flops": case["points"] * NETWORK_FLOPS}
    if case["path"] == "train":
        n = case["batch"] * case["steps"]
        return {"bytes": n * 4 * (case["inputs"] + 1) + 8 * NETWORK_FLOPS, "flops": 3 * n * NETWORK_FLOPS}
    if case["path"] == "unweight":
        # the share inside the cuts is listed; the network sees it (two stages) or the runner does (plain)
        inside = (0.28 if case["process"] == "pp3j" else 0.056) * case["points"]
        flops = 200 * case["points"]
        for name, n in _split(case):
            share = inside * n / case["points"]
            flops += share * (NETWORK_FLOPS if case["stages"] == 2 else _point_work(name)[1])
        return {"bytes": 16 * inside, "flops": flops}
    b = f = 0
    for name, n in _split(case):
        bytes_, flops = _point_work(name)
        b += n * (32 * 5 + 12 if case["path"] == "umami" else bytes_)
        f += n * flops * (2 if case["path"] == "stable" else 1)
    return {"bytes": b, "flops": f}


# ---- the same values in 64 bits -------------------------------------------------------------------

# the fields of a row's word after its op (4 bits): widths by kind, numbers are bits
FIELDS = {1: "PP", 7: "PFX", 8: "PFX", 9: "PFX", 10: "PKX", 11: "PPAXXK", 12: "PFXSt",
          **{op: "iSPPPFFX" for op in (2, 3, 4, 5, 6)}}


def _rows(t):
    for w in (int(w) for w in t.words):
        op, row = w & 15, []
        w >>= 4
        for kind in FIELDS[op]:
            bits = {"i": 1, "t": 10}.get(kind) or int(t.width["PAFXSK".index(kind)])
            row.append(w & ((1 << bits) - 1))
            w >>= bits
        yield (op, *row)


def _wavefunction(code, p):
    """The massless gluon's or Weyl spinor's components for momenta p [4][point]; all points of a leg
    have one sign of energy."""
    family, orientation, h, ch = code & 7, (code >> 3) & 3, ((code >> 5) & 7) - 2, ((code >> 8) & 3) - 1
    (e, px, py, pz), pos = p, bool(p[0, 0] > 0)
    zero = torch.zeros_like(e)
    cx = lambda re, im: torch.complex(re + zero, im + zero)  # noqa: E731
    if family == 3:
        c, hel, sgn = math.sqrt(0.5), (h if pos else -h), (1.0 if pos else -1.0)
        pt = torch.hypot(px, py)
        if bool((pt == 0).all()):
            return torch.stack([cx(zero, zero), cx(zero - hel * c, zero), cx(zero, sgn * c * pz.sign()), cx(zero, zero)])
        a = pz / (e.abs() * pt) * c * hel
        return torch.stack([cx(zero, zero), cx(-px * a, -sgn * c * py / pt), cx(-py * a, sgn * c * px / pt),
                            cx(hel * c * pt / e.abs(), zero)])
    if family != 1:
        raise ValueError("massless gluons and Weyl spinors only")
    anti, s = orientation != 0, 1.0 if pos else -1.0
    back = (px == 0) & (py == 0) & (pz * s < 0)
    root = torch.where(back, zero, (s * (e + pz)).clamp_min(0).sqrt()) * (-1.0 if anti == pos else 1.0)
    safe = torch.where(root == 0, torch.ones_like(root), root)
    along = cx(-h * (2 * e.abs()).sqrt(), zero)
    if pos:
        across = cx(-h * px / safe, py / safe) if anti else cx(h * px / safe, -py / safe)
    else:
        across = cx(-h * px / safe, -py / safe) if anti else cx(h * px / safe, py / safe)
    a, b = cx(root, zero), torch.where(root == 0, along, across)
    first = (h == 1 and ch == 1) if pos else (h == -1 and ch == 1)
    second = (h == -1 and ch == -1) if pos else (h == 1 and ch == -1)
    if not first and not second:
        return torch.stack([cx(zero, zero)] * 2)
    return torch.stack([a, b] if (second if anti else first) else [b, a])


def _dot(l, r):
    return l[0] * r[0] - l[1] * r[1] - l[2] * r[2] - l[3] * r[3]


def _contribution(op, l, r, u, v):
    i = 1j
    if op == 2:
        return torch.stack([-i * l[0] * r[3] - i * l[1] * r[1] + l[1] * r[2] + i * l[0] * r[0],
                            -l[0] * r[2] - i * l[0] * r[1] + i * l[1] * r[0] + i * l[1] * r[3]])
    if op == 3:
        return torch.stack([-l[1] * r[2] + i * l[0] * r[0] + i * l[0] * r[3] + i * l[1] * r[1],
                            -i * l[1] * r[3] + l[0] * r[2] + i * l[0] * r[1] + i * l[1] * r[0]])
    if op == 4:
        return torch.stack([l[0] * r[1] + l[1] * r[2] + l[2] * r[3], l[0] * r[0] + l[3] * r[2] + l[4] * r[3],
                            l[1] * r[0] - l[3] * r[1] + l[5] * r[3], l[2] * r[0] - l[4] * r[1] - l[5] * r[2]])
    if op == 5:
        return torch.stack([l[a] * r[b] - l[b] * r[a] for a in range(4) for b in range(a + 1, 4)])
    return _dot(l, r) * (u - v) + 2 * (_dot(l, v) * r - _dot(r, u) * l)


def _evaluate(t, p):
    """The plan's helicity outputs [point][output] at momenta p [leg][component][point]."""
    forms = [sum(float(t.term_coefficients[j]) * p[int(t.term_slots[j])] for j in range(a, a + n))
             for a, n in np.asarray(t.form_terms).reshape(-1, 2).tolist()]
    scale = [complex(a, b) for a, b in zip(t.scale_re, t.scale_im)]
    factor = [complex(a, b) for a, b in zip(t.factor_re, t.factor_im)]
    cur, amp = {}, {}
    for op, *f in _rows(t):
        if op == 12:
            cur[f[0]] = factor[f[2]] * _wavefunction(f[4], forms[f[1]])
        elif op in (2, 3, 4, 5, 6):
            init, s, a, b, dst, u, v, x = f
            o = _contribution(op, cur[a], cur[b], forms[u], forms[v]) * (scale[s] * factor[x])
            cur[dst] = o if init else cur[dst] + o
        elif op in (7, 8, 9):
            c, q, s = cur[f[0]], forms[f[1]], factor[f[2]] / _dot(forms[f[1]], forms[f[1]])
            if op == 9:
                cur[f[0]] = c * (-1j * s)
            elif op == 7:
                cur[f[0]] = s * torch.stack([-1j * c[0] * q[3] - 1j * c[1] * q[1] + c[1] * q[2] + 1j * c[0] * q[0],
                                             -c[0] * q[2] - 1j * c[0] * q[1] + 1j * c[1] * q[0] + 1j * c[1] * q[3]])
            else:
                cur[f[0]] = s * torch.stack([-c[1] * q[2] + 1j * c[0] * q[0] + 1j * c[0] * q[3] + 1j * c[1] * q[1],
                                             -1j * c[1] * q[3] + c[0] * q[2] + 1j * c[0] * q[1] + 1j * c[1] * q[0]])
        elif op == 11:
            a, b, m, x, y, n = f
            w = torch.tensor(factor[y:y + n], dtype=torch.complex128, device=p.device).unsqueeze(1)
            z = factor[x] * (cur[a][:n] * cur[b][:n] * w).sum(0)
            amp[m] = amp[m] + z if m in amp else z
        else:
            raise ValueError("op %d" % op)
    out = torch.zeros(p.shape[2], t.outputs, dtype=torch.float64, device=p.device)
    for o in range(t.outputs):
        for j in range(int(t.offsets[o]), int(t.offsets[o + 1])):
            z = amp[int(t.planes[j])]
            out[:, o] += float(t.weights[j]) * (z.real * z.real + z.imag * z.imag)
    return out


def _exact_outputs(name, p):
    """Per plan part, its outputs at all points, a piece of the points at a time."""
    step = 1 << (13 if p.shape[0] == 6 else 16)
    return [torch.cat([_evaluate(t, p[:, :, k:k + step]) for k in range(0, p.shape[2], step)]) for t in _templates(name)]


def _network64(params, x, hidden=False):
    shapes = [(256, 64), (256,), (256, 256), (256,), (256, 256), (256,), (256, 256), (256,), (256,), (1,)]
    parts = [q.view(s) for q, s in zip(params.split([math.prod(s) for s in shapes]), shapes)]
    h = torch.nn.functional.pad(x.double(), (0, 64 - x.shape[1]))
    for k in range(4):
        z = h @ parts[2 * k].T + parts[2 * k + 1]
        h = z * (1 + torch.tanh(z / 2)) / 2
    return h if hidden else h @ parts[8] + parts[9]


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    params = torch.tensor(s["net"].params(), dtype=torch.float64, device="cuda")
    m, v, total, b = torch.zeros_like(params), torch.zeros_like(params), 0.0, case["batch"]
    for k in range(case["steps"]):
        params.requires_grad_(True)
        e = _network64(params, s["x"][k * b:(k + 1) * b]) - s["y"][k * b:(k + 1) * b].double()
        loss = (e * e).sum()
        g, = torch.autograd.grad(loss / b, params)
        params, total = params.detach(), total + loss.detach()
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        params = params - RATE * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": params, "loss": total.view(1)}


def exact(case, seed):
    if case["path"] == "unweight":
        return None  # a candidate is kept or not: a decision, not a computed number
    if case["path"] == "forward":
        s = _prepare_forward(case, seed)
        return _network64(torch.tensor(s["net"].params(), dtype=torch.float64, device="cuda"), s["x"])
    if case["path"] == "train":
        return _exact_train(case, seed)
    got = [_exact_outputs(name, p) for name, p in _mix_points(case, seed)]
    if case["path"] == "umami":
        me = []
        for (name, _), parts in zip(_split(case), got):
            num, den = _templates(name)[0].meta["group_factor"]
            me.append(sum(parts).sum(1) * (num / den))
        return torch.cat(me)
    out = [o.view(-1) for parts in got for o in parts]
    return out[0] if case["path"] == "abi" else {"out": out, "redone": None} if case["path"] == "stable" else out
