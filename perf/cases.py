"""The work that a user of lfts_cpu_b200 has it do, as cases that can be timed and compared.

A case is one call, or one turn of a loop, of a simulation program: the concentrations of given fields
(``calc_concs``), a Langevin step (``full_step_device``: W- update, Anderson mixing of w+, the extra
``calc_concs``), the sampling that runs every so many steps (H, S(k)), the gradients of H (``backward``), the
bare contour step on the caller's device arrays (``lfts_step_fwd_noalloc``), and steps of a replica ensemble
(``Ensemble.run``).  Meshes, chain lengths and parameters are those of the reference's inputs (16^3, 64^3 and
128^3, N = 64 and 90, the N = 64 benchmark configurations) and boxes with sides of the supported lengths.

Fields: W- is white noise of the size that the Langevin dynamics keep up at the case's parameters (a step's
noise has variance 2 M dt / (C V), the drift term damps it by 2 dt / XbN a step), w+ a small random field.

Results: the FP64 path hands on its FP64 fields; the FP32-mixed path computes its propagators in single
precision, and its fields are handed on in single precision.
"""
import ctypes
import math

import numpy as np
import torch

import lfts_cpu_b200 as lfts
from lfts_cpu_b200.capi import Params, lib

# sides with a compiled transform and the (my, mz) pairs of uneven boxes
SIDES = (8, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128)
UNEVEN = ((12, 20), (24, 16), (16, 32), (32, 64))
ENSEMBLE_SIDES = (16, 24, 32, 48, 64, 96)
MOST_POINTS = 128 ** 3


def _case(name, kind, prec, m, N, NA, **more):
    c = {"kind": kind, "prec": prec, "mx": m[0], "my": m[1], "mz": m[2], "N": N, "NA": NA}
    c.update({"XbN": 16.0, "C": 100.0, "dt": 0.5, "dx": 0.0625}, **more)
    if name:
        c["name"] = name
    return c


def listed():
    cube = lambda n: (n, n, n)  # noqa: E731
    return [
        # one contour step on device arrays, for a host framework that owns the memory: the smallest call
        _case("step_fwd_24", "step_fwd", "fp64", cube(24), 64, 24, at=20),
        # concentrations of the small mesh of the reference's checking input: latency
        _case("concs_fp64_16", "concs", "fp64", cube(16), 40, 16),
        # a whole Langevin step of the plain FP64 configuration (mixing to the usual tolerance)
        _case("langevin_fp64_32", "langevin", "fp64", cube(32), 64, 32, XbN=14.0, C=50.0, dx=0.125, cap=200, tol=1e-4),
        # a mid-sized mesh with radix-3 sides, single precision
        _case("concs_fp32_48", "concs", "fp32", cube(48), 64, 27, C=50.0),
        # an uneven box with an odd chain length, as a box-shape study has
        _case("concs_fp64_box", "concs", "fp64", (40, 32, 64), 47, 13),
        # the FP64 configuration at 64^3
        _case("concs_fp64_64", "concs", "fp64", cube(64), 64, 32, dx=0.1),
        # the reference's own 64^3 input runs N = 90; here in the mixed precision
        _case("concs_fp32_64", "concs", "fp32", cube(64), 90, 45),
        # gradients with respect to the box and chi N, propagators checkpointed every 8 steps
        _case("backward_fp64_64", "backward", "fp64", cube(64), 64, 32, XbN=15.0, C=50.0, dx=0.09375, every=8),
        # what a sampling step adds: H, one S(k) sample and its spherical average
        _case("sampling_fp64_64", "sampling", "fp64", cube(64), 64, 32, dx=0.1),
        # the replica ensemble of uneven meshes, a short run of every replica and its fields, the mixing capped
        _case("ensemble_32", "ensemble", "fp32", cube(96), 64, 24, C=50.0, n32=12, n48=7, n64=5, n96=8, cap=8,
              tol=1e-4, steps=3),
        # the headline configuration, mixing capped so that every pass does the same work
        _case("langevin_fp32_128", "langevin", "fp32", cube(128), 64, 25, XbN=20.0, cap=12, tol=1e-4),
        # the same mesh in FP64: the largest amount of data
        _case("concs_fp64_128", "concs", "fp64", cube(128), 64, 25, XbN=20.0),
    ]


def _draw_mesh(rng, most):
    while True:
        if rng.random() < 0.6:
            n = rng.choice(SIDES[2:])
            m = (n, n, n)
        else:
            ny, nz = rng.choice(UNEVEN + tuple((n, n) for n in SIDES))
            m = (rng.choice(SIDES), ny, nz)
        if 1000 <= m[0] * m[1] * m[2] <= most:
            return m


def draw(rng):
    kind = rng.choice(("concs", "concs", "concs", "concs", "langevin", "langevin", "sampling", "backward", "step_fwd",
                       "ensemble"))
    N = int(round(math.exp(rng.uniform(math.log(12), math.log(100)))))
    NA = rng.randint(1, N - 1)
    XbN, C = round(rng.uniform(12.0, 20.0), 2), round(rng.uniform(50.0, 200.0), 1)
    dx = round(rng.uniform(0.06, 0.125), 4)
    prec = rng.choice(("fp64", "fp32"))
    more = {"XbN": XbN, "C": C, "dx": dx}
    if kind == "ensemble":
        n = [rng.randint(0, 6), rng.randint(0, 4), rng.randint(0, 3), rng.randint(0, 3)]
        n[rng.randrange(4)] += 1
        return _case(None, kind, "fp32", (96, 96, 96), min(N, 64), min(NA, 63), n32=n[0], n48=n[1], n64=n[2],
                     n96=n[3], cap=rng.randint(4, 8), tol=1e-4, steps=rng.randint(2, 3), **more)
    if kind == "step_fwd":
        return _case(None, kind, "fp64", _draw_mesh(rng, 64 ** 3), N, NA, at=rng.randint(1, N - 1), **more)
    if kind == "backward":
        return _case(None, kind, "fp64", _draw_mesh(rng, 64 ** 3), min(N, 64), min(NA, 63),
                     every=rng.choice((0, 4, 8, 16)), **more)
    if kind == "sampling":
        return _case(None, kind, prec, _draw_mesh(rng, 64 ** 3), N, NA, **more)
    if kind == "langevin":
        # FP64 to the tolerance; FP32-mixed with a cap, so that the amount of work is fixed
        most = 64 ** 3 if prec == "fp64" else MOST_POINTS
        cap = 200 if prec == "fp64" else rng.randint(4, 12)
        return _case(None, kind, prec, _draw_mesh(rng, most), min(N, 64), min(NA, 63), cap=cap, tol=1e-4, **more)
    return _case(None, kind, prec, _draw_mesh(rng, MOST_POINTS), min(N, 64), min(NA, 63), **more)


# ---- inputs -------------------------------------------------------------------------------------------------

def _mesh(case):
    return case["mx"], case["my"], case["mz"]


def _box(case, m):
    return tuple(case["dx"] * n for n in m)


def _noise_sd(case, m):
    M, V = math.prod(m), math.prod(_box(case, m))
    return math.sqrt(2.0 * M * case["dt"] / (case["C"] * V))


def _fields(case, m, seed):
    """W- (M) and w+ (M) on the host, from the seed."""
    rng = np.random.default_rng(seed)
    M = math.prod(m)
    sd = _noise_sd(case, m) / math.sqrt(2.0 * 2.0 * case["dt"] / case["XbN"])
    w = rng.standard_normal(2 * M)
    w[:M] *= sd
    w[M:] *= 0.1
    return w


def _noise(case, m, seed, which):
    rng = np.random.default_rng((seed, which))
    return rng.standard_normal(math.prod(m)) * _noise_sd(case, m)


class _DeviceArray:
    """A system's field array as one that torch can wrap; it holds the system for as long as a tensor uses it."""

    def __init__(self, system, n):
        self.system = system
        ptr = system.fields_device_ptr()
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _system(case, m):
    prec = lfts.LFTS_FP64 if case["prec"] == "fp64" else lfts.LFTS_FP32_MIXED
    return lfts.System(case["N"], case["NA"], case["XbN"], case["C"], case["dt"], m, _box(case, m), precision=prec)


def _replicas(case, seed):
    sides = [32] * case["n32"] + [48] * case["n48"] + [64] * case["n64"] + [96] * case["n96"]
    return [{"N": case["N"], "NA": case["NA"], "XbN": case["XbN"], "C": case["C"], "dt": case["dt"], "m": (n, n, n),
             "L": _box(case, (n, n, n)), "seed": 1000 * seed + r} for r, n in enumerate(sides)]


def prepare(case, seed):
    kind, m = case["kind"], _mesh(case)
    if kind == "step_fwd":
        M = math.prod(m)
        rng = np.random.default_rng(seed)
        p = Params()
        p.N, p.NA, p.XbN, p.C, p.dt = case["N"], case["NA"], case["XbN"], case["C"], case["dt"]
        for d in range(3):
            p.m[d], p.L[d] = m[d], _box(case, m)[d]
        h = np.exp(-_fields(case, m, seed) / case["N"])
        q = torch.from_numpy(rng.uniform(0.2, 1.8, 2 * M)).cuda()
        return {"case": case, "p": p, "q": q, "h": torch.from_numpy(h).cuda(), "out": torch.empty_like(q)}
    if kind == "ensemble":
        reps = _replicas(case, seed)
        ens = lfts.Ensemble(reps)
        for r, d in enumerate(reps):
            ens.set_fields(r, _fields(case, d["m"], (seed, r)))
        ens.mix(2, case["tol"])
        return {"case": case, "ens": ens, "n": len(reps)}
    s = _system(case, m)
    s.set_fields(_fields(case, m, seed))
    M = math.prod(m)
    state = {"case": case, "sys": s, "stream": torch.cuda.ExternalStream(s.stream),
             "w": torch.as_tensor(_DeviceArray(s, 4 * M), device="cuda")}
    if kind == "langevin":
        s.calc_concs()
        s.langevin_init(_noise(case, m, seed, 0))
        state["noise"] = torch.from_numpy(_noise(case, m, seed, 1)).cuda()
    return state


# ---- one pass -----------------------------------------------------------------------------------------------

def _handed_on(state, first):
    """The fields from `first` (in M values) on, in the precision that the path computes them in."""
    case, w = state["case"], state["w"]
    M = w.numel() // 4
    if case["prec"] == "fp64":
        return w[first * M:]
    with torch.cuda.stream(state["stream"]):
        return w[first * M:].to(torch.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step_fwd":
        rc = lib().lfts_step_fwd_noalloc(ctypes.byref(state["p"]), state["q"].data_ptr(), state["out"].data_ptr(),
                                         state["h"].data_ptr(), case["at"], torch.cuda.current_stream().cuda_stream)
        if rc:
            raise lfts.LftsError(rc, "lfts_step_fwd_noalloc")
        return state["out"]
    if kind == "ensemble":
        ens = state["ens"]
        k, lnq = ens.run(case["steps"], case["cap"], case["tol"])
        return {"k": k, "lnQ": lnq.astype(np.float32),
                "w": [ens.get_fields(r).astype(np.float32) for r in range(state["n"])]}
    s = state["sys"]
    if kind == "concs":
        lnq = s.calc_concs()
        return {"lnQ": lnq, "phi": _handed_on(state, 2)}
    if kind == "langevin":
        k, lnq = s.full_step_device(state["noise"].data_ptr(), case["cap"], case["tol"])
        return {"k": k, "lnQ": lnq, "w": _handed_on(state, 0)}
    if kind == "sampling":
        H = s.get_H()
        s.sk_reset()
        s.sk_sample()
        K, S = s.sk_bin()
        return {"H": H, "K": K, "S": S}
    if kind == "backward":
        dL, dX, H = s.backward(case["every"])
        return {"dL": dL, "dXbN": dX, "H": H}
    raise ValueError(kind)


# ---- what a pass cannot do without ----------------------------------------------------------------------------

def _concs_work(m, N, word):
    """Fields in, phi out; both chains' transforms (2.5 M log2 M flops a real transform, two a step and chain);
    the propagators are written once and read once where they exceed the on-chip memory they could stay in."""
    M = math.prod(m)
    flops = (N - 1) * 2 * 2 * 2.5 * M * math.log2(M)
    kept = 2.0 * N * M * word
    return 8.0 * 4 * M + 2 * max(0.0, kept - 100e6), flops


def work(case):
    kind, m, N = case["kind"], _mesh(case), case["N"]
    M = math.prod(m)
    word = 8 if case["prec"] == "fp64" else 4
    if kind == "step_fwd":
        return {"bytes": 8.0 * 6 * M, "flops": 2 * 2 * 2.5 * M * math.log2(M)}
    if kind == "ensemble":
        bytes_, flops = 0.0, 0.0
        for n in [32] * case["n32"] + [48] * case["n48"] + [64] * case["n64"] + [96] * case["n96"]:
            b, f = _concs_work((n, n, n), N, word)
            bytes_ += case["steps"] * case["cap"] * b
            flops += case["steps"] * case["cap"] * f
        return {"bytes": bytes_, "flops": flops}
    b, f = _concs_work(m, N, word)
    if kind == "langevin":
        # the capped loop runs cap - 1 iterations and the extra calc_concs; to the tolerance it takes about 30
        turns = min(case["cap"], 31)
        return {"bytes": turns * b + (turns - 1) * 22.0 * M * word, "flops": turns * f}
    if kind == "sampling":
        return {"bytes": b + 8.0 * 3 * M, "flops": f + 2.5 * M * math.log2(M)}
    if kind == "backward":
        # the chains once, q's recomputation, and two forward transforms per step
        return {"bytes": b, "flops": f * (1.5 if case["every"] else 1.0) + (N - 1) * 2 * 2.5 * M * math.log2(M)}
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, by plain torch and numpy ------------------------------------------------------------

def _g(m, L, N, device):
    k = [torch.fft.fftfreq(m[d], 1.0 / m[d], dtype=torch.float64, device=device) / L[d] for d in (0, 1)]
    kz = torch.arange(m[2] // 2 + 1, dtype=torch.float64, device=device) / L[2]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + kz[None, None, :] ** 2
    return k2, torch.exp(-4.0 * math.pi ** 2 * k2 / (6.0 * N))


def _chains(case, m, wm, wp):
    """q_1..q_N, q^_1..q^_N (lists of mesh tensors), hA, hB, g tables."""
    N, NA = case["N"], case["NA"]
    k2, g = _g(m, _box(case, m), N, wm.device)
    hA, hB = torch.exp(-(wm + wp) / N), torch.exp(-(wp - wm) / N)
    q, qd = [hA], [hB]
    conv = lambda t: torch.fft.irfftn(g * torch.fft.rfftn(t), s=m)  # noqa: E731
    if NA < 1:
        q = [hB]
    if N - NA < 1:
        qd = [hA]
    for i in range(1, N):
        q.append((hA if i < NA else hB) * conv(q[-1]))
        qd.append((hB if i < N - NA else hA) * conv(qd[-1]))
    return q, qd, hA, hB, k2, g


def _concs(case, m, wm, wp):
    N, NA = case["N"], case["NA"]
    q, qd, hA, hB, _, _ = _chains(case, m, wm, wp)
    Q = q[-1].mean()
    A = sum((q[i] * qd[N - 1 - i] for i in range(NA)), torch.zeros_like(wm)) / (hA * Q * N)
    B = sum((q[i] * qd[N - 1 - i] for i in range(NA, N)), torch.zeros_like(wm)) / (hB * Q * N)
    return float(torch.log(Q)), A - B, A + B


def _mix(case, m, wm, wp):
    """Anderson mixing with history 10; (k, w+)."""
    hist, err, k = [], 1.0, 1
    while k < case["cap"] and err > case["tol"]:
        _, _, pp = _concs(case, m, wm, wp)
        d = pp - 1.0
        err = float(torch.sqrt((d * d).mean()))
        lam = 1.0 - 0.9 ** k
        new = wp + lam * d
        if hist:
            U = torch.stack([torch.stack([((d - a[0]) * (d - b[0])).sum() for b in hist]) for a in hist])
            V = torch.stack([(d * (d - a[0])).sum() for a in hist])
            c = torch.linalg.solve(U, V)
            for ci, (dn, wn) in zip(c, hist):
                new = new + ci * ((wn - wp) + lam * (dn - d))
        hist = (hist + [(d, wp)])[-10:]
        wp = new
        k += 1
    return k, wp


def _exact_sampling(case, m, wm, wp):
    lnq, _, _ = _concs(case, m, wm, wp)
    M, L = math.prod(m), _box(case, m)
    H = -lnq + float(((wm ** 2) / case["XbN"] - wp).mean())
    k2 = _g(m, L, case["N"], torch.device("cpu"))[0].numpy()
    K = (2.0 * math.pi * np.sqrt(k2)).reshape(-1)
    CV = case["C"] * math.prod(L)
    S = torch.fft.rfftn(wm).abs().square().reshape(-1).cpu().numpy() * CV / (case["XbN"] * M) ** 2
    S = S - 0.5 / case["XbN"]
    wt = np.full(K.shape, 2.0).reshape(m[0], m[1], -1)
    wt[:, :, 0] = wt[:, :, -1] = 1.0
    wt = wt.reshape(-1)
    order = np.argsort(K, kind="stable")
    ends = np.flatnonzero(np.abs(np.diff(K[order])) > 1e-5)
    starts = np.concatenate([[0], ends + 1])
    last = np.concatenate([ends, [K.size - 1]])
    num = np.add.reduceat((wt * S)[order], starts)
    den = np.add.reduceat(wt[order], starts)
    return {"H": H, "K": K[order][last], "S": num / den}


def _exact_backward(case, m, wm, wp):
    N, NA = case["N"], case["NA"]
    L, M = _box(case, m), math.prod(m)
    q, qd, hA, hB, _, g = _chains(case, m, wm, wp)
    Q = q[-1].mean()
    # dQ/dL_a = (1/M) sum_i <conv_i', .> with q^_{N-i} the adjoint of q_{i+1} apart from h
    dQ = [0.0, 0.0, 0.0]
    wt = torch.full(g.shape, 2.0, dtype=torch.float64, device=g.device)
    wt[..., 0] = wt[..., -1] = 1.0
    ks = [torch.fft.fftfreq(m[d], 1.0 / m[d], dtype=torch.float64, device=g.device) for d in (0, 1)]
    ks.append(torch.arange(m[2] // 2 + 1, dtype=torch.float64, device=g.device))
    shape = ([-1, 1, 1], [1, -1, 1], [1, 1, -1])
    acc = torch.zeros_like(g)
    for i in range(1, N):
        a, b = torch.fft.rfftn(q[i - 1]), torch.fft.rfftn(qd[N - i - 1])
        acc += (a * b.conj()).real
    acc = acc * wt * g / (float(M) * M)
    for d in range(3):
        dgdL = 2.0 * 4.0 * math.pi ** 2 * ks[d].reshape(shape[d]) ** 2 / (6.0 * N * L[d] ** 3)
        dQ[d] = float((dgdL * acc).sum())
    H = -float(torch.log(Q)) + float(((wm ** 2) / case["XbN"] - wp).mean())
    dX = -float((wm ** 2).mean()) / case["XbN"] ** 2
    return {"dL": np.array([-x / float(Q) for x in dQ]), "dXbN": dX, "H": H}


def exact(case, seed):
    kind, m = case["kind"], _mesh(case)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "ensemble":
        return None  # the noise is the ensemble's own generator's
    w = torch.from_numpy(_fields(case, m, seed)).to(dev)
    wm, wp = (t.reshape(m) for t in w.chunk(2))
    if kind == "step_fwd":
        M = math.prod(m)
        rng = np.random.default_rng(seed)
        q = torch.from_numpy(rng.uniform(0.2, 1.8, 2 * M)).to(dev).reshape((2,) + m)
        h = torch.exp(-w / case["N"]).reshape((2,) + m)
        g, N, NA, i = _g(m, _box(case, m), case["N"], dev)[1], case["N"], case["NA"], case["at"]
        conv = [torch.fft.irfftn(g * torch.fft.rfftn(t), s=m) for t in q]
        return torch.cat([(conv[0] * h[0 if i < NA else 1]).reshape(-1),
                          (conv[1] * h[1 if i < N - NA else 0]).reshape(-1)])
    if kind == "concs":
        lnq, pm, pp = _concs(case, m, wm, wp)
        return {"lnQ": lnq, "phi": torch.cat([pm.reshape(-1), pp.reshape(-1)])}
    if kind == "sampling":
        return _exact_sampling(case, m, wm, wp)
    if kind == "backward":
        return _exact_backward(case, m, wm, wp)
    # a Langevin step; in the mixed precision w+ follows rounding through the least squares of every iteration,
    # so it has no value of its own to be held to
    if case["prec"] != "fp64":
        return None
    _, pm, _ = _concs(case, m, wm, wp)
    eta = [torch.from_numpy(_noise(case, m, seed, j)).to(dev).reshape(m) for j in (0, 1)]
    wm = wm - (pm + 2.0 * wm / case["XbN"]) * case["dt"] + 0.5 * (eta[0] + eta[1])
    k, wp = _mix(case, m, wm, wp)
    lnq, pm, pp = _concs(case, m, wm, wp)
    return {"k": None, "lnQ": lnq, "w": torch.cat([t.reshape(-1) for t in (wm, wp, pm, pp)])}
