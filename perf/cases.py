"""What a program built on this package has it do, as cases that can be timed.

A case is one call, or one short chain of calls, through the package's public
entry points (`twochnrg_gb300.Engine`, `sweep_batch`, and the C entry point
for callers that cannot allocate).  Its `kind` says which:

  noalloc    nrg_diag_block_noalloc on a device matrix: the smallest call
  diag       Engine.diag_blocks: the blocks of one iteration, or one large one
  sweep      Engine.sweep: the Wilson-chain sweep of a model
  batch      sweep_batch: independent (Q,Sz) sweeps
  thermo     Engine.thermo: impurity and free-chain sweeps side by side
  dm         sweep_dm, dm_backprop, lehmann: the spectral function A(omega)
  grad       grad_forward, grad_backward: derivatives of T chi and <n_d>
  grad_dm    grad_forward_dm, dm_backprop, lehmann_grad: derivatives of A(omega)

Model parameters are drawn from the seed around the package's own workloads
(U of [0.1, 1], a level near -U/2, a hybridization of [1e-3, 5e-2]), so the
block structure of two seeds differs as it does between two parameter points.
"""
import ctypes
import math

import numpy as np
import torch

import twochnrg_gb300 as tg

# Householder reduction flops of one iteration per kept^3 (4/3 sum n_b^3 over
# the blocks): the two-channel site has 16 states, the one-channel site 4.
_ITER_FLOPS = {"1chQS": 5.0, "1chQSz": 3.0, "2chQS": 18.0}
# states (multiplets) of one iteration per kept state
_ITER_STATES = {"1chQS": 4.0, "1chQSz": 4.0, "2chQS": 15.5}
# the most states one iteration can have per kept state, and sectors in all
_MOST_STATES = {"1chQS": 4, "1chQSz": 4, "2chQS": 16}
_MOST_BLOCKS = 1024
# iterations before the truncation sets in, roughly: log(kept) over the growth
_GROWTH = {"1chQS": math.log(3.0), "1chQSz": math.log(4.0), "2chQS": math.log(10.0)}


def listed():
    return [
        # one block of an early iteration or of a host program's own solver
        {"name": "noalloc_64", "kind": "noalloc", "n": 64},
        # the blocks of one one-channel iteration at 500 kept, at the DiagHN call site
        {"name": "diag_iteration", "kind": "diag", "blocks": 21, "nmax": 257},
        # one sector of a two-channel iteration, every eigenvector
        {"name": "diag_one_large", "kind": "diag", "blocks": 1, "nmax": 1901},
        # a quick look at a parameter point: launches and latency
        {"name": "sweep_qsz_small", "kind": "sweep", "model": "1chQSz", "nsites": 14, "kept": 80},
        # the one-channel (Q,S) sweep at the usual 500 kept
        {"name": "sweep_qs_500", "kind": "sweep", "model": "1chQS", "nsites": 40, "kept": 500},
        # a two-channel sweep at a tenth of the full kept count
        {"name": "sweep_2ch_300", "kind": "sweep", "model": "2chQS", "nsites": 16, "kept": 300},
        # the two-channel sweep up to its first iteration at the full 3000 kept
        {"name": "sweep_2ch_3000", "kind": "sweep", "model": "2chQS", "nsites": 4, "kept": 3000},
        # a parameter scan: independent (Q,Sz) sweeps of 200 to 1000 kept
        {"name": "batch_16", "kind": "batch", "instances": 16, "nsites": 40, "kmin": 200, "kmax": 1000},
        # T chi and S of the impurity, the free chain subtracted
        {"name": "thermo_qs_300", "kind": "thermo", "model": "1chQS", "nsites": 24, "kept": 300},
        # the spectral function on 2000 frequencies
        {"name": "dm_qs_500", "kind": "dm", "nsites": 40, "kept": 500, "nomega": 2000},
        # derivatives of the thermodynamics for a fit
        {"name": "grad_qsz_200", "kind": "grad", "nsites": 20, "kept": 200},
        # derivatives of the spectral function for a fit
        {"name": "grad_dm_200", "kind": "grad_dm", "nsites": 20, "kept": 200, "nomega": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "diag", "diag", "sweep", "sweep", "sweep", "batch", "thermo", "dm", "grad",
                       "grad_dm"])
    if kind == "noalloc":
        return {"kind": kind, "n": _log_int(rng, 5, 256)}
    if kind == "diag":
        nmax = _log_int(rng, 9, 1901)
        return {"kind": kind, "blocks": 1 if nmax > 900 else rng.randint(1, 25), "nmax": nmax}
    if kind == "sweep":
        model = rng.choice(["1chQS", "1chQSz", "2chQS"])
        if model == "2chQS":
            kept = _log_int(rng, 40, 1500)
            return {"kind": kind, "model": model, "nsites": rng.randint(4, 6 if kept > 500 else 14), "kept": kept}
        return {"kind": kind, "model": model, "nsites": rng.randint(8, 40), "kept": _log_int(rng, 40, 700)}
    if kind == "batch":
        kmin = _log_int(rng, 50, 300)
        return {"kind": kind, "instances": rng.randint(3, 14), "nsites": rng.randint(12, 36), "kmin": kmin,
                "kmax": kmin + rng.randint(10, 500)}
    if kind == "thermo":
        return {"kind": kind, "model": rng.choice(["1chQS", "1chQSz"]), "nsites": rng.randint(8, 30),
                "kept": _log_int(rng, 50, 400)}
    if kind == "dm":
        return {"kind": kind, "nsites": rng.randint(12, 40), "kept": _log_int(rng, 60, 500),
                "nomega": 2 * rng.randint(50, 1000)}
    if kind == "grad":
        return {"kind": kind, "nsites": rng.randint(8, 24), "kept": _log_int(rng, 60, 250)}
    return {"kind": kind, "nsites": rng.randint(10, 22), "kept": _log_int(rng, 60, 220),
            "nomega": 2 * rng.randint(50, 256)}


def _sizes(case):
    """Block sizes as an iteration has them: most sectors well below the largest."""
    n = case["nmax"]
    rng = np.random.default_rng([n, case["blocks"]])
    return [n] + [int(max(1, round(n * x))) for x in rng.beta(0.8, 1.2, size=case["blocks"] - 1)]


def _block(n, rng):
    """A block with the spectrum of an H_N sector: levels spread over the
    rescaled bandwidth, couplings of a few tenths of it between them."""
    a = rng.standard_normal((n, n)) * (0.6 / math.sqrt(n))
    a = a + a.T
    a[np.diag_indices(n)] += rng.uniform(0.0, 10.0, n)
    return a


def _point(rng):
    U = float(rng.uniform(0.1, 1.0))
    return {"U": U, "ed": float(-U / 2 + rng.uniform(-0.1, 0.1)),
            "gamma": float(np.exp(rng.uniform(np.log(1e-3), np.log(5e-2))))}


def _frequencies(n):
    h = n // 2
    return np.concatenate([-np.logspace(0, -10, h), np.logspace(-10, 0, h)])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "noalloc":
        n = case["n"]
        s["a"] = torch.from_numpy(_block(n, rng)).cuda()
        s["ev"] = torch.empty(n, dtype=torch.float64, device="cuda")
        s["vec"] = torch.empty(n, n, dtype=torch.float64, device="cuda")
        fn = tg.load_library().nrg_diag_block_noalloc
        fn.argtypes = [ctypes.c_int] + 4 * [ctypes.c_void_p]
        s["call"] = fn
        return s
    if kind == "batch":
        s["instances"] = []
        for _ in range(case["instances"]):
            p = _point(rng)
            B = float(np.exp(rng.uniform(np.log(1e-8), np.log(1e-3))))
            s["instances"].append(dict(model="1chQSz", nsites=case["nsites"],
                                       ncutoff=int(rng.integers(case["kmin"], case["kmax"] + 1)), lam=2.5,
                                       U=p["U"], ed=p["ed"], gamma1=p["gamma"], gamma2_or_B=B))
        return s
    s["engine"] = tg.Engine(0)
    if kind == "diag":
        blocks = [_block(n, rng) for n in _sizes(case)]
        s["sizes"] = [len(b) for b in blocks]
        s["packed"] = np.concatenate([b[np.triu_indices(len(b))] for b in blocks])
        return s
    s.update(_point(rng))
    s["B"] = float(np.exp(rng.uniform(np.log(1e-6), np.log(1e-3))))
    if "nomega" in case:
        s["omegas"] = _frequencies(case["nomega"])
    return s


def _iterations(r, model, kept):
    """A sweep's iterations as tables of one row per iteration, as a program
    stores them: rows padded with zeros, so that the tables of two parameter
    points have one shape whatever their sectors."""
    # the 1 % window of the cut lets more states through than asked for
    most = _MOST_STATES[model] * (2 * kept + 64)

    def table(f, width):
        rows = [np.ravel(f(it)) for it in r.iters]
        out = np.zeros((len(rows), width), dtype=rows[0].dtype)
        for k, row in enumerate(rows):
            out[k, :len(row)] = row
        return out

    return {"en": table(lambda it: it.en, most), "bsize": table(lambda it: it.bsize, _MOST_BLOCKS),
            "qn": table(lambda it: it.qn, 2 * _MOST_BLOCKS),
            "kept_bsize": table(lambda it: it.kept_bsize, _MOST_BLOCKS),
            "thermo": np.array([it.thermo for it in r.iters]), "opavg": np.array([it.opavg for it in r.iters]),
            "emin": np.array([it.emin for it in r.iters]), "ecut": np.array([it.ecut for it in r.iters]),
            "nkept": np.array([it.nkept for it in r.iters])}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "noalloc":
        stream = torch.cuda.current_stream().cuda_stream
        st = state["call"](c["n"], state["a"].data_ptr(), state["ev"].data_ptr(), state["vec"].data_ptr(), stream)
        if st != 0:
            raise RuntimeError(f"nrg_diag_block_noalloc: status {st}")
        vec = state["vec"]
        # eigenvectors are determined up to a sign: fix it, as a program that
        # stores or compares them does
        return {"ev": state["ev"], "vec": vec * torch.sign(vec.sum(1, keepdim=True))}
    if kind == "batch":
        r = tg.sweep_batch(state["instances"])
        return {"thermo": r.thermo, "opavg": r.opavg, "nkept": r.nkept}
    eng = state["engine"]
    if kind == "diag":
        ev, vec = eng.diag_blocks(state["sizes"], state["packed"])
        for v in vec:
            v *= np.sign(v.sum(axis=1, keepdims=True))
        return {"ev": np.concatenate(ev), "vec": np.concatenate([v.ravel() for v in vec])}
    U, ed, g = state["U"], state["ed"], state["gamma"]
    if kind == "sweep":
        x = {"1chQS": 0.0, "1chQSz": state["B"], "2chQS": g}[c["model"]]
        return _iterations(eng.sweep(c["model"], c["nsites"], c["kept"], 2.5, U, ed, g, x), c["model"], c["kept"])
    if kind == "thermo":
        x = state["B"] if c["model"] == "1chQSz" else 0.0
        t = eng.thermo(c["model"], c["nsites"], c["kept"], 2.5, U, ed, g, x, reuse_chain=False)
        return {"temp": t.temp, "suscep": t.suscep, "suscep_imp": t.suscep_imp, "entropy": t.entropy,
                "entropy_imp": t.entropy_imp}
    if kind == "grad":
        r = eng.grad_forward("1chQSz", c["nsites"], c["kept"], 2.5, U, ed, g, state["B"])
        w = np.zeros((c["nsites"], 4, 4))
        w[:, :, 2] = 1.0 / (4.0 * c["nsites"])  # the mean of T chi over the sweep's temperatures
        return {"d_tchi": r.d_thermo[:, :, :, 2], "d_opavg": r.d_opavg, "d_egs": r.d_egs, "egs": r.egs,
                "loss_grad": eng.grad_backward(g_thermo=w), **_iterations(r.sweep, "1chQSz", c["kept"])}
    # the temperature two thirds down the chain
    temp = 2.5 ** (-(c["nsites"] * 2 // 3) / 2.0)
    if kind == "dm":
        eng.sweep_dm(c["nsites"], c["kept"], 2.5, U, ed, g)
        prm = eng.dm_params(temp=temp, bbroad=0.6)
        trace = eng.dm_backprop(prm)
        _, A = eng.lehmann(prm, omegas=state["omegas"])
        return {"trace": trace, "A": A}
    eng.grad_forward_dm(c["nsites"], c["kept"], 2.5, U, ed, g)
    prm = eng.dm_params(temp=temp, bbroad=0.6)
    trace = eng.dm_backprop(prm)
    _, A, dA = eng.lehmann_grad(prm, omegas=state["omegas"])
    return {"trace": trace, "A": A, "dA": dA}


def _sweep_work(model, nsites, kept):
    """Iterations at the kept count, the growing ones before them neglected."""
    full = max(1.0, nsites - math.log(kept / 4.0) / _GROWTH[model])
    return {"bytes": 8.0 * full * _ITER_STATES[model] * kept, "flops": full * _ITER_FLOPS[model] * float(kept) ** 3}


def work(case):
    kind = case["kind"]
    if kind == "noalloc":
        n = float(case["n"])
        return {"bytes": 8 * (2 * n * n + n), "flops": (4 / 3 + 2) * n ** 3}
    if kind == "diag":
        n, m = float(case["nmax"]), case["blocks"] - 1
        # beta(0.8, 1.2) sizes: mean square and cube of the fraction
        s2, s3 = n * n * (1 + 0.24 * m), n ** 3 * (1 + 0.168 * m)
        return {"bytes": 8 * 1.5 * s2, "flops": (4 / 3 + 2) * s3}
    if kind == "batch":
        k = 0.5 * (case["kmin"] + case["kmax"])
        w = _sweep_work("1chQSz", case["nsites"], k)
        return {q: case["instances"] * v for q, v in w.items()}
    if kind in ("sweep", "thermo"):
        w = _sweep_work(case["model"], case["nsites"], case["kept"])
        return {q: (2 if kind == "thermo" else 1) * v for q, v in w.items()}
    # every eigenvector of every block, and with derivatives four tangents of
    # the block matrices (two products of the block size each)
    model = "1chQSz" if kind == "grad" else "1chQS"
    w = _sweep_work(model, case["nsites"], case["kept"])
    per = {"dm": 2.5, "grad": 1 + 4 * 3.0, "grad_dm": 2.5 + 4 * 6.0}[kind]
    return {"bytes": w["bytes"] + 16.0 * case.get("nomega", 0), "flops": per * w["flops"]}


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("noalloc", "diag"):
        return None  # a whole sweep is not a few lines of numpy
    if case.get("nmax", 0) > 2500:
        return None
    rng = np.random.default_rng(seed)
    sizes = [case["n"]] if kind == "noalloc" else _sizes(case)
    ev, vec = [], []
    for n in sizes:
        w, v = np.linalg.eigh(_block(n, rng))
        v = v.T
        ev.append(w)
        vec.append(v * np.sign(v.sum(axis=1, keepdims=True)))
    if kind == "noalloc":
        return {"ev": ev[0], "vec": vec[0]}
    return {"ev": np.concatenate(ev), "vec": np.concatenate([v.ravel() for v in vec])}
