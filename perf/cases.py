"""The calls that users of this framework make, for measuring their speed.

Four families, each through the public entry points of the Python binding
(the same C ABI a Fortran host calls):

  step      one adaptive RK4(5) step on host arrays (runge4_adapt2), the call
            that replaces the reference's: 2-D and 3-D tanks, wavemaker of
            first and second order
  interval  the time loop over one output interval with its step control on
            the device (advance), one tank or an ensemble (advance_many)
  lines     cos / sin transforms of device lines by the entry point that
            allocates nothing (transform_noalloc), both directions
  gemm      the surrogate's tensor-core contraction: the raw call (tc_gemm)
            and a linear layer forward and backward (surrogate.tc_matmul)

A tank's fields are random sums of the tank's own modes under a wave
spectrum, with the wave height and period of its sea state.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hos-nwt_gb300"))
import hosnwt  # noqa: E402
import surrogate  # noqa: E402
import workloads  # noqa: E402

MAX_STEP_COST = 1025 * 513 * 8 * 8 * 7 * 7.0  # grid points x orders squared of the largest tank


def listed():
    return [
        # a sloshing tank between two output times: the smallest time loop,
        # a few steps of short launches (the sloshing benchmark's n1 = 129)
        {"name": "interval_sloshing", "kind": "interval", "icase": 1, "tanks": 1, "n1": 129, "M": 3, "f_out": 10.0},
        # an uneven ensemble of irregular-wave tanks advanced together
        {"name": "interval_ensemble", "kind": "interval", "icase": 4, "tanks": 6, "n1": 1025, "M": 5, "f_out": 25.0},
        # the plain 2-D benchmarks: regular wave, and JONSWAP from a wave file
        {"name": "step_regular_2d", "kind": "step", "n1": 257, "n2": 1, "n3": 33, "M": 3, "p1": 3, "p2": 1,
         "wmk": 1, "wave": "mono", "Hs": 0.05, "Tp": 1.0},
        {"name": "step_irregular_2d", "kind": "step", "n1": 1025, "n2": 1, "n3": 65, "M": 5, "p1": 5, "p2": 1,
         "wmk": 1, "wave": "file", "Hs": 0.10, "Tp": 1.4},
        # a narrow basin with ragged lengths (511, 31; dealiased 511, 63) and
        # the second-order wavemaker, sizes of the reference's 3-D benchmarks
        {"name": "step_basin_3d", "kind": "step", "n1": 256, "n2": 32, "n3": 16, "M": 3, "p1": 3, "p2": 3,
         "wmk": 2, "wave": "mono", "Hs": 0.10, "Tp": 1.8},
        # the directional benchmark tank, partial dealiasing (p < M)
        {"name": "step_directional_3d", "kind": "step", "n1": 513, "n2": 257, "n3": 33, "M": 5, "p1": 4, "p2": 4,
         "wmk": 1, "wave": "file", "Hs": 0.08, "Tp": 1.2},
        # the steep M = 7 tank, the largest configuration (dealiased 4100 x 2052)
        {"name": "step_steep_3d", "kind": "step", "n1": 1025, "n2": 513, "n3": 33, "M": 7, "p1": 7, "p2": 7,
         "wmk": 1, "wave": "file", "Hs": 0.15, "Tp": 1.3},
        # one line of a 2-D tank for a host that owns the device memory
        {"name": "lines_one", "kind": "lines", "n": 1025, "lines": 1, "dir": 1, "cs": "cos"},
        # the lines of a 3-D dealiased grid, modes to space
        {"name": "lines_grid", "kind": "lines", "n": 2052, "lines": 513, "dir": -1, "cs": "sin"},
        # the surrogate: a channel mix on the dealiased points of a training
        # batch and the truncated cosine transform of its channels, forward
        # and backward; the truncated x transform of a whole 3-D grid
        {"name": "linear_channels", "kind": "linear", "rows": 32 * 2052, "K": 32, "N": 32},
        {"name": "linear_modes", "kind": "linear", "rows": 32 * 32, "K": 2052, "N": 64},
        {"name": "gemm_grid_modes", "kind": "gemm", "rows": 32896, "K": 2056, "N": 64, "act": 1, "bf16": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "interval", "lines", "linear", "gemm"])
    if kind == "interval":
        icase = rng.choice([1, 4])
        return {"kind": kind, "icase": icase, "tanks": rng.choice([1, 1, 2, 4]), "n1": _log(rng, 65, 1025),
                "M": rng.choice([1, 3, 5]), "f_out": 10.0 if icase == 1 else 25.0}
    if kind == "lines":
        n = _log(rng, 65, 8193)
        return {"kind": kind, "n": n, "lines": _log(rng, 1, max(1.0, min(513.0, 513 * (2052.0 / n) ** 2))),
                "dir": rng.choice([1, -1]), "cs": rng.choice(["cos", "sin"])}
    if kind == "linear":
        return {"kind": kind, "rows": _log(rng, 500, 70000), "K": rng.choice([4, 32, 64, 513, 1025]),
                "N": rng.choice([1, 32, 33, 64, 128])}
    if kind == "gemm":
        return {"kind": kind, "rows": _log(rng, 257, 66000), "K": 8 * _log(rng, 4, 257), "N": _log(rng, 16, 512),
                "act": rng.choice([0, 1]), "bf16": rng.choice([True, False])}
    # a tank: 2-D in two of five; half of the lengths odd powers of two plus
    # one, as users choose them, the rest anything
    M = rng.choice([1, 2, 3, 3, 4, 5, 5, 7])
    two_d = rng.random() < 0.4
    while True:
        n1 = rng.choice([65, 129, 257, 513, 1025]) if rng.random() < 0.5 else _log(rng, 64, 1025)
        n2 = 1 if two_d else (rng.choice([17, 33, 65, 129, 257]) if rng.random() < 0.5 else _log(rng, 16, 300))
        p = rng.choice([q for q in (1, 2, 3, 4, 5, 7) if q <= M and 2 * q >= M])
        if n1 * n2 * (p + 1) ** (2 if n2 > 1 else 1) * M * M <= 0.25 * MAX_STEP_COST:
            break
    return {"kind": "step", "n1": n1, "n2": n2, "n3": rng.choice([9, 17, 33, 40]), "M": M, "p1": p,
            "p2": p if n2 > 1 else 1, "wmk": rng.choice([1, 1, 2]), "wave": rng.choice(["mono", "jonswap"]),
            "Hs": round(rng.uniform(0.03, 0.08), 3), "Tp": round(rng.uniform(1.2, 1.8), 3)}


# ------------------------------------------------------------------ tanks

def _field_pair(rng, n1, n2, Hs, Tp, h=5.0, xlen=50.0, ylen=30.0):
    """Surface elevation and surface potential (n1 x n2, nondimensional) of
    random standing waves of the tank's modes around the peak period, cut at
    twice the peak frequency, and the amplitudes of the potential (modes)."""
    ts = math.sqrt(h / 9.81)
    k1 = np.pi * np.arange(n1)[:, None] / (xlen / h)
    k2 = np.pi * np.arange(n2)[None, :] / (ylen / h)
    k = np.sqrt(k1 ** 2 + k2 ** 2)
    w = np.sqrt(k * np.tanh(k))
    wp = 2.0 * np.pi * ts / Tp
    r = np.where(w > 0, w, 1.0) / wp
    amp = np.exp(-1.25 * 0.5 * r ** -4.0) * r ** -2.5 * (r < 2.0) * (w > 0)
    amp = amp * np.exp(-(np.arctan2(k2, np.maximum(k1, 1e-9)) / 0.6) ** 2)
    amp[(np.arange(n1) > 0.6 * n1), :] = 0.0
    amp[:, (np.arange(n2) > 0.6 * n2) & (n2 > 1)] = 0.0
    a = amp * rng.standard_normal((n1, n2))
    b = amp * rng.standard_normal((n1, n2))
    c1 = np.cos(np.pi * np.outer(np.arange(n1), np.arange(n1)) / (n1 - 1))
    c2 = np.cos(np.pi * np.outer(np.arange(n2), np.arange(n2)) / max(n2 - 1, 1))
    dev = "cuda"
    c1, c2 = torch.tensor(c1, device=dev), torch.tensor(c2, device=dev)
    eta = (c1 @ torch.tensor(a, device=dev) @ c2).cpu().numpy()
    scale = Hs / 4.0 / h / max(float(eta.std()), 1e-30)
    b = b * scale / np.where(w > 0, w, 1.0)
    phis = (c1 @ torch.tensor(b, device=dev) @ c2).cpu().numpy()
    return np.asfortranarray(eta * scale), np.asfortranarray(phis), np.asfortranarray(b)


def _tank(case, seed, n1, M, directory):
    """The tank of a case and its workload's wave, phases from the seed."""
    g = case.get
    kw = dict(Hs=g("Hs", 0.08), Tp=g("Tp", 1.4), T_stop=200.0, toler=1e-7, f_out=g("f_out", 10.0),
              i_wmk=g("wmk", 1), iseed=1000 + seed % 1000)
    n2, n3, p1, p2 = g("n2", 1), g("n3", 33), g("p1", M), g("p2", 1)
    if g("icase") == 1:
        inp = workloads.base_input(icase=1, islosh=3, aslosh=0.02, iabsnb=0, **kw)
    elif g("icase") == 4 or g("wave") == "jonswap":
        inp = workloads.base_input(icase=4, **kw)
    elif g("wave") == "mono":
        inp = workloads.base_input(icase=2, amp_mono=0.5 * g("Hs"), nu_mono=1.0 / g("Tp"),
                                   theta_mono=20.0 if n2 > 1 else 0.0, ph_mono=(seed % 628) * 0.01, **kw)
    else:
        make = workloads.irregular_2d if n2 == 1 else (workloads.steep_3d if M >= 7 else workloads.directional_3d)
        inp = dict(make(directory, seed=seed)["inp"], T_stop=200.0)
    return hosnwt.Tank(inp, n1, n2, n3, M, p1, p2, wave_dir=directory)


def _prepare_step(case, seed):
    rng = np.random.default_rng(seed)
    n1, n2 = case["n1"], case["n2"]
    with tempfile.TemporaryDirectory() as tmp:
        tank = _tank(case, seed, n1, case["M"], tmp)
    inf = tank.info()
    arrs = tank.get_rk_state()
    arrs[0], arrs[1], _ = _field_pair(rng, n1, n2, case["Hs"], case["Tp"])
    # eta1st (space) and a1st (modes): the linear waves of the wavemaker
    arrs[6], _, arrs[8] = _field_pair(rng, n1, n2, case["Hs"], case["Tp"])
    if case["wmk"] == 2:
        arrs[7], _, arrs[9] = _field_pair(rng, n1, n2, 0.05 * case["Hs"], 0.8 * case["Tp"])
    return {"tank": tank, "arrs": arrs, "t": 8.0 / inf["Tscale"], "h": inf["delt"]}


def _prepare_interval(case, seed):
    rng = np.random.default_rng(seed)
    tanks = []
    with tempfile.TemporaryDirectory() as tmp:
        for k in range(case["tanks"]):
            # uneven sizes and orders: n1, n1/2, n1/4, ... and back
            n1 = max(65, (case["n1"] - 1) // (1 << (k % 4)) + 1)
            M = [case["M"], 3, case["M"]][k % 3]
            tanks.append(_tank(case, seed + k, n1, M, tmp))
            tanks[-1].set_state(*_field_pair(rng, n1, 1, 0.02, 1.8)[:2])
    return {"tanks": tanks, "dt_out": [t.info()["delt_out"] for t in tanks],
            "h": [t.info()["delt"] for t in tanks]}


def _run_interval(s):
    # the next output interval of the running tanks
    tanks = s["tanks"]
    ends = [t.info()["time_cur"] + d for t, d in zip(tanks, s["dt_out"])]
    if len(tanks) == 1:
        s["h"][0] = tanks[0].advance(ends[0], s["h"][0])[0]
    else:
        s["h"] = hosnwt.advance_many(tanks, ends, s["h"])
    return [t.get_state() for t in tanks]


def _transforms_per_rhs(M):
    """2-D transforms of the dealiased grid that one right-hand side needs:
    the order products and their way back, the surface gradients, the
    additional potential and the filters."""
    return M * (M + 1) // 2 + (M - 1) + 5 + 6 + 2 * (M // 2)


def _tank_work(n1, n2, M, p1, p2, steps):
    nd = (p1 + 1) * n1 / 2 * (max(1.0, (p2 + 1) * n2 / 2) if n2 > 1 else 1.0)
    flops = 5.0 * _transforms_per_rhs(M) * 2.5 * nd * math.log2(max(nd, 2.0))
    return {"bytes": 2.0 * 8 * 6 * n1 * n2 * steps, "flops": flops * steps}


# ------------------------------------------------------------------ lines

def _lines_input(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(case["lines"], case["n"], device="cuda", dtype=torch.float64, generator=g)
    if case["dir"] < 0:  # modal amplitudes decay like a wave spectrum's
        x = x / (1.0 + 0.02 * torch.arange(case["n"], device="cuda", dtype=torch.float64)) ** 2
    return x


def _lines_exact(case, seed):
    x = _lines_input(case, seed).cpu().numpy()
    n, D = case["n"], case["n"] - 1
    if case["cs"] == "cos":
        f = np.fft.rfft(np.concatenate([x, x[:, D - 1:0:-1]], axis=1), axis=1).real
        if case["dir"] > 0:
            f = f / D
            f[:, [0, D]] *= 0.5
            return f
        sign = 1.0 - 2.0 * (np.arange(n) % 2)
        return 0.5 * (f + x[:, :1] + x[:, D:] * sign)
    x[:, [0, D]] = 0.0
    f = -0.5 * np.fft.rfft(np.concatenate([x, -x[:, D - 1:0:-1]], axis=1), axis=1).imag
    f[:, [0, D]] = 0.0
    return f * (2.0 / D) if case["dir"] > 0 else f


# ------------------------------------------------------------------ gemm

def _gemm_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    M, N, K = case["rows"], case["N"], case["K"]
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)
    v = torch.randn(N, device="cuda", generator=g)
    if case["kind"] == "linear":
        return x, w, torch.randn(M, N, device="cuda", generator=g)
    return x.to(torch.bfloat16), w.to(torch.bfloat16), v


def _gemm_exact(case, seed):
    x, w, v = _gemm_inputs(case, seed)
    b = lambda t: t.to(torch.bfloat16).double()  # noqa: E731  the contractions take BF16 operands
    if case["kind"] == "linear":
        return [b(x) @ b(w).T, b(v) @ b(w), b(v).T @ b(x)]
    y = b(x) @ b(w).T + v.double()
    return torch.nn.functional.gelu(y, approximate="tanh") if case["act"] else y


# ------------------------------------------------------------------ interface

def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return dict(_prepare_step(case, seed), kind=kind)
    if kind == "interval":
        return dict(_prepare_interval(case, seed), kind=kind)
    if kind == "lines":
        x = _lines_input(case, seed)
        return dict(case, x=x, out=torch.empty_like(x))
    x, w, v = _gemm_inputs(case, seed)
    if kind == "linear":
        return {"kind": kind, "x": x.requires_grad_(), "w": w.requires_grad_(), "gy": v}
    out = torch.empty(case["rows"], case["N"], device="cuda", dtype=torch.bfloat16 if case["bf16"] else torch.float32)
    return {"kind": kind, "x": x, "w": w, "bias": v, "out": out, "act": case["act"],
            "err": torch.zeros(1, dtype=torch.int32, device="cuda")}


def run(s):
    kind = s["kind"]
    if kind == "step":
        arrs, err = s["tank"].runge4_adapt2(s["t"], *s["arrs"], s["h"])
        return list(arrs), err
    if kind == "interval":
        return _run_interval(s)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "lines":
        hosnwt.transform_noalloc(s["dir"], s["cs"], s["n"], s["lines"], s["x"].data_ptr(), s["out"].data_ptr(), stream)
        return s["out"]
    if kind == "linear":
        y = surrogate.tc_matmul(s["x"], s["w"])
        gx, gw = torch.autograd.grad(y, (s["x"], s["w"]), s["gy"])
        return [y.detach(), gx, gw]
    return hosnwt.tc_gemm(s["x"], s["w"], bias=s["bias"], act=s["act"], out=s["out"], err=s["err"], stream=stream)


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _tank_work(case["n1"], case["n2"], case["M"], case["p1"], case["p2"], 1)
    if kind == "interval":
        tot = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["tanks"]):
            n1 = max(65, (case["n1"] - 1) // (1 << (k % 4)) + 1)
            M = [case["M"], 3, case["M"]][k % 3]
            # RK4 stability: steps of about 9 / (n1 - 1) depth units in time
            steps = max(1.0, (1.0 / case["f_out"]) / 0.714 * (n1 - 1) / 8.5)
            w = _tank_work(n1, 1, M, M, 1, steps)
            tot = {q: tot[q] + w[q] for q in tot}
        return tot
    if kind == "lines":
        n, L = case["n"], case["lines"]
        return {"bytes": 16.0 * n * L, "flops": 2.5 * n * math.log2(n) * L}
    M, N, K = case["rows"], case["N"], case["K"]
    if kind == "linear":  # operands read once, results written once, in FP32
        return {"bytes": 4.0 * (2 * M * K + 2 * N * K + 2 * M * N), "flops": 6.0 * M * N * K}
    return {"bytes": 2.0 * (M * K + N * K) + (2.0 if case["bf16"] else 4.0) * M * N + 4.0 * N, "flops": 2.0 * M * N * K}


def exact(case, seed):
    kind = case["kind"]
    if kind == "lines":
        return _lines_exact(case, seed)
    if kind in ("linear", "gemm"):
        return _gemm_exact(case, seed)
    return None  # whole steps and intervals: no 64-bit value without the solver itself
