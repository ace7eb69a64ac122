"""The work a user of this framework has it do, as measurable cases.

Kinds of case, each through a public entry point of the gsfft package:

* ``plan``    one sparse FFT of a device-resident signal with a plan that the
              program keeps (Plan.run), FP64 or mixed precision;
* ``batch``   many small signals in one graph launch (Batch.capture / launch);
* ``drop_in`` the reference's own entry, outer_loop: everything in one call,
              candidates returned in host memory;
* ``host``    a host signal through the whole call: ingest, run, results;
* ``fft``     the batched power-of-two FFT building block;
* ``filter``  the flat-window filter design a program does once per configuration.

Sizes are the ones of this repository's benchmark (n = 2^27 with k = 16000 and
k = 43000, the batch of small signals), of its tests (n = 2^14 .. 2^20) and of
the reference's experiment (n = 2^20, k = 1000).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gpu-sfft_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import gsfft  # noqa: E402
from gsfft import synth  # noqa: E402

CAP = 524288  # a plan's default candidate capacity


def _sfft(name, kind, q, k, bcst, loc, thr, est, rcst, rloops=2, prec="mixed", noise_db=0.0):
    return {"name": name, "kind": kind, "q": q, "k": k, "Bcst": bcst, "loops_loc": loc,
            "loops_thresh": thr, "loops_est": est, "RLFC_cst": rcst, "RLFC_loops": rloops,
            "precision": prec, "noise_db": noise_db}


def listed():
    return [
        # the headline step: one 2^27-point signal, 16000 tones, mixed precision
        _sfft("plan_n27_mixed", "plan", 27, 16000, 0.65, 2, 2, 7, 4096),
        # the same step for a program that keeps the reference's double precision
        _sfft("plan_n27_fp64", "plan", 27, 16000, 0.65, 2, 2, 7, 4096, prec="fp64"),
        # a measured (noisy) signal: no bin is an exact zero, the cutoffs do real work
        _sfft("plan_n27_mixed_noise40", "plan", 27, 16000, 0.65, 2, 2, 7, 4096, noise_db=40.0),
        # the largest: 43000 tones at 30 dB, three location loops, W = 2^24
        _sfft("plan_n27_k43000_mixed", "plan", 27, 43000, 0.8, 3, 2, 8, 32768, noise_db=30.0),
        # the reference's experiment size in double precision, noisy
        _sfft("plan_n20_fp64", "plan", 20, 1000, 1.40, 2, 2, 5, 128, prec="fp64", noise_db=30.0),
        # the smallest call: latency and launches are everything
        _sfft("plan_n14_mixed", "plan", 14, 10, 2.5, 2, 2, 5, 16),
        # many small signals of mixed sizes in flight (q 18 .. 24, k 50 .. 4000)
        {"name": "batch24_mixed", "kind": "batch", "count": 24, "mix": 2024, "qmin": 18, "qmax": 24,
         "streams": 16},
        # a program written against the reference: plan, run and results in one call
        _sfft("drop_in_n20", "drop_in", 20, 1000, 1.40, 2, 2, 5, 128, prec="fp64", noise_db=30.0),
        # a double-precision host recording of 2^22 samples through ingest, run and results
        # into the program's spectrum
        _sfft("host_n22_mixed", "host", 22, 1501, 1.2, 2, 2, 5, 512),
        # the RLFC transform's shape as a call of its own, double precision
        {"name": "fft_fp64_2p22x2", "kind": "fft", "log2n": 22, "batch": 2, "sign": -1, "precision": "fp64"},
        # the bucket transform's shape, single precision, inverse
        {"name": "fft_fp32_2p17x9", "kind": "fft", "log2n": 17, "batch": 9, "sign": 1, "precision": "mixed"},
        # the once-per-configuration filter design
        _sfft("filter_n22", "filter", 22, 2000, 1.0, 2, 2, 5, 512, prec="fp64"),
    ]


def _floor2(x):
    return 1 << (int(x).bit_length() - 1) if x >= 1 else 0


def _derived(c):
    """(n, B, W, w, b_f, t0, tolerance, valid): the run parameters of a configuration."""
    q, k, tol = c["q"], c["k"], 1e-8
    n = 1 << q
    bb = int(c["Bcst"] * math.sqrt(float(n) * k / math.log2(n)))
    B = _floor2(bb)
    W = _floor2(c["RLFC_cst"] * n / B) if B else 0
    w = _taps(bb, tol) if bb else 0
    b_f = int(1.2 * 1.1 * (float(n) / bb)) if bb else 0
    t0 = math.cosh(math.acosh(1 / tol) / (w - 1)) if w > 1 else 1.0
    ok = (256 <= B <= n // 2 and 256 <= W < n and W > n // B and 2 * k < min(W, B) and 3 <= w <= n
          and 1 <= b_f <= n and c["loops_thresh"] <= c["loops_loc"])
    return n, B, W, w, b_f, t0, tol, ok


def _mix(c):
    """The configurations of a batch of small signals (drawn as the benchmark draws them)."""
    rng = np.random.default_rng(c["mix"])
    out = []
    while len(out) < c["count"]:
        q = int(rng.integers(c["qmin"], c["qmax"] + 1))
        k = int(round(float(np.exp(rng.uniform(np.log(50), np.log(4000))))))
        one = _sfft("", "plan", q, k, float(rng.uniform(0.6, 1.5)), 2, 2, 5, 128)
        if _derived(one)[-1]:
            out.append(one)
    return out


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "plan", "batch", "drop_in", "host", "fft", "fft", "filter"])
    if kind == "batch":
        lo = rng.randint(16, 20)
        return {"kind": "batch", "count": rng.randint(5, 24), "mix": rng.randint(0, 10**6), "qmin": lo,
                "qmax": rng.randint(lo, 23), "streams": rng.choice([4, 8, 16, 32])}
    if kind == "fft":
        log2n = rng.randint(8, 24)
        most = max(1, min(512, 1 << (24 - log2n)))
        return {"kind": "fft", "log2n": log2n, "batch": int(round(math.exp(rng.uniform(0, math.log(most))))),
                "sign": rng.choice([-1, 1]), "precision": rng.choice(["fp64", "mixed"])}
    while True:
        prec = "fp64" if kind in ("drop_in", "filter") else rng.choice(["fp64", "mixed"])
        q = {"plan": rng.randint(14, 27 if prec == "mixed" else 26), "drop_in": rng.randint(15, 22),
             "host": rng.randint(16, 22), "filter": rng.randint(14, 22)}[kind]
        k = int(round(math.exp(rng.uniform(math.log(10), math.log(16000)))))
        noise = 30.0 if kind == "drop_in" else rng.choice([0.0, 0.0, 30.0, 40.0]) if kind == "plan" else 0.0
        loc = rng.choice([2, 2, 2, 3])
        c = _sfft("", kind, q, k, rng.uniform(0.6, 1.5), loc, 2, rng.randint(5, 8),
                  rng.choice([128, 512, 4096]), rng.choice([1, 2, 2]), prec, noise)
        del c["name"]
        W, ok = _derived(c)[2], _derived(c)[-1]
        if ok and W <= (1 << 22 if prec == "fp64" else 1 << 24):  # no dearer than the listed ones
            return c


class _View:
    """A device buffer of the library as an array of 8-byte words; it keeps the
    plan that owns the buffer, so tensors made from it stay valid."""

    def __init__(self, plan, ptr, words):
        self.plan = plan
        self.__cuda_array_interface__ = {"shape": (words,), "typestr": "<i8", "data": (ptr, False),
                                         "version": 3, "strides": None}


def _nodes(plan, ptr, count):
    """(keys, values) views of `count` result nodes (key, padding, two doubles)."""
    words = torch.as_tensor(_View(plan, ptr, 3 * count), device="cuda").view(count, 3)
    words.zero_()  # nodes that a run does not fill stay zero
    return words[:, 0], words.view(torch.float64)[:, 1:3]


def _results(plan, k, candidates):
    """Device views of a plan's results: the k largest and, where asked, every candidate."""
    p = [ctypes.c_void_p() for _ in range(4)]
    gsfft.check(gsfft.lib().gsfft_device_results(plan.h, *[ctypes.byref(v) for v in p]), "gsfft_device_results")
    keys, values = _nodes(plan, p[2].value, k)
    out = {"top_keys": keys, "top_values": values}
    if candidates:
        out["cand_keys"], out["cand_values"] = _nodes(plan, p[0].value, CAP)
    return out


def _params(c):
    p, status = gsfft.derive_params(c["q"], c["k"], c["Bcst"], c["loops_loc"], c["loops_thresh"],
                                    c["loops_est"], c["RLFC_cst"], c["RLFC_loops"])
    gsfft.check(status, "gsfft_derive_params")
    return p


def _filter(p):
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    gsfft.design_filter(p, ft.data_ptr(), ff.data_ptr())
    return ft, ff


def _signal(c, p, seed):
    x, loc, coef, _ = synth.signal_torch(p.n, p.k, seed, c["noise_db"] or None)
    return x if c["precision"] == "fp64" else x.to(torch.complex64), loc, coef


def _plan(c, p):
    plan = gsfft.Plan(p, gsfft.FP64 if c["precision"] == "fp64" else gsfft.MIXED)
    ft, ff = _filter(p)
    plan.set_filter(ft.data_ptr(), ff.data_ptr())
    return plan


def prepare(case, seed):
    kind = case["kind"]
    gsfft.lib()
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "fft":
        f64 = case["precision"] == "fp64"
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["batch"], 1 << case["log2n"])
        x = torch.randn(shape, dtype=torch.complex128 if f64 else torch.complex64, device="cuda", generator=g)
        return {"case": case, "x": x, "y": torch.empty_like(x), "stream": stream,
                "prec": gsfft.FP64 if f64 else gsfft.MIXED}
    if kind == "batch":
        plans, xs, draws, outs = [], [], [], []
        for i, c in enumerate(_mix(case)):
            p = _params(c)
            plans.append(_plan(c, p))
            xs.append(_signal(c, p, 1000 * seed + i)[0])
            draws.append(synth.draws(1000 * seed + i, p.n, p.W_RLFC, p.RLFC_loops, p.loops))
            outs.append(_results(plans[-1], p.k, False))
        torch.cuda.synchronize()
        batch = gsfft.Batch(plans, streams=case["streams"])
        batch.capture([x.data_ptr() for x in xs], draws)
        return {"case": case, "batch": batch, "xs": xs, "outs": outs, "stream": stream}
    p = _params(case)
    if kind == "filter":
        # the design has no input but the configuration: the tolerance follows the seed
        p, status = gsfft.derive_params(case["q"], case["k"], case["Bcst"], case["loops_loc"],
                                        case["loops_thresh"], case["loops_est"], case["RLFC_cst"],
                                        case["RLFC_loops"], _tolerance(case, seed))
        gsfft.check(status, "gsfft_derive_params")
        return {"case": case, "p": p, "stream": stream,
                "ft": torch.zeros(p.w, dtype=torch.complex128, device="cuda"),
                "ff": torch.zeros(p.n, dtype=torch.complex128, device="cuda")}
    x, loc, coef = _signal(case, p, seed)
    draws = synth.draws(seed, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    if kind == "drop_in":
        ft, ff = _filter(p)
        return {"case": case, "p": p, "x": x, "ft": ft, "ff": ff, "seed": seed, "libc": ctypes.CDLL(None),
                "keys": np.zeros(CAP, np.int64), "values": np.zeros((CAP, 2))}
    plan = _plan(case, p)
    if kind == "host":
        d_x = torch.empty_like(x)
        return {"case": case, "plan": plan, "hx": x.to(torch.complex128).cpu().numpy(), "d_x": d_x,
                "draws": draws, "stream": stream, "spectrum": np.zeros(p.n, np.complex128)}
    # Mixed precision on a noisy signal: the program takes the k largest (the
    # candidates past them are picks from the noise floor).  Otherwise the whole
    # candidate list is a result as well.
    whole = case["precision"] == "fp64" or not case["noise_db"]
    out = _results(plan, p.k, whole)
    return {"case": case, "plan": plan, "x": x, "draws": draws, "out": out, "stream": stream}


def _taps(bb, tol):
    w = int((1 / math.pi) * (1 / (0.5 / bb)) * math.acosh(1.0 / tol))
    return w - (1 - w % 2)


def _tolerance(case, seed):
    """A tolerance near 1e-8 that leaves the number of taps as it is at 1e-8."""
    bb = int(case["Bcst"] * math.sqrt(float(1 << case["q"]) * case["k"] / math.log2(1 << case["q"])))
    step = 1e-8 * (seed % 997)
    return 1e-8 * (1 + step if _taps(bb, 1e-8 * (1 + step)) == _taps(bb, 1e-8) else 1 - step)


def run(s):
    kind = s["case"]["kind"]
    if kind == "plan":
        s["plan"].run(s["x"].data_ptr(), *s["draws"], stream=s["stream"])
        return s["out"]
    if kind == "batch":
        s["batch"].launch(stream=s["stream"])
        return s["outs"]
    if kind == "fft":
        c = s["case"]
        gsfft.fft(s["x"].data_ptr(), s["y"].data_ptr(), 1 << c["log2n"], c["batch"], c["sign"], s["prec"],
                  stream=s["stream"])
        return s["y"]
    if kind == "filter":
        gsfft.design_filter(s["p"], s["ft"].data_ptr(), s["ff"].data_ptr(), stream=s["stream"])
        return [s["ft"], s["ff"]]
    if kind == "host":
        plan = s["plan"]
        gsfft.ingest(s["hx"], plan.precision, s["d_x"].data_ptr(), stream=s["stream"])
        plan.run(s["d_x"].data_ptr(), *s["draws"], stream=s["stream"])
        top = plan.results(stream=s["stream"])["topk"]
        s["spectrum"][top["key"]] = top["x"] + 1j * top["y"]
        return s["spectrum"]
    # drop_in: glibc's generators give the draws, as in the reference's program
    p, libc, L = s["p"], s["libc"], gsfft.lib()
    libc.srand48(ctypes.c_long(s["seed"]))
    libc.srandom(ctypes.c_uint(s["seed"]))
    count = ctypes.c_int(0)
    ptr = L.outer_loop(s["x"].data_ptr(), p.n, s["ft"].data_ptr(), s["ff"].data_ptr(), p.w, p.B, p.B_thresh,
                       p.W_RLFC, p.RLFC_loops, p.loops_thresh, p.loops_loc, p.loops, ctypes.byref(count),
                       ctypes.c_float(0.0))
    if not ptr:
        raise RuntimeError("outer_loop: " + gsfft.last_error())
    nodes = np.ctypeslib.as_array(ctypes.cast(ptr, ctypes.POINTER(ctypes.c_uint8)),
                                  (count.value * gsfft.NODE.itemsize,)).copy().view(gsfft.NODE)
    libc.free(ctypes.c_void_p(ptr))
    m = count.value
    s["keys"][:m], s["values"][:m, 0], s["values"][:m, 1] = nodes["key"], nodes["x"], nodes["y"]
    return [s["keys"], s["values"]]


def _work_sfft(c):
    n, B, W, w = _derived(c)[:4]
    es = 16 if c["precision"] == "fp64" else 8
    loops, R = c["loops_loc"] + c["loops_est"], c["RLFC_loops"]
    samples = min(n, loops * w + R * W)  # signal samples that the taps and the RLFC rows touch
    nbytes = es * (samples + w) + 24 * c["k"]
    flops = (8.0 * loops * w + 5.0 * loops * B * math.log2(B) + 5.0 * R * W * math.log2(W)
             + 8.0 * loops * 2 * c["k"])
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind == "fft":
        es = 16 if case["precision"] == "fp64" else 8
        N = case["batch"] << case["log2n"]
        return {"bytes": 2.0 * es * N, "flops": 5.0 * N * case["log2n"]}
    if kind == "batch":
        each = [_work_sfft(c) for c in _mix(case)]
        return {"bytes": float(sum(e[0] for e in each)), "flops": float(sum(e[1] for e in each))}
    if kind == "filter":
        n, _, _, w = _derived(case)[:4]
        return {"bytes": 16.0 * (w + n), "flops": 2 * 5.0 * n * case["q"] + 5.0 * w * math.log2(w)}
    nbytes, flops = _work_sfft(case)
    if kind == "host":
        nbytes = 16.0 * (1 << case["q"]) + 24 * case["k"]  # the host signal, read once
    return {"bytes": float(nbytes), "flops": float(flops)}


def _exact_filter(case, seed):
    q, tol = case["q"], _tolerance(case, seed)
    n = 1 << q
    bb = int(case["Bcst"] * math.sqrt(float(n) * case["k"] / math.log2(n)))
    w = _taps(bb, tol)
    b_f, t0 = int(1.2 * 1.1 * (float(n) / bb)), math.cosh(math.acosh(1 / tol) / (w - 1))
    f64 = dict(dtype=torch.float64, device="cuda")
    x = t0 * torch.cos(math.pi * torch.arange(w, **f64) / w)
    cheb = torch.where(x.abs() <= 1, torch.cos((w - 1) * torch.acos(x.clamp(-1, 1))),
                       torch.cosh((w - 1) * torch.acosh(x.clamp(min=1))))
    win = torch.where(x < -1, torch.zeros_like(x), cheb * tol)  # acosh below -1 is not a number: 0
    X = torch.fft.fft(win.to(torch.complex128)).real
    h = w // 2
    g = torch.zeros(n, **f64)
    g[:h] = X[:h]
    g[n - h:] = X[h + 1:2 * h + 1]
    G = torch.fft.fft(g.to(torch.complex128))
    # sums of b_f neighbours by doubling: few additions per output
    box, have, piece, size = None, 0, G, 1
    while size <= b_f:
        if b_f & size:
            box = piece if box is None else box + torch.roll(piece, -have)
            have += size
        piece, size = piece + torch.roll(piece, -size), size * 2
    ff = torch.roll(box, b_f // 2)
    ff = ff / ff.abs().max()
    m = (h * torch.arange(n, dtype=torch.int64, device="cuda")) % n
    ang = -2.0 * math.pi * (m.to(torch.float64) / n)
    ff = ff * torch.complex(torch.cos(ang), torch.sin(ang))
    return [torch.fft.ifft(ff)[:w].contiguous(), ff]


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        x = prepare(case, seed)["x"].to(torch.complex128)
        return torch.fft.fft(x) if case["sign"] < 0 else torch.fft.ifft(x, norm="forward")
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind == "host":
        loc, coef = synth.sparse_spectrum(1 << case["q"], case["k"], seed)  # no noise: the tones themselves
        spectrum = np.zeros(1 << case["q"], np.complex128)
        spectrum[loc] = coef
        return spectrum
    # The other kinds list their results in the order that the method's own
    # candidates have, which a plain transform does not give.
    return None
