"""Ordered perm+filter pass (FP32): its bins against the gather form's, and the RLFC
candidates against an FP64 transform of the sub-samples.

Both forms add the same at most 33 products of a bucket, in another order: each bin
differs by at most 2 * 33 * 2^-24 of the sum of the products' magnitudes, which for
noise and taps of about one size is below 8 sqrt(33) times the row's root mean
square; the B-point FFT that follows keeps that ratio, with log2(B) <= 17 more
roundings of each side.  An FP32 transform of W points is within 4 log2(W) 2^-24 of
the spectrum's root mean square of its exact values: only samples that close to the
cutoff may be on either side of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFGS = [  # (q, k, Bcst, loops_loc, loops_thresh, loops_est, RLFC_cst, RLFC_loops), tolerance, row groups, radix
    ((14, 10, 2.5, 2, 2, 5, 16, 2), 1e-8, 0, 0),      # 64 rows: one tile an item
    ((16, 50, 1.0, 2, 2, 5, 128, 2), 1e-8, 1, 0),     # n/W = 2: eight RLFC columns a tile
    ((18, 100, 1.0, 3, 2, 13, 32, 8), 1e-8, 1, 0),    # 16 loops, 8 RLFC loops, n/W = 32
    ((18, 100, 1.0, 2, 2, 5, 32, 2), 0.6, 1, 0),      # w < B: no full tile
    ((22, 777, 0.93, 2, 2, 7, 512, 2), 1e-8, 0, 0),
    ((22, 777, 0.93, 2, 2, 7, 4096, 2), 1e-8, 2, 0),  # y in row blocks (radix 2^11), two row groups
    ((23, 2000, 0.93, 2, 2, 7, 4096, 3), 1e-8, 0, 0),
    ((24, 1000, 2.5, 2, 2, 5, 16384, 2), 1e-8, 1, 12),  # row blocks, radix 2^12: 16 columns of y a row
    ((24, 1000, 2.5, 2, 2, 5, 8192, 2), 1e-8, 1, 10),   # radix 2^10: y in order
]


@pytest.mark.parametrize("cfg,tol,groups,radix", CFGS)
def test_stream_tiles(G, torch_cuda, cfg, tol, groups, radix):
    torch = torch_cuda
    from gsfft import synth
    p, st = G.derive_params(*cfg, tolerance=tol)
    assert st == 0
    g = torch.Generator(device="cuda").manual_seed(sum(cfg[:2]))
    rnd = dict(dtype=torch.complex64, device="cuda", generator=g)
    x, ft = torch.randn(p.n, **rnd), torch.randn(p.w, **rnd)
    ff = torch.randn(p.n, dtype=torch.complex128, device="cuda", generator=g) + 2.0
    ft64 = ft.to(torch.complex128)
    draws = synth.draws(7, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    res = []
    for flag in (G.FLAG_FORCE_STREAM, G.FLAG_FORCE_GATHER):
        t = G.Tuning()
        t.rlfc_first_radix = radix
        if flag == G.FLAG_FORCE_STREAM:
            t.row_groups = groups
        plan = G.Plan(p, G.MIXED, flag, tuning=t)
        plan.set_filter(ft64.data_ptr(), ff.data_ptr())
        plan.run(x.data_ptr(), *draws)
        torch.cuda.synchronize()
        res.append(plan.debug_stages())
        assert plan.describe()["streaming"] == (flag == G.FLAG_FORCE_STREAM)
        plan.close()
    a, b = res
    rms = np.sqrt((np.abs(b["bins"]) ** 2).mean(1, keepdims=True))
    tol_b = (2 * 33 * 8 * np.sqrt(33) + 2 * 4 * 17) * 2.0 ** -24
    assert (np.sqrt((np.abs(a["bins"] - b["bins"]) ** 2).mean(1, keepdims=True)) <= tol_b * rms).all()
    must = torch.zeros(p.W_RLFC, dtype=torch.bool, device="cuda")
    may = must.clone()
    for off in draws[0]:
        X = torch.fft.fft(x[int(off)::p.n // p.W_RLFC].to(torch.complex128)).abs()
        dev = 4 * np.log2(p.W_RLFC) * 2.0 ** -24 * float(X.square().mean().sqrt())
        cut = float(torch.topk(X, p.B_thresh).values[-1])
        must |= X > cut + 2 * dev
        may |= X >= cut - 2 * dev
    got = torch.zeros_like(must)
    got[torch.as_tensor(a["J2"].astype(np.int64), device="cuda")] = True  # union of the loops' picks
    assert bool((may | ~got).all()) and bool((got | ~must).all())
