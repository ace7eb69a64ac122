"""FP64 perm+filter in column order against the bucket-order gathers.

Both add the same at most 32 products of a bucket, in another order: each bin
differs by at most 2 * 32 * 2^-53 of the sum of the products' magnitudes, and
the B-point FFT that follows keeps that ratio (it is unitary up to scale).  With
noise for a signal and taps of about one size, that sum is below 8 times the
row's root mean square times sqrt(32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFGS = [  # (q, k, Bcst, loops_loc, loops_thresh, loops_est, RLFC_cst, RLFC_loops), tolerance
    ((14, 10, 2.5, 2, 2, 5, 16, 2), 1e-8),    # B = 256, n/W = 16
    ((16, 50, 1.0, 2, 2, 5, 128, 2), 1e-8),   # n/W = 2: sixteen RLFC columns a block
    ((16, 20, 1.0, 2, 2, 5, 8, 1), 1e-8),     # one RLFC loop
    ((18, 100, 1.0, 3, 2, 13, 32, 8), 1e-8),  # 16 loops, 8 RLFC loops
    ((20, 1000, 1.4, 2, 2, 5, 128, 2), 1e-8),  # n/W = 64: blocks without RLFC columns
    ((18, 100, 1.0, 2, 2, 5, 32, 2), 0.6),    # w < B: no full tile
    ((18, 100, 1.9, 2, 2, 5, 32, 2), 0.4),    # one full tile
    ((22, 777, 0.93, 2, 2, 7, 512, 2), 1e-8),
    # RLFC rows in pairs (first radix 2^10, 2^11, 2^12)
    ((20, 500, 1.0, 2, 2, 5, 2048, 2), 1e-8),
    ((22, 777, 0.93, 2, 2, 7, 4096, 2), 1e-8),
    ((23, 2000, 0.93, 2, 2, 7, 4096, 3), 1e-8),
    ((24, 1000, 2.5, 2, 2, 5, 16384, 2), 1e-8),
]


@pytest.mark.parametrize("cfg,tol", CFGS)
@pytest.mark.parametrize("quirk", [0, 1])
def test_column_order_matches_bucket_order(G, torch_cuda, cfg, tol, quirk):
    torch = torch_cuda
    from gsfft import synth
    p, st = G.derive_params(*cfg, tolerance=tol)
    assert st == 0
    g = torch.Generator(device="cuda").manual_seed(sum(cfg[:2]))
    rnd = dict(dtype=torch.complex128, device="cuda", generator=g)
    x, ft, ff = torch.randn(p.n, **rnd), torch.randn(p.w, **rnd), torch.randn(p.n, **rnd) + 2.0
    draws = synth.draws(7, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    flags = G.FLAG_QUIRK_RESIDUE if quirk else 0
    res = []
    for f in (flags, flags | G.FLAG_FORCE_GATHER):
        plan = G.Plan(p, G.FP64, f)
        plan.set_filter(ft.data_ptr(), ff.data_ptr())
        plan.run(x.data_ptr(), *draws)
        r = plan.results()
        res.append((plan.debug_stages(), r["nodes"]["key"].copy(), r["topk"]["key"].copy()))
        assert not plan.describe()["streaming"]
        plan.close()
    (a, ka, ta), (b, kb, tb) = res
    rms = np.sqrt((np.abs(b["bins"]) ** 2).mean(1, keepdims=True))
    assert (np.sqrt((np.abs(a["bins"] - b["bins"]) ** 2).mean(1, keepdims=True))
            <= 2 * 32 * 2.0 ** -53 * 8 * np.sqrt(32) * rms).all()
    np.testing.assert_array_equal(a["J2"], b["J2"])
    np.testing.assert_array_equal(a["J"], b["J"])
    np.testing.assert_array_equal(ka, kb)
    np.testing.assert_array_equal(ta, tb)
