"""Plans of small signals: bucket FFTs spread over two passes with all loops' rows in
one launch (B = 2^12, 2^13 in FP64), vote tables cleared by the run's first kernel up
to n = 2^20.

Bins against numpy: a bucket adds at most 33 products and its FFT has 13 levels, each
rounding to 2^-53 twice at most on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFGS = [(20, 1000, 1.4, 2, 2, 5, 128, 2), (18, 300, 1.0, 2, 2, 5, 128, 2), (20, 500, 1.0, 2, 2, 5, 128, 2),
        (21, 1000, 1.4, 2, 2, 5, 128, 2)]


def _plan(G, torch, cfg, prec):
    p, st = G.derive_params(*cfg, tolerance=1e-8)
    assert st == 0
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr())
    plan = G.Plan(p, prec)
    plan.set_filter(ft.data_ptr(), ff.data_ptr())
    return p, plan, ft


@pytest.mark.parametrize("cfg", CFGS)
def test_bins_of_every_loop(G, torch_cuda, cfg):
    torch = torch_cuda
    from gsfft import synth
    p, plan, ft = _plan(G, torch, cfg, G.FP64)
    rng = np.random.default_rng(5)
    x = rng.standard_normal(p.n) + 1j * rng.standard_normal(p.n)
    d_x = torch.as_tensor(x, device="cuda")
    offs, a, ai = synth.draws(3, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    plan.run(d_x.data_ptr(), offs, a, ai)
    torch.cuda.synchronize()
    bins = plan.debug_stages()["bins"]
    plan.close()
    taps, i = ft.cpu().numpy(), np.arange(p.w, dtype=np.int64)
    for l in range(p.loops):
        y = np.zeros(-(-p.w // p.B) * p.B, np.complex128)
        y[:p.w] = x[(i * int(ai[l])) % p.n] * taps
        ref = np.fft.fft(y.reshape(-1, p.B).sum(0))
        err = np.sqrt((np.abs(bins[l] - ref) ** 2).mean() / (np.abs(ref) ** 2).mean())
        assert err <= 2 * (33 + 2 * 13) * 2.0 ** -53


@pytest.mark.parametrize("cfg", [(14, 10, 2.5, 2, 2, 5, 16, 2)] + CFGS)
@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
def test_runs_leave_no_votes_behind(G, torch_cuda, cfg, prec):
    torch = torch_cuda
    from gsfft import synth
    prec = getattr(G, prec)
    p, plan, _ = _plan(G, torch, cfg, prec)
    xs = [synth.signal_torch(p.n, p.k, s)[0] for s in (1, 2)]
    xs = [x if prec == G.FP64 else x.to(torch.complex64) for x in xs]
    draws = [synth.draws(s, p.n, p.W_RLFC, p.RLFC_loops, p.loops) for s in (1, 2)]
    first = {}
    for k in (0, 1, 1, 0, 1):
        plan.run(xs[k].data_ptr(), *draws[k])
        r = plan.results()
        got = (r["nodes"].tobytes(), r["topk"].tobytes())
        if k not in first:
            _, fresh, _ = _plan(G, torch, cfg, prec)
            fresh.run(xs[k].data_ptr(), *draws[k])
            f = fresh.results()
            first[k] = (f["nodes"].tobytes(), f["topk"].tobytes())
            fresh.close()
        assert got == first[k]
    plan.close()
