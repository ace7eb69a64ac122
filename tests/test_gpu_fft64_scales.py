"""FP64 transforms of samples on very different scales, and plans of very small or very
large signals (the passes' FP64 form with its gathers, row pairs, |X|^2 and row maxima)."""
import numpy as np
import pytest

from gsfft import synth

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("log2n,batch", [(8, 1), (8, 17), (9, 3), (10, 2), (11, 3), (12, 1), (13, 1), (14, 2), (17, 1), (20, 1)])
@pytest.mark.parametrize("small", [1e-20, 1e-90, 2.0 ** -24])
def test_small_samples_beside_large_ones(G, torch_cuda, log2n, batch, small):
    """Ones at the even positions cancel exactly in all but two outputs; the others are
    the transform of the small samples at the odd positions, each output within
    log2(n) roundings of 2^-53 of them (relative L2, both sides)."""
    torch, n = torch_cuda, 1 << log2n
    rng = np.random.default_rng(log2n)
    odd = np.zeros((batch, n), np.complex128)
    odd[:, 1::2] = rng.standard_normal((batch, n // 2)) + 1j * rng.standard_normal((batch, n // 2))
    x = odd * small
    x[:, ::2] = 1.0
    d = torch.from_numpy(x).cuda()
    y = torch.empty_like(d)
    G.fft(d.data_ptr(), y.data_ptr(), n, batch, -1, G.FP64)
    y = y.cpu().numpy()
    want = np.fft.fft(odd.astype(np.clongdouble), axis=1)
    rest = np.ones(n, bool)
    rest[[0, n // 2]] = False
    assert np.allclose(y[:, 0], n / 2, rtol=1e-6) and np.allclose(y[:, n // 2], n / 2, rtol=1e-6)
    e = y[:, rest].astype(np.clongdouble) / np.longdouble(small) - want[:, rest]
    rel = np.sqrt((np.abs(e) ** 2).sum(1) / (np.abs(want[:, rest]) ** 2).sum(1))
    assert float(rel.max()) <= 2 * log2n * U


CFGS = [  # (configuration, flags by name)
    ((14, 10, 2.5, 2, 2, 5, 16, 2), ()),                      # B = 256: sixteen rows a CTA
    ((18, 100, 1.0, 2, 2, 5, 128, 2), ("FLAG_FORCE_GATHER",)),  # gathers in the first pass
    ((20, 1000, 1.4, 2, 2, 5, 128, 2), ()),                   # B = 2^13 in two passes
    ((20, 500, 1.0, 2, 2, 5, 2048, 2), ()),                   # W = 2^19
    ((22, 777, 0.93, 2, 2, 7, 4096, 2), ()),                  # W = 2^20: RLFC rows in pairs
    ((22, 777, 0.93, 3, 2, 5, 4096, 1), ("FLAG_FORCE_GATHER",)),
]


@pytest.mark.parametrize("cfg,flags", CFGS)
def test_plan_of_scaled_signal(G, torch_cuda, cfg, flags):
    """Powers of two scale everything exactly: the same bits inside the fixed-point range
    (2^+-200), the same picks and keys outside it (2^+-300), where the estimates are
    within rounding (one part in 10^12 of the largest, some 10^4 roundings)."""
    torch = torch_cuda
    p, st = G.derive_params(*cfg)
    assert st == G.OK
    x, *_ = synth.signal_torch(p.n, p.k, 3, 30.0)
    draws = synth.draws(3, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr())
    plan = G.Plan(p, G.FP64, sum(getattr(G, f) for f in flags))
    plan.set_filter(ft.data_ptr(), ff.data_ptr())

    def run(scale):
        z = x * scale
        plan.run(z.data_ptr(), *draws)
        r, d = plan.results(), plan.debug_stages()
        assert r["status"] == G.OK
        v = (r["nodes"]["x"] + 1j * r["nodes"]["y"]) / scale
        return d["J2"], d["J"], r["nodes"]["key"], r["topk"]["key"], v

    base = run(1.0)
    for scale in (2.0 ** -200, 2.0 ** 200, 2.0 ** -300, 2.0 ** 300):
        got = run(scale)
        for a, b in zip(got[:4], base[:4]):
            np.testing.assert_array_equal(a, b)
        if abs(np.log2(scale)) < 250:
            np.testing.assert_array_equal(got[4], base[4])
        else:
            assert np.abs(got[4] - base[4]).max() <= 1e-12 * np.abs(base[4]).max()
    plan.close()
