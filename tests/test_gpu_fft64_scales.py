"""FP64 plans of very small or very large signals (the passes' FP64 form with its gathers,
row pairs, |X|^2 and row maxima)."""
import numpy as np
import pytest

from gsfft import synth

pytestmark = pytest.mark.gpu

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
