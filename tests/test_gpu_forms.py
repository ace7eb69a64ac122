"""That FP64 plans take the column order by default: its sums run in another order than
bucket order's (GSFFT_FLAG_FORCE_GATHER), so of thousands of bins some differ in their
last bits, where the same form twice gives the same bits."""
import numpy as np
import pytest

from gsfft import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [(14, 10, 2.5, 2, 2, 5, 16, 2), (18, 100, 1.0, 3, 2, 13, 32, 8),
                                 (22, 777, 0.93, 2, 2, 7, 4096, 2)])
def test_fp64_default_is_column_order(G, torch_cuda, cfg):
    torch = torch_cuda
    p, st = G.derive_params(*cfg)
    assert st == G.OK and p.w >= 4 * p.B
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = dict(dtype=torch.complex128, device="cuda", generator=g)
    x, ft, ff = torch.randn(p.n, **rnd), torch.randn(p.w, **rnd), torch.randn(p.n, **rnd) + 2.0
    bins = []
    for flags in (0, 0, G.FLAG_FORCE_GATHER):
        plan = G.Plan(p, G.FP64, flags)
        plan.set_filter(ft.data_ptr(), ff.data_ptr())
        plan.run(x.data_ptr(), *synth.draws(7, p.n, p.W_RLFC, p.RLFC_loops, p.loops))
        torch.cuda.synchronize()
        bins.append(plan.debug_stages()["bins"])
        plan.close()
    np.testing.assert_array_equal(bins[0], bins[1])
    assert (bins[0] != bins[2]).mean() > 0.1
