"""The tuning cache of FP64 plans: bucket-order and column-order gathers are different
plans (GSFFT_FLAG_FORCE_GATHER), and lines from before the column order are no answer."""
import pytest

from gsfft import synth

pytestmark = pytest.mark.gpu


def test_gather_orders_do_not_share_lines(G, torch_cuda, tmp_path):
    torch = torch_cuda
    p, st = G.derive_params(18, 100, 1.0, 2, 2, 5, 128, 2)
    assert st == G.OK
    x, *_ = synth.signal_torch(p.n, p.k, 1, 30.0)
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr())
    draws = synth.draws(1, p.n, p.W_RLFC, p.RLFC_loops, p.loops)
    cache = tmp_path / "tuning.txt"

    def tune(flags):
        t, ms = G.autotune_plan(p, G.FP64, flags, x.data_ptr(), ft.data_ptr(), ff.data_ptr(), *draws, reps=2,
                                cache_path=str(cache))
        return t.as_dict(), ms, cache.read_text().splitlines()

    _, _, lines = tune(0)
    assert len(lines) == 1
    _, _, lines = tune(G.FLAG_FORCE_GATHER)
    assert len(lines) == 2 and lines[0].split()[1] != lines[1].split()[1]
    # a line as it was written when the ordered pass and bucket order were the forms
    tag, key = lines[0].split()[:2]
    old = key.replace("|gather=cols", "")
    assert old != key
    cache.write_text(f"{tag} {old} pf=1 groups=1 br=0 rr=0 sel=1 ms=0.00001\n")
    _, ms, lines = tune(0)
    assert ms > 0.001 and len(lines) == 2
