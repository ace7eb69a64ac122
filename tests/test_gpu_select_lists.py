"""Cutoffs against a stable sort over value distributions that take each branch of
the single-launch selection: ranks inside noise, ties at the threshold, fewer
non-zero samples than wanted (the first zeros fill up), large values lying together
(a warp's list runs over), one value everywhere, rows of odd length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(kind, rng, batch, size, num):
    x = rng.standard_exponential((batch, size))
    if kind == "ties":
        x = np.floor(4 * x) / 4
    elif kind == "few":
        x[rng.random((batch, size)) > 0.4 * num / size] = 0.0
    elif kind == "exact":  # num non-zero samples
        for r in x:
            r[rng.permutation(size)[num:]] = 0.0
    elif kind == "one_over":
        for r in x:
            r[rng.permutation(size)[num + 1:]] = 0.0
    elif kind == "together":
        x *= 1e-6
        a = size // 3
        x[:, a:a + num + num // 4] += 5.0
    elif kind == "equal":
        x[:] = 0.25
    elif kind == "wide":
        x = np.exp(12 * rng.standard_normal((batch, size)))
    elif kind == "zeros":
        x[:] = 0.0
        x[:, -1] = 1.0
    elif kind == "mixed":  # rows that settle in different ways behind one barrier
        x[0, rng.permutation(size)[num // 2:]] = 0.0
        x[-1] = np.floor(x[-1])
    return x


def expect(x, num, floor_rel, dtype):
    out = []
    for r in x.astype(dtype):
        f = dtype(np.float64(r.max()) * floor_rel)
        r = np.where(r < f, dtype(0), r)
        out.append(np.sort(np.argsort(-r, kind="stable")[:num]))
    return np.array(out, np.int32)


SHAPES = [(300, 7, 1), (2049, 1000, 2), (8192, 2000, 5), (65537, 1234, 1), (131072, 32000, 2), (262144, 86000, 2),
          (300001, 4000, 2), (1 << 20, 5000, 3), (1 << 20, 100, 1), (1 << 22, 32000, 2)]


@pytest.mark.parametrize("size,num,batch", SHAPES)
@pytest.mark.parametrize("kind", ["noise", "ties", "few", "exact", "one_over", "together", "equal", "wide", "zeros",
                                  "mixed"])
@pytest.mark.parametrize("prec", [0, 1])
def test_cutoff_branches(G, torch_cuda, size, num, batch, kind, prec):
    torch = torch_cuda
    dtype = (np.float64, np.float32)[prec]
    x = rows(kind, np.random.default_rng(size + num), batch, size, num).astype(dtype)
    d = torch.from_numpy(x).cuda()
    for floor_rel in (0.0, 1e-10):
        want = expect(x, num, floor_rel, dtype)
        for _ in range(2):  # the second call finds the scratch as the first left it
            out = torch.full((batch, num), -1, dtype=torch.int32, device="cuda")
            G.cutoff_floor(d.data_ptr(), size, num, batch, prec, floor_rel, out.data_ptr())
            np.testing.assert_array_equal(out.cpu().numpy(), want)
    if size <= G.NOALLOC_MAX_SIZE and batch <= G.NOALLOC_MAX_BATCH:
        out = torch.full((batch, num), -1, dtype=torch.int32, device="cuda")
        G.cutoff_noalloc(d.data_ptr(), size, num, batch, prec, out.data_ptr())
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), expect(x, num, 0.0, dtype))


@pytest.mark.parametrize("prec", [0, 1])
def test_selection_leaves_its_scratch_clean(G, torch_cuda, prec):
    """A plan keeps its selection scratch: runs of rows that settle in different
    ways, one after the other, on the same plan."""
    torch = torch_cuda
    from gsfft import synth
    p, st = G.derive_params(20, 1000, 1.40, 2, 2, 5, 128, 2)
    assert st == 0
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr())
    plan = G.Plan(p, prec)
    plan.set_filter(ft.data_ptr(), ff.data_ptr())
    seen = {}
    for k, snr in ((1, None), (2, 30.0), (3, None), (1, None), (2, 30.0), (3, None)):
        x, _, _, _ = synth.signal_torch(p.n, p.k, k, snr)
        if k == 3:
            x = torch.zeros_like(x)
            x[5] = 1.0  # every bin equal in magnitude
        x = x if prec == 0 else x.to(torch.complex64)
        plan.run(x.data_ptr(), *synth.draws(k, p.n, p.W_RLFC, p.RLFC_loops, p.loops))
        r = plan.results()
        key = r["topk"]["key"].tolist()
        assert seen.setdefault(k, key) == key
