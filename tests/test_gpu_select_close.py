"""Cutoffs of samples that lie close together: the digit of the num-th largest holds more
samples than are ranked (it is counted again in finer parts, down to single values), the
lists of a whole octave would run over, many samples share the deciding value, rows of
one call settle at different depths.  Against a stable sort (ties: lowest index)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(kind, rng, batch, size, num):
    x = rng.random((batch, size))
    if kind == "near one":  # estimates of a noiseless signal
        x = 1.0 + 1e-6 * x
        x[:, ::7] *= 1e-9
    elif kind == "seven":
        x = np.floor(7 * x)
    elif kind == "steps":  # runs of equal values at every depth of the digits
        x = 1.0 + np.floor(2 * x) * 2.0 ** -4 + np.floor(3 * rng.random(x.shape)) * 2.0 ** -14 + np.floor(
            2 * rng.random(x.shape)) * 2.0 ** -22
    elif kind == "last bits":
        x = 1.0 + np.floor(x * 3 * size) * 2.0 ** -52
    elif kind == "rows":  # uniform, ties, spread, few
        x[0] = np.floor(5 * x[0])
        if batch > 2:
            x[1] = np.exp(20 * x[1])
            x[2, num // 2:] = 0.0
        x[-1] = 0.5 + x[-1] * 2.0 ** -30
    return x


def expect(x, num):
    return np.array([np.sort(np.argsort(-r, kind="stable")[:num]) for r in x], np.int32)


# one CTA, clusters, one grid over the rows; few and many of the samples wanted
SHAPES = [(500, 300, 3), (2048, 100, 8), (4096, 1000, 2), (30001, 9000, 2), (131072, 2000, 3), (262144, 40000, 1),
          (262145, 40000, 4), (1 << 20, 1 << 18, 1), ((1 << 21) + 6, 3000, 2), (1 << 22, 32000, 1)]


@pytest.mark.parametrize("size,num,batch", SHAPES)
@pytest.mark.parametrize("kind", ["uniform", "near one", "seven", "steps", "last bits", "rows"])
@pytest.mark.parametrize("prec", [0, 1])
def test_close_samples(G, torch_cuda, size, num, batch, kind, prec):
    torch = torch_cuda
    x = rows(kind, np.random.default_rng(size + num), batch, size, num).astype((np.float64, np.float32)[prec])
    want = expect(x, num)
    d = torch.from_numpy(x).cuda()
    for floor_rel in (0.0, 1e-300):  # without and with row maxima; again on the same scratch
        out = torch.full((batch, num), -1, dtype=torch.int32, device="cuda")
        G.cutoff_floor(d.data_ptr(), size, num, batch, prec, floor_rel, out.data_ptr())
        np.testing.assert_array_equal(out.cpu().numpy(), want)
    for _ in range(2):
        out = torch.full((batch, num), -1, dtype=torch.int32, device="cuda")
        G.cutoff_noalloc(d.data_ptr(), size, num, batch, prec, out.data_ptr())
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
