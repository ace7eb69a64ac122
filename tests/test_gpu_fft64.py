"""The FP64 FFT (fixed-point passes) against an extended-precision transform.

A pass rounds every output once (half a unit of 2^-53 per component) and its
fixed-point part adds less than a quarter of that, so a transform of p passes
is within p * 1.25 * 2^-53 of the exact one (relative L2).  Samples spread over
many orders of magnitude share one exponent per sub-transform: two bits less.
Values outside the fixed-point range take the FP64 form of the pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def run(G, torch, x, sign):
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    y = torch.empty_like(d)
    G.fft(d.data_ptr(), y.data_ptr(), x.shape[1], x.shape[0], sign, G.FP64)
    return y.cpu().numpy()


def exact(x, sign):
    x = x.astype(np.clongdouble)
    return np.fft.fft(x) if sign < 0 else np.fft.ifft(x) * x.shape[1]


def worst(y, X):
    e, n = np.sqrt((np.abs(y - X) ** 2).sum(1)), np.sqrt((np.abs(X) ** 2).sum(1))
    return float((e / n).max())  # in extended precision: rows may be tiny


def passes(log2n):
    return 1 if log2n <= 13 else (2 if log2n <= 24 else 3)


# every radix 2^7 .. 2^13 as the only pass, first and second passes of all
# radices, batches that leave the last CTA's rows partly empty
SIZES = [(8, 1), (8, 7), (9, 3), (10, 3), (11, 1), (11, 3), (12, 1), (13, 2), (14, 1), (15, 3), (16, 1), (17, 3),
         (18, 1), (19, 1)]


@pytest.mark.parametrize("log2n,batch", SIZES)
@pytest.mark.parametrize("sign", [-1, 1])
def test_fft64_error(G, torch_cuda, log2n, batch, sign):
    n, tol = 1 << log2n, passes(log2n) * 1.25 * U
    rng = np.random.default_rng(100 * log2n + batch)
    noise = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    impulse = np.zeros((batch, n), np.complex128)
    impulse[np.arange(batch), rng.integers(0, n, batch)] = 0.7 - 0.3j
    tone = np.exp(2j * np.pi * ((np.arange(n)[None, :] * rng.integers(1, n, (batch, 1))) % n) / n)
    rows = noise * 10.0 ** (-30.0 * np.arange(batch))[:, None]  # each row keeps its own scale
    for x, t in ((noise, tol), (impulse, tol), (tone, tol), (rows, tol),
                 (noise * np.exp(10 * rng.standard_normal(noise.shape)), 4 * tol)):
        assert worst(run(G, torch_cuda, x, sign), exact(x, sign)) <= t


@pytest.mark.parametrize("log2n,batch", [(8, 3), (11, 3), (13, 2), (14, 2), (17, 1)])
def test_fft64_outside_fixed_point(G, torch_cuda, log2n, batch):
    """FP64 arithmetic (about log2 n roundings of 2^-53 per point) for very
    large and very small samples; zeros stay zeros; infinities and NaN do not
    disappear."""
    n = 1 << log2n
    rng = np.random.default_rng(log2n)
    x = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    X = exact(x, -1)
    for scale in (1e-200, 1e-90, 1e200, 1e-280):
        y = run(G, torch_cuda, x * scale, -1)
        assert worst(y.astype(np.clongdouble) / np.longdouble(scale), X) <= 2 * log2n * U
    mixed = x.copy()
    mixed[0] *= 1e200  # a row in FP64 beside rows in fixed point
    y = run(G, torch_cuda, mixed, -1)
    y[0] /= 1e200
    assert worst(y, X) <= 2 * log2n * U
    assert not run(G, torch_cuda, np.zeros_like(x), -1).any()
    tiny = np.full((batch, n), 3 * 2.0 ** -1074 + 0j)  # subnormals: their sum is exact
    y = run(G, torch_cuda, tiny, -1)
    assert (y[:, 0] == 3 * n * 2.0 ** -1074).all()
    for bad in (np.inf, np.nan):
        z = x.copy()
        z[batch - 1, n // 3] = bad
        y = run(G, torch_cuda, z, -1)
        assert not np.isfinite(y[batch - 1]).any()
        if batch > 1:
            assert np.isfinite(y[0]).all()
