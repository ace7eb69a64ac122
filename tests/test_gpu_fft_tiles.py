"""Two-pass FP32 transforms whose array between the passes is kept in tiles (radices
2^11 / 2^12, then 2^10 .. 2^12), against FP64.  Each of the L radix-2 levels adds
rounding of at most about 2^-24 of the row's root mean square, the twiddle products
as much again."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,batch", [(21, 1), (21, 3), (22, 2), (23, 1), (24, 2)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_tiled_passes(G, torch_cuda, L, batch, sign):
    torch = torch_cuda
    n = 1 << L
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn(batch, n, dtype=torch.complex64, device="cuda", generator=g)
    x[:, 1] += 100.0  # a row that is not symmetric under the tile's index swaps
    y = torch.empty_like(x)
    G.fft(x.data_ptr(), y.data_ptr(), n, batch, sign, G.MIXED)
    torch.cuda.synchronize()
    for b in range(batch):
        ref = torch.fft.fft(x[b].to(torch.complex128)) if sign < 0 else torch.fft.ifft(x[b].to(torch.complex128)) * n
        rms = float(ref.abs().square().mean().sqrt())
        assert float((y[b] - ref).abs().square().mean().sqrt()) <= 2 * L * 2.0 ** -24 * rms


@pytest.mark.parametrize("L,batch", [(20, 2), (21, 1), (22, 2), (23, 1)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_tiled_passes_fp64(G, torch_cuda, L, batch, sign):
    """Pairs of sub-transforms, radices 2^10 .. 2^12; the second run's values lie below
    the fixed-point range (exponents under -800), so both passes take their FP64 form."""
    torch = torch_cuda
    n = 1 << L
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn(batch, n, dtype=torch.complex128, device="cuda", generator=g)
    x[:, 1] += 100.0
    refs = [torch.fft.fft(r) if sign < 0 else torch.fft.ifft(r) * n for r in x]
    for scale in (1.0, 2.0 ** -850):
        xs = x * scale
        y = torch.empty_like(x)
        G.fft(xs.data_ptr(), y.data_ptr(), n, batch, sign, G.FP64)
        torch.cuda.synchronize()
        for b in range(batch):
            rms = float(refs[b].abs().square().mean().sqrt())
            err = y[b] / scale - refs[b]
            assert float(err.abs().square().mean().sqrt()) <= 4 * L * 2.0 ** -53 * rms  # both sides round
