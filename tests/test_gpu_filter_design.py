"""Filter design kernels against plain torch in double precision.

Five transforms in a chain, each within about log2 n roundings of 2^-53 on
either side, and sums and products of a few more: relative L2 within
5 log2(n) 2^-53 for the taps and the response."""
import math

import pytest

pytestmark = pytest.mark.gpu

# (q, k, Bcst, ...): n below and above one boxcar tile of 4096 outputs, odd and even
# b_f, windows from a fraction of n to almost all of it, one- and two-pass transforms
CFGS = [(13, 60, 1.4, 2, 2, 5, 16, 2), (13, 60, 2.8, 2, 2, 5, 16, 2), (14, 10, 2.5, 2, 2, 5, 16, 2),
        (15, 30, 1.7, 2, 2, 5, 16, 2), (17, 200, 0.8, 2, 2, 5, 64, 2), (19, 77, 1.1, 2, 2, 5, 128, 2)]


def design(torch, p):
    """The flat window of cuExperiment.cu:277-448 with torch.fft."""
    n, w, f64 = p.n, p.w, dict(dtype=torch.float64, device="cuda")
    x = p.t0 * torch.cos(math.pi * torch.arange(w, **f64) / w)
    cheb = torch.where(x.abs() <= 1, torch.cos((w - 1) * torch.acos(x.clamp(-1, 1))),
                       torch.cosh((w - 1) * torch.acosh(x.clamp(min=1))))
    win = torch.where(x < -1, torch.zeros_like(x), cheb * p.tolerance)
    X, h = torch.fft.fft(win.to(torch.complex128)).real, w // 2
    g = torch.zeros(n, **f64)
    g[:h], g[n - h:] = X[:h], X[h + 1:2 * h + 1]
    G = torch.fft.fft(g.to(torch.complex128))
    box, have, piece, size = None, 0, G, 1  # sums of b_f neighbours by doubling
    while size <= p.b_f:
        if p.b_f & size:
            box = piece if box is None else box + torch.roll(piece, -have)
            have += size
        piece, size = piece + torch.roll(piece, -size), size * 2
    ff = torch.roll(box, p.b_f // 2)
    ff = ff / ff.abs().max()
    ang = -2.0 * math.pi * ((h * torch.arange(n, dtype=torch.int64, device="cuda")) % n).double() / n
    ff = ff * torch.complex(torch.cos(ang), torch.sin(ang))
    return torch.fft.ifft(ff)[:w], ff


@pytest.mark.parametrize("cfg", CFGS)
@pytest.mark.parametrize("b_f_step", [0, 1])
@pytest.mark.parametrize("keep_response", [True, False])
def test_filter_design_matches_torch(G, torch_cuda, cfg, b_f_step, keep_response):
    torch = torch_cuda
    p, _ = G.derive_params(*cfg)
    p.b_f += b_f_step  # either parity
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr() if keep_response else 0)
    want_t, want_f = design(torch, p)
    tol = 5 * p.q * 2.0 ** -53
    assert float((ft - want_t).norm() / want_t.norm()) <= tol
    if keep_response:
        assert float((ff - want_f).norm() / want_f.norm()) <= tol
