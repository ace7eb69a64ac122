"""The filter design, to the bit.

Mixed-precision plans round the taps and the response to FP32, where a change in the
last FP64 bits of the design shows as a change in the last FP32 bit of estimates
(relative 1e-7).  So the design's bits are part of what a mixed plan returns: these
are digests of the taps and of the response as FP64 arithmetic gives them, in the
order of the sums and with the transforms of the design as it was first built (one,
two and three passes; the two largest are the shapes of the 2^27-point plans)."""
import hashlib

import pytest

pytestmark = pytest.mark.gpu

DIGESTS = [
    ((13, 60, 1.4, 2, 2, 5, 16, 2), "a745e299a2306c3f", "40e537fda5bc05bf"),
    ((14, 10, 2.5, 2, 2, 5, 16, 2), "75543e8b840710ec", "12f637a4c3d041fd"),
    ((17, 200, 0.8, 2, 2, 5, 64, 2), "96d1dc1e8aa91c6c", "9b2c692c47322d71"),
    ((20, 1000, 1.4, 2, 2, 5, 128, 2), "3a400a97a1f09961", "f15113a85a090816"),
    ((22, 2000, 1.0, 2, 2, 5, 512, 2), "d43dfae445d078bf", "b7f8f0b564d544cf"),
    ((25, 700, 0.9, 2, 2, 7, 512, 2), "46c18f203dabaed4", "9086b3b1a18e6bc0"),
    ((27, 16000, 0.65, 2, 2, 7, 4096, 2), "8196762337932778", "a76af8ff28ae5c2a"),
    ((27, 43000, 0.8, 3, 2, 8, 32768, 2), "240c3cda0bd671dc", "54e9f4947f97a635"),
]


def digest(t):
    return hashlib.sha256(t.cpu().numpy().tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("cfg,taps,response", DIGESTS)
def test_design_bits(G, torch_cuda, cfg, taps, response):
    torch = torch_cuda
    p, st = G.derive_params(*cfg)
    assert st == G.OK
    ft = torch.zeros(p.w, dtype=torch.complex128, device="cuda")
    ff = torch.zeros(p.n, dtype=torch.complex128, device="cuda")
    G.design_filter(p, ft.data_ptr(), ff.data_ptr())
    assert digest(ft) == taps
    assert digest(ff) == response
