"""Reverse-hash voting against the oracle at the shapes where the walk changes:
windows of 2 to 4096 positions (1 to 32 lanes a bucket, one and several steps),
write passes with a thread and with a warp per bucket, buckets with more
candidates than slots in both, windows that wrap around the residues."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n, B, W, heavy buckets, residues, how they lie
CASES = [
    (1 << 16, 1 << 15, 256, 9001, 20, "spread"),
    (1 << 16, 1 << 11, 128, 1500, 40, "spread"),
    (1 << 20, 1 << 14, 8192, 9000, 500, "spread"),
    (1 << 20, 1 << 14, 8192, 100, 8000, "spread"),     # nearly every position
    (1 << 19, 1 << 11, 1024, 1100, 90, "together"),    # few buckets, over 32 candidates
    (1 << 22, 1 << 12, 16384, 3000, 700, "spread"),
    (1 << 22, 1 << 10, 65536, 901, 300, "ends"),       # windows of 4096, wrapping residues
    (1 << 24, 1 << 14, 32768, 9000, 200, "together"),  # many buckets, some over 32 candidates
    (1 << 23, 1 << 15, 2048, 20000, 300, "spread"),    # many buckets, dense windows
]


@pytest.mark.parametrize("n,B,W,Bt,nres,lie", CASES)
@pytest.mark.parametrize("thresh", [1, 2])
def test_vote_walk_matches_oracle(G, O, torch_cuda, n, B, W, Bt, nres, lie, thresh):
    torch = torch_cuda
    rng = np.random.default_rng(n + nres)
    if lie == "spread":
        J2 = rng.choice(W, nres, replace=False)
    elif lie == "together":
        J2 = W // 3 + np.arange(nres)
    else:
        J2 = (W - nres // 2 + np.arange(nres)) % W
    J2 = np.sort(J2).astype(np.int32)
    cap, cand_o, count = 1 << 21, [], 0
    vote_o = np.zeros(n, np.int32)
    d_vote = torch.zeros(n, dtype=torch.int32, device="cuda")
    d_cand = torch.zeros(cap, dtype=torch.int32, device="cuda")
    d_J2 = torch.from_numpy(J2).cuda()
    for _ in range(2):
        # a = 1 keeps the residues as they lie; then a random permutation
        a = 1 if not len(cand_o) and thresh == 1 else int(rng.integers(0, n // 2)) * 2 + 1
        ai = pow(a, -1, n)
        J = np.sort(rng.choice(B, Bt, replace=False)).astype(np.int32)
        c, vote_o, _ = O.reverse_hash(J, J2, n, B, W, a, ai, thresh, vote=vote_o, cand=cand_o, cap=cap)
        cand_o = list(c)
        d_J = torch.from_numpy(J).cuda()
        s, count = G.stage_reverse_hash(d_J.data_ptr(), J.size, d_J2.data_ptr(), J2.size, n, B, W, a, ai, thresh, 0,
                                        d_vote.data_ptr(), d_cand.data_ptr(), cap, count)
        assert s == G.OK
    assert count == len(cand_o)
    np.testing.assert_array_equal(d_cand.cpu().numpy()[:count], np.array(cand_o, np.int32))
    np.testing.assert_array_equal(d_vote.cpu().numpy(), vote_o)
