// Device code of the voting stage (A7): the block bodies of the mark, count
// and write passes, with the block index and block count as arguments, so
// that the per-plan kernels (vote.cu) and the persistent kernel that runs the
// tails of a whole batch (batch_tail.cu) run the same code.  Loads of data
// that another block of the same launch may have written (the vote table, the
// bucket counts, the stashed candidates, the loop's first candidate) bypass L1
// (ld.global.cg), so the persistent kernel sees what its earlier work items wrote.
#pragma once
#include "stages.cuh"

namespace gsfft {

namespace {

constexpr int VT = 256;  // threads per block in this file

__device__ __forceinline__ unsigned blk_excl_scan(unsigned v, unsigned *ws, unsigned *total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[wid] = x;
  __syncthreads();
  if (wid == 0) {
    unsigned w = lane < VT / 32 ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < VT / 32) ws[lane] = w;
  }
  __syncthreads();
  unsigned base = wid ? ws[wid - 1] : 0;
  unsigned tot = ws[VT / 32 - 1];
  __syncthreads();
  if (total) *total = tot;
  return base + x - v;
}

__device__ __forceinline__ unsigned blk_sum(unsigned v, unsigned *ws) {
  unsigned t;
  blk_excl_scan(v, ws, &t);
  return t;
}

// ------------------------------------------------------------ voting
struct WalkArgs {
  const int *J;
  int Bt, n, nb, W;
  const unsigned *bm;
  const int *fmax;
  unsigned a;
  int packed;  // vote tables of 2-bit counters (16 per word; two tables used on alternate
               // runs) instead of epoch-tagged 32-bit entries
};

// The vote table.  Epoch-tagged: entry = epoch << 8 | count, never cleared
// between runs, read and written plainly (a location is visited at most once
// per pass).  Packed (at most 3 location loops, so counts fit 2 bits): 16
// counters per word, n / 4 bytes -- small enough to stay in L2 -- updated
// with word atomics, since neighbouring locations share a word.  There are
// two packed tables, the run with epoch e using table e & 1; after a run's
// voting the other one is cleared for the next run (vote_clear_kernel), so
// the clear overlaps the run's latency-bound tail; for small n the run's first
// kernel clears both.
__device__ __forceinline__ unsigned *packed_table(const WalkArgs &w, unsigned *vote, unsigned epoch) {
  return vote + ((epoch & 1u) ? ((unsigned)w.n >> 4) : 0u);
}
// vote_update: the votes of up to four visited locations, independent so
// that their table accesses overlap; cnt[q] = the count after the vote.
__device__ __forceinline__ void vote_update(const WalkArgs &w, unsigned epoch, unsigned *vote,
                                            const unsigned (&loc)[4], int nq, unsigned (&cnt)[4]) {
  if (w.packed) {
    unsigned *tab = packed_table(w, vote, epoch);
    unsigned old[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < nq) old[q] = atomicAdd(&tab[loc[q] >> 4], 1u << (2 * (loc[q] & 15u)));
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < nq) cnt[q] = ((old[q] >> (2 * (loc[q] & 15u))) & 3u) + 1u;
    return;
  }
  unsigned e[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (q < nq) e[q] = __ldcg(&vote[loc[q]]);
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (q < nq) {
      const unsigned cv = ((e[q] >> 8) == epoch) ? (e[q] & 255u) + 1u : 1u;
      vote[loc[q]] = (epoch << 8) | cv;
      cnt[q] = cv;
    }
}
// whether location loc's count is exactly the threshold (after a pass's votes)
__device__ __forceinline__ bool vote_at_threshold(const WalkArgs &w, unsigned epoch, const unsigned *vote,
                                                  unsigned loc, unsigned thresh) {
  if (w.packed) {
    const unsigned *tab = vote + ((epoch & 1u) ? ((unsigned)w.n >> 4) : 0u);
    return ((__ldcg(&tab[loc >> 4]) >> (2 * (loc & 15u))) & 3u) == thresh;
  }
  return __ldcg(&vote[loc]) == ((epoch << 8) | thresh);
}

// low = ceil((J - 0.5) * n/B) reduced mod n (innerLoop.cu:792), in integers.
__device__ __forceinline__ int window_low(int J, int n, int nb) {
  const long long v = (2LL * J - 1) * nb;  // 2 * (J - 0.5) * nb
  const long long c = v >= 0 ? (v + 1) / 2 : -((-v) / 2);
  return (int)((c + n) & (long long)(n - 1));
}

// A group of lpb lanes walks a heavy bucket: lane s of the group holds the 32
// offsets c0 + 32 s .. + 31 of its window [low, low + n/B) as one mask (two bitmap
// words and a funnel shift, whatever the alignment), so a window of 1024 offsets is
// one step and all its table accesses overlap; 32 / lpb buckets share a warp.
// Lanes, then bits, in ascending order give the window in ascending order.
__host__ __device__ __forceinline__ int lanes_per_bucket(int nb) {
  int l = 1;
  while (l < 32 && 32 * l < nb) l <<= 1;
  return l;
}

// chunk_fn(mask, off) for every step, by every lane (the trip count is the same for
// all groups); bit b of mask is the visited position low + off + b.
template <class F>
__device__ __forceinline__ void for_each_chunk(const WalkArgs &w, int low, bool live, int sub, int lpb,
                                               F &&chunk_fn) {
  const int key = low & (w.W - 1);
  if (key > *w.fmax) live = false;  // reference clamp: nothing visited
  for (int c0 = 0; c0 < w.nb; c0 += 32 * lpb) {
    unsigned mask = 0;
    const int off = c0 + 32 * sub;
    if (live && off < w.nb) {
      int r = key + off;
      if (r >= w.W) r -= w.W;
      const int wi = r >> 5, wn = wi + 1 == (w.W >> 5) ? 0 : wi + 1;
      mask = __funnelshift_r(__ldg(&w.bm[wi]), __ldg(&w.bm[wn]), r & 31);
      if (w.nb - off < 32) mask &= (1u << (w.nb - off)) - 1u;
    }
    chunk_fn(mask, off);
  }
}

// exclusive scan over groups of lpb lanes
__device__ __forceinline__ unsigned group_excl_scan(unsigned v, int sub, int lpb, unsigned *total) {
  unsigned x = v;
  for (int o = 1; o < lpb; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o, lpb);
    if (sub >= o) x += y;
  }
  *total = __shfl_sync(0xffffffffu, x, lpb - 1, lpb);
  return x - v;
}

constexpr int STASH = 32;     // candidates recorded per heavy bucket by the count pass

// buckets per block of the mark and count passes
__host__ __device__ __forceinline__ int buckets_per_block(int nb) { return VT / lanes_per_bucket(nb); }
__host__ __device__ __forceinline__ int walk_blocks(int Bt, int nb) {
  return (Bt + buckets_per_block(nb) - 1) / buckets_per_block(nb);
}
// Lanes per bucket in the write pass.  One where buckets are many and have few
// candidates (n = 2^27, k = 16000: 4000 blocks of warps 15 us, 125 of threads 7 us); a
// warp where they are few, or where more than 24 visited positions a window (nres
// residues of W) can bring more candidates than slots, which are walked again.
__host__ __device__ __forceinline__ int write_lanes(int Bt, int nb, int nres, int W) {
  return Bt <= 8192 || (long long)nb * nres > 24LL * W ? 32 : 1;
}
__host__ __device__ __forceinline__ int write_blocks(int Bt, int lw) { return (Bt + VT / lw - 1) / (VT / lw); }

// Takes up to four visited positions of a lane's mask (low bits first).
__device__ __forceinline__ int take_four(unsigned &mask, unsigned first, unsigned a, unsigned nmask,
                                         unsigned (&loc)[4], unsigned (&bit)[4]) {
  int nq = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (mask) {
      bit[q] = (unsigned)__ffs(mask) - 1u;
      mask &= mask - 1;
      loc[q] = ((first + bit[q]) * a) & nmask;
      nq = q + 1;
    }
  }
  return nq;
}

// Votes of heavy bucket t (one group of lanes): returns the number of visited
// positions whose count reached the threshold, and records the bucket's first STASH
// of them, in window order, at slot[].
__device__ __forceinline__ unsigned count_walk(const WalkArgs &w, int t, int sub, int lpb, unsigned epoch,
                                               unsigned thresh, unsigned *vote, int *slot) {
  const unsigned nmask = (unsigned)w.n - 1u;
  const bool live = t < w.Bt;
  const int low = live ? window_low(w.J[t], w.n, w.nb) : 0;
  unsigned recorded = 0;  // this bucket's candidates so far (the same in its group)
  for_each_chunk(w, low, live, sub, lpb, [&](unsigned mask, int off) {
    const unsigned first = (unsigned)low + (unsigned)off;
    unsigned app = 0;  // bits of this lane's mask whose count reached the threshold
    while (mask) {
      unsigned loc[4], bit[4], cv[4];
      const int nq = take_four(mask, first, w.a, nmask, loc, bit);
      vote_update(w, epoch, vote, loc, nq, cv);
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q < nq && cv[q] == thresh) app |= 1u << bit[q];
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, app != 0u)) {
      unsigned ctot;
      unsigned o = recorded + group_excl_scan((unsigned)__popc(app), sub, lpb, &ctot);
      while (app) {
        const int b = __ffs(app) - 1;
        app &= app - 1;
        if (o < (unsigned)STASH) slot[o] = (int)(((first + (unsigned)b) * w.a) & nmask);
        o++;
      }
      recorded += ctot;
    }
  });
  return recorded;
}

// One block of the count pass: votes of the location loop, each bucket's candidate
// count and first STASH candidates, and the sum of the block's counts (csum[bid]).
__device__ __forceinline__ void vote_count_block(const WalkArgs &w, unsigned epoch, unsigned thresh,
                                                 unsigned *vote, int *cnt, int *csum, int *stash, int bid) {
  const int lpb = lanes_per_bucket(w.nb), sub = threadIdx.x & (lpb - 1);
  const int t = bid * (VT / lpb) + (int)threadIdx.x / lpb;
  const unsigned c = count_walk(w, t, sub, lpb, epoch, thresh, vote, stash + (size_t)t * STASH);
  __shared__ int s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  if (sub == 0 && t < w.Bt) {
    cnt[t] = (int)c;
    if (c) atomicAdd(&s_sum, (int)c);
  }
  __syncthreads();
  if (threadIdx.x == 0) csum[bid] = s_sum;
}

// One block of a location loop before the (loops_thresh - 1)-th, which cannot bring
// any count to the threshold: votes only.
__device__ __forceinline__ void vote_mark_block(const WalkArgs &w, unsigned epoch, unsigned *vote,
                                                int bid) {
  const int lpb = lanes_per_bucket(w.nb), sub = threadIdx.x & (lpb - 1);
  const int t = bid * (VT / lpb) + (int)threadIdx.x / lpb;
  const unsigned nmask = (unsigned)w.n - 1u;
  const bool live = t < w.Bt;
  const int low = live ? window_low(w.J[t], w.n, w.nb) : 0;
  for_each_chunk(w, low, live, sub, lpb, [&](unsigned mask, int off) {
    while (mask) {
      unsigned loc[4], bit[4], cv[4];
      const int nq = take_four(mask, (unsigned)low + (unsigned)off, w.a, nmask, loc, bit);
      vote_update(w, epoch, vote, loc, nq, cv);
    }
  });
}

// Heavy bucket t with more candidates than slots (a whole warp): walks the window
// and the vote table again and appends its candidates at cand[next ..].
__device__ __forceinline__ void write_walk(const WalkArgs &w, int t, unsigned epoch, unsigned thresh,
                                           const unsigned *vote, int *cand, int cap, long long next) {
  const int lane = threadIdx.x & 31;
  const unsigned nmask = (unsigned)w.n - 1u;
  const int low = window_low(w.J[t], w.n, w.nb);
  for_each_chunk(w, low, true, lane, 32, [&](unsigned mask, int off) {
    const unsigned first = (unsigned)low + (unsigned)off;
    unsigned app = 0;
    while (mask) {
      unsigned loc[4], bit[4];
      const int nq = take_four(mask, first, w.a, nmask, loc, bit);
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q < nq && vote_at_threshold(w, epoch, vote, loc[q], thresh)) app |= 1u << bit[q];
    }
    __syncwarp();
    unsigned ctot;
    long long o = next + group_excl_scan((unsigned)__popc(app), lane, 32, &ctot);
    while (app) {
      const int b = __ffs(app) - 1;
      app &= app - 1;
      if (o < cap) cand[o] = (int)(((first + (unsigned)b) * w.a) & nmask);
      o++;
    }
    next += ctot;
  });
}

// One block of the write pass of location loop l, lw lanes per bucket (1 or 32):
// appends the block's candidates at their canonical offsets, after those of the
// earlier buckets (the count pass's block sums); the last block stores the next
// loop's offset and the candidate count.
__device__ __forceinline__ void vote_write_block(const WalkArgs &w, int l, int lw, unsigned epoch, unsigned thresh,
                                                 const unsigned *vote, const int *cnt, const int *csum,
                                                 const int *stash, int *cand, int cap, RunCtl *ctl, int bid,
                                                 int nblk) {
  __shared__ unsigned ws[VT / 32];
  const int base = __ldcg(&ctl->base[l]);
  const int t0 = bid * (VT / lw), t = t0 + (int)threadIdx.x / lw, lane = threadIdx.x & 31;
  unsigned before = 0;
  // whole blocks of the count pass, four sums a load, then the buckets left
  const int bpb = buckets_per_block(w.nb), nsum = t0 / bpb, n4 = nsum / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < n4; i += VT) {
    const int4 v = __ldcg(reinterpret_cast<const int4 *>(csum) + i);
    before += (unsigned)(v.x + v.y + v.z + v.w);
  }
  for (int i = 4 * n4 + (int)threadIdx.x; i < nsum; i += VT) before += (unsigned)__ldcg(&csum[i]);
  for (int i = nsum * bpb + (int)threadIdx.x; i < t0; i += VT) before += (unsigned)__ldcg(&cnt[i]);
  unsigned c = t < w.Bt && (lw == 1 || lane == 0) ? (unsigned)__ldcg(&cnt[t]) : 0u;
  before = blk_sum(before, ws);
  unsigned tot;
  const unsigned pre = blk_excl_scan(c, ws, &tot);
  long long next = (long long)base + before + pre;
  if (lw == 1) {
    if (c && c <= (unsigned)STASH) {
      const int4 *slot = reinterpret_cast<const int4 *>(stash + (size_t)t * STASH);
      for (unsigned j = 0; j < c; j += 4) {
        const int4 v = __ldcg(slot + j / 4);
        const int vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (unsigned q = 0; q < 4; q++)
          if (j + q < c && next + j + q < cap) cand[next + j + q] = vs[q];
      }
    }
    unsigned big = __ballot_sync(0xffffffffu, c > (unsigned)STASH);
    while (big) {
      const int src = __ffs(big) - 1;
      big &= big - 1;
      write_walk(w, t - lane + src, epoch, thresh, vote, cand, cap, __shfl_sync(0xffffffffu, next, src));
    }
  } else {
    c = __shfl_sync(0xffffffffu, c, 0);
    next = __shfl_sync(0xffffffffu, next, 0);
    if (c > (unsigned)STASH)
      write_walk(w, t, epoch, thresh, vote, cand, cap, next);
    else if ((unsigned)lane < c && next + lane < cap)
      cand[next + lane] = __ldcg(&stash[(size_t)t * STASH + lane]);
  }
  if (bid == nblk - 1 && threadIdx.x == 0) {
    const long long nc = (long long)base + before + tot;
    const int count = (int)(nc > 0x7fffffffLL ? 0x7fffffffLL : nc);
    ctl->base[l + 1] = count;
    ctl->cand_count = count;
    if (nc > cap) ctl->overflow = 1;
  }
}

}  // namespace

}  // namespace gsfft
