// A5 + the RLFC sub-sampling of A4 in one ordered pass over the signal.
//
// The gather form (pf.cu) reads each tap's sample at a random address; at the
// n = 2^27 sizes every such read costs a whole DRAM burst (~64-96 bytes for
// an 8-byte sample).  When loops * w random reads cost more than reading x
// once, this kernel streams x through shared memory with TMA instead.
//
// View x as an (n/B) x B matrix, x[r*B + c].  For loop l the tap of position
// t = r*B + c is i = t*a_l mod n (t = i*ai_l mod n, innerLoop.cu:738,769):
//   i = B * ((q_l + r*alpha_l) mod nb) + b_l,    nb = n/B,
//   b_l = (c*a_l) mod B,  q_l = ((c*a_l) mod n) / B,  alpha_l = a_l mod nb.
// Every tap of column c therefore belongs to the one bucket b_l (c -> b_l is
// a bijection since a_l is odd), and tap j of that bucket sits in row
//   r_j = (j*beta_l + s_l) mod nb,  beta_l = alpha_l^-1 mod nb,  s_l = -q_l*beta_l,
// i.e. the column's hit rows are one per-loop set {j*beta_l mod nb} shifted by
// s_l.  The host sorts that set once per run; one thread per (column, loop)
// walks its rotated copy in ascending row order, so it touches only its own
// ~w/B hits while the CTA streams every row of its columns exactly
// once.  Sums run in ascending row (= signal position) order: fixed, no
// atomics.
//
// Tiles of 256 rows x 16 columns (FP32) arrive by cp.async.bulk.tensor.2d, issued
// by a producer warp, into a shared-memory ring guarded by full / empty mbarriers
// whose waits are bounded (a timeout sets an error flag instead of hanging).  Each
// consumer warp copies its walks' taps into shared memory with cp.async at the
// start of an item; where they do not fit beside two tiles, each hit's tap is
// loaded from a bucket-major table in L2, one hit ahead.
//
// RLFC loop r samples positions off_r + m*(n/W) (restLocFreqCoeffKernel,
// innerLoop.cu:693-703); (n/W) divides B, so those are whole columns and the
// CTA copies them from the tile to y_r[t / (n/W)].  A tile holds few columns of a
// loop, so y written in order is written in parts of 32-byte sectors, which cost
// 104 us of the n = 2^27, k = 16000 step (250 at k = 43000): where the FFT can
// read it so, y is in blocks of four rows instead, whole sectors.
//
// What bounds it: 2^27 FP32 samples are 1.07 GB, 150 us with no consumer.  Whole
// steps went 438 -> 400 us (k = 16000), 1013 -> 896 (k = 43000, 8 columns of y a
// tile) and 539 -> 466 (24 signals of 2^18 .. 2^24) from 64 x 64 tiles; what is
// left above the stream is the RLFC copies (about 25 us at k = 16000) and the
// scattered stores of the bins (16).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "stages.cuh"

namespace gsfft {

namespace {

constexpr int ST = 128;      // B must be a multiple of this
// Columns of a tile: 128 bytes of a row in FP32.  Of 2^27 samples in rows of 2^17,
// 16 columns x 256 rows stream at 7.0 TB/s with no consumer (64 x 64: 7.2, 8 x 256:
// 5.7), and a walk meets its hits in a quarter of the tiles of 64 rows: the warps'
// instructions a tile, not the memory, were the limit there.
constexpr int LOGCW = 4, CW = 1 << LOGCW;
constexpr int MINNS = 2, MAXNS = 8;  // tiles of the ring
constexpr int MAXT = 32;     // full tiles of taps per bucket (w / B) supported
constexpr int MAXL = 16;     // loops supported
// Two CTAs an SM, so that one loads an item's taps while the other walks.  Whole
// step at n = 2^27, k = 16000 / 43000, RLFC copies off: 32 KiB tiles 401 / 836 us,
// 16 KiB 428 / 952; one CTA with 32 KiB tiles 508 / 1036.
constexpr int CTAS_PER_SM = 2;
constexpr int PF_TILE = 32 * 1024;  // bytes of a tile, halved where the taps leave no room for two
constexpr int PF_SMEM = (228 / CTAS_PER_SM - 1) * 1024 - 5 * 1024;  // dynamic bytes a CTA
constexpr int MAXRW = 4;     // RLFC warps
constexpr int MAXTH = 32 * (CW * MAXL / 32 + 1 + MAXRW);
constexpr unsigned NONE = 0x7fffffffu;

// taps per bucket in the bucket-major table: the w/B full-tile taps plus the
// partial one, rounded up to even so that every bucket's row is a multiple of
// 16 bytes (bulk copies)
__host__ __device__ inline int taps_per_bucket(int tiles) { return (tiles + 2) & ~1; }

struct HitTab {
  unsigned s[MAXL][MAXT];  // (row offset << 8) | j, sorted by row offset
  unsigned beta[MAXL];
  unsigned xrow[MAXL];     // (tiles * beta) mod nb: row offset of the partial tap
};

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ unsigned long long policy_evict_first() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long policy_evict_last() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ void tma_load_tile(void *dst, const CUtensorMap *tm, int x0, int y0,
                                              unsigned long long *bar, unsigned bytes,
                                              unsigned long long pol) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(tm)), "r"(x0), "r"(y0), "r"(smem_u32(bar)), "l"(pol)
      : "memory");
}

// read-only tap load that asks L2 to keep the line
__device__ __forceinline__ float2 ld_tap(const float2 *p, unsigned long long pol) {
  float2 v;
  asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;"
               : "=f"(v.x), "=f"(v.y)
               : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double2 ld_tap(const double2 *p, unsigned long long pol) {
  double2 v;
  asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
               : "=d"(v.x), "=d"(v.y)
               : "l"(p), "l"(pol));
  return v;
}

// Bounded wait on an mbarrier phase; false after ~0.5 s without completion.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity) {
  return mbar_wait_bounded(smem_u32(bar), parity);
}

// Persistent, warp-specialised.  A work item is (block of CW columns, row
// group); CTA b takes items b, b + grid, ...  Warp roles:
//  * the first NCW warps: consumers.  Thread (l, col) walks loop l of column
//    col; its taps come from its shared-memory slot (staged form) or from the
//    bucket-major tap table one hit ahead, so the L2 reads overlap the stream.
//  * the next warp: producer.  One lane streams every tile of the CTA's
//    items, in order, into a ring of NS tiles (full[s]: tile landed,
//    tx-counted; empty[s]: every releasing warp is done with it).
//  * the last warps (RLFC loops only): copy the RLFC sub-samples out of each
//    tile.
// No block-wide barrier inside the stream.
// swz: 14 where the tile is stored with TMA's 128-byte swizzle (column c of row r
// at c ^ 2 (r mod 8)), else 0.  The RLFC warps read down a column, 16 rows in one
// bank without it: n = 2^27 step 414 -> 402 us.
template <typename T, bool STG>
__global__ void __launch_bounds__(MAXTH, CTAS_PER_SM)
pf_tma_kernel(const __grid_constant__ CUtensorMap tmap, const typename Cx<T>::V *__restrict__ filt,
              int logn, int logB, int w, int rt, int ord, int NS, int tiles, int rows_per_group,
              int groups, int L, Draws d, HitTab ht, typename Cx<T>::V *__restrict__ bins, int swz, int nrlfc,
              int logsig, int logyr, typename Cx<T>::V *__restrict__ y, int W, int *err) {
  pdl_enter();
  typedef typename Cx<T>::V V;
  const int NCT = CW * L;  // walks of an item
  const int NCW = (NCT + 31) / 32;
  const int nrw = (int)blockDim.x / 32 - NCW - 1;  // RLFC warps
  extern __shared__ __align__(1024) unsigned char dsm[];
  // each loop's sorted list twice in a row, so a rotated walk needs no wrap
  __shared__ unsigned S2[MAXL][2 * MAXT];
  __shared__ unsigned s_a[MAXL], s_beta[MAXL], s_xrow[MAXL];
  __shared__ __align__(8) unsigned long long full[MAXNS], empty[MAXNS];
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int B = 1 << logB;
  const int lognb = logn - logB;
  const int nb = 1 << lognb;
  const unsigned nbm = (unsigned)nb - 1u;
  const unsigned nmask = (1u << logn) - 1u;
  const int TT = taps_per_bucket(tiles);  // row length of the bucket-major table
  const unsigned stage_bytes = (unsigned)(rt * CW * sizeof(V));
  const int ntile = rows_per_group / rt;
  const int ncb = B / CW;
  const int items = ncb * groups;
  const int xmul = (int)(sizeof(V) / 8);  // tensor elements are 8-byte words
  V *tile0 = reinterpret_cast<V *>(dsm);

  for (int e = tid; e < L * 2 * MAXT; e += blockDim.x) {
    const int l = e / (2 * MAXT), m = e % (2 * MAXT);
    S2[l][m] = m < tiles ? ht.s[l][m] : (m < 2 * tiles ? ht.s[l][m - tiles] : 0u);
  }
  if (tid < L) {
    s_a[tid] = (unsigned)d.a[tid];
    s_beta[tid] = ht.beta[tid];
    s_xrow[tid] = ht.xrow[tid];
  }
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < NS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], (unsigned)(NCW + nrw));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  int st = 0;       // stage of the current tile ...
  unsigned ph = 0;  // ... and its phase
  auto next_tile = [&]() {
    if (++st == NS) {
      st = 0;
      ph ^= 1u;
    }
  };

  if (warp > NCW) {
    // ---------------- RLFC warps: loop r samples positions off_r + m*(n/W)
    // (restLocFreqCoeffKernel, innerLoop.cu:693-703); n/W divides B, so those
    // are whole columns, copied from the tile to y_r[t / (n/W)]
    const unsigned smask = (1u << logsig) - 1u;
    const int lognc = logsig >= LOGCW ? 0 : LOGCW - logsig;  // log2 of a loop's columns in a block
    // A loop's samples in a tile, in order: row within its block, column, block of
    // rows.  A thread's next sample is whole blocks of rows on (32 nrw threads are a
    // multiple of a block's samples), in the same column.
    const int e0 = tid - 32 * (NCW + 1);
    const int ci = (e0 >> logyr) & ((1 << lognc) - 1);
    const int row0 = ((e0 >> (logyr + lognc)) << logyr) + (e0 & ((1 << logyr) - 1));
    const int rstep = (32 * nrw >> (logyr + lognc)) << logyr;
    const size_t ystep = (size_t)rstep << (logB - logsig);
    constexpr int U = 4;  // copies in flight per thread
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      const int cb = it % ncb, g = it / ncb;
      const unsigned c0 = (unsigned)(cb * CW);
      for (int t = 0; t < ntile; t++, next_tile()) {
        const V *tl = tile0 + (size_t)st * rt * CW;
        if (!__all_sync(0xffffffffu, mbar_wait(&full[st], ph))) {
          abort_flag = 1;
          atomicExch(err, 1);
          return;
        }
        const unsigned r0 = (unsigned)(g * rows_per_group + t * rt);
        for (int rr = 0; rr < nrlfc; rr++) {
          const unsigned off = (unsigned)d.offs[rr];
          const unsigned first = (off - c0) & smask;  // first matching column
          if (first >= (unsigned)CW) continue;
          const unsigned ci0 = (c0 + first - off) >> logsig;
          const unsigned scol = first + ((unsigned)ci << logsig);
          V *yp = y + (size_t)rr * W + (e0 & ((1 << logyr) - 1)) +
                  (((size_t)((r0 + row0) >> logyr) << (logB - logsig)) + ci0 + ci << logyr);
          for (int row = row0; row < rt; row += U * rstep) {
            V v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
              const int ru = row + u * rstep;
              if (ru < rt) v[u] = tl[(ru << LOGCW) + (scol ^ ((ru << 1) & swz))];
            }
#pragma unroll
            for (int u = 0; u < U; u++, yp += ystep)
              if (row + u * rstep < rt) *yp = v[u];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
      }
    }
    return;
  }
  if (warp == NCW) {
    // ---------------- producer
    if (lane == 0) {
      const unsigned long long pol = policy_evict_first();
      int k = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        const int cb = it % ncb, g = it / ncb;
        for (int t = 0; t < ntile; t++, k++, next_tile()) {
          if (!mbar_wait(&empty[st], ph ^ 1u) || abort_flag) {
            abort_flag = 1;
            ok = false;
            break;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          tma_load_tile(reinterpret_cast<char *>(tile0) + (size_t)st * stage_bytes, &tmap,
                        cb * CW * xmul, g * rows_per_group + t * rt, &full[st], stage_bytes, pol);
        }
      }
      // stay until the last load of every stage has landed (bounded)
      for (int j = k - NS < 0 ? 0 : k - NS; j < k; j++)
        if (!mbar_wait(&full[j % NS], (unsigned)((j / NS) & 1))) {
          atomicExch(err, 1);
          break;
        }
    }
    return;
  }

  // ---------------- consumers
  const bool act = tid < NCT;  // the last warp of an odd loop count is half full
  const int col = tid & (CW - 1), l = act ? tid >> LOGCW : 0;
  const int residue = w & (B - 1);
  const unsigned a = s_a[l], beta = s_beta[l], xrow = s_xrow[l];
  const unsigned *S = S2[l];
  const unsigned long long keep = policy_evict_last();
  // staged form: this thread's slot of TT taps after the tile ring
  V *const tslot = reinterpret_cast<V *>(dsm + (size_t)NS * stage_bytes) + (size_t)tid * TT;
  const int nch = (int)(TT * sizeof(V) / 16);  // 16-byte pieces of a slot
  const int dq = 32 / nch, dr = 32 - dq * nch;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int cb = it % ncb, g = it / ncb;
    const int c0 = cb * CW;
    const unsigned c = (unsigned)(c0 + col);
    const int rbeg = g * rows_per_group;
    // Walk state.  Rotated position k of the column's hit list is
    // doubled-list entry m = mw + k; its row is (v + s) mod nb.
    const unsigned prod = c * a;
    const int bl = (int)(prod & (unsigned)(B - 1));
    const unsigned q = (prod & nmask) >> logB;
    const unsigned sl = (0u - q * beta) & nbm;
    const V *fcol = filt + (size_t)bl * TT;  // the bucket's taps, contiguous
    if constexpr (STG) {
      // the warp copies its walks' taps together, 16 bytes a lane, so that a
      // load covers whole rows; every lane is past its last read of the old ones
      __syncwarp();
      int row = (warp << 5) + lane / nch, part = lane - lane / nch * nch;
      const int end = min(NCT, (warp + 1) << 5);
      unsigned dst = smem_u32(tslot - (size_t)lane * TT) + (unsigned)lane * 16u;
      while (row < end) {
        const unsigned br = ((unsigned)(c0 + (row & (CW - 1))) * s_a[row >> LOGCW]) & (unsigned)(B - 1);
        const char *src = reinterpret_cast<const char *>(filt + (size_t)br * TT) + part * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        dst += 512u;
        row += dq;
        part += dr;
        if (part >= nch) {
          part -= nch;
          row++;
        }
      }
    }
    // mw: first sorted entry with v >= nb - s (binary search)
    int lo = 0, hi = tiles;
    const unsigned lim = (unsigned)nb - sl;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((S[mid] >> 8) < lim) lo = mid + 1;
      else hi = mid;
    }
    const int mw = lo;
    // first rotated position with row >= rbeg (binary search)
    lo = 0;
    hi = rbeg ? tiles : 0;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((((S[mw + mid] >> 8) + sl) & nbm) < (unsigned)rbeg) lo = mid + 1;
      else hi = mid;
    }
    int mc = mw + lo;
    const int me = act ? mw + tiles : 0;
    // the next hit's row, its tap and the entry after it, loaded a hit ahead, so
    // that a hit waits for its sample alone (S has entries past the last, and
    // the tap of one is a valid one)
    auto tap = [&](unsigned j) {
      if constexpr (STG) return tslot[j];
      else return ld_tap(fcol + j, keep);
    };
    unsigned nm = NONE, er = NONE, ent = S[mc];
    if (mc < me) nm = ((ent >> 8) + sl) & nbm;
    if (act && bl < residue) {
      er = (xrow + sl) & nbm;
      if (er < (unsigned)rbeg) er = NONE;
    }
    if constexpr (STG) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
    }
    V fe = mk((T)0, (T)0), ftap = fe;
    if (er != NONE) fe = tap((unsigned)tiles);
    if (act) ftap = tap(ent & 255u);
    ent = S[mc + 1];
    T re = 0, im = 0;

    for (int t = 0; t < ntile; t++, next_tile()) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full[st], ph))) {
        abort_flag = 1;
        atomicExch(err, 1);
        return;
      }
      const unsigned r0 = (unsigned)(rbeg + t * rt), r1 = r0 + (unsigned)rt;
      const V *tl = tile0 + (size_t)st * rt * CW;
      auto add = [&](unsigned row, V f) {
        const V xv = tl[((row - r0) << LOGCW) + ((unsigned)col ^ ((row << 1) & (unsigned)swz))];
        re = fma(xv.x, f.x, re);
        re = fma(-xv.y, f.y, re);
        im = fma(xv.x, f.y, im);
        im = fma(xv.y, f.x, im);
      };
      // full-tile taps in ascending row order, the partial tap after those of
      // its block of ord rows (the order of the sums does not depend on rt)
      while (nm < r1) {
        if ((er | (unsigned)(ord - 1)) < nm) {
          add(er, fe);
          er = NONE;
        }
        add(nm, ftap);
        const int m = ++mc;
        nm = m < me ? ((ent >> 8) + sl) & nbm : NONE;
        ftap = tap(ent & 255u);
        ent = S[m + 1];
      }
      if (er < r1) {
        add(er, fe);
        er = NONE;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[st]);
    }
    // partial sums of this row group: bins[group][l][b]
    if (act) bins[((size_t)g * L + l) * B + bl] = mk(re, im);
  }
}

// FP64 form: the same column-ordered walk, with each hit's sample gathered from
// global memory instead of streamed.
//
// What bounds it: DRAM lines.  A 16-byte sample costs its 128-byte line.  In
// bucket order (pf.cu) the loops * w gathers are random and nearly every one
// fetches a line of its own: 2.45 GB at n = 2^27, k = 16000, 434 us, and the RLFC
// rows, gathered by the W-point FFT's first pass, another 1.07 GB.  Here a CTA
// owns 32 columns (four lines a row); its warps walk the loops of those columns in
// ascending row order side by side (a barrier every PC_U hits keeps them together:
// 482 -> 448 us), and its threads copy the RLFC columns at the same pace, so
// samples that share a line are read close together, and stored by pairs of rows
// where the W-point FFT reads them so (whole sectors: step 860 -> 843 us).  At n =
// 2^27 the kernel took 440 us with the RLFC rows in order, and the W-point FFT fell
// from 392 to 297 us; at
// n = 2^14 .. 2^26 it is faster by itself (27 -> 11, 33 -> 17 at 2^20, 175 -> 107
// at 2^25, 289 -> 224 us at 2^26), so every FP64 plan whose sizes allow it takes it.
// Streaming the whole signal through shared memory (pf_tma_kernel) took 489 us at
// n = 2^27: the divergent hit loop wastes FP64 issue slots (1.73 operations a clock
// and SM); here every lane has a hit at every step.
//
// quirk: the partial tap as permFilterTillKernel indexes it (innerLoop.cu:745-754),
// id = bucket * tiles + B, from the bucket-order taps qfilt.
constexpr int PC_U = 3;  // hits in flight per thread
__global__ void __launch_bounds__(512, 2)
pf_cols_kernel(const double2 *__restrict__ x, const double2 *__restrict__ filt,
               const double2 *__restrict__ qfilt, int logn, int logB, int w, int tiles, int L, Draws d,
               HitTab ht, double2 *__restrict__ bins, int nrlfc, int logsig, int logyr,
               double2 *__restrict__ y, int W, int quirk) {
  pdl_enter();
  __shared__ unsigned S2[MAXL][2 * MAXT];
  const int tid = threadIdx.x, lane = tid & 31, l = tid >> 5;
  const int B = 1 << logB, lognb = logn - logB, nb = 1 << lognb;
  const unsigned nbm = (unsigned)nb - 1u, nmask = (1u << logn) - 1u;
  const int TT = taps_per_bucket(tiles);
  for (int e = lane; e < 2 * MAXT; e += 32) S2[l][e] = e < tiles ? ht.s[l][e] : (e < 2 * tiles ? ht.s[l][e - tiles] : 0u);
  __syncwarp();
  const unsigned *S = S2[l];
  const unsigned c = blockIdx.x * 32u + (unsigned)lane;
  const unsigned a = (unsigned)d.a[l], beta = ht.beta[l];
  const unsigned prod = c * a;
  const int bl = (int)(prod & (unsigned)(B - 1));
  const unsigned sl = (0u - ((prod & nmask) >> logB) * beta) & nbm;
  const double2 *fcol = filt + (size_t)bl * TT;
  const double2 *xcol = x + c;
  const unsigned long long keep = policy_evict_last();
  // first sorted entry whose row wraps past nb (pf_tma_kernel)
  int lo = 0, hi = tiles;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((S[mid] >> 8) < (unsigned)nb - sl) lo = mid + 1;
    else hi = mid;
  }
  // RLFC samples of this block: rows x (loops r) x (columns c = off_r mod n/W)
  const int logcpr = logsig >= 5 ? 0 : 5 - logsig;  // log2 of a loop's columns in the block
  const int steps = max((tiles + PC_U - 1) / PC_U, 1);
  const int total = (nb * nrlfc) << logcpr;
  const int per = ((total + steps - 1) / steps + 1) & ~1;
  const int nthr = 32 * L;
  double re = 0.0, im = 0.0;
  auto accumulate = [&](double2 xv, double2 f) {
    re = fma(xv.x, f.x, re);
    re = fma(-xv.y, f.y, re);
    im = fma(xv.x, f.y, im);
    im = fma(xv.y, f.x, im);
  };
  int k = 0;
  for (int st = 0; st < steps; st++, k += PC_U) {
    __syncthreads();  // keeps the warps on the same rows
    double2 xv[PC_U], f[PC_U];
#pragma unroll
    for (int u = 0; u < PC_U; u++) {
      if (k + u < tiles) {
        const int m = lo + k + u;
        const unsigned ent = S[m];
        const unsigned row = (ent >> 8) + sl - (m < tiles ? (unsigned)nb : 0u);
        xv[u] = __ldg(xcol + ((size_t)row << logB));
        f[u] = ld_tap(fcol + (ent & 255u), keep);
      }
    }
    const int e1 = min((st + 1) * per, total);
    for (int e = st * per + tid; e < e1; e += nthr) {
      // logyr = 1: two rows of a column side by side, whole 32-byte sectors of y
      const int ci = (e >> logyr) & ((1 << logcpr) - 1), q = e >> (logcpr + logyr);
      const int rr = q % nrlfc, row = (q / nrlfc << logyr) + (e & logyr);
      const unsigned off = (unsigned)d.offs[rr];
      const unsigned cc = ((off - blockIdx.x * 32u) & ((1u << logsig) - 1u)) + ((unsigned)ci << logsig);
      if (cc < 32u) {
        const unsigned t = ((unsigned)row << logB) + blockIdx.x * 32u + cc;
        const unsigned col = (blockIdx.x * 32u + cc - off) >> logsig;
        y[(size_t)rr * W + (((((unsigned)row >> logyr) << (logB - logsig)) + col) << logyr) + (e & logyr)] = __ldg(x + t);
      }
    }
#pragma unroll
    for (int u = 0; u < PC_U; u++)
      if (k + u < tiles) accumulate(xv[u], f[u]);
  }
  if (bl < (w & (B - 1))) {  // the partial tap
    if (quirk && tiles > 0) {
      const unsigned id = (unsigned)bl * (unsigned)tiles + (unsigned)B;
      accumulate(__ldg(x + ((id * (unsigned)d.ai[l]) & nmask)), __ldg(qfilt + id));
    } else {
      accumulate(__ldg(xcol + ((size_t)((ht.xrow[l] + sl) & nbm) << logB)), ld_tap(fcol + tiles, keep));
    }
  }
  bins[(size_t)l * B + bl] = make_double2(re, im);
}

// Bucket-major copy of the taps: tb[b * TT + j] = filt[j * B + b] (0 past w).
template <typename V>
__global__ void bucket_major_kernel(const V *__restrict__ filt, int w, int B, int TT, V *tb) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)B * TT) return;
  const int b = (int)(i / TT), j = (int)(i % TT);
  const long long src = (long long)j * B + b;
  V v = filt[src < w ? src : 0];
  if (src >= w) v.x = v.y = 0;
  tb[i] = v;
}

template <typename V>
__global__ void sum_partials_kernel(const V *__restrict__ part, int groups, long long count, V *out) {
  pdl_enter();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= count) return;
  V v = part[i];
  for (int g = 1; g < groups; g++) v = cadd(v, part[(long long)g * count + i]);
  out[i] = v;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  // the driver's entry point is the same for every context; looked up once,
  // thread-safely (function-local static initialisation)
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return nullptr;
  }();
  return fn;
}

int ilog2(long long v) {
  int l = 0;
  while ((1LL << l) < v) l++;
  return l;
}

unsigned inv_odd(unsigned a) {  // a^-1 mod 2^32 for odd a (Newton)
  unsigned x = a;
  for (int i = 0; i < 5; i++) x *= 2u - a * x;
  return x;
}

// Tile of a pass: its rows, the ring's depth, and whether the taps are staged in
// shared memory (always but for the longest windows of the most loops).
struct PfTile {
  int rt, ns, swz;
  bool staged;
};
inline PfTile pf_tile(int rows_per_group, int es, int loops, int tiles, int ord) {
  PfTile t;
  const int slots = CW * loops * taps_per_bucket(tiles) * es;
  const int rt = std::min(rows_per_group, PF_TILE / (CW * es));
  t.rt = rt;
  if (PF_SMEM - slots < MINNS * rt * CW * es && rt / 2 >= ord) t.rt = rt / 2;
  t.staged = PF_SMEM - slots >= MINNS * t.rt * CW * es;
  if (!t.staged) t.rt = rt;
  t.ns = std::min(MAXNS, (PF_SMEM - (t.staged ? slots : 0)) / (t.rt * CW * es));
  // the swizzle spans 128-byte rows, in groups of eight from the tile's start
  t.swz = CW * es == 128 && t.rt % 8 == 0 ? 14 : 0;
  return t;
}

template <typename T, bool STG>
int launch_T(const CUtensorMap &tm, const void *filt, int logn, int logB, int w, const PfTile &pt, int ord,
             int tiles, int groups, int loops, const Draws &d, const HitTab &ht, void *bins, int nrlfc,
             int logsig, int logyr, void *y, int W, int *err, cudaStream_t st) {
  typedef typename Cx<T>::V V;
  const int B = 1 << logB;
  const int smem = (int)sizeof(V) * (pt.ns * pt.rt * CW + (STG ? CW * loops * taps_per_bucket(tiles) : 0));
  // RLFC warps: a power of two, one for 256 samples of a tile (one for 512 held
  // the ring back: 424 against 402 us), and whole blocks of rows a step
  int rw = 0;
  if (nrlfc) {
    const int lognc = std::max(0, LOGCW - logsig), per_tile = std::max(pt.rt * nrlfc * CW >> logsig, 1);
    rw = 1;
    while (rw < MAXRW && (rw * 256 < per_tile || 32 * rw < 1 << (logyr + lognc))) rw *= 2;
  }
  const int threads = 32 * ((CW * loops + 31) / 32 + 1 + rw);
  static PerContext<int> attr;  // the kernel's dynamic shared memory limit, per context
  GS_CHECK(attr.ensure_at_least(smem, [](int v) {
    if (cudaFuncSetAttribute(pf_tma_kernel<T, STG>, cudaFuncAttributeMaxDynamicSharedMemorySize, v) ==
        cudaSuccess)
      return (int)GSFFT_OK;
    set_last_error("pf_tma_kernel: %d bytes of shared memory refused: %s", v,
                   cudaGetErrorString(cudaGetLastError()));
    return (int)GSFFT_ERR_CUDA;
  }));
  int dev = 0, sms = 0, per_sm = 0;
  GS_CUDA(cudaGetDevice(&dev));
  GS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pf_tma_kernel<T, STG>, threads, smem));
  const int items = (B / CW) * groups;
  const int grid = std::max(1, std::min(items, std::max(per_sm, 1) * sms));
  const int rows_per_group = (1 << (logn - logB)) / groups;
  GS_CUDA(launch_pdl(pf_tma_kernel<T, STG>, dim3(grid), dim3(threads), smem, st, tm, (const V *)filt, logn,
                     logB, w, pt.rt, ord, pt.ns, tiles, rows_per_group, groups, loops, d, ht, (V *)bins, pt.swz, nrlfc,
                     logsig, logyr, (V *)y, W, err));
  return GSFFT_OK;
}

}  // namespace

int stream_taps_count(int w, int B) { return B * taps_per_bucket(w / B); }

int launch_stream_taps(int precision, const void *filt, int w, int B, void *taps_bm,
                       cudaStream_t st) {
  const int TT = taps_per_bucket(w / B);
  const long long cnt = (long long)B * TT;
  const unsigned grid = (unsigned)((cnt + 255) / 256);
  if (precision == GSFFT_FP64)
    bucket_major_kernel<double2><<<grid, 256, 0, st>>>((const double2 *)filt, w, B, TT, (double2 *)taps_bm);
  else
    bucket_major_kernel<float2><<<grid, 256, 0, st>>>((const float2 *)filt, w, B, TT, (float2 *)taps_bm);
  GS_LAUNCHED();
  return GSFFT_OK;
}

int launch_sum_partials(int precision, const void *part, int groups, long long count, void *out,
                        cudaStream_t st) {
  const unsigned grid = (unsigned)((count + 255) / 256);
  if (precision == GSFFT_FP64)
    GS_CUDA(launch_pdl(sum_partials_kernel<double2>, dim3(grid), dim3(256), 0, st,
                       (const double2 *)part, groups, count, (double2 *)out));
  else
    GS_CUDA(launch_pdl(sum_partials_kernel<float2>, dim3(grid), dim3(256), 0, st,
                       (const float2 *)part, groups, count, (float2 *)out));
  GS_LAUNCHED();
  return GSFFT_OK;
}

bool stream_pf_supported(int n, int B, int loops, int W, int RLFC_loops) {
  if (loops < 2 || loops > MAXL || B < ST || (B % ST) != 0 || n / B < 2) return false;
  if (RLFC_loops > MAX_RLFC_LOOPS || (W > 0 && n / W > B)) return false;
  if (n / B > (1 << 23)) return false;  // row offsets must fit 24 bits
  return encode_fn() != nullptr;
}

// Blocks of rows after which a column's partial tap is added, whatever the tiles are.
static int stream_rows_per_tile(int n, int B, int precision) {
  return std::min(n / B, precision == GSFFT_FP64 ? 32 : 64);
}

int stream_pf_groups(int n, int B, int w, int loops, int precision) {
  const int nb = n / B;
  const int rt = stream_rows_per_tile(n, B, precision);
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // The number of groups fixes the order of a bin's sums and so its last FP32 bit:
  // it is part of what a plan returns, and not derived from the kernel's tiles (16
  // columns, two CTAs an SM).  It doubles until there are 6 or 12 items of 64 columns (32
  // above 15 loops) per SM: 6 where an item's FP32 taps and four tiles of 32 KiB (three
  // above 9 loops) fit 218 KiB, as a kernel of one CTA an SM had them.
  const int cw = 64 * loops + 64 <= 1024 ? 64 : 32;
  const int slots = 8 * cw * loops * taps_per_bucket(w / B), tile = 8 * rt * cw;
  const bool few = precision != GSFFT_FP64 && cw == 64 &&
                   (loops <= 9 ? 4 : 3) * tile + slots <= 218 * 1024;
  const long long want = (few ? 6LL : 12LL) * sms;
  int groups = 1;
  while ((long long)(B / cw) * groups < want && nb / (groups * 2) >= 4 * rt) groups *= 2;
  return groups;
}

bool stream_pf_groups_valid(int n, int B, int groups, int precision) {
  if (groups < 1 || (groups & (groups - 1))) return false;
  if (groups == 1) return true;
  const int nb = n / B;
  return nb / groups >= 4 * stream_rows_per_tile(n, B, precision) && nb % groups == 0;
}

// sorted hit rows of each loop: j * beta mod nb for j < tiles
static void hit_table(int n, int B, int tiles, int loops, const Draws &d, HitTab &ht) {
  const unsigned nbm = (unsigned)(n / B) - 1u;
  memset(&ht, 0, sizeof(ht));
  std::pair<unsigned, unsigned> v[MAXT];
  for (int l = 0; l < loops; l++) {
    const unsigned alpha = (unsigned)d.a[l] & nbm;
    const unsigned beta = inv_odd(alpha) & nbm;
    ht.beta[l] = beta;
    ht.xrow[l] = ((unsigned)tiles * beta) & nbm;
    for (int j = 0; j < tiles; j++) v[j] = {((unsigned)j * beta) & nbm, (unsigned)j};
    std::sort(v, v + tiles);
    for (int j = 0; j < tiles; j++) ht.s[l][j] = (v[j].first << 8) | v[j].second;
  }
}

int launch_perm_filter_cols(const void *x, int n, const void *filt, const void *qfilt, int w, int B, int loops,
                            const Draws &d, void *bins, int nrlfc, void *y, int W, bool quirk, cudaStream_t st, int logyr) {
  if (!stream_pf_supported(n, B, loops, W, nrlfc) || w / B >= MAXT) return GSFFT_ERR_UNSUPPORTED;
  HitTab ht;
  hit_table(n, B, w / B, loops, d, ht);
  GS_CUDA(launch_pdl(pf_cols_kernel, dim3(B / 32), dim3(32 * loops), 0, st, (const double2 *)x,
                     (const double2 *)filt, (const double2 *)qfilt, ilog2(n), ilog2(B), w, w / B, loops, d, ht,
                     (double2 *)bins, nrlfc, ilog2(n / W), logyr, (double2 *)y, W, quirk ? 1 : 0));
  GS_LAUNCHED();
  return GSFFT_OK;
}

int launch_perm_filter_stream(int precision, const void *x, int n, const void *filt, int w, int B,
                              int loops, const Draws &d, void *bins, int nrlfc, void *y, int W,
                              int *err, cudaStream_t st, int groups_req, int logyr) {
  if (!stream_pf_supported(n, B, loops, W, nrlfc)) return GSFFT_ERR_UNSUPPORTED;
  const int tiles = w / B;
  if (tiles >= MAXT || tiles > 255) return GSFFT_ERR_UNSUPPORTED;
  const int logn = ilog2(n), logB = ilog2(B), logsig = ilog2(n / W);
  const int nb = n / B;
  HitTab ht;
  hit_table(n, B, tiles, loops, d, ht);
  // x as a 2-D tensor of 8-byte words: nb rows of B (FP32) or 2B (FP64) words
  const bool dbl = precision == GSFFT_FP64;
  const int es = dbl ? 16 : 8;
  const int ord = stream_rows_per_tile(n, B, precision);
  int groups = stream_pf_groups(n, B, w, loops, precision);
  if (groups_req > 0) {
    if (!stream_pf_groups_valid(n, B, groups_req, precision)) return GSFFT_ERR_PARAM;
    groups = groups_req;
  }
  const PfTile pt = pf_tile(nb / groups, es, loops, tiles, ord);
  CUtensorMap tm;
  const cuuint64_t gdim[2] = {(cuuint64_t)B * (es / 8), (cuuint64_t)nb};
  const cuuint64_t gstride[1] = {(cuuint64_t)B * es};
  const cuuint32_t box[2] = {(cuuint32_t)(CW * (es / 8)), (cuuint32_t)pt.rt};
  const cuuint32_t estr[2] = {1, 1};
  // 128-byte L2 fetches: with 256 the neighbour's half was fetched twice (1.55 GB
  // read for 1.07, the first-read data being evicted first)
  CUresult cr = encode_fn()(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void *>(x), gdim,
                            gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            pt.swz ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return GSFFT_ERR_CUDA;
  }
  auto go = [&](auto launch) {
    return launch(tm, filt, logn, logB, w, pt, ord, tiles, groups, loops, d, ht, bins, nrlfc, logsig, logyr, y,
                  W, err, st);
  };
  const int s = dbl ? (pt.staged ? go(launch_T<double, true>) : go(launch_T<double, false>))
                    : (pt.staged ? go(launch_T<float, true>) : go(launch_T<float, false>));
  if (s != GSFFT_OK) return s;
  GS_LAUNCHED();
  return GSFFT_OK;
}

}  // namespace gsfft
