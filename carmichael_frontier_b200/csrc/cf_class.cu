// cf_class.cu -- class join: the exchange join of one modulus split by residue class, with the
// table of each class in shared memory.
//
// A fused probe (cf_fused.cu) reads one random 32-byte L2 sector per record and spends four warp
// instructions on it; both are at their limits.  Here the join is cut into the phi(d) unit classes
// modulo a small divisor d of the odd part m of M.  Records of different classes never match, and
// because the class is multiplicative, the records of ONE class can be enumerated directly: a
// record is a prefix (A-subset) times a suffix (b-subset), both grouped by class, and the records
// of class c are, for every suffix class e, the pairs (prefix of class c/e) x (suffix of class e)
// whose last prefix index is below the first suffix index.  So a class's build records (about
// 3e4) fit a Bloom filter in shared memory (192 KB, two bits in one 32-bit word per record) and
// its probe records are tested there at shared-memory speed.
//
// The filter hashes the residue modulo a second divisor m' < 2^32 of m, coprime to d, in its
// scaled form V = floor(2^32 * frac(x / m')): with w = floor(2^64 * prefix / m') kept per prefix,
// a record costs two integer multiply-adds,
//     V = w_hi * s + mulhi(w_lo, s)   (mod 2^32),   s = suffix residue,
// which is floor(2^32 * frac) or one less (w is short by less than 1, so V by less than
// s / 2^32 < 1).  Records are therefore equal mod m' only if their V differ by at most one, and
// the build side sets the bits of V - 1, V and V + 1, so no match is lost.
//
//   k_cj_count    every prefix and suffix of both sides: class, residue mod m', place in its bin
//   k_cj_rows / k_cj_rowscan / k_cj_scatter   counting sort by (class, bounding index): prefixes
//                 by last index, suffixes by first index; a class's suffixes are padded to whole
//                 blocks of 32 * U, so a block has one class, and prefixes that go with a block
//                 are a leading run of the class's prefix row
//   k_cj_build    per class: filter of the build side, written to global memory
//   k_cj_probe    per class (or part of one): filter in shared memory, every probe record tested;
//                 survivors (prefix, suffix) to per-class chunk lists
//   k_cj_resolve  per class: second filter of the survivors, build records swept against it,
//                 the few that pass chained and looked up by the survivors: pairs equal mod d, m'
//   k_cj_emit     pairs whose residues mod M are equal (recomputed exactly), with their ranks
//
// Pairs go to cf_check_pairs like the fused probe's candidates.  Every equal-residue pair of the
// two rank ranges is found, with all duplicates (gpu/mitm_gpu2.py:107-119, src/mitm64.cpp:85-101).
#include <math.h>
#include <string.h>
#include <algorithm>
#include <vector>
#include "cf_abi_internal.h"
#include "cf_enum.cuh"

namespace {

constexpr int kCjBlock = 1024;
constexpr int kCjWarps = kCjBlock / 32;
constexpr u32 kCjWords = 49152;          // filter words of one class (192 KB: one CTA per SM)
constexpr u32 kCjWords2 = 32768;         // resolve: filter words of the survivors of one round (128 KB)
constexpr u32 kCjHeads = 16384;          // resolve: chain heads of the build records that pass it (64 KB)
constexpr u32 kCjChunk = 128;            // survivors per chunk
constexpr u32 kCjRoundChunks = 16;       // resolve: chunks a warp takes per round (65,536 survivors a round)
constexpr u32 kCjListCap = 32768;        // resolve: build records one round may keep, at most (see listcap)
constexpr u32 kCjCands = kCjWords2 / 4;  // resolve: record pairs equal mod d and m' in one round (64 KB)
constexpr u32 kCjMaxD = 8192;            // class modulus
constexpr u64 kCjMaxList = 1ull << 24;   // prefixes or suffixes of one side
constexpr u32 kCjMinMp = 1u << 27;       // least m': below it too many records share a V
constexpr int kCjMaxR = 8;
constexpr u64 kCjMagic = 0x43464a4f494e3031ull;

struct CjSide {
  u32 n, R, A, b, bw;      // pool size, radius, prefix and suffix sizes, bits of a packed index
  u32 U;                   // suffix entries per lane and block: a block is 32 * U entries of one class
  u32 mult_m, mult_d;      // constant factor of every record, mod m' and mod d
  u32 nP, nT;              // prefixes (of the rank window) and suffixes
  u32 elP, elT;            // their first element in the temporary arrays
  u32 binP, binT;          // first bin: class * n + bounding index
  u32 capT;                // suffix entries with padding (upper bound)
  u64 p_lo;                // first prefix rank
  u64 oTX, oTI, oPW, oPI, oBlk;  // workspace byte offsets
};

}  // namespace

// Host plan of one class join (cf_class_plan_bytes() bytes; the first fields are read by the caller).
struct CfClassPlan {
  u64 magic;
  u32 ok, d, mp, phi;      // ok: the class join applies; class modulus, filter modulus, classes
  u64 ws_bytes;            // workspace of cf_class_join
  u32 r, swap, elems, run; // run: list elements per thread of k_cj_count
  u64 i_lo, i_n;
  u64 zero_bytes;
  u32 maxchunks, maxcands;
  u32 listcap, pad;
  u64 oCtr, oBins, oHeads, oUnits, oInv, oRowBase, oRowTot, oRowCnt, oTmp, oBm, oCmeta, oChunkV, oChunks, oList, oCands;
  CjSide side[2];          // 0: build side, 1: probe side
};

namespace {

enum { kCtrChunks = 0, kCtrBuild = 1, kCtrResolve = 3, kCtrUnits = 4, kCtrCands = 7, kCtrNb0 = 5, kCtrNb1 = 6 };

struct CjArgs {
  CfClassPlan p;
  unsigned char* ws;
  const u64* pool[2];      // pool tables of the build and probe sides
  CfPair* pairs;
  u32 *npairs, *err;
  u32 max_pairs;
};

template <class T>
__device__ __forceinline__ T* at(const CjArgs& a, u64 off) {
  return (T*)(a.ws + off);
}

// c * v mod d for c, v < d <= 8192.
__device__ __forceinline__ u32 mulmod_d(u32 c, u32 v, u32 d) { return c * v % d; }

__device__ __forceinline__ void cj_unrank(u64 rank, int n, const u64* __restrict__ binom, int stride, int K,
                                          int (&idx)[4]) {
  int start = 0;
#pragma unroll
  for (int pos = 0; pos < 4; ++pos) {
    if (pos >= K) break;
    const int rem = K - pos - 1;
    if (rem == 0) {
      idx[pos] = start + (int)rank;
      break;
    }
    const u64 total = binom[(size_t)(n - start) * stride + rem + 1];
    const u64 Y = total - rank;
    int lo = start, hi = n - 1 - rem;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (binom[(size_t)(n - mid) * stride + rem + 1] >= Y) lo = mid; else hi = mid - 1;
    }
    idx[pos] = lo;
    rank -= total - binom[(size_t)(n - lo) * stride + rem + 1];
    start = lo + 1;
  }
}

// Element e of the four lists, in this order: suffixes then prefixes of the build side, then of
// the probe side.
__device__ __forceinline__ bool cj_element(const CjArgs& a, u32 e, int& s, bool& prefix, u32& i) {
  for (s = 0; s < 2; ++s) {
    const CjSide& sd = a.p.side[s];
    if (e - sd.elT < sd.nT) { prefix = false; i = e - sd.elT; return true; }
    if (e - sd.elP < sd.nP) { prefix = true; i = e - sd.elP; return true; }
  }
  return false;
}

// Next K-subset in lexicographic order.
__device__ __forceinline__ void cj_next(int n, int K, int (&idx)[4]) {
  int j = K - 1;
#pragma unroll
  for (int t = 3; t > 0; --t)
    if (t == j && t < K && idx[t] == n - K + t) --j;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    if (t == j) idx[t] += 1;
    else if (t > j && t > 0 && t < K) idx[t] = idx[t - 1] + 1;
  }
}

// A thread takes `run` consecutive elements and unranks the first only: 4 where the lists fill the GPU
// all the same (6.4e5 elements: 21 us with runs of 1, 25 with 4; 3.5e6: 138 and 102).
__global__ void __launch_bounds__(256) k_cj_count(const __grid_constant__ CjArgs a) {
  u32* bins = at<u32>(a, a.p.oBins);
  u32* t_bin = at<u32>(a, a.p.oTmp);
  u32 *t_pos = t_bin + a.p.elems, *t_x = t_pos + a.p.elems, *t_pk = t_x + a.p.elems;
  const u32 runs = (a.p.elems + a.p.run - 1) / a.p.run;
  for (u32 g = blockIdx.x * blockDim.x + threadIdx.x; g < runs; g += gridDim.x * blockDim.x) {
    int idx[4] = {0, 0, 0, 0};
    int in = -1;                                   // list of the previous element: 2 * side + prefix
#pragma unroll 1
    for (u32 e = g * a.p.run; e < min(a.p.elems, (g + 1) * a.p.run); ++e) {
      int s;
      bool prefix;
      u32 i;
      if (!cj_element(a, e, s, prefix, i)) continue;
      const CjSide& sd = a.p.side[s];
      const u64* pool = a.pool[s];
      const int K = (int)(prefix ? sd.A : sd.b), n = (int)sd.n;
      if (in == 2 * s + (int)prefix) cj_next(n, K, idx);
      else cj_unrank(prefix ? sd.p_lo + i : (u64)i, n, pool + cf_pool_off_binom(n), (int)sd.R + 1, K, idx);
      in = 2 * s + (int)prefix;
      const u64* pr = pool + cf_pool_off_prime(n);
      u64 x = prefix ? sd.mult_m : 1u;
      u32 c = prefix ? sd.mult_d : 1u % a.p.d;
      u32 pk = 0;
      int last = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j >= K) break;
        const u64 q = pr[idx[j]];                  // below 2^31, x below 2^32
        x = x * q % a.p.mp;
        c = c * ((u32)q % a.p.d) % a.p.d;
        pk |= (u32)idx[j] << (sd.bw * j);
        last = idx[j];
      }
      const u32 bin = (prefix ? sd.binP : sd.binT) + c * sd.n + (u32)(prefix ? last : idx[0]);
      t_bin[e] = bin;
      t_pos[e] = atomicAdd(&bins[bin], 1u);
      t_x[e] = (u32)x;
      t_pk[e] = pk;
    }
  }
}

__device__ u32 cj_inverse(u32 v, u32 d) {          // v^-1 mod d, or 0 when there is none (or d == 1)
  int r0 = (int)d, r1 = (int)v, t0 = 0, t1 = 1;
  while (r1) {
    const int q = r0 / r1, r2 = r0 - q * r1, t2 = t0 - q * t1;
    r0 = r1; r1 = r2; t0 = t1; t1 = t2;
  }
  if (r0 != 1) return 0;
  return (u32)(t0 < 0 ? t0 + (int)d : t0) % d;
}

// One warp per row (list, class): exclusive prefix of its bins in place, and the row's length
// (suffix rows rounded up to whole blocks).  Lists: 0, 1 suffixes and prefixes of the build side,
// 2, 3 of the probe side.
__global__ void __launch_bounds__(256) k_cj_rows(const __grid_constant__ CjArgs a) {
  const u32 row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const u32 d = a.p.d;
  if (row >= 4 * d) return;
  const u32 l = row / d, c = row % d;
  const CjSide& sd = a.p.side[l >> 1];
  const bool prefix = l & 1;
  u32* b = at<u32>(a, a.p.oBins) + (prefix ? sd.binP : sd.binT) + (size_t)c * sd.n;
  u32 run = 0;
  for (u32 o = 0; o < sd.n; o += 32) {
    const u32 v = o + lane < sd.n ? b[o + lane] : 0u;
    u32 incl = v;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, incl, k);
      if (lane >= (u32)k) incl += x;
    }
    if (o + lane < sd.n) b[o + lane] = run + incl - v;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) {
    const u32 w = 32 * sd.U;
    at<u32>(a, a.p.oRowCnt)[row] = run;
    at<u32>(a, a.p.oRowTot)[row] = prefix ? run : (run + w - 1) / w * w;
    if (l == 0) {
      const u32 inv = d == 1 ? 0u : cj_inverse(c, d);
      at<u32>(a, a.p.oInv)[c] = inv;
      if (inv || d == 1) {
        const u32 u = atomicAdd(at<u32>(a, a.p.oCtr) + kCtrUnits, 1u);
        if (u < a.p.phi) at<u32>(a, a.p.oUnits)[u] = c;
      }
    }
  }
}

// Exclusive prefix of each list's row lengths (one CTA), and the suffix block counts.
__global__ void __launch_bounds__(kCjBlock) k_cj_rowscan(const __grid_constant__ CjArgs a) {
  __shared__ u32 s_w[kCjWarps];
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5, d = a.p.d;
  const u32* tot = at<u32>(a, a.p.oRowTot);
  u32* base = at<u32>(a, a.p.oRowBase);
  for (u32 l = 0; l < 4; ++l) {
    u32 run = 0;
    for (u32 o = 0; o < d; o += kCjBlock) {
      const u32 i = o + threadIdx.x;
      const u32 v = i < d ? tot[l * d + i] : 0u;
      u32 incl = v;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const u32 x = __shfl_up_sync(0xffffffffu, incl, k);
        if (lane >= (u32)k) incl += x;
      }
      if (lane == 31) s_w[wid] = incl;
      __syncthreads();
      if (wid == 0) {
        u32 t = s_w[lane];
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
          const u32 x = __shfl_up_sync(0xffffffffu, t, k);
          if (lane >= (u32)k) t += x;
        }
        s_w[lane] = t;
      }
      __syncthreads();
      if (i < d) base[l * d + i] = run + (wid ? s_w[wid - 1] : 0u) + incl - v;
      run += s_w[kCjWarps - 1];
      __syncthreads();
    }
    if (threadIdx.x == 0 && !(l & 1)) at<u32>(a, a.p.oCtr)[l ? kCtrNb1 : kCtrNb0] = run / (32 * a.p.side[l >> 1].U);
  }
}

__global__ void __launch_bounds__(256) k_cj_scatter(const __grid_constant__ CjArgs a) {
  const u32* bins = at<u32>(a, a.p.oBins);
  const u32* t_bin = at<u32>(a, a.p.oTmp);
  const u32 *t_pos = t_bin + a.p.elems, *t_x = t_pos + a.p.elems, *t_pk = t_x + a.p.elems;
  const u32* base = at<u32>(a, a.p.oRowBase);
  const u32* inv = at<u32>(a, a.p.oInv);
  const u32 d = a.p.d;
  for (u32 e = blockIdx.x * blockDim.x + threadIdx.x; e < a.p.elems; e += gridDim.x * blockDim.x) {
    int s;
    bool prefix;
    u32 i;
    if (!cj_element(a, e, s, prefix, i)) continue;
    const CjSide& sd = a.p.side[s];
    const u32 bin = t_bin[e];
    const u32 c = (bin - (prefix ? sd.binP : sd.binT)) / sd.n;
    const u32 to = base[(2 * s + (prefix ? 1 : 0)) * d + c] + bins[bin] + t_pos[e];
    const u32 x = t_x[e], pk = t_pk[e];
    if (prefix) {                                  // w = floor(x * 2^64 / m')
      const u64 n1 = (u64)x << 32;
      const u64 hi = n1 / a.p.mp, rem = n1 - hi * a.p.mp;
      at<u64>(a, sd.oPW)[to] = (hi << 32) | ((rem << 32) / a.p.mp);
      at<u32>(a, sd.oPI)[to] = pk;
    } else {
      at<u32>(a, sd.oTX)[to] = x;                  // a unit mod m': never 0, the padding's value
      at<u32>(a, sd.oTI)[to] = pk;
    }
  }
  // per suffix block: inverse of its class and the first index of its last entry (a warp per class row)
  const u32 lane = threadIdx.x & 31;
  for (u32 row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < 2 * d; row += (gridDim.x * blockDim.x) >> 5) {
    const u32 s = row >= d, c = row - s * d;
    const CjSide& sd = a.p.side[s];
    const u32 w = 32 * sd.U, nb = at<u32>(a, a.p.oRowTot)[2 * s * d + c] / w,
              cnt = at<u32>(a, a.p.oRowCnt)[2 * s * d + c];
    const u32* b = bins + sd.binT + (size_t)c * sd.n;
    for (u32 i = lane; i < nb; i += 32) {
      const u32 at_end = min((i + 1) * w, cnt) - 1;
      u32 lo = 0, hi = sd.n - 1;                   // bin of the block's last entry: largest f with b[f] <= at_end
      while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (b[mid] <= at_end) lo = mid; else hi = mid - 1;
      }
      at<u32>(a, sd.oBlk)[base[2 * s * d + c] / w + i] = (inv[c] << 16) | lo;
    }
  }
}

// Scaled residue of prefix w times suffix x.
__device__ __forceinline__ u32 cj_v(u64 w, u32 x) { return (u32)(w >> 32) * x + __umulhi((u32)w, x); }

// Filter place of V: word and two bits (the second may equal the first), from the bits 22 and up of
// V * kCjWords; returns the bits below.
__device__ __forceinline__ u32 cj_place(u32 V, u32& word, u32& mask) {
  const u64 q = (u64)V * kCjWords;
  const u32 lo = (u32)q;
  word = (u32)(q >> 32);
  mask = (1u << (lo >> 27)) | (1u << ((lo >> 22) & 31u));
  return lo & 0x3fffffu;
}

// One warp's share of the suffix blocks [b0, b1) of a class, 32 blocks at a time, one per lane: the
// loads that lead from a block to its prefix run (block -> class of the prefixes -> run length) are
// one latency for 32 blocks.  Long ranges go out in chunks of 32 consecutive blocks (whole sectors
// of the lookups); in short ones, where a chunk more or less per warp would show, round i takes
// block 32 * i + (warp + 7 * i) % 32, so that no warp keeps meeting the same place of equally long
// class rows.
constexpr u32 kCjLongRange = 1u << 14;
struct CjRun {
  u32 b, first, cnt, k;    // block, first prefix entry, prefixes that go with it, their class
};
__device__ __forceinline__ CjRun cj_lookup(const CjArgs& a, const CjSide& sd, int s, u32 c, u32 b0, u32 b1, u32 i0) {
  CjRun r;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = i0 + lane;
  r.b = b0 + 32 * i0 + (b1 - b0 >= kCjLongRange ? 32 * warp + lane : 32 * lane + ((warp + 7 * i) & 31u));
  r.cnt = 0;
  r.first = r.k = 0;
  if (r.b < b1) {
    const u32 info = at<u32>(a, sd.oBlk)[r.b];
    r.k = mulmod_d(c, info >> 16, a.p.d);
    r.cnt = at<u32>(a, a.p.oBins)[sd.binP + r.k * sd.n + (info & 0xffffu)];
    r.first = at<u32>(a, a.p.oRowBase)[(2 * s + 1) * a.p.d + r.k];
  }
  return r;
}

// Run f(V, prefix entry, suffix entry) for every build-side record of class c (this warp's blocks).
// Class rows of the smaller side are short (tens of entries), so the block set-up and the lanes past
// their last prefix weigh as much as the records: 7.6e6 records in 40 us (build) at 144 classes; 49 with the
// places of V - 1 and V + 1 computed for every record (r = 7, 6.2e8 records: 7.9 and 9.7 ms).
template <int U, class F>
__device__ __forceinline__ void cj_sweep(const CjArgs& a, const CjSide& sd, int s, u32 c, u32 nblk, F f) {
  const u32 lane = threadIdx.x & 31;
  const u32* TX = at<u32>(a, sd.oTX);
  const u32* TI = at<u32>(a, sd.oTI);
  const u64* PW = at<u64>(a, sd.oPW);
  const u32* bins = at<u32>(a, a.p.oBins) + sd.binP;
  const u32 fm = (1u << sd.bw) - 1u;
  for (u32 i0 = 0; i0 * 32 < nblk; i0 += 32) {
    const CjRun mine = cj_lookup(a, sd, s, c, 0, nblk, i0);
    for (u32 todo = __ballot_sync(0xffffffffu, mine.cnt != 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const u32 b = __shfl_sync(0xffffffffu, mine.b, src), cnt = __shfl_sync(0xffffffffu, mine.cnt, src);
      const u32 first = __shfl_sync(0xffffffffu, mine.first, src), k = __shfl_sync(0xffffffffu, mine.k, src);
      u32 x[U], ti[U], lim[U];
      const u32 t0 = b * 32 * U + lane;
      u64 w = lane < cnt ? PW[first + lane] : 0ull;
#pragma unroll
      for (int u = 0; u < U; ++u) { x[u] = TX[t0 + 32 * u]; ti[u] = TI[t0 + 32 * u]; }
#pragma unroll
      for (int u = 0; u < U; ++u) lim[u] = x[u] ? bins[k * sd.n + (ti[u] & fm)] : 0u;   // prefixes ending before it
      for (u32 j0 = 0; j0 < cnt; j0 += 32) {
        const u32 m = min(32u, cnt - j0);
        if (j0) w = lane < m ? PW[first + j0 + lane] : 0ull;
        for (u32 j = 0; j < m; ++j) {
          const u64 wj = __shfl_sync(0xffffffffu, w, j);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j0 + j < lim[u]) f(cj_v(wj, x[u]), first + j0 + j, t0 + 32 * u);
        }
      }
    }
  }
}

template <class F>
__device__ __forceinline__ void cj_sweep_u(const CjArgs& a, const CjSide& sd, int s, u32 c, u32 nblk, F f) {
  if (sd.U == 4) cj_sweep<4>(a, sd, s, c, nblk, f);
  else if (sd.U == 2) cj_sweep<2>(a, sd, s, c, nblk, f);
  else cj_sweep<1>(a, sd, s, c, nblk, f);
}

__global__ void __launch_bounds__(kCjBlock, 1) k_cj_build(const __grid_constant__ CjArgs a) {
  extern __shared__ __align__(16) u32 s_bm[];
  __shared__ u32 s_unit;
  u32* ctr = at<u32>(a, a.p.oCtr);
  const u32 nblk = ctr[kCtrNb0];
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_unit = atomicAdd(ctr + kCtrBuild, 1u);
    for (u32 i = threadIdx.x; i < kCjWords / 4; i += kCjBlock) ((uint4*)s_bm)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const u32 ci = s_unit;
    if (ci >= a.p.phi) return;
    const u32 c = at<u32>(a, a.p.oUnits)[ci];
    cj_sweep_u(a, a.p.side[0], 0, c, nblk, [&](u32 V, u32, u32) {
      u32 w0, m0;
      const u32 rest = cj_place(V, w0, m0);
      atomicOr(&s_bm[w0], m0);
      // V - 1 and V + 1 have the same place unless kCjWords less or more leaves the bits below it: 1 in 85 each
      const bool down = rest < kCjWords, up = rest >= 0x400000u - kCjWords;
      if (down || up) {
        cj_place(down ? V - 1u : V + 1u, w0, m0);
        atomicOr(&s_bm[w0], m0);
      }
    });
    __syncthreads();
    uint4* out = at<uint4>(a, a.p.oBm) + (size_t)ci * (kCjWords / 4);
    for (u32 i = threadIdx.x; i < kCjWords / 4; i += kCjBlock) out[i] = ((uint4*)s_bm)[i];
  }
}

// Survivors of one warp: chunks of kCjChunk, linked per (class, warp).
struct CjSink {
  u32 chunk, fill;         // open chunk + 1 (0: none) and its entries
};
__device__ __forceinline__ void cj_close(const CjArgs& a, CjSink& k) {
  if (k.chunk && (threadIdx.x & 31) == 0) at<u32>(a, a.p.oCmeta)[2 * (size_t)(k.chunk - 1) + 1] = k.fill;
  k.chunk = 0;
  k.fill = 0;
}
__device__ __forceinline__ void cj_push(const CjArgs& a, CjSink& k, u32 ci, bool have, u32 V, u64 v) {
  const u32 act = __ballot_sync(0xffffffffu, have), n = __popc(act);
  const u32 lane = threadIdx.x & 31;
  if (n == 0) return;
  if (k.chunk == 0 || k.fill + n > kCjChunk) {
    cj_close(a, k);
    u32 id = 0;
    if (lane == 0) id = atomicAdd(at<u32>(a, a.p.oCtr) + kCtrChunks, 1u);
    id = __shfl_sync(0xffffffffu, id, 0);
    if (id >= a.p.maxchunks) {                     // lost survivors: the caller repeats the join another way
      if (lane == 0) atomicOr(a.err, CF_ERR_PART_OVERFLOW);
      return;
    }
    if (lane == 0) {                               // a (class, warp) list may grow in several CTAs
      const u32 nxt = atomicExch(at<u32>(a, a.p.oHeads) + (size_t)ci * kCjWarps + (threadIdx.x >> 5), id + 1);
      at<u32>(a, a.p.oCmeta)[2 * (size_t)id] = nxt;
    }
    k.chunk = id + 1;
  }
  if (have) {
    const size_t to = (size_t)(k.chunk - 1) * kCjChunk + k.fill + __popc(act & ((1u << lane) - 1u));
    at<u32>(a, a.p.oChunkV)[to] = V;
    at<u64>(a, a.p.oChunks)[to] = v;
  }
  k.fill += n;
}

// The first 32 (or the last n) survivors of a warp's ring, one per lane: the records among them go to
// the chunk list with their V.  A prefix that reaches past the suffix's first index is no record.
__device__ __forceinline__ void cj_drain(const CjArgs& a, CjSink& k, u32 ci, const uint2* ring, u32 n) {
  const CjSide& sd = a.p.side[1];
  const u32 lane = threadIdx.x & 31;
  u32 V = 0;
  bool rec = false;
  uint2 e = make_uint2(0u, 0u);                    // prefix entry, suffix entry
  if (lane < n) {
    e = ring[lane];
    const u32 first = at<u32>(a, sd.oTI)[e.y] & ((1u << sd.bw) - 1u);
    const u32 last = at<u32>(a, sd.oPI)[e.x] >> (sd.bw * (sd.A - 1));
    V = cj_v(at<u64>(a, sd.oPW)[e.x], at<u32>(a, sd.oTX)[e.y]);
    rec = first > last;
  }
  cj_push(a, k, ci, rec, V, ((u64)e.x << 32) | e.y);
}

template <int U>
__device__ __forceinline__ void cj_probe_range(const CjArgs& a, const u32* s_bm, uint2* ring, u32 ci, u32 c, u32 b0,
                                               u32 b1) {
  const CjSide& sd = a.p.side[1];
  const u32 lane = threadIdx.x & 31;
  const u32* TX = at<u32>(a, sd.oTX);
  const u64* PW = at<u64>(a, sd.oPW);
  constexpr u32 G = 32 / U;                        // prefixes per word of outcome bits
  constexpr u32 kPat = U == 4 ? 0x11111111u : U == 2 ? 0x55555555u : 0xffffffffu;
  const u32 below = (1u << lane) - 1u;
  CjSink sink{0, 0};
  u32 held = 0;                                    // survivors in the ring
  for (u32 i0 = 0; b0 + i0 * 32 < b1; i0 += 32) {
    const CjRun mine = cj_lookup(a, sd, 1, c, b0, b1, i0);
    for (u32 todo = __ballot_sync(0xffffffffu, mine.cnt != 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const u32 t0 = __shfl_sync(0xffffffffu, mine.b, src) * 32 * U + lane;
      const u32 cnt = __shfl_sync(0xffffffffu, mine.cnt, src), first = __shfl_sync(0xffffffffu, mine.first, src);
      u32 x[U], keep = 0;                          // keep: outcome bits of entries that are not padding
      u64 w = lane < cnt ? PW[first + lane] : 0ull;
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = TX[t0 + 32 * u];
#pragma unroll
      for (int u = 0; u < U; ++u) keep |= x[u] ? kPat << (U - 1 - u) : 0u;
      for (u32 j0 = 0; j0 < cnt; j0 += 32) {
        const u32 m = min(32u, cnt - j0);
        if (j0) w = lane < m ? PW[first + j0 + lane] : 0ull;
        for (u32 g0 = 0; g0 < m; g0 += G) {
          const u32 g1 = min(m, g0 + G);
          u32 acc = 0;                             // bit (prefix, entry), the last one lowest
#pragma unroll 2
          for (u32 j = g0; j < g1; ++j) {
            const u64 wj = __shfl_sync(0xffffffffu, w, j);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const u64 q = (u64)cj_v(wj, x[u]) * kCjWords;
              const u32 lo = (u32)q, f = s_bm[q >> 32];
              acc = acc + acc + (__funnelshift_r(f, f, lo >> 27) & __funnelshift_r(f, f, lo >> 22) & 1u);
            }
          }
          acc &= keep;
          const u32 top = (g1 - g0) * U - 1u, pf = first + j0 + g0;
          for (u32 act; (act = __ballot_sync(0xffffffffu, acc != 0)) != 0;) {
            if (acc) {
              const u32 q = top - ((u32)__ffs(acc) - 1u);           // (prefix - g0) * U + entry
              ring[held + __popc(act & below)] = make_uint2(pf + q / U, t0 + 32 * (q % U));
              acc &= acc - 1u;
            }
            held += __popc(act);
            if (held >= 32) {                      // a full warp of survivors at a time
              __syncwarp();
              cj_drain(a, sink, ci, ring, 32);
              held -= 32;
              const uint2 rest = ring[32 + lane];
              __syncwarp();
              if (lane < held) ring[lane] = rest;
              __syncwarp();
            }
          }
        }
      }
    }
  }
  if (held) {
    __syncwarp();
    cj_drain(a, sink, ci, ring, held);
  }
  __syncwarp();
  cj_close(a, sink);
}

// Bound by integer issue: k = 64, r = 5, 5.9e8 I records in 0.60 ms (9.8e11 records/s; the fused
// probe 3.2 ms), issue slots 68% busy, ALU pipe 62%, the multiplier pipe 57%, shared memory 55%; 24
// instructions per 32 records, of which 12 test, the rest survivors, prefixes past their suffix (10 to
// 30%) and the block set-up.  Survivors wait in a ring per warp until 32 can be looked up at once
// (pushed as found, with their V from registers: 0.64 ms).  32 warps of 64 registers: more registers
// would halve the warps that hide the shared-memory latency.  CTA g of G takes the g-th of G equal parts of the (class, suffix block) sequence: whole classes
// and a part of one at either end, so a filter is loaded phi + G times in all.
__global__ void __launch_bounds__(kCjBlock, 1) k_cj_probe(const __grid_constant__ CjArgs a) {
  extern __shared__ __align__(16) u32 s_bm[];
  uint2* ring = (uint2*)(s_bm + kCjWords) + (threadIdx.x >> 5) * 64;   // this warp's survivors
  const u32 nblk = at<u32>(a, a.p.oCtr)[kCtrNb1];
  const u64 total = (u64)a.p.phi * nblk;
  u64 lo = total * blockIdx.x / gridDim.x;
  const u64 hi = total * (blockIdx.x + 1) / gridDim.x;
  while (lo < hi) {
    const u32 ci = (u32)(lo / nblk), b0 = (u32)(lo - (u64)ci * nblk);
    const u32 b1 = (u32)min((u64)nblk, b0 + (hi - lo));
    const u32 c = at<u32>(a, a.p.oUnits)[ci];
    const uint4* in = at<uint4>(a, a.p.oBm) + (size_t)ci * (kCjWords / 4);
    __syncthreads();
#pragma unroll 12
    for (u32 i = threadIdx.x; i < kCjWords / 4; i += kCjBlock) ((uint4*)s_bm)[i] = __ldcg(in + i);
    __syncthreads();
    if (a.p.side[1].U == 4) cj_probe_range<4>(a, s_bm, ring, ci, c, b0, b1);
    else if (a.p.side[1].U == 2) cj_probe_range<2>(a, s_bm, ring, ci, c, b0, b1);
    else cj_probe_range<1>(a, s_bm, ring, ci, c, b0, b1);
    lo += b1 - b0;
  }
}

// ---- resolve -------------------------------------------------------------------

// Second hash, of V without its three lowest bits: records equal mod m' have V within one, so
// their V >> 3 is equal or neighbouring.
__device__ __forceinline__ void cj_place2(u32 v3, u32& word, u32& mask) {
  const u32 h = v3 * 0x9E3779B1u;
  word = h >> 17;                                  // kCjWords2 words
  mask = (1u << ((h >> 12) & 31u)) | (1u << ((h >> 7) & 31u));
}
__device__ __forceinline__ u32 cj_head(u32 v3) { return (v3 * 0x85EBCA6Bu) >> 18; }   // kCjHeads heads

// Packed indices of record (p, t) of a side, ascending.
__device__ __forceinline__ void cj_indices(const CjArgs& a, const CjSide& sd, u32 p, u32 t, int (&idx)[kCjMaxR]) {
  const u32 pk = at<u32>(a, sd.oPI)[p], tk = at<u32>(a, sd.oTI)[t], m = (1u << sd.bw) - 1u;
  for (u32 j = 0; j < sd.A; ++j) idx[j] = (int)((pk >> (sd.bw * j)) & m);
  for (u32 j = 0; j < sd.b; ++j) idx[sd.A + j] = (int)((tk >> (sd.bw * j)) & m);
}
__device__ __forceinline__ u64 cj_full_key(const u64* __restrict__ pool, int n, int r, const int (&idx)[kCjMaxR]) {
  const CfPoolHdr* hd = (const CfPoolHdr*)pool;
  const CfMod32 md = cf_mod32_from_hdr(hd);
  const u64* pr = pool + cf_pool_off_prime(n);
  CfElt32 e;
  e.X = hd->X0;
  e.x2 = hd->x20;
  for (int j = 0; j < r; ++j) e = cf_mul32(e, (u32)pr[idx[j]], md);
  return cf_key32(e, md);
}
__device__ __forceinline__ u64 cj_rank(const u64* __restrict__ pool, int n, int r, const int (&idx)[kCjMaxR]) {
  const u64* binom = pool + cf_pool_off_binom(n);
  u64 rank = 0;
  int start = 0;
  for (int j = 0; j < r; ++j) {
    rank += binom[(size_t)(n - start) * (r + 1) + r - j] - binom[(size_t)(n - idx[j]) * (r + 1) + r - j];
    start = idx[j] + 1;
  }
  return rank;
}

// Build record (bp, bt) and probe record (pp, pt) agree mod d and m': append them when their full
// residues agree and the I record lies in the rank window.
__device__ __forceinline__ void cj_emit(const CjArgs& a, u32 bp, u32 bt, u32 pp, u32 pt) {
  const CjSide &sb = a.p.side[0], &sp = a.p.side[1];
  const int r = (int)a.p.r;
  int ib[kCjMaxR], ip[kCjMaxR];
  cj_indices(a, sb, bp, bt, ib);
  cj_indices(a, sp, pp, pt, ip);
  if (cj_full_key(a.pool[0], (int)sb.n, r, ib) != cj_full_key(a.pool[1], (int)sp.n, r, ip)) return;
  const u64 rb = cj_rank(a.pool[0], (int)sb.n, r, ib), rp = cj_rank(a.pool[1], (int)sp.n, r, ip);
  CfPair pr;
  pr.d_id = a.p.swap ? rp : rb;
  pr.i_id = a.p.swap ? rb : rp;
  if (pr.i_id - a.p.i_lo >= a.p.i_n) return;
  const u32 k = atomicAdd(a.npairs, 1u);
  if (k < a.max_pairs) a.pairs[k] = pr;
  else atomicOr(a.err, CF_ERR_PAIR_OVERFLOW);
}

// f(V, place in the chunk arrays) for the survivors in up to kCjRoundChunks chunks from `chunk`
// (1-based) of this warp's list; returns the next chunk.
template <class F>
__device__ __forceinline__ u32 cj_survivors(const CjArgs& a, u32 chunk, F f) {
  const u32 lane = threadIdx.x & 31;
  static_assert(kCjChunk == 128, "four entries per lane");
  for (u32 i = 0; i < kCjRoundChunks && chunk; ++i) {
    const uint2 meta = *(at<uint2>(a, a.p.oCmeta) + (chunk - 1));
    const u32 base = (chunk - 1) * kCjChunk + 4 * lane;
    const uint4 v = *(const uint4*)(at<u32>(a, a.p.oChunkV) + base);   // entries from the fill on are not used
    if (4 * lane + 0 < meta.y) f(v.x, base);
    if (4 * lane + 1 < meta.y) f(v.y, base + 1);
    if (4 * lane + 2 < meta.y) f(v.z, base + 2);
    if (4 * lane + 3 < meta.y) f(v.w, base + 3);
    chunk = meta.x;
  }
  return chunk;
}

struct CjKept {
  u32 V, p, t, next;
};

__global__ void __launch_bounds__(kCjBlock, 1) k_cj_resolve(const __grid_constant__ CjArgs a) {
  extern __shared__ __align__(16) u32 smem[];
  u32* s_bm = smem;
  u32* s_head = smem + kCjWords2;
  uint2* s_cand = (uint2*)(smem + kCjWords2 / 2);   // after the first filter: the kept records' filter, candidates
  __shared__ u32 s_unit, s_n, s_m, s_at;
  u32* ctr = at<u32>(a, a.p.oCtr);
  const u32 nblk = ctr[kCtrNb0];
  CjKept* list = at<CjKept>(a, a.p.oList) + (size_t)blockIdx.x * a.p.listcap;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_unit = atomicAdd(ctr + kCtrResolve, 1u);
    __syncthreads();
    const u32 ci = s_unit;
    if (ci >= a.p.phi) return;
    const u32 c = at<u32>(a, a.p.oUnits)[ci];
    u32 chunk = at<u32>(a, a.p.oHeads)[(size_t)ci * kCjWarps + (threadIdx.x >> 5)];
    while (__syncthreads_or(chunk != 0)) {         // rounds of at most 32 * 16 * 128 survivors
      for (u32 i = threadIdx.x; i < (kCjWords2 + kCjHeads) / 4; i += kCjBlock)
        ((uint4*)smem)[i] = make_uint4(0u, 0u, 0u, 0u);
      if (threadIdx.x == 0) s_n = s_m = 0;
      __syncthreads();
      const u32 next = cj_survivors(a, chunk, [&](u32 V, u32) {
        u32 w, m;
        cj_place2(V >> 3, w, m);
        atomicOr(&s_bm[w], m);
        if ((V & 7u) == 0u || (V & 7u) == 7u) {
          cj_place2((V & 7u) ? (V + 1u) >> 3 : (V - 1u) >> 3, w, m);
          atomicOr(&s_bm[w], m);
        }
      });
      __syncthreads();
      cj_sweep_u(a, a.p.side[0], 0, c, nblk, [&](u32 V, u32 p, u32 t) {
        u32 w, m;
        cj_place2(V >> 3, w, m);
        if ((s_bm[w] & m) == m) {
          const u32 k = atomicAdd(&s_n, 1u);
          if (k < a.p.listcap) {
            CjKept e;
            e.V = V;
            e.p = p;
            e.t = t;
            e.next = atomicExch(&s_head[cj_head(V >> 3)], k + 1u);
            list[k] = e;
          } else {
            atomicOr(a.err, CF_ERR_PART_OVERFLOW);
          }
        }
      });
      __syncthreads();
      // the kept records' own filter (64 KB of the first one's place): nearly every survivor stops there
      const u32 kept = min(s_n, a.p.listcap);
      for (u32 i = threadIdx.x; i < kCjWords2 / 8; i += kCjBlock) ((uint4*)s_bm)[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      for (u32 i = threadIdx.x; i < kept; i += kCjBlock) {
        u32 w, m;
        cj_place2(list[i].V >> 3, w, m);
        atomicOr(&s_bm[w >> 1], m);
      }
      __syncthreads();
      cj_survivors(a, chunk, [&](u32 V, u32 pos) {
        const u32 lo = (V - 1u) >> 3, hi = (V + 1u) >> 3;
        for (u32 v3 = V >> 3, step = 0; step < 2; ++step) {
          u32 w, m;
          cj_place2(v3, w, m);
          if ((s_bm[w >> 1] & m) == m)
            for (u32 k = s_head[cj_head(v3)]; k;) {
              const CjKept e = list[k - 1];
              if ((e.V >> 3) == v3 && e.V - V + 1u <= 2u) {
                const u32 q = atomicAdd(&s_m, 1u);
                if (q < kCjCands) s_cand[q] = make_uint2(k - 1u, pos);
                else atomicOr(a.err, CF_ERR_PART_OVERFLOW);
              }
              k = e.next;
            }
          if (lo != v3) v3 = lo;
          else if (hi != v3) v3 = hi;
          else break;
        }
      });
      __syncthreads();
      const u32 nc = min(s_m, kCjCands);
      if (threadIdx.x == 0 && nc) s_at = atomicAdd(ctr + kCtrCands, nc);
      __syncthreads();
      for (u32 i = threadIdx.x; i < nc; i += kCjBlock) {
        const CjKept e = list[s_cand[i].x];
        const u64 pt = at<u64>(a, a.p.oChunks)[s_cand[i].y];
        if (s_at + i < a.p.maxcands) at<uint4>(a, a.p.oCands)[s_at + i] = make_uint4(e.p, e.t, (u32)(pt >> 32), (u32)pt);
        else atomicOr(a.err, CF_ERR_PART_OVERFLOW);
      }
      chunk = next;
    }
  }
}

// The record pairs that agree mod d and m': a kernel of their own, so that their chains of loads
// run side by side on the whole GPU.
__global__ void __launch_bounds__(128) k_cj_emit(const __grid_constant__ CjArgs a) {
  const u32 n = min(at<u32>(a, a.p.oCtr)[kCtrCands], a.p.maxcands);
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 c = at<uint4>(a, a.p.oCands)[i];
    cj_emit(a, c.x, c.y, c.z, c.w);
  }
}

u64 up256(u64 x) { return (x + 255) & ~(u64)255; }

u64 binom_sat(u64 n, u64 k) {
  if (k > n) return 0;
  unsigned __int128 v = 1;
  for (u64 i = 1; i <= k; ++i) {
    v = v * (n - k + i) / i;
    if (v >> 63) return ~0ull;
  }
  return (u64)v;
}

// Estimated warp instructions of one (class, class) item of a side cut into A-prefixes and
// b-suffixes with U entries per lane: a block costs about 30 where it has prefixes, and 5 + 11.5 U
// per prefix of its run, which goes up to the block's largest first index.  Of a row's suffixes
// (Poisson with the expected counts) the last block's largest first index is the row's.
void shape_cost(u32 n, u32 A, u32 b, double phi, double (&cost)[3]) {
  const double row = (double)binom_sat(n, b) / phi;
  double end[3], seen = 0, before = exp(-row);     // before: probability of no entry from index f on
  for (int v = 0; v < 3; ++v) { end[v] = 32 << v; cost[v] = 1.0 + row / end[v]; }
  double w = (double)binom_sat(n - 1, b - 1) / phi, run = 0;   // suffixes from f, prefixes ending below f
  for (u32 f = 0; f + b <= n; ++f) {
    const double left = row - seen - w, after = left > 30 ? 0.0 : exp(-std::max(0.0, left));
    const double some = run > 30 ? 30.0 : 30.0 * (1.0 - exp(-run));
    seen += w;
    for (int v = 0; v < 3; ++v) {
      const double block = some + run * (5.0 + 11.5 * (1 << v));
      cost[v] += (after - before) * block;
      for (; seen >= end[v] && end[v] < row; end[v] += 32 << v) cost[v] += block;
    }
    before = after;
    w *= (double)(n - b - f) / (double)(n - 1 - f > 0 ? n - 1 - f : 1);   // C(n-2-f, b-1) / phi
    run = f + 1 < A ? 0.0 : f + 1 == A ? 1.0 / phi : run * (double)(f + 1) / (double)(f + 1 - A);
  }
}

// Rank among the A-subsets of {0..n-1} of the first A indices of the r-subset at `rank`.
u64 prefix_rank(u64 rank, u64 n, u64 r, u64 A) {
  u64 start = 0, out = 0;
  for (u64 pos = 0; pos < A; ++pos) {
    u64 c = start;
    for (;; ++c) {
      const u64 cnt = binom_sat(n - 1 - c, r - pos - 1);
      if (rank < cnt) break;
      rank -= cnt;
      out += binom_sat(n - 1 - c, A - pos - 1);
    }
    start = c + 1;
  }
  return out;
}

// Largest divisor below 2^32 of prod p^e (the m' of a class modulus that takes the other primes).
u64 best_divisor(const std::vector<std::pair<u64, int>>& f) {
  std::vector<u64> ds{1};
  for (const auto& pe : f) {
    const size_t n = ds.size();
    u64 q = 1;
    for (int e = 0; e < pe.second; ++e) {
      if (q > 0xffffffffull / pe.first) break;
      q *= pe.first;
      for (size_t i = 0; i < n; ++i)
        if (ds[i] <= 0xffffffffull / q) ds.push_back(ds[i] * q);
    }
    if (ds.size() > 200000) break;
  }
  return *std::max_element(ds.begin(), ds.end());
}

}  // namespace

extern "C" size_t cf_class_plan_bytes(void) { return sizeof(CfClassPlan); }

// Plan the class join of the D side C(nD, r) against the I ranks [i_lo, i_lo + i_n) for a modulus
// with odd part m; swap: the I window is the smaller (build) side.  plan->ok is 0 when the class
// join does not apply: no class modulus with about the wanted number of classes and an m' of at
// least 2^27 beside it, lists above 2^24 entries, or a radius outside 2..8.  Host code, no device call.
extern "C" int cf_class_plan(u64 m, int nD, int nI, int r, u64 i_lo, u64 i_n, int swap, void* plan,
                             size_t plan_bytes) try {
  if (!plan || plan_bytes < sizeof(CfClassPlan) || nD < 1 || nI < 1 || nD > CF_MAX_POOL || nI > CF_MAX_POOL) {
    cf_set_error("cf_class_plan: bad arguments%s", "");
    return CF_EBADARG;
  }
  CfClassPlan* P = (CfClassPlan*)plan;
  memset(P, 0, sizeof *P);
  P->magic = kCjMagic;
  if (r < 2 || r > kCjMaxR || !(m & 1) || nD < r || nI < r) return CF_OK;
  const u64 totD = binom_sat(nD, r), totI = binom_sat(nI, r);
  if (totD == ~0ull || totI == ~0ull || i_n == 0 || i_lo >= totI || i_n > totI - i_lo) return CF_OK;
  const double n_build = swap ? (double)i_n : (double)totD, n_probe = swap ? (double)totD : (double)i_n;
  // odd primes of m below the class limit
  std::vector<std::pair<u64, int>> f;
  u64 rest = m;
  for (u64 p = 3; p < kCjMaxD && p * p <= rest; p += 2) {
    int e = 0;
    while (rest % p == 0) { rest /= p; ++e; }
    if (e) f.push_back({p, e});
  }
  if (rest > 1 && rest < kCjMaxD) f.push_back({rest, 1});
  else if (rest > 1 && rest < (1ull << 32)) f.push_back({rest, 1});
  if (f.size() > 14) f.resize(14);
  // One wave of classes (148 SMs; build and resolve take a class per CTA), until a class would hold
  // more than 100,000 build records.  k = 64, r = 5, 5.9e8 I records: 0.86 ms at 144 classes, 1.17
  // at 72, 1.08 at 288; r = 4, 3.0e7 I records: 0.19 ms at 144, 0.37 at 12; r = 6, 4.7e8 I records:
  // 2.2 ms at 1.0e5 records per class, 2.6 at 71,000, 3.4 at 45,000 (the number of (class, class)
  // items grows with the square of the classes, the filter's false positives with the records).
  const double want = std::max(140.0, n_build / 100000);
  struct Cand { double score; u32 mask, d, phi; };
  std::vector<Cand> cs;
  cs.push_back({0.0, 0u, 1u, 1u});                 // the subsets of f with a product up to kCjMaxD: about 130 of 2^14
  for (size_t i = 0; i < f.size(); ++i)            // (a walk over all masks took half of a plan's 40 us)
    for (size_t k = 0, n = cs.size(); k < n; ++k)
      if (cs[k].d * f[i].first <= kCjMaxD)
        cs.push_back({0.0, cs[k].mask | 1u << i, (u32)(cs[k].d * f[i].first), (u32)(cs[k].phi * (f[i].first - 1))});
  for (Cand& x : cs) x.score = fabs(log2(x.phi / want)) + 0.4 * log2(ceil(x.phi / 148.0) * 148.0 / x.phi);
  std::sort(cs.begin(), cs.end(), [](const Cand& x, const Cand& y) { return x.score < y.score || (x.score == y.score && x.mask < y.mask); });
  u64 mp = 0;
  size_t pick = 0;
  for (; pick < cs.size(); ++pick) {
    std::vector<std::pair<u64, int>> g;
    u64 left = m;                                  // m without the class primes: m' divides it
    for (size_t i = 0; i < f.size(); ++i) {
      if (!(cs[pick].mask >> i & 1)) g.push_back(f[i]);
      else
        for (int e = 0; e < f[i].second; ++e) left /= f[i].first;
    }
    // fewer classes than a quarter of the wanted leave most SMs idle (r = 4, 1.4e7 I records, 12
    // classes: 0.31 ms, the table join 0.23)
    if (left < kCjMinMp || 4.0 * cs[pick].phi < want) continue;
    mp = best_divisor(g);
    if (mp >= kCjMinMp) break;
  }
  if (mp < kCjMinMp || pick >= cs.size()) return CF_OK;
  const u32 d = cs[pick].d, phi = cs[pick].phi;
  const double per = n_build / phi;
  if (per > 6.0 * kCjWords) return CF_OK;          // the filter would pass nearly everything
  P->d = d; P->phi = phi; P->mp = (u32)mp;
  P->r = (u32)r; P->swap = (u32)(swap != 0); P->i_lo = i_lo; P->i_n = i_n;
  u64 off = 0, el = 0, bin = 0;
  for (int s = 0; s < 2; ++s) {
    CjSide& sd = P->side[s];
    const bool isI = (s == 0) == (swap != 0);
    sd.n = (u32)(isI ? nI : nD);
    sd.R = (u32)r;
    // prefix size and entries per lane: least estimated cost of all items, with the lists in it (an
    // entry takes about 80 issue slots to make and sort)
    double best = -1;
    u64 nT = 0, p0 = 0, p1 = 0;
    for (int A = 1; A < r; ++A) {
      const int b = r - A, mx = std::max(A, b);
      if (mx > 4 || (mx > 3 && sd.n > 256)) continue;
      const u64 t = binom_sat(sd.n, b);
      u64 q0 = 0, q1 = binom_sat(sd.n, A);
      const u64 pall = q1;
      if (isI && (i_lo || i_n < totI)) {
        q0 = prefix_rank(i_lo, sd.n, r, A);
        q1 = prefix_rank(i_lo + i_n - 1, sd.n, r, A) + 1;
      }
      if (t > kCjMaxList || q1 - q0 > kCjMaxList) continue;
      double cost[3];
      shape_cost(sd.n, (u32)A, (u32)b, phi, cost);
      for (u32 U = 1; U <= 4; U *= 2) {
        const double share = (double)(q1 - q0) / (double)pall;   // of the prefixes, in a rank window
        const double c = cost[U / 2] * phi * phi * share * (s == 0 ? 2 : 1) + 80.0 * (t + q1 - q0);
        if (best >= 0 && c >= best) continue;
        best = c;
        sd.A = (u32)A; sd.b = (u32)b; sd.U = U;
        sd.bw = mx <= 3 ? 10 : 8;
        nT = t; p0 = q0; p1 = q1;
      }
    }
    if (best < 0) return CF_OK;
    sd.nT = (u32)nT;
    sd.nP = (u32)(p1 - p0);
    sd.p_lo = p0;
    sd.capT = (u32)(nT + (u64)phi * 32 * sd.U);
    sd.elT = (u32)el; el += sd.nT;
    sd.elP = (u32)el; el += sd.nP;
    sd.binT = (u32)bin; bin += (u64)d * sd.n;
    sd.binP = (u32)bin; bin += (u64)d * sd.n;
    sd.mult_m = 1; sd.mult_d = 1 % d;
  }
  P->elems = (u32)el;
  P->run = el >= (2u << 20) ? 4 : 1;
  const double lam = per / kCjWords, fp = std::min(0.5, (lam + lam * lam) / 256.0);
  const double chunks = 4096.0 + (double)(phi + 148) * kCjWarps + n_probe * std::min(0.6, 1.5 * fp) / 96.0;
  if (chunks > 3.0e7) return CF_OK;               // entry places stay below 2^32
  P->maxchunks = (u32)chunks;
  // zeroed region first
  P->oCtr = off; off += 256;
  P->oBins = off; off = up256(off + bin * 4);
  for (int s = 0; s < 2; ++s) { P->side[s].oBlk = off; off = up256(off + (P->side[s].capT / (32 * P->side[s].U) + 1) * 4ull); }
  for (int s = 0; s < 2; ++s) { P->side[s].oTX = off; off = up256(off + P->side[s].capT * 4ull); }
  P->oHeads = off; off = up256(off + (u64)phi * kCjWarps * 4);
  P->zero_bytes = off;
  P->oUnits = off; off = up256(off + (u64)phi * 4);
  P->oInv = off; off = up256(off + (u64)d * 4);
  P->oRowBase = off; off = up256(off + (u64)d * 16);
  P->oRowTot = off; off = up256(off + (u64)d * 16);
  P->oRowCnt = off; off = up256(off + (u64)d * 16);
  P->oTmp = off; off = up256(off + el * 16);
  for (int s = 0; s < 2; ++s) {
    CjSide& sd = P->side[s];
    sd.oTI = off; off = up256(off + sd.capT * 4ull);
    sd.oPW = off; off = up256(off + sd.nP * 8ull);
    sd.oPI = off; off = up256(off + sd.nP * 4ull);
  }
  // the filters are read by the probe, the kept records' lists by the resolve after it: one place.  A round
  // keeps about one build record in fifty, and the candidates of one round bound the true matches
  P->listcap = (u32)std::min<double>(kCjListCap, per / 8 + kCjCands + 4096);
  P->oBm = P->oList = off;
  off = up256(off + std::max((u64)phi * kCjWords * 4, 148ull * P->listcap * sizeof(CjKept)));
  P->oCmeta = off; off = up256(off + (u64)P->maxchunks * 8);
  P->oChunkV = off; off = up256(off + (u64)P->maxchunks * kCjChunk * 4);
  P->oChunks = off; off = up256(off + (u64)P->maxchunks * kCjChunk * 8);
  // record pairs that agree mod d and m' by chance, V within one: twice 3 n n' / (phi m') and more
  const double cands = 65536.0 + 6.0 * n_build * n_probe / ((double)phi * mp);
  if (cands > 1e8) return CF_OK;
  P->maxcands = (u32)cands;
  P->oCands = off; off = up256(off + (u64)P->maxcands * 16);
  P->ws_bytes = off;
  P->ok = 1;
  return CF_OK;
} catch (...) {                                    // the lists of divisors did not fit host memory
  cf_set_error("cf_class_plan: out of host memory%s", "");
  return CF_ENOMEM;
}

// Whether a plan was made for these sides, this window and a modulus with odd part m.
bool cf_class_plan_fits(const void* plan, u64 m, int nD, int nI, int r, u64 i_lo, u64 i_n, int swap) {
  const CfClassPlan* P = (const CfClassPlan*)plan;
  if (P->magic != kCjMagic || !P->ok || P->r != (u32)r || P->swap != (u32)(swap != 0) || P->i_lo != i_lo || P->i_n != i_n)
    return false;
  return P->side[P->swap ? 1 : 0].n == (u32)nD && P->side[P->swap ? 0 : 1].n == (u32)nI && P->mp && P->d && m % P->mp == 0 &&
         m % P->d == 0;
}

// Run a planned class join on the stream: equal-residue pairs {D rank, I rank} are appended through
// *npairs (zeroed by the caller).  poolD, poolI: device pool tables (cf_pool_prepare) of the two
// sides, D with the multiplier whose residues mod plan->mp and plan->d are multD_m and multD_d, I
// with multiplier 1; every prime below 2^31.  ws: plan->ws_bytes of device memory, 256-byte
// aligned, used until the call's kernels have run.  *err receives CF_ERR_PART_OVERFLOW when a
// survivor list ran out (repeat the join with cf_dtab_build / cf_fused_probe) and
// CF_ERR_PAIR_OVERFLOW when more than max_pairs pairs were found.
extern "C" int cf_class_join(const void* plan, const void* poolD, const void* poolI, u32 multD_m, u32 multD_d,
                             void* ws, size_t ws_bytes, void* pairs, u32 max_pairs, u32* npairs, u32* err,
                             void* ev_built, void* stream) {
  const CfClassPlan* P = (const CfClassPlan*)plan;
  if (!P || P->magic != kCjMagic || !P->ok || !poolD || !poolI || !ws || ws_bytes < P->ws_bytes ||
      ((uintptr_t)ws & 255u) || (max_pairs && !pairs) || !npairs || !err || multD_m >= P->mp || multD_d >= P->d) {
    cf_set_error("cf_class_join: bad arguments%s", "");
    return CF_EBADARG;
  }
  const cudaStream_t st = (cudaStream_t)stream;
  CjArgs a;
  a.p = *P;
  a.ws = (unsigned char*)ws;
  CjSide& sD = a.p.side[P->swap ? 1 : 0];
  sD.mult_m = multD_m;
  sD.mult_d = multD_d;
  a.pool[0] = (const u64*)(P->swap ? poolI : poolD);
  a.pool[1] = (const u64*)(P->swap ? poolD : poolI);
  a.pairs = (CfPair*)pairs;
  a.npairs = npairs;
  a.err = err;
  a.max_pairs = max_pairs;
  const int smem1 = (int)(kCjWords * 4), smemP = smem1 + kCjWarps * 64 * 8, smem2 = (int)((kCjWords2 + kCjHeads) * 4);
  cudaError_t e = cudaFuncSetAttribute(k_cj_build, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cj_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, smemP);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cj_resolve, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2);
  if (e == cudaSuccess) e = cudaMemsetAsync(ws, 0, P->zero_bytes, st);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_class_join: set-up");
  const unsigned ge = std::min<u32>((P->elems + 255) / 256, 148 * 16);
  k_cj_count<<<std::min<u32>((P->elems / P->run + 256) / 256, 148 * 16), 256, 0, st>>>(a);
  k_cj_rows<<<(4 * P->d * 32 + 255) / 256, 256, 0, st>>>(a);
  k_cj_rowscan<<<1, kCjBlock, 0, st>>>(a);
  k_cj_scatter<<<ge, 256, 0, st>>>(a);
  const unsigned g = std::min<u32>(P->phi, 148);
  k_cj_build<<<g, kCjBlock, smem1, st>>>(a);
  if (ev_built) {
    e = cudaEventRecord((cudaEvent_t)ev_built, st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_class_join: event");
  }
  k_cj_probe<<<148, kCjBlock, smemP, st>>>(a);
  k_cj_resolve<<<g, kCjBlock, smem2, st>>>(a);
  k_cj_emit<<<148 * 4, 128, 0, st>>>(a);
  CF_LAUNCH_CHECK("cf_class_join");
  return CF_OK;
}
