// cf_sort.cu -- stable LSD onesweep radix sort of (u64 key, u64 id) records and
// the sorted-side merge join: the drop-ins for the reference's sort_side
// (gpu/mitm_gpu2.py:101-104, a stable argsort plus two gathers) and
// join_sorted (gpu/mitm_gpu2.py:107-119).
//
// Sort: one histogram kernel reads every key once and counts all digits of all
// passes; each pass is then ONE kernel (onesweep): a CTA takes the next tile
// ticket, ranks its keys stably in shared memory (per warp, item by item over a
// warp-striped tile, lanes of one digit matched through a shared mask, so equal
// digits keep input order), publishes its per-digit counts, resolves its global
// digit offsets by decoupled look-back over the tiles before it (bounded spin),
// and scatters keys, then ids.  The digit is 8 or 9 bits wide (one width for all
// passes of a sort; the autotuner picks it per size class).  Passes whose digit
// is equal for every key are skipped by the host, so keys below M cost at most
// ceil(log2 M / width) passes.
//
// Merge join: a CTA takes a tile of consecutive sorted I keys, brings the D
// range they can match into shared memory and searches it;
// every I row with at least one equal D key is appended as (row, first D
// position, count) to a compact run list (pairs are rare).  The host expands
// runs into pairs in I-row order, which is join_sorted's output order.
#include <string.h>
#include <type_traits>
#include <vector>
#include "cf_abi_internal.h"

namespace {

using u16 = unsigned short;

constexpr int kSortBlock = 512;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortBlock * kSortItems;  // 4096
constexpr int kWarps = kSortBlock / 32;
constexpr int kMaxPasses = 8;                       // 64 bits at 8 or 9 bits per digit
// Look-back status word of one digit of one tile: flag (aggregate / inclusive) in the top two bits,
// count below.  32-bit words when n < 2^30 (half the status traffic), 64-bit words otherwise.
template <typename SW>
struct Status {
  static constexpr int kBits = (int)sizeof(SW) * 8;
  static constexpr SW kAgg = (SW)1 << (kBits - 2);
  static constexpr SW kInc = (SW)2 << (kBits - 2);
  static constexpr SW kVal = ((SW)1 << (kBits - 2)) - 1;
};
constexpr u32 kSpinLimit = 1u << 24;

// Digit counts of every pass, one read of the keys: hist[p][d] for the digit of
// width db at bit p * db, p < np.  Dynamic shared memory: np << db counters.
__global__ void __launch_bounds__(kSortBlock)
k_sort_hist(const u64* __restrict__ keys, u64 n, u64* __restrict__ hist /*[np][1 << db]*/, int np, int db) {
  extern __shared__ u32 s_h[];
  const int bins = np << db;
  const u64 mask = (1ull << db) - 1;
  for (int i = threadIdx.x; i < bins; i += kSortBlock) s_h[i] = 0;
  __syncthreads();
  for (u64 i = (u64)blockIdx.x * kSortBlock + threadIdx.x; i < n; i += (u64)gridDim.x * kSortBlock) {
    const u64 k = keys[i];
#pragma unroll
    for (int p = 0; p < kMaxPasses; ++p)
      if (p < np) atomicAdd(&s_h[(p << db) + (int)((k >> (p * db)) & mask)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < bins; i += kSortBlock) {
    const u32 v = s_h[i];
    if (v) atomicAdd((unsigned long long*)&hist[i], (unsigned long long)v);
  }
}

// exclusive scan of each pass's histogram of 1 << db bins (one warp per pass)
__global__ void k_sort_hist_scan(const u64* __restrict__ hist, u64* __restrict__ excl, int db) {
  const int p = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bins = 1 << db;
  u64 run = 0;
  for (int c = 0; c < bins; c += 32) {
    const u64 v = hist[p * bins + c + lane];
    u64 incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    excl[p * bins + c + lane] = run + incl - v;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
}

__device__ __forceinline__ u32 lanemask_lt() {
  u32 m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Bulk (TMA) copies of a tile into shared memory, completed on an mbarrier.
__device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(u64* bar, u32 count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(u64* bar, u32 bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// global -> shared, `bytes` a multiple of 16, both addresses 16-byte aligned
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, u32 bytes, u64* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Bounded wait for phase `parity` of an mbarrier; false if the limit ran out.
__device__ __forceinline__ bool mbar_wait(u64* bar, u32 parity, u32 limit) {
  const u32 a = smem_addr(bar);
  for (u32 i = 0; i < limit; ++i) {
    u32 done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Global places of the staged elements j = threadIdx.x + k * kSortBlock (staged element j has
// digit s_dj[j]): computed once per tile and used for the keys and again for the ids.
template <typename Dig>
__device__ __forceinline__ void tile_places(const Dig* s_dj, const u64* s_gbase, int tv, u64 (&dst)[kSortItems]) {
  u32 d[kSortItems];
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const int j = threadIdx.x + k * kSortBlock;
    d[k] = j < tv ? (u32)s_dj[j] : 0u;
  }
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) dst[k] = s_gbase[d[k]] + (u64)(threadIdx.x + k * kSortBlock);
}

// Write a staged tile to its global places, kSortItems elements per thread with their
// shared-memory loads issued together.
__device__ __forceinline__ void write_tile(const u64* s_v, const u64 (&dst)[kSortItems], u64* __restrict__ out,
                                           int tv) {
  u64 v[kSortItems];
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const int j = threadIdx.x + k * kSortBlock;
    v[k] = s_v[j < tv ? j : 0];
  }
#pragma unroll
  for (int k = 0; k < kSortItems; ++k)
    if (threadIdx.x + k * kSortBlock < tv) out[dst[k]] = v[k];
}

constexpr u32 kMbarLimit = 1u << 22;  // try_wait rounds (each suspends for a while) before giving up

// Dynamic shared memory of one pass with DB-bit digits (R = 2^DB bins):
//   tile keys [4096] u64 | tile ids [4096] u64 | warp digit counters [16][R] Cnt |
//   union { peer masks [16][R] u32 (ranking only),
//           staged digits [4096] Dig, gbase [R] u64, dcnt [R] u32, doff [R] u32 (after ranking) }.
// A warp's count of one digit is at most 256 and the exclusive over warps at most 4096, so the
// 9-bit pass keeps its counters in 16 bits; with the union that keeps it at 112 KB, two CTAs per SM.
template <int DB>
struct PassLayout {
  static constexpr int R = 1 << DB;
  using Cnt = typename std::conditional<DB == 8, u32, u16>::type;
  using Dig = typename std::conditional<DB == 8, unsigned char, u16>::type;
  static constexpr size_t kTile = (size_t)kSortTile * 16;
  static constexpr size_t kWc = (size_t)kWarps * R * sizeof(Cnt);
  static constexpr size_t kMm = (size_t)kWarps * R * 4;
  static constexpr size_t kDj = (size_t)kSortTile * sizeof(Dig);
  static constexpr size_t kAfter = kDj + (size_t)R * 16;
  static constexpr size_t kUnion = kMm > kAfter ? kMm : kAfter;
  static constexpr size_t kSmem = kTile + kWc + kUnion;
  static_assert(R <= kSortBlock, "one thread per digit in the scan and look-back");
  static_assert(kWc % 16 == 0 && kDj % 16 == 0, "aligned sub-arrays");
  static_assert(2 * (kSmem + 1024 + 256) <= 233472, "two CTAs per SM");
};

// Control words of the segment sort (below) and its scaled key.
constexpr int kSegLog = 64 * 32;   // pieces of the logarithmic map: 32 per power of two
struct SegCtl {
  u32 cdf[kSegLog + 2];    // f at the start of each piece; the rest is zeroed before the sort:
  u32 full[kSegLog];       // all keys per piece
  u32 hist[kSegLog];       // sampled keys per piece
  u64 scale, max_key;      // from here on also for the sides of k_seg_front
  u64 cap;                 // largest key of kMapNarrow
  u32 top;                 // 2^L NS - 1
  u32 mode;                // f(key), see SegScale
  u32 met;                 // sampled keys that met their equal from another run
  u32 max_seg, err, bail;  // bail: the LSD sort takes these keys, nothing is moved
  u32 blocks_done, pieces_done, tickets[2];
};
// Piece of a key (0 counts as 1) and its place in the piece, 26 bits.
__device__ __forceinline__ u32 seg_piece(u64 key, u32& frac) {
  const u64 k = key ? key : 1ull;
  const int z = __clzll((long long)k);
  const u32 h = (u32)((k << z) >> 32);
  frac = h & 0x3ffffffu;
  return ((u32)(63 - z) << 5) | ((h >> 26) & 31u);
}
// f of a key, monotone, at most top.  (One linear form for narrow keys too, a minimum and a shift more, costs the
// passes 2%: a mode of its own.)
enum { kMapPieces = 0, kMapEven = 1, kMapNarrow = 2 };
struct SegScale {
  u64 s, cap;
  u32 top, mode;
  const u32* cdf;
  __device__ __forceinline__ u32 even(u64 key) const {
    const u64 f = __umul64hi(key, s);
    return f < top ? (u32)f : top;
  }
  __device__ __forceinline__ u32 narrow(u64 key) const { return (u32)((key < cap ? key : cap) * s >> 32); }
  __device__ __forceinline__ u32 operator()(u64 key) const {
    if (mode == kMapEven) return even(key);            // uniform over the launch
    if (mode == kMapNarrow) return narrow(key);
    u32 frac;
    const u32 i = seg_piece(key, frac), c0 = __ldg(cdf + i), c1 = __ldg(cdf + i + 1);
    return (u32)min((u64)c0 + (((u64)(c1 - c0) * frac) >> 26), (u64)top);
  }
};
__device__ __forceinline__ SegScale seg_map(const SegCtl* c) {
  SegScale r;
  r.s = c->scale;
  r.cap = c->cap;
  r.top = c->top;
  r.mode = c->mode;
  r.cdf = c->cdf;
  return r;
}

// One onesweep pass over the DB-bit digit at bit `shift`.  Two CTAs per SM.  BULK:
// the tile's keys and ids are brought into shared memory by two bulk copies at
// the start (every pointer 16-byte aligned), so the id load overlaps the ranking;
// otherwise by plain coalesced loads.  Each item's digit (DB + 1 bits, R = no
// item) rides in the top bits of its local offset.
// MSD: the digit is taken from the scaled key (SegScale) instead of the key.
//
// Bound by the shared-memory pipe (69% busy) and barriers (a quarter of the stalls): about 50
// wavefronts per 32 records for ranking, staging and write-out, DRAM at 32% under the profiler.  Peers
// found by 8 ballots instead of the shared mask: 7% slower; two items ranked at a time: no difference;
// tiles of 2048 records on 256 threads, four CTAs per SM: 5% slower (runs of 64 bytes, twice the status words).
template <int DB, bool BULK, typename SW, bool MSD>
__global__ void __launch_bounds__(kSortBlock, 2)
k_sort_pass(const u64* __restrict__ kin, const u64* __restrict__ iin, u64* __restrict__ kout,
            u64* __restrict__ iout, u64 n, int shift, const SegCtl* __restrict__ scale, const u64* __restrict__ gexcl /*[R]*/,
            SW* __restrict__ status /*[tiles][R]*/, u32* __restrict__ ticket, u32* __restrict__ err) {
  using St = Status<SW>;
  using L = PassLayout<DB>;
  using Cnt = typename L::Cnt;
  using Dig = typename L::Dig;
  constexpr int R = L::R;
  constexpr u32 kNone = (u32)R;
  // predecessor tiles read per look-back round trip: every round reads R status words per tile, so
  // narrow windows win (measured at 2^28 records: 8-bit digits 5 > 4, 6 > 8 > 12; 9-bit 2 > 3, 4 > 8)
  constexpr int kLookWin = DB == 8 ? 5 : 2;
  extern __shared__ __align__(128) unsigned char smem[];
  u64* s_kin = (u64*)smem;                                   // tile keys; later the staging area
  u64* s_iin = s_kin + kSortTile;                            // tile ids
  Cnt* s_wc = (Cnt*)(smem + L::kTile);                       // [kWarps][R] warp digit counts
  unsigned char* s_un = smem + L::kTile + L::kWc;
  u32* s_mm = (u32*)s_un;                                    // [kWarps][R] lanes holding each digit
  Dig* s_dj = (Dig*)s_un;                                    // digit of staged element j
  u64* s_gbase = (u64*)(s_un + L::kDj);  // global position of staged element j of digit d: s_gbase[d] + j
  u32* s_dcnt = (u32*)(s_gbase + R);
  u32* s_doff = s_dcnt + R;
  __shared__ __align__(8) u64 s_bar[2];
  __shared__ u32 s_tile;
  __shared__ u32 s_scan[kWarps];

  if (threadIdx.x == 0) {
    const u32 stop = MSD ? scale->bail : 0u;
    const u32 mine = atomicAdd(ticket, 1u);
    s_tile = stop ? ~0u : mine;
    if (BULK) {
      mbar_init(&s_bar[0], 1);
      mbar_init(&s_bar[1], 1);
      mbar_fence_init();
    }
  }
  __syncthreads();
  SegScale sc{};
  if constexpr (MSD) {
    if (s_tile == ~0u) return;                // uniform, before any copy is started
    sc = seg_map(scale);
  }
  const u32 tile = s_tile;
  const u64 base = (u64)tile * kSortTile;
  const u64 left = n - base;
  const int tv = (int)(left < (u64)kSortTile ? left : (u64)kSortTile);
  if (BULK) {
    if (threadIdx.x == 0) {
      const u32 bytes = (u32)(tv & ~1) * 8u;   // whole 16-byte units; an odd last record is loaded below
      mbar_expect_tx(&s_bar[0], bytes);
      if (bytes) bulk_g2s(s_kin, kin + base, bytes, &s_bar[0]);
      mbar_expect_tx(&s_bar[1], bytes);
      if (bytes) bulk_g2s(s_iin, iin + base, bytes, &s_bar[1]);
      if (tv & 1) {
        s_kin[tv - 1] = kin[base + tv - 1];
        s_iin[tv - 1] = iin[base + tv - 1];
      }
    }
  } else {
    for (int j = threadIdx.x; j < tv; j += kSortBlock) {
      s_kin[j] = kin[base + j];
      s_iin[j] = iin[base + j];
    }
  }
  for (int i = threadIdx.x; i < (int)((L::kWc + L::kMm) / 4); i += kSortBlock)   // counters and masks
    ((u32*)(smem + L::kTile))[i] = 0;
  __syncthreads();
  // A tile whose keys never arrived (both bounded waits ran out, practically unreachable) is
  // ranked as empty: it publishes zero counts, so its successors' look-back still ends and
  // every position they compute stays below n, and it writes nothing.  The error word makes
  // the call return CF_ETIMEOUT.
  bool keys_lost = false;
  if (BULK) {
    bool ok = mbar_wait(&s_bar[0], 0, kMbarLimit);
    if (!ok) {
      atomicOr(err, CF_ERR_SPIN_LIMIT);
      ok = mbar_wait(&s_bar[0], 0, kMbarLimit);
    }
    keys_lost = __syncthreads_or(!ok) != 0;
  }
  const int tr = keys_lost ? 0 : tv;          // items ranked and written
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u64 key[kSortItems];
  u32 loc[kSortItems];                      // local offset (low 16 bits) | digit << 16
  const u32 lt = lanemask_lt();
  Cnt* wc = s_wc + wid * R;
  u32* mm = s_mm + wid * R;
#pragma unroll
  for (int it = 0; it < kSortItems; ++it) {
    const int e = wid * 32 * kSortItems + it * 32 + lane;
    key[it] = e < tr ? s_kin[e] : 0ull;
  }
  // stable rank within the warp, item by item: the lanes of one digit find each other
  // through a shared mask (one atomic OR each), the group's lowest lane takes the
  // group's slice of the warp's digit counter and clears the mask, and the slice's
  // start reaches the group by shuffle
#pragma unroll
  for (int it = 0; it < kSortItems; ++it) {
    const int e = wid * 32 * kSortItems + it * 32 + lane;
    const u64 kd = MSD ? (u64)sc(key[it]) : key[it];
    const u32 d = e < tr ? (u32)((kd >> shift) & (u64)(R - 1)) : kNone;
    const bool valid = d < kNone;
    if (valid) atomicOr(&mm[d], 1u << lane);
    __syncwarp();
    const u32 peers = valid ? mm[d] : 0u;
    const int leader = valid ? __ffs(peers) - 1 : lane;
    __syncwarp();
    u32 base = 0;
    if (valid && lane == leader) {
      base = wc[d];
      wc[d] = (Cnt)(base + __popc(peers));
      mm[d] = 0u;
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    __syncwarp();
    loc[it] = (d << 16) | (base + __popc(peers & lt));
  }
  __syncthreads();
  if (threadIdx.x < R) {                      // per digit: exclusive over warps, tile total
    const int d = threadIdx.x;
    u32 v[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v[w] = s_wc[w * R + d];
    u32 run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      s_wc[w * R + d] = (Cnt)run;
      run += v[w];
    }
    s_dcnt[d] = run;
    // flag and count share one 64-bit word and readers read nothing else that this
    // tile writes, so the status store needs no fence before it
    const SW pub = (tile == 0) ? (St::kInc | (SW)run) : (St::kAgg | (SW)run);
    ((volatile SW*)status)[(u64)tile * R + d] = pub;
    u32 incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_scan[wid] = incl;
    s_doff[d] = incl - run;
  }
  __syncthreads();
  if (threadIdx.x < R) {
    u32 add = 0;
    for (int w = 0; w < wid; ++w) add += s_scan[w];
    s_doff[threadIdx.x] += add;
  }
  __syncthreads();
  // keys and ids are staged before the look-back, while the predecessors publish their counts (2^26
  // records of 61 bits, LSD: 8-bit passes 6.28 -> 6.08 ms, 9-bit 6.54 -> 6.33 against the look-back first
  // and the ids staged after the keys were written)
  {
    u32 add[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const u32 d = loc[it] >> 16;
      add[it] = d < kNone ? s_doff[d] + (u32)wc[d] : 0u;
    }
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const u32 d = loc[it] >> 16;
      if (d < kNone) {
        const u32 l = (loc[it] & 0xffffu) + add[it];
        loc[it] = l | (d << 16);
        s_kin[l] = key[it];
        s_dj[l] = (Dig)d;
      }
    }
  }
  bool lost = keys_lost;
  if (BULK) {
    bool ok = mbar_wait(&s_bar[1], 0, kMbarLimit);
    if (!ok) {
      atomicOr(err, CF_ERR_SPIN_LIMIT);
      ok = mbar_wait(&s_bar[1], 0, kMbarLimit);
    }
    lost |= !ok;
  }
  {
    u64 idv[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const int e = wid * 32 * kSortItems + it * 32 + lane;
      idv[it] = (loc[it] >> 16) < kNone ? s_iin[e] : 0ull;
    }
    lost = __syncthreads_or(lost) != 0;
    if (!lost) {
#pragma unroll
      for (int it = 0; it < kSortItems; ++it)
        if ((loc[it] >> 16) < kNone) s_iin[loc[it] & 0xffffu] = idv[it];
    }
  }
  if (threadIdx.x < R) {
    const int d = threadIdx.x;
    u64 excl = 0;
    if (tile > 0) {
      // decoupled look-back, kLookWin predecessors per round trip, bounded.  Tile 0
      // always publishes an inclusive prefix, so the walk ends at tile 0 at the latest.
      int j = (int)tile - 1;
      u32 spins = 0;
      for (;;) {
        SW v[kLookWin];
#pragma unroll
        for (int w = 0; w < kLookWin; ++w)
          v[w] = (j - w >= 0) ? ((volatile const SW*)status)[(u64)(j - w) * R + d] : St::kInc;
        int used = 0;
        bool stop = false, stall = false;
#pragma unroll
        for (int w = 0; w < kLookWin; ++w) {
          if (stop || stall) continue;
          const SW f = v[w] & (SW)~St::kVal;
          if (f == 0) { stall = true; continue; }
          excl += (u64)(v[w] & St::kVal);
          ++used;
          if (f == St::kInc) stop = true;
        }
        if (stop) break;
        j -= used;
        if (used == 0) {                       // predecessor not published yet: back off briefly
          if (++spins > kSpinLimit) { atomicOr(err, CF_ERR_SPIN_LIMIT); break; }
          __nanosleep(64);
        }
      }
      ((volatile SW*)status)[(u64)tile * R + d] = St::kInc | (SW)(excl + s_dcnt[d]);
    }
    s_gbase[d] = gexcl[d] + excl - s_doff[d];   // wraps mod 2^64; j >= s_doff[d] brings it back
  }
  __syncthreads();
  if (lost) {
    // nothing is written; before the CTA gives up its shared memory, wait (bounded) once
    // more for copies still in flight, so a late copy is unlikely to land in a later CTA's tile
    if (keys_lost) mbar_wait(&s_bar[0], 0, kMbarLimit);
    mbar_wait(&s_bar[1], 0, kMbarLimit);
    return;
  }
  u64 dst[kSortItems];
  tile_places(s_dj, s_gbase, tr, dst);
  write_tile(s_kin, dst, kout, tr);
  write_tile(s_iin, dst, iout, tr);
}

// ---------------------------------------------------------------------------
// Segment sort: the sort of sides whose keys spread over their range (residues do).
//
// An LSD sort moves every record once per digit, 7 or 8 times.  Here the scaled key
//     f = min(mulhi(key, S), 2^L NS - 1),  S = floor(2^(64 + L) NS / (m + 1))
// (monotone in the key, even over the range for m the largest key, whatever its size) is sorted by
// f >> L only, in one or two onesweep passes, which leaves NS segments of about 3,400 records in
// order; each is then sorted in shared memory by one CTA: the low L bits of f are its bin (about
// 0.4 records per bin), one atomic per record gives bin sizes and slots, and a record's place is its
// bin's start plus the records of the bin before it in (key, position) order.  A record moves 32
// bytes per onesweep pass and 32 in the segment sort.
//
// Residues are even over [0, M) once products wrap; the D side's are not (products of few small
// primes stay below M).  The keys are sampled by pieces of their logarithm (32 per power of two),
// and where the sample is not even, all keys are counted by piece and f runs through each piece by the
// piece's share of them.  Even keys below 2^L NS are spread by a factor instead of mulhi.
//
// A segment above kSegCap records (few distinct keys, clusters) leaves the records as
// the passes left them, a stable reordering, and the caller runs the LSD sort on that.  Where the
// sample meets the same key often, the LSD sort, which skips digits that all keys share, is the faster
// one: nothing is moved then (seg_dup_limit).
// ---------------------------------------------------------------------------
constexpr int kSegBlock = 512;
constexpr int kSegItems = 8;
constexpr int kSegCap = kSegBlock * kSegItems;         // 4096 records
constexpr u64 kSegMean = 3400;                         // records per segment: 12 sigma below the capacity
constexpr int kSegBits = 13;                           // L: bins of a segment, log2
constexpr int kSegBins = 1 << kSegBits;
constexpr int kSegBinMax = 32;                         // larger bins: the segment goes to the bitonic sort
constexpr size_t kSegSmem = (size_t)kSegCap * 20 + (size_t)kSegBins * 2;
constexpr u32 kSegFrontMax = 1u << 16;                 // up to here one CTA samples, counts and scans (65,000 records
                                                       // 62 us; 65,537 by three kernels 86)
constexpr u64 kSegMaxN = kSegMean << 18;               // 8.9e8: two 9-bit digits

__device__ __forceinline__ u64 seg_scale(u64 max_key, u32 segs) {   // S of the linear map
  const u64 d = max_key + 1, range = (u64)segs << kSegBits;
  if (d == 0) return range;                            // max = 2^64 - 1
  if (d <= range) return ~0ull;                        // f = key - 1: below the range already
  return (u64)(((unsigned __int128)range << 64) / d);
}

template <int T>
__device__ __forceinline__ u64 block_max(u64 m, u64* s_m) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const u64 x = __shfl_xor_sync(0xffffffffu, m, o);
    m = x > m ? x : m;
  }
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  m = s_m[0];
  for (u32 w = 1; w < T / 32; ++w) m = s_m[w] > m ? s_m[w] : m;
  __syncthreads();
  return m;
}

// Keys that a sample of 1 in `step` (at least 2^19 keys, runs of 32) may have missed above its largest:
// sorted input hides up to 32 * step of them, 2^-14 of the records.
__device__ __forceinline__ u64 seg_reach(u64 max_key, u32 step) {
  const u64 more = step > 1 ? max_key >> 13 : 0;
  return max_key + more < max_key ? ~0ull : max_key + more;
}

// The map of the keys counted in h (shared memory, kSegLog pieces), by one CTA of T threads: linear
// when every piece holds what even keys below the maximum would (within six deviations and a
// twentieth), else (or with `pieces`) piecewise, f rising by a piece's share of the keys over the piece --
// over the part of it below `reach` in the last one, which even keys may fill up to there.
// FRONT: the map also in h (kSegLog + 1 entries) and *sc, for the CTA itself.
template <int T, bool FRONT>
__device__ __forceinline__ void seg_make_map(u32* h, u64 max_key, u64 reach, u32 segs, bool pieces, SegCtl* ctl, u32* s_w,
                                             SegScale* sc) {
  constexpr int P = kSegLog / T;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 c[P], sum = 0;
#pragma unroll
  for (int q = 0; q < P; ++q) sum += c[q] = h[threadIdx.x * P + q];
  u32 incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_w[wid] = incl;
  __syncthreads();
  u32 run = incl - sum, total = 0;
  for (int w = 0; w < T / 32; ++w) {
    if (w < wid) run += s_w[w];
    total += s_w[w];
  }
  const u64 range = (u64)segs << kSegBits;
  const float per = (float)total / ((float)max_key + 1.0f);
  bool even = !pieces;
  u32 unused, over = 0;                                // over: end of the last piece's own range
  const u32 last = seg_piece(reach, unused);
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const u32 i = threadIdx.x * P + q;
    const u64 c0 = (u64)run * range / (total ? total : 1u);
    run += c[q];
    if (i <= last) {
      ctl->cdf[i] = (u32)c0;
      if (FRONT) h[i] = (u32)c0;
    }
    // keys [2^e (1 + j/32), 2^e (1 + (j+1)/32)) cut at the maximum
    const float lo = ldexpf(1.0f + (float)(i & 31u) / 32.0f, (int)(i >> 5)), w = ldexpf(1.0f / 32.0f, (int)(i >> 5));
    if (i == last) {
      const float have = fminf(w, (float)reach + 1.0f - lo);
      const float end = (float)c0 + ((float)range - (float)c0) * (have > 0.0f ? fminf(w / have, 1024.0f) : 1.0f);
      over = end < 4.2e9f ? max((u32)end, (u32)range) : 4200000000u;
    }
    const float e = per * fminf(w, fmaxf(0.0f, (float)max_key + 1.0f - lo));
    even = even && (i < 160u || fabsf((float)c[q] - e) <= 0.05f * e + 6.0f * sqrtf(e) + 16.0f);   // keys below 32: pieces below one key
  }
  const int lin = __syncthreads_and(even);
  if (over) s_w[0] = over;
  __syncthreads();
  over = s_w[0];                                       // the pieces above hold no key, or a few that were not sampled
  for (u32 i = last + 1 + threadIdx.x; i <= (u32)kSegLog; i += T) {
    ctl->cdf[i] = over;
    if (FRONT) h[i] = over;
  }
  if (threadIdx.x == 0) {
    SegScale r{};
    r.mode = !lin ? kMapPieces : reach < range ? kMapNarrow : kMapEven;
    r.s = r.mode == kMapNarrow ? (range << 32) / (reach + 1) : seg_scale(reach, segs);   // (reach + 1) s <= 2^32 range
    r.cap = reach;
    r.top = (u32)(range - 1);
    ctl->scale = r.s;
    ctl->cap = r.cap;
    ctl->top = r.top;
    ctl->mode = r.mode;
    if (FRONT) *sc = r;
  }
}

// Sampled keys (one run of 32 of every 32 * step): their maximum, their pieces, and how many met their
// equal from another run in a table of the CTA's last keys; the last CTA makes the map.  (Equal
// keys within a run are not counted: in ordered input every key that occurs twice is beside its equal.)
constexpr u32 kSegSeen = 8192;                         // table entries: 24 bits of hash, 8 of the run
// Records per key from which the LSD sort is taken: equal keys share a bin, where records are compared with one
// another, and make segments uneven (deviation sqrt(3400 (g + 1)) for g records a key).  Segment sort / LSD
// sort, us: 7.6e6 records, g = 4, 50-bit keys 447 / 791, narrow keys 424 / 455; g = 8 974 / 789 and 486 / 454; 2^26
// narrow, g = 4 2946 / 3033, g = 8 3427 / 3008; 2^20 wide, g = 12 184 / 212, g = 16 233 / 214.  Below 2^19 records
// finding out costs what the LSD sort gains (25 us: 3.0e5, g = 32 130 / 108).
__device__ __forceinline__ float seg_dup_limit(u64 n) {
  return n < (1ull << 19) ? 3.0e38f : n < (1ull << 22) ? 12.0f : 7.0f;
}
__global__ void __launch_bounds__(512) k_seg_sample(const u64* __restrict__ keys, u64 n, u32 step, u32 segs, SegCtl* ctl) {
  __shared__ u64 s_m[16];
  __shared__ u32 s_h[kSegLog], s_seen[kSegSeen], s_w[16], s_last, s_met;
  for (int i = threadIdx.x; i < kSegLog; i += 512) s_h[i] = 0;
  for (u32 i = threadIdx.x; i < kSegSeen; i += 512) s_seen[i] = 0;
  if (threadIdx.x == 0) s_met = 0;
  __syncthreads();
  u64 m = 0;
  u32 met = 0;
  const u64 lanes = (u64)gridDim.x * 512;
  for (u64 t = (u64)blockIdx.x * 512 + threadIdx.x;; t += lanes) {
    const u64 i = (t >> 5) * 32 * step + (t & 31);
    if (i >= n) break;
    const u64 k = keys[i];
    m = k > m ? k : m;
    u32 frac;
    atomicAdd(&s_h[seg_piece(k, frac)], 1u);
    const u64 h = (k ^ (k >> 32)) * 0x9E3779B97F4A7C15ull;
    const u32 tag = ((u32)(h >> 19) & 0xffffff00u) | (u32)((t >> 5) & 255u);
    const u32 old = atomicExch(&s_seen[h >> 51], tag);
    met += ((old ^ tag) >> 8) == 0u && ((old ^ tag) & 255u) != 0u;
  }
  if (met) atomicAdd(&s_met, met);
  m = block_max<512>(m, s_m);
  for (int i = threadIdx.x; i < kSegLog; i += 512)
    if (s_h[i]) atomicAdd(&ctl->hist[i], s_h[i]);
  if (threadIdx.x == 0) {
    atomicMax((unsigned long long*)&ctl->max_key, (unsigned long long)m);
    if (s_met) atomicAdd(&ctl->met, s_met);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int i = threadIdx.x; i < kSegLog; i += 512) s_h[i] = __ldcg(&ctl->hist[i]);
  __syncthreads();
  const u64 max_key = __ldcg(&ctl->max_key);
  seg_make_map<512, false>(s_h, max_key, seg_reach(max_key, step), segs, false, ctl, s_w, nullptr);
  if (threadIdx.x == 0) {
    // a CTA's x table-fulls of keys leave 1 - (1 - e^-x) / x of a table for the average key to meet; of those a
    // key that occurs g times equals g / n
    const float sampled = (float)(n + 32ull * step - 1) / (float)step, x = sampled / gridDim.x / (float)kSegSeen;
    const float seen = (float)kSegSeen * (1.0f - (1.0f - __expf(-x)) / x);
    const float g = (float)__ldcg(&ctl->met) * (float)n / (sampled * seen);
    if (__ldcg(&ctl->met) >= 8u && g > seg_dup_limit(n)) {
      ctl->bail = 1;
      ctl->max_seg = ~0u;
    }
  }
}

// All keys by piece where the sample was not even and thin (above 1.0e7 records: fewer than 340 sampled keys a
// segment; 2^26 records: 50, and pieces of few segments then miss the capacity: products of small primes
// 7.3 ms with the LSD sort behind it, 2.8 so).
__global__ void __launch_bounds__(512) k_seg_pieces(const u64* __restrict__ keys, u64 n, u32 step, u32 segs, SegCtl* ctl) {
  if (ctl->mode != kMapPieces || ctl->bail) return;    // uniform over the launch
  __shared__ u32 s_h[kSegLog], s_w[16], s_last;
  for (int i = threadIdx.x; i < kSegLog; i += 512) s_h[i] = 0;
  __syncthreads();
  constexpr int kU = 8;
  for (u64 i0 = (u64)blockIdx.x * 512 * kU + threadIdx.x; i0 < n; i0 += (u64)gridDim.x * 512 * kU) {
    u64 k[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) k[u] = i0 + u * 512 < n ? keys[i0 + u * 512] : 0ull;
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (i0 + u * 512 >= n) break;
      u32 frac;
      atomicAdd(&s_h[seg_piece(k[u], frac)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kSegLog; i += 512)
    if (s_h[i]) atomicAdd(&ctl->full[i], s_h[i]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ctl->pieces_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int i = threadIdx.x; i < kSegLog; i += 512) s_h[i] = __ldcg(&ctl->full[i]);
  __syncthreads();
  seg_make_map<512, false>(s_h, ctl->max_key, seg_reach(ctl->max_key, step), segs, true, ctl, s_w, nullptr);
}

// Histograms of the one or two digits of f >> L: db low bits, then the rest.
__global__ void __launch_bounds__(512)
k_seg_hist(const u64* __restrict__ keys, u64 n, const SegCtl* __restrict__ ctl, u64* __restrict__ hist, int np, int db) {
  if (ctl->bail) return;                               // uniform over the launch
  __shared__ u32 s_h[2 << 9];
  const int bins = np << db;
  const u32 mask = (1u << db) - 1u;
  for (int i = threadIdx.x; i < bins; i += blockDim.x) s_h[i] = 0;
  const SegScale sc = seg_map(ctl);
  __syncthreads();
  constexpr int kU = 8;                                // loads in flight per thread
  for (u64 i0 = (u64)blockIdx.x * 512 * kU + threadIdx.x; i0 < n; i0 += (u64)gridDim.x * 512 * kU) {
    u64 k[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) k[u] = i0 + u * 512 < n ? keys[i0 + u * 512] : 0ull;
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (i0 + u * 512 >= n) break;
      const u32 v = sc(k[u]) >> kSegBits;
      atomicAdd(&s_h[v & mask], 1u);
      if (np > 1) atomicAdd(&s_h[(1u << db) + (v >> db)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < bins; i += blockDim.x)
    if (s_h[i]) atomicAdd((unsigned long long*)&hist[i], (unsigned long long)s_h[i]);
}

// Up to kSegFrontMax records, one digit (segs <= 256): map, counts, offsets and starts in one CTA.
__global__ void __launch_bounds__(1024, 1)
k_seg_front(const u64* __restrict__ keys, u32 n, u32 segs, SegCtl* __restrict__ ctl, u64* __restrict__ excl,
            u32* __restrict__ starts) {
  __shared__ u64 s_m[32];
  __shared__ u32 s_l[kSegLog + 1], s_h[256], s_w[32];
  __shared__ SegScale s_sc;
  for (int i = threadIdx.x; i < kSegLog; i += 1024) s_l[i] = 0;
  if (threadIdx.x < 256) s_h[threadIdx.x] = 0;
  __syncthreads();
  u64 m = 0;
#pragma unroll 4
  for (u32 i = 4 * (threadIdx.x & ~31u) + (threadIdx.x & 31u); i < n; i += 4096) {   // 32 of every 128 keys
    const u64 k = keys[i];
    m = k > m ? k : m;
    u32 frac;
    atomicAdd(&s_l[seg_piece(k, frac)], 1u);
  }
  m = block_max<1024>(m, s_m);
  seg_make_map<1024, true>(s_l, m, m, segs, false, ctl, s_w, &s_sc);
  __syncthreads();
  const SegScale sc = s_sc;
  bool differ = sc.mode == kMapEven;                   // even over 2^L NS values and more
  if (differ) {
#pragma unroll 8
    for (u32 i = threadIdx.x; i < n; i += 1024) atomicAdd(&s_h[sc.even(keys[i]) >> kSegBits], 1u);
  } else {
    const u64 k0 = keys[0];
#pragma unroll 4
    for (u32 i = threadIdx.x; i < n; i += 1024) {
      const u64 k = keys[i];
      differ = differ || k != k0;
      u32 frac;
      const u32 q = seg_piece(k, frac), c0 = s_l[q], c1 = s_l[q + 1];   // as SegScale, from shared memory
      const u32 f = sc.mode == kMapNarrow ? sc.narrow(k) : (u32)min((u64)c0 + (((u64)(c1 - c0) * frac) >> 26), (u64)sc.top);
      atomicAdd(&s_h[f >> kSegBits], 1u);
    }
  }
  const bool one_key = __syncthreads_or(differ) == 0;  // in order as it is: the pass copies it, no segment is sorted
  const int lane = threadIdx.x & 31;
  u32 v = 0, incl = 0;
  if (threadIdx.x < 256) {
    v = incl = s_h[threadIdx.x];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_w[threadIdx.x >> 5] = incl;
    if (!one_key) atomicMax(&ctl->max_seg, v);
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    u32 add = 0;
    for (u32 w = 0; w < threadIdx.x >> 5; ++w) add += s_w[w];
    excl[threadIdx.x] = add + incl - v;
    if (threadIdx.x <= segs) starts[threadIdx.x] = one_key ? 0u : add + incl - v;
  }
}

// First record of each segment (records ordered by f >> L), and the largest segment.  A warp per
// segment, 32 probes a round: five or six dependent loads (a thread's binary search made 23 to 26 of
// them: 24 us for the 2,243 segments of 7.6e6 records, 9.5 here).
constexpr int kBoundWarps = 8;                         // segments per CTA; one warp more for the last one's end
__global__ void __launch_bounds__((kBoundWarps + 1) * 32)
k_seg_bounds(const u64* __restrict__ keys, u32 n, u32 segs, SegCtl* __restrict__ ctl, u32* __restrict__ starts) {
  __shared__ u32 s_at[kBoundWarps + 1];
  if (ctl->bail) return;                               // uniform over the launch
  const u32 wid = threadIdx.x >> 5, lane = threadIdx.x & 31, s = blockIdx.x * kBoundWarps + wid;
  const SegScale sc = seg_map(ctl);
  u32 lo = 0, hi = n;                                  // lower bound of segment s
  if (s < segs) {
    while (hi - lo > 32) {
      const u32 step = (hi - lo) / 33 + 1, p = lo + (lane + 1) * step - 1;
      const bool less = p < hi && (sc(keys[p]) >> kSegBits) < s;
      lo += __popc(__ballot_sync(0xffffffffu, less)) * step;
      hi = min(hi, lo + step - 1);
    }
    const bool less = lo + lane < hi && (sc(keys[lo + lane]) >> kSegBits) < s;
    lo += __popc(__ballot_sync(0xffffffffu, less));
  } else {
    lo = n;
  }
  if (lane == 0) s_at[wid] = lo;
  __syncthreads();
  if (lane == 0 && wid < kBoundWarps && s <= segs) {
    starts[s] = lo;
    if (s < segs) atomicMax(&ctl->max_seg, s_at[wid + 1] - lo);
  }
}

// Sort one segment by (key, position).  Bound by its chain of shared-memory phases, the neighbours'
// comparisons above all: 2^26 records in 0.85 ms, 2.5 TB/s (0.95 ms with half the bins, 1.02 with the
// bins recomputed from the keys); the onesweep pass takes 0.71 ms for the same records and the whole
// sort 2.5 ms (6.28 ms as eight LSD passes).  Two CTAs of 512 threads per SM (98 KB of shared memory, 64
// registers): while one loads or stores, the other ranks.  starts == nullptr: the whole array is one
// segment (n <= kSegCap) and its largest key is found here.
__global__ void __launch_bounds__(kSegBlock, 2)
k_seg_sort(const u64* kin, const u64* iin, u64* kout, u64* iout, u32 n, const SegCtl* __restrict__ ctl,
           const u32* __restrict__ starts) {
  extern __shared__ __align__(16) unsigned char smem[];
  u64* s_key = (u64*)smem;                             // [kSegCap] in bin order
  u64* s_id = s_key + kSegCap;                         // [kSegCap] ids in input order
  u16* s_pos = (u16*)(s_id + kSegCap);                 // [kSegCap] input position of s_key's record
  u16* s_bid = s_pos + kSegCap;                        // [kSegCap] bin of s_key's record
  u32* s_bin = (u32*)(s_bid + kSegCap);                // [kSegBins] sizes, then starts, two 16-bit halves a word
  const u16* s_start = (const u16*)s_bin;
  __shared__ u32 s_w[kSegBlock / 32];
  __shared__ u64 s_m[kSegBlock / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (starts && ctl->max_seg > (u32)kSegCap) return;   // uniform: the caller takes the LSD sort
  const u32 first = starts ? starts[blockIdx.x] : 0u;
  const u32 m = starts ? starts[blockIdx.x + 1] - first : n;
  if (m == 0) return;
  u64 key[kSegItems];
#pragma unroll
  for (int k = 0; k < kSegItems; ++k) {
    const u32 j = threadIdx.x + k * kSegBlock;
    key[k] = j < m ? kin[first + j] : 0ull;
  }
#pragma unroll
  for (int k = 0; k < kSegItems; ++k) {
    const u32 j = threadIdx.x + k * kSegBlock;
    if (j < m) s_id[j] = iin[first + j];
  }
  for (int i = threadIdx.x; i < kSegBins / 2; i += kSegBlock) s_bin[i] = 0;
  SegScale sc{};
  if (starts) {
    sc = seg_map(ctl);
    __syncthreads();
  } else {
    u64 mx = 0;
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) mx = key[k] > mx ? key[k] : mx;
    mx = block_max<kSegBlock>(mx, s_m);
    if (threadIdx.x == 0) s_m[0] = seg_scale(mx, 1u);
    __syncthreads();
    sc.s = s_m[0];
    sc.top = kSegBins - 1u;
    sc.mode = kMapEven;
  }
  u32 bs[kSegItems];                                   // bin << 16 | slot in the bin
#pragma unroll
  for (int k = 0; k < kSegItems; ++k) {
    const u32 j = threadIdx.x + k * kSegBlock;
    const u32 b = sc(key[k]) & (kSegBins - 1u);
    const u32 sh = 16 * (b & 1u);
    bs[k] = j < m ? (b << 16) | ((atomicAdd(&s_bin[b >> 1], 1u << sh) >> sh) & 0xffffu) : 0u;
  }
  __syncthreads();
  // exclusive scan of the bin sizes, 16 bins (8 words) per thread
  constexpr int kPer = kSegBins / 2 / kSegBlock;
  u32 c[kPer], sum = 0, big = 0;
#pragma unroll
  for (int q = 0; q < kPer; q += 4) {
    const uint4 v = *(const uint4*)&s_bin[threadIdx.x * kPer + q];
    c[q] = v.x; c[q + 1] = v.y; c[q + 2] = v.z; c[q + 3] = v.w;
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const u32 lo = c[q] & 0xffffu, hi = c[q] >> 16;
    big = max(big, max(lo, hi));
    sum += lo + hi;
  }
  u32 incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_w[wid] = incl;
  const bool heavy = __syncthreads_or(big > (u32)kSegBinMax) != 0;
  if (!heavy) {
    u32 run = incl - sum;
    for (int w = 0; w < wid; ++w) run += s_w[w];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const u32 lo = c[q] & 0xffffu, hi = c[q] >> 16;
      c[q] = run | ((run + lo) << 16);
      run += lo + hi;
    }
#pragma unroll
    for (int q = 0; q < kPer; q += 4)
      *(uint4*)&s_bin[threadIdx.x * kPer + q] = make_uint4(c[q], c[q + 1], c[q + 2], c[q + 3]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) {
      const u32 j = threadIdx.x + k * kSegBlock;
      if (j < m) {
        const u32 to = s_start[bs[k] >> 16] + (bs[k] & 0xffffu);
        s_key[to] = key[k];
        s_pos[to] = (u16)j;
        s_bid[to] = (u16)(bs[k] >> 16);
      }
    }
    __syncthreads();
    // place q of the bin order: its record moves within its bin only, by the records of the bin
    // that come before it
#pragma unroll
    for (int k = 0; k < kSegItems; ++k) {
      const u32 q = threadIdx.x + k * kSegBlock;
      if (q >= m) continue;
      const u64 kq = s_key[q];
      const u32 pq = s_pos[q], f = s_bid[q];
      u32 to = q;
      for (u32 x = q; x-- > 0;) {
        if (s_bid[x] != f) break;
        const u64 o = s_key[x];
        to -= (o > kq || (o == kq && s_pos[x] > pq)) ? 1u : 0u;
      }
      for (u32 x = q + 1; x < m; ++x) {
        if (s_bid[x] != f) break;
        const u64 o = s_key[x];
        to += (o < kq || (o == kq && s_pos[x] < pq)) ? 1u : 0u;
      }
      kout[first + to] = kq;
      iout[first + to] = s_id[pq];
    }
    return;
  }
  // many records in one bin: bitonic sort of (key, position); the padding (~0, 0xffff) stays last
  u32 p2 = 2;
  while (p2 < m) p2 <<= 1;
#pragma unroll
  for (int k = 0; k < kSegItems; ++k) {
    const u32 j = threadIdx.x + k * kSegBlock;
    if (j < p2) {
      s_key[j] = j < m ? key[k] : ~0ull;
      s_pos[j] = j < m ? (u16)j : (u16)0xffff;
    }
  }
  __syncthreads();
  for (u32 w = 2; w <= p2; w <<= 1)
    for (u32 h = w >> 1; h; h >>= 1) {
      for (u32 t = threadIdx.x; t < p2 / 2; t += kSegBlock) {
        const u32 x = 2 * t - (t & (h - 1)), y = x + h;
        const u64 ka = s_key[x], kb = s_key[y];
        const u16 pa = s_pos[x], pb = s_pos[y];
        const bool gt = ka > kb || (ka == kb && pa > pb);
        if (gt == ((x & w) == 0)) {
          s_key[x] = kb; s_key[y] = ka;
          s_pos[x] = pb; s_pos[y] = pa;
        }
      }
      __syncthreads();
    }
  for (u32 j = threadIdx.x; j < m; j += kSegBlock) {
    kout[first + j] = s_key[j];
    iout[first + j] = s_id[s_pos[j]];
  }
}

// ---------------------------------------------------------------------------
// Merge join of two sorted key arrays.
// ---------------------------------------------------------------------------
constexpr int kMergeBlock = 256;
constexpr int kMergeItems = 8;
constexpr int kMergeTile = kMergeBlock * kMergeItems;  // I keys of one CTA
constexpr u32 kMergeD = 4096;                          // D keys of its range that fit shared memory (32 KB)

struct CfRun {
  u64 irow, dlo, cnt;
};

__device__ __forceinline__ u64 lower_bound_u64(const u64* __restrict__ a, u64 lo, u64 hi, u64 key) {
  while (lo < hi) {
    const u64 mid = lo + ((hi - lo) >> 1);
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// First position of a[0, n) whose key is >= key (UPPER: > key), by the whole warp: 32 probes a round.
template <bool UPPER>
__device__ __forceinline__ u64 warp_bound(const u64* __restrict__ a, u64 n, u64 key, int lane) {
  u64 lo = 0, hi = n;                                  // the answer lies in [lo, hi]
  while (hi - lo > 32) {
    const u64 step = (hi - lo) / 33 + 1;
    const u64 p = lo + (u64)(lane + 1) * step - 1;
    const bool less = p < hi && (UPPER ? a[p] <= key : a[p] < key);
    const u32 k = __popc(__ballot_sync(0xffffffffu, less));
    const u64 l2 = lo + (u64)k * step;                 // probes 0..k-1 are before the answer, probe k is not
    hi = min(hi, l2 + step - 1);
    lo = l2;
  }
  const bool less = lo + lane < hi && (UPPER ? a[lo + lane] <= key : a[lo + lane] < key);
  return lo + __popc(__ballot_sync(0xffffffffu, less));
}

// A CTA takes 2048 consecutive I keys: the D range they can match is found by two warp-wide searches
// and brought into shared memory, where each key is searched; keys are read coalesced.  (One thread
// per 16 I keys with its own binary search of all of D was bound by the latency of its chain: 192 us
// for 6.4e5 x 1.0e7 sorted keys, 30 here; reading the I keys takes 13.)
__global__ void __launch_bounds__(kMergeBlock)
k_merge_runs(const u64* __restrict__ Dk, u64 nD, const u64* __restrict__ Ik, u64 nI, CfRun* __restrict__ runs,
             u64 max_runs, unsigned long long* __restrict__ nruns, u64* __restrict__ npairs, u32* __restrict__ err) {
  __shared__ u64 s_d[kMergeD];
  __shared__ u64 s_lo, s_hi;
  const u64 t0 = (u64)blockIdx.x * kMergeTile;
  const u32 tv = (u32)min((u64)kMergeTile, nI - t0);
  u64 key[kMergeItems];
#pragma unroll
  for (int k = 0; k < kMergeItems; ++k) {
    const u32 j = threadIdx.x + k * kMergeBlock;
    key[k] = j < tv ? Ik[t0 + j] : 0ull;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid == 0) {
    const u64 v = warp_bound<false>(Dk, nD, Ik[t0], lane);
    if (lane == 0) s_lo = v;
  } else if (wid == 1) {
    const u64 v = warp_bound<true>(Dk, nD, Ik[t0 + tv - 1], lane);
    if (lane == 0) s_hi = v;
  }
  __syncthreads();
  const u64 lo = s_lo, hi = s_hi;
  if (lo >= hi) return;                                // uniform
  const u32 nd = (u32)min(hi - lo, (u64)kMergeD + 1);
  const bool near = nd <= kMergeD;
  if (near)
    for (u32 i = threadIdx.x; i < nd; i += kMergeBlock) s_d[i] = Dk[lo + i];
  __syncthreads();
  u64 local_pairs = 0;
#pragma unroll
  for (int k = 0; k < kMergeItems; ++k) {
    const u32 j = threadIdx.x + k * kMergeBlock;
    if (j >= tv) continue;
    u64 pos, cnt = 0;
    if (near) {
      u32 a = 0, b = nd;
      while (a < b) {
        const u32 mid = (a + b) >> 1;
        if (s_d[mid] < key[k]) a = mid + 1; else b = mid;
      }
      pos = lo + a;
      while (a < nd && s_d[a] == key[k]) { ++a; ++cnt; }
    } else {
      pos = lower_bound_u64(Dk, lo, hi, key[k]);
      while (pos + cnt < hi && Dk[pos + cnt] == key[k]) ++cnt;
    }
    if (cnt) {
      const u64 q = atomicAdd(nruns, 1ull);
      if (q < max_runs) {
        CfRun run;
        run.irow = t0 + j; run.dlo = pos; run.cnt = cnt;
        runs[q] = run;
      } else {
        atomicOr(err, CF_ERR_PAIR_OVERFLOW);
      }
      local_pairs += cnt;
    }
  }
  if (local_pairs) atomicAdd((unsigned long long*)npairs, (unsigned long long)local_pairs);
}

}  // namespace

// Workspace of one sort of n records with np passes of db-bit digits: second
// key/id buffers, histograms, the look-back status words of every pass and the
// tile tickets.
static size_t sort_tmp_bytes(u64 n, int np, int db) {
  const u64 tiles = (n + kSortTile - 1) / kSortTile;
  const u64 bins = (u64)np << db;
  return (size_t)(2 * n * 8) + (size_t)(2 * bins * 8) + (size_t)(tiles * bins * 8) + kMaxPasses * 4 + 64;
}

static int sort_passes(int key_bits, int db) { return (key_bits + db - 1) / db; }

template <int DB, typename SW, bool MSD>
static cudaError_t sort_pass_attrs() {
  cudaError_t e = cudaFuncSetAttribute(k_sort_pass<DB, true, SW, MSD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PassLayout<DB>::kSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sort_pass<DB, false, SW, MSD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)PassLayout<DB>::kSmem);
  return e;
}

template <int DB, typename SW, bool MSD = false>
static void sort_pass_launch(bool bulk, unsigned tiles, cudaStream_t st, const u64* ka, const u64* ia, u64* kb,
                             u64* ib, u64 n, int shift, const u64* excl, SW* status, u32* ticket, u32* errw,
                             const SegCtl* scale = nullptr) {
  if (bulk)
    k_sort_pass<DB, true, SW, MSD><<<tiles, kSortBlock, PassLayout<DB>::kSmem, st>>>(ka, ia, kb, ib, n, shift, scale,
                                                                                     excl, status, ticket, errw);
  else
    k_sort_pass<DB, false, SW, MSD><<<tiles, kSortBlock, PassLayout<DB>::kSmem, st>>>(ka, ia, kb, ib, n, shift, scale,
                                                                                      excl, status, ticket, errw);
}

template <typename SW>
static cudaError_t sort_passes_attrs(int db) { return db == 8 ? sort_pass_attrs<8, SW, false>() : sort_pass_attrs<9, SW, false>(); }

// The sort behind cf_sort_pairs and cf_sort_pairs_digits: np = ceil(key_bits / db)
// passes of db-bit digits (8 or 9), passes whose digit is constant skipped.
static int sort_pairs(u64* keys, u64* ids, u64 n, int key_bits, int db, void* tmp, size_t tmp_bytes, size_t need,
                      cudaStream_t st) {
  const int np = sort_passes(key_bits, db);
  const int bins = 1 << db;
  const u64 tiles = (n + kSortTile - 1) / kSortTile;
  if (tmp_bytes < need) { cf_set_error("cf_sort_pairs: workspace too small%s", ""); return CF_ENOMEM; }
  unsigned char* w = (unsigned char*)tmp;
  u64* k2 = (u64*)w; w += n * 8;
  u64* i2 = (u64*)w; w += n * 8;
  u64* hist = (u64*)w; w += (size_t)np * bins * 8;
  u64* excl = (u64*)w; w += (size_t)np * bins * 8;
  const bool narrow = n < (1ull << 30);           // 32-bit status words hold every count
  unsigned char* status = w; w += (size_t)np * tiles * bins * 8;   // room for 64-bit words
  u32* tickets = (u32*)w; w += kMaxPasses * 4;
  u32* errw = (u32*)w;
  cudaError_t e = cudaMemsetAsync(hist, 0, (size_t)np * bins * 8, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(status, 0, (size_t)np * tiles * bins * (narrow ? 4 : 8), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(tickets, 0, kMaxPasses * 4 + 4, st);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs: memset");
  const unsigned hgrid = (unsigned)((n + kSortBlock * 8 - 1) / (kSortBlock * 8));
  k_sort_hist<<<hgrid < 2048 ? hgrid : 2048, kSortBlock, (size_t)(np << db) * 4, st>>>(keys, n, hist, np, db);
  k_sort_hist_scan<<<1, 32 * np, 0, st>>>(hist, excl, db);
  CF_LAUNCH_CHECK("cf_sort_pairs: histogram");
  std::vector<u64> hh((size_t)np * bins);
  e = cudaMemcpyAsync(hh.data(), hist, hh.size() * 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs: histogram read");
  e = narrow ? sort_passes_attrs<u32>(db) : sort_passes_attrs<u64>(db);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs: smem attribute");
  u64 *ka = keys, *ia = ids, *kb = k2, *ib = i2;
  int done = 0;
  for (int p = 0; p < np; ++p) {
    bool trivial = false;
    for (int d = 0; d < bins; ++d) if (hh[(size_t)p * bins + d] == n) trivial = true;
    if (trivial) continue;
    // bulk copies read 16-byte units from 16-byte boundaries: every tile starts at
    // a multiple of 4096 records, so aligned source arrays suffice
    const bool bulk = ((((uintptr_t)ka) | ((uintptr_t)ia)) & 15u) == 0;
    const u64 pw = (u64)p * tiles * bins;           // this pass's status words
    const u64* pex = excl + p * bins;
    if (narrow) {
      u32* pst = (u32*)status + pw;
      if (db == 8) sort_pass_launch<8, u32>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, 8 * p, pex, pst, tickets + p, errw);
      else sort_pass_launch<9, u32>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, 9 * p, pex, pst, tickets + p, errw);
    } else {
      u64* pst = (u64*)status + pw;
      if (db == 8) sort_pass_launch<8, u64>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, 8 * p, pex, pst, tickets + p, errw);
      else sort_pass_launch<9, u64>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, 9 * p, pex, pst, tickets + p, errw);
    }
    CF_LAUNCH_CHECK("cf_sort_pairs: pass");
    u64* t = ka; ka = kb; kb = t;
    t = ia; ia = ib; ib = t;
    ++done;
  }
  if (done & 1) {      // result sits in the workspace: copy back
    e = cudaMemcpyAsync(keys, ka, n * 8, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ids, ia, n * 8, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs: copy back");
  }
  u32 herr = 0;
  e = cudaMemcpyAsync(&herr, errw, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs: error word");
  if (herr & CF_ERR_SPIN_LIMIT) { cf_set_error("cf_sort_pairs: look-back wait exceeded its limit%s", ""); return CF_ETIMEOUT; }
  return CF_OK;
}

static int sort_args_ok(const u64* keys, const u64* ids, u64 n, int key_bits, const void* tmp, const char* who) {
  if (!keys || !ids || !tmp) { cf_set_error("%s: null buffer", who); return CF_EBADARG; }
  if (key_bits < 1 || key_bits > 64) { cf_set_error("%s: key_bits must be 1..64", who); return CF_EBADARG; }
  if (n > (1ull << 40)) { cf_set_error("%s: n too large", who); return CF_EBADARG; }
  return CF_OK;
}

extern "C" size_t cf_sort_tmp_bytes(u64 n) { return sort_tmp_bytes(n, kMaxPasses, 8); }

// Sort (keys, ids) of length n by key, stably, in place (results end in the
// caller's arrays), 8-bit digits.  key_bits: bits of the largest key (1..64);
// passes whose digit is constant are skipped.  Synchronises the stream once (to
// read the digit histogram).
extern "C" int cf_sort_pairs(u64* keys, u64* ids, u64 n, int key_bits, void* tmp, size_t tmp_bytes, void* stream) {
  if (n <= 1) return CF_OK;
  const int rc = sort_args_ok(keys, ids, n, key_bits, tmp, "cf_sort_pairs");
  if (rc != CF_OK) return rc;
  return sort_pairs(keys, ids, n, key_bits, 8, tmp, tmp_bytes, cf_sort_tmp_bytes(n), (cudaStream_t)stream);
}

// Workspace of cf_sort_pairs_digits; 0 for a digit width other than 8 or 9 or
// key_bits outside 1..64.
extern "C" size_t cf_sort_digits_tmp_bytes(u64 n, int key_bits, int digit_bits) {
  if ((digit_bits != 8 && digit_bits != 9) || key_bits < 1 || key_bits > 64) return 0;
  return sort_tmp_bytes(n, sort_passes(key_bits, digit_bits), digit_bits);
}

// cf_sort_pairs with the digit width chosen by the caller (8 or 9 bits):
// ceil(key_bits / digit_bits) passes, constant-digit passes skipped.  Same
// result for every width.
extern "C" int cf_sort_pairs_digits(u64* keys, u64* ids, u64 n, int key_bits, int digit_bits, void* tmp,
                                    size_t tmp_bytes, void* stream) {
  if (digit_bits != 8 && digit_bits != 9) {
    cf_set_error("cf_sort_pairs_digits: digit_bits must be 8 or 9%s", "");
    return CF_EBADARG;
  }
  if (n <= 1) return CF_OK;
  const int rc = sort_args_ok(keys, ids, n, key_bits, tmp, "cf_sort_pairs_digits");
  if (rc != CF_OK) return rc;
  return sort_pairs(keys, ids, n, key_bits, digit_bits, tmp, tmp_bytes,
                    cf_sort_digits_tmp_bytes(n, key_bits, digit_bits), (cudaStream_t)stream);
}

// Workspace of cf_sort_pairs_to for n records.
extern "C" size_t cf_sort_to_tmp_bytes(u64 n) {
  const size_t lsd = sort_tmp_bytes(n, kMaxPasses, 8), lsd9 = sort_tmp_bytes(n, sort_passes(64, 9), 9);
  return (lsd > lsd9 ? lsd : lsd9) + ((size_t)8 << 18) + 65536;
}

// Stable sort of (kin, iin)[n] by key into (kout, iout), which must not overlap the inputs; the
// inputs are left as they are.  digit_bits (8 or 9): the digit width of the LSD sort that takes the
// sides the segment sort does not (above 8.9e8 records, or a segment above 4096 records).
// Synchronises the stream once at the end (twice where the LSD sort runs).
extern "C" int cf_sort_pairs_to(const u64* kin, const u64* iin, u64* kout, u64* iout, u64 n, int digit_bits, void* tmp,
                                size_t tmp_bytes, void* stream) {
  if (digit_bits != 8 && digit_bits != 9) {
    cf_set_error("cf_sort_pairs_to: digit_bits must be 8 or 9%s", "");
    return CF_EBADARG;
  }
  if (n == 0) return CF_OK;
  if (!kin || !iin || !kout || !iout || !tmp) { cf_set_error("cf_sort_pairs_to: null buffer%s", ""); return CF_EBADARG; }
  if (n > (1ull << 40)) { cf_set_error("cf_sort_pairs_to: n too large%s", ""); return CF_EBADARG; }
  if (tmp_bytes < cf_sort_to_tmp_bytes(n)) { cf_set_error("cf_sort_pairs_to: workspace too small%s", ""); return CF_ENOMEM; }
  const cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaFuncSetAttribute(k_seg_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSegSmem);
  if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs_to: smem attribute");
  if (n <= (u64)kSegCap) {                             // one segment: one launch
    k_seg_sort<<<1, kSegBlock, kSegSmem, st>>>(kin, iin, kout, iout, (u32)n, nullptr, nullptr);
    CF_LAUNCH_CHECK("cf_sort_pairs_to: one segment");
    return cf_cuda_status(cudaStreamSynchronize(st), "cf_sort_pairs_to");
  }
  const u64 *src_k = kin, *src_i = iin;
  if (n <= kSegMaxN) {
    const u32 segs = (u32)((n + kSegMean - 1) / kSegMean);
    const int np = segs <= 512 ? 1 : 2, db = segs <= 256 || (np == 2 && segs <= 65536) ? 8 : 9, bins = 1 << db;
    const bool front = n <= kSegFrontMax;              // segs <= 20
    const u64 tiles = (n + kSortTile - 1) / kSortTile;
    // workspace: second buffers, then the zeroed control words, histograms and status words
    unsigned char* w = (unsigned char*)tmp;
    const size_t side = (size_t)(n + (n & 1)) * 8;     // 16-byte aligned ids for the bulk copies
    u64* k2 = (u64*)w; w += side;
    u64* i2 = (u64*)w; w += side;
    // whole lines of 128 bytes for the status rows (7.6e6 records 359 us with rows across lines, 351)
    SegCtl* ctl = (SegCtl*)(((uintptr_t)w + 255) & ~(uintptr_t)255);
    w = (unsigned char*)ctl + ((sizeof(SegCtl) + 255) & ~(size_t)255);
    unsigned char* zero = front ? (unsigned char*)&ctl->scale : (unsigned char*)ctl->full;
    u32* errw = &ctl->err;
    u64* hist = (u64*)w; w += (size_t)np * bins * 8;
    u32* status = (u32*)w; w += (size_t)np * tiles * bins * 4;
    const size_t zeroed = (size_t)(w - zero);
    u64* excl = (u64*)(((uintptr_t)w + 7) & ~(uintptr_t)7); w = (unsigned char*)(excl + (size_t)np * bins);
    u32* starts = (u32*)w; w += (size_t)4 * segs + 4;
    if ((size_t)(w - (unsigned char*)tmp) > tmp_bytes) { cf_set_error("cf_sort_pairs_to: workspace too small%s", ""); return CF_ENOMEM; }
    e = db == 8 ? sort_pass_attrs<8, u32, true>() : sort_pass_attrs<9, u32, true>();
    if (e == cudaSuccess) e = cudaMemsetAsync(zero, 0, zeroed, st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs_to: set-up");
    const unsigned g = (unsigned)((n + 4095) / 4096), gm = g < 148 * 4 ? g : 148 * 4;
    if (front) {
      k_seg_front<<<1, 1024, 0, st>>>(kin, (u32)n, segs, ctl, excl, starts);
    } else {
      const u32 step = (u32)(n >> 20) + 1;             // 2^19 to 2^20 sampled keys
      k_seg_sample<<<gm < 148 ? gm : 148, 512, 0, st>>>(kin, n, step, segs, ctl);
      if (step > 10) k_seg_pieces<<<148 * 2, 512, 0, st>>>(kin, n, step, segs, ctl);
      k_seg_hist<<<gm, 512, 0, st>>>(kin, n, ctl, hist, np, db);
      k_sort_hist_scan<<<1, 32 * np, 0, st>>>(hist, excl, db);
    }
    for (int p = 0; p < np; ++p) {
      const u64 *ka = p ? k2 : kin, *ia = p ? i2 : iin;
      u64 *kb = p + 1 == np ? kout : k2, *ib = p + 1 == np ? iout : i2;
      const bool bulk = ((((uintptr_t)ka) | ((uintptr_t)ia)) & 15u) == 0;
      const int shift = kSegBits + p * db;
      u32* pst = status + (size_t)p * tiles * bins;
      if (db == 8)
        sort_pass_launch<8, u32, true>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, shift, excl + p * bins, pst,
                                       ctl->tickets + p, errw, ctl);
      else
        sort_pass_launch<9, u32, true>(bulk, (unsigned)tiles, st, ka, ia, kb, ib, n, shift, excl + p * bins, pst,
                                       ctl->tickets + p, errw, ctl);
    }
    if (!front) k_seg_bounds<<<segs / kBoundWarps + 1, (kBoundWarps + 1) * 32, 0, st>>>(kout, (u32)n, segs, ctl, starts);
    k_seg_sort<<<segs, kSegBlock, kSegSmem, st>>>(kout, iout, kout, iout, (u32)n, ctl, starts);
    CF_LAUNCH_CHECK("cf_sort_pairs_to: segments");
    u32 h[3];                                          // largest segment, error word, no segments at all
    static_assert(offsetof(SegCtl, err) == offsetof(SegCtl, max_seg) + 4 && offsetof(SegCtl, bail) == offsetof(SegCtl, err) + 4,
                  "read together");
    e = cudaMemcpyAsync(h, &ctl->max_seg, 12, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs_to: control words");
    if (h[1] & CF_ERR_SPIN_LIMIT) { cf_set_error("cf_sort_pairs_to: look-back wait exceeded its limit%s", ""); return CF_ETIMEOUT; }
    if (!h[2] && h[0] <= (u32)kSegCap) return CF_OK;
    if (!h[2]) {
      src_k = kout;                                    // ordered by the top bits, equal keys in input order
      src_i = iout;
    }
  }
  if (src_k == kin) {
    e = cudaMemcpyAsync(kout, src_k, n * 8, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(iout, src_i, n * 8, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return cf_cuda_status(e, "cf_sort_pairs_to: copy");
  }
  return sort_pairs(kout, iout, n, 64, digit_bits, tmp, tmp_bytes, sort_tmp_bytes(n, sort_passes(64, digit_bits), digit_bits), st);
}

extern "C" size_t cf_merge_run_bytes(void) { return sizeof(CfRun); }

// Equal-key runs between sorted Dk[nD] and sorted Ik[nI]: runs[k] = (I row, first
// D position, count), unordered; *nruns and *npairs (device u64 counters,
// zeroed by the caller) receive the run and pair totals.
extern "C" int cf_merge_join_runs(const u64* Dk, u64 nD, const u64* Ik, u64 nI, void* runs, u64 max_runs,
                                  u64* nruns, u64* npairs, u32* err, void* stream) {
  if (nD == 0 || nI == 0) return CF_OK;
  if (!Dk || !Ik || !nruns || !npairs || !err || (max_runs && !runs)) {
    cf_set_error("cf_merge_join_runs: null buffer%s", "");
    return CF_EBADARG;
  }
  const u64 grid = (nI + kMergeTile - 1) / kMergeTile;
  if (grid > 0x7fffffffull) { cf_set_error("cf_merge_join_runs: n too large%s", ""); return CF_EBADARG; }
  k_merge_runs<<<(unsigned)grid, kMergeBlock, 0, (cudaStream_t)stream>>>(
      Dk, nD, Ik, nI, (CfRun*)runs, max_runs, (unsigned long long*)nruns, npairs, err);
  CF_LAUNCH_CHECK("cf_merge_join_runs");
  return CF_OK;
}
