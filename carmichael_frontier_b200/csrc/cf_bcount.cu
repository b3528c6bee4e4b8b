// cf_bcount.cu -- exact sizes of the product-bounded sides, without enumerating their records.
//
// The number of r-subsets I of the ascending pool with prod(I) < Icap, and of r-subsets D of the
// base with prod(D) >= Dmin: the record counts of the reference's filtered sides
// (src/mitm64_idump_stream2.cpp, src/mitm64_ddump.cpp), which a join that finds its pairs another
// way still reports.  The test is A a_x <= H[y] = floor((Icap-1) / a_y) (I), A b_x >= G[y] =
// ceil(Dmin / b_y) (D), the row t = 0 of the bound tables (cf_igen_bounds, cf_ddump_bounds), A the
// product of r - 2 primes; the y inside the bound are those up to some y*, which falls as x rises.
// The D side runs over mirrored indices (largest prime first).
//
// Up to 2^20 (r-2)-subsets, a warp takes one, its lanes the x, and y* is a binary search: every pair
// (subset, x) is its own lane (k = 78, r = 4, 2.6e7 subsets of 159 primes: 16 us).  Beyond, a warp
// takes an (r-3)-subset, its lanes the next index, and each lane walks x up and y* down, O(n) steps
// for up to n^2 / 2 pairs (r = 6, 4.3e9 subsets of 124 primes: 1.24 ms; binary searches 3.0 ms, and
// the walk takes 94 us where the searches take 16).  Both are bound by the issue of 128-bit products
// and compares.
#include "cf_abi_internal.h"

namespace {

struct U128c {
  u64 lo, hi;
};
// a * b, false on a product of 2^128 or more
__device__ __forceinline__ bool mul_fits(U128c a, u64 b, U128c& r) {
  const u64 c = __umul64hi(a.lo, b), t = a.hi * b;
  if (__umul64hi(a.hi, b)) return false;
  r.lo = a.lo * b;
  r.hi = t + c;
  return r.hi >= t;
}
__device__ __forceinline__ bool leq(U128c a, U128c b) { return a.hi < b.hi || (a.hi == b.hi && a.lo <= b.lo); }

template <int SIDE>
__global__ void __launch_bounds__(256)
k_bound_count(const u64* __restrict__ pool, const u64* __restrict__ bounds, int n, int r, int q, u64 nprefix,
              unsigned long long* __restrict__ out) {
  extern __shared__ u64 s[];                        // primes in order of enumeration, then bounds (lo, hi)
  U128c* s_b = (U128c*)(s + ((n + 1) & ~1));
  const u64* pr = pool + cf_pool_off_prime(n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int x = SIDE == 0 ? i : n - 1 - i;
    s[i] = pr[x];
    s_b[i].lo = bounds[2 * x];
    s_b[i].hi = bounds[2 * x + 1];
  }
  __syncthreads();
  const u64* binom = pool + cf_pool_off_binom(n);
  const int lane = threadIdx.x & 31;
  u64 total = 0;
  for (u64 p = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < nprefix;
       p += ((u64)gridDim.x * blockDim.x) >> 5) {
    U128c A{1, 0};
    u64 rank = p;
    int start = 0;
    bool fits = true;
    for (int pos = 0; pos < q; ++pos) {             // the p-th q-subset, and its product
      const int rem = q - pos - 1;
      int c = start;
      if (rem == 0) {
        c = start + (int)rank;
      } else {
        const u64 tot = binom[(size_t)(n - start) * (r + 1) + rem + 1], Y = tot - rank;
        int lo = start, hi = n - 1 - rem;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (binom[(size_t)(n - mid) * (r + 1) + rem + 1] >= Y) lo = mid; else hi = mid - 1;
        }
        c = lo;
        rank -= tot - binom[(size_t)(n - c) * (r + 1) + rem + 1];
      }
      fits = fits && mul_fits(A, s[c], A);
      start = c + 1;
    }
    if (!fits) continue;                            // I: above every bound; D: the caller's products fit
    if (q == r - 2) {
      for (int x0 = start; x0 < n - 1; x0 += 32) {
        const int x = x0 + lane;
        int lo = x;                                 // y* (x: none)
        U128c A2;
        if (x < n - 1 && mul_fits(A, s[x], A2)) {
          int hi = n - 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const bool in = SIDE == 0 ? leq(A2, s_b[mid]) : leq(s_b[mid], A2);
            if (in) lo = mid; else hi = mid - 1;
          }
          total += (u64)(lo - x);
        }
        if (!__any_sync(0xffffffffu, lo > x)) break;   // larger x: none either
      }
    } else {
      for (int w = start + lane; w < n - 2; w += 32) {
        U128c A1;
        if (!mul_fits(A, s[w], A1)) continue;
        int y = n - 1;
        for (int x = w + 1; x < y; ++x) {
          U128c A2;
          if (!mul_fits(A1, s[x], A2)) break;
          if (SIDE == 0) {
            while (y > x && !leq(A2, s_b[y])) --y;
          } else {
            while (y > x && !leq(s_b[y], A2)) --y;
          }
          total += (u64)(y - x);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if (lane == 0 && total) atomicAdd(out, (unsigned long long)total);
}

template <int SIDE>
int launch_bound_count(const void* pool, const void* bounds, int n, int r, int q, u64 nprefix, u64* out, cudaStream_t st) {
  const size_t smem = (size_t)((n + 1) & ~1) * 8 + (size_t)n * 16;
  const u64 g = (nprefix + 7) / 8;
  k_bound_count<SIDE><<<(unsigned)(g < 148 * 16 ? g : 148 * 16), 256, smem, st>>>(
      (const u64*)pool, (const u64*)bounds, n, r, q, nprefix, (unsigned long long*)out);
  CF_LAUNCH_CHECK("cf_bounded_count");
  return CF_OK;
}

}  // namespace

// *out (device, zeroed by the caller) += the number of r-subsets inside the bound: side 0, products
// below the Icap of the cf_igen_bounds table; side 1, products of at least the Dmin of the
// cf_ddump_bounds table, whose r largest primes multiply below 2^128.  pool, bounds: the side's
// device tables for radius r, 3 <= r <= 16, n >= r; at most 2^40 (r-3)-subsets.
extern "C" int cf_bounded_count(int side, const void* pool, const void* bounds, int n, int r, u64* out, void* stream) {
  if ((side != 0 && side != 1) || !pool || !bounds || !out || r < 3 || r > CF_MAX_R || n < r || n > CF_MAX_POOL) {
    cf_set_error("cf_bounded_count: bad arguments%s", "");
    return CF_EBADARG;
  }
  u64 prefixes[2] = {1, 1};                         // (r-2)- and (r-3)-subsets
  for (int k = 0; k < 2; ++k) {
    const int q = r - 2 - k;
    unsigned __int128 c = 1;
    for (int i = 1; i <= q && c; ++i) {
      c = c * (unsigned)(n - q + i) / (unsigned)i;
      if (c >> 62) c = 0;                           // too many
    }
    prefixes[k] = (u64)c;
  }
  // a warp per (r-2)-subset while unranking each is cheap against the rest
  const int k = prefixes[0] && prefixes[0] <= (1u << 20) ? 0 : 1;
  if (!prefixes[k] || prefixes[k] >> 40) { cf_set_error("cf_bounded_count: too many prefixes%s", ""); return CF_EBADARG; }
  return side == 0 ? launch_bound_count<0>(pool, bounds, n, r, r - 2 - k, prefixes[k], out, (cudaStream_t)stream)
                   : launch_bound_count<1>(pool, bounds, n, r, r - 2 - k, prefixes[k], out, (cudaStream_t)stream);
}
