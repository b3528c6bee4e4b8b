// cf_check.cuh -- exact check of one candidate (D, I) pair of one modulus
// (shared by the single-modulus and the batched pair-check kernels), one warp per pair.
//
// A pair that passes the size screen costs (n + R)^2 modular products (Korselt) and a 2048-bit
// product of n + R primes; on one thread that is 20 us at 64 primes and 5 ms of a join whose bound
// lets many pairs through (k = 90, r = 5).  Over a warp the Korselt moduli go to the lanes, and the
// product keeps two 32-bit limbs per lane with the carries one step behind (a carry out of a lane is
// added to the next lane's limb before the next factor multiplies it), so a factor is one shuffle.
#pragma once
#include "cf_abi_internal.h"
#include "cf_enum.cuh"

// Limbs 2 * lane and 2 * lane + 1 of a number below 2^2048, with a carry pending on each.
struct CfWarpBig {
  u32 l0, l1, c0, c1;
  bool over;               // lane 31: something carried out of the top
};
__device__ __forceinline__ void cf_big_settle(CfWarpBig& b, int lane) {
  while (__any_sync(0xffffffffu, (b.c0 | b.c1) != 0u)) {
    const u64 s0 = (u64)b.l0 + b.c0;
    const u64 s1 = (u64)b.l1 + b.c1 + (s0 >> 32);
    b.l0 = (u32)s0;
    b.l1 = (u32)s1;
    const u32 out = (u32)(s1 >> 32);
    const u32 in = __shfl_up_sync(0xffffffffu, out, 1);
    b.over |= lane == 31 && out != 0u;
    b.c0 = lane ? in : 0u;
    b.c1 = 0u;
  }
}
__device__ __forceinline__ void cf_big_mul(CfWarpBig& b, u32 q, int lane) {
  if (q >> 31) cf_big_settle(b, lane);            // (limb + carry) * q stays below 2^64 for q < 2^31
  const u64 t0 = ((u64)b.l0 + b.c0) * q, t1 = ((u64)b.l1 + b.c1) * q;
  const u32 out = (u32)(t1 >> 32);
  const u32 in = __shfl_up_sync(0xffffffffu, out, 1);
  b.over |= lane == 31 && out != 0u;
  b.l0 = (u32)t0;
  b.l1 = (u32)t1;
  b.c0 = lane ? in : 0u;
  b.c1 = (u32)(t0 >> 32);
}

// cf_unrank_lex by a warp: 32 candidates of a position at a time.
template <int R>
__device__ __forceinline__ void cf_unrank_warp(u64 rank, int n, const u64* __restrict__ binom, int (&idx)[R], int lane) {
  int start = 0;
#pragma unroll
  for (int pos = 0; pos < R - 1; ++pos) {
    const int rem = R - pos - 1;
    const u64 total = cf_binom(binom, R, n - start, rem + 1), Y = total - rank;
    int lo = start;                               // largest c with C(n-c, rem+1) >= Y
    for (int base = start; base <= n - 1 - rem; base += 32) {
      const int c = base + lane;
      const int k = __popc(__ballot_sync(0xffffffffu, c <= n - 1 - rem && cf_binom(binom, R, n - c, rem + 1) >= Y));
      lo = k ? base + k - 1 : lo;
      if (k < 32) break;
    }
    idx[pos] = lo;
    rank -= total - cf_binom(binom, R, n - lo, rem + 1);
    start = lo + 1;
  }
  idx[R - 1] = start + (int)rank;
}

// x-th prime of S = (B0 without the primes at di) and the primes at ii, x < nD; false: deleted.
template <int R>
__device__ __forceinline__ bool cf_in_base(const int (&di)[R], int x) {
  bool in = true;
#pragma unroll
  for (int j = 0; j < R; ++j) in &= di[j] != x;
  return in;
}

// Check one candidate pair (lexicographic ranks) of one modulus; the whole warp calls it with the
// same pair and every lane gets the result.
template <int R>
__device__ __forceinline__ CfPairResult cf_check_warp(const u64* __restrict__ poolD, const u64* __restrict__ poolI,
                                     const CfScreen* __restrict__ scr, CfPair pr, int lane) {
  const CfPoolHdr* hD = (const CfPoolHdr*)poolD;
  const CfPoolHdr* hI = (const CfPoolHdr*)poolI;
  const int nD = (int)hD->n, nI = (int)hI->n;
  const bool fast = hD->fast32 && hI->fast32;
  CfArithWide wD, wI;
  wD.md = cf_mod_from_hdr(hD);
  wI.md = wD.md;
  const CfMod32 md32 = cf_mod32_from_hdr(hD);
  const u64* bD = poolD + cf_pool_off_binom(nD);
  const u64* bI = poolI + cf_pool_off_binom(nI);
  wD.pk = poolD + cf_pool_off_pkey(nD);
  wI.pk = poolI + cf_pool_off_pkey(nI);
  const u64* pD = poolD + cf_pool_off_prime(nD);
  const u64* pI = poolI + cf_pool_off_prime(nI);
  const double* lD = (const double*)(poolD + cf_pool_off_lg(nD));
  const double* lI = (const double*)(poolI + cf_pool_off_lg(nI));
  CfPairResult out;
  out.flags = 0;
  out.r = R;
  for (int j = 0; j < CF_MAX_R; ++j) { out.d_idx[j] = 0; out.i_idx[j] = 0; }
  int di[R], ii[R];
  cf_unrank_warp<R>(pr.d_id, nD, bD, di, lane);
  cf_unrank_warp<R>(pr.i_id, nI, bI, ii, lane);
  u64 kd, ki;
  if (fast) {
    CfElt32 eD, eI;
    eD.X = hD->X0; eD.x2 = hD->x20;
    eI.X = hI->X0; eI.x2 = hI->x20;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      eD = cf_mul32(eD, (u32)pD[di[j]], md32);
      eI = cf_mul32(eI, (u32)pI[ii[j]], md32);
    }
    kd = cf_key32(eD, md32);
    ki = cf_key32(eI, md32);
  } else {
    kd = cf_subset_key<R>(di, wD, hD->mult_key);
    ki = cf_subset_key<R>(ii, wI, hI->mult_key);
  }
  double lg = scr->lgP0;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    lg += lI[ii[j]] - lD[di[j]];
    out.d_idx[j] = (unsigned short)di[j];
    out.i_idx[j] = (unsigned short)ii[j];
  }
  if (kd == ki) out.flags |= CF_HIT_KEY_EQUAL;
  if (kd == ki && lg <= scr->lgB + scr->eps) {
    out.flags |= CF_HIT_SCREEN;
    // --- distinctness of S = (B0 \ D) u I: D indices are distinct by construction
    //     (strictly increasing), I primes must avoid B0 and each other.
    bool distinct = true;
    for (int j = 0; j < R; ++j) {
      const u64 q = pI[ii[j]];
      for (int x = lane; x < nD; x += 32) distinct &= (pD[x] != q);
      for (int y = 0; y < j; ++y) distinct &= (pI[ii[y]] != q);
    }
    if (__all_sync(0xffffffffu, distinct)) out.flags |= CF_HIT_DISJOINT;
    // --- exact size: n = prod(S) in 32-bit limbs against B
    CfWarpBig n;
    n.l0 = lane == 0 ? 1u : 0u;
    n.l1 = n.c0 = n.c1 = 0u;
    n.over = false;
    for (int x = 0; x < nD + R; ++x) {
      if (x < nD && !cf_in_base<R>(di, x)) continue;
      const u64 q = x < nD ? pD[x] : pI[ii[x - nD]];
      if (q >> 32) { n.over = true; continue; }
      cf_big_mul(n, (u32)q, lane);
    }
    cf_big_settle(n, lane);
    if (!__any_sync(0xffffffffu, n.over)) {
      const u32 b0 = 2 * lane < (int)scr->nlimbs ? scr->limbsB[2 * lane] : 0u;
      const u32 b1 = 2 * lane + 1 < (int)scr->nlimbs ? scr->limbsB[2 * lane + 1] : 0u;
      const u64 v = ((u64)n.l1 << 32) | n.l0, w = ((u64)b1 << 32) | b0;
      const u32 gt = __ballot_sync(0xffffffffu, v > w), lt = __ballot_sync(0xffffffffu, v < w);
      if (gt <= lt) out.flags |= CF_HIT_SIZE_EXACT;   // the highest differing limbs decide
    }
    // --- Korselt: prod(S) == 1 mod (p-1) for every p in S, a prime per lane
    bool korselt = true;
    for (int x0 = 0; x0 < nD + R; x0 += 32) {
      const int x = x0 + lane;
      const bool mine = x < nD + R && (x >= nD || cf_in_base<R>(di, x));
      const u64 mod = mine ? (x < nD ? pD[x] : pI[ii[x - nD]]) - 1 : 1;
      if (mod == 0) korselt = false;
      if (!__all_sync(0xffffffffu, korselt)) break;
      u64 prod = 1 % mod;
      for (int y = 0; y < nD + R; ++y) {
        if (y < nD && !cf_in_base<R>(di, y)) continue;
        const u64 q = y < nD ? pD[y] : pI[ii[y - nD]];
        prod = ((mod | q) >> 32) == 0 ? prod * ((u32)q % (u32)mod) % mod
                                      : (u64)(((unsigned __int128)prod * (q % mod)) % mod);
      }
      korselt = prod == 1 % mod;
      if (!__all_sync(0xffffffffu, korselt)) break;
    }
    if (__all_sync(0xffffffffu, korselt)) out.flags |= CF_HIT_KORSELT;
  }
  return out;
}

