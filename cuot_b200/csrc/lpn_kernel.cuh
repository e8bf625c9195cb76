// lpn_kernel.cuh -- device code of the Ferret primal LPN rows (emp-ot
// LpnF2::__compute4 / __compute1, lpn_f2.h:46-79), shared by the single-
// instance kernel (lpn.cu) and the batched engine (batch.cu).
#pragma once
#include "ctx.cuh"

namespace cuot {
namespace {

struct LpnArgs {
  AesKey key;
  const uint32_t *t0;
  const Blk *kk;
  Blk *e;                 // row `row_lo` of the n-row matrix
  // Dual-role launches (both roles of one extension on this GPU): the second
  // role's kk and rows, XORed with the same public index matrix; else null.
  const Blk *kk2;
  Blk *e2;
  // Both roles' kk, block j of each in 32 bytes (lpn_interleave), or null.
  Blk *kk12;
  int64_t n, k, tail;     // tail: first row handled by the one-row path
  int64_t row_lo;         // first row held in e (a multiple of 4)
  int64_t g0, ngroups;    // 4-row groups [g0, g0 + ngroups)
  int64_t j0, ntail;      // one-row rows [j0, j0 + ntail)
  uint32_t mask;
  int d;
};

constexpr int kLpnThreads = 256;

__device__ __forceinline__ uint32_t lpn_idx(uint32_t w, uint32_t mask, uint32_t k) {
  uint32_t x = w & mask;
  return x >= k ? x - k : x;
}

// Which rows a d = 10 kernel computes: one role's, both roles' from kk and kk2,
// or both from the interleaved kk12 (one 32-byte sector per index then serves
// both; the gathers are what the dual-role kernel waits for).
enum LpnRoles { kOneRole, kTwoRoles, kInterleaved };

// Block j of kk and kk2 side by side.
__device__ __forceinline__ void lpn_interleave(const LpnArgs &a, int64_t j) {
  st_blk(a.kk12 + 2 * j, ldg_blk(a.kk + j));
  st_blk(a.kk12 + 2 * j + 1, ldg_blk(a.kk2 + j));
}
__device__ __forceinline__ void ldg_pair(const Blk *p, Blk &u, Blk &v) {  // 32 bytes, 32-byte aligned
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(u.w[0]), "=r"(u.w[1]), "=r"(u.w[2]), "=r"(u.w[3]), "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3])
      : "l"(p));
}

// Groups [g, g + 6) for d = 10 by a warp: lane 5 s + p takes index blocks 2p and
// 2p + 1 of group g + s, whose terms 8p..8p+7 belong to row 8p / 10 and the
// next one.  Row p - 1 (p > 0) is then this lane's first sum and the lane
// before's second one (for p = 1 its first: that lane has one row only).
// `end`: groups at or above it are left out.  The D plaintexts makeBlock(i, m)
// = {m, 0, i_lo, i_hi} (m < 10) differ only in byte 0, so after AddRoundKey
// they differ only in byte 0 of column 0.  Round 1 reads that byte only for
// output column 0 (ShiftRows keeps row 0 in place); output columns 1..3 and
// three of column 0's four lookups are the same for a lane's two blocks.
// A thread per whole group (round 1 once for ten blocks, 10 x 2 gathers in
// turn) needed a third fewer round-1 lookups but held both roles' eight sums
// (two CTAs per SM) and was slower at every size: 65,536 rows 26.1 / 31.3 us
// (one role / both) against 19.3 / 22.4 here, 470,016 rows 60.6 / 84.1 against
// 49.6 / 66.8, 10,485,760 rows 912 / 1261 against 802 / 1197.
template <LpnRoles ROLES>
__device__ __forceinline__ void lpn_split6(const LpnArgs &a, const TabRef &T, int64_t g, int64_t end) {
  constexpr bool DUAL = ROLES != kOneRole;
  const int lane = threadIdx.x & 31, s = lane / 5, p = lane % 5;
  const int64_t i = 4 * (g + s);
  const bool on = s < 6 && g + s < end;
  const uint32_t k = uint32_t(a.k), mask = a.mask;
  const AesKey &K = a.key;
  Blk acc[2][2];
#pragma unroll
  for (int m = 0; m < 2; m++) acc[m][0] = acc[m][1] = Blk{{0, 0, 0, 0}};
  if (on) {
    const uint32_t s1 = K.rk[1], s2 = uint32_t(uint64_t(i)) ^ K.rk[2], s3 = uint32_t(uint64_t(i) >> 32) ^ K.rk[3];
    const uint32_t s0hi = K.rk[0];
    const uint32_t c1 = round_col(T, s1, s2, s3, s0hi, K.rkr[5]);
    const uint32_t c2 = round_col(T, s2, s3, s0hi, s1, K.rkr[6]);
    const uint32_t c3 = round_col(T, s3, s0hi, s1, s2, K.rkr[7]);
    const uint32_t c0x = t2<2>(T, s2) ^ rotl8(t0<1>(T, s1) ^ t2<3>(T, s3) ^ K.rkr[4]);
    uint32_t x[2][4] = {{t0<0>(T, uint32_t(2 * p) ^ K.rk[0]) ^ c0x, c1, c2, c3},
                        {t0<0>(T, uint32_t(2 * p + 1) ^ K.rk[0]) ^ c0x, c1, c2, c3}};
    aes_enc2_from_round2(T, x[0], x[1], K);
    const int first = p ? 2 * p : 8;  // terms of the first row
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint32_t idx = lpn_idx(x[q / 4][q % 4], mask, k);
      const uint32_t m = q < first ? ~0u : 0u;
      Blk u, v;
      if constexpr (ROLES == kInterleaved) {
        ldg_pair(a.kk12 + 2 * uint64_t(idx), u, v);
      } else {
        u = ldg_blk(a.kk + idx);
        if constexpr (DUAL) v = ldg_blk(a.kk2 + idx);
      }
#pragma unroll
      for (int w = 0; w < 4; w++) {
        acc[0][0].w[w] ^= u.w[w] & m;
        acc[0][1].w[w] ^= u.w[w] & ~m;
      }
      if constexpr (DUAL) {
#pragma unroll
        for (int w = 0; w < 4; w++) {
          acc[1][0].w[w] ^= v.w[w] & m;
          acc[1][1].w[w] ^= v.w[w] & ~m;
        }
      }
    }
  }
  const int64_t at = i - a.row_lo + p - 1;
#pragma unroll
  for (int r = 0; r < (DUAL ? 2 : 1); r++) {
    const Blk give = p == 0 ? acc[r][0] : acc[r][1];
    Blk row = acc[r][0];
#pragma unroll
    for (int w = 0; w < 4; w++) row.w[w] ^= __shfl_up_sync(0xffffffffu, give.w[w], 1);
    Blk *o = (r ? a.e2 : a.e) + at;
    if (on && p) st_blk_cs(o, blk_xor(ld_blk(o), row));
  }
}

// Rows 4g..4g+3 for any d (1..32); the second role too when a.kk2 is set.
__device__ void lpn_group4_dyn(const LpnArgs &a, const TabRef &T, int64_t g) {
  const int64_t i = 4 * g;
  const uint32_t k = uint32_t(a.k), mask = a.mask;
  const bool dual = a.kk2 != nullptr;
  Blk acc[4] = {{{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}};
  Blk acc2[4] = {{{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}};
  const uint32_t ilo = uint32_t(uint64_t(i)), ihi = uint32_t(uint64_t(i) >> 32);
  for (int m = 0; m < a.d; m++) {
    uint32_t x[4] = {uint32_t(m), 0u, ilo, ihi};
    aes_enc(T, x, a.key);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int word = 4 * m + q;
      const uint32_t idx = lpn_idx(x[q], mask, k);
      const Blk v = ldg_blk(a.kk + idx);
      const Blk v2 = dual ? ldg_blk(a.kk2 + idx) : Blk{{0, 0, 0, 0}};
      const int row = word / a.d;
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (r == row) {
          acc[r] = blk_xor(acc[r], v);
          acc2[r] = blk_xor(acc2[r], v2);
        }
    }
  }
#pragma unroll
  for (int m = 0; m < 4; m++) {
    Blk *p = a.e + (i - a.row_lo) + m;
    st_blk_cs(p, blk_xor(ld_blk(p), acc[m]));
    if (dual) {
      Blk *p2 = a.e2 + (i - a.row_lo) + m;
      st_blk_cs(p2, blk_xor(ld_blk(p2), acc2[m]));
    }
  }
}

// One tail row (emp-ot __compute1, lpn_f2.h:61-70); both roles when a.kk2
// is set.
__device__ void lpn_row1(const LpnArgs &a, const TabRef &T, int64_t j) {
  const int nb = (a.d + 3) / 4;
  const uint32_t k = uint32_t(a.k);
  const bool dual = a.kk2 != nullptr;
  const uint32_t jlo = uint32_t(uint64_t(j)), jhi = uint32_t(uint64_t(j) >> 32);
  Blk acc{{0, 0, 0, 0}}, acc2{{0, 0, 0, 0}};
  int done = 0;
  for (int m = 0; m < nb; m++) {
    uint32_t x[4] = {uint32_t(m), 0u, jlo, jhi};
    aes_enc(T, x, a.key);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (done < a.d) {
        acc = blk_xor(acc, ldg_blk(a.kk + (x[q] % k)));
        if (dual) acc2 = blk_xor(acc2, ldg_blk(a.kk2 + (x[q] % k)));
      }
      done++;
    }
  }
  Blk *p = a.e + (j - a.row_lo);
  st_blk(p, blk_xor(ld_blk(p), acc));
  if (dual) {
    Blk *p2 = a.e2 + (j - a.row_lo);
    st_blk(p2, blk_xor(ld_blk(p2), acc2));
  }
}

}  // namespace
}  // namespace cuot
