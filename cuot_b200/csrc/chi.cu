// chi.cu -- per-tree chi sums of Ferret's malicious consistency check.
//
// For tree j with seed s_j (the first 16 bytes of Hash(secret_sum_j)), the
// sender's check value is V_j = sum_{i < 2^h} s_j^(i+1) * v_{j,i} over
// GF(2^128), and the receiver computes the same sum W_j over its leaves
// (spcot_sender.h:88-98, spcot_recver.h:97-107: uni_hash_coeff_gen followed
// by vector_inn_prdt_sum_red).  Field: natural bit order (bit i of the
// little-endian block is the coefficient of x^i), reduction polynomial
// x^128 + x^7 + x^2 + x + 1 (emp-tool's gfmul).
//
// B200 has no carry-less multiply, so one CTA per tree turns the sum into
// polynomial evaluations with repeated multipliers:
//   thread j (of 128) runs Horner over its leaves i = j + 128 q with the
//   multiplier u = s^128:  P_j = sum_q v_{j+128q} u^q;
//   warp w (of 4) runs Horner over P_{w+4q} with s^4, and warp 0 over the four
//   results with s, the last product with s included.
// The leaves' products use nibble tables of u in shared memory: u * x = XOR_k
// T[k][nibble k of x], 32 lookups of 16 bytes.  Every entry is held eight
// times, once per group of four banks, and a lane reads the copy of its own
// group: four wavefronts per lookup, where 256-entry byte tables (16 lookups,
// also 64 KiB) met about eleven, and an eighth of the entries to compute.  The
// 128 products of the fold are a warp's each: lane l holds c x^(4l + b), b < 4,
// for the multiplier c and adds those whose bits of x are set; four XOR
// reductions over the warp give the product (bit-serial ones by single
// threads, level by level, took as long as the leaves).
// Bound by the lookups' wavefronts: 32 x 4 per 32 leaves and SM, 145 us for
// 2,507 trees of depth 12.  Measured there 675 -> 178 us (64 trees of depth 10: 45 -> 8).
#include <atomic>

#include "ctx.cuh"

namespace cuot {
namespace {

constexpr int kChiThreads = 128;
constexpr int kChiTableBytes = 32 * 16 * 8 * 16;  // [nibble][value][copy]

struct U128 {
  uint64_t lo, hi;
};

__device__ __forceinline__ U128 u128(const uint4 v) {
  return U128{uint64_t(v.x) | (uint64_t(v.y) << 32), uint64_t(v.z) | (uint64_t(v.w) << 32)};
}
__device__ __forceinline__ uint4 to_u4(U128 a) {
  return make_uint4(uint32_t(a.lo), uint32_t(a.lo >> 32), uint32_t(a.hi), uint32_t(a.hi >> 32));
}
// a * x, reduced (x^128 = x^7 + x^2 + x + 1)
__device__ __forceinline__ U128 mulx(U128 a) {
  const uint64_t c = a.hi >> 63;
  return U128{(a.lo << 1) ^ (c * 0x87ull), (a.hi << 1) | (a.lo >> 63)};
}
// r3:r2:r1:r0 mod x^128 + x^7 + x^2 + x + 1 (the first fold spills at most 7 bits)
__device__ __forceinline__ U128 reduce256(uint64_t r0, uint64_t r1, uint64_t r2, uint64_t r3) {
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const uint64_t h0 = r2, h1 = r3;
    r2 = r3 = 0;
    r0 ^= h0 ^ (h0 << 1) ^ (h0 << 2) ^ (h0 << 7);
    r1 ^= h1 ^ (h1 << 1) ^ (h1 << 2) ^ (h1 << 7) ^ (h0 >> 63) ^ (h0 >> 62) ^ (h0 >> 57);
    r2 ^= (h1 >> 63) ^ (h1 >> 62) ^ (h1 >> 57);
  }
  return U128{r0, r1};
}
// a * x^m, 0 <= m < 128
__device__ __forceinline__ U128 mulxn(U128 a, int m) {
  const int b = m & 63;
  const uint64_t lo = a.lo << b, mid = (a.hi << b) | (b ? a.lo >> (64 - b) : 0), hi = b ? a.hi >> (64 - b) : 0;
  return m < 64 ? reduce256(lo, mid, hi, 0) : reduce256(0, lo, mid, hi);
}
// bits i -> 2i of a 32-bit word
__device__ __forceinline__ uint64_t spread32(uint32_t x) {
  uint64_t v = x;
  v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
  v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
  v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
  v = (v | (v << 2)) & 0x3333333333333333ull;
  v = (v | (v << 1)) & 0x5555555555555555ull;
  return v;
}
// a^2: squaring is GF(2)-linear (bit i -> bit 2i)
__device__ __forceinline__ U128 gsqr(U128 a) {
  return reduce256(spread32(uint32_t(a.lo)), spread32(uint32_t(a.lo >> 32)), spread32(uint32_t(a.hi)),
                   spread32(uint32_t(a.hi >> 32)));
}

// u * x with the nibble tables; T: this lane's copies.
__device__ __forceinline__ U128 tmul(const char *T, const uint4 x) {
  uint4 r = make_uint4(0, 0, 0, 0);
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int k = 0; k < 32; k++) {
    const int sh = 4 * (k & 7);  // nibble at bits 7..10: its entry's offset
    const uint32_t off = (sh > 7 ? w[k >> 3] >> (sh > 7 ? sh - 7 : 0) : w[k >> 3] << (sh > 7 ? 0 : 7 - sh)) & 0x780u;
    const uint4 e = *reinterpret_cast<const uint4 *>(T + k * 2048 + off);
    r.x ^= e.x; r.y ^= e.y; r.z ^= e.z; r.w ^= e.w;
  }
  return u128(r);
}

// A warp's products with a fixed c: lane l holds c x^(4l), ..., c x^(4l + 3).
struct WarpMul {
  uint4 y[4];
  __device__ __forceinline__ WarpMul(U128 c, int lane) {
    U128 v = mulxn(c, 4 * lane);
#pragma unroll
    for (int b = 0; b < 4; b++) {
      y[b] = to_u4(v);
      v = mulx(v);
    }
  }
  // c * x, x and the result in every lane
  __device__ __forceinline__ uint4 operator()(uint4 x, int lane) const {
    const uint32_t lo = lane & 8 ? x.y : x.x, hi = lane & 8 ? x.w : x.z;
    const uint32_t n = (lane & 16 ? hi : lo) >> (4 * (lane & 7));
    uint4 r = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const uint32_t m = 0u - ((n >> b) & 1u);
      r.x ^= y[b].x & m; r.y ^= y[b].y & m; r.z ^= y[b].z & m; r.w ^= y[b].w & m;
    }
    return make_uint4(__reduce_xor_sync(0xffffffffu, r.x), __reduce_xor_sync(0xffffffffu, r.y),
                      __reduce_xor_sync(0xffffffffu, r.z), __reduce_xor_sync(0xffffffffu, r.w));
  }
};
__device__ __forceinline__ uint4 xor4(uint4 a, uint4 b) {
  return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w);
}

template <bool CHAINED>
__global__ void __launch_bounds__(kChiThreads) chi_sum_kernel(const uint4 *__restrict__ leaves, int h,
                                                              const uint4 *__restrict__ seeds,
                                                              uint4 *__restrict__ out) {
  extern __shared__ uint4 T[];       // [32][16][8]
  __shared__ uint4 P[kChiThreads];   // u x^m, then the threads' partial sums
  __shared__ uint4 R[4];
  const int tree = blockIdx.x, j = threadIdx.x, lane = j & 31, warp = j >> 5;
  const int64_t L = int64_t(1) << h, Q = L / kChiThreads;  // leaves per thread (0: some threads have one)
  const uint32_t zero = chain_begin<CHAINED>();
  const uint4 *lv = leaves + tree * L + zero;
  seeds += zero;
  const U128 s = u128(__ldg(&seeds[tree])), s4 = gsqr(gsqr(s));
  uint4 acc = make_uint4(0, 0, 0, 0);
  if (Q > 1) {
    // Leaves are loaded four steps ahead, the first ones beside the table: one step
    // covers L2's latency and not that of memory, which few deep trees have nothing
    // else to hide behind (16 trees of depth 20 4,978 us so, 2,673 four ahead).
    // Chained calls' leaves fit L2: two (one tree of depth 16 162 us, four 184).
    constexpr int kAhead = CHAINED ? 2 : 4;
    uint4 first[kAhead];
    const uint4 *p = lv + j + kChiThreads * (Q - 1);
#pragma unroll
    for (int i = 0; i < kAhead; i++)
      if (i < Q) first[i] = __ldg(p - kChiThreads * i);
    U128 u = s4;
#pragma unroll 1
    for (int l = 0; l < 5; l++) u = gsqr(u);
    P[j] = to_u4(mulxn(u, j));
    __syncthreads();
    // four threads per nibble k: value v = 4 (j % 4) + i, eight copies each
    const int k = j >> 2, v4 = j & 3;
    uint4 base = make_uint4(0, 0, 0, 0);
    if (v4 & 1) base = xor4(base, P[4 * k + 2]);
    if (v4 & 2) base = xor4(base, P[4 * k + 3]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint4 e = base;
      if (i & 1) e = xor4(e, P[4 * k]);
      if (i & 2) e = xor4(e, P[4 * k + 1]);
#pragma unroll
      for (int c = 0; c < 8; c++) T[(k * 16 + 4 * v4 + i) * 8 + ((c + lane) & 7)] = e;
    }
    __syncthreads();
    const char *mine = reinterpret_cast<const char *>(T + (lane & 7));
    if (Q < kAhead) {  // Q = 2
      acc = xor4(to_u4(tmul(mine, first[0])), first[1]);
    } else {
      acc = first[0];
#pragma unroll 1
      for (int64_t q = Q - kAhead; q >= 0; q -= kAhead) {  // leaves q + kAhead - 1 .. q
        uint4 x[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; i++) x[i] = first[i];
        p -= kChiThreads * kAhead;
        if (q) {
#pragma unroll
          for (int i = 0; i < kAhead; i++) first[i] = __ldg(p - kChiThreads * i);
        }
        if (q != Q - kAhead) acc = xor4(to_u4(tmul(mine, acc)), x[0]);
#pragma unroll
        for (int i = 1; i < kAhead; i++) acc = xor4(to_u4(tmul(mine, acc)), x[i]);
      }
    }
  } else if (j < L) {
    acc = __ldg(&lv[j]);
  }
  P[j] = acc;  // (the table's readers of P are past the barrier above)
  __syncthreads();
  {
    const WarpMul mul(s4, lane);
    uint4 r = P[warp + 4 * 31];
#pragma unroll 1
    for (int q = 30; q >= 0; q--) r = xor4(mul(r, lane), P[warp + 4 * q]);
    if (lane == 0) R[warp] = r;
  }
  __syncthreads();
  if (warp == 0) {
    const WarpMul mul(s, lane);
    uint4 r = R[3];
#pragma unroll
    for (int q = 2; q >= 0; q--) r = xor4(mul(r, lane), R[q]);
    r = mul(r, lane);
    if (lane == 0) out[tree] = r;
  }
}

}  // namespace
}  // namespace cuot

using namespace cuot;

extern "C" {

int cuot_ferret_chi_sum(cuot_ctx *ctx, const cuot_block *leaves_d, uint64_t t, int h,
                        const cuot_block *seeds_d, cuot_block *out_d, void *stream) {
  if (!ctx || !leaves_d || !seeds_d || !out_d) return fail(CUOT_EINVAL, "null argument");
  if (t < 1 || t > 0x7fffffffull) return fail(CUOT_EINVAL, "t=%llu out of range", (unsigned long long)t);
  if (h < 1 || h > 30) return fail(CUOT_EINVAL, "h=%d out of range [1,30]", h);
  DeviceGuard g(ctx);
  static std::atomic<bool> attr_set[64];
  const int dev = ctx->device;
  if (dev >= 64 || !attr_set[dev].load()) {
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (cudaFuncSetAttribute(chi_sum_kernel<false>, kAttr, kChiTableBytes) != cudaSuccess ||
        cudaFuncSetAttribute(chi_sum_kernel<true>, kAttr, kChiTableBytes) != cudaSuccess) {
      cudaGetLastError();
      return fail(CUOT_ECUDA, "chi kernel attribute failed");
    }
    if (dev < 64) attr_set[dev].store(true);
  }
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool chained = chain_launches(t << h, st);
  launch_as(chained, chained ? chi_sum_kernel<true> : chi_sum_kernel<false>, dim3((unsigned)t), dim3(kChiThreads),
            kChiTableBytes, st, reinterpret_cast<const uint4 *>(leaves_d), h, reinterpret_cast<const uint4 *>(seeds_d),
            reinterpret_cast<uint4 *>(out_d));
  return launch_status();
}

}  // extern "C"
