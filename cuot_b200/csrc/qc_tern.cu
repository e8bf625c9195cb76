// qc_tern.cu -- exact quasi-cyclic dual LPN of n = 2^e blocks, 14 <= e <= 22,
// by the ternary transform of qc_tern.cuh: out = a * in mod (x^n - 1) for all
// 128 bit planes at once, with blocks read and written as they are (a block
// is the 128 planes' bits of one coefficient, so no bit transpose is needed)
// and XORs only.
//
// Kernels of one dual LPN, between two buffers of P points x L pairs of words
// per 32 planes ([word group][point][part][coefficient]):
//   tern_pass27            pieces of the input -> first pass of every coset
//   tern_pass27 / pass9    the other forward passes
//   tern_inner             per point and 32 planes: the product in R_L, in
//                          shared memory (in place)
//   tern_pass27 / pass9    inverse passes
//   tern_final             pieces -> coefficients mod x^n - 1 (XORed with xor_in)
// Measured on B200, one dual LPN through a plan, the fp64 FFT path against this:
// n = 2^14 35 / 33 us, 2^15 47 / 38, 2^16 65 / 49, 2^17 102 / 69, 2^18 184 / 92,
// 2^19 371 / 169, 2^20 727 / 375, 2^21 1542 / 928, 2^22 3346 / 1946.
#include "ctx.cuh"
#include "qc_tern.cuh"

namespace cuot {
namespace {

struct TernJobs {
  const uint32_t *in[kTernMaxJobs];
  const uint32_t *xor_in[kTernMaxJobs];
  uint32_t *out[kTernMaxJobs];
  const uint32_t *consts[kTernMaxJobs];
};

// sigma of every node of every pass and size (host: for nothing but the upload).
__constant__ TernSigmas c_sigmas = tern_sigmas();

// What a pass reads and writes: src != dst, or the pieces of jobs.in first.
struct PassArgs {
  int e, pass;
  int W;  // word groups: 4 or a caller's 2 or 1 (kFirstSome: jobs.in from the first of them), 1 for the bits of `a`
  const uint32_t *src;
  uint32_t *dst;
  uint64_t job_words;
  TernJobs jobs;
};
enum PassKind { kFirst, kFirstSome, kFirstBits, kForward, kInverse, kLastInverse };
constexpr bool pass_first(PassKind k) { return k == kFirst || k == kFirstSome || k == kFirstBits; }
constexpr bool pass_inverse(PassKind k) { return k == kInverse || k == kLastInverse; }

// Rotation table of a pass in shared memory, and the one of its rotated stores.
template <int L, PassKind KIND>
__device__ __forceinline__ void fill_tables(RotEntry *load, RotEntry *store) {
  for (int i = threadIdx.x; i < kRotEntries; i += blockDim.x) {
    load[i] = pass_first(KIND) ? rot_entry_first(L, i) : rot_entry(L, i, false);
    if (KIND == kLastInverse) store[i] = rot_entry(L, i, true);
  }
}

// The pieces (children) k0 + dk k (k < N) of a butterfly, blocks i0 + 3c (c < 3)
// of residue r.  All words are loaded before the first is touched: the masks
// of the rotations are looked up again afterwards, since holding them would
// halve the loads in flight.
template <int L, int RAD, int N, PassKind KIND>
__device__ __forceinline__ void load_slots(const PassArgs &a, const Butterfly &b, const uint16_t *sigmas,
                                           const uint32_t *src, const RotEntry *tab, int k0, int dk, int i0, int r,
                                           int w, G4 (&f)[N][3]) {
  int ti[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int slot = k0 + dk * k;
    const RotBase rb =
        rot_base<L>(pass_inverse(KIND) ? inv_rotation<L>(b, sigmas, slot) : fwd_rotation<RAD>(b, slot), r);
    ti[k] = rb.i + i0;
    if constexpr (pass_first(KIND)) {
      const int at = (b.piece + slot * b.step) * L + rb.off;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int j = at + tab[ti[k] + 3 * c].x;
        uint32_t x = 0;
        if (j < (1 << a.e)) x = KIND == kFirstBits ? __ldg(&src[j >> 5]) >> (j & 31) : __ldg(&src[j * 4 + w]);
        f[k][c].a = x;
      }
    } else {
      const uint32_t *p = src + (b.first + slot * b.step) * tern_element(L) + rb.off;
#pragma unroll
      for (int c = 0; c < 3; c++) f[k][c] = load_raw(p, tab[ti[k] + 3 * c]);
    }
  }
  asm volatile("" ::: "memory");  // or the compiler keeps the masks of the first lookup
#pragma unroll
  for (int k = 0; k < N; k++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const RotEntry t = tab[ti[k] + 3 * c];
      if constexpr (pass_first(KIND)) {
        const uint32_t x = KIND == kFirstBits ? 0u - (f[k][c].a & 1u) : f[k][c].a;
        f[k][c] = G4{x & t.m1, x & t.m2};
      } else {
        f[k][c] = load_fix(t, f[k][c]);
      }
    }
}

// A thread's word group w and residue r from its index over both.  The first
// pass reads whole blocks (word groups fastest), the others contiguous words.
struct Lane {
  int w, r;
  bool on;
};
template <int L, PassKind KIND>
__device__ __forceinline__ Lane lane_of(int id, int W) {
  constexpr int B = tern_block(L);
  const Lane l = pass_first(KIND) ? Lane{id % W, id / W, false} : Lane{id / B, id % B, false};
  return Lane{l.w, l.r, l.w < W && l.r < L / 9};
}

// Radix 27: butterfly blockIdx.x, 32 (word group, residue) indices per
// CTA (blockIdx.y), job blockIdx.z.  Nine warps: a warp first takes the 9-point
// DFTs over k1 of one k2 and one coefficient class i0, then the three-point
// ones of one q1; the 243 pairs of every lane change hands in shared memory.
constexpr int kExchangeBytes = 243 * 2 * 32 * 4;
// (CTAs per SM: three leave the other passes 72 registers for their 54 words and
// fewer loads in flight, 34-46 us at 2^20 against 31-41 with two; the first
// pass has 27 words, 27 us against 30)
template <int L, PassKind KIND, bool CHAINED>
__global__ void __launch_bounds__(288, pass_first(KIND) ? 3 : 2) tern_pass27(PassArgs a) {
  constexpr int B = tern_block(L);
  const int W = KIND == kFirst ? 4 : KIND == kFirstBits ? 1 : a.W;
  extern __shared__ uint32_t X[];  // [q1][k2][coefficient][word][lane]
  __shared__ RotEntry tab[kRotEntries], stab[KIND == kLastInverse ? kRotEntries : 1];
  fill_tables<L, KIND>(tab, stab);
  const TernShape s = tern_shape(a.e);
  const uint16_t *sigmas = c_sigmas.v[a.e - kTernMinE];
  const Butterfly b = tern_butterfly(s, sigmas, a.pass, blockIdx.x, pass_inverse(KIND));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Lane ln = lane_of<L, KIND>(blockIdx.y * 32 + lane, W);
  const int w = ln.w, r = ln.r;
  const uint64_t group = uint64_t(tern_points(s)) * tern_element(L);
  const uint64_t at = uint64_t(blockIdx.z) * a.job_words + uint64_t(w) * group;
  __syncthreads();
  const uint32_t zero = chain_begin<CHAINED>();
  {
    const uint32_t *src = pass_first(KIND) ? a.jobs.in[blockIdx.z] + zero : a.src + at + zero;
    const int k2 = warp / 3, i0 = warp % 3;
    G4 f[9][3];
    if (ln.on) {
      load_slots<L, 27, 9, KIND>(a, b, sigmas, src, tab, k2, 3, i0, r, w, f);
      dft<9>(f);
#pragma unroll
      for (int q1 = 0; q1 < 9; q1++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          uint32_t *x = X + ((q1 * 3 + k2) * 9 + i0 + 3 * c) * 64 + lane;
          x[0] = f[dft_slot<9>(q1)][c].a;
          x[32] = f[dft_slot<9>(q1)][c].b;
        }
    }
  }
  __syncthreads();
  if (!ln.on) return;
  const int q1 = warp;
  uint32_t *o[3];
  RotBase rb[3];
#pragma unroll
  for (int q2 = 0; q2 < 3; q2++) {
    const int q = q1 + 9 * q2, k = pass_inverse(KIND) ? (27 - q) % 27 : q;
    rb[q2] = rot_base<L>(KIND == kLastInverse ? fwd_rotation<27>(b, k) : 0, r);
    o[q2] = a.dst + at + (b.first + k * b.step) * tern_element(L) + rb[q2].off;
  }
#pragma unroll
  for (int i = 0; i < 9; i++) {
    G4 y[3];
#pragma unroll
    for (int k2 = 0; k2 < 3; k2++) {
      const int d = i - q1 * k2, wraps = (8 - d) / 9;
      const uint32_t *x = X + ((q1 * 3 + k2) * 9 + d + 9 * wraps) * 64 + lane;
      y[k2] = dft27_twiddle(G4{x[0], x[32]}, wraps);
    }
    dft3(y[0], y[1], y[2]);
#pragma unroll
    for (int q2 = 0; q2 < 3; q2++) {
      if constexpr (KIND == kLastInverse) {
        store_pair(o[q2], stab[rb[q2].i + i], y[q2]);
      } else {
        o[q2][i * B] = y[q2].a;
        o[q2][i * B + tern_part(L)] = y[q2].b;
      }
    }
  }
}

// Radix 9 or 3: a thread holds three blocks' coefficients of all pieces.
template <int L, int RAD, PassKind KIND, bool CHAINED>
__global__ void __launch_bounds__(128, 5) tern_pass9(PassArgs a) {  // 5: all 54 loads in flight (at 80 registers 150 us a pass at 2^22, at 96 125)
  constexpr int B = tern_block(L);
  __shared__ RotEntry tab[kRotEntries];
  fill_tables<L, KIND>(tab, nullptr);
  const TernShape s = tern_shape(a.e);
  const uint16_t *sigmas = c_sigmas.v[a.e - kTernMinE];
  const Butterfly b = tern_butterfly(s, sigmas, a.pass, blockIdx.x, pass_inverse(KIND));
  const int id = blockIdx.y * 128 + threadIdx.x, i0 = id / (a.W * B);
  const Lane ln = lane_of<L, KIND>(id % (a.W * B), a.W);
  __syncthreads();
  const uint32_t zero = chain_begin<CHAINED>();
  if (!ln.on || i0 >= 3) return;
  const uint64_t at = uint64_t(blockIdx.z) * a.job_words + uint64_t(ln.w) * tern_points(s) * tern_element(L);
  G4 f[RAD][3];
  load_slots<L, RAD, RAD, KIND>(a, b, sigmas, a.src + at + zero, tab, 0, 1, i0, ln.r, ln.w, f);
  dft<RAD>(f);
  uint32_t *o = a.dst + at + b.first * tern_element(L) + i0 * B + ln.r;
  const int step = b.step * tern_element(L);
#pragma unroll
  for (int k = 0; k < RAD; k++) {
    const int slot = pass_inverse(KIND) ? idft_slot<RAD>(k) : dft_slot<RAD>(k);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      o[k * step + 3 * c * B] = f[slot][c].a;
      o[k * step + 3 * c * B + tern_part(L)] = f[slot][c].b;
    }
  }
}

// The product in R_L of one point and 32 planes (blockIdx.x: point, y: word
// group, z: job).
// It is bound by the integer pipe (61-63 % busy in ncu), so CTAs are small:
// fewer warps wait at the barriers between steps whose task counts differ, and
// more registers per thread keep more independent XORs in flight.  288 threads
// (one round of leaf products for L = 729) took 60 us at n = 2^18, 245 at 2^20,
// 1268 at 2^22; these sizes 47, 221 and 1038.
template <class S>
constexpr int inner_threads() {
  return S::L == 243 ? 96 : S::L == 1458 ? 256 : 192;
}
template <class S>
constexpr int inner_blocks() {
  return S::L == 243 ? 8 : S::L == 729 ? 5 : S::L == 1458 ? 3 : 2;
}
// Steps 0..2: the element x -> the threads' radix-3 results (below TASK2).
template <class S, int NT>
__device__ __forceinline__ void inner_forward(const uint32_t *x, uint32_t *V, int tid, const Task2 &t2, G4 (&f2)[3][S::G]) {
  static_assert(S::TASK1 <= NT && S::TASK2 <= NT, "one round of butterflies: every load before the first store");
  for (int i = tid; i < S::TASK0; i += NT) p0<S>(x, V, i);
  __syncthreads();
  {
    const Task1 t = task1<S>(tid);
    G4 f[S::R1][3];
    if (tid < S::TASK1) p1_load<S>(V, t, f);
    __syncthreads();
    if (tid < S::TASK1) {
      dft<S::R1>(f);
      p1_store<S>(V, t, f);
    }
  }
  __syncthreads();
  if (tid < S::TASK2) p2_load<S>(V, t2, f2);
  __syncthreads();
}

template <class S, bool CHAINED>
__global__ void __launch_bounds__(inner_threads<S>(), inner_blocks<S>()) tern_inner(uint32_t *buf, uint64_t job_words,
                                                                                   TernJobs jobs) {
  extern __shared__ uint32_t V[];
  constexpr int NT = inner_threads<S>();
  const int tid = threadIdx.x;
  const uint32_t zero = chain_begin<CHAINED>();
  uint32_t *x = buf + zero + uint64_t(blockIdx.z) * job_words +
                (uint64_t(blockIdx.y) * gridDim.x + blockIdx.x) * tern_element(S::L);
  const uint32_t *cs = jobs.consts[blockIdx.z] + zero + uint64_t(blockIdx.x) * kLeafWords * S::LEAVES;
  const Task2 t2 = task2<S>(tid);
  uint32_t next[kLeafWords] = {};
  {
    G4 f[3][S::G];
    inner_forward<S, NT>(x, V, tid, t2, f);
    if (tid < S::LEAVES) {
#pragma unroll
      for (int j = 0; j < kLeafWords; j++) next[j] = __ldg(&cs[j * S::LEAVES + tid]);
    }
    if (tid < S::TASK2) p2_store<S>(V, t2, f);
  }
  __syncthreads();
  // the next product's constants are on their way while this one is computed
  for (int i = tid; i < S::LEAVES; i += NT) {
    uint32_t v[18], w[kLeafWords];
#pragma unroll
    for (int j = 0; j < kLeafWords; j++) {
      w[j] = next[j];
      if (i + NT < S::LEAVES) next[j] = __ldg(&cs[j * S::LEAVES + i + NT]);
    }
#pragma unroll
    for (int j = 0; j < 18; j++) v[j] = V[j * S::SL + i];
    leaf9(v, w);
#pragma unroll
    for (int j = 0; j < 18; j++) V[j * S::SL + i] = v[j];
  }
  __syncthreads();
  {
    G4 f[3][S::G];
    if (tid < S::TASK2) p4_load<S>(V, t2, f);
    __syncthreads();
    if (tid < S::TASK2) p4_store<S>(V, t2, f);
  }
  __syncthreads();
  {
    const Task1 t = task1<S>(tid);
    G4 f[S::R1][3];
    if (tid < S::TASK1) p5_load<S>(V, t, f);
    __syncthreads();
    if (tid < S::TASK1) {
      dft<S::R1>(f);
      p5_store<S>(V, t, f);
    }
  }
  __syncthreads();
  for (int i = tid; i < S::TASK0; i += NT) p6<S>(V, x, i);
}

// The leaf constants of a point of the transform of `a`.
template <class S, bool CHAINED>
__global__ void __launch_bounds__(192) tern_consts(const uint32_t *buf, uint32_t *consts) {
  extern __shared__ uint32_t V[];
  const int tid = threadIdx.x;
  const Task2 t2 = task2<S>(tid);
  const uint32_t zero = chain_begin<CHAINED>();
  {
    G4 f[3][S::G];
    inner_forward<S, 192>(buf + zero + uint64_t(blockIdx.x) * tern_element(S::L), V, tid, t2, f);
    if (tid < S::TASK2) {
#pragma unroll
      for (int q = 0; q < 3; q++)
#pragma unroll
        for (int c = 0; c < S::G; c++) fwd_store<S::LP>(V + (t2.group * 3 + q) * S::ES, t2.r + 9 * c, f[q][c]);
    }
  }
  __syncthreads();
  uint32_t *o = consts + uint64_t(blockIdx.x) * kLeafWords * S::LEAVES, *D = V + S::BASE;
#pragma unroll 1
  for (int h = 0; h < S::E / 5; h++) {
    for (int i = tid; i < S::NE * 53; i += 192) {
      const int el = i / 53, d = i % 53;
      const G4 t = const_top<S>(V + el * S::ES, h, d - 26);
      D[el * S::DIAGS + d] = t.a;
      D[el * S::DIAGS + 53 + d] = t.b;
    }
    __syncthreads();
    for (int i = tid; i < 5 * S::NE; i += 192) {
      // a warp's evaluations are (nearly) one: little divergence between its cases
      const int e1 = i / S::NE, q = i / (2 * S::R1) % 3, group = i % (2 * S::R1);
      const uint32_t *d = D + (group * 3 + q) * S::DIAGS;
      uint32_t w[kLeafWords];
      leaf_consts(Diag{d, d + 53}, e1, w);
      const int id = leaf_id<S>(group, q, 5 * h + e1);
#pragma unroll
      for (int j = 0; j < kLeafWords; j++) o[j * S::LEAVES + id] = w[j];
    }
    __syncthreads();
  }
}

// A thread per coefficient: the word groups' coefficients of a warp are each
// contiguous, and its blocks are written whole.
template <int E, bool CHAINED>
__global__ void __launch_bounds__(256) tern_final(const uint32_t *buf, uint64_t job_words, TernJobs jobs) {
  constexpr TernShape s = tern_shape(E);
  const uint32_t j = blockIdx.x * 256 + threadIdx.x;
  const uint32_t zero = chain_begin<CHAINED>();
  const uint32_t *b = buf + zero + uint64_t(blockIdx.z) * job_words;
  constexpr uint64_t group = uint64_t(tern_points(s)) * tern_element(s.L);
  uint4 v = make_uint4(tern_coefficient<E>(b, j), tern_coefficient<E>(b + group, j), tern_coefficient<E>(b + 2 * group, j),
                       tern_coefficient<E>(b + 3 * group, j));
  const uint4 *xi = reinterpret_cast<const uint4 *>(jobs.xor_in[blockIdx.z]);
  if (xi) {
    const uint4 x = xi[j + zero];
    v = make_uint4(v.x ^ x.x, v.y ^ x.y, v.z ^ x.z, v.w ^ x.w);
  }
  reinterpret_cast<uint4 *>(jobs.out[blockIdx.z])[j] = v;
}

// The same for word groups w0 .. w0 + W - 1 (W = 1 or 2) of a dual LPN that takes them
// in turn: a thread per coefficient and group.
template <int E>
__global__ void __launch_bounds__(256) tern_final_some(const uint32_t *buf, uint64_t job_words, TernJobs jobs, int W,
                                                       int w0) {
  constexpr TernShape s = tern_shape(E);
  constexpr uint64_t group = uint64_t(tern_points(s)) * tern_element(s.L);
  const uint32_t id = blockIdx.x * 256 + threadIdx.x, j = id / W, w = id % W;
  uint32_t v = tern_coefficient<E>(buf + uint64_t(blockIdx.z) * job_words + w * group, j);
  const uint64_t at = uint64_t(j) * 4 + w0 + w;
  if (jobs.xor_in[blockIdx.z]) v ^= jobs.xor_in[blockIdx.z][at];
  jobs.out[blockIdx.z][at] = v;
}

uint64_t group_words(int e) {
  const TernShape s = tern_shape(e);
  return uint64_t(tern_points(s)) * tern_element(s.L);
}

template <typename F>
int set_smem(F fn, int bytes) {
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) return CUOT_OK;
  cudaGetLastError();
  return fail(CUOT_ECUDA, "QC shared-memory attribute failed: %s", cudaGetErrorString(e));
}

// One call's launches: njobs side by side on st, chained or not; W word groups.
struct Run {
  int njobs, W;
  bool chained;
  cudaStream_t st;
};
template <int L, PassKind KIND, bool C>
int pass27(const Run &r, const PassArgs &a) {
  CUOT_TRY(set_smem(tern_pass27<L, KIND, C>, kExchangeBytes));
  const dim3 grid(tern_points(tern_shape(a.e)) / 27, (a.W * tern_block(L) + 31) / 32, r.njobs);
  launch_as(C, tern_pass27<L, KIND, C>, grid, dim3(288), kExchangeBytes, r.st, a);
  return CUOT_OK;
}
template <int L, int RAD, PassKind KIND, bool C>
int pass9(const Run &r, const PassArgs &a) {
  const dim3 grid(tern_points(tern_shape(a.e)) / RAD, (3 * a.W * tern_block(L) + 127) / 128, r.njobs);
  launch_as(C, tern_pass9<L, RAD, KIND, C>, grid, dim3(128), 0, r.st, a);
  return CUOT_OK;
}
// Pass a.pass of the transform (KIND kForward: of the passes after the first).
template <int L, bool C>
int pass_of(const Run &r, const PassArgs &a, PassKind kind) {
  const int rad = tern_radix(tern_shape(a.e).m, a.pass);
  switch (kind) {
    case kFirst: return pass27<L, kFirst, C>(r, a);
    case kFirstSome: return pass27<L, kFirstSome, C>(r, a);
    case kFirstBits: return pass27<L, kFirstBits, C>(r, a);
    case kLastInverse: return pass27<L, kLastInverse, C>(r, a);
    case kForward:
      return rad == 27  ? pass27<L, kForward, C>(r, a)
             : rad == 9 ? pass9<L, 9, kForward, C>(r, a)
                        : pass9<L, 3, kForward, C>(r, a);
    default:
      return rad == 27  ? pass27<L, kInverse, C>(r, a)
             : rad == 9 ? pass9<L, 9, kInverse, C>(r, a)
                        : pass9<L, 3, kInverse, C>(r, a);
  }
}
template <class S, bool C>
int inner_of(const Run &r, int P, uint32_t *buf, uint64_t job_words, const TernJobs &jobs) {
  CUOT_TRY(set_smem(tern_inner<S, C>, S::WORDS * 4));
  launch_as(C, tern_inner<S, C>, dim3(P, r.W, r.njobs), dim3(inner_threads<S>()), S::WORDS * 4, r.st, buf, job_words, jobs);
  return CUOT_OK;
}
template <class S, bool C>
int consts_of(const Run &r, int P, const uint32_t *buf, uint32_t *consts) {
  constexpr int smem = (S::BASE + S::NE * S::DIAGS) * 4;
  CUOT_TRY(set_smem(tern_consts<S, C>, smem));
  launch_as(C, tern_consts<S, C>, dim3(P), dim3(192), smem, r.st, buf, consts);
  return CUOT_OK;
}
// The sizes that are ever chained (kChainBlocks) have L = 243 or 729.
#define TERN_DISPATCH(L_, F, ...)                                                         \
  switch (L_) {                                                                           \
    case 243: return r.chained ? F<TERN_##F(243, 27), true> __VA_ARGS__                   \
                               : F<TERN_##F(243, 27), false> __VA_ARGS__;                 \
    case 729: return r.chained ? F<TERN_##F(729, 27), true> __VA_ARGS__                   \
                               : F<TERN_##F(729, 27), false> __VA_ARGS__;                 \
    case 1458: return F<TERN_##F(1458, 54), false> __VA_ARGS__;                           \
    default: return F<TERN_##F(2187, 81), false> __VA_ARGS__;                             \
  }
#define TERN_pass_of(L, LP) L
#define TERN_inner_of(L, LP) Inner<L, LP>
#define TERN_consts_of(L, LP) Inner<L, LP>
int pass(const Run &r, const PassArgs &a, PassKind kind) {
  TERN_DISPATCH(tern_shape(a.e).L, pass_of, (r, a, kind))
}
int inner(const Run &r, int e, uint32_t *buf, uint64_t job_words, const TernJobs &jobs) {
  const int P = tern_points(tern_shape(e));
  TERN_DISPATCH(tern_shape(e).L, inner_of, (r, P, buf, job_words, jobs))
}
int consts(const Run &r, int e, const uint32_t *buf, uint32_t *out) {
  const int P = tern_points(tern_shape(e));
  TERN_DISPATCH(tern_shape(e).L, consts_of, (r, P, buf, out))
}
#undef TERN_pass_of
#undef TERN_inner_of
#undef TERN_consts_of
#undef TERN_DISPATCH

// Word groups w0 .. w0 + W - 1.
template <int E>
void final_of(const Run &r, const uint32_t *buf, uint64_t job_words, const TernJobs &jobs, int W, int w0) {
  if (W < 4) {
    launch_as(false, tern_final_some<E>, dim3((1u << E) / 256 * W, 1, r.njobs), dim3(256), 0, r.st, buf, job_words,
              jobs, W, w0);
    return;
  }
  constexpr bool kMayChain = (1ull << E) <= kChainBlocks;
  launch_as(kMayChain && r.chained, kMayChain && r.chained ? tern_final<E, kMayChain> : tern_final<E, false>,
            dim3((1u << E) / 256, 1, r.njobs), dim3(256), 0, r.st, buf, job_words, jobs);
}

// Passes first.. of the transform in half[0] (forward; the result's half in *at),
// or back to pass 0.
int passes_on(const Run &r, int e, int from, uint32_t *const half[2], uint64_t job_words, int *at) {
  PassArgs a{e, 0, r.W, nullptr, nullptr, job_words, TernJobs{}};
  for (a.pass = from; a.pass < tern_passes(tern_shape(e).m); a.pass++, *at ^= 1) {
    a.src = half[*at];
    a.dst = half[*at ^ 1];
    CUOT_TRY(pass(r, a, kForward));
  }
  return CUOT_OK;
}
int passes_back(const Run &r, int e, uint32_t *const half[2], uint64_t job_words, int *at) {
  const TernShape s = tern_shape(e);
  PassArgs a{e, 0, r.W, nullptr, nullptr, job_words, TernJobs{}};
  for (a.pass = tern_passes(s.m) - 1; a.pass >= 0; a.pass--, *at ^= 1) {
    a.src = half[*at];
    a.dst = half[*at ^ 1];
    // a single coset's pieces (y^m = 1) need no rotation in the end
    CUOT_TRY(pass(r, a, a.pass || s.cosets == 1 ? kInverse : kLastInverse));
  }
  return CUOT_OK;
}

}  // namespace

bool tern_supported(int e) { return e >= kTernMinE && e <= kTernMaxE; }

uint64_t tern_ahat_bytes(int e) {
  const TernShape s = tern_shape(e);
  return uint64_t(tern_points(s)) * 2 * (s.L / s.Lp) * tern_evals(s.Lp) * kLeafWords * 4;
}

uint64_t tern_build_bytes(int e) { return 2 * group_words(e) * 4; }
uint64_t tern_job_bytes(int e, int groups) { return 2 * group_words(e) * 4 * groups; }

int tern_build_ahat(int e, const uint64_t *a_d, void *scratch, void *ahat, cudaStream_t st) {
  uint32_t *half[2] = {static_cast<uint32_t *>(scratch), static_cast<uint32_t *>(scratch) + group_words(e)};
  const Run r{1, 1, chain_launches(1ull << e, st), st};
  PassArgs a{e, 0, 1, nullptr, half[0], 0, TernJobs{}};
  a.jobs.in[0] = reinterpret_cast<const uint32_t *>(a_d);
  int at = 0;
  CUOT_TRY(pass(r, a, kFirstBits));
  CUOT_TRY(passes_on(r, e, 1, half, 0, &at));
  CUOT_TRY(consts(r, e, half[at], static_cast<uint32_t *>(ahat)));
  return launch_status(1 + tern_passes(tern_shape(e).m));
}

// Word groups w0 .. w0 + W - 1 of the dual LPNs `jobs`, in scratch.
static int tern_groups(int e, const TernJobs &jobs, int njobs, int W, int w0, void *scratch, TernAux *aux,
                       cudaStream_t st) {
  const TernShape s = tern_shape(e);
  const uint64_t group = group_words(e), job_words = group * W;
  uint32_t *half[2] = {static_cast<uint32_t *>(scratch), static_cast<uint32_t *>(scratch) + njobs * job_words};
  const int passes = tern_passes(s.m);
  Run r{njobs, W, chain_launches(uint64_t(njobs) << e, st), st};
  PassArgs first{e, 0, W, nullptr, half[0], job_words, jobs};
  for (int j = 0; j < njobs; j++) first.jobs.in[j] += w0;
  CUOT_TRY(pass(r, first, W == 4 ? kFirst : kFirstSome));
  int at = 0, launches = 2 * passes + 2;
  const int turn = e > 20 ? 1 : 2;
  if (aux && turn < W) {
    // The word groups are independent from here to the end: they alternate
    // between two streams, so that one's kernels fill the other's wave tails
    // and its passes (memory) run beside inner products (integer pipe).  Two
    // groups at a time while a group's kernels are small (2^19: 187 us on one
    // stream, 169 with pairs, 189 one by one; 2^20 386, 375, 377), one by one
    // above (2^21 976, 940, 928; 2^22 2006, 1973, 1946).
    r.W = turn;
    if (cudaEventRecord(aux->ev[0], st) != cudaSuccess || cudaStreamWaitEvent(aux->stream, aux->ev[0], 0) != cudaSuccess)
      return launch_status(1);
    for (int w = 0; w < W; w += r.W) {
      r.st = (w / r.W) & 1 ? aux->stream : st;
      uint32_t *part[2] = {half[0] + w * group, half[1] + w * group};
      at = 0;
      CUOT_TRY(passes_on(r, e, 1, part, job_words, &at));
      CUOT_TRY(inner(r, e, part[at], job_words, jobs));
      CUOT_TRY(passes_back(r, e, part, job_words, &at));
    }
    r.st = st;
    if (cudaEventRecord(aux->ev[1], aux->stream) != cudaSuccess || cudaStreamWaitEvent(st, aux->ev[1], 0) != cudaSuccess)
      return launch_status(1);
    launches += (W / r.W - 1) * 2 * passes;
  } else {
    CUOT_TRY(passes_on(r, e, 1, half, job_words, &at));
    CUOT_TRY(inner(r, e, half[at], job_words, jobs));
    CUOT_TRY(passes_back(r, e, half, job_words, &at));
  }
  switch (e) {
#define TERN_FINAL(E) \
  case E: final_of<E>(r, half[at], job_words, jobs, W, w0); break;
    TERN_FINAL(14) TERN_FINAL(15) TERN_FINAL(16) TERN_FINAL(17) TERN_FINAL(18)
    TERN_FINAL(19) TERN_FINAL(20) TERN_FINAL(21) TERN_FINAL(22)
#undef TERN_FINAL
  }
  return launch_status(launches);
}

int tern_dual(int e, const TernJob *job, int njobs, int groups, void *scratch, TernAux *aux, cudaStream_t st) {
  if (njobs > kTernMaxJobs) return fail(CUOT_EINVAL, "%d dual LPNs in one launch (at most %d)", njobs, kTernMaxJobs);
  TernJobs jobs{};
  for (int j = 0; j < njobs; j++) {
    jobs.in[j] = reinterpret_cast<const uint32_t *>(job[j].in);
    jobs.xor_in[j] = reinterpret_cast<const uint32_t *>(job[j].xor_in);
    jobs.out[j] = reinterpret_cast<uint32_t *>(job[j].out);
    jobs.consts[j] = static_cast<const uint32_t *>(job[j].ahat);
  }
  for (int w0 = 0; w0 < 4; w0 += groups) CUOT_TRY(tern_groups(e, jobs, njobs, groups, w0, scratch, aux, st));
  return CUOT_OK;
}

}  // namespace cuot
