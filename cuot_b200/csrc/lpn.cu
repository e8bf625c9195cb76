// lpn.cu -- Ferret primal LPN and plain AES-128 ECB.
//
// LPN: e[i] ^= XOR_{j<d} kk[idx(i, j)] with emp-ot's index matrix
// (lpn_f2.h:46-79, one task over [0, n)):
//   rows i..i+3 (i % 4 == 0, i < tail): the d blocks makeBlock(i, m), m < d,
//     are AES-encrypted under the seed key; their 4d little-endian u32 words
//     give row i + q/d, term q%d: idx = w & mask, minus k if >= k.
//   rows j >= tail (tail = first multiple of 4 >= n-4): ceil(d/4) blocks
//     makeBlock(j, m), idx = w % k.
// The index AES runs in the same kernel as the gather, so the n*d index
// matrix never touches HBM (cuOT materialises it, dev_layer.cu:171-173).
// kk (k blocks) is read through the read-only path and stays L2-resident.
#include <mutex>

#include "lpn_kernel.cuh"

namespace cuot {

// Any d (a.d), both roles when a.kk2 is set: a thread per 4-row group.
__global__ void __launch_bounds__(kLpnThreads) lpn_kernel(LpnArgs a) {
  extern __shared__ __align__(16) uint32_t smem_tab[];
  stage_table(smem_tab, a.t0);
  __syncthreads();
  const TabRef T{reinterpret_cast<const char *>(smem_tab), uint32_t(threadIdx.x & 31) * 4u};
  const int64_t total = a.ngroups + a.ntail;
  for (int64_t w = int64_t(blockIdx.x) * kLpnThreads + threadIdx.x; w < total;
       w += int64_t(gridDim.x) * kLpnThreads) {
    if (w < a.ngroups) lpn_group4_dyn(a, T, a.g0 + w);
    else lpn_row1(a, T, a.j0 + (w - a.ngroups));
  }
}

// d = 10: five lanes per group (lpn_split6), persistent CTAs.
template <LpnRoles ROLES, bool CHAINED>
__global__ void __launch_bounds__(kLpnThreads, 3) lpn_split_kernel(LpnArgs a) {
  extern __shared__ __align__(16) uint32_t smem_tab[];
  stage_table(smem_tab, a.t0);
  __syncthreads();
  const uint32_t zero = chain_begin<CHAINED>();
  const TabRef T{reinterpret_cast<const char *>(smem_tab), uint32_t(threadIdx.x & 31) * 4u};
  const int64_t warps = int64_t(gridDim.x) * (kLpnThreads / 32), end = a.g0 + a.ngroups;
  const int64_t warp = int64_t(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  for (int64_t g = a.g0 + 6 * warp + zero; g < end; g += 6 * warps) lpn_split6<ROLES>(a, T, g, end);
  if (blockIdx.x == gridDim.x - 1)
    for (int64_t j = threadIdx.x + zero; j < a.ntail; j += kLpnThreads) lpn_row1(a, T, a.j0 + j);
}

__global__ void __launch_bounds__(256) lpn_interleave_kernel(LpnArgs a) {
  for (int64_t j = int64_t(blockIdx.x) * 256 + threadIdx.x; j < a.k; j += int64_t(gridDim.x) * 256) lpn_interleave(a, j);
}

// Plain in-place AES-128 ECB, two blocks per thread.
__global__ void __launch_bounds__(kLpnThreads) ecb_kernel(AesKey key, const uint32_t *t0,
                                                          Blk *io, uint64_t n) {
  extern __shared__ __align__(16) uint32_t smem_tab[];
  stage_table(smem_tab, t0);
  __syncthreads();
  const TabRef T{reinterpret_cast<const char *>(smem_tab), uint32_t(threadIdx.x & 31) * 4u};
  const uint64_t half = (n + 1) / 2;
  for (uint64_t i = uint64_t(blockIdx.x) * kLpnThreads + threadIdx.x; i < half;
       i += uint64_t(gridDim.x) * kLpnThreads) {
    const uint64_t j = i + half;  // second block, keeps both accesses coalesced
    Blk p = ld_blk(io + i);
    uint32_t x[4] = {p.w[0], p.w[1], p.w[2], p.w[3]};
    if (j < n) {
      Blk q = ld_blk(io + j);
      uint32_t y[4] = {q.w[0], q.w[1], q.w[2], q.w[3]};
      aes_enc2(T, x, key, y, key);
      st_blk(io + j, Blk{{y[0], y[1], y[2], y[3]}});
    } else {
      aes_enc(T, x, key);
    }
    st_blk(io + i, Blk{{x[0], x[1], x[2], x[3]}});
  }
}

static int grid_for(cuot_ctx *ctx, const void *fn, int64_t work, int *grid) {
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kLpnThreads, kTableBytes);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  if (per_sm < 1) per_sm = 1;
  int64_t need = (work + kLpnThreads - 1) / kLpnThreads;
  int64_t cap = int64_t(per_sm) * sms * 8;
  *grid = int(need < cap ? (need > 0 ? need : 1) : cap);
  return CUOT_OK;
}

template <typename F>
static int set_smem(F fn) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CUOT_ECUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(e));
  }
  return CUOT_OK;
}

int launch_any(cuot_ctx *ctx, const LpnArgs &a, cudaStream_t st) {
  CUOT_TRY(set_smem(lpn_kernel));
  int grid = 1;
  grid_for(ctx, (const void *)lpn_kernel, a.ngroups + a.ntail, &grid);
  lpn_kernel<<<grid, kLpnThreads, kTableBytes, st>>>(a);
  return launch_status();
}

template <LpnRoles ROLES, bool CHAINED>
int launch_split_as(cuot_ctx *ctx, const LpnArgs &a, cudaStream_t st) {
  CUOT_TRY(set_smem(lpn_split_kernel<ROLES, CHAINED>));
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lpn_split_kernel<ROLES, CHAINED>, kLpnThreads, kTableBytes);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int64_t tasks = (a.ngroups + 5) / 6, cap = int64_t(per_sm < 1 ? 1 : per_sm) * sms;
  launch_as(CHAINED, lpn_split_kernel<ROLES, CHAINED>, dim3(unsigned(tasks < 1 ? 1 : tasks < cap ? tasks : cap)),
            dim3(kLpnThreads), kTableBytes, st, a);
  return launch_status();
}
template <LpnRoles ROLES>
int launch_split(cuot_ctx *ctx, const LpnArgs &a, cudaStream_t st) {
  return chain_launches(uint64_t(a.ngroups) * 4, st) ? launch_split_as<ROLES, true>(ctx, a, st)
                                                     : launch_split_as<ROLES, false>(ctx, a, st);
}

// Memory of its own for one call on `st`, given back to the context's pool in stream
// order: no other call's arena, captured graph or stream holds it.  Null if there is
// none to be had.
static void *pool_alloc(cuot_ctx *ctx, uint64_t bytes, cudaStream_t st) {
  static std::mutex mu;
  // other streams of the program may be under capture, which forbids a plain cudaMalloc
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  void *p = nullptr;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!ctx->pool) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location = {cudaMemLocationTypeDevice, ctx->device};
      uint64_t keep = kPoolKeeps;
      if (cudaMemPoolCreate(&ctx->pool, &props) != cudaSuccess) {
        ctx->pool = nullptr;
        cudaGetLastError();
      } else {
        cudaMemPoolSetAttribute(ctx->pool, cudaMemPoolAttrReleaseThreshold, &keep);
      }
    }
  }
  if (ctx->pool && cudaMallocFromPoolAsync(&p, bytes, ctx->pool, st) != cudaSuccess) {
    p = nullptr;
    cudaGetLastError();
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  return p;
}

// Both roles, d = 10.  From kInterleaveRows rows on, kk and kk2 are first copied
// side by side (470,016 rows 66.8 -> 58.6 us with the copy, 10,485,760 rows 1197 ->
// 927; at 131,072 rows the 3 us that the gathers would save are the copy's launch),
// unless `st` is captured, kk has more than half as many blocks as there are rows
// (262,144 of both: nothing gained), or there is no memory.  Without the copy two arrays of
// more than about 32 MB each fall out of L2 together: one role after the other
// is then faster (10,485,760 rows, k = 1.6 / 2 / 2.6 / 4 million: 1,227 / 1,623 / 2,128 /
// 2,762 us together, 1,602 / 1,602 / 1,603 / 1,758 in turn; copied 950 / 1,058 / 1,224).
constexpr int64_t kInterleaveRows = 1 << 18, kTogether = 2000000;
int launch_dual(cuot_ctx *ctx, LpnArgs a, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) return launch_status(0);
  if (a.ngroups * 4 >= kInterleaveRows && a.k <= 2 * a.ngroups && cap == cudaStreamCaptureStatusNone)
    a.kk12 = static_cast<Blk *>(pool_alloc(ctx, uint64_t(a.k) * 32, st));
  if (a.kk12) {
    const int64_t grid = (a.k + 255) / 256;
    lpn_interleave_kernel<<<unsigned(grid < 148 * 8 ? grid : 148 * 8), 256, 0, st>>>(a);
    int rc = launch_status();
    if (rc == CUOT_OK) rc = launch_split<kInterleaved>(ctx, a, st);
    if (cudaFreeAsync(a.kk12, st) != cudaSuccess && rc == CUOT_OK) rc = launch_status(0);
    return rc;
  }
  if (a.k <= kTogether) return launch_split<kTwoRoles>(ctx, a, st);
  LpnArgs b = a;
  a.kk2 = nullptr;
  a.e2 = nullptr;
  b.kk = b.kk2;
  b.e = b.e2;
  b.kk2 = nullptr;
  b.e2 = nullptr;
  CUOT_TRY(launch_split<kOneRole>(ctx, a, st));
  return launch_split<kOneRole>(ctx, b, st);
}

// Rows [row_lo, row_hi) of one task over [0, n) (lpn_f2.h:72-79), for one
// role (kk2 == e2 == nullptr) or for both roles of one extension.
int lpn_rows(cuot_ctx *ctx, const uint8_t seed[16], const cuot_block *kk_d, const cuot_block *kk2_d,
             int64_t k, int d, cuot_block *e_rows_d, cuot_block *e2_rows_d, int64_t row_lo, int64_t row_hi,
             int64_t n, void *stream) {
  if (k < 1 || k > 0x7fffffffll) return fail(CUOT_EINVAL, "k=%lld out of range", (long long)k);
  if (d < 1 || d > 32) return fail(CUOT_EINVAL, "d=%d out of range [1,32]", d);
  if (n < 0 || row_lo < 0 || row_hi < row_lo || row_hi > n)
    return fail(CUOT_EINVAL, "bad row range [%lld,%lld) of n=%lld", (long long)row_lo,
                (long long)row_hi, (long long)n);
  if (row_lo % 4 || (row_hi % 4 && row_hi != n))
    return fail(CUOT_EINVAL, "row range must start at a multiple of 4 and end at one or at n");
  if (row_hi == row_lo) return CUOT_OK;
  DeviceGuard g(ctx);
  LpnArgs a{};
  host_aes_key_expand(seed, &a.key);
  a.t0 = ctx->t0_d;
  a.kk = reinterpret_cast<const Blk *>(kk_d);
  a.e = reinterpret_cast<Blk *>(e_rows_d);
  a.kk2 = reinterpret_cast<const Blk *>(kk2_d);
  a.e2 = reinterpret_cast<Blk *>(e2_rows_d);
  a.n = n; a.k = k; a.d = d; a.row_lo = row_lo;
  uint32_t mask = 1;
  while (int64_t(mask) < k) mask = (mask << 1) | 1u;  // lpn_f2.h:27-31
  a.mask = mask;
  int64_t tail = 0;
  if (n > 4) tail = ((n - 4) + 3) / 4 * 4;  // lpn_f2.h:75: groups while j < n - 4
  a.tail = tail;
  const int64_t gend = (row_hi < tail ? row_hi : tail);
  a.g0 = row_lo / 4;
  a.ngroups = gend > row_lo ? (gend - row_lo) / 4 : 0;
  a.j0 = row_lo > tail ? row_lo : tail;
  a.ntail = row_hi > a.j0 ? row_hi - a.j0 : 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool dual = kk2_d != nullptr;
  if (d == 10) return dual ? launch_dual(ctx, a, st) : launch_split<kOneRole>(ctx, a, st);
  return launch_any(ctx, a, st);
}

}  // namespace cuot

using namespace cuot;

extern "C" {

int cuot_lpn_primal_dual(cuot_ctx *ctx, const uint8_t seed[16], const cuot_block *kk_send_d,
                         const cuot_block *kk_recv_d, int64_t k, int d, cuot_block *e_send_io_d,
                         cuot_block *e_recv_io_d, int64_t n, void *stream) {
  if (!ctx || !seed || ((!kk_send_d || !kk_recv_d || !e_send_io_d || !e_recv_io_d) && n > 0))
    return fail(CUOT_EINVAL, "null argument");
  if (n > 0 && e_send_io_d == e_recv_io_d) return fail(CUOT_EINVAL, "the two roles' rows must not alias");
  return lpn_rows(ctx, seed, kk_send_d, kk_recv_d, k, d, e_send_io_d, e_recv_io_d, 0, n, n, stream);
}

int cuot_lpn_primal_range(cuot_ctx *ctx, const uint8_t seed[16], const cuot_block *kk_d,
                          int64_t k, int d, cuot_block *e_rows_d, int64_t row_lo, int64_t row_hi,
                          int64_t n, void *stream) {
  if (!ctx || !seed || ((!kk_d || !e_rows_d) && row_hi > row_lo)) return fail(CUOT_EINVAL, "null argument");
  return lpn_rows(ctx, seed, kk_d, nullptr, k, d, e_rows_d, nullptr, row_lo, row_hi, n, stream);
}

int cuot_lpn_primal(cuot_ctx *ctx, const uint8_t seed[16], const cuot_block *kk_d,
                    int64_t k, int d, cuot_block *e_io_d, int64_t n, void *stream) {
  return cuot_lpn_primal_range(ctx, seed, kk_d, k, d, e_io_d, 0, n, n, stream);
}

int cuot_aes128_ecb(cuot_ctx *ctx, const uint8_t key[16], cuot_block *io_d,
                    uint64_t nblocks, void *stream) {
  if (!ctx || !key || (!io_d && nblocks)) return fail(CUOT_EINVAL, "null argument");
  if (nblocks == 0) return CUOT_OK;
  DeviceGuard g(ctx);
  AesKey k;
  host_aes_key_expand(key, &k);
  CUOT_TRY(set_smem(ecb_kernel));
  int grid = 1;
  grid_for(ctx, (const void *)ecb_kernel, int64_t((nblocks + 1) / 2), &grid);
  ecb_kernel<<<grid, kLpnThreads, kTableBytes, static_cast<cudaStream_t>(stream)>>>(
      k, ctx->t0_d, reinterpret_cast<Blk *>(io_d), nblocks);
  return launch_status();
}

}  // extern "C"
