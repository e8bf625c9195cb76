// pprf_kernel.cuh -- the GGM PPRF tree kernel (a group of threads per tree),
// shared by the translation units that launch it.  Each including file gets its own
// copy of the fixed-key schedule in constant memory and must upload it once
// per device before the first launch (pprf_upload_keys).
#pragma once
#include "ctx.cuh"

namespace cuot {
// Internal linkage: every including translation unit gets its own kernel
// instances bound to its own constant-memory key copy.
namespace {

// Fixed GGM keys: k0 = zero_block, k1 = makeBlock(0, 1) (spcot_sender.h:63).
__constant__ AesKey c_ggm_rk[2];

// Uploads this translation unit's copy of the GGM key schedules to the
// current device.
inline cudaError_t pprf_upload_keys() {
  AesKey k[2];
  uint8_t key[16] = {0};
  host_aes_key_expand(key, &k[0]);
  key[0] = 1;
  host_aes_key_expand(key, &k[1]);
  return cudaMemcpyToSymbol(c_ggm_rk, k, sizeof k);
}

enum PprfMode { FERRET_SEND = 0, FERRET_RECV = 1, SOT_SEND = 2, SOT_RECV = 3 };

struct PprfArgs {
  uint64_t t;
  int h;
  const uint32_t *t0;
  const Blk *roots;  // senders
  Blk *leaves, *scratch;
  Blk delta;
  // Ferret sender outputs [t][h], [t]
  Blk *lsum, *rsum, *ss_out;
  // receivers
  const Blk *mc;          // Ferret [t][h]; SOT [h][t]
  const uint8_t *choice;  // Ferret [t][h]; SOT [h][t]
  const Blk *ss_in;       // Ferret [t]
  // SOT sender inputs [h][t], outputs [h+1][t]; SOT receiver inputs [h+1][t]
  const Blk *base0, *base1;
  Blk *m0, *m1;
  const Blk *m0_in, *m1_in;
};

// Threads per CTA at most: one group of 256 or 128 threads, two of 128, four of 64.
constexpr int kPprfThreads = 256;

__device__ __forceinline__ Blk mask_lsb(Blk b) {
  b.w[0] &= ~1u;  // emp-ot `& one`, one = makeBlock(~0, ~1)
  return b;
}

// Shared-memory state of a group of G threads (256, 128 or 64): the levels of up to G nodes and the
// warps' level sums (left, right), double-buffered by level parity.
template <int G>
struct PprfSmem {
  Blk lev[G + G / 2];
  Blk red[2][2][G / 32];
  // Level of 2^k <= G nodes: levels alternate between the two parts.
  __device__ Blk *level(int k) {
    constexpr int kLog = G == 256 ? 8 : G == 128 ? 7 : 6;
    return lev + ((k ^ kLog) & 1 ? G : 0);
  }
};
// Dynamic shared memory of a CTA: the T-table, then the groups' states.
template <int G>
constexpr int pprf_smem_bytes() {
  return kTableBytes + kPprfThreads / G * int(sizeof(PprfSmem<G>));
}
// Barrier of the group (named, since a CTA may hold several).
template <int G>
__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(G) : "memory");
}

// XOR of a block value over the lanes of `mask` (all that call), in each of them.
__device__ __forceinline__ Blk mask_xor(uint32_t mask, Blk v) {
#pragma unroll
  for (int i = 0; i < 4; i++) v.w[i] = __reduce_xor_sync(mask, v.w[i]);
  return v;
}

// Expands tree `tree` of the instance described by `a` with a group of G
// threads (tid: thread of the group).  slot: 2^h blocks for the ping-pong of the
// levels above G nodes; smaller ones stay in shared memory, where a level costs
// one AES latency and a barrier and no trip to L2 and back.
// The T-table must already be staged (and synced) in shared memory.
extern __shared__ __align__(16) uint32_t smem_tab[];
// sot: SOT modes (an argument, so that a kernel over trees of both kinds holds
// the AES loop once).
template <bool SEND, int G>
__device__ __forceinline__ void pprf_tree(const PprfArgs &a, bool sot, uint64_t tree, Blk *slot, int group, int tid) {
  PprfSmem<G> &sm = reinterpret_cast<PprfSmem<G> *>(smem_tab + kTableWords)[group];
  const TabRef T{reinterpret_cast<const char *>(smem_tab), uint32_t(tid & 31) * 4u};
  // Senders: the sums of level l leave the group (global stores by its first
  // warp) and nothing of them is read back, so one barrier per level suffices,
  // with the warp sums double-buffered by level parity: the first warp reads
  // red[l & 1] before it enters level l + 1, and red[l & 1] is written again
  // only after the barrier that ends level l + 1.  Receivers patch a node of
  // the level just written, which the next level reads, so they keep a
  // second barrier.
  const int lane = tid & 31, warp = tid >> 5;
  const int h = a.h;
  const uint64_t W = 1ull << h;
  Blk *const leaves = a.leaves + tree * W;
  Blk root{{0, 0, 0, 0}};
  uint32_t bits = 0;  // receivers: choice bit of level l in bit l (h <= 30)
  if (SEND) {
    root = ldg_blk(a.roots + tree);
  } else {
    const bool c = lane < h && a.choice[sot ? uint64_t(lane) * a.t + tree : tree * h + lane];
    bits = __ballot_sync(0xffffffffu, c);
  }
  uint64_t ap = 0;  // receivers' path
  // Senders' outputs of level l from its left and right sums (one thread).
  const auto send_sums = [&](int l, bool last, const Blk(&S)[2]) {
    const uint64_t of = tree * h + l, os = uint64_t(l) * a.t + tree;
    if (!sot) {
      // ot_msg_0/1 of level l (spcot_sender.h:66-84), host layout [t][h]
      st_blk(a.lsum + of, S[0]);
      st_blk(a.rsum + of, S[1]);
      if (last)  // secret_sum = XOR(masked leaves) ^ delta (spcot_sender.h:49-58)
        st_blk(a.ss_out + tree, blk_xor(mask_lsb(blk_xor(S[0], S[1])), a.delta));
    } else {
      const Blk b0 = ldg_blk(a.base0 + os), b1 = ldg_blk(a.base1 + os);
      st_blk(a.m0 + os, blk_xor(b0, S[0]));
      st_blk(a.m1 + os, blk_xor(b1, S[1]));
      if (last) {  // extra row that carries delta (silent/sender.cu:97-102)
        st_blk(a.m0 + os + a.t, blk_xor(blk_xor(b0, S[1]), a.delta));
        st_blk(a.m1 + os + a.t, blk_xor(blk_xor(b1, S[0]), a.delta));
      }
    }
  };

  for (int l = 0; l < h; l++) {
    const bool last = (l == h - 1);
    const uint32_t np = 1u << l;  // h <= 30
    const Blk *in = np <= unsigned(G) ? sm.level(l) : (h - l) & 1 ? slot : leaves;
    Blk *out = !last && 2 * np <= unsigned(G) ? sm.level(l + 1) : (h - l) & 1 ? leaves : slot;
    // receivers: the level's message (and its mask), on the way during the AES
    Blk x0{{0, 0, 0, 0}}, x1{{0, 0, 0, 0}};
    const int bit = (bits >> l) & 1;
    const uint64_t os = uint64_t(l) * a.t + tree;
    const bool quick = np <= 32 && !last;
    if (!SEND && (quick ? warp == bit && lane == int(ap) : tid == 0)) {
      x0 = ldg_blk(a.mc + (sot ? os : tree * h + l));
      if (sot) x1 = ldg_blk((bit ? a.m1_in : a.m0_in) + os);
    }
    // (without it the loading thread ran on by itself: 479 -> 679 us for 1,280 trees
    // of depth 13)
    if (!SEND) __syncwarp();
    if (quick) {
      // The chain of levels is what a small call waits for: about 2,000 cycles each
      // here when one thread made both children (1,590 of issue and latency for the
      // two AES) and one warp then finished the sums (570).  So a warp per side, a node
      // per lane (1,100), and no sums on the chain: the senders' last warp adds up the
      // children in shared memory while the others go on, and the receivers' sum of
      // side `bit` is in one warp, whose lane `ap` has the node to mend.  16 trees of
      // depth 10: Ferret 18.4 / 19.8 -> 16.9 / 18.2 us (sender / receiver), SOT
      // 20.0 / 22.1 -> 17.1 / 18.7; 5,000 of depth 9: 163 / 169 -> 148 / 152.
      if (warp < 2 && lane < int(np)) {
        const Blk p = (l == 0) ? root : ld_blk(in + lane);
        uint32_t x[4] = {p.w[0], p.w[1], p.w[2], p.w[3]};
        aes_enc(T, x, c_ggm_rk[warp]);
        Blk c{{x[0] ^ p.w[0], x[1] ^ p.w[1], x[2] ^ p.w[2], x[3] ^ p.w[3]}};
        if (!SEND && warp == bit) {
          const Blk s = mask_xor(uint32_t((1ull << np) - 1), c);
          if (lane == int(ap)) c = blk_xor(blk_xor(c, s), blk_xor(x0, x1));
        }
        st_blk(out + 2 * lane + warp, c);
      }
      ap = 2 * ap + 1 - bit;
      group_sync<G>(group);
      if (SEND && warp == G / 32 - 1) {
        Blk S[2] = {Blk{{0, 0, 0, 0}}, Blk{{0, 0, 0, 0}}};
        if (lane < int(np)) {
          S[0] = ld_blk(out + 2 * lane);
          S[1] = ld_blk(out + 2 * lane + 1);
        }
        S[0] = warp_xor(S[0]);
        S[1] = warp_xor(S[1]);
        if (lane == 0) send_sums(l, last, S);
      }
      continue;
    }
    const uint32_t keep = last && !sot ? ~1u : ~0u;  // Ferret leaves: emp-ot `& one`
    Blk accL{{0, 0, 0, 0}}, accR{{0, 0, 0, 0}};
    for (uint32_t i = tid; i < np; i += G) {
      const Blk p = (l == 0) ? root : ld_blk(in + i);
      uint32_t L[4] = {p.w[0], p.w[1], p.w[2], p.w[3]};
      uint32_t R[4] = {p.w[0], p.w[1], p.w[2], p.w[3]};
      aes_enc2(T, L, c_ggm_rk[0], R, c_ggm_rk[1]);
      Blk cl{{L[0] ^ p.w[0], L[1] ^ p.w[1], L[2] ^ p.w[2], L[3] ^ p.w[3]}};
      Blk cr{{R[0] ^ p.w[0], R[1] ^ p.w[1], R[2] ^ p.w[2], R[3] ^ p.w[3]}};
      accL = blk_xor(accL, cl);
      accR = blk_xor(accR, cr);
      cl.w[0] &= keep;
      cr.w[0] &= keep;
      if (last) {
        st_blk_cs(out + 2 * i, cl);
        st_blk_cs(out + 2 * i + 1, cr);
      } else {
        st_blk(out + 2 * i, cl);
        st_blk(out + 2 * i + 1, cr);
      }
    }
    // Warps that had nodes (np: a power of two) add up theirs.
    const int nw = np >= unsigned(G) ? G / 32 : np > 32 ? int(np / 32) : 1;
    Blk(&red)[2][G / 32] = sm.red[l & 1];
    if (warp < nw) {
      accL = warp_xor(accL);
      accR = warp_xor(accR);
      if (nw > 1 && lane == 0) {
        red[0][warp] = accL;
        red[1][warp] = accR;
      }
    }
    group_sync<G>(group);
    if (warp == 0) {
      Blk S[2] = {accL, accR};
      if (nw > 1) {  // lanes 0..: left sums, lanes 16..: right sums
        Blk v{{0, 0, 0, 0}};
        if ((lane & 15) < nw) v = ld_blk(&red[lane >> 4][lane & 15]);
#pragma unroll
        for (int o = G / 64; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < 4; i++) v.w[i] ^= __shfl_xor_sync(0xffffffffu, v.w[i], o);
        S[0] = S[1] = v;
#pragma unroll
        for (int i = 0; i < 4; i++) S[1].w[i] = __shfl_down_sync(0xffffffffu, v.w[i], 16);
      }
      if (lane == 0) {
        if (SEND) {
          send_sums(l, last, S);
        } else if (!sot) {
          // spcot_recver.h:71-95: b = 0 -> fill the even child, puncture the odd.
          const uint64_t f = 2 * ap + bit, pun = 2 * ap + 1 - bit;
          // The node at f currently holds X (garbage, derived from the unknown
          // punctured parent).  S_b includes X, so X ^ S_b ^ m is the XOR of
          // the other same-side nodes with m: the sender's node.
          const Blk fix = blk_xor(bit ? S[1] : S[0], x0);
          if (!last) {
            st_blk(out + f, blk_xor(ld_blk(out + f), fix));
          } else {
            // Leaves are stored masked.  Filled leaf (masked) = X' ^ mask(fix).
            st_blk(out + f, blk_xor(ld_blk(out + f), mask_lsb(fix)));
            // Punctured leaf = XOR of all other masked leaves ^ secret_sum
            // (spcot_recver.h:53-64) = mask(S0 ^ S1 ^ fix) ^ G' ^ ss, with G'
            // the masked garbage leaf at `pun` (its term cancels).
            const Blk g = ld_blk(out + pun);
            Blk r = blk_xor(mask_lsb(blk_xor(blk_xor(S[0], S[1]), fix)), g);
            r = blk_xor(r, ldg_blk(a.ss_in + tree));
            st_blk(out + pun, r);
          }
          ap = pun;
        } else {  // SOT_RECV (silent/recver.cu:98-115, 143-155)
          const uint64_t f = 2 * ap + bit, pun = 2 * ap + 1 - bit;
          st_blk(out + f, blk_xor(ld_blk(out + f), blk_xor(blk_xor(x0, x1), bit ? S[1] : S[0])));
          if (last) {
            const Blk dec2 = blk_xor(ldg_blk((bit ? a.m1_in : a.m0_in) + os + a.t), ldg_blk(a.mc + os));
            st_blk(out + pun, blk_xor(ld_blk(out + pun), blk_xor(dec2, bit ? S[0] : S[1])));
          }
          ap = pun;
        }
      }
    }
    if (!SEND) group_sync<G>(group);
  }
}

// Trees of a single instance: every group takes trees group, group + groups,
// ... (persistent: the table is staged once per CTA, and a group's slot of the
// scratch stays in L2 from tree to tree).
template <int MODE, int G, bool CHAINED>
__global__ void __launch_bounds__(kPprfThreads, 3) pprf_tree_kernel(PprfArgs a) {
  const int per_cta = blockDim.x / G;
  stage_table(smem_tab, a.t0);
  __syncthreads();
  const uint32_t zero = chain_begin<CHAINED>();
  const int group = threadIdx.x / G;
  // groups of one CTA take trees far apart, so that few trees spread over CTAs
  const uint64_t id = uint64_t(group) * gridDim.x + blockIdx.x, groups = uint64_t(gridDim.x) * per_cta;
  for (uint64_t tree = id + zero; tree < a.t; tree += groups) {
    pprf_tree<MODE == FERRET_SEND || MODE == SOT_SEND, G>(a, MODE == SOT_SEND || MODE == SOT_RECV, tree,
                                                          a.scratch + (id << a.h), group, threadIdx.x % G);
    group_sync<G>(group);  // the next tree's writes to the shared state
  }
}

// Threads per tree for `trees` trees (the deepest of depth h) on `ctas` resident
// CTAs.  Shallow levels leave most of a large group idle, so with enough trees
// to fill the chip several smaller groups share a CTA.  Measured on B200
// (Ferret sender, 256 / 128 / 64 threads): 64 trees of depth 10 17.4 / 17.6 /
// 24.6 us, 300 33.5 / 32.9 / 39.2, 918 of depth 9 45 / 41 / 41, 1,280 of depth 13
// 463 / 468 / 485, 1,500 of depth 10 102 / 99 / 90, 4,971 of depth 11 519 / 490 /
// 458, 5,000 of depth 9 203 / 194 / 148 (one CTA per tree and launch before: 277).
// Deep trees that two groups per CTA would share out badly (more than 1.2 times the
// CTAs, but not two per CTA; more than 13 / 6, but not 8 / 3) go one by one to CTAs as
// these get free: dealt out beforehand they leave SMs waiting for the fullest one
// (one by one / dealt out: 500 trees of depth 13 209 / 208 us, 592 209 / 260, 740 258 /
// 302, 888 322 / 302, 950 359 / 350, 1,036 359 / 396, 1,184 408 / 464, 1,280 468 / 465).
inline int pprf_group_size(uint64_t trees, int h, uint64_t ctas) {
  if (trees <= ctas) return 256;
  const bool uneven = (5 * trees > 6 * ctas && 3 * trees <= 5 * ctas) || (6 * trees > 13 * ctas && 3 * trees <= 8 * ctas);
  if (h >= 12 && uneven) return 256;
  return trees <= 3 * ctas || h > 12 ? 128 : 64;
}

}  // namespace
}  // namespace cuot
