// qc_tern.cuh -- shapes and per-thread steps of the ternary transform behind
// the exact dual LPN (qc_tern.cu).  Everything here is host/device code, so a
// CPU test runs the same steps thread by thread.
//
// Product of two polynomials over GF(2) by A. Schoenhage, "Schnelle
// Multiplikation von Polynomen ueber Koerpern der Charakteristik 2", Acta
// Informatica 7 (1977): with y = x^L, a polynomial of n bits is one of
// I = ceil(n / L) pieces of L bits in y, and the pieces' products (degree
// below 2L - 1) are taken in
//   R_L = GF(2)[x] / (x^2L + x^L + 1),
// where w = x^L is a primitive cube root of unity and x a root of unity of
// order 3L: transforms in y of length 3^j need only XORs and rotations.  An
// element of R_L is L pairs (a, b) = a + b w with x^L = w, i.e. a polynomial
// over GF(4); w (a, b) = (b, a ^ b), w^2 (a, b) = (a ^ b, a).
//
// Outer level: the 2I - 1 pieces of the product are found from its values at
//   C: y^m = 1 (m points, m >= 2I - 1), or
//   F: y^2m + y^m + 1 = 0 (2m points: y^m = w and y^m = w^2).
// Inner level, per point: a product in R_L is a product in z = x^L' modulo
// z^2T + z^T + 1 (T = L / L', since z^T = x^L = w) of 2T pieces of L' bits, so
// its values at the 2T points z^T = w, w^2 in R_L' give it exactly.
// Leaf: a product in R_L' = GF(4)[x] / (x^L' - w) by a fixed element is a
// Toeplitz matrix times a vector; it is split into 9 x 9 Toeplitz products by
// the transpose of Toom-Cook over GF(4) (points 0, 1, w, w^2, infinity: five
// products per three-way split; Karatsuba for a two-way split), and each of
// those once more into five 3 x 3 ones.
//
// Data words hold 32 bit planes, so one XOR works on 32 of the 128 products
// that share the polynomial `a`; `a` itself only enters as leaf constants.
#pragma once
#include <stdint.h>

#define TERN_HD __host__ __device__ __forceinline__

namespace cuot {

// ---- shapes ------------------------------------------------------------------
struct TernShape {
  int L, Lp;      // ring sizes: R_L (outer), R_Lp (inner); T = L / Lp points per half
  int m, cosets;  // 1: C (y^m = 1); 2: F
};
constexpr int kTernMinE = 14, kTernMaxE = 22;
constexpr TernShape tern_shape(int e) {
  return e == 14   ? TernShape{243, 27, 81, 2}
         : e == 15 ? TernShape{243, 27, 243, 2}
         : e == 16 ? TernShape{243, 27, 729, 1}
         : e == 17 ? TernShape{729, 27, 243, 2}
         : e == 18 ? TernShape{729, 27, 729, 1}
         : e == 19 ? TernShape{729, 27, 729, 2}
         : e == 20 ? TernShape{1458, 54, 729, 2}
         : e == 21 ? TernShape{2187, 81, 2187, 1}
                   : TernShape{2187, 81, 2187, 2};
}
constexpr int tern_points(const TernShape &s) { return s.m * s.cosets; }
constexpr int tern_pieces(const TernShape &s, int e) { return int(((1ll << e) + s.L - 1) / s.L); }
// 9 x 9 products per R_Lp product.
constexpr int tern_evals(int Lp) { return Lp == 27 ? 5 : Lp == 54 ? 15 : 25; }
// Outer passes: radix 27 first, then what is left of m.
constexpr int tern_passes(int m) { return m == 2187 ? 3 : 2; }
constexpr int tern_radix(int m, int p) { return p == 0 || (m == 729 && p == 1) ? 27 : m == 81 ? 3 : 9; }
constexpr bool tern_shape_ok(int e) {
  const TernShape s = tern_shape(e);
  return (s.cosets == 2 ? 2 : 1) * s.m >= 2 * tern_pieces(s, e) - 1 && tern_pieces(s, e) <= s.m &&
         s.L % (s.cosets == 2 ? s.m : s.m / 3) == 0;
}
static_assert(tern_shape_ok(14) && tern_shape_ok(15) && tern_shape_ok(16) && tern_shape_ok(17) && tern_shape_ok(18) &&
                  tern_shape_ok(19) && tern_shape_ok(20) && tern_shape_ok(21) && tern_shape_ok(22),
              "points must determine the product and their roots of unity must lie in R_L");

// ---- GF(4) pairs of 32-plane words --------------------------------------------
struct G4 {
  uint32_t a, b;
};
TERN_HD G4 g_add(G4 x, G4 y) { return G4{x.a ^ y.a, x.b ^ y.b}; }
TERN_HD G4 g_w1(G4 x) { return G4{x.b, x.a ^ x.b}; }
TERN_HD G4 g_w2(G4 x) { return G4{x.a ^ x.b, x.a}; }

// (x0, x1, x2) -> sums with 1, w^k, w^2k, k = 0, 1, 2: eight three-input XORs.
TERN_HD void dft3(G4 &x0, G4 &x1, G4 &x2) {
  const G4 y0{x0.a ^ x1.a ^ x2.a, x0.b ^ x1.b ^ x2.b};
  const G4 y1{x0.a ^ x1.b ^ (x2.a ^ x2.b), x0.b ^ x2.a ^ (x1.a ^ x1.b)};
  x2 = G4{x0.a ^ y0.a ^ y1.a, x0.b ^ y0.b ^ y1.b};  // y0 + y1 + y2 = x0
  x1 = y1;
  x0 = y0;
}

// RAD-point DFT over elements whose three coefficients lie L/3 apart, so that
// t = x^(L/3) (t^3 = w, a ninth root of unity) only renames them.  Output q
// stands in slot dft_slot<RAD>(q).
template <int RAD>
TERN_HD constexpr int dft_slot(int q) { return RAD == 9 ? 3 * (q % 3) + q / 3 : q; }
TERN_HD void mul_t(G4 (&f)[3]) {
  const G4 x = f[2];
  f[2] = f[1];
  f[1] = f[0];
  f[0] = g_w1(x);
}
template <int RAD>
TERN_HD void dft(G4 (&f)[RAD][3]) {
  if constexpr (RAD == 3) {
#pragma unroll
    for (int c = 0; c < 3; c++) dft3(f[0][c], f[1][c], f[2][c]);
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
      for (int c = 0; c < 3; c++) dft3(f[k][c], f[3 + k][c], f[6 + k][c]);
    mul_t(f[4]);
    mul_t(f[5]);
    mul_t(f[5]);
    mul_t(f[7]);
    mul_t(f[7]);
    mul_t(f[8]);  // t^4 = w t
#pragma unroll
    for (int c = 0; c < 3; c++) f[8][c] = g_w1(f[8][c]);
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
      for (int c = 0; c < 3; c++) dft3(f[3 * q][c], f[3 * q + 1][c], f[3 * q + 2][c]);
  }
}
// Output k of the inverse DFT (w -> w^-1; 1 / RAD = 1): slot of DFT output -k.
template <int RAD>
TERN_HD constexpr int idft_slot(int k) { return dft_slot<RAD>((RAD - k) % RAD); }

// ---- outer passes ------------------------------------------------------------------
// A node of M pieces holds the product mod y^M - x^sigma; a pass of radix RAD
// turns it into RAD nodes of M / RAD pieces with sigma_q = (sigma + 3 L q) / RAD:
// the DFT of its pieces k M/RAD + i, each times x^(k sigma / RAD).  Nodes are
// numbered in place (child q of node v is v RAD + q), over all cosets.
constexpr int tern_node_size(int m, int pass) {
  int v = m;
  for (int p = 0; p < pass; p++) v /= tern_radix(m, p);
  return v;
}
// Shift of a coset's root node: y^m = x^sigma (C: 1; F: w and w^2).
constexpr int tern_root_sigma(const TernShape &s, int coset) { return s.cosets == 1 ? 0 : (coset + 1) * s.L; }
// sigma of every node of passes 0, 1, ...: pass p from tern_sigma_at on.
constexpr int tern_sigma_at(const TernShape &s, int pass) {
  int at = 0;
  for (int p = 0; p < pass; p++) at += tern_points(s) / tern_node_size(s.m, p);
  return at;
}
constexpr int kTernSigmas = 2 + 54 + 486;  // the most of any shape
struct TernSigmas {
  uint16_t v[kTernMaxE - kTernMinE + 1][kTernSigmas];
};
constexpr TernSigmas tern_sigmas() {
  TernSigmas t{};
  for (int e = kTernMinE; e <= kTernMaxE; e++) {
    const TernShape s = tern_shape(e);
    for (int c = 0; c < s.cosets; c++) t.v[e - kTernMinE][c] = uint16_t(tern_root_sigma(s, c));
    for (int p = 0; p + 1 < tern_passes(s.m); p++) {
      const int nodes = tern_points(s) / tern_node_size(s.m, p), rad = tern_radix(s.m, p);
      for (int n = 0; n < nodes; n++)
        for (int q = 0; q < rad; q++)
          t.v[e - kTernMinE][tern_sigma_at(s, p + 1) + n * rad + q] =
              uint16_t((t.v[e - kTernMinE][tern_sigma_at(s, p) + n] + 3 * s.L * q) / rad);
    }
  }
  return t;
}

// Butterfly beta of a pass.
struct Butterfly {
  int sigma;        // of its node
  int first, step;  // its points
  int piece;        // their index in their node, and in the next pass's child
  int kids;         // INV: index of its first child's sigma (-1: last pass, no rotation)
  int kn, rn;       // INV: the piece's slot in the next forward pass, and that pass's radix
};
TERN_HD Butterfly tern_butterfly(const TernShape &s, const uint16_t *sigmas, int pass, int beta, bool inv) {
  const int M = tern_node_size(s.m, pass), rad = tern_radix(s.m, pass), step = M / rad;
  const int node = beta / step, piece = beta % step;
  Butterfly b{};
  b.sigma = sigmas[tern_sigma_at(s, pass) + node];
  b.first = node * M + piece;
  b.step = step;
  b.piece = piece;
  b.kids = -1;
  if (inv && pass + 1 < tern_passes(s.m)) {
    b.kids = tern_sigma_at(s, pass + 1) + node * rad;
    b.rn = tern_radix(s.m, pass + 1);
    b.kn = piece / (step / b.rn);
  }
  return b;
}
// Rotation of slot k's load: forward, piece k by k sigma / RAD; inverse, child
// k back by what the next forward pass rotated this piece of it by.
template <int RAD>
TERN_HD int fwd_rotation(const Butterfly &b, int k) { return k * b.sigma / RAD; }
template <int L>
TERN_HD int inv_rotation(const Butterfly &b, const uint16_t *sigmas, int k) {
  if (b.kids < 0) return 0;
  const int f = b.kn * sigmas[b.kids + k] / b.rn;
  return f ? 3 * L - f : 0;
}

// Elements in memory: two parts of nine blocks of L/9 words, each block padded
// to whole 32-byte sectors.
constexpr int tern_block(int L) { return (L / 9 + 7) & ~7; }
constexpr int tern_part(int L) { return 9 * tern_block(L); }
constexpr int tern_element(int L) { return 2 * tern_part(L); }
template <int L>
TERN_HD int tern_word(int r) { return r + r / (L / 9) * (tern_block(L) - L / 9); }  // of coefficient r in its part

// x^s of an element, s in [0, 3L): with s = a L/9 + lo, coefficient r of block i
// (r < L/9, i < 9) comes from block d = i - a - [r < lo], d in [-27, 9), at
// r - lo (+ L/9 if r < lo) there.  Table entry d + 27: block d mod 9, times
// w^(wraps), as the two words to load: x in part wraps != 0 and y in the other
// one give (x ^ (y & m2), y ^ (x & m1)).  A rotated store by -s goes to the same
// place with w^-wraps, as (a ^ (b & m1)) -> x, (b ^ (a & m2)) -> y.
struct RotEntry {
  int x, y;
  uint32_t m1, m2;
};
constexpr int kRotEntries = 36;
TERN_HD RotEntry rot_entry(int L, int i, bool store) {
  const int d = i - 27;
  int g = (8 - d) / 9;  // -floor(d / 9), 0..3
  const int at = (d + g * 9) * tern_block(L);
  g = store ? (6 - g) % 3 : g % 3;
  return RotEntry{at + (g ? tern_part(L) : 0), at + (g ? 0 : tern_part(L)), g == 1 ? ~0u : 0u, g == 2 ? ~0u : 0u};
}
// The first pass's input is one word per coefficient (at x, unpadded), with the
// masks of w^g's two words.
TERN_HD RotEntry rot_entry_first(int L, int i) {
  const int d = i - 27, g = (8 - d) / 9;
  return RotEntry{(d + g * 9) * (L / 9), 0, g % 3 != 1 ? ~0u : 0u, g % 3 != 0 ? ~0u : 0u};
}
// What a load puts into the pair first (raw), and after all loads are issued.
TERN_HD G4 load_raw(const uint32_t *p, const RotEntry &e) { return G4{p[e.x], p[e.y]}; }
TERN_HD G4 load_fix(const RotEntry &e, G4 v) { return G4{v.a ^ (v.b & e.m2), v.b ^ (v.a & e.m1)}; }
TERN_HD void store_pair(uint32_t *p, const RotEntry &e, G4 v) {
  p[e.x] = v.a ^ (v.b & e.m1);
  p[e.y] = v.b ^ (v.a & e.m2);
}
struct RotBase {
  int off;  // to add to a table entry's words
  int i;    // table index of block 0
};
template <int L>
TERN_HD RotBase rot_base(int s, int r) {
  const int a = s / (L / 9), lo = s % (L / 9), low = r < lo;
  return RotBase{r - lo + (low ? L / 9 : 0), 27 - a - low};
}

// 27-point DFT of elements whose nine coefficients lie L/9 apart, as 9-point
// DFTs over k1 (k = 3 k1 + k2) by threads that hold coefficients i0 + 3c, then,
// for each q1, three-point ones over k2 of x^(q1 k2 L/9) times the results:
// output q1 + 9 q2.  dft27_shift: block and wraps of coefficient i of that.
TERN_HD G4 dft27_twiddle(G4 v, int wraps) { return wraps == 0 ? v : wraps == 1 ? g_w1(v) : g_w2(v); }

// ---- inner level ---------------------------------------------------------------
// Working copy of an R_Lp element: four blocks of Lp words, a window of the
// cyclic sequence [a | a ^ b | b], in which the two words of coefficient P of
// x^s times the element stand at P - s and P - s - Lp.  The window is chosen
// so that no index wraps: the forward steps rotate by s in [0, 2 Lp) (indices
// [-3 Lp, Lp)), the inverse ones by -s (indices [-Lp, 3 Lp)).  The fourth
// block is one more store per pair; wrapping would be four more operations
// per load, and the lookups are bound by the integer pipe.
template <int LP>
TERN_HD void fwd_store(uint32_t *V, int p, G4 v) {
  V[p] = v.a;
  V[LP + p] = v.a ^ v.b;
  V[2 * LP + p] = v.b;
  V[3 * LP + p] = v.a;
}
template <int LP>
TERN_HD G4 fwd_load(const uint32_t *V, int q) { return G4{V[3 * LP + q], V[2 * LP + q]}; }
template <int LP>
TERN_HD void inv_store(uint32_t *V, int p, G4 v) {
  V[p] = v.b;
  V[LP + p] = v.a;
  V[2 * LP + p] = v.a ^ v.b;
  V[3 * LP + p] = v.b;
}
template <int LP>
TERN_HD G4 inv_load(const uint32_t *V, int q) { return G4{V[LP + q], V[q]}; }

// Compile-time shape of the inner level.
template <int L_, int LP_>
struct Inner {
  static constexpr int L = L_, LP = LP_, T = L_ / LP_, R1 = T / 3;  // passes of radix R1 (9 or 3) and 3
  static constexpr int G = LP_ / 9, E = tern_evals(LP_);
  static constexpr int NE = 2 * T;             // elements (points)
  static constexpr int TASK1 = 2 * 3 * (LP_ / 3);  // radix-R1 butterflies: half, piece, residue
  static constexpr int TASK2 = 2 * R1 * 9;     // radix-3 butterflies with evaluation: half, node, residue
  static constexpr int LEAVES = NE * E;
  // Words between the 18 words of a leaf product: LEAVES rounded up to 9 mod
  // 16, so that a warp of consecutive groups (2 R1 of them) and residues
  // writes distinct banks.
  static constexpr int SL = LEAVES + ((9 - LEAVES % 16) + 16) % 16;
  // Words of a working copy: its four blocks, padded so that consecutive
  // elements lie (about) Lp / 3 banks apart, as a warp of radix-R1 butterflies
  // wants them, and an odd number, as one of radix-3 butterflies does.
  static constexpr int ES = LP_ == 27 ? 137 : LP_ == 54 ? 243 : 347;
  static constexpr int BASE = NE * ES;
  // Steps 0 and 6: a thread takes one coefficient p < Lp of CH consecutive pieces.
  static constexpr int CH = LP_ == 27 ? 3 : LP_ == 54 ? 6 : 9;
  static constexpr int CHUNKS = (T + CH - 1) / CH, TASK0 = LP_ * CHUNKS;
  // Word of coefficient p of piece i in a part of an R_L element.
  TERN_HD static constexpr int word(int i, int p) { return i / (T / 9) * tern_block(L_) + i % (T / 9) * LP_ + p; }
  static constexpr int WORDS = 18 * SL > BASE ? 18 * SL : BASE;
  static constexpr int DIAGS = 2 * 53;         // words of a 27 x 27 matrix's diagonals
  static_assert(R1 == 9 || R1 == 3, "inner passes");
};

// Step 0: an R_L element x into the two halves' pieces: z^T = w takes (a, b) of
// pieces i and i + T as they are, z^T = w^2 takes (a ^ b, b).
template <class S>
TERN_HD void p0(const uint32_t *x, uint32_t *V, int id) {
  const int p = id % S::LP, i0 = id / S::LP * S::CH;
#pragma unroll
  for (int c = 0; c < S::CH; c++) {
    const int i = i0 + c;
    if (S::T % S::CH && i >= S::T) break;
    const G4 u{x[S::word(i, p)], x[S::word(i, p) + tern_part(S::L)]};
    fwd_store<S::LP>(V + i * S::ES, p, u);
    fwd_store<S::LP>(V + (S::T + i) * S::ES, p, G4{u.a ^ u.b, u.b});
  }
}

struct Task1 {
  int half, piece, r;
};
template <class S>
TERN_HD Task1 task1(int id) {
  return Task1{id / (3 * (S::LP / 3)), (id / (S::LP / 3)) % 3, id % (S::LP / 3)};
}
template <class S>
TERN_HD void p1_load(const uint32_t *V, const Task1 &t, G4 (&f)[S::R1][3]) {
#pragma unroll
  for (int k = 0; k < S::R1; k++) {
    const uint32_t *e = V + (t.half * S::T + t.piece + 3 * k) * S::ES;
    const int rot = k * (t.half + 1) * (S::LP / S::R1);
#pragma unroll
    for (int c = 0; c < 3; c++) f[k][c] = fwd_load<S::LP>(e, t.r - rot + c * (S::LP / 3));
  }
}
template <class S>
TERN_HD void p1_store(uint32_t *V, const Task1 &t, const G4 (&f)[S::R1][3]) {
#pragma unroll
  for (int q = 0; q < S::R1; q++)
#pragma unroll
    for (int c = 0; c < 3; c++)
      fwd_store<S::LP>(V + (t.half * S::T + q * 3 + t.piece) * S::ES, t.r + c * (S::LP / 3), f[dft_slot<S::R1>(q)][c]);
}

// Radix-3 pass: group = half * R1 + node (fastest over lanes), residue r mod 9.
struct Task2 {
  int group, r;
};
template <class S>
TERN_HD Task2 task2(int id) {
  return Task2{id % (2 * S::R1), id / (2 * S::R1)};
}
// sigma / 3 of a node of the radix-3 pass.
template <class S>
TERN_HD int sigma3(int group) {
  return (group / S::R1 + 1 + 3 * (group % S::R1)) * (S::LP / (3 * S::R1));
}
template <class S>
TERN_HD void p2_load(const uint32_t *V, const Task2 &t, G4 (&f)[3][S::G]) {
  const int s3 = sigma3<S>(t.group);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const uint32_t *e = V + (t.group * 3 + k) * S::ES;
    const int rot = k * s3;  // below 2 Lp
#pragma unroll
    for (int c = 0; c < S::G; c++) f[k][c] = fwd_load<S::LP>(e, t.r - rot + 9 * c);
  }
#pragma unroll
  for (int c = 0; c < S::G; c++) dft3(f[0][c], f[1][c], f[2][c]);
}

// Transposed Toom-Cook of a three-way Toeplitz split: (v0, v1, v2) -> the five
// vectors at 0, 1, w, w^2, infinity of v2 + v1 Y + v0 Y^2, and back.
TERN_HD void toom_eval(G4 v0, G4 v1, G4 v2, G4 (&e)[5]) {
  e[0] = v2;
  e[4] = v0;
  dft3(v2, v1, v0);
  e[1] = v2;
  e[2] = v1;
  e[3] = v0;
}
TERN_HD void toom_join(const G4 (&q)[5], G4 &o0, G4 &o1, G4 &o2) {
  G4 x = q[1], y = q[2], z = q[3];
  dft3(x, y, z);
  o0 = g_add(x, q[0]);
  o1 = y;
  o2 = g_add(z, q[4]);
}
// A residue's G coefficients (9 apart) -> its words of the E leaf vectors.
template <int G>
TERN_HD void leaf_eval(const G4 (&v)[G], G4 (&e)[G == 3 ? 5 : G == 6 ? 15 : 25]) {
  if constexpr (G == 3) {
    toom_eval(v[0], v[1], v[2], e);
  } else {
    constexpr int H = G == 6 ? 3 : 5;
    G4 u[H][3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
      if constexpr (G == 6) {  // Karatsuba: V1, V0, V0 + V1
        u[0][b] = v[3 + b];
        u[1][b] = v[b];
        u[2][b] = g_add(v[b], v[3 + b]);
      } else {
        G4 t[5];
        toom_eval(v[b], v[3 + b], v[6 + b], t);
#pragma unroll
        for (int h = 0; h < 5; h++) u[h][b] = t[h];
      }
    }
#pragma unroll
    for (int h = 0; h < H; h++) {
      G4 t[5];
      toom_eval(u[h][0], u[h][1], u[h][2], t);
#pragma unroll
      for (int j = 0; j < 5; j++) e[5 * h + j] = t[j];
    }
  }
}
template <int G>
TERN_HD void leaf_join(const G4 (&e)[G == 3 ? 5 : G == 6 ? 15 : 25], G4 (&v)[G]) {
  if constexpr (G == 3) {
    toom_join(e, v[0], v[1], v[2]);
  } else {
    constexpr int H = G == 6 ? 3 : 5;
    G4 u[H][3];
#pragma unroll
    for (int h = 0; h < H; h++) {
      G4 t[5];
#pragma unroll
      for (int j = 0; j < 5; j++) t[j] = e[5 * h + j];
      toom_join(t, u[h][0], u[h][1], u[h][2]);
    }
#pragma unroll
    for (int b = 0; b < 3; b++) {
      if constexpr (G == 6) {
        v[b] = g_add(u[0][b], u[2][b]);
        v[3 + b] = g_add(u[1][b], u[2][b]);
      } else {
        const G4 t[5] = {u[0][b], u[1][b], u[2][b], u[3][b], u[4][b]};
        toom_join(t, v[b], v[3 + b], v[6 + b]);
      }
    }
  }
}

// Leaf vectors: word j (0..17) of leaf (element group * 3 + q, evaluation ev)
// at [j][(q E + ev) 2 R1 + group].
template <class S>
TERN_HD int leaf_id(int group, int q, int ev) {
  return (q * S::E + ev) * (2 * S::R1) + group;
}
template <class S>
TERN_HD void p2_store(uint32_t *V, const Task2 &t, const G4 (&f)[3][S::G]) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    G4 e[S::E];
    leaf_eval<S::G>(f[q], e);
#pragma unroll
    for (int j = 0; j < S::E; j++) {
      uint32_t *o = V + 2 * t.r * S::SL + leaf_id<S>(t.group, q, j);
      o[0] = e[j].a;
      o[S::SL] = e[j].b;
    }
  }
}
// Leaf products -> inverse radix-3 butterfly -> pieces (rotated back by the
// next step's loads).
template <class S>
TERN_HD void p4_load(const uint32_t *V, const Task2 &t, G4 (&f)[3][S::G]) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    G4 e[S::E];
#pragma unroll
    for (int j = 0; j < S::E; j++) {
      const uint32_t *o = V + 2 * t.r * S::SL + leaf_id<S>(t.group, q, j);
      e[j] = G4{o[0], o[S::SL]};
    }
    leaf_join<S::G>(e, f[q]);
  }
#pragma unroll
  for (int c = 0; c < S::G; c++) dft3(f[0][c], f[1][c], f[2][c]);
}
template <class S>
TERN_HD void p4_store(uint32_t *V, const Task2 &t, const G4 (&f)[3][S::G]) {
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int c = 0; c < S::G; c++)
      inv_store<S::LP>(V + (t.group * 3 + k) * S::ES, t.r + 9 * c, f[(3 - k) % 3][c]);
}
template <class S>
TERN_HD void p5_load(const uint32_t *V, const Task1 &t, G4 (&f)[S::R1][3]) {
#pragma unroll
  for (int q = 0; q < S::R1; q++) {
    const int group = t.half * S::R1 + q;
    const int rot = t.piece * sigma3<S>(group);  // below 2 Lp
    const uint32_t *e = V + (group * 3 + t.piece) * S::ES;
#pragma unroll
    for (int c = 0; c < 3; c++) f[q][c] = inv_load<S::LP>(e, t.r + rot + c * (S::LP / 3));
  }
}
template <class S>
TERN_HD void p5_store(uint32_t *V, const Task1 &t, const G4 (&f)[S::R1][3]) {
#pragma unroll
  for (int k = 0; k < S::R1; k++)
#pragma unroll
    for (int c = 0; c < 3; c++)
      inv_store<S::LP>(V + (t.half * S::T + t.piece + 3 * k) * S::ES, t.r + c * (S::LP / 3), f[idft_slot<S::R1>(k)][c]);
}
// Step 6: the R_L product.  With A, B the halves' pieces, piece i + T of the
// product is A + B and piece i is w^2 A + w B; each has 2 Lp coefficients, so
// its upper half falls on the next piece's lower half, and the last one's on
// pieces 0 and T (z^2T = z^T + 1).
template <class S>
TERN_HD void in_piece(const uint32_t *V, int i, int p, G4 &A, G4 &B) {
  const int rot = i / 3 * (S::LP / S::R1);  // slot of the radix-R1 pass: rotated back by slot (half + 1) Lp / R1
  A = inv_load<S::LP>(V + i * S::ES, p + rot);
  B = inv_load<S::LP>(V + (S::T + i) * S::ES, p + 2 * rot);
}
template <class S>
TERN_HD void p6(const uint32_t *V, uint32_t *x, int id) {
  const int p = id % S::LP, i0 = id / S::LP * S::CH;
  G4 A, B, C, D;
  in_piece<S>(V, i0 ? i0 - 1 : S::T - 1, p, C, D);
#pragma unroll
  for (int c = 0; c < S::CH; c++) {
    const int i = i0 + c;
    if (S::T % S::CH && i >= S::T) break;
    in_piece<S>(V, i, p, A, B);
    // lower halves of pieces i and i + T, and the upper halves of those before
    uint32_t ulo = C.a ^ D.a ^ D.b, uhi = C.b ^ D.b;
    if (i == 0) {
      const uint32_t t = ulo;
      ulo = uhi;
      uhi ^= t;
    }
    x[S::word(i, p)] = A.a ^ A.b ^ B.b ^ ulo;
    x[S::word(i, p) + tern_part(S::L)] = A.a ^ B.a ^ uhi;
    C = A;
    D = B;
  }
}

// ---- leaves ----------------------------------------------------------------------
// Constants of a 9 x 9 product: for each of its five 3 x 3 Toeplitz products
// the five diagonals c = c0 + c1 w, as bits c0, c1, c0 ^ c1: bit j % 32 of word
// j / 32, j = (e2 5 + diagonal) 3 + {0, 1, 2}.
constexpr int kLeafMasks = 75, kLeafWords = 3;

// (a, b) of the N pairs o += c v, c of bits j, j + 1, j + 2.  On the device the
// bits become predicates of the XORs (one operation each).
template <int N>
TERN_HD void leaf_diagonal(const uint32_t (&w)[kLeafWords], int j, const G4 *v0, G4 *o0) {
#ifdef __CUDA_ARCH__
  if constexpr (N == 1)
    asm("{ .reg .pred p0, p1, p2; .reg .u32 t;\n"
        "and.b32 t, %4, %7; setp.ne.u32 p0, t, 0; and.b32 t, %5, %8; setp.ne.u32 p1, t, 0;"
        "and.b32 t, %6, %9; setp.ne.u32 p2, t, 0;\n"
        "@p0 xor.b32 %0, %0, %2; @p1 xor.b32 %0, %0, %3; @p1 xor.b32 %1, %1, %2; @p2 xor.b32 %1, %1, %3; }"
        : "+r"(o0[0].a), "+r"(o0[0].b)
        : "r"(v0[0].a), "r"(v0[0].b), "r"(w[j / 32]), "r"(w[(j + 1) / 32]), "r"(w[(j + 2) / 32]),
          "r"(1u << j % 32), "r"(1u << (j + 1) % 32), "r"(1u << (j + 2) % 32));
  else if constexpr (N == 2)
    asm("{ .reg .pred p0, p1, p2; .reg .u32 t;\n"
        "and.b32 t, %8, %11; setp.ne.u32 p0, t, 0; and.b32 t, %9, %12; setp.ne.u32 p1, t, 0;"
        "and.b32 t, %10, %13; setp.ne.u32 p2, t, 0;\n"
        "@p0 xor.b32 %0, %0, %4; @p1 xor.b32 %0, %0, %5; @p1 xor.b32 %1, %1, %4; @p2 xor.b32 %1, %1, %5;\n"
        "@p0 xor.b32 %2, %2, %6; @p1 xor.b32 %2, %2, %7; @p1 xor.b32 %3, %3, %6; @p2 xor.b32 %3, %3, %7; }"
        : "+r"(o0[0].a), "+r"(o0[0].b), "+r"(o0[1].a), "+r"(o0[1].b)
        : "r"(v0[0].a), "r"(v0[0].b), "r"(v0[1].a), "r"(v0[1].b), "r"(w[j / 32]), "r"(w[(j + 1) / 32]),
          "r"(w[(j + 2) / 32]), "r"(1u << j % 32), "r"(1u << (j + 1) % 32), "r"(1u << (j + 2) % 32));
  else
    asm("{ .reg .pred p0, p1, p2; .reg .u32 t;\n"
        "and.b32 t, %12, %15; setp.ne.u32 p0, t, 0; and.b32 t, %13, %16; setp.ne.u32 p1, t, 0;"
        "and.b32 t, %14, %17; setp.ne.u32 p2, t, 0;\n"
        "@p0 xor.b32 %0, %0, %6; @p1 xor.b32 %0, %0, %7; @p1 xor.b32 %1, %1, %6; @p2 xor.b32 %1, %1, %7;\n"
        "@p0 xor.b32 %2, %2, %8; @p1 xor.b32 %2, %2, %9; @p1 xor.b32 %3, %3, %8; @p2 xor.b32 %3, %3, %9;\n"
        "@p0 xor.b32 %4, %4, %10; @p1 xor.b32 %4, %4, %11; @p1 xor.b32 %5, %5, %10; @p2 xor.b32 %5, %5, %11; }"
        : "+r"(o0[0].a), "+r"(o0[0].b), "+r"(o0[1].a), "+r"(o0[1].b), "+r"(o0[2].a), "+r"(o0[2].b)
        : "r"(v0[0].a), "r"(v0[0].b), "r"(v0[1].a), "r"(v0[1].b), "r"(v0[2].a), "r"(v0[2].b), "r"(w[j / 32]),
          "r"(w[(j + 1) / 32]), "r"(w[(j + 2) / 32]), "r"(1u << j % 32), "r"(1u << (j + 1) % 32),
          "r"(1u << (j + 2) % 32));
#else
  uint32_t m[3];
  for (int k = 0; k < 3; k++) m[k] = (w[(j + k) / 32] >> (j + k) % 32) & 1u ? ~0u : 0u;
  for (int n = 0; n < N; n++) {
    o0[n].a ^= (v0[n].a & m[0]) ^ (v0[n].b & m[1]);
    o0[n].b ^= (v0[n].a & m[1]) ^ (v0[n].b & m[2]);
  }
#endif
}

// v (nine pairs) <- Toeplitz product.
TERN_HD void leaf9(uint32_t (&v)[18], const uint32_t (&w)[kLeafWords]) {
  G4 e[5][3], q[5][3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    G4 t[5];
    toom_eval(G4{v[2 * i], v[2 * i + 1]}, G4{v[6 + 2 * i], v[7 + 2 * i]}, G4{v[12 + 2 * i], v[13 + 2 * i]}, t);
#pragma unroll
    for (int h = 0; h < 5; h++) e[h][i] = t[h];
  }
#pragma unroll
  for (int h = 0; h < 5; h++) {
    // diagonal d: output r takes input r + 2 - d
#pragma unroll
    for (int r = 0; r < 3; r++) q[h][r] = G4{0u, 0u};
    leaf_diagonal<1>(w, 15 * h, &e[h][2], &q[h][0]);
    leaf_diagonal<2>(w, 15 * h + 3, &e[h][1], &q[h][0]);
    leaf_diagonal<3>(w, 15 * h + 6, &e[h][0], &q[h][0]);
    leaf_diagonal<2>(w, 15 * h + 9, &e[h][0], &q[h][1]);
    leaf_diagonal<1>(w, 15 * h + 12, &e[h][0], &q[h][2]);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const G4 t[5] = {q[0][i], q[1][i], q[2][i], q[3][i], q[4][i]};
    G4 o0, o1, o2;
    toom_join(t, o0, o1, o2);
    v[2 * i] = o0.a;
    v[2 * i + 1] = o0.b;
    v[6 + 2 * i] = o1.a;
    v[7 + 2 * i] = o1.b;
    v[12 + 2 * i] = o2.a;
    v[13 + 2 * i] = o2.b;
  }
}

// The constants' side: diagonal d of the Toeplitz matrix of an R_Lp element c is
// c_d (d >= 0) or w c_(d + Lp), i.e. the rotated read; a three-way split's
// block diagonals T_-2..T_2 combine (interpolation, transposed) to
//   0: T_-2 + T_1, 1: T_-1 + T_0 + T_1, w: w^2 T_-1 + w T_0 + T_1,
//   w^2: w T_-1 + w^2 T_0 + T_1, infinity: T_2 + T_-1,
// a two-way split's to T_-1 + T_0, T_0 + T_1, T_0.
TERN_HD G4 toom_const(int e, G4 tm2, G4 tm1, G4 t0, G4 t1, G4 t2) {
  if (e == 0) return g_add(tm2, t1);
  if (e == 1) return g_add(g_add(tm1, t0), t1);
  if (e == 2) return g_add(g_add(g_w2(tm1), g_w1(t0)), t1);
  if (e == 3) return g_add(g_add(g_w1(tm1), g_w2(t0)), t1);
  return g_add(t2, tm1);
}
// Diagonal d (|d| <= 26) of evaluation h's 27 x 27 Toeplitz matrix, from the
// element's working copy at V.
template <class S>
TERN_HD G4 const_top(const uint32_t *V, int h, int d) {
  if constexpr (S::G == 3) {
    return fwd_load<S::LP>(V, d);
  } else if constexpr (S::G == 6) {
    const G4 t = fwd_load<S::LP>(V, d);
    return h < 2 ? g_add(t, fwd_load<S::LP>(V, h == 0 ? d - 27 : d + 27)) : t;
  } else {
    return toom_const(h, fwd_load<S::LP>(V, d - 54), fwd_load<S::LP>(V, d - 27), fwd_load<S::LP>(V, d),
                      fwd_load<S::LP>(V, d + 27), fwd_load<S::LP>(V, d + 54));
  }
}
// Leaf words of evaluation e1 of the 27 x 27 matrix whose diagonals d are at
// t[d + 26].  Word bits come from bit 0 of the data words.
struct Diag {
  const uint32_t *a, *b;  // words of diagonal -26
};
TERN_HD void leaf_consts(const Diag &t, int e1, uint32_t (&w)[kLeafWords]) {
  G4 s1[17];
#pragma unroll
  for (int i = 0; i < 17; i++) {
    const int d = i - 8 + 26;
    s1[i] = toom_const(e1, G4{t.a[e1 ? d : d - 18], t.b[e1 ? d : d - 18]}, G4{t.a[d - 9], t.b[d - 9]}, G4{t.a[d], t.b[d]},
                       G4{t.a[d + 9], t.b[d + 9]}, G4{t.a[d + (e1 < 4 ? 0 : 18)], t.b[d + (e1 < 4 ? 0 : 18)]});
  }
  w[0] = w[1] = w[2] = 0;
#pragma unroll
  for (int e2 = 0; e2 < 5; e2++)
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const int d = i - 2 + 8;
      const G4 c = toom_const(e2, s1[d - 6], s1[d - 3], s1[d], s1[d + 3], s1[d + 6]);
      const int j = (5 * e2 + i) * 3;
      w[j / 32] |= (c.a & 1u) << j % 32;
      w[(j + 1) / 32] |= (c.b & 1u) << (j + 1) % 32;
      w[(j + 2) / 32] |= ((c.a ^ c.b) & 1u) << (j + 2) % 32;
    }
}

// Coefficient j of the product mod x^n - 1 from the pieces c_i (after the last
// inverse pass): coefficients j and j + n of sum_i c_i x^(iL), where c_i has 2L
// coefficients.  F: with A, B the cosets' pieces, c_i = w^2 A_i + w B_i and
// c_(i + m) = A_i + B_i.
template <int E>
TERN_HD uint32_t tern_piece(const uint32_t *buf, int i, int part, int at) {  // at: word of the coefficient in its part
  constexpr TernShape s = tern_shape(E);
  constexpr int el = tern_element(s.L), pt = tern_part(s.L);
  if (s.cosets == 1) return buf[i * el + part * pt + at];
  if (i >= s.m) {
    const uint32_t *A = buf + (i - s.m) * el + part * pt + at;
    return A[0] ^ A[s.m * el];
  }
  const uint32_t *A = buf + i * el + at, *B = A + s.m * el;
  return A[0] ^ B[pt] ^ (part ? B[0] : A[pt]);
}
template <int E>
TERN_HD uint32_t tern_coefficient(const uint32_t *buf, uint32_t j) {
  constexpr TernShape s = tern_shape(E);
  uint32_t v = 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t t = j + (uint32_t(h) << E);
    const int i = int(t / uint32_t(s.L)), at = tern_word<s.L>(int(t % uint32_t(s.L)));
    if (i < tern_points(s)) v ^= tern_piece<E>(buf, i, 0, at);
    if (i) v ^= tern_piece<E>(buf, i - 1, 1, at);
  }
  return v;
}

}  // namespace cuot
