// Host run of the ternary transform's per-thread steps (qc_tern.cuh), in the
// order in which the kernels of qc_tern.cu take them: out = a * in mod
// (x^n - 1) for 32 bit planes (word j of in / out: coefficient j).
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../cuot_b200/csrc/qc_tern.cuh"

using namespace cuot;
using std::vector;

static const TernSigmas kSigmas = tern_sigmas();

// The pass's DFT of one residue: f[k][i], nine coefficients L/9 apart.
template <int RAD>
static void dft_all(G4 (&f)[RAD][9]) {
  if constexpr (RAD != 27) {
    for (int i0 = 0; i0 < 3; i0++) {
      G4 h[RAD][3];
      for (int k = 0; k < RAD; k++)
        for (int c = 0; c < 3; c++) h[k][c] = f[k][i0 + 3 * c];
      dft<RAD>(h);
      for (int q = 0; q < RAD; q++)
        for (int c = 0; c < 3; c++) f[q][i0 + 3 * c] = h[dft_slot<RAD>(q)][c];
    }
  } else {
    G4 x[9][3][9];  // [q1][k2][coefficient]
    for (int k2 = 0; k2 < 3; k2++)
      for (int i0 = 0; i0 < 3; i0++) {
        G4 h[9][3];
        for (int k1 = 0; k1 < 9; k1++)
          for (int c = 0; c < 3; c++) h[k1][c] = f[3 * k1 + k2][i0 + 3 * c];
        dft<9>(h);
        for (int q1 = 0; q1 < 9; q1++)
          for (int c = 0; c < 3; c++) x[q1][k2][i0 + 3 * c] = h[dft_slot<9>(q1)][c];
      }
    for (int q1 = 0; q1 < 9; q1++)
      for (int i = 0; i < 9; i++) {
        G4 y[3];
        for (int k2 = 0; k2 < 3; k2++) {
          const int d = i - q1 * k2, wraps = (8 - d) / 9;
          y[k2] = dft27_twiddle(x[q1][k2][d + 9 * wraps], wraps);
        }
        dft3(y[0], y[1], y[2]);
        for (int q2 = 0; q2 < 3; q2++) f[q1 + 9 * q2][i] = y[q2];
      }
  }
}

template <int L, int RAD>
static void pass_steps(int e, vector<uint32_t> &buf, int pass, bool inv, const uint32_t *in) {
  const TernShape s = tern_shape(e);
  const uint16_t *sig = kSigmas.v[e - kTernMinE];
  const vector<uint32_t> src(buf);
  for (int beta = 0; beta < tern_points(s) / RAD; beta++) {
    const Butterfly b = tern_butterfly(s, sig, pass, beta, inv);
    for (int r = 0; r < L / 9; r++) {
      G4 f[RAD][9];
      for (int k = 0; k < RAD; k++) {
        const RotBase rb = rot_base<L>(inv ? inv_rotation<L>(b, sig, k) : fwd_rotation<RAD>(b, k), r);
        for (int i = 0; i < 9; i++) {
          if (in) {
            const RotEntry t = rot_entry_first(L, rb.i + i);
            const int j = (b.piece + k * b.step) * L + rb.off + t.x;
            const uint32_t x = j < (1 << e) ? in[j] : 0u;
            f[k][i] = G4{x & t.m1, x & t.m2};
          } else {
            const RotEntry t = rot_entry(L, rb.i + i, false);
            f[k][i] = load_fix(t, load_raw(src.data() + (b.first + k * b.step) * tern_element(L) + rb.off, t));
          }
        }
      }
      dft_all<RAD>(f);
      for (int q = 0; q < RAD; q++) {
        const int k = inv ? (RAD - q) % RAD : q;
        uint32_t *o = buf.data() + (b.first + k * b.step) * tern_element(L);
        const RotBase rb = rot_base<L>(inv && pass == 0 ? fwd_rotation<RAD>(b, k) : 0, r);
        for (int i = 0; i < 9; i++) store_pair(o + rb.off, rot_entry(L, rb.i + i, true), f[q][i]);
      }
    }
  }
}

template <int L>
static void outer(int e, vector<uint32_t> &buf, int pass, bool inv, const uint32_t *in = nullptr) {
  const int rad = tern_radix(tern_shape(e).m, pass);
  if (rad == 27)
    pass_steps<L, 27>(e, buf, pass, inv, in);
  else if (rad == 9)
    pass_steps<L, 9>(e, buf, pass, inv, in);
  else
    pass_steps<L, 3>(e, buf, pass, inv, in);
}

// Pieces of in (n words) -> values at the points.
template <int L>
static void forward(int e, const uint32_t *in, vector<uint32_t> &buf) {
  for (int p = 0; p < tern_passes(tern_shape(e).m); p++) outer<L>(e, buf, p, false, p ? nullptr : in);
}

template <class S>
static void inner_forward(const uint32_t *x, vector<uint32_t> &V, vector<vector<G4>> &f2) {
  for (int id = 0; id < S::TASK0; id++) p0<S>(x, V.data(), id);
  vector<G4> keep(size_t(S::TASK1) * S::R1 * 3);
  for (int id = 0; id < S::TASK1; id++) {
    G4 f[S::R1][3];
    p1_load<S>(V.data(), task1<S>(id), f);
    dft<S::R1>(f);
    std::memcpy(&keep[size_t(id) * S::R1 * 3], f, sizeof f);
  }
  for (int id = 0; id < S::TASK1; id++) {
    G4 f[S::R1][3];
    std::memcpy(f, &keep[size_t(id) * S::R1 * 3], sizeof f);
    p1_store<S>(V.data(), task1<S>(id), f);
  }
  f2.assign(S::TASK2, vector<G4>(3 * S::G));
  for (int id = 0; id < S::TASK2; id++) {
    G4 f[3][S::G];
    p2_load<S>(V.data(), task2<S>(id), f);
    std::memcpy(f2[id].data(), f, sizeof f);
  }
}

template <class S>
static void point_consts(const uint32_t *x, uint32_t *consts) {  // [word][leaf]
  vector<uint32_t> V(S::WORDS);
  vector<vector<G4>> f2;
  inner_forward<S>(x, V, f2);
  for (int id = 0; id < S::TASK2; id++) {
    const Task2 t = task2<S>(id);
    for (int q = 0; q < 3; q++)
      for (int c = 0; c < S::G; c++)
        fwd_store<S::LP>(V.data() + (t.group * 3 + q) * S::ES, t.r + 9 * c, f2[id][q * S::G + c]);
  }
  for (int el = 0; el < S::NE; el++)
    for (int h = 0; h < S::E / 5; h++) {
      uint32_t diag[S::DIAGS];
      for (int d = -26; d <= 26; d++) {
        const G4 t = const_top<S>(V.data() + el * S::ES, h, d);
        diag[d + 26] = t.a;
        diag[53 + d + 26] = t.b;
      }
      for (int e1 = 0; e1 < 5; e1++) {
        uint32_t w[kLeafWords];
        leaf_consts(Diag{diag, diag + 53}, e1, w);
        for (int j = 0; j < kLeafWords; j++) consts[j * S::LEAVES + leaf_id<S>(el / 3, el % 3, 5 * h + e1)] = w[j];
      }
    }
}

template <class S>
static void point_product(uint32_t *x, const uint32_t *consts) {
  vector<uint32_t> V(S::WORDS);
  vector<vector<G4>> f2;
  inner_forward<S>(x, V, f2);
  for (int id = 0; id < S::TASK2; id++) {
    G4 f[3][S::G];
    std::memcpy(f, f2[id].data(), sizeof f);
    p2_store<S>(V.data(), task2<S>(id), f);
  }
  for (int l = 0; l < S::LEAVES; l++) {
    uint32_t v[18], w[kLeafWords];
    for (int j = 0; j < 18; j++) v[j] = V[j * S::SL + l];
    for (int j = 0; j < kLeafWords; j++) w[j] = consts[j * S::LEAVES + l];
    leaf9(v, w);
    for (int j = 0; j < 18; j++) V[j * S::SL + l] = v[j];
  }
  for (int id = 0; id < S::TASK2; id++) {
    G4 f[3][S::G];
    p4_load<S>(V.data(), task2<S>(id), f);
    std::memcpy(f2[id].data(), f, sizeof f);
  }
  for (int id = 0; id < S::TASK2; id++) {
    G4 f[3][S::G];
    std::memcpy(f, f2[id].data(), sizeof f);
    p4_store<S>(V.data(), task2<S>(id), f);
  }
  vector<G4> keep(size_t(S::TASK1) * S::R1 * 3);
  for (int id = 0; id < S::TASK1; id++) {
    G4 f[S::R1][3];
    p5_load<S>(V.data(), task1<S>(id), f);
    dft<S::R1>(f);
    std::memcpy(&keep[size_t(id) * S::R1 * 3], f, sizeof f);
  }
  for (int id = 0; id < S::TASK1; id++) {
    G4 f[S::R1][3];
    std::memcpy(f, &keep[size_t(id) * S::R1 * 3], sizeof f);
    p5_store<S>(V.data(), task1<S>(id), f);
  }
  for (int id = 0; id < S::TASK0; id++) p6<S>(V.data(), x, id);
}

template <class S>
static void points(const TernShape &s, uint32_t *buf, uint32_t *abuf) {
  vector<uint32_t> consts(size_t(kLeafWords) * S::LEAVES);
  for (int p = 0; p < tern_points(s); p++) {
    point_consts<S>(abuf + size_t(p) * tern_element(s.L), consts.data());
    point_product<S>(buf + size_t(p) * tern_element(s.L), consts.data());
  }
}

template <int E, class S>
static void dual(const uint64_t *a, const uint32_t *in, uint32_t *out) {
  constexpr TernShape s = tern_shape(E);
  static_assert(s.L == S::L && s.Lp == S::LP, "inner level of this shape");
  const size_t n = size_t(1) << E, words = size_t(tern_points(s)) * tern_element(s.L);
  vector<uint32_t> abits(n), abuf(words), buf(words);
  for (size_t j = 0; j < n; j++) abits[j] = (a[j / 64] >> (j % 64)) & 1u ? ~0u : 0u;
  forward<S::L>(E, abits.data(), abuf);
  forward<S::L>(E, in, buf);
  points<S>(s, buf.data(), abuf.data());
  for (int p = tern_passes(s.m) - 1; p >= 0; p--) outer<S::L>(E, buf, p, true);
  for (size_t j = 0; j < n; j++) out[j] = tern_coefficient<E>(buf.data(), uint32_t(j));
}

extern "C" int tern_host_dual(int e, const uint64_t *a, const uint32_t *in, uint32_t *out) {
  switch (e) {
    case 14: dual<14, Inner<243, 27>>(a, in, out); break;
    case 15: dual<15, Inner<243, 27>>(a, in, out); break;
    case 16: dual<16, Inner<243, 27>>(a, in, out); break;
    case 17: dual<17, Inner<729, 27>>(a, in, out); break;
    case 18: dual<18, Inner<729, 27>>(a, in, out); break;
    case 19: dual<19, Inner<729, 27>>(a, in, out); break;
    case 20: dual<20, Inner<1458, 54>>(a, in, out); break;
    case 21: dual<21, Inner<2187, 81>>(a, in, out); break;
    case 22: dual<22, Inner<2187, 81>>(a, in, out); break;
    default: return 1;
  }
  return 0;
}
