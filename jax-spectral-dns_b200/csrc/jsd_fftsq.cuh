// Register-resident FFTs of square length N = S * S, one line per group of S
// lanes of a warp.
//
// Four-step form with n = S n1 + n2 and k = k1 + S k2:
//   X[k1 + S k2] = sum_n2 w_S^(n2 k2) w_N^(n2 k1) [ sum_n1 x[S n1 + n2] w_S^(n1 k1) ]
// Lane t of a group holds the elements at positions t + S m (m = 0..S-1) of
// its line. Stage 1: lane t (= n2) takes the S-point DFT over m, multiplies
// entry k1 by w_N^(t k1) and writes it to row k1, column t of the group's
// exchange buffer; stage 2: lane t (= k1) reads row t and takes the S-point
// DFT over the columns. The result X[t + S k2] lands in register k2, so every
// lane holds the same positions of the output as of the input: pointwise work
// between an inverse and a forward transform stays in registers, and the only
// synchronisation is a __syncwarp around the exchange.
//
// S-point DFTs in registers: radices 2, 3, 4, 5, 7, 8 directly (jsd_fft.cuh), 9
// and 16 as squares of 3 and 4 with twiddles (dft_square), composite S with
// coprime factors by the prime-factor (Good-Thomas) mapping, which needs no
// twiddles: n = (B n1 + A n2) mod S, k = (B (B^-1 mod A) k1 + A (A^-1 mod B)
// k2) mod S for S = A B.
#pragma once

#include "jsd_common.cuh"
#include "jsd_fft.cuh"

namespace jsd {

__host__ __device__ constexpr int sq_inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return 1;
}

// first factor A of the prime-factor split used for S (0: S is a base radix)
__host__ __device__ constexpr int sq_split(int s) {
  return s == 6 ? 2 : s == 10 ? 2 : s == 12 ? 4 : s == 14 ? 2 : s == 15 ? 3 : s == 20 ? 4 : s == 21 ? 3
       : s == 24 ? 8 : s == 28 ? 4 : s == 30 ? 2 : 0;
}

template <int R, bool INV, typename C>
__host__ __device__ __forceinline__ void dft_reg(C* x);

// cos and sin of 2 pi m / R, R = 9 and 16, for the twiddles inside dft_square
template <int R>
__host__ __device__ __forceinline__ void square_root_table(int m, double& c, double& s) {
  if (R == 9) {
    const double C[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
    const double S[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676,
                         0.34202014332566873304};
    c = C[m];
    s = S[m];
  } else {
    const double C[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                          -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0,
                          -0.92387953251128675613};
    const double S[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0,
                          0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                          -0.38268343236508977173};
    c = C[m];
    s = S[m];
  }
}

// A * A points as A-point DFTs with twiddles between (A = 3, 4)
template <int A, bool INV, typename C>
__host__ __device__ __forceinline__ void dft_square(C* x) {
  using Rl = typename real_of<C>::type;
#pragma unroll
  for (int n2 = 0; n2 < A; ++n2) {
    C a[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) a[n1] = x[A * n1 + n2];
    dft_reg<A, INV>(a);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      if (n2 * k1) {
        double c, s;
        square_root_table<A * A>(n2 * k1, c, s);
        a[k1] = cmul(a[k1], cmake<C>((Rl)c, (Rl)(INV ? s : -s)));
      }
      x[A * k1 + n2] = a[k1];
    }
  }
  C y[A * A];
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C b[A];
#pragma unroll
    for (int n2 = 0; n2 < A; ++n2) b[n2] = x[A * k1 + n2];
    dft_reg<A, INV>(b);
#pragma unroll
    for (int k2 = 0; k2 < A; ++k2) y[k1 + A * k2] = b[k2];
  }
#pragma unroll
  for (int k = 0; k < A * A; ++k) x[k] = y[k];
}

template <int A, int B, bool INV, typename C>
__host__ __device__ __forceinline__ void dft_pfa(C* x) {
  constexpr int N = A * B;
  constexpr int binv = sq_inv_mod(B % A, A);
  constexpr int ainv = sq_inv_mod(A % B, B);
  C t[N];
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1)
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) t[n1 * B + n2] = x[(B * n1 + A * n2) % N];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    C a[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) a[n1] = t[n1 * B + n2];
    dft_reg<A, INV>(a);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) t[k1 * B + n2] = a[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C b[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) b[n2] = t[k1 * B + n2];
    dft_reg<B, INV>(b);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) x[(B * binv * k1 + A * ainv * k2) % N] = b[k2];
  }
}

template <int R, bool INV, typename C>
__host__ __device__ __forceinline__ void dft_reg(C* x) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    dft2<INV>(x);
  } else if constexpr (R == 4) {
    dft4<INV>(x);
  } else if constexpr (R == 8) {
    dft8<INV>(x);
  } else if constexpr (R == 3 || R == 5 || R == 7) {
    dft_odd<R, INV>(x);
  } else if constexpr (R == 9) {
    dft_square<3, INV>(x);
  } else if constexpr (R == 16) {
    dft_square<4, INV>(x);
  } else {
    static_assert(sq_split(R) != 0, "unsupported register DFT length");
    dft_pfa<sq_split(R), R / sq_split(R), INV>(x);
  }
}

// Exchange buffer of a group: rows an odd number of elements apart (16-byte
// elements of one column then fall on distinct slots; S + 1 would put all seven
// rows of S = 7 on one), and with three and more groups per warp groups S more
// than a multiple of 16 apart, so that the lanes of a warp write one run of slots.
template <int S>
__host__ __device__ constexpr int sq_row() {
  return S | 1;
}
template <int S>
__host__ __device__ constexpr int sq_xbuf() {
  return S * sq_row<S>() + (S <= 10 ? ((S - S * sq_row<S>()) % 16 + 16) % 16 : 0);
}

// Stage 1 of a transform of the line held by the S lanes of a group (t =
// lane in the group): x[m] = element t + S m on entry; the S-point DFT over m,
// times w_N^(t j), goes to row j, column t of the group's exchange buffer xb.
// tw[j - 1] = w_N^(t j) with the forward sign, j = 1..S-1.
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ void sq_stage1(C* x, const C* tw, C* xb, int t) {
  dft_reg<S, INV>(x);
#pragma unroll
  for (int j = 1; j < S; ++j) {
    C w = tw[j - 1];
    if (INV) w.y = -w.y;
    x[j] = cmul(x[j], w);
  }
#pragma unroll
  for (int j = 0; j < S; ++j) xb[j * sq_row<S>() + t] = x[j];
}

// Stage 2: lane t reads row t and transforms it; x[m] = X[t + S m] on exit.
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ void sq_stage2(C* x, const C* xb, int t) {
#pragma unroll
  for (int j = 0; j < S; ++j) x[j] = xb[t * sq_row<S>() + j];
  dft_reg<S, INV>(x);
}

// The whole transform. Every lane of the warp must call it, since the exchange
// is synchronised warp-wide; lanes outside any group pass live = false.
template <int S, bool INV, typename C>
__device__ __forceinline__ void sq_fft(C* x, const C* tw, C* xb, int t, bool live) {
  if (live) sq_stage1<S, INV>(x, tw, xb, t);
  __syncwarp();
  if (live) sq_stage2<S, INV>(x, xb, t);
  __syncwarp();
}

// Row stride of the lane-major twiddle table: entry (j, t) = w_N^(t j) sits at
// (j - 1) * stride + t, so the lanes of a group read consecutive entries.
__host__ __device__ constexpr int sq_tw_stride(int s) {
  return s <= 16 ? 16 : 32;
}

// sq_fft with the twiddles read from the lane-major table (sq_tw_stride;
// typically in shared memory) instead of registers.
template <int S, bool INV, typename C>
__device__ __forceinline__ void sq_fft_tab(C* x, const C* tab, C* xb, int t, bool live) {
  constexpr int TS = sq_tw_stride(S);
  if (live) {
    dft_reg<S, INV>(x);
#pragma unroll
    for (int j = 1; j < S; ++j) {
      C w = tab[(j - 1) * TS + t];
      if (INV) w.y = -w.y;
      x[j] = cmul(x[j], w);
    }
#pragma unroll
    for (int j = 0; j < S; ++j) xb[j * sq_row<S>() + t] = x[j];
  }
  __syncwarp();
  if (live) sq_stage2<S, INV>(x, xb, t);
  __syncwarp();
}

// Half-split form for even S = 2H: a line on 2S lanes, lane (t, h) holding
// the H elements at positions t + S (2 j + h), j = 0..H-1.
//   stage 1, decimation in time over m = 2 j + h: lane h transforms its own
//     H values (E for h = 0, O for h = 1), swaps them with its partner lane
//     (same t, other h), and forms Y[h H + k] = E[k] +- w_S^k O[k], times
//     w_N^(t (h H + k)), into the exchange buffer;
//   stage 2, decimation in frequency: lane (t, h) reads row t and forms
//     c[n] = b[n] + b[n+H] (h = 0) or (b[n] - b[n+H]) w_S^n (h = 1), whose
//     H-point DFT is X[t + S (2 j + h)].
// Input and output positions of a lane coincide, as in sq_fft. tab = w_N^e.
// Stage-1 butterfly of the half-split form for one k: own = this lane's
// H-point DFT value at k, other = the partner lane's.
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ C sq2_butterfly(C own, C other, int k, const C* tab, int t, int h) {
  constexpr int H = S / 2;
  const C E = h ? other : own;
  C O = h ? own : other;
  C w = tab[S * k];
  if (INV) w.y = -w.y;
  O = cmul(O, w);
  const C y = h ? csub(E, O) : cadd(E, O);
  C tw = tab[t * (h * H + k)];
  if (INV) tw.y = -tw.y;
  return cmul(y, tw);
}

// Stage 2 of the half-split form: read row t of the exchange buffer, combine
// for output parity h, H-point DFT; x[j] = X[t + S (2 j + h)] on exit.
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ void sq2_stage2(C* x, const C* xb, const C* tab, int t, int h) {
  constexpr int H = S / 2;
#pragma unroll
  for (int n = 0; n < H; ++n) {
    const C b0 = xb[t * (S + 1) + n], b1 = xb[t * (S + 1) + n + H];
    if (h) {
      C w = tab[S * n];
      if (INV) w.y = -w.y;
      x[n] = cmul(csub(b0, b1), w);
    } else {
      x[n] = cadd(b0, b1);
    }
  }
  dft_reg<H, INV>(x);
}

template <int S, bool INV, typename C>
__device__ __forceinline__ void sq2_fft(C* x, const C* tab, C* xb, int t, int h, int partner, bool live) {
  constexpr int H = S / 2;
  static_assert(2 * H == S, "half-split transform needs an even side");
  dft_reg<H, INV>(x);
#pragma unroll
  for (int k = 0; k < H; ++k) {
    C o;
    o.x = __shfl_sync(0xffffffffu, x[k].x, partner);
    o.y = __shfl_sync(0xffffffffu, x[k].y, partner);
    x[k] = sq2_butterfly<S, INV>(x[k], o, k, tab, t, h);
  }
  if (live) {
#pragma unroll
    for (int k = 0; k < H; ++k) xb[(h * H + k) * (S + 1) + t] = x[k];
  }
  __syncwarp();
  if (live) sq2_stage2<S, INV>(x, xb, tab, t, h);
  __syncwarp();
}

// Half-split form on lane pairs (S = 12, 14, 16): lane 2 t + h of a line holds
// element positions t + S m, its partner the other half of column t.
//   S = 2 H, H odd: prime-factor mapping, m = (H h + 2 r) mod S on entry and
//     (H h + (H + 1) r) mod S on exit in register r: the split into H-point
//     DFTs and pairs needs no twiddles.
//   H even: m = 2 r + h both ways, twiddles w_S^r on the odd half as in sq2_fft.
// The exchange buffer has 16 columns per row; column c of row j sits at
// c ^ swizzle(j). The two rows a lane pair writes differ by 4 in the swizzle and
// eight neighbouring rows have distinct ones, so the writes of eight lanes, and
// the reads of eight rows (the lanes of a pair read the same entry), hit
// distinct 16-byte slots. The twiddle table is swizzled likewise.
template <int S>
struct Sq2p {
  static constexpr int H = S / 2, XS = 16;
  static constexpr bool PF = H % 2 == 1;
  static_assert(S == 12 || S == 14 || S == 16, "swizzles are laid out for these sides");
  // m, and the exchange row, of register r in lane half h: m0 + (h ? step(m0) : 0)
  static __host__ __device__ constexpr int out0(int r) { return PF ? (H + 1) * r % S : 2 * r; }
  static __host__ __device__ constexpr int row0(int r) { return PF ? out0(r) : r; }
  static __host__ __device__ constexpr int step(int m0) { return PF ? (m0 < H ? H : -H) : 1; }
  static __host__ __device__ constexpr int rstep(int j0) { return PF ? step(j0) : H; }
  // entry register of the element that leaves a transform in register r
  static __host__ __device__ constexpr int entry(int r) { return PF ? (H + 1) / 2 * r % H : r; }
  static __host__ __device__ constexpr bool second(int j) { return PF ? j % 2 == 1 : j >= H; }
  static __host__ __device__ constexpr int swizzle(int j) {
    const int e = !second(j) ? j : PF ? (j >= H ? j - H : j + H) : j - H;  // the first row of j's pair
    const int f = PF ? (e < 8 ? e / 2 : (e - 6) / 2) : S == 12 ? (e < 4 ? e : e + 2) : e;
    return second(j) ? f ^ 4 : f;
  }
  static __host__ __device__ constexpr int xbuf() { return S * XS; }
  static __host__ __device__ constexpr int tab() { return S * XS; }
};

// Entry e of the swizzled twiddle table (Sq2p::tab entries): w_N^(t j) at j * 16 + (t ^ 4 second(j))
template <int S, typename C>
__host__ __device__ __forceinline__ C sq2p_table_entry(const C* __restrict__ table, int e) {
  const int j = e / Sq2p<S>::XS, t = (e % Sq2p<S>::XS) ^ (Sq2p<S>::second(j) ? 4 : 0);
  return t < S ? table[t * j] : cmake<C>(0, 0);
}

// First half: the H-point DFT over a lane's own values, ready for the pair.
// wS (even H only): 1 for the even half, then w_S^k, k < H, for the odd one (no
// branch on the half).
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ void sq2p_first(C* x, const C* wS, int h) {
  using Q = Sq2p<S>;
  dft_reg<Q::H, INV>(x);
  if constexpr (!Q::PF) {
#pragma unroll
    for (int k = 1; k < Q::H; ++k) {
      C w = wS[h * Q::H + k];
      if (INV) w.y = -w.y;
      x[k] = cmul(x[k], w);
    }
  }
}

// The pair's value for the row that lane half sg (+1, -1) writes, times its twiddle
template <bool INV, typename C, typename Rl>
__host__ __device__ __forceinline__ C sq2p_pair(C own, C other, C w, Rl sg) {
  if (INV) w.y = -w.y;
  return cmul(cmake<C>(fma(sg, own.x, other.x), fma(sg, own.y, other.y)), w);
}

// Second half: x[n] = entry n0 of the row +- entry n1 (sq2p_n0, sq2p_n1), transformed
template <int S>
__host__ __device__ constexpr int sq2p_n0(int n) {
  return Sq2p<S>::PF ? 2 * n : n;
}
template <int S>
__host__ __device__ constexpr int sq2p_n1(int n) {
  return Sq2p<S>::PF ? (S / 2 + 2 * n) % S : n + S / 2;
}
template <int S, bool INV, typename C>
__host__ __device__ __forceinline__ void sq2p_second(C* x, const C* wS, int h) {
  using Q = Sq2p<S>;
  if constexpr (!Q::PF) {
#pragma unroll
    for (int n = 1; n < Q::H; ++n) {
      C w = wS[h * Q::H + n];
      if (INV) w.y = -w.y;
      x[n] = cmul(x[n], w);
    }
  }
  dft_reg<Q::H, INV>(x);
}

#if defined(__CUDACC__)
// 16-byte shared-memory accesses by 32-bit address: an address with the line's
// buffer on a 128-byte boundary takes a swizzle as an exclusive or
// (volatile, so that they stay between the barriers of an exchange; table loads need not)
__device__ __forceinline__ double2 lds16(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ double2 lds16_table(unsigned a) {
  double2 v;
  asm("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts16(unsigned a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};\n" ::"r"(a), "d"(v.x), "d"(v.y));
}

// Shared-memory addresses of a lane: its column of the exchange rows (and of
// the twiddle table) that its half writes, for rows whose step is +H or -H (or
// the one step of even H), and its own row for reading, swizzles included
struct Sq2pAddr {
  unsigned wp, wm, tp, tm, row;
};
template <int S>
__device__ __forceinline__ Sq2pAddr sq2p_addr(unsigned xb, unsigned tab, int t, int h) {
  using Q = Sq2p<S>;
  const unsigned th = 16u * (unsigned)(t ^ (h ? 4 : 0)), hs = h ? 16u * Q::XS * Q::H : 0u;
  Sq2pAddr a;
  a.wp = xb + th + hs;
  a.tp = tab + th + hs;
  a.wm = xb + th - hs;  // only used for rows of at least H
  a.tm = tab + th - hs;
  a.row = xb + 16u * (unsigned)(t * Q::XS + Q::swizzle(t));
  return a;
}

template <int S, bool INV>
__device__ __forceinline__ void sq2p_fft(double2* x, const double2* wS, const Sq2pAddr& ad, int h, bool live) {
  using Q = Sq2p<S>;
  constexpr unsigned ROW = 16u * Q::XS;
  const double sg = h ? -1.0 : 1.0;
  sq2p_first<S, INV>(x, wS, h);
#pragma unroll
  for (int k = 0; k < Q::H; ++k) {
    double2 o;
    o.x = __shfl_xor_sync(0xffffffffu, x[k].x, 1);
    o.y = __shfl_xor_sync(0xffffffffu, x[k].y, 1);
    const int j0 = Q::row0(k);
    const bool up = Q::rstep(j0) > 0;
    const double2 v = sq2p_pair<INV>(x[k], o, lds16_table((up ? ad.tp : ad.tm) + j0 * ROW), sg);
    if (live) sts16(((up ? ad.wp : ad.wm) ^ (16u * Q::swizzle(j0))) + j0 * ROW, v);
  }
  __syncwarp();
#pragma unroll
  for (int n = 0; n < Q::H; ++n) {
    constexpr unsigned LOW = 7u;
    const unsigned n0 = sq2p_n0<S>(n), n1 = sq2p_n1<S>(n);
    const double2 b0 = lds16((ad.row ^ (16u * (n0 & LOW))) + 16u * (n0 & ~LOW));
    const double2 b1 = lds16((ad.row ^ (16u * (n1 & LOW))) + 16u * (n1 & ~LOW));
    x[n] = make_double2(fma(sg, b1.x, b0.x), fma(sg, b1.y, b0.y));
  }
  sq2p_second<S, INV>(x, wS, h);
  __syncwarp();
}
#endif

// Lane t's twiddles w_N^(t j), j = 1..S-1, from the table w_N^e, e = 0..N-1.
template <int S, typename C>
__host__ __device__ __forceinline__ void sq_twiddles(C* tw, const C* __restrict__ table, int t) {
#pragma unroll
  for (int j = 1; j < S; ++j) tw[j - 1] = table[t * j];
}

}  // namespace jsd
