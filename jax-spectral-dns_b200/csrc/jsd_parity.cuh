// FP64 y-contractions on even and odd parts.
//
// The Gauss-Lobatto points are symmetric about y = 0, so every y-operator maps
// even profiles to even ones and odd to odd (D and its products: even to odd
// and odd to even), and every eigenvector of the interior D^2 is even or odd.
// An Ny x Ny product on a profile is then two products of half the size in
// each direction on its even and odd parts, half the multiplications:
//   input on the points  (FOLD): s_k = b_k + b_{n-1-k}, d_k = b_k - b_{n-1-k}
//   output on the points (unfold): c_i = S_i + T_i, c_{n-1-i} = S_i - T_i
//   eigen rows: even modes first, then odd ones (the plan orders them so)
//
// k_parity: C_e (M x N) = A_e B_e for a batch of entries, each operator given
// as two halves in DMMA fragment order. Both halves of an operator live in the
// registers of the CTA's 2 W warps (warps 0..W-1 the first half, TM row tiles
// of 8 each): operand A costs no shared-memory reads, and a B fragment read
// from the tile serves TM tensor instructions. Column tiles of 32 stream
// through two shared buffers by cp.async; persistent CTAs walk a contiguous
// range of (entry, tile), so an operator is loaded once or twice per CTA. A
// half with one row or column more than its tiles (Ny = 16 j + 1) takes that row
// as plain dot products and that column as an outer product, which beats padding
// 65 to 72.
// Bound: the FP64 tensor pipe (44 us of 79 for the three products back from the
// eigenbasis at 129 x 129 columns, Ny = 129; pipe 56 to 67% active); the rest is the
// stretch between two tiles of a CTA that the other CTA of the SM only partly
// fills. Whole-operator tiles (k_dgemm_t) take 126 us for the same call, 103
// against 67 us for the y-derivatives of two fields.
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "../../include/jsd.h"
#include "jsd_common.cuh"
#include "jsd_gemm.cuh"

namespace jsd {

constexpr int kParN = 32;          // columns per tile
constexpr int kParBS = kParN + 4;  // tile row stride: the fragment reads of a half-warp hit distinct banks

struct ParityEntry {
  const double* a[2];  // halves in fragment order (parity_pack)
  const double* B;     // kin x N
  double* C;           // mout x N
  int M[2], K[2];      // rows and columns of the halves
  int part[2];         // input part each half reads: 0 sums / even rows, 1 differences / odd rows
  int kin, mout;       // rows of B and C
};

struct ParityBatch {
  ParityEntry e[kGemmMaxBatch];
  int count;
  int N;       // columns = row stride of B and C
  int unfold;  // outputs on the points (else: rows of half 0, then of half 1)
  int rows;    // rows of a tile buffer (parity_rows)
  int accumulate;  // C += A B (unfolded outputs only)
};

// row tiles of 8 that hold M rows, one row beyond them left to the dot products
inline int parity_row_tiles(int m) { return m > 8 && m % 8 == 1 ? m / 8 : (m + 7) / 8; }

// Warps per half and row tiles per warp for `rt` row tiles, chosen by time at
// 129 x 129 (rt = 8: (4, 2) 77 / 79 us with and without folding, (2, 4) 81 /
// 87, (8, 1) 97 / 94), 161 x 161 columns at Ny = 145 (rt = 9: (3, 3) 150 / 161,
// (9, 1) 177 / 176) and 33 x 33 x 8 runs at Ny = 97 (rt = 6: (2, 3) 29 / 29,
// (3, 2) 30 / 31, (6, 1) 32 / 31): pairs of row tiles keep the tensor
// instructions large, but two warps of each CTA per quarter of an SM fill the
// pipe better than one.
inline bool parity_shape(int rt, int& w, int& tm) {
  static const int shapes[][2] = {{1, 1}, {2, 1}, {3, 1}, {2, 2}, {5, 1}, {2, 3}, {4, 2}, {3, 3}, {5, 2}, {6, 2}};
  for (const auto& s : shapes)
    if (s[0] * s[1] >= rt) {
      w = s[0];
      tm = s[1];
      return true;
    }
  return false;
}

// k steps of 4 held per row tile; a half with one column more (at most 8 rt + 1,
// as many as rows) starts its accumulators with that column's outer product
__host__ __device__ constexpr int parity_ksteps(int row_tiles) { return 2 * row_tiles; }

// position of element (row, k) of a half in fragment order: [row tile][k step][lane]
inline size_t parity_slot(int row_tiles, int row, int k) {
  return ((size_t)(row / 8) * parity_ksteps(row_tiles) + k / 4) * 32 + (row % 8) * 4 + k % 4;
}

// A half (M x K, row-major) in fragment order, zero padded, followed by its
// column 8 row_tiles (row by row) and its row 8 row_tiles (zeros without one).
inline size_t parity_frag(int row_tiles) { return (size_t)row_tiles * parity_ksteps(row_tiles) * 32; }
inline std::vector<double> parity_pack(const std::vector<double>& h, int M, int K, int row_tiles) {
  const int edge = 8 * row_tiles;
  const size_t frag = parity_frag(row_tiles);
  std::vector<double> out(frag + edge + K, 0.0);
  for (int r = 0; r < M; ++r)
    for (int k = 0; k < K; ++k) {
      const double v = h[(size_t)r * K + k];
      if (r >= edge) out[frag + edge + k] = v;
      else if (k >= edge) out[frag + r] = v;
      else out[parity_slot(row_tiles, r, k)] = v;
    }
  return out;
}

// The eigenbasis tables of a plan with every eigenvector exactly even or odd
// and the even modes first (the order of the eigen rows is the plan's own),
// and D exactly odd under y -> -y. An eigenvector as a solver returns it has
// the other parity mixed in at the level its eigenvalue's neighbour allows
// (7e-11 at Ny = 129), D is odd to its own round-off (5e-15 of its largest
// entry; its first rows are kept and mirrored, so rows still sum to zero). The
// boundary vectors belong to the same tables: kept from the unsymmetrised ones,
// w0 differs from D[0, int] V by 8e-11 of itself at Ny = 129.
struct SymTables {
  bool ok = false;
  int n_even = 0;
  std::vector<double> D, V, Vinv, lam, sgn, c0, cN, w0, wN;
};

inline SymTables symmetric_tables(const jsd_desc* d) {
  SymTables t;
  const int ny = d->ny, n = ny - 2;
  auto D = [&](int r, int c) { return d->D[(size_t)r * ny + c]; };
  auto V = [&](int r, int c) { return d->V[(size_t)r * n + c]; };
  auto W = [&](int r, int c) { return d->Vinv[(size_t)r * n + c]; };
  double dmax = 0, vmax = 0, wmax = 0;
  for (int i = 0; i < ny * ny; ++i) dmax = std::max(dmax, std::fabs(d->D[i]));
  for (int i = 0; i < n * n; ++i) {
    vmax = std::max(vmax, std::fabs(d->V[i]));
    wmax = std::max(wmax, std::fabs(d->Vinv[i]));
  }
  std::vector<int> order;
  for (int want : {1, -1})
    for (int j = 0; j < n; ++j)
      if (d->sgn[j] == want) order.push_back(j);
  if ((int)order.size() != n) return t;
  for (int j = 0; j < n; ++j) t.n_even += d->sgn[j] == 1;
  if (t.n_even != (n + 1) / 2) return t;
  // (comparisons written so that a NaN fails them)
  for (int r = 0; r < ny; ++r)
    for (int c = 0; c < ny; ++c)
      if (!(std::fabs(D(r, c) + D(ny - 1 - r, ny - 1 - c)) <= 1e-10 * dmax)) return t;
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c)
      if (!(std::fabs(V(r, c) - d->sgn[c] * V(n - 1 - r, c)) <= 1e-8 * vmax) ||
          !(std::fabs(W(r, c) - d->sgn[r] * W(r, n - 1 - c)) <= 1e-8 * wmax))
        return t;
  t.ok = true;
  t.D.resize((size_t)ny * ny);
  for (int r = 0; r < ny; ++r)
    for (int c = 0; c < ny; ++c)
      t.D[(size_t)r * ny + c] = 2 * r < ny - 1   ? D(r, c)
                                : 2 * r > ny - 1 ? -D(ny - 1 - r, ny - 1 - c)
                                                 : 0.5 * (D(r, c) - D(r, ny - 1 - c));
  t.V.resize((size_t)n * n);
  t.Vinv.resize((size_t)n * n);
  for (int j = 0; j < n; ++j) {
    const int o = order[j];
    for (int r = 0; r < n; ++r) {
      t.V[(size_t)r * n + j] = 0.5 * (V(r, o) + d->sgn[o] * V(n - 1 - r, o));
      t.Vinv[(size_t)j * n + r] = 0.5 * (W(o, r) + d->sgn[o] * W(o, n - 1 - r));
    }
    const double sg = d->sgn[o];
    t.lam.push_back(d->lam[o]);
    t.sgn.push_back(sg);
    // the boundary columns of D^2 mirror each other, so the new rows of V^-1 give
    // the definite part of (c0, cN); w0 and wN are formed again from the new D, V
    t.c0.push_back(0.5 * (d->c0[o] + sg * d->cN[o]));
    t.cN.push_back(sg * t.c0[j]);
    long double w = 0;
    for (int r = 0; r < n; ++r) w += (long double)t.D[r + 1] * t.V[(size_t)r * n + j];
    t.w0.push_back((double)w);
    t.wN.push_back(-sg * t.w0[j]);
  }
  return t;
}

// Halves of a whole operator A (mout x kin, row-major). fold / unfold: its
// columns / rows are points; otherwise they are eigen rows, the first n_even
// of them even. A column or row pair enters the halves through its even or odd
// combination, so whatever of A breaks the symmetry (round-off) drops out.
struct ParityHalves {
  std::vector<double> h[2];
  int M[2], K[2], part[2];
};
inline ParityHalves parity_halves(const double* A, int mout, int kin, bool fold, bool unfold, int n_even) {
  ParityHalves o;
  const int kh = (kin + 1) / 2, kp = kin / 2, mh = (mout + 1) / 2, mp = mout / 2;
  auto at = [&](int r, int k) { return (long double)A[(size_t)r * kin + k]; };
  // does the first half (even modes, or even output) read the even input?
  bool straight = false;
  if (!(fold && unfold)) {
    long double even = 0, odd = 0;
    const int rows = unfold ? mp : n_even, cols = fold ? kp : n_even;
    for (int r = 0; r < rows; ++r)
      for (int k = 0; k < cols; ++k) {
        const long double a = at(r, k), b = fold ? at(r, kin - 1 - k) : at(mout - 1 - r, k);
        even += (a + b) * (a + b);
        odd += (a - b) * (a - b);
      }
    straight = even >= odd;
  }  // D maps even to odd
  for (int p = 0; p < 2; ++p) {
    o.part[p] = straight ? p : 1 - p;
    o.M[p] = unfold ? (p ? mp : mh) : (p ? mout - n_even : n_even);
    o.K[p] = fold ? (o.part[p] ? kp : kh) : (o.part[p] ? kin - n_even : n_even);
    o.h[p].resize((size_t)o.M[p] * o.K[p]);
    const long double so = p ? -1 : 1, si = o.part[p] ? -1 : 1;
    for (int r = 0; r < o.M[p]; ++r)
      for (int k = 0; k < o.K[p]; ++k) {
        const int row = unfold ? r : (p ? n_even : 0) + r, col = fold ? k : (o.part[p] ? n_even : 0) + k;
        long double v = at(row, col), w = 1;
        if (fold) {
          v += si * at(row, kin - 1 - col);
          w *= col == kin - 1 - col ? 4 : 2;  // the mid-plane's sum is twice its value
        }
        if (unfold) {
          v += so * at(mout - 1 - row, col);
          if (fold) v += so * si * at(mout - 1 - row, kin - 1 - col);
          w *= 2;
        }
        o.h[p][(size_t)r * o.K[p] + k] = (double)(v / w);
      }
  }
  return o;
}

__device__ __forceinline__ void dmma16(double* c0, double* c1, double a0, double a1, double a2, double a3, double b0,
                                       double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Rows of a tile buffer. The k loop runs over whole steps: past the last column
// of a half it reads rows against zeros of A, which lie inside the tile when
// folding (kin >= 4 KS, which the plan asks for) and are zero rows after it
// otherwise (all entries then have the same kin).
inline int parity_rows(const ParityBatch& b, bool fold, int ksteps) {
  int rows = 0;
  for (int i = 0; i < b.count; ++i) {
    const ParityEntry& e = b.e[i];
    const int even = e.part[0] == 0 ? e.K[0] : e.K[1];
    rows = std::max(rows, fold ? e.kin : std::max(e.kin, even + 4 * ksteps));
  }
  return rows;
}

template <int W, int TM>
struct ParityCfg {
  static constexpr int RT = W * TM, KS = parity_ksteps(RT), THREADS = 64 * W;
  static constexpr int ACC = TM * (kParN / 8) * 2;  // results per lane
  static constexpr int XCH = W * ACC * 32;          // doubles handed between the halves' warps
  static constexpr int XROW = 2 * 2 * W * kParN;    // partial dot products of the extra rows
  static constexpr int XA = 2 * (4 * KS + 4);       // extra rows of the operator's halves
  // column groups of 8 per pass over k, and CTAs per SM: two CTAs where operand,
  // accumulators and about 36 more registers per thread allow it, if need be
  // with two passes over the tile
  static constexpr bool two(int ntp) { return (4 * TM * RT + 4 * TM * ntp + 36) * THREADS * 2 <= 65536; }
  static constexpr int NTP = !two(4) && two(2) ? 2 : 4;
  static constexpr int MIN_BLOCKS = two(NTP) ? 2 : 1;
  static size_t smem(int rows) { return sizeof(double) * (2 * (size_t)rows * kParBS + XCH + XROW + XA); }
};

template <int W, int TM, bool FOLD>
__global__ void __launch_bounds__(64 * W, ParityCfg<W, TM>::MIN_BLOCKS) k_parity(ParityBatch batch) {
  using Cfg = ParityCfg<W, TM>;
  constexpr int RT = Cfg::RT, KS = Cfg::KS, NT = kParN / 8, NTP = Cfg::NTP, BS = kParBS;
  extern __shared__ __align__(16) double psm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = warp / W, w = warp - half * W;
  const int g = lane >> 2, t = lane & 3;
  const int N = batch.N;
  const int ntiles = (N + kParN - 1) / kParN;
  const long long total = (long long)ntiles * batch.count;
  // (never empty: the grid has at most one CTA per tile)
  const int first = (int)(total * blockIdx.x / gridDim.x), last = (int)(total * (blockIdx.x + 1) / gridDim.x);

  const int bufd = batch.rows * BS;  // doubles per tile buffer
  double* xch = psm + 2 * bufd;      // [pass][W][...][32]
  double* xrow = xch + Cfg::XCH;     // [half][2 W warps][32]
  double* xas = xrow + Cfg::XROW;    // [half][4 KS + 4]

  // a thread copies one 16-byte column of the tile, every THREADS / 16th row
  constexpr int RSTEP = Cfg::THREADS / (kParN / 2);
  const int lr = tid / (kParN / 2), lc = (tid % (kParN / 2)) * 2;
  auto load_tile = [&](int ei, int n0, double* buf) {
    const int rows = batch.e[ei].kin;
    const bool ok = n0 + lc < N;
    const double* src = batch.e[ei].B + (ok ? (size_t)lr * N + n0 + lc : 0);
    const size_t step = ok ? (size_t)RSTEP * N : 0;
    double* dst = buf + lr * BS + lc;
#pragma unroll 4
    for (int r = lr; r < rows; r += RSTEP, src += step, dst += RSTEP * BS) cp_async16(dst, src, ok ? 16 : 0);
    cp_async_commit();
  };

  if (!FOLD)  // zero rows past the tile, never overwritten
    for (int i = batch.e[0].kin * BS + tid; i < bufd; i += Cfg::THREADS) psm[i] = psm[bufd + i] = 0.0;

  double a[TM][KS], ax[TM];  // operand fragments; the extra column's entries of rows g
  const double* loaded = nullptr;
  auto load_operator = [&](const ParityEntry& e) {
    loaded = e.a[half];
    const double* src = loaded + (size_t)w * TM * KS * 32 + lane;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
#pragma unroll
      for (int s = 0; s < KS; ++s) a[i][s] = src[(i * KS + s) * 32];
      ax[i] = loaded[RT * KS * 32 + (w * TM + i) * 8 + g];
    }
    for (int k = w * 32 + lane; k < e.K[half]; k += W * 32)
      xas[half * (4 * KS + 4) + k] = loaded[RT * KS * 32 + 8 * RT + k];
  };
  int ei = first / ntiles, n0 = (first - ei * ntiles) * kParN, buf = 0;
  load_operator(batch.e[ei]);  // fixed at plan creation: needs no earlier kernel
  pdl();
  load_tile(ei, n0, psm);
  for (int tile = first; tile < last; ++tile) {
    const double* Bs = psm + buf * bufd;
    const ParityEntry& e = batch.e[ei];
    const int M = e.M[half], K = e.K[half], kin = e.kin, mout = e.mout;
    if (e.a[half] != loaded) {
      __syncthreads();  // the extra rows of the last operator are no longer read
      load_operator(e);
    }
    cp_async_wait<0>();
    __syncthreads();  // the tile is here, and every warp is done with the other buffer and with xch
    const int ein = n0 + kParN < N ? ei : ei + 1, nn = n0 + kParN < N ? n0 + kParN : 0;
    buf ^= 1;
    if (tile + 1 < last) load_tile(ein, nn, psm + buf * bufd);

    // the row beyond the tiles (outputs on the points only): every warp sums a
    // stretch of k for all 32 columns, lane = column; warp 0 adds them up below
    if (batch.unfold && (mout + 1) / 2 > 8 * RT) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int Kh = e.K[h], ph = e.part[h];
        const double* xb = Bs + (FOLD || ph == 0 ? 0 : (kin - Kh) * BS) + lane;
        const double* xm = Bs + (kin - 1) * BS + lane;
        const double* xa = xas + h * (4 * KS + 4);
        double x = 0.0;
        if (e.M[h] > 8 * RT) {
          const int ke = Kh * (warp + 1) / (2 * W);
#pragma unroll 4
          for (int k = Kh * warp / (2 * W); k < ke; ++k) {
            double b = xb[k * BS];
            if (FOLD) b = fma(ph ? -1.0 : 1.0, xm[-k * BS], b);
            x = fma(xa[k], b, x);
          }
        }
        xrow[(h * 2 * W + warp) * kParN + lane] = x;
      }
    }

    // rows of this lane's fragments: 4 s + t from b0 (and, folding, its mirror from b1)
    const int part = e.part[half];
    const double* b0 = Bs + (FOLD || part == 0 ? t : kin - K + t) * BS + g;
    const double* b1 = Bs + (kin - 1 - t) * BS + g;
    const double sign = part ? -1.0 : 1.0;
    double* C = e.C + (batch.unfold || !half ? 0 : (size_t)(mout - M) * N) + n0;
    const int r0 = w * TM * 8 + g;
    const bool full = n0 + kParN <= N;  // every column of the tile exists
#pragma unroll
    for (int j0 = 0; j0 < NT; j0 += NTP) {
      double acc[TM][NTP][2];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < NTP; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
      if (K > 8 * RT) {
#pragma unroll
        for (int j = 0; j < NTP; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int o = 8 * (j0 + j) + 2 * t - g + q;
            double bx = b0[(8 * RT - t) * BS + o];
            if (FOLD) bx = fma(sign, b1[o - (8 * RT - t) * BS], bx);
#pragma unroll
            for (int i = 0; i < TM; ++i) acc[i][j][q] = ax[i] * bx;
          }
      }
#pragma unroll
      for (int s = 0; s < KS; s += 2) {
        double b[2][NTP];
#pragma unroll
        for (int d = 0; d < 2; ++d) {
#pragma unroll
          for (int j = 0; j < NTP; ++j) {
            b[d][j] = b0[4 * (s + d) * BS + 8 * (j0 + j)];
            if (FOLD) b[d][j] = fma(sign, b1[8 * (j0 + j) - 4 * (s + d) * BS], b[d][j]);
          }
        }
#pragma unroll
        for (int i = 0; i < TM - 1; i += 2)
#pragma unroll
          for (int j = 0; j < NTP; ++j)
            dmma16(acc[i][j], acc[i + 1][j], a[i][s], a[i + 1][s], a[i][s + 1], a[i + 1][s + 1], b[0][j], b[1][j]);
        if (TM % 2) {
#pragma unroll
          for (int d = 0; d < 2; ++d)
#pragma unroll
            for (int j = 0; j < NTP; ++j)
              dmma(acc[TM - 1][j][0], acc[TM - 1][j][1], a[TM - 1][s + d], b[d][j]);
        }
      }
      if (!batch.unfold) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          double* Ci = C + (size_t)(r0 + 8 * i) * N + 8 * j0 + 2 * t;
          if (r0 + 8 * i < M) {
#pragma unroll
            for (int j = 0; j < NTP; ++j)
              if (full || n0 + 8 * (j0 + j) + 2 * t < N)
                *reinterpret_cast<double2*>(Ci + 8 * j) = make_double2(acc[i][j][0], acc[i][j][1]);
          }
        }
        continue;
      }
      // c_i = S_i + T_i, c_{n-1-i} = S_i - T_i: the two warps of a row group hand
      // each other half of the pass's column groups (half 0 keeps the first HJ),
      // then both combine and store
      constexpr int HJ = NTP / 2;
      double* xc = xch + ((size_t)(j0 / NTP) * W + w) * (2 * TM * HJ * 2 * 32) + lane;
      const int pairs = mout / 2;  // rows with a mirror of their own; row `pairs` is the mid-plane when mout is odd
      auto hand = [&](auto H) {
        constexpr int h = decltype(H)::value;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < HJ; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) xc[(((h * TM + i) * HJ + j) * 2 + q) * 32] = acc[i][(1 - h) * HJ + j][q];
      };
      auto combine = [&](auto H) {
        constexpr int h = decltype(H)::value;
        const int col = n0 + 8 * (j0 + h * HJ) + 2 * t;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const int r = r0 + 8 * i;
          double* Cu = C + (size_t)r * N + (col - n0);
          double* Cd = C + (size_t)(mout - 1 - r) * N + (col - n0);
#pragma unroll
          for (int j = 0; j < HJ; ++j) {
            double o[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) o[q] = xc[((((1 - h) * TM + i) * HJ + j) * 2 + q) * 32];
            const double* m = acc[i][h * HJ + j];
            double2 up = make_double2(m[0] + o[0], m[1] + o[1]);
            double2 dn = h ? make_double2(o[0] - m[0], o[1] - m[1]) : make_double2(m[0] - o[0], m[1] - o[1]);
            if (full || col + 8 * j < N) {
              if (batch.accumulate) {
                if (r < mout - pairs) up = cadd(up, *reinterpret_cast<double2*>(Cu + 8 * j));
                if (r < pairs) dn = cadd(dn, *reinterpret_cast<double2*>(Cd + 8 * j));
              }
              if (r < mout - pairs) *reinterpret_cast<double2*>(Cu + 8 * j) = up;
              if (r < pairs) *reinterpret_cast<double2*>(Cd + 8 * j) = dn;
            }
          }
        }
      };
      using H0 = std::integral_constant<int, 0>;
      using H1 = std::integral_constant<int, 1>;
      if (half) hand(H1{});
      else hand(H0{});
      __syncthreads();
      if (half) combine(H1{});
      else combine(H0{});
      if (j0 + NTP == NT && warp == 0 && mout - pairs > 8 * RT && n0 + lane < N) {
        double S = 0.0, T = 0.0;
#pragma unroll
        for (int q = 0; q < 2 * W; ++q) {
          S += xrow[q * kParN + lane];
          T += xrow[(2 * W + q) * kParN + lane];
        }
        double* Cu = C + (size_t)(8 * RT) * N + lane;
        double* Cd = C + (size_t)(mout - 1 - 8 * RT) * N + lane;
        *Cu = S + T + (batch.accumulate ? *Cu : 0.0);
        if (pairs > 8 * RT) *Cd = S - T + (batch.accumulate ? *Cd : 0.0);
      }
    }
    ei = ein;
    n0 = nn;
  }
}

}  // namespace jsd
