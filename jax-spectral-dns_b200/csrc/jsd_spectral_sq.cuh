// Transform kernels of the nonlinear terms on register-resident square FFTs
// (jsd_fftsq.cuh), used when the plan's FFT lengths are S * S. Same three
// passes and the same intermediate layouts as the shared-memory kernels in
// jsd_spectral.cuh, with one line per group of S lanes:
//   k_zinv_sq : group per (y, kx): Hermitian part, 9 (18) inverse z transforms
//               (k_zinv_staged: large boxes, input rows through shared memory);
//   k_xmid_sq : mixed form: block per (y, run of z columns), group per z column:
//               packed pairs of fields through inverse x transforms, the products in
//               registers (every lane owns the same x positions in every line),
//               2 forward x transforms (k_xmid_h2: the line on 2 S lanes);
//   k_xmid_park : the same for the FP64 form, finished components in shared
//               memory, columns across planes (k_xmid_dual_sq: the dual's);
//   k_zfwd_sq : group per (y, kx) on three warps, one forward z transform each,
//               then truncation and the spectral combinations of write_terms.
// All sizes are compile-time, so index arithmetic is shifts and multiplies,
// and the only synchronisation inside a transform is a __syncwarp.
#pragma once

#include <type_traits>

#include "jsd_fftsq.cuh"
#include "jsd_gemm.cuh"
#include "jsd_spectral.cuh"

namespace jsd {

constexpr int kSqWarps = 4;  // warps per block

// Lane roles. HW: with two groups per warp (11 <= S <= 16) each group takes
// its own half-warp (lanes 16 gi + t, t < S): a 64-bit shared-memory request
// is served per half-warp, so the groups' accesses never share a bank cycle.
// Otherwise 32 / S groups of S consecutive lanes, the last 32 - G S idle.
template <int S, bool HW = true>
struct SqLane {
  static constexpr int G = 32 / S;                        // line groups per warp
  static constexpr int W = (HW && G == 2) ? 16 : S;       // lane stride of the groups
  int warp, gi, t;
  bool live;  // lane belongs to a group (the other lanes idle)
  __device__ __forceinline__ SqLane() {
    const int lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    gi = lane / W;
    t = lane - gi * W;
    live = gi < G && t < S;
    if (!live) {
      gi = 0;
      if (HW) t = 0;
    }
  }
};

// src.f[i] by selects over the parameter array (a runtime index into the
// kernel parameter would copy the array to local memory)
__device__ __forceinline__ const double2* zinv_field(const ZinvSrc& src, int i) {
  const double2* r = src.f[0];
#pragma unroll
  for (int k = 1; k < 12; ++k)
    if (i == k) r = src.f[k];
  return r;
}

// ---------------------------------------------------------------------------
// inverse z pass (same output as k_zinv)
// ---------------------------------------------------------------------------
template <typename C, int S>
__global__ void __launch_bounds__(kSqWarps * 32) k_zinv_sq(Geo g, const C* __restrict__ twtab, ZinvSrc src,
                                                           C* inter) {
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, XB = sq_xbuf<S>();
  // The two forms keep their best measured shapes: FP32 lines on half-warp
  // groups with the next field's rows prefetched into L2 and per-position
  // bound tests resolved at compile time; FP64 lines on consecutive-lane
  // groups with plain bound tests and no prefetch (the compiler then keeps
  // all 2 S loads of a line in flight; with the FP32 shape the FP64 pass
  // took 175 us instead of 109 us cold at 128 x 129 x 128).
  constexpr bool F32 = sizeof(C) == sizeof(float2);
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const SqLane<S, F32> ln;
  C* xb = reinterpret_cast<C*>(sq_raw) + (ln.warp * SqLane<S>::G + ln.gi) * XB;
  const int K1 = g.kx_max + 1, K = g.kz_max;
  const int pair = (blockIdx.x * kSqWarps + ln.warp) * SqLane<S>::G + ln.gi;
  const bool act = ln.live && pair < g.ny * K1;
  const int y = act ? pair / K1 : 0;
  const int kx = act ? pair - y * K1 : 0;
  C tw[S - 1];
  sq_twiddles<S>(tw, twtab, ln.t);
  pdl();
  // the group's two rows (kx and -kx) of field `i` into L2: the loads of a
  // field then wait for L2, not DRAM (one field ahead; rows are 16-byte
  // aligned and mz * 16 bytes long)
  auto prefetch = [&](int i) {
    if (F32 && act && ln.t == 0 && i < 6 * src.nsets) {
      const double2* f = zinv_field(src, i);
      l2_prefetch(f + sidx(g, y, kx, 0), (unsigned)(g.mz * sizeof(double2)));
      if (kx) l2_prefetch(f + sidx(g, y, g.mx - kx, 0), (unsigned)(g.mz * sizeof(double2)));
    }
  };
  const int step = gridDim.y;
  prefetch(blockIdx.y + step);
#pragma unroll 1
  for (int i = blockIdx.y; i < 6 * src.nsets; i += step) {
    const int set = i / 6, fi = i - 6 * set;
    const double2* f = zinv_field(src, i);
    prefetch(i + 2 * step);
    C x[S], xz[S];
    // K < N / 2: positions below N / 2 hold kz >= 0 modes, those above kz < 0
#pragma unroll
    for (int m = 0; m < S; ++m) {
      const int p = ln.t + S * m;
      const bool below = F32 && S * m + S - 1 < N / 2, above = F32 && S * m >= N / 2;
      const bool lo = !above && p <= K, hi = !below && p >= N - K;
      const int kz = below ? p : above ? p - N : lo ? p : p - N;
      const C v = (act && (lo || hi)) ? to_c<C>(sym_at(g, f, y, kx, kz)) : cmake<C>(0, 0);
      x[m] = v;
      xz[m] = cmul_ik(v, (Rl)(kz * g.az));
    }
    sq_fft<S, true>(x, tw, xb, ln.t, ln.live);
    C* o = inter + (((size_t)(set * kZinvLines + fi) * g.ny + y) * K1 + kx) * N + ln.t;
    if (act) {
#pragma unroll
      for (int m = 0; m < S; ++m) o[S * m] = x[m];
    }
    if (fi < 3) {
      sq_fft<S, true>(xz, tw, xb, ln.t, ln.live);
      C* oz = inter + (((size_t)(set * kZinvLines + 6 + fi) * g.ny + y) * K1 + kx) * N + ln.t;
      if (act) {
#pragma unroll
        for (int m = 0; m < S; ++m) oz[S * m] = xz[m];
      }
    }
  }
}

template <typename C, int S>
size_t zinv_sq_smem() {
  return sizeof(C) * (size_t)kSqWarps * SqLane<S>::G * sq_xbuf<S>();
}

// ---------------------------------------------------------------------------
// inverse z pass, input rows staged (same output as k_zinv_sq, bit for bit): a
// group's two rows (kx and -kx) of the next field come by cp.async into shared
// memory while the transforms of the current one run, so a field's loads wait
// for nothing; twiddles come from a shared table.
// Bound: HBM, 4.5 TB/s at 129 x 129 modes x 129 planes in FP64 (what is left:
// eight warps per SM alternate between transforms and line stores). Measured
// there 98 us, 119 with k_zinv_sq's loads into registers; FP32 69 from 93; FP64
// 161 x 161 x 145 169 from 257 (there the register loads spill).
// The rows' way through shared memory costs 2 us where the fields lie in the
// L2, so k_zinv_sq keeps boxes of fewer than kStagedMin entries per field (all
// runs; six fields in and nine line sets out then share the L2): steps of 65 x
// 65 x 89 modes 405 against 407 us, 29 x 19 x 85 150 against 158; above the line
// 65 x 65 x 129 578 against 560, 97 x 97 x 97 1104 against 1061, four runs of 41 x
// 97 x 41 623 against 600. FP64 S <= 7 stays with k_zinv_sq (twelve runs of 33 x 97
// x 33 1166 against 1176), S = 16 is always staged (33 x 33 x 161 298 against 283).
// ---------------------------------------------------------------------------
constexpr size_t kStagedMin = 1u << 19;

template <typename C, int S>
struct ZinvStaged {
  static constexpr bool F32 = sizeof(C) == sizeof(float2);
  using Lane = SqLane<S, F32>;
  static constexpr int GROUPS = kSqWarps * Lane::G, XB = sq_xbuf<S>(), TAB = (S - 1) * sq_tw_stride(S);
  // whether the kernel is built for the side, and whether it then takes every box
  static constexpr bool EVER = F32 ? S >= 7 : S >= 8, ALWAYS = !F32 && S == 16;
  // registers: x, i kz x and the DFT's temporaries (238 at S = 14 in FP64: with
  // three blocks it spills, 136 against 98 us)
  static constexpr int BLOCKS = F32 ? 4 : S <= 10 ? 3 : 2;
  // elements between the groups' row pairs: with consecutive-lane groups the
  // lanes of a warp read one run of slots
  static __host__ __device__ int row_stride(int mz) { return 2 * mz + ((S - 2 * mz) % 8 + 8) % 8; }
  static size_t smem(const Geo& g) {
    return sizeof(double2) * (size_t)GROUPS * row_stride(g.mz) + sizeof(C) * ((size_t)GROUPS * XB + TAB);
  }
};

template <typename C, int S>
__global__ void __launch_bounds__(kSqWarps * 32, ZinvStaged<C, S>::BLOCKS) k_zinv_staged(
    Geo g, const C* __restrict__ twtab, ZinvSrc src, C* inter) {
  using Z = ZinvStaged<C, S>;
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, TS = sq_tw_stride(S);
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const typename Z::Lane ln;
  const int group = ln.warp * Z::Lane::G + ln.gi, mz = g.mz;
  double2* ra = reinterpret_cast<double2*>(sq_raw) + group * Z::row_stride(mz);
  C* xb = reinterpret_cast<C*>(reinterpret_cast<double2*>(sq_raw) + Z::GROUPS * Z::row_stride(mz));
  C* tab = xb + Z::GROUPS * Z::XB;
  xb += group * Z::XB;
  for (int e = threadIdx.x; e < Z::TAB; e += kSqWarps * 32) {
    const int j = e / TS + 1, t = e % TS;
    if (t < S) tab[e] = twtab[t * j];
  }
  const int K1 = g.kx_max + 1, K = g.kz_max;
  const int pair = blockIdx.x * Z::GROUPS + group;
  const bool act = ln.live && pair < g.ny * K1;
  const int y = act ? pair / K1 : 0;
  const int kx = act ? pair - y * K1 : 0;
  const double2* rb = kx ? ra + mz : ra;  // the row of -kx
  const size_t oa = sidx(g, y, kx, 0), ob = sidx(g, y, kx ? g.mx - kx : 0, 0);
  // the group's rows of field i, by its own lanes
  auto stage = [&](int i) {
    if (act && i < 6 * src.nsets) {
      const double2* f = zinv_field(src, i);
#pragma unroll
      for (int m = 0; m < S; ++m) {
        const int p = ln.t + S * m;
        if (p < mz) {
          cp_async16(ra + p, f + oa + p, 16);
          if (kx) cp_async16(ra + mz + p, f + ob + p, 16);
        }
      }
    }
    cp_async_commit();
  };
  pdl();
  stage(0);
  __syncthreads();  // the twiddle table
#pragma unroll 1
  for (int i = 0; i < 6 * src.nsets; ++i) {
    const int set = i / 6, fi = i - 6 * set;
    cp_async_wait<0>();
    __syncwarp();
    int t = ln.t;
    asm volatile("" : "+r"(t));  // positions and wavenumbers formed here, not kept over the loop
    C x[S], xz[S];
    // K < N / 2: positions below N / 2 hold kz >= 0 modes, those above kz < 0
#pragma unroll
    for (int m = 0; m < S; ++m) {
      const int p = t + S * m;
      const bool below = S * m + S - 1 < N / 2, above = S * m >= N / 2;
      const bool lo = !above && p <= K, hi = !below && p >= N - K;
      const int kz = below ? p : above ? p - N : lo ? p : p - N;
      C v = cmake<C>(0, 0);
      if (act && (lo || hi)) {
        const double2 a = ra[mode_pos(kz, mz)], b = rb[mode_pos(-kz, mz)];
        v = to_c<C>(make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y)));
      }
      x[m] = v;
      xz[m] = cmul_ik(v, (Rl)(kz * g.az));
    }
    __syncwarp();  // every lane has read the rows
    stage(i + 1);
    sq_fft_tab<S, true>(x, tab, xb, ln.t, ln.live);
    C* o = inter + (((size_t)(set * kZinvLines + fi) * g.ny + y) * K1 + kx) * N + ln.t;
    if (act) {
#pragma unroll
      for (int m = 0; m < S; ++m) o[S * m] = x[m];
    }
    if (fi < 3) {
      sq_fft_tab<S, true>(xz, tab, xb, ln.t, ln.live);
      C* oz = inter + (((size_t)(set * kZinvLines + 6 + fi) * g.ny + y) * K1 + kx) * N + ln.t;
      if (act) {
#pragma unroll
        for (int m = 0; m < S; ++m) oz[S * m] = xz[m];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// forward z pass (same output as k_zfwd)
// ---------------------------------------------------------------------------
// Truncation and spectral combinations of a group's three transformed lines
// lb[f * XB + position], by threads j, j + stride, ... of those that share it
template <typename C, int S>
__device__ __forceinline__ void zfwd_outputs(const Geo& g, const C* lb, int y, int kx, int j, int stride,
                                             double2* __restrict__ q, double2* __restrict__ H1,
                                             double2* __restrict__ hg, double2* __restrict__ conv00) {
  constexpr int N = S * S, XB = sq_xbuf<S>();
  const int K = g.kx_max;
  const double cf = g.c_fwd;
  auto getF = [&](int f, int kz) -> double2 {
    const C v = lb[f * XB + (kz >= 0 ? kz : N + kz)];
    return make_double2((double)v.x * cf, (double)v.y * cf);
  };
  // rows this group owns: kx itself; -kx for 1 <= kx < K; the -K slot when kx = K
  int rows[2];
  int nrows = 1;
  rows[0] = kx;
  if (kx >= 1 && kx < K) rows[nrows++] = g.mx - kx;
  if (kx == K) rows[nrows++] = K + 1;
  for (int i = j; i < nrows * g.mz; i += stride) {
    const int rr = i >= g.mz ? 1 : 0;
    const int iz = i - rr * g.mz;
    const int ix = rows[rr];
    int sx, sz;
    bool cj;
    truncation_source(g, ix, iz, sx, sz, cj);
    double2 h[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const double2 val = (sx >= 0) ? getF(f, sz) : cconj(getF(f, -sz));
      h[f] = cj ? cconj(val) : val;
    }
    write_terms(g, y, ix, iz, h[0], h[1], h[2], q, H1, hg, conv00);
  }
}

// Three warps per G line groups, each transforming one of a group's three lines;
// then all of a group's lanes form the outputs. Bound: HBM in large boxes (181.9
// MB in 41 us at 129 x 129 modes x 129 planes), one transform and the exchange in
// small ones. One warp that transforms the three lines in turn and forms the
// outputs takes 45 and, at 33 x 33 x 65, 10.7 us against 8.7; steps: 49 x 97 x 49
// 336 -> 296 us, 161 x 145 x 161 3786 -> 3742, 129 x 129 x 129 2117 -> 2105.
constexpr int kZfwdThreads = 96;

template <typename C, int S>
__global__ void __launch_bounds__(kZfwdThreads) k_zfwd_sq(Geo g, const C* __restrict__ twtab,
                                                          const C* out3, double2* q,
                                                          double2* H1, double2* hg,
                                                          double2* conv00) {
  constexpr int N = S * S, XB = sq_xbuf<S>();
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const SqLane<S> ln;
  C* lb = reinterpret_cast<C*>(sq_raw) + ln.gi * 3 * XB;
  const int K1 = g.kx_max + 1, f = ln.warp;
  const int pair = blockIdx.x * SqLane<S>::G + ln.gi;
  const bool act = ln.live && pair < g.ny * K1;
  const int y = act ? pair / K1 : 0;
  const int kx = act ? pair - y * K1 : 0;
  C tw[S - 1];
  sq_twiddles<S>(tw, twtab, ln.t);
  pdl();
  const C* src = out3 + (((size_t)f * g.ny + y) * K1 + kx) * N + ln.t;
  C x[S];
#pragma unroll
  for (int m = 0; m < S; ++m) x[m] = act ? src[S * m] : cmake<C>(0, 0);
  sq_fft<S, false>(x, tw, lb + f * XB, ln.t, ln.live);
  if (ln.live) {
#pragma unroll
    for (int m = 0; m < S; ++m) lb[f * XB + ln.t + S * m] = x[m];
  }
  __syncthreads();
  if (act) zfwd_outputs<C, S>(g, lb, y, kx, ln.t + S * f, 3 * S, q, H1, hg, conv00);
}

template <typename C, int S>
size_t zfwd_sq_smem() {
  return sizeof(C) * (size_t)SqLane<S>::G * 3 * sq_xbuf<S>();
}

// ---------------------------------------------------------------------------
// x pass with the products
// ---------------------------------------------------------------------------
// Shared-memory layout of the x pass, chosen so that every 64-bit request is
// served at the minimum number of wavefronts:
//   input tile [field][zl][kx], row stride KP: the staging copies (8 z columns
//     x 2 rows per half-warp) need KP = 2 mod 16 when ZC = 8; with more columns
//     per block an odd KP;
//   output tile [row][zl] with the 8 z columns of a row swizzled by
//     (row / 2) mod 8: the lanes of a group write 14 consecutive rows of one
//     column, the store reads 2 rows of 8 columns per half-warp;
//   twiddles lane-major (sq_tw_stride).
template <int ZC>
__host__ __device__ __forceinline__ int xsq_kp(int k1) {
  return ZC == 8 ? k1 + ((2 - k1) % 16 + 16) % 16 : k1 | 1;
}

template <typename C, int S>
struct XmidSq {
  static constexpr int G = SqLane<S>::G;
  static constexpr int ZC = kSqWarps * G;  // z columns per block
  static __host__ __device__ int kp(int k1) { return xsq_kp<ZC>(k1); }
  static constexpr int twn = (S - 1) * sq_tw_stride(S);  // twiddle table entries
  static size_t smem(const Geo& g, int nfields) {
    const int K1 = g.kx_max + 1;
    return sizeof(C) * ((size_t)nfields * ZC * kp(K1) + 3 * (size_t)K1 * ZC + (size_t)kSqWarps * G * sq_xbuf<S>() +
                        (size_t)twn);
  }
};

// slot of (row, z column) in the output tile
template <int ZC>
__device__ __forceinline__ int xsq_oslot(int row, int zl) {
  return ZC == 8 ? row * 8 + (zl ^ ((row >> 1) & 7)) : row * ZC + zl;
}

// Block-wide: the lane-major twiddle table from the table w_N^e, e = 0..N-1.
template <typename C, int S>
__device__ __forceinline__ void xsq_twiddle_table(C* stab, const C* __restrict__ twtab) {
  constexpr int TS = sq_tw_stride(S);
  for (int e = threadIdx.x; e < XmidSq<C, S>::twn; e += blockDim.x) {
    const int j = e / TS + 1, t = e - (j - 1) * TS;
    stab[e] = t < S ? twtab[t * j] : cmake<C>(0, 0);
  }
}

// 8- or 16-byte asynchronous copy global -> shared (zero fill when !ok)
template <typename C>
__device__ __forceinline__ void cp_async_elem(C* smem, const C* gmem, bool ok) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if constexpr (sizeof(C) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(ok ? 8 : 0));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(ok ? 16 : 0));
}

// Block-wide: start asynchronous copies of the input tile [f][zl][kx]
// (kx >= 0) of nfields fields; the caller waits (cp_async_wait<0>) and syncs.
template <typename C, int ZC>
__device__ __forceinline__ void xsq_stage_tile(const Geo& g, const C* __restrict__ inter, C* tile, int nfields,
                                               int y, int z0) {
  constexpr int RSTEP = kSqWarps * 32 / ZC;  // tile rows per pass of the block
  const int K1 = g.kx_max + 1, KP = xsq_kp<ZC>(K1);
  if (threadIdx.x < RSTEP * ZC) {
    const int zl = threadIdx.x % ZC;
    const int z = z0 + zl;
    const bool zok = z < g.pz;
    const C* base = inter + (size_t)y * K1 * g.pz + (zok ? z : 0);
    const size_t fstride = (size_t)g.ny * K1 * g.pz;
    int row = threadIdx.x / ZC;
    int f = row / K1, kx = row - (row / K1) * K1;
    for (; row < nfields * K1; row += RSTEP) {
      cp_async_elem(tile + (f * ZC + zl) * KP + kx, base + f * fstride + (size_t)kx * g.pz, zok);
      kx += RSTEP;
      while (kx >= K1) {
        kx -= K1;
        ++f;
      }
    }
  }
  cp_async_commit();
}

// Packed line a + i b of the column's fields (fa, fb), x-derivatives on request,
// at positions t + S m (same packing as fill_pair).
template <typename C, int S>
__device__ __forceinline__ void xsq_fill(const Geo& g, const C* tile, int zl, int t, bool live, C* x, int fa,
                                         bool dxa, int fb, bool dxb) {
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, ZC = XmidSq<C, S>::ZC;
  const int K = g.kx_max, KP = XmidSq<C, S>::kp(K + 1);
  const C* ta = tile + (fa * ZC + zl) * KP;
  const C* tb = tile + (fb * ZC + zl) * KP;
  // K < N / 2, so positions below N / 2 can only be kx >= 0 modes and those
  // above only kx < 0 modes: after unrolling, each m but a straddling one
  // needs one bound check and no select of the packing
#pragma unroll
  for (int m = 0; m < S; ++m) {
    const int p = t + S * m;
    const bool below = S * m + S - 1 < N / 2, above = S * m >= N / 2;
    const bool lo = !above && p <= K, hi = !below && p >= N - K;
    C out = cmake<C>(0, 0);
    if (live && (lo || hi)) {
      const int kx = below ? p : above ? N - p : lo ? p : N - p;
      C A = ta[kx], B = tb[kx];
      const Rl k = (Rl)(kx * g.ax);
      if (dxa) A = cmul_ik(A, k);
      if (dxb) B = cmul_ik(B, k);
      if (m == 0 && p == 0) out = cmake<C>(A.x, B.x);
      else if (below || (!above && lo)) out = cmake<C>(A.x - B.y, A.y + B.x);
      else out = cmake<C>(A.x + B.y, B.x - A.y);
    }
    x[m] = out;
  }
}

// Forward transforms of (h0 + i h1) and (h2 + 0 i) of the column, kx >= 0
// outputs to the block's output tile [f][kx][zl].
template <typename C, int S>
__device__ __forceinline__ void xsq_forward(const Geo& g, const C* tab, C* xb, C* otile, int zl, int t, bool live,
                                            C* z01, C* z2) {
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, ZC = XmidSq<C, S>::ZC;
  const int K = g.kx_max, K1 = K + 1;
  sq_fft_tab<S, false>(z01, tab, xb, t, live);
  sq_fft_tab<S, false>(z2, tab, xb, t, live);
  if (live) {
#pragma unroll
    for (int m = 0; m < S; ++m) {
      xb[t + S * m] = z01[m];
      const int p = t + S * m;
      if (p <= K) otile[xsq_oslot<ZC>(2 * K1 + p, zl)] = z2[m];
    }
  }
  __syncwarp();
  if (live) {
    const Rl half = (Rl)0.5;
    for (int kx = t; kx <= K; kx += S) {
      const C a = xb[kx];
      const C b = xb[kx == 0 ? 0 : N - kx];
      // H0 = (Z[k] + conj Z[-k]) / 2, H1 = (Z[k] - conj Z[-k]) / (2 i)
      otile[xsq_oslot<ZC>(0 * K1 + kx, zl)] = cmake<C>(half * (a.x + b.x), half * (a.y - b.y));
      otile[xsq_oslot<ZC>(1 * K1 + kx, zl)] = cmake<C>(half * (a.y + b.y), -half * (a.x - b.x));
    }
  }
}

// Block-wide: coalesced store of the output tile.
template <typename C, int ZC>
__device__ __forceinline__ void xsq_store(const Geo& g, const C* otile, C* __restrict__ out3, int y, int z0) {
  constexpr int RSTEP = kSqWarps * 32 / ZC;
  const int K1 = g.kx_max + 1;
  if (threadIdx.x >= RSTEP * ZC) return;
  const int zl = threadIdx.x % ZC;
  const int z = z0 + zl;
  if (z >= g.pz) return;
  C* base = out3 + (size_t)y * K1 * g.pz + z;
  const size_t fstride = (size_t)g.ny * K1 * g.pz;
  int row = threadIdx.x / ZC;
  int f = row / K1, kx = row - (row / K1) * K1;
  for (; row < 3 * K1; row += RSTEP) {
    base[f * fstride + (size_t)kx * g.pz] = otile[xsq_oslot<ZC>(row, zl)];
    kx += RSTEP;
    while (kx >= K1) {
      kx -= K1;
      ++f;
    }
  }
}

// Resident blocks per SM the FP32 x pass is compiled for (registers capped at
// 168 per lane: a little spilling, 12 warps per SM instead of 8).
constexpr int kXsqBlocks = 3;

// NS / perturbation products of the mixed form (the FP64 form runs k_xmid_park), as in k_xmid:
//   hel_i = -lam (u . grad) u_i + lam/2 (div u) u_i - U d_x u_i - delta_i0 (v U' - (div u) U / 2)
template <typename C, int S>
__global__ void __launch_bounds__(kSqWarps * 32, kXsqBlocks) k_xmid_sq(Geo g, const C* __restrict__ twtab,
                                                           const C* inter, C* out3,
                                                           const double* ubase,
                                                           const double* dubase, double lam_d) {
  static_assert(sizeof(C) == sizeof(float2), "FP64 lines: k_xmid_park");
  pdl();
  using Rl = typename real_of<C>::type;
  constexpr int G = SqLane<S>::G, ZC = XmidSq<C, S>::ZC, XB = sq_xbuf<S>();
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const int K1 = g.kx_max + 1, KP = XmidSq<C, S>::kp(K1);
  C* tile = reinterpret_cast<C*>(sq_raw);
  C* otile = tile + kZinvLines * ZC * KP;
  const SqLane<S> ln;
  C* xb = otile + 3 * K1 * ZC + (ln.warp * G + ln.gi) * XB;
  const int z0 = blockIdx.x * ZC, y = blockIdx.y;
  const int zl = ln.warp * G + ln.gi;
  const Rl ub = ubase ? (Rl)ubase[y / g.nb] : (Rl)0;
  const Rl dub = dubase ? (Rl)dubase[y / g.nb] : (Rl)0;
  const Rl c = (Rl)g.c_inv, lam = (Rl)lam_d, half = (Rl)0.5;
  xsq_stage_tile<C, ZC>(g, inter, tile, kZinvLines, y, z0);
  // twiddle table in shared memory (read by stage 1 of every transform)
  C* stab = otile + 3 * K1 * ZC + kSqWarps * G * XB;
  xsq_twiddle_table<C, S>(stab, twtab);
  cp_async_wait<0>();
  __syncthreads();
  const bool live = ln.live;
  const int t = ln.t;
  // intermediate: 0 u, 1 v, 2 w, 3 du/dy, 4 dv/dy, 5 dw/dy, 6 du/dz, 7 dv/dz, 8 dw/dz
  Rl U[S], V[S], W[S], DIV[S], A0[S], A1[S], A2[S];
  C x[S];
  xsq_fill<C, S>(g, tile, zl, t, live, x, 0, false, 1, false);  // (u, v)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#pragma unroll
  for (int m = 0; m < S; ++m) {
    U[m] = x[m].x * c;
    V[m] = x[m].y * c;
  }
  xsq_fill<C, S>(g, tile, zl, t, live, x, 2, false, 0, true);  // (w, du/dx)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#pragma unroll
  for (int m = 0; m < S; ++m) {
    W[m] = x[m].x * c;
    const Rl dxu = x[m].y * c;
    DIV[m] = dxu;
    A0[m] = lam * U[m] * dxu + ub * dxu;
  }
  xsq_fill<C, S>(g, tile, zl, t, live, x, 1, true, 2, true);  // (dv/dx, dw/dx)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#pragma unroll
  for (int m = 0; m < S; ++m) {
    const Rl dxv = x[m].x * c, dxw = x[m].y * c;
    A1[m] = lam * U[m] * dxv + ub * dxv;
    A2[m] = lam * U[m] * dxw + ub * dxw;
  }
  xsq_fill<C, S>(g, tile, zl, t, live, x, 4, false, 8, false);  // (dv/dy, dw/dz)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#pragma unroll
  for (int m = 0; m < S; ++m) {
    const Rl dyv = x[m].x * c, dzw = x[m].y * c;
    DIV[m] += dyv + dzw;
    A1[m] += lam * V[m] * dyv;
    A2[m] += lam * W[m] * dzw;
  }
  xsq_fill<C, S>(g, tile, zl, t, live, x, 3, false, 5, false);  // (du/dy, dw/dy)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#pragma unroll
  for (int m = 0; m < S; ++m) {
    const Rl dyu = x[m].x * c, dyw = x[m].y * c;
    A0[m] += lam * V[m] * dyu;
    A2[m] += lam * V[m] * dyw;
  }
  xsq_fill<C, S>(g, tile, zl, t, live, x, 6, false, 7, false);  // (du/dz, dv/dz)
  sq_fft_tab<S, true>(x, stab, xb, t, live);
  C z2[S];
#pragma unroll
  for (int m = 0; m < S; ++m) {
    const Rl dzu = x[m].x * c, dzv = x[m].y * c;
    const Rl a0 = A0[m] + lam * W[m] * dzu;
    const Rl a1 = A1[m] + lam * W[m] * dzv;
    const Rl d = DIV[m];
    const Rl h0 = -a0 + half * lam * d * U[m] - V[m] * dub + half * d * ub;
    const Rl h1 = -a1 + half * lam * d * V[m];
    const Rl h2 = -A2[m] + half * lam * d * W[m];
    x[m] = cmake<C>(h0, h1);
    z2[m] = cmake<C>(h2, (Rl)0);
  }
  xsq_forward<C, S>(g, stab, xb, otile, zl, t, live && z0 + zl < g.pz, x, z2);
  __syncthreads();
  xsq_store<C, ZC>(g, otile, out3, y, z0);
}

// Adjoint products, as in k_xmid_dual (lam = 1; dual v, frozen forward u,
// base U(y) e_x, Ut = U + u):
//   hel_i = -(Ut . grad) v_i + sum_j v_j d_i Ut_j + [(div u) v_i + (div v) Ut_i] / 4
// Intermediate lines 0..8 hold v (v, dv/dy, dv/dz), 9..17 the same for u.
template <typename C, int S>
__global__ void __launch_bounds__(kSqWarps * 32) k_xmid_dual_sq(Geo g, const C* __restrict__ twtab,
                                                                const C* inter, C* out3,
                                                                const double* ubase,
                                                                const double* dubase) {
  pdl();
  using Rl = typename real_of<C>::type;
  constexpr int G = SqLane<S>::G, ZC = XmidSq<C, S>::ZC, XB = sq_xbuf<S>();
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const int K1 = g.kx_max + 1, KP = XmidSq<C, S>::kp(K1);
  C* tile = reinterpret_cast<C*>(sq_raw);
  C* otile = tile + 2 * kZinvLines * ZC * KP;
  const SqLane<S> ln;
  C* xb = otile + 3 * K1 * ZC + (ln.warp * G + ln.gi) * XB;
  const int z0 = blockIdx.x * ZC, y = blockIdx.y;
  const int zl = ln.warp * G + ln.gi;
  const Rl ub = (Rl)ubase[y / g.nb];
  const Rl dub = (Rl)dubase[y / g.nb];
  const Rl c = (Rl)g.c_inv, q4 = (Rl)0.25;
  xsq_stage_tile<C, ZC>(g, inter, tile, 2 * kZinvLines, y, z0);
  // twiddle table in shared memory (read by stage 1 of every transform)
  C* stab = otile + 3 * K1 * ZC + kSqWarps * G * XB;
  xsq_twiddle_table<C, S>(stab, twtab);
  cp_async_wait<0>();
  __syncthreads();
  const bool live = ln.live;
  const int t = ln.t;
  Rl V0[S], V1[S], V2[S], U0[S], U1[S], U2[S], A0[S], A1[S], A2[S], DV[S], DU[S];
  C x[S];
#define JSD_LINE(fa, dxa, fb, dxb)                           \
  xsq_fill<C, S>(g, tile, zl, t, live, x, fa, dxa, fb, dxb); \
  sq_fft_tab<S, true>(x, stab, xb, t, live);
#define JSD_EACH(body)                                       \
  _Pragma("unroll") for (int m = 0; m < S; ++m) {            \
    const Rl pa = x[m].x * c, pb = x[m].y * c;               \
    body                                                     \
  }
  JSD_LINE(0, false, 1, false)  // (v0, v1)
  JSD_EACH(V0[m] = pa; V1[m] = pb;)
  JSD_LINE(2, false, 9, false)  // (v2, u0)
  JSD_EACH(V2[m] = pa; U0[m] = pb;)
  JSD_LINE(10, false, 11, false)  // (u1, u2)
  JSD_EACH(U1[m] = pa; U2[m] = pb;)
  JSD_LINE(0, true, 1, true)  // (dv0/dx, dv1/dx)
  JSD_EACH(const Rl ut = ub + U0[m]; A0[m] = -ut * pa; A1[m] = -ut * pb; DV[m] = pa;)
  JSD_LINE(2, true, 3, false)  // (dv2/dx, dv0/dy)
  JSD_EACH(A2[m] = -(ub + U0[m]) * pa; A0[m] -= U1[m] * pb;)
  JSD_LINE(4, false, 5, false)  // (dv1/dy, dv2/dy)
  JSD_EACH(A1[m] -= U1[m] * pa; A2[m] -= U1[m] * pb; DV[m] += pa;)
  JSD_LINE(6, false, 7, false)  // (dv0/dz, dv1/dz)
  JSD_EACH(A0[m] -= U2[m] * pa; A1[m] -= U2[m] * pb;)
  JSD_LINE(8, false, 9, true)  // (dv2/dz, du0/dx)
  JSD_EACH(A2[m] -= U2[m] * pa; DV[m] += pa; A0[m] += V0[m] * pb; DU[m] = pb;)
  JSD_LINE(10, true, 11, true)  // (du1/dx, du2/dx)
  JSD_EACH(A0[m] += V1[m] * pa + V2[m] * pb;)
  JSD_LINE(12, false, 13, false)  // (du0/dy, du1/dy)
  JSD_EACH(A1[m] += V0[m] * pa + V1[m] * pb; DU[m] += pb;)
  JSD_LINE(14, false, 15, false)  // (du2/dy, du0/dz)
  JSD_EACH(A1[m] += V2[m] * pa; A2[m] += V0[m] * pb;)
  JSD_LINE(16, false, 17, false)  // (du1/dz, du2/dz)
  C z2[S];
  JSD_EACH(
      A2[m] += V1[m] * pa + V2[m] * pb; DU[m] += pb; const Rl du = DU[m]; const Rl dv = DV[m];
      const Rl h0 = A0[m] + q4 * du * V0[m] + q4 * dv * (ub + U0[m]);
      const Rl h1 = A1[m] + dub * V0[m] + q4 * du * V1[m] + q4 * dv * U1[m];
      const Rl h2 = A2[m] + q4 * du * V2[m] + q4 * dv * U2[m]; x[m] = cmake<C>(h0, h1); z2[m] = cmake<C>(h2, (Rl)0);)
#undef JSD_LINE
#undef JSD_EACH
  xsq_forward<C, S>(g, stab, xb, otile, zl, t, live && z0 + zl < g.pz, x, z2);
  __syncthreads();
  xsq_store<C, ZC>(g, otile, out3, y, z0);
}

// ---------------------------------------------------------------------------
// x pass of the mixed form, half-split lanes (even S): a z column's lines on 2 S
// lanes, H = S / 2 points per lane (sq2_fft). Half the registers per lane of
// k_xmid_sq; the autotuner's alternative to it (129 x 129 modes x 129 planes: 172 us
// against 134).
// ---------------------------------------------------------------------------
template <int S>
struct SqLane2 {
  static constexpr int H = S / 2, L = 2 * S, G = 32 / L;  // lines per warp
  int warp, gi, t, h, partner;
  bool live;
  __device__ __forceinline__ SqLane2() {
    const int lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    gi = lane / L;
    const int r = lane - gi * L;
    h = r / S;
    t = r - h * S;
    live = gi < G;
    if (!live) {
      gi = 0;
      h = 0;
      t = 0;
    }
    partner = live ? (h ? lane - S : lane + S) : lane;
  }
};

template <typename C, int S>
struct XmidH2 {
  static constexpr int G = SqLane2<S>::G;
  static constexpr int ZC = kSqWarps * G;
  static size_t smem(const Geo& g, int nfields) {
    const int K1 = g.kx_max + 1;
    return sizeof(C) * ((size_t)nfields * ZC * (K1 | 1) + 3 * (size_t)K1 * ZC + (size_t)kSqWarps * G * sq_xbuf<S>() +
                        (size_t)S * S);
  }
};

// packed line of fields (fa, fb) at this lane's positions t + S (2 j + h)
template <typename C, int S, int ZC>
__device__ __forceinline__ void xh2_fill(const Geo& g, const C* tile, int zl, int t, int h, bool live, C* x, int fa,
                                         bool dxa, int fb, bool dxb) {
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, H = S / 2;
  const int K = g.kx_max, KP = (K + 1) | 1;
  const C* ta = tile + (fa * ZC + zl) * KP;
  const C* tb = tile + (fb * ZC + zl) * KP;
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const int p = t + S * (2 * j + h);
    const bool lo = p <= K, hi = p >= N - K;
    C out = cmake<C>(0, 0);
    if (live && (lo || hi)) {
      const int kx = lo ? p : N - p;
      C A = ta[kx], B = tb[kx];
      const Rl k = (Rl)(kx * g.ax);
      if (dxa) A = cmul_ik(A, k);
      if (dxb) B = cmul_ik(B, k);
      if (p == 0) out = cmake<C>(A.x, B.x);
      else if (lo) out = cmake<C>(A.x - B.y, A.y + B.x);
      else out = cmake<C>(A.x + B.y, B.x - A.y);
    }
    x[j] = out;
  }
}

template <typename C, int S>
__global__ void __launch_bounds__(kSqWarps * 32) k_xmid_h2(Geo g, const C* __restrict__ twtab,
                                                           const C* inter, C* out3,
                                                           const double* ubase,
                                                           const double* dubase, double lam_d) {
  static_assert(sizeof(C) == sizeof(float2), "FP64 lines: k_xmid_park");
  pdl();
  using Rl = typename real_of<C>::type;
  constexpr int N = S * S, H = S / 2, G = SqLane2<S>::G, ZC = XmidH2<C, S>::ZC, XB = sq_xbuf<S>();
  extern __shared__ __align__(16) unsigned char sq_raw[];
  const int K = g.kx_max, K1 = K + 1, KP = K1 | 1;
  C* tile = reinterpret_cast<C*>(sq_raw);
  C* otile = tile + kZinvLines * ZC * KP;
  const SqLane2<S> ln;
  C* xb = otile + 3 * K1 * ZC + (ln.warp * G + ln.gi) * XB;
  C* stab = otile + 3 * K1 * ZC + kSqWarps * G * XB;
  const int z0 = blockIdx.x * ZC, y = blockIdx.y;
  const int zl = ln.warp * G + ln.gi;
  const Rl ub = ubase ? (Rl)ubase[y / g.nb] : (Rl)0;
  const Rl dub = dubase ? (Rl)dubase[y / g.nb] : (Rl)0;
  const Rl c = (Rl)g.c_inv, lam = (Rl)lam_d, half = (Rl)0.5;
  xsq_stage_tile<C, ZC>(g, inter, tile, kZinvLines, y, z0);
  for (int e = threadIdx.x; e < N; e += blockDim.x) stab[e] = twtab[e];
  cp_async_wait<0>();
  __syncthreads();
  const bool live = ln.live;
  const int t = ln.t, h = ln.h, pr = ln.partner;
  Rl U[H], V[H], W[H], DIV[H], A0[H], A1[H], A2[H];
  C x[H];
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 0, false, 1, false);  // (u, v)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
#pragma unroll
  for (int j = 0; j < H; ++j) {
    U[j] = x[j].x * c;
    V[j] = x[j].y * c;
  }
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 2, false, 0, true);  // (w, du/dx)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
#pragma unroll
  for (int j = 0; j < H; ++j) {
    W[j] = x[j].x * c;
    const Rl dxu = x[j].y * c;
    DIV[j] = dxu;
    A0[j] = lam * U[j] * dxu + ub * dxu;
  }
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 1, true, 2, true);  // (dv/dx, dw/dx)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const Rl dxv = x[j].x * c, dxw = x[j].y * c;
    A1[j] = lam * U[j] * dxv + ub * dxv;
    A2[j] = lam * U[j] * dxw + ub * dxw;
  }
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 4, false, 8, false);  // (dv/dy, dw/dz)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const Rl dyv = x[j].x * c, dzw = x[j].y * c;
    DIV[j] += dyv + dzw;
    A1[j] += lam * V[j] * dyv;
    A2[j] += lam * W[j] * dzw;
  }
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 3, false, 5, false);  // (du/dy, dw/dy)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const Rl dyu = x[j].x * c, dyw = x[j].y * c;
    A0[j] += lam * V[j] * dyu;
    A2[j] += lam * V[j] * dyw;
  }
  xh2_fill<C, S, ZC>(g, tile, zl, t, h, live, x, 6, false, 7, false);  // (du/dz, dv/dz)
  sq2_fft<S, true>(x, stab, xb, t, h, pr, live);
  C z2[H];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    const Rl dzu = x[j].x * c, dzv = x[j].y * c;
    const Rl a0 = A0[j] + lam * W[j] * dzu;
    const Rl a1 = A1[j] + lam * W[j] * dzv;
    const Rl d = DIV[j];
    const Rl h0 = -a0 + half * lam * d * U[j] - V[j] * dub + half * d * ub;
    const Rl h1 = -a1 + half * lam * d * V[j];
    const Rl h2 = -A2[j] + half * lam * d * W[j];
    x[j] = cmake<C>(h0, h1);
    z2[j] = cmake<C>(h2, (Rl)0);
  }
  // forward transforms and the kx >= 0 outputs of the column
  const bool colok = live && z0 + zl < g.pz;
  sq2_fft<S, false>(x, stab, xb, t, h, pr, colok);
  sq2_fft<S, false>(z2, stab, xb, t, h, pr, colok);
  if (colok) {
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const int p = t + S * (2 * j + h);
      xb[p] = x[j];
      if (p <= K) otile[(2 * K1 + p) * ZC + zl] = z2[j];
    }
  }
  __syncwarp();
  if (colok) {
    for (int kx = h * S + t; kx <= K; kx += 2 * S) {
      const C a = xb[kx];
      const C b = xb[kx == 0 ? 0 : N - kx];
      otile[xsq_oslot<ZC>(0 * K1 + kx, zl)] = cmake<C>(half * (a.x + b.x), half * (a.y - b.y));
      otile[xsq_oslot<ZC>(1 * K1 + kx, zl)] = cmake<C>(half * (a.y + b.y), -half * (a.x - b.x));
    }
  }
  __syncthreads();
  xsq_store<C, ZC>(g, otile, out3, y, z0);
}

// ---------------------------------------------------------------------------
// x pass of the FP64 form. The products take seven arrays per line besides the
// line being transformed; what bounds the kernel is how many of them a lane
// must hold (registers: warps in flight), then shared-memory wavefronts. So
//  * the lines are paired by velocity component: (u, du/dx), (dv/dx, dw/dx),
//    then (v, dv/dy), (du/dy, dw/dy), then (w, dw/dz), (du/dz, dv/dz); once a
//    component has met its derivatives it goes to shared memory until the end
//    and only four arrays live across a transform;
//  * (u, du/dx) is one field times 1 - k (1 + k on the negative side): one load
//    per position instead of two;
//  * c_inv enters once, squared, at the end instead of scaling every line.
// Lane policies: a line on S lanes (S points each), or, where 16 S registers
// do not fit, on 2 S lanes (S / 2 points each, sq2p_fft).
// Bound: shared-memory wavefronts (67% of the pipe at 129 x 129 modes, 129
// planes, S = 14; FP64 pipe 34%, HBM 15%). Measured there 240 us, 344 us with
// seven arrays live, lanes (t, h) at t + S h and branches on the mode range;
// 33 x 33 modes x 776 planes (S = 7) 85 us from 163, 49 x 49 x 65 24 from 49
// (S = 9 in place of 10), 161 x 161 x 145 435 from 1127 (S = 16 in place of
// shared-memory passes of length 243).
// ---------------------------------------------------------------------------
template <int S_>
struct LineFull {
  static constexpr int S = S_, R = S, L = S, G = 32 / L, XB = sq_xbuf<S>(), TAB = S * sq_tw_stride(S);
  // Registers per thread: 4 arrays, the line and its temporaries. Caps of 128 (four
  // blocks), 168 (three) and 255: S = 9 spills 108 bytes at 168, 7 32, 4 and 5 8;
  // sides 3, 6, 8 and 10 none.
  static constexpr int BLOCKS = S <= 5 ? 4 : S <= 9 ? 3 : 2;
  static __device__ __forceinline__ int column(int li) { return li; }
  static __device__ __forceinline__ int half(int) { return 0; }
  static __device__ __forceinline__ int pos(int t, int, int r) { return t + S * r; }
  // +1 where register r holds k >= 0 modes, -1 where k < 0 (K < N / 3: the
  // positions between hold none)
  static __device__ __forceinline__ double side(int, int r) { return 2 * r < S ? 1.0 : -1.0; }
  static __device__ __forceinline__ constexpr int entry(int r) { return r; }
  static __device__ __forceinline__ double2 twiddle(const double2* __restrict__ table, int e) {
    const int j = e / sq_tw_stride(S), t = e % sq_tw_stride(S);
    return t < S ? table[t * j] : make_double2(0.0, 0.0);
  }
  struct Addr {
    const double2* tab;
    double2* xb;
  };
  static __device__ __forceinline__ Addr addr(double2* xb, const double2* tab, int, int) { return {tab, xb}; }
  static __device__ __forceinline__ void settle(Addr&) {}
  template <bool INV>
  static __device__ __forceinline__ void fft(double2* x, const double2*, const Addr& a, int t, int, bool live) {
    sq_fft_tab<S, INV>(x, a.tab + sq_tw_stride(S), a.xb, t, live);
  }
};

template <int S_>
struct LineHalf {
  using Q = Sq2p<S_>;
  static constexpr int S = S_, R = S / 2, L = 2 * S, G = 32 / L, XB = Q::xbuf(), TAB = Q::tab();
  static constexpr int BLOCKS = 3;  // 168 registers: S = 14 fits, 12 spills 4 bytes, 16 56
  static __device__ __forceinline__ int column(int li) { return li >> 1; }
  static __device__ __forceinline__ int half(int li) { return li & 1; }
  static __device__ __forceinline__ int pos(int t, int h, int r) {
    const int m = Q::out0(r);
    return t + S * (m + (h ? Q::step(m) : 0));
  }
  static __device__ __forceinline__ double side(int h, int r) {
    const int m = Q::out0(r);
    if (!Q::PF) return 2 * m < S ? 1.0 : -1.0;
    return (2 * m < S) == (h == 0) ? 1.0 : -1.0;
  }
  static __device__ __forceinline__ constexpr int entry(int r) { return Q::entry(r); }
  static __device__ __forceinline__ double2 twiddle(const double2* __restrict__ table, int e) {
    return sq2p_table_entry<S>(table, e);
  }
  using Addr = Sq2pAddr;
  static __device__ __forceinline__ Addr addr(double2* xb, const double2* tab, int t, int h) {
    return sq2p_addr<S>((unsigned)__cvta_generic_to_shared(xb), (unsigned)__cvta_generic_to_shared(tab), t, h);
  }
  // ties the table's addresses to this place: its loads do not move above it
  // (nor are they kept in registers from one transform to the next)
  static __device__ __forceinline__ void settle(Addr& a) { asm volatile("" : "+r"(a.tp), "+r"(a.tm)); }
  template <bool INV>
  static __device__ __forceinline__ void fft(double2* x, const double2* wS, const Addr& a, int, int h, bool live) {
    sq2p_fft<S, INV>(x, wS, a, h, live);
  }
};

template <int S>
using XLineLanes = std::conditional_t<(S <= 10), LineFull<S>, LineHalf<S>>;

template <class P>
struct XmidPark {
  static constexpr int S = P::S, ZC = kSqWarps * P::G;
  // Input tile [zl][kx][field]: the nine fields of a mode lie together, so a
  // line's reads along kx step over an odd number of 16-byte slots and a
  // field is a fixed offset. kp rows per column, ZERO rows of zeros after the
  // modes for the positions that have none (lane pairs pick the one four slots
  // from the partner's mode); the staging copies of 8 threads (4 or 8 columns)
  // hit distinct slots. The output tile [field][zl][kx] takes its place.
  static constexpr int ZERO = P::L > S ? 8 : 1;
  static __host__ __device__ int kp(int k1) {
    return ZC == 4 ? k1 + ZERO + ((2 - ZERO - k1) % 8 + 8) % 8 : (k1 + ZERO) | 1;
  }
  static size_t smem(const Geo& g) {
    return sizeof(double2) * ((size_t)kZinvLines * ZC * kp(g.kx_max + 1) + (size_t)ZC * P::XB + P::TAB + S) +
           sizeof(double) * 2 * (size_t)ZC * P::R * P::L;
  }
};

// Columns of the pass, plane after plane: a block's ZC columns may span two
// planes, so a box narrower than ZC leaves no lanes idle. Offset of column c
// in a field of the intermediate ([y][kx][z]); y = c / pz.
__device__ __forceinline__ size_t xpark_column(const Geo& g, int c, int& y) {
  y = c / g.pz;
  return (size_t)y * (g.kx_max + 1) * g.pz + (c - y * g.pz);
}

// Asynchronous copies of the input tile
template <int ZC, int ZERO>
__device__ __forceinline__ void xpark_stage(const Geo& g, const double2* __restrict__ inter, double2* tile, int c0,
                                            int kp) {
  constexpr int RSTEP = kSqWarps * 32 / ZC;
  const int K1 = g.kx_max + 1;
  if (threadIdx.x < RSTEP * ZC) {
    const int zl = threadIdx.x % ZC;
    const bool ok = c0 + zl < g.ny * g.pz;
    int y;
    const double2* src = inter + (ok ? xpark_column(g, c0 + zl, y) : 0);
    const size_t fstride = (size_t)g.ny * K1 * g.pz;
    for (int kx = threadIdx.x / ZC; kx < K1; kx += RSTEP) {
      const double2* s = src + (size_t)kx * g.pz;
      double2* d = tile + (zl * kp + kx) * kZinvLines;
#pragma unroll
      for (int f = 0; f < kZinvLines; ++f) cp_async_elem(d + f, s + f * fstride, ok);
    }
  }
  cp_async_commit();
  constexpr int Z = ZERO * kZinvLines;
  for (int i = threadIdx.x; i < ZC * Z; i += blockDim.x)
    tile[((i / Z) * kp + K1) * kZinvLines + i % Z] = make_double2(0.0, 0.0);
}

enum XLine { kOwnDx, kBothDx, kPlain };  // (a, da/dx), (da/dx, db/dx), (a, b)

// One position of a packed line a + i b at signed wavenumber k = side |k|:
// a + i b for k >= 0, conj(a) + i conj(b) for k < 0 (k = 0: a, b are real)
template <XLine KIND, int FA, int FB>
__device__ __forceinline__ double2 xpark_value(const double2* mode, double side, double k) {
  const double2 A = mode[FA];
  if (KIND == kOwnDx) return make_double2(A.x * (1.0 - k), side * A.y * (1.0 - k));
  const double2 B = mode[FB];
  const double2 v = make_double2(fma(-side, B.y, A.x), fma(side, A.y, B.x));
  return KIND == kPlain ? v : make_double2(-k * v.y, k * v.x);
}

template <class P>
__global__ void __launch_bounds__(kSqWarps * 32, P::BLOCKS) k_xmid_park(Geo g, const double2* __restrict__ twtab,
                                                                        const double2* inter,
                                                                        double2* out3,
                                                                        const double* ubase,
                                                                        const double* dubase) {
  pdl();
  using X = XmidPark<P>;
  constexpr int S = P::S, N = S * S, R = P::R, G = P::G, ZC = X::ZC, XB = P::XB;
  extern __shared__ __align__(128) unsigned char park_raw[];
  const int K = g.kx_max, K1 = K + 1, KP = X::kp(K1);
  double2* xball = reinterpret_cast<double2*>(park_raw);  // first: the swizzles want 128-byte boundaries
  double2* tab = xball + ZC * XB;
  double2* wS = tab + P::TAB;
  double2* tile = wS + S;
  double* park = reinterpret_cast<double*>(tile + kZinvLines * ZC * KP);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gi0 = lane / P::L, li = lane - gi0 * P::L;
  const bool live = gi0 < G;
  const int gi = live ? gi0 : 0;
  const int h = live ? P::half(li) : 0, t = live ? P::column(li) : 0;
  const int zl = warp * G + gi;
  double2* xb = xball + zl * XB;
  double* pk = park + (size_t)zl * 2 * R * P::L + (live ? li : 0);  // [2][R][L]
  const int c0 = blockIdx.x * ZC, ncol = g.ny * g.pz;
  xpark_stage<ZC, X::ZERO>(g, inter, tile, c0, KP);
  for (int e = threadIdx.x; e < P::TAB; e += blockDim.x) tab[e] = P::twiddle(twtab, e);
  if (threadIdx.x < S) wS[threadIdx.x] = 2 * threadIdx.x < S ? make_double2(1.0, 0.0) : twtab[(threadIdx.x - S / 2) * S];
  // in units of c_inv: products of two fields take c_inv^2 at the end
  const int yb = min(c0 + zl, ncol - 1) / g.pz / g.nb;
  const double ub = ubase ? ubase[yb] / g.c_inv : 0.0, dub = dubase ? dubase[yb] / g.c_inv : 0.0;
  const double c2 = g.c_inv * g.c_inv;
  cp_async_wait<0>();
  __syncthreads();
  typename P::Addr ad = P::addr(xb, tab, t, h);
  P::settle(ad);
  // |mode| at each position, a zero row where there is none
  auto mode_at = [&](int p) { return p <= K ? p : p >= N - K ? N - p : -1; };
  int kxr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int kx = mode_at(P::pos(t, h, r));
    kxr[r] = kx >= 0 ? kx : X::ZERO == 1 ? K1 : K1 + ((mode_at(P::pos(t, 1 - h, r)) + 4 - K1) & 7);
  }
  const double2* column = tile + zl * KP * kZinvLines;
  auto line = [&](auto kind, auto fa, auto fb, double2* x) {
    constexpr XLine KIND = decltype(kind)::value;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double side = P::side(h, r);
      x[P::entry(r)] = xpark_value<KIND, decltype(fa)::value, decltype(fb)::value>(
          column + kxr[r] * kZinvLines, side, KIND == kPlain ? 0.0 : side * (kxr[r] * g.ax));
    }
    P::settle(ad);
    P::template fft<true>(x, wS, ad, t, h, live);
  };
  using OwnDx = std::integral_constant<XLine, kOwnDx>;
  using BothDx = std::integral_constant<XLine, kBothDx>;
  using Plain = std::integral_constant<XLine, kPlain>;
#define JSD_LINE(kind, fa, fb) line(kind{}, std::integral_constant<int, fa>{}, std::integral_constant<int, fb>{}, x)
  // intermediate: 0 u, 1 v, 2 w, 3 du/dy, 4 dv/dy, 5 dw/dy, 6 du/dz, 7 dv/dz, 8 dw/dz
  double2 x[R];
  double A0[R], A1[R], A2[R], D[R], W[R];
  JSD_LINE(OwnDx, 0, 0);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    W[r] = x[r].x + ub;  // U + u: the base flow advects like u
    D[r] = x[r].y;
    A0[r] = W[r] * x[r].y;
    if (live) pk[r * P::L] = W[r];
  }
  JSD_LINE(BothDx, 1, 2);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    A1[r] = W[r] * x[r].x;
    A2[r] = W[r] * x[r].y;
  }
  JSD_LINE(Plain, 1, 4);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    W[r] = x[r].x;
    D[r] += x[r].y;
    A1[r] = fma(W[r], x[r].y, A1[r]);
    if (live) pk[(R + r) * P::L] = W[r];
  }
  JSD_LINE(Plain, 3, 5);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    A0[r] = fma(W[r], x[r].x, A0[r]);
    A2[r] = fma(W[r], x[r].y, A2[r]);
  }
  JSD_LINE(Plain, 2, 8);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    W[r] = x[r].x;
    D[r] += x[r].y;
    A2[r] = fma(W[r], x[r].y, A2[r]);
  }
  JSD_LINE(Plain, 6, 7);
#undef JSD_LINE
  // hel_i = -(u . grad) u_i + (div u) u_i / 2 - U d_x u_i - delta_i0 (v U' - (div u) U / 2)
  double2 z01[R], z2[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double d = 0.5 * D[r], U = pk[r * P::L], V = pk[(R + r) * P::L];
    const double a0 = fma(W[r], x[r].x, A0[r]), a1 = fma(W[r], x[r].y, A1[r]);
    const double h0 = fma(-V, dub, fma(d, U, -a0)), h1 = fma(d, V, -a1), h2 = fma(d, W[r], -A2[r]);
    z01[P::entry(r)] = make_double2(c2 * h0, c2 * h1);
    z2[P::entry(r)] = make_double2(c2 * h2, 0.0);
  }
  P::template fft<false>(z01, wS, ad, t, h, live);
  P::template fft<false>(z2, wS, ad, t, h, live);
  __syncthreads();  // every line has read the input tile: outputs [f][zl][kx] take its place
  if (live) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int p = P::pos(t, h, r);
      xb[p] = z01[r];
      if (p <= K) tile[(2 * ZC + zl) * KP + p] = z2[r];
    }
  }
  __syncwarp();
  if (live) {
    for (int kx = li; kx <= K; kx += P::L) {
      const double2 a = xb[kx], b = xb[kx == 0 ? 0 : N - kx];
      // H0 = (Z[k] + conj Z[-k]) / 2, H1 = (Z[k] - conj Z[-k]) / (2 i)
      tile[(0 * ZC + zl) * KP + kx] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
      tile[(1 * ZC + zl) * KP + kx] = make_double2(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));
    }
  }
  __syncthreads();
  constexpr int RSTEP = kSqWarps * 32 / ZC;
  const int zs = threadIdx.x % ZC;
  if (threadIdx.x < RSTEP * ZC && c0 + zs < ncol) {
    int y;
    double2* base = out3 + xpark_column(g, c0 + zs, y);
    const size_t fstride = (size_t)g.ny * K1 * g.pz;
    for (int kx = threadIdx.x / ZC; kx < K1; kx += RSTEP) {
#pragma unroll
      for (int f = 0; f < 3; ++f)
        base[f * fstride + (size_t)kx * g.pz] = tile[(f * ZC + zs) * KP + kx];
    }
  }
}

}  // namespace jsd
