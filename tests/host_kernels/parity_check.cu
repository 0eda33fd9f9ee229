// Host check of the operators on even and odd parts (jsd_parity.cuh): random
// operators with each symmetry the kernel takes, cut with parity_halves and
// parity_pack, read back through parity_slot and applied the way k_parity does
// (fold, two halves with their extra column and row, unfold), against the whole
// product in long double. Prints per case: kind, rows, columns, largest error
// over |A| |B|, and that of the whole product in double.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../jax-spectral-dns_b200/csrc/jsd_parity.cuh"

using namespace jsd;

static double urand(unsigned long long& s) {
  s = s * 6364136223846793005ull + 1442695040888963407ull;
  return ((s >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
}

static void run_case(const char* kind, int ny, int mout, int kin, bool fold, bool unfold, int flip, int n_even,
                     unsigned long long seed) {
  std::vector<double> A((size_t)mout * kin), B(kin);
  for (double& b : B) b = urand(seed);
  for (int r = 0; r < mout; ++r)
    for (int k = 0; k < kin; ++k) {
      // the sign of the mirrored entry: along the points, by the parity of the eigen row or column
      double v = urand(seed);
      const int rm = unfold ? mout - 1 - r : r, km = fold ? kin - 1 - k : k;
      const double sgn = fold && unfold ? -1.0 : flip * ((fold ? r : k) < n_even ? 1.0 : -1.0);
      if (rm < r || (rm == r && km < k)) v = sgn * A[(size_t)rm * kin + km];
      else if (rm == r && km == k && sgn < 0) v = 0.0;
      A[(size_t)r * kin + k] = v;
    }
  int w = 0, tm = 0;
  if (!parity_shape(parity_row_tiles((ny + 1) / 2), w, tm)) exit(1);  // one shape for all of a plan's operators
  const int rt = w * tm, edge = 8 * rt;
  const ParityHalves h = parity_halves(A.data(), mout, kin, fold, unfold, n_even);
  std::vector<double> half[2];
  for (int p = 0; p < 2; ++p) {
    const std::vector<double> pk = parity_pack(h.h[p], h.M[p], h.K[p], rt);
    if (pk.size() != parity_frag(rt) + edge + h.K[p] || h.M[p] > edge + 1 || h.K[p] > edge + 1) exit(2);
    half[p].assign(h.M[p], 0.0);
    for (int r = 0; r < h.M[p]; ++r)
      for (int k = 0; k < h.K[p]; ++k) {
        const double a = r >= edge ? pk[parity_frag(rt) + edge + k] : k >= edge ? pk[parity_frag(rt) + r]
                                                                               : pk[parity_slot(rt, r, k)];
        const int base = h.part[p] ? kin - h.K[p] : 0;
        const double b = fold ? (h.part[p] ? B[k] - B[kin - 1 - k] : B[k] + B[kin - 1 - k]) : B[base + k];
        half[p][r] += a * b;
      }
  }
  double err = 0, plain = 0;
  for (int r = 0; r < mout; ++r) {
    long double want = 0, mag = 0;
    double c = 0;
    for (int k = 0; k < kin; ++k) {
      want += (long double)A[(size_t)r * kin + k] * B[k];
      mag += fabsl((long double)A[(size_t)r * kin + k] * B[k]);
      c += A[(size_t)r * kin + k] * B[k];
    }
    double got;
    if (unfold) {
      const int i = r < mout - 1 - r ? r : mout - 1 - r;
      const double S = half[0][i], T = i < h.M[1] ? half[1][i] : 0.0;
      got = r == i ? S + T : S - T;
    } else {
      got = r < h.M[0] ? half[0][r] : half[1][r - h.M[0]];
    }
    err = std::max(err, (double)(fabsl(got - want) / (mag + 1e-300L)));
    plain = std::max(plain, (double)(fabsl(c - want) / (mag + 1e-300L)));
  }
  printf("%s %d %d %.3e %.3e\n", kind, mout, kin, err, plain);
}

int main() {
  for (int ny : {10, 11, 17, 18, 24, 33, 34, 35, 49, 50, 65, 66, 82, 97, 98, 129, 130, 131, 145, 161, 193}) {
    const int n = ny - 2, ne = (n + 1) / 2;
    run_case("D", ny, ny, ny, true, true, 1, 0, ny);
    run_case("VinvD", ny, n, ny, true, false, -1, ne, ny + 1);
    run_case("Vinv", ny, n, n, true, false, 1, ne, ny + 2);
    run_case("V", ny, ny, n, false, true, 1, ne, ny + 3);
    run_case("DV", ny, ny, n, false, true, -1, ne, ny + 4);
    run_case("VinvT", ny, n, n, false, true, 1, ne, ny + 5);
  }
  return 0;
}
