// Host-side check of the lane-pair half-split transform (sq2p_*, jsd_fftsq.cuh)
// and of the 9- and 16-point register DFTs: lanes emulated one after another
// through the swizzled exchange buffer and twiddle table, against a direct DFT.
// Also that no two entries share a place in either, and that the eight places a
// shared-memory phase touches are distinct modulo 8 (the slots of a 128-byte
// row). Prints, per form, the largest relative error of both directions.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>

#include "../../jax-spectral-dns_b200/csrc/jsd_fftsq.cuh"

using namespace jsd;

static double urand(unsigned& s) {
  s = s * 1664525u + 1013904223u;
  return ((s >> 8) & 0xffffff) / double(0x1000000) - 0.5;
}

static std::vector<double2> direct(const std::vector<double2>& x, bool inv) {
  const int N = (int)x.size();
  const long double pi = 3.14159265358979323846264338327950288L;
  std::vector<double2> ref(N);
  for (int k = 0; k < N; ++k) {
    long double re = 0, im = 0;
    for (int n = 0; n < N; ++n) {
      const long double a = (inv ? 2 : -2) * pi * (long double)((long long)n * k % N) / N;
      re += x[n].x * cosl(a) - x[n].y * sinl(a);
      im += x[n].x * sinl(a) + x[n].y * cosl(a);
    }
    ref[k] = make_double2((double)re, (double)im);
  }
  return ref;
}

static double error(const std::vector<double2>& a, const std::vector<double2>& b) {
  double err = 0, mag = 0;
  for (size_t k = 0; k < a.size(); ++k) {
    err = fmax(err, fmax(fabs(a[k].x - b[k].x), fabs(a[k].y - b[k].y)));
    mag = fmax(mag, fmax(fabs(b[k].x), fabs(b[k].y)));
  }
  return err / mag;
}

static void need(bool ok) {
  if (!ok) exit(1);
}

template <int S, bool INV>
static double pairs() {
  using Q = Sq2p<S>;
  constexpr int N = S * S, H = S / 2, XS = Q::XS;
  unsigned seed = 31u + S + INV;
  std::vector<double2> x(N), table(N), out(N);
  for (auto& v : x) v = make_double2(urand(seed), urand(seed));
  for (int e = 0; e < N; ++e) {
    const long double a = -2 * 3.14159265358979323846264338327950288L * e / N;
    table[e] = make_double2((double)cosl(a), (double)sinl(a));
  }
  std::vector<double2> tab(Q::tab()), xb(Q::xbuf()), wS(S);
  for (int e = 0; e < Q::tab(); ++e) tab[e] = sq2p_table_entry<S>(table.data(), e);
  for (int k = 0; k < S; ++k) wS[k] = k < H ? make_double2(1.0, 0.0) : table[(k - H) * S];
  double2 reg[S][2][H];
  auto pos = [](int t, int h, int r) {
    const int m = Q::out0(r);
    return t + S * (m + (h ? Q::step(m) : 0));
  };
  for (int t = 0; t < S; ++t)
    for (int h = 0; h < 2; ++h) {
      for (int r = 0; r < H; ++r) reg[t][h][Q::entry(r)] = x[pos(t, h, r)];
      sq2p_first<S, INV>(reg[t][h], wS.data(), h);
    }
  std::set<int> used;
  for (int k = 0; k < H; ++k) {
    std::vector<int> place(2 * S), look(2 * S);
    for (int t = 0; t < S; ++t)
      for (int h = 0; h < 2; ++h) {
        const int j0 = Q::row0(k), th = t ^ (h ? 4 : 0), j = j0 + (h ? Q::rstep(j0) : 0);
        look[2 * t + h] = j * XS + th;
        place[2 * t + h] = j * XS + (th ^ Q::swizzle(j0));
        need(place[2 * t + h] < Q::xbuf() && used.insert(place[2 * t + h]).second);
        xb[place[2 * t + h]] = sq2p_pair<INV>(reg[t][h][k], reg[t][1 - h][k], tab[look[2 * t + h]], h ? -1.0 : 1.0);
      }
    for (auto* v : {&place, &look})
      for (int l = 0; l + 8 <= 2 * S; l += 8) {
        std::set<int> slots;
        for (int i = 0; i < 8; ++i) slots.insert((*v)[l + i] % 8);
        need(slots.size() == 8);
      }
  }
  for (int t = 0; t < S; t += 8) {  // eight neighbouring rows, any one entry
    std::set<int> slots;
    for (int i = t; i < t + 8 && i < S; ++i) slots.insert(Q::swizzle(i));
    need((int)slots.size() == (S - t < 8 ? S - t : 8));
  }
  for (int t = 0; t < S; ++t)
    for (int h = 0; h < 2; ++h) {
      double2* v = reg[t][h];
      for (int n = 0; n < H; ++n) {
        const double2 b0 = xb[t * XS + (sq2p_n0<S>(n) ^ Q::swizzle(t))], b1 = xb[t * XS + (sq2p_n1<S>(n) ^ Q::swizzle(t))];
        v[n] = h ? csub(b0, b1) : cadd(b0, b1);
      }
      sq2p_second<S, INV>(v, wS.data(), h);
      for (int r = 0; r < H; ++r) out[pos(t, h, r)] = v[r];
    }
  return error(out, direct(x, INV));
}

template <int R, bool INV>
static double registers() {
  unsigned seed = 5u + R + INV;
  std::vector<double2> x(R);
  for (auto& v : x) v = make_double2(urand(seed), urand(seed));
  const std::vector<double2> ref = direct(x, INV);
  dft_reg<R, INV>(x.data());
  return error(x, ref);
}

int main() {
  printf("pairs12 %.3e %.3e\n", pairs<12, false>(), pairs<12, true>());
  printf("pairs14 %.3e %.3e\n", pairs<14, false>(), pairs<14, true>());
  printf("pairs16 %.3e %.3e\n", pairs<16, false>(), pairs<16, true>());
  printf("dft9 %.3e %.3e\n", registers<9, false>(), registers<9, true>());
  printf("dft16 %.3e %.3e\n", registers<16, false>(), registers<16, true>());
  return 0;
}
