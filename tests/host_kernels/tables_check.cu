// Host check of the symmetrised eigenbasis tables (jsd_parity.cuh): reads ny
// (int32) and the tables D, V, V^-1, lam, sgn, c0, cN, w0, wN (doubles) from
// standard input, writes ok (int32), the number of even modes (int32) and the
// new tables in the same order.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../jax-spectral-dns_b200/csrc/jsd_parity.cuh"

int main() {
  int ny = 0;
  if (fread(&ny, sizeof ny, 1, stdin) != 1) return 1;
  const size_t n = ny - 2, sizes[9] = {(size_t)ny * ny, n * n, n * n, n, n, n, n, n, n};
  std::vector<double> t[9];
  for (int i = 0; i < 9; ++i) {
    t[i].resize(sizes[i]);
    if (fread(t[i].data(), sizeof(double), sizes[i], stdin) != sizes[i]) return 1;
  }
  jsd_desc d = {};
  d.ny = ny;
  const double** fields[9] = {&d.D, &d.V, &d.Vinv, &d.lam, &d.sgn, &d.c0, &d.cN, &d.w0, &d.wN};
  for (int i = 0; i < 9; ++i) *fields[i] = t[i].data();
  const jsd::SymTables o = jsd::symmetric_tables(&d);
  const int head[2] = {o.ok ? 1 : 0, o.n_even};
  fwrite(head, sizeof(int), 2, stdout);
  for (const std::vector<double>* v : {&o.D, &o.V, &o.Vinv, &o.lam, &o.sgn, &o.c0, &o.cN, &o.w0, &o.wN})
    fwrite(v->data(), sizeof(double), v->size(), stdout);
  return 0;
}
