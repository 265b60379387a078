// The flux-form transposed RHS (nsf_rhs_adjoint_flux.cuh) on the host, for tests/test_adjoint_flux_cpu.py: the adjoint
// of every node of a grid of n[0] x n[1] x n[2] nodes from the RHS adjoint lam (5 fields) and the inputs (10 fields: the
// momenta, rho_E, u, v, w, p, T, mu); out: the same 10 fields.
#define __device__
#define __forceinline__ inline
#include "nsf_rhs_adjoint_flux.cuh"

struct C {
  double ax, ay, az, h0, pf, e_xx23, e_xx12, e_yx6, e_zx6, e_yx4, e_zx4, e_yy12, e_yy23, e_zy6, e_zy4, e_zz12, e_zz23;
};

extern "C" void rhs_adjoint_flux(const C* c, const int* n, const double* lam, const double* in, double* out) {
  const long N = long(n[0]) * n[1] * n[2];
  for (int i = 0; i < n[0]; ++i)
    for (int j = 0; j < n[1]; ++j)
      for (int k = 0; k < n[2]; ++k) {
        auto at = [&](const double* f, int di, int dj, int dk) {
          const int a = i + di, b = j + dj, d = k + dk;
          return a < 0 || b < 0 || d < 0 || a >= n[0] || b >= n[1] || d >= n[2] ? 0.0 : f[(long(a) * n[1] + b) * n[2] + d];
        };
        auto l = [&](int e, int di, int dj, int dk) { return at(lam + e * N, di, dj, dk); };
        const int row[5] = {4, 5, 6, 8, 9};
        auto v = [&](int q, int di, int dj, int dk) { return at(in + row[q] * N, di, dj, dk); };
        const long x = (long(i) * n[1] + j) * n[2] + k;
        const double m[3] = {in[x], in[N + x], in[2 * N + x]};
        const int ijk[3] = {i, j, k};
        auto inner = [&](int a, int s) { return ijk[a] + s >= 1 && ijk[a] + s <= n[a] - 2; };
        auto node = [&](int a) { return inner((a + 1) % 3, 0) && inner((a + 2) % 3, 0); };
        auto near = [&](int a, int s) { return inner(a, s); };
        auto face = [&](int a, int s) { return node(a) && ijk[a] + s >= 0 && ijk[a] + s < n[a]; };
        const nsf::adj::Bar o = nsf::adj::rhs_adjoint(*c, l, v, m, in[3 * N + x], in[7 * N + x], node, near, face);
        const double r[10] = {o.m[0], o.m[1], o.m[2], o.rE, o.u[0], o.u[1], o.u[2], o.p, o.T, o.mu};
        for (int q = 0; q < 10; ++q) out[q * N + x] = r[q];
      }
}
