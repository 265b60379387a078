// Transposed right-hand side in flux form.
//
// The right-hand side of a node P (nsf_physics.cuh) is, per direction a, a difference of per-node quantities G_a and
// of per-face quantities F_a:
//   RHS(P) = sum_a [G_a(P + a) - G_a(P - a)] + [F_a(P, P + a) - F_a(P - a, P)],
// so with lam the adjoint of the RHS the adjoint of G_a(X) is lam(X - a) - lam(X + a), and that of F_a(X, Y) is
// lam(X) - lam(Y). The adjoint of a node's inputs is then three parts:
//   G at the node itself (its own values and the in-line differences D_b u_c of its velocities),
//   the faces to its six neighbours,
//   the differences D_b u_c of its neighbours, which read this node's velocities: S_bc(X - b) - S_bc(X + b) with S_bc
//   the adjoint of D_b u_c at a node (mixed_adjoint).
// Each product is formed once per node or face, about 500 FP64 operations a node, where the term-by-term gather over
// the 19 RHS nodes that read a node takes 2,000 (nsf_rhs_adjoint.cuh, which no kernel uses any more: the tests evaluate
// it against the term table of gen_rhs_adjoint.py, and this form against the same table).
//
// lam(e, di, dj, dk): RHS adjoint of equation e at offset (di, dj, dk), zero where no RHS is taken. val(q, di, dj, dk):
// u, v, w, T, mu for q = 0..4. kappa = pf mu is not an input of its own: its adjoint is part of mu's.
#ifndef NSF_RHS_ADJOINT_FLUX_CUH
#define NSF_RHS_ADJOINT_FLUX_CUH

namespace nsf {
namespace adj {

struct Bar {  // adjoints of a node's inputs
  double m[3], rE, u[3], p, T, mu;
};

template <int A>
struct Dir {
  static constexpr int i = A == 0, j = A == 1, k = A == 2;
};
// coefficients of the mixed terms of directions a != b (symmetric in a, b), -1/(6 da db) and 1/(4 da db); of the
// inviscid terms, -1/(2 da); of the faces, 2/(3 da^2) for a's own velocity and 1/(2 da^2) else
template <int A, int B, class CT>
__device__ __forceinline__ double c6(const CT& C) {
  return A + B == 1 ? C.e_yx6 : A + B == 2 ? C.e_zx6 : C.e_zy6;
}
template <int A, int B, class CT>
__device__ __forceinline__ double c4(const CT& C) {
  return A + B == 1 ? C.e_yx4 : A + B == 2 ? C.e_zx4 : C.e_zy4;
}
template <int A, class CT>
__device__ __forceinline__ double cA(const CT& C) {
  return A == 0 ? C.ax : A == 1 ? C.ay : C.az;
}
template <int A, class CT>
__device__ __forceinline__ double b23(const CT& C) {
  return A == 0 ? C.e_xx23 : A == 1 ? C.e_yy23 : C.e_zz23;
}
template <int A, class CT>
__device__ __forceinline__ double b12(const CT& C) {
  return A == 0 ? C.e_xx12 : A == 1 ? C.e_yy12 : C.e_zz12;
}

// Adjoint of G_a's equation e at the node at offset (oi, oj, ok).
template <int A, class Lam>
__device__ __forceinline__ double dl(const Lam& lam, int e, int oi, int oj, int ok) {
  return lam(e, oi - Dir<A>::i, oj - Dir<A>::j, ok - Dir<A>::k) - lam(e, oi + Dir<A>::i, oj + Dir<A>::j, ok + Dir<A>::k);
}

// S[c]: the adjoint of D_b u_c (u_c at + b minus u_c at - b) of the node at offset (oi, oj, ok).
template <int B, class CT, class Lam, class Val>
__device__ __forceinline__ void mixed_adjoint(const CT& C, const Lam& lam, const Val& val, int oi, int oj, int ok,
                                              double S[3]) {
  constexpr int A1 = (B + 1) % 3, A2 = (B + 2) % 3;
  const double h1 = dl<A1>(lam, 4, oi, oj, ok), h2 = dl<A2>(lam, 4, oi, oj, ok);
  const double uB = val(B, oi, oj, ok), u1 = val(A1, oi, oj, ok), u2 = val(A2, oi, oj, ok), mu = val(4, oi, oj, ok);
  S[B] = mu * (c6<A1, B>(C) * (dl<A1>(lam, 1 + A1, oi, oj, ok) + u1 * h1) +
               c6<A2, B>(C) * (dl<A2>(lam, 1 + A2, oi, oj, ok) + u2 * h2));
  S[A1] = c4<A1, B>(C) * mu * (dl<A1>(lam, 1 + B, oi, oj, ok) + uB * h1);
  S[A2] = c4<A2, B>(C) * mu * (dl<A2>(lam, 1 + B, oi, oj, ok) + uB * h2);
}

// The differences D_b u_c of the neighbour at s b, which read this node's velocities (with the sign -s).
template <int B, int S, class CT, class Lam, class Val>
__device__ __forceinline__ void mixed_part(const CT& C, const Lam& lam, const Val& val, Bar& o) {
  double s[3];
  mixed_adjoint<B>(C, lam, val, S * Dir<B>::i, S * Dir<B>::j, S * Dir<B>::k, s);
#pragma unroll
  for (int c = 0; c < 3; ++c) o.u[c] -= S * s[c];
}

// G_a at the node.
template <int A, class CT, class Lam, class Val>
__device__ __forceinline__ void node_part(const CT& C, const Lam& lam, const Val& val, const double m[3], double rE,
                                          const double u[3], double p, double mu, Bar& o) {
  constexpr int B1 = (A + 1) % 3, B2 = (A + 2) % 3;
  auto diff = [&](int c, auto dir) {  // D_b u_c
    constexpr int i = decltype(dir)::i, j = decltype(dir)::j, k = decltype(dir)::k;
    return val(c, i, j, k) - val(c, -i, -j, -k);
  };
  const double a = cA<A>(C);
  double g[5];
#pragma unroll
  for (int e = 0; e < 5; ++e) g[e] = dl<A>(lam, e, 0, 0, 0);
  const double au = a * u[A];
  o.m[A] += a * g[0];
#pragma unroll
  for (int c = 0; c < 3; ++c) o.m[c] += au * g[1 + c];
  const double t = au * g[4];
  o.rE += t;
  o.p += t + a * g[1 + A];
  double ub = m[0] * g[1] + m[1] * g[2] + m[2] * g[3] + (C.h0 + rE + p) * g[4];
  const double q = g[1 + A] + u[A] * g[4], mg = mu * g[4];
  const double s = c6<A, B1>(C) * diff(B1, Dir<B1>{}) + c6<A, B2>(C) * diff(B2, Dir<B2>{});
  const double t1 = c4<A, B1>(C) * diff(A, Dir<B1>{}), t2 = c4<A, B2>(C) * diff(A, Dir<B2>{});
  o.mu += q * s + t1 * (g[1 + B1] + u[B1] * g[4]) + t2 * (g[1 + B2] + u[B2] * g[4]);
  o.u[A] += a * ub + mg * s;
  o.u[B1] += mg * t1;
  o.u[B2] += mg * t2;
}

// The face to the neighbour at s a (s = 1 or -1); lX: lam at the node.
template <int A, int S, class CT, class Lam, class Val>
__device__ __forceinline__ void face_part(const CT& C, const Lam& lam, const Val& val, const double lX[5],
                                          const double u[3], double T, double mu, Bar& o) {
  constexpr int di = S * Dir<A>::i, dj = S * Dir<A>::j, dk = S * Dir<A>::k;
  const double muY = val(4, di, dj, dk), ms = mu + muY;
  const double w = lX[4] - lam(4, di, dj, dk);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double b = c == A ? b23<A>(C) : b12<A>(C);
    const double uY = val(c, di, dj, dk), du = uY - u[c], phi = lX[1 + c] - lam(1 + c, di, dj, dk);
    // F = b ms du (momentum), b (mu u + muY uY) du (energy)
    o.u[c] += b * (w * (mu * du - (mu * u[c] + muY * uY)) - ms * phi);
    o.mu += b * du * (phi + w * u[c]);
  }
  const double h = b12<A>(C) * C.pf * w;  // heat flux pf ms (T_Y - T)
  o.T -= h * ms;
  o.mu += h * (val(3, di, dj, dk) - T);
}

// Adjoints of the inputs of the node at offset 0. m, rE, p: its momenta, rho_E and pressure.
// node(a): the node's G_a is read by a right-hand side, i.e. its coordinates other than a's are interior;
// near(a, s): its neighbour at s a is interior in a's coordinate; face(a, s): the face to that neighbour has one.
// Where they are false every lam of the part is zero. They also end the compiler's scheduling regions: in one region
// the parts' loads would all be in flight, and in registers, at once.
template <class CT, class Lam, class Val, class Node, class Near, class Face>
__device__ __forceinline__ Bar rhs_adjoint(const CT& C, const Lam& lam, const Val& val, const double m[3], double rE,
                                           double p, const Node& node, const Near& near, const Face& face) {
  Bar o;
#pragma unroll
  for (int c = 0; c < 3; ++c) o.m[c] = o.u[c] = 0.0;
  o.rE = o.p = o.T = o.mu = 0.0;
  const double u[3] = {val(0, 0, 0, 0), val(1, 0, 0, 0), val(2, 0, 0, 0)}, T = val(3, 0, 0, 0), mu = val(4, 0, 0, 0);
  if (node(0)) node_part<0>(C, lam, val, m, rE, u, p, mu, o);
  if (node(1)) node_part<1>(C, lam, val, m, rE, u, p, mu, o);
  if (node(2)) node_part<2>(C, lam, val, m, rE, u, p, mu, o);
  if (near(0, -1)) mixed_part<0, -1>(C, lam, val, o);
  if (near(0, 1)) mixed_part<0, 1>(C, lam, val, o);
  if (near(1, -1)) mixed_part<1, -1>(C, lam, val, o);
  if (near(1, 1)) mixed_part<1, 1>(C, lam, val, o);
  if (near(2, -1)) mixed_part<2, -1>(C, lam, val, o);
  if (near(2, 1)) mixed_part<2, 1>(C, lam, val, o);
  double lX[5];
#pragma unroll
  for (int e = 0; e < 5; ++e) lX[e] = lam(e, 0, 0, 0);
  if (face(0, -1)) face_part<0, -1>(C, lam, val, lX, u, T, mu, o);
  if (face(0, 1)) face_part<0, 1>(C, lam, val, lX, u, T, mu, o);
  if (face(1, -1)) face_part<1, -1>(C, lam, val, lX, u, T, mu, o);
  if (face(1, 1)) face_part<1, 1>(C, lam, val, lX, u, T, mu, o);
  if (face(2, -1)) face_part<2, -1>(C, lam, val, lX, u, T, mu, o);
  if (face(2, 1)) face_part<2, 1>(C, lam, val, lX, u, T, mu, o);
  return o;
}

}  // namespace adj
}  // namespace nsf
#endif
