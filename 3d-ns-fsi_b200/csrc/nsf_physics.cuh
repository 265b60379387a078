// Device helpers shared by the kernels: thermodynamics (primitive values from conserved values and
// back), dt-limit terms, block reductions, and the right-hand side of the reference's five flux loops.
#ifndef NSF_PHYSICS_CUH
#define NSF_PHYSICS_CUH

#include "nsf_device.cuh"

namespace nsf {

// ----------------------------------------------------------------------------------------------
// Thermodynamics (updatePrimitiveVariables, Solver.cpp:446-479; derive*, FlowVariableGroupStructs.h).
// pow(1+T, 1.5) is evaluated as x*sqrt(x); the three divisions by (1+rho) share one reciprocal.
// Both differ from the reference by rounding only.
struct Prim {
  double u, v, w, p, T, mu, ka;
};

// The constants prims_of_nr reads, small enough to keep in registers.
struct ThermoConsts {
  double gamma, gm1, muA, muRe, pf;
};

__device__ __forceinline__ Prim prims_of(const Consts& C, double rho, double ru, double rv, double rw, double rE) {
  Prim q;
  const double r1 = 1.0 / (rho + 1.0);
  q.u = ru * r1;
  q.v = rv * r1;
  q.w = rw * r1;
  q.p = C.gm1 * (rE - (rho + 1.0) * 0.5 * (q.u * q.u + q.v * q.v + q.w * q.w));
  q.T = (C.gamma * q.p - rho) * r1;
  const double x = 1.0 + q.T;
  q.mu = x * sqrt(x) * C.sc1 / (C.re * (q.T + C.sc1));
  q.ka = q.mu * C.pf;
  return q;
}

// Reciprocal and square root by Newton-Raphson refinement of the hardware approximations
// (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64): y <- y (2 - a y) and r <- r (3 - a r^2) / 2, each iteration
// doubling the correct bits, two of them from the approximation's ~20 bits, then one Heron correction of
// s = a r for the square root. Arguments are positive normal numbers here (1 + rho, 1 + T, and the
// viscosity denominator); results are within a couple of ulps of the correctly rounded ones.
__device__ __forceinline__ double recip_nr(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  double e = fma(-a, y, 1.0);
  y = fma(y, e, y);
  e = fma(-a, y, 1.0);
  return fma(y, e, y);
}
__device__ __forceinline__ double sqrt_nr(double a) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  const double h = 0.5 * a;
  r = r * fma(-h * r, r, 1.5);
  r = r * fma(-h * r, r, 1.5);
  const double s = a * r;
  return fma(fma(-s, s, a), 0.5 * r, s);
}

// a / b from b's refined reciprocal r, corrected by the quotient's residual: rounded as the division but for rare cases
// next to a midpoint, where the product a r is off by one in the last place every few values.
__device__ __forceinline__ double quot_nr(double a, double b, double r) {
  const double q = a * r;
  return fma(r, fma(-b, q, a), q);
}

// Sutherland's viscosity x sqrt(x) sc1 / (re (T + sc1)), x = 1 + T, as x^2 / sqrt(x d^2) with d = re + T re/sc1 (C.muRe,
// C.muA), with d's sign: one Newton-Raphson inverse square root in place of a square root and a reciprocal, twelve FP64
// operations in place of twenty. The last iteration is written as a correction of r, which keeps its rounding out of the
// result: measured against extended precision over |T| <= 0.2, rms error 1.25-1.33e-16 by the coefficients (the quotient
// form: 1.28-1.50e-16), largest 5.4e-16 (6.6e-16); tests/test_viscosity_gpu.py.
template <class CT>
__device__ __forceinline__ double mu_nr(const CT& C, double x, double T) {
  const double d = fma(T, C.muA, C.muRe);
  const double z = (x * d) * d;
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(z));
  const double h = 0.5 * z;
  r = r * fma(-h * r, r, 1.5);
  r = fma(r, fma(-h * r, r, 0.5), r);
  const double mu = x * (x * r);
  return __hiloint2double(__double2hiint(mu) ^ (__double2hiint(d) & int(0x80000000u)), __double2loint(mu));
}

// prims_of with Newton-Raphson reciprocal and inverse square root (the stage kernel's staging warps, where
// the IEEE division and square root sequences are the longest dependency chains of a plane). CT: Consts or ThermoConsts.
template <class CT>
__device__ __forceinline__ Prim prims_of_nr(const CT& C, double rho, double ru, double rv, double rw, double rE) {
  Prim q;
  const double r1 = recip_nr(rho + 1.0);
  q.u = ru * r1;
  q.v = rv * r1;
  q.w = rw * r1;
  q.p = C.gm1 * (rE - 0.5 * (ru * q.u + rv * q.v + rw * q.w));
  q.T = (C.gamma * q.p - rho) * r1;
  q.mu = mu_nr(C, 1.0 + q.T, q.T);
  q.ka = q.mu * C.pf;
  return q;
}

// Conserved values from primitive values (deriveConservedVariables, FlowVariableGroupStructs.h:152-161).
__device__ __forceinline__ void cons_of(const Consts& C, double u, double v, double w, double p, double T,
                                        double out[5]) {
  const double rho = (C.gamma * p - T) / (1.0 + T);
  out[0] = rho;
  out[1] = (1.0 + rho) * u;
  out[2] = (1.0 + rho) * v;
  out[3] = (1.0 + rho) * w;
  out[4] = p / C.gm1 + (1.0 + rho) * 0.5 * (u * u + v * v + w * w);
}

// Non-negative doubles compare like their bit patterns, so maxima reduce with integer atomicMax.
__device__ __forceinline__ void atomic_max_pos(unsigned long long* a, double v) {
  if (v > 0) atomicMax(a, static_cast<unsigned long long>(__double_as_longlong(v)));
}

struct DtAcc {
  double sx = 0, sy = 0, sz = 0, nu = 0;
  __device__ __forceinline__ void add(const Consts& C, double rho, double u, double v, double w, double p, double mu) {
    // getInviscidTimeStepLimit / getViscousTimeStepLimit terms, Solver.cpp:100-122
    const double c = sqrt((1.0 + C.gamma * p) / (1.0 + rho));
    sx = fmax(sx, c + fabs(u));
    sy = fmax(sy, c + fabs(v));
    sz = fmax(sz, c + fabs(w));
    nu = fmax(nu, mu / (rho + 1.0) * C.vmod);
  }
};

// dt-limit terms of a node (getInviscidTimeStepLimit / getViscousTimeStepLimit, Solver.cpp:91-126) with one
// reciprocal of 1 + rho for all the divisions by it, reciprocals and square roots by Newton-Raphson (recip_nr,
// sqrt_nr). The terms only enter maxima, so their last-bit rounding moves dt by at most an ulp or two.
// dt_terms: the stage kernels' interior nodes. dt_terms_bc: edge, ghost and inactive nodes, whose quotients are
// corrected by their residuals (the rounding of the divisions); dt_terms_known: the same with velocities, pressure and
// temperature known.
__device__ __forceinline__ void dt_terms(const Consts& C, const double (&u)[5], DtAcc& a) {
  const double r1 = recip_nr(u[0] + 1.0);
  const double vx = u[1] * r1, vy = u[2] * r1, vz = u[3] * r1;
  const double p = C.gm1 * (u[4] - 0.5 * (u[1] * vx + u[2] * vy + u[3] * vz));
  const double T = (C.gamma * p - u[0]) * r1;
  const double c = sqrt_nr((1.0 + C.gamma * p) * r1);
  a.sx = fmax(a.sx, c + fabs(vx));
  a.sy = fmax(a.sy, c + fabs(vy));
  a.sz = fmax(a.sz, c + fabs(vz));
  a.nu = fmax(a.nu, mu_nr(C, 1.0 + T, T) * r1 * C.vmod);
}
__device__ __forceinline__ void dt_terms_at(const Consts& C, double r, double r1, double u, double v, double w, double p,
                                            double T, DtAcc& a) {
  const double c = sqrt_nr(quot_nr(1.0 + C.gamma * p, r, r1));
  const double x = 1.0 + T, den = C.re * (T + C.sc1);
  const double mu = quot_nr(x * sqrt_nr(x) * C.sc1, den, recip_nr(den));
  a.sx = fmax(a.sx, c + fabs(u));
  a.sy = fmax(a.sy, c + fabs(v));
  a.sz = fmax(a.sz, c + fabs(w));
  a.nu = fmax(a.nu, quot_nr(mu, r, r1) * C.vmod);
}
__device__ __forceinline__ void dt_terms_bc(const Consts& C, const double (&u)[5], DtAcc& a) {
  const double r = u[0] + 1.0, r1 = recip_nr(r);
  const double vx = u[1] * r1, vy = u[2] * r1, vz = u[3] * r1;
  const double p = C.gm1 * (u[4] - r * 0.5 * (vx * vx + vy * vy + vz * vz));
  const double T = (C.gamma * p - u[0]) * r1;
  dt_terms_at(C, r, r1, vx, vy, vz, p, T, a);
}
__device__ __forceinline__ void dt_terms_known(const Consts& C, double rho, double u, double v, double w, double p,
                                               double T, DtAcc& a) {
  const double r = rho + 1.0;
  dt_terms_at(C, r, recip_nr(r), u, v, w, p, T, a);
}

__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Linear thread index and thread count of the block (1-D or 2-D blocks).
__device__ __forceinline__ int block_tid() { return threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z); }
__device__ __forceinline__ int block_threads() { return blockDim.x * blockDim.y * blockDim.z; }

// Block-wide reduction of the four dt maxima into ctl->mx (order independent). Thread count % 32 == 0.
__device__ inline void flush_dt(StepCtl* ctl, DtAcc a, double* scratch /*[4*32]*/) {
  const int tid = block_tid(), lane = tid & 31, wid = tid >> 5, nw = block_threads() >> 5;
  double v[4] = {warp_max(a.sx), warp_max(a.sy), warp_max(a.sz), warp_max(a.nu)};
  __syncthreads();
  if (lane == 0)
    for (int q = 0; q < 4; ++q) scratch[q * 32 + wid] = v[q];
  __syncthreads();
  if (wid == 0) {
    for (int q = 0; q < 4; ++q) {
      double m = lane < nw ? scratch[q * 32 + lane] : 0.0;
      m = warp_max(m);
      if (lane == 0) atomic_max_pos(&ctl->mx[q], m);
    }
  }
  __syncthreads();
}

// Block-wide sums of the five change-norm partials into a per-block slot (fixed order: deterministic).
__device__ inline void flush_norms(double* slot, const double s[5], double* scratch /*[5*32]*/) {
  const int tid = block_tid(), lane = tid & 31, wid = tid >> 5, nw = block_threads() >> 5;
  double v[5];
  for (int q = 0; q < 5; ++q) v[q] = warp_sum(s[q]);
  __syncthreads();
  if (lane == 0)
    for (int q = 0; q < 5; ++q) scratch[q * 32 + wid] = v[q];
  __syncthreads();
  if (wid == 0)
    for (int q = 0; q < 5; ++q) {
      double m = lane < nw ? scratch[q * 32 + lane] : 0.0;
      m = warp_sum(m);
      if (lane == 0) slot[q] = m;
    }
  __syncthreads();
}


// Bounded grid barrier over nb blocks on a 64-bit arrival counter that only grows: every barrier instance
// takes exactly nb arrivals, so an arrival that reads `old` belongs to instance old / nb and waits until
// the counter reaches (old / nb + 1) * nb (release on arrival, acquire on the poll). A wait longer than
// kBarrierPolls polls sets *timeout (a StepCtl::timeout) and goes on: the run is then reported invalid,
// nothing hangs.
constexpr long long kBarrierPolls = 1ll << 24;
__device__ __forceinline__ unsigned long long atom_add_release(unsigned long long* a, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.add.release.gpu.u64 %0, [%1], %2;" : "=l"(old) : "l"(a), "l"(v) : "memory");
  return old;
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* a) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
  return v;
}
__device__ inline void grid_barrier(unsigned long long* S, unsigned nb, int* timeout) {
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0) {  // one arrival per block, any block shape
    const unsigned long long old = atom_add_release(S, 1ull);
    const unsigned long long target = (old / nb + 1) * nb;
    long long it = 0;
    while (ld_acquire(S) < target) {
      if (++it > kBarrierPolls) {
        atomicExch(timeout, 1);
        break;
      }
    }
  }
  __syncthreads();  // with the acquire: the block's later loads see what the other blocks wrote before they arrived
}

// ---------------------------------------------------------------------------------------------------
// Right-hand side of the five flux loops (continuity Solver.cpp:181-196, x/y/z momentum :199-339, energy
// :342-418) split by direction, for kernels that stream along i and keep the thread's own (j, k) column in
// registers. For the x direction the reference's terms are differences of
// per-node quantities and of per-face quantities along the column:
//   x-part(P) = [G(E) - G(W)] + [F(P,E) - F(W,P)]
// with G the convective/inviscid flux and the mixed-derivative products of a node, and F the normal
// viscous and heat-flux products of an x-face, e.g. for x-momentum
//   G = ax (rho_u u + p) + e_yx6 mu (v_N - v_S) + e_zx6 mu (w_U - w_D),   F = e_xx23 (mu_a + mu_b)(u_b - u_a).
// F(W,P) is the reference's (mu_W + mu_P)(u_P - u_W) (addition commutes); G differences regroup the
// reference's sums and differ from it by rounding only. Here and in yz_part the energy equation's mixed
// terms reuse the momentum equations' products (mu_N u_N (v_EN - v_WN) is formed as u_N [mu_N (v_EN - v_WN)])
// and the heat flux (kappa_a + kappa_b)(T_b - T_a) is formed as pf (mu_a + mu_b)(T_b - T_a), kappa = pf mu:
// the same sums, rounded differently. Terms of one factor are summed before it multiplies them (the momentum
// equations' coefficients equal the energy's: seventeen are read instead of 45), and the energy takes the work of a
// face's stress on the face's velocity with the stress the momentum uses, e.g. v_N (ay h_N + s_N): about twenty FP64
// operations fewer of 265 a node, and for an ensemble, whose coefficients lie in shared memory, 28 loads fewer
// (64 members 3883 -> 3693 us per step, 16 spheres 855 -> 843, Taylor-Green 256^3 2872 -> 2850).
struct XNode {  // G of one node for the five equations
  double g[5];
};
struct XOwn {  // a node's values that the next x-face needs
  double mu, u, v, w, T;
};

// G at one node. own: rho_u, rho_v, rho_w, rho_E, u, v, w, p, mu; d*: in-plane differences at the node
// (v_N - v_S, u_N - u_S, w_U - w_D, u_U - u_D).
// x_node and x_face spell out every rounding (__dmul_rn, __dadd_rn, __fma_rn are never contracted or
// reordered by the compiler): the stage kernel evaluates them in two places (the first planes of a work item
// and its main loop), and a plane's G and F must come out bit for bit the same in either, whatever the
// i-planes a work item covers (a grid run whole or in x-slabs gives identical values).
__device__ __forceinline__ XNode x_node(const Consts& C, double ru, double rv, double rw, double rE, double u,
                                        double v, double w, double p, double mu, double dyv, double dyu, double dzw,
                                        double dzu) {
  XNode n;
  const double myv = __dmul_rn(mu, dyv), mzw = __dmul_rn(mu, dzw), myu = __dmul_rn(mu, dyu), mzu = __dmul_rn(mu, dzu);
  // the mixed-derivative stresses, shared by the momenta and the energy (their work)
  const double sx = __fma_rn(C.e_zx6, mzw, __dmul_rn(C.e_yx6, myv));
  const double sy = __dmul_rn(C.e_yx4, myu), sz = __dmul_rn(C.e_zx4, mzu);
  n.g[0] = __dmul_rn(C.ax, ru);
  n.g[1] = __fma_rn(C.ax, __fma_rn(ru, u, p), sx);
  n.g[2] = __fma_rn(C.ax, __dmul_rn(rv, u), sy);
  n.g[3] = __fma_rn(C.ax, __dmul_rn(rw, u), sz);
  const double h = __dadd_rn(__dadd_rn(C.h0, rE), p);
  n.g[4] = __fma_rn(u, __fma_rn(C.ax, h, sx), __fma_rn(v, sy, __dmul_rn(w, sz)));
  return n;
}

// F of the x-face between a (lower i) and b.
__device__ __forceinline__ void x_face(const Consts& C, const XOwn& a, const XOwn& b, double f[5]) {
  const double ms = __dadd_rn(a.mu, b.mu);
  const double du = __dsub_rn(b.u, a.u), dv = __dsub_rn(b.v, a.v), dw = __dsub_rn(b.w, a.w);
  f[0] = 0.0;
  f[1] = __dmul_rn(C.e_xx23, __dmul_rn(ms, du));
  f[2] = __dmul_rn(C.e_xx12, __dmul_rn(ms, dv));
  f[3] = __dmul_rn(C.e_xx12, __dmul_rn(ms, dw));
  const double su = __fma_rn(a.mu, a.u, __dmul_rn(b.mu, b.u));
  const double sv = __fma_rn(a.mu, a.v, __dmul_rn(b.mu, b.v));
  const double sw = __fma_rn(a.mu, a.w, __dmul_rn(b.mu, b.w));
  double e4 = __fma_rn(sw, dw, __dmul_rn(sv, dv));  // the terms of weight 1/(2dx^2)
  e4 = __fma_rn(C.pf, __dmul_rn(ms, __dsub_rn(b.T, a.T)), e4);
  f[4] = __fma_rn(C.e_xx12, e4, __dmul_rn(C.e_xx23, __dmul_rn(su, du)));
}

// The velocities at a node's in-plane neighbours (N, S: +j, -j; U, D: +k, -k) that the mixed x-differences read, in
// registers (Cross) or read from the staged plane at each use (CrossMem: plane pointer p, node c).
struct Cross {
  double vn, vs, un, us, wu, wd, uu, ud;
  __device__ __forceinline__ double vN() const { return vn; }
  __device__ __forceinline__ double vS() const { return vs; }
  __device__ __forceinline__ double uN() const { return un; }
  __device__ __forceinline__ double uS() const { return us; }
  __device__ __forceinline__ double wU() const { return wu; }
  __device__ __forceinline__ double wD() const { return wd; }
  __device__ __forceinline__ double uU() const { return uu; }
  __device__ __forceinline__ double uD() const { return ud; }
};
template <int HK, int FS>
struct CrossMem {
  const double* p;
  int c;
  __device__ __forceinline__ double vN() const { return p[1 * FS + c + HK]; }
  __device__ __forceinline__ double vS() const { return p[1 * FS + c - HK]; }
  __device__ __forceinline__ double uN() const { return p[0 * FS + c + HK]; }
  __device__ __forceinline__ double uS() const { return p[0 * FS + c - HK]; }
  __device__ __forceinline__ double wU() const { return p[2 * FS + c + 1]; }
  __device__ __forceinline__ double wD() const { return p[2 * FS + c - 1]; }
  __device__ __forceinline__ double uU() const { return p[0 * FS + c + 1]; }
  __device__ __forceinline__ double uD() const { return p[0 * FS + c - 1]; }
  __device__ __forceinline__ Cross load() const { return Cross{vN(), vS(), uN(), uS(), wU(), wD(), uU(), uD()}; }
};
// y- and z-direction part of the right-hand side at P (the reference's terms not covered by G and F).
// cP/pP: staged centre plane; xW, xP, xE: the in-plane neighbours' velocities on the planes at -x, P and +x (of the
// neighbour planes only these are read, for the mixed x-derivatives); own: P's own values. The staged planes
// hold u, v, w, p, T, mu (fields 0..5); kappa = pf mu is formed here, as prims_of forms it.
template <int HK, int FS, class X>
__device__ __forceinline__ void yz_part(const Consts& C, const double* __restrict__ cP, const double* __restrict__ pP,
                                        const X& xW, const X& xP, const X& xE, int c, const XOwn& own, double out[5]) {
  enum { RU = 1, RV = 2, RW = 3, RE = 4 };
  enum { U = 0, V = 1, W = 2, P = 3, TT = 4, MU = 5 };
#define F_(b, v, o) (b)[(v)*FS + c + (o)]
  constexpr int oN = HK, oS = -HK, oU = 1, oD = -1;
  const double muP = own.mu, uP = own.u, vP = own.v, wP = own.w, TP = own.T;
  const double muN = F_(pP, MU, oN), muS = F_(pP, MU, oS), muU = F_(pP, MU, oU), muD = F_(pP, MU, oD);
  const double uN = xP.uN(), uS = xP.uS(), uU = xP.uU(), uD = xP.uD();
  const double vN = xP.vN(), vS = xP.vS(), vU = F_(pP, V, oU), vD = F_(pP, V, oD);
  const double wN = F_(pP, W, oN), wS = F_(pP, W, oS), wU = xP.wU(), wD = xP.wD();
  const double pN = F_(pP, P, oN), pS = F_(pP, P, oS), pU = F_(pP, P, oU), pD = F_(pP, P, oD);
  // face viscosity sums (mu_N + mu_P) ... of the normal viscous and heat-flux terms
  const double msN = muN + muP, msS = muS + muP, msU = muU + muP, msD = muD + muP;
  // mixed-derivative products mu_X (difference across X), shared by momentum and energy
  const double mNdxv = muN * (xE.vN() - xW.vN()), mSdxv = muS * (xE.vS() - xW.vS());
  const double mNdxu = muN * (xE.uN() - xW.uN()), mSdxu = muS * (xE.uS() - xW.uS());
  const double mUdxw = muU * (xE.wU() - xW.wU()), mDdxw = muD * (xE.wD() - xW.wD());
  const double mUdxu = muU * (xE.uU() - xW.uU()), mDdxu = muD * (xE.uD() - xW.uD());
  const double wNU = F_(pP, W, oN + oU), wND = F_(pP, W, oN + oD), wSU = F_(pP, W, oS + oU), wSD = F_(pP, W, oS + oD);
  const double vNU = F_(pP, V, oN + oU), vND = F_(pP, V, oN + oD), vSU = F_(pP, V, oS + oU), vSD = F_(pP, V, oS + oD);
  const double mNdzw = muN * (wNU - wND), mSdzw = muS * (wSU - wSD);  // w_U - w_D at N, S
  const double mUdyw = muU * (wNU - wSU), mDdyw = muD * (wND - wSD);  // w_N - w_S at U, D
  const double mNdzv = muN * (vNU - vND), mSdzv = muS * (vSU - vSD);  // v_U - v_D at N, S
  const double mUdyv = muU * (vNU - vSU), mDdyv = muD * (vND - vSD);  // v_N - v_S at U, D
  const double duN = uN - uP, duS = uP - uS, duU = uU - uP, duD = uP - uD;
  const double dvN = vN - vP, dvS = vP - vS, dvU = vU - vP, dvD = vP - vD;
  const double dwN = wN - wP, dwS = wP - wS, dwU = wU - wP, dwD = wP - wD;
  // mixed-derivative stresses of a y-face's v and of a z-face's w, shared by the momentum and the energy (its work)
  const double sN = fma(C.e_zy6, mNdzw, C.e_yx6 * mNdxu), sS = fma(C.e_zy6, mSdzw, C.e_yx6 * mSdxu);
  const double sU = fma(C.e_zy6, mUdyv, C.e_zx6 * mUdxu), sD = fma(C.e_zy6, mDdyv, C.e_zx6 * mDdxu);
  out[0] = fma(C.ay, F_(cP, RV, oN) - F_(cP, RV, oS), C.az * (F_(cP, RW, oU) - F_(cP, RW, oD)));
  {
    const double ruN = F_(cP, RU, oN), ruS = F_(cP, RU, oS), ruU = F_(cP, RU, oU), ruD = F_(cP, RU, oD);
    double e = C.ay * fma(ruN, vN, -(ruS * vS));
    e = fma(C.az, fma(ruU, wU, -(ruD * wD)), e);
    e = fma(C.e_yy12, fma(msN, duN, -(msS * duS)), e);
    e = fma(C.e_zz12, fma(msU, duU, -(msD * duD)), e);
    e = fma(C.e_yx4, mNdxv - mSdxv, e);
    out[1] = fma(C.e_zx4, mUdxw - mDdxw, e);
  }
  {
    const double rvN = F_(cP, RV, oN), rvS = F_(cP, RV, oS), rvU = F_(cP, RV, oU), rvD = F_(cP, RV, oD);
    double e = fma(C.ay, fma(rvN, vN, pN), sN) - fma(C.ay, fma(rvS, vS, pS), sS);
    e = fma(C.az, fma(rvU, wU, -(rvD * wD)), e);
    e = fma(C.e_yy23, fma(msN, dvN, -(msS * dvS)), e);
    e = fma(C.e_zz12, fma(msU, dvU, -(msD * dvD)), e);
    out[2] = fma(C.e_zy4, mUdyw - mDdyw, e);
  }
  {
    const double rwN = F_(cP, RW, oN), rwS = F_(cP, RW, oS), rwU = F_(cP, RW, oU), rwD = F_(cP, RW, oD);
    double e = fma(C.az, fma(rwU, wU, pU), sU) - fma(C.az, fma(rwD, wD, pD), sD);
    e = fma(C.ay, fma(rwN, vN, -(rwS * vS)), e);
    e = fma(C.e_yy12, fma(msN, dwN, -(msS * dwS)), e);
    e = fma(C.e_zz23, fma(msU, dwU, -(msD * dwD)), e);
    out[3] = fma(C.e_zy4, mNdzv - mSdzv, e);
  }
  {
    const double hN = C.h0 + F_(cP, RE, oN) + pN, hS = C.h0 + F_(cP, RE, oS) + pS;
    const double hU = C.h0 + F_(cP, RE, oU) + pU, hD = C.h0 + F_(cP, RE, oD) + pD;
    double e = vN * fma(C.ay, hN, sN);
    e = fma(-vS, fma(C.ay, hS, sS), e);
    e = fma(wU, fma(C.az, hU, sU), e);
    e = fma(-wD, fma(C.az, hD, sD), e);
    const double muu = muP * uP, muv = muP * vP, muw = muP * wP;
    // the terms of weight 1/(2dy^2), 2/(3dy^2), 1/(2dz^2), 2/(3dz^2)
    double t = fma(muN, uN, muu) * duN;
    t = fma(-fma(muS, uS, muu), duS, t);
    t = fma(fma(muN, wN, muw), dwN, t);
    t = fma(-fma(muS, wS, muw), dwS, t);
    t = fma(C.pf, fma(msN, F_(pP, TT, oN) - TP, -(msS * (TP - F_(pP, TT, oS)))), t);
    e = fma(C.e_yy12, t, e);
    e = fma(C.e_yy23, fma(fma(muN, vN, muv), dvN, -(fma(muS, vS, muv) * dvS)), e);
    t = fma(muU, uU, muu) * duU;
    t = fma(-fma(muD, uD, muu), duD, t);
    t = fma(fma(muU, vU, muv), dvU, t);
    t = fma(-fma(muD, vD, muv), dvD, t);
    t = fma(C.pf, fma(msU, F_(pP, TT, oU) - TP, -(msD * (TP - F_(pP, TT, oD)))), t);
    e = fma(C.e_zz12, t, e);
    e = fma(C.e_zz23, fma(fma(muU, wU, muw), dwU, -(fma(muD, wD, muw) * dwD)), e);
    // the remaining mixed terms' work
    e = fma(C.e_yx4, fma(uN, mNdxv, -(uS * mSdxv)), e);
    e = fma(C.e_zx4, fma(uU, mUdxw, -(uD * mDdxw)), e);
    t = fma(wN, mNdzv, -(wS * mSdzv));
    t = fma(vU, mUdyw, t);
    t = fma(-vD, mDdyw, t);
    out[4] = fma(C.e_zy4, t, e);
  }
#undef F_
}

}  // namespace nsf
#endif
