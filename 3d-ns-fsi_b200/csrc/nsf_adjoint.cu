// Discrete adjoint of the RK4 time step: one kernel per forward kernel, in gather form.
//
// The forward step (nsf_kernels.cu, nsf_stage_ws.cu) is a sequence of kernels that read and write the
// physical field buffers (three per conserved field, the RK4 accumulator, the near-body filter's pre- and
// post-filter values). The adjoint keeps one adjoint array per physical buffer and runs the transpose of
// every kernel in reverse order: a kernel that overwrites values consumes (zeroes) their adjoints and adds
// its Jacobian-transposed contributions to the adjoints of the values it read. Because the adjoint state
// mirrors the physical buffers, the reference's stale-buffer semantics (values that persist across the
// buffer swaps, primitives of filter nodes taken before the near-body filter) are differentiated exactly
// as the forward path reproduces them. Every kernel writes only adjoints of its own nodes (gathers over
// precomputed reverse maps where the forward kernel scatters): no atomics, deterministic results.
//
// The dt sequence is frozen (the gradient does not differentiate the CFL limit), as the gradient checks
// against finite differences and the dual-number oracle do.
#include <cuda_runtime.h>

#include <algorithm>

#include "nsf_adjoint.h"
#include "nsf_device.cuh"
#include "nsf_internal.h"
#include "nsf_physics.cuh"
#include "nsf_rhs_adjoint_flux.cuh"

namespace nsf {
namespace {

// Pressure of conserved values (prims_of's p).
__device__ __forceinline__ double pressure(const Consts& C, const double u[5], double g[5]) {
  const double r1 = 1.0 / (u[0] + 1.0);
  const double vx = u[1] * r1, vy = u[2] * r1, vz = u[3] * r1;
  const double K = 0.5 * (vx * vx + vy * vy + vz * vz);
  if (g) {  // gradient of p with respect to the five conserved values
    g[0] = C.gm1 * K;
    g[1] = -C.gm1 * vx;
    g[2] = -C.gm1 * vy;
    g[3] = -C.gm1 * vz;
    g[4] = C.gm1;
  }
  return C.gm1 * (u[4] - (u[0] + 1.0) * K);
}

// --------------------------------------------------------------------------------------- objective
// F_x = -dA * sum_g p(U_g) n_x(g) over the ghost nodes of the current state (the buffers the step just
// finished in, StepCtl::perm[f][0]); one block, fixed summation order.
__global__ void k_objective(const Grid* __restrict__ gp, const double* __restrict__ nx, double dA, double weight,
                            double* acc) {
  __shared__ double red[32];
  const Grid& G = *gp;
  const StepCtl* c = G.ctl;
  double s = 0;
  for (int q = threadIdx.x; q < G.nGhost; q += blockDim.x) {
    const long long n = G.gnode[q];
    double u[5];
    for (int f = 0; f < 5; ++f) u[f] = G.bufs[c->perm[f][0]][f][n];
    s += -dA * nx[q] * pressure(G.C, u, nullptr);
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += red[w];
    *acc += weight * t;
  }
}

// The adjoint of the objective's pressure at ghost q (added to the adjoint of the step's result there).
__device__ __forceinline__ void adj_objective_term(const Grid& G, const double* const val[5], const double* nx,
                                                   double dA, double weight, int q, double lam[5]) {
  const long long n = G.gnode[q];
  double u[5], g[5];
  for (int f = 0; f < 5; ++f) u[f] = val[f][n];
  pressure(G.C, u, g);
  for (int f = 0; f < 5; ++f) lam[f] += weight * (-dA * nx[q]) * g[f];
}

// ------------------------------------------------------------------------------------------- ghosts
// k_ghost writes the ghost values (weights x cell values, momenta negated) and writes the filtered
// values back to the filter nodes. Phase 1: consume the adjoints of everything k_ghost wrote (with, on a
// step whose result enters J, the objective's adjoint at the ghost nodes first).
__device__ __forceinline__ void adj_ghost_consume_item(const Grid& G, const AdjPtrs& A, double* ipbar,
                                                       const AdjBcParams& P, int q) {
  if (q < G.nGhost) {
    const long long n = G.gnode[q];
    const double sgn[5] = {1, -1, -1, -1, 1};
    double lam[5];
    for (int f = 0; f < 5; ++f) lam[f] = A.lamO[f][n];
    if (P.objective) adj_objective_term(G, P.objVal, P.nx, P.dA, P.weight, q, lam);
    for (int f = 0; f < 5; ++f) {
      ipbar[f * (long long)G.nGhost + q] = sgn[f] * lam[f];
      A.lamO[f][n] = 0.0;
    }
  } else {
    const int f = q - G.nGhost;
    const long long n = G.fnode[f];
    A.lamFnew[2 * f] += A.lamO[0][n];
    A.lamFnew[2 * f + 1] += A.lamO[4][n];
    A.lamO[0][n] = 0.0;
    A.lamO[4][n] = 0.0;
  }
}

// Phase 2: every image-point cell node gathers weight x image-point adjoint from the ghosts that read it
// (reverse map in CSR form: entries 8 * ghost + corner).
__device__ __forceinline__ void adj_ghost_gather_item(const Grid& G, const AdjPtrs& A, const double* ipbar,
                                                      const AdjBcParams& P, int c) {
  const long long m = P.cnode[c];
  const int e0 = P.coff[c], e1 = P.coff[c + 1];
  // the node's own values first (they depend on m only), so their loads overlap the entries' loads
  const bool filt = (G.type[m] & FILTER_BIT) != 0;
  const int fi = filt ? G.fidx[m] : 0;
  double* const t0 = filt ? A.lamFnew + 2 * fi : A.lamO[0] + m;  // where the density's adjoint goes
  double* const t4 = filt ? A.lamFnew + 2 * fi + 1 : A.lamO[4] + m;
  double o[5];
  o[0] = *t0;
  o[4] = *t4;
  for (int f = 1; f < 4; ++f) o[f] = A.lamO[f][m];
  double a[5] = {0, 0, 0, 0, 0};
  for (int e = e0; e < e1; ++e) {
    const int q = P.cent[e] >> 3, slot = P.cent[e] & 7;
    const double wn = G.gw[16 * (long long)q + slot], wd = G.gw[16 * (long long)q + 8 + slot];
    a[0] += wn * ipbar[q];
    a[4] += wn * ipbar[4 * (long long)G.nGhost + q];
    for (int f = 1; f < 4; ++f) a[f] += wd * ipbar[f * (long long)G.nGhost + q];
  }
  *t0 = o[0] + a[0];  // filter node: k_ghost read its filtered values
  *t4 = o[4] + a[4];
  for (int f = 1; f < 4; ++f) A.lamO[f][m] = o[f] + a[f];
}

// ------------------------------------------------------------------------------- near-body filter
// k_body_filter: fpre = O at the filter node, fnew = (6 O[n] + sum of the 6 neighbours)/12 (rho, rho_E).
// Every node of the filter stencils gathers from the filter nodes whose stencil holds it. slots[7 q ..]:
// the node's own filter slot, then those of its neighbours at +-i, +-j, +-k (-1: not a filter node),
// listed at setup so that an item's loads take two round trips (indices, then values).
__device__ __forceinline__ void adj_filter_item(const AdjPtrs& A, const long long* nodes, const int* slots, int q) {
  const long long m = nodes[q];
  int sl[7];
  for (int d = 0; d < 7; ++d) sl[d] = slots[7 * (long long)q + d];
  double fn[7][2], fp[2] = {0, 0};
  for (int d = 0; d < 7; ++d)
    for (int c = 0; c < 2; ++c) fn[d][c] = sl[d] >= 0 ? A.lamFnew[2 * sl[d] + c] : 0.0;
  if (sl[0] >= 0)
    for (int c = 0; c < 2; ++c) fp[c] = A.lamFpre[2 * sl[0] + c];
  const double o0 = A.lamO[0][m], o4 = A.lamO[4][m];
  double ar = 0, ae = 0;
  if (sl[0] >= 0) {
    ar += 0.5 * fn[0][0] + fp[0];
    ae += 0.5 * fn[0][1] + fp[1];
  }
  for (int d = 1; d < 7; ++d) {
    if (sl[d] < 0) continue;
    ar += fn[d][0] / 12;
    ae += fn[d][1] / 12;
  }
  A.lamO[0][m] = o0 + ar;
  A.lamO[4][m] = o4 + ae;
}

// -------------------------------------------------------------------------------- edge boundaries
// One node of an edge block (k_edge_bc's geometry: 32 x kEdgeRows nodes, (tx, ty) within it). Phase 1
// (periodic, outlet, inlet part 1): consume the adjoint of the edge node; periodic and outlet add to their
// (one-to-one) source nodes, the inlet keeps the adjoint of its filtered extrapolated density per node for
// phase 2.
__device__ __forceinline__ void adj_edge_item(const Grid& G, const EdgeBlock& eb, int tx, int ty, const AdjPtrs& A,
                                              const double* const val[5], int axis, double stageT, double* fbar,
                                              double* lamInflow) {
  const Consts& C = G.C;
  const int e = eb.e;
  const int* b = G.eBox[e];
  const int ax1 = axis == 0 ? 1 : 0, ax2 = axis == 2 ? 1 : 2;
  const int a = eb.a0 + ty;
  const int bb = eb.b0 + tx;
  if (a > b[2 * ax1 + 1] || bb > b[2 * ax2 + 1]) return;
  int ijk[3];
  ijk[axis] = b[2 * axis];
  ijk[ax1] = a;
  ijk[ax2] = bb;
  const long long st = axis == 0 ? G.sI : axis == 1 ? G.sJ : 1;
  const long long n = ijk[0] * G.sI + ijk[1] * G.sJ + ijk[2];
  const int side = G.eSide[e], bc = G.eBc[e];
  // Every load of an item is issued before its first store (one memory round trip, not two): the nodes
  // an item reads and writes are its own -- no other item of the phase touches them.
  double lam[5];
  if (bc == NSF_BC_PERIODIC) {
    int src[3] = {ijk[0], ijk[1], ijk[2]};
    const int nAx = axis == 0 ? G.NI : axis == 1 ? G.NJ : G.NK;
    src[axis] = side == 0 ? nAx - 2 : 1;
    const long long m = src[0] * G.sI + src[1] * G.sJ + src[2];
    double acc[5];
    for (int f = 0; f < 5; ++f) {
      lam[f] = A.lamO[f][n];
      acc[f] = A.lamO[f][m];
    }
    for (int f = 0; f < 5; ++f) {
      A.lamO[f][n] = 0.0;
      A.lamO[f][m] = acc[f] + lam[f];
    }
    return;
  }
  if (bc == NSF_BC_OUTLET) {
    const long long a1 = side == 0 ? n + st : n - st, a2 = side == 0 ? n + 2 * st : n - 2 * st;
    double v1[4], v2[4], l1[4], l2[4];
    for (int f = 0; f < 5; ++f) lam[f] = A.lamO[f][n];
    for (int f = 0; f < 4; ++f) {
      v1[f] = val[f][a1];
      v2[f] = val[f][a2];
      l1[f] = A.lamO[f][a1];
      l2[f] = A.lamO[f][a2];
    }
    for (int f = 0; f < 5; ++f) A.lamO[f][n] = 0.0;
    const double rho = 2 * v1[0] - v2[0];
    double u[3];
    for (int f = 1; f < 4; ++f) u[f - 1] = (2 * v1[f] - v2[f]) / (1 + rho);
    // rho_E = (1 + rho)/2 |u|^2 with u = m/(1 + rho): d/drho = -|u|^2/2, d/dm = u
    const double rbar = lam[0] - 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]) * lam[4];
    A.lamO[0][a1] = l1[0] + 2 * rbar;
    A.lamO[0][a2] = l2[0] - rbar;
    for (int f = 1; f < 4; ++f) {
      const double mbar = lam[f] + u[f - 1] * lam[4];
      A.lamO[f][a1] = l1[f] + 2 * mbar;
      A.lamO[f][a2] = l2[f] - mbar;
    }
    return;
  }
  if (bc == NSF_BC_INLET) {
    // rho = f (filtered extrapolation); u_axis = ramp * M0 * profile; T = 0; p = rho / gamma
    for (int f = 0; f < 5; ++f) lam[f] = A.lamO[f][n];
    const long long s1 = ax1 == 0 ? G.sI : G.sJ, s2 = ax2 == 1 ? G.sJ : 1;
    // (a neighbour outside the box reads the node's own values, which are not used)
    const bool has[4] = {a < b[2 * ax1 + 1], a > b[2 * ax1], bb < b[2 * ax2 + 1], bb > b[2 * ax2]};
    const long long off[4] = {s1, -s1, s2, -s2};
    double r1[5], r2[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const long long m = q < 4 && has[q & 3] ? n + off[q & 3] : n;
      r1[q] = val[0][side == 0 ? m + st : m - st];
      r2[q] = val[0][side == 0 ? m + 2 * st : m - 2 * st];
    }
    auto ext = [&](int q) { return 2 * r1[q] - r2[q]; };
    double f = 0;
    unsigned nn = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (has[q]) {
        f += ext(q);
        ++nn;
      }
    f += nn * ext(4);
    f /= 2 * nn;
    const double ramp = fmin(1., stageT / 10.) * C.m0 * (side == 1 ? -1.0 : 1.0);
    const double prof = (G.inflow && axis == 0) ? G.inflow[a * G.NKp + bb] : 1.0;
    const double inflowBar = axis == 0 ? lamInflow[a * G.NKp + bb] : 0.0;
    for (int f = 0; f < 5; ++f) A.lamO[f][n] = 0.0;
    const double vel = ramp * prof;
    const double fb = lam[0] + vel * lam[axis + 1] + (1 / (C.gamma * C.gm1) + 0.5 * vel * vel) * lam[4];
    const double velbar = (1 + f) * (lam[axis + 1] + vel * lam[4]);
    if (axis == 0) lamInflow[a * G.NKp + bb] = inflowBar + velbar * ramp;
    fbar[(long long)a * G.NKp + bb + (side ? (long long)G.NJ * G.NKp : 0)] = fb;
    return;
  }
  for (int f = 0; f < 5; ++f) A.lamO[f][n] = 0.0;  // any other condition: the value is consumed
}

// Inlet phase 2 (x faces only): every node of the two planes behind the inlet gathers from the inlet
// nodes whose filtered extrapolation used it.
__device__ __forceinline__ void adj_inlet_gather_item(const Grid& G, const EdgeBlock& eb, int tx, int ty,
                                                      const AdjPtrs& A, const double* fbar) {
  const int e = eb.e;  // the x faces' blocks; only inlet faces gather
  if (G.eBc[e] != NSF_BC_INLET) return;
  const int* b = G.eBox[e];
  const int a = eb.a0 + ty;   // j
  const int bb = eb.b0 + tx;  // k
  if (a > b[3] || bb > b[5]) return;
  const int side = G.eSide[e];
  const long long base = side ? (long long)G.NJ * G.NKp : 0;
  auto nnOf = [&](int ca, int cb) {
    return unsigned(ca < b[3]) + unsigned(ca > b[2]) + unsigned(cb < b[5]) + unsigned(cb > b[4]);
  };
  double g = 0;
  const int da[5] = {0, 1, -1, 0, 0}, db[5] = {0, 0, 0, 1, -1};
  for (int c = 0; c < 5; ++c) {
    const int ca = a + da[c], cb = bb + db[c];
    if (ca < b[2] || ca > b[3] || cb < b[4] || cb > b[5]) continue;
    const unsigned nn = nnOf(ca, cb);
    const double w = c == 0 ? double(nn) / (2 * nn) : 1.0 / (2 * nn);
    g += w * fbar[base + (long long)ca * G.NKp + cb];
  }
  const long long n = (long long)b[0] * G.sI + (long long)a * G.sJ + bb;
  const long long st = G.sI;
  A.lamO[0][side == 0 ? n + st : n - st] += 2 * g;
  A.lamO[0][side == 0 ? n + 2 * st : n - 2 * st] -= g;
}

// ------------------------------------------------------------------------------------------ stage
// Before the stage kernel's adjoint: the RK4 combine's adjoint and the stage's RHS input quantities.
// Combine (interior fluid nodes; lam is zero elsewhere): with o = the adjoint of the stage output,
//   stage 1:    k = dt/2 o + acc, acc = 0      stages 2, 3: k = inc o + 2 acc      stage 4: k = dt/6 o, acc += k
// (inc = dt/2, dt), lam = k is the adjoint of the stage's RHS; U0 receives o, o is consumed.
// Values: momenta and rho_E from I, density from R, filter nodes' density and rho_E from fpre (for the
// primitives), then the primitives and transport properties, as the stage kernel stages them.
// With periodic z faces (Grid::zFused) the stage kernel also wrote the z copies of the nodes at k = 1 and
// k = NK-2 it computed, with periodic y faces (Grid::yFused) the y copies of those at j = 1 and j = NJ-2:
// their adjoints are gathered here, before the combine's (edge blocks left with only such nodes are not
// listed, so the edge phase has not consumed them).
// Solid nodes (ghost and inactive): the adjoint of k_solid_copy, which copied the stage input into the
// output of the fields in solidMask (bit 0: the density from R) before the edge conditions.
__device__ __forceinline__ void adj_prepare_item(const Grid& G, const AdjPtrs& A, int s, double dtUsed, int solidMask,
                                                 double* __restrict__ lam, double* __restrict__ V, long long n) {
  const double inc = s == 2 ? dtUsed : dtUsed / 2, dtF = dtUsed / 6;
  // every load first (about twenty independent loads in flight per thread), then the arithmetic
  const uint8_t ty = G.type[n];
  const bool interior = (ty & TYPE_MASK) == FLUID_INTERIOR;
  const double m1 = A.val[1][n], m2 = A.val[2][n], m3 = A.val[3][n], e4 = A.val[4][n];
  double rho = A.valR[n], rE = e4;
  double o[5], acc[5], u0[5], oz[5] = {0, 0, 0, 0, 0}, oy[5] = {0, 0, 0, 0, 0};
  for (int f = 0; f < 5; ++f) {  // whatever the node's type, which is still on its way
    o[f] = A.lamO[f][n];
    acc[f] = A.lamAcc[f][n];
    u0[f] = A.lamU0[f][n];
  }
  // the z and y copies the stage kernel wrote with this node
  const bool zCopy = (ty & (ZCOPY_UP_BIT | ZCOPY_DOWN_BIT)) != 0;
  const long long nz = (ty & ZCOPY_UP_BIT) ? n + (G.NK - 2) : n - (G.NK - 2);
  const bool yCopy = (ty & YCOPY_BIT) != 0;
  const long long ny = yCopy && (n % G.sI) / G.sJ == 1 ? n + (G.NJ - 2) * G.sJ : n - (G.NJ - 2) * G.sJ;
  if (interior)
    for (int f = 0; f < 5; ++f) {
      if (zCopy) oz[f] = A.lamO[f][nz];
      if (yCopy) oy[f] = A.lamO[f][ny];
    }
  if (ty & FILTER_BIT) {
    const int f = G.fidx[n];
    rho = A.valFpre[2 * f];
    rE = A.valFpre[2 * f + 1];
    // the near-body filter's adjoints were consumed by the filter phase: clear them for the transposed
    // RHS (fpre) and the previous stage's ghosts (fnew)
    A.lamFpre[2 * f] = 0.0;
    A.lamFpre[2 * f + 1] = 0.0;
    A.lamFnew[2 * f] = 0.0;
    A.lamFnew[2 * f + 1] = 0.0;
  }
  const Prim pr = prims_of_nr(G.C, rho, m1, m2, m3, rE);  // as the stage kernel's staging warps
  const double q[10] = {m1, m2, m3, e4, pr.u, pr.v, pr.w, pr.p, pr.T, pr.mu};
  for (int v = 4; v < 10; ++v) V[v * G.N + n] = q[v];  // 0..3 are the stage input's own values (A.val)
  if (!interior) {
    for (int f = 0; f < 5; ++f) lam[f * G.N + n] = 0.0;
    const uint8_t t = ty & TYPE_MASK;
    if (solidMask && (t == SOLID_GHOST || t == SOLID_INACTIVE)) {
      if (solidMask & 1) {
        A.lamR[n] += A.lamO[0][n];
        A.lamO[0][n] = 0.0;
      }
      for (int f = 1; f < 5; ++f)
        if (solidMask & (1 << f)) {
          A.lamI[f][n] += A.lamO[f][n];
          A.lamO[f][n] = 0.0;
        }
    }
    return;
  }
  if (zCopy)
    for (int f = 0; f < 5; ++f) {
      o[f] += oz[f];
      A.lamO[f][nz] = 0.0;
    }
  if (yCopy)
    for (int f = 0; f < 5; ++f) {
      o[f] += oy[f];
      A.lamO[f][ny] = 0.0;
    }
  for (int f = 0; f < 5; ++f) {
    double k;
    if (s == 0) {
      k = inc * o[f] + acc[f];
      A.lamAcc[f][n] = 0.0;
    } else if (s < 3) {
      k = inc * o[f] + 2 * acc[f];
    } else {
      k = dtF * o[f];
      A.lamAcc[f][n] = acc[f] + dtF * o[f];
    }
    lam[f * G.N + n] = k;
    A.lamU0[f][n] = u0[f] + o[f];
    A.lamO[f][n] = 0.0;
  }
}

// ----------------------------------------------------------------------- two launches per stage
// Everything of a stage's adjoint before the transposed RHS, in the forward kernels' reverse order. The
// boundary work runs as phases of one cooperative launch: ghost consume (and the objective) | ghost gather
// | near-body filter | edges z | y | x | inlet gather. Each phase reads what the one before it wrote
// anywhere in the grid, so a grid barrier (bounded: a wait that gives up marks the run invalid through
// StepCtl::timeout) separates non-empty phases. Every phase is a thread-stride loop over its items; an
// edge block counts 64 items (32 x kEdgeRows nodes). The RK4 combine and RHS inputs, one item per node,
// follow as a kernel of their own (measured faster than a last phase of the cooperative launch, whose
// grid is sized for the few boundary items).
constexpr int kAdjBcThreads = 256;  // the grid is sized by the largest phase: a few dozen blocks
__global__ void __launch_bounds__(kAdjBcThreads)
    k_adj_bc(const __grid_constant__ Grid G, const __grid_constant__ AdjBcParams P, int s) {
  const AdjPtrs& A = P.A;
  // One chain of phases over all blocks, or (P.bodyBlocks > 0: the host found the bodies' nodes and the
  // face planes disjoint) two independent chains -- the body phases on the first bodyBlocks blocks, the
  // edge phases on the rest -- each with its own barrier counter.
  const bool split = P.bodyBlocks > 0;
  const bool bodyChain = !split || int(blockIdx.x) < P.bodyBlocks;
  const bool edgeChain = !split || int(blockIdx.x) >= P.bodyBlocks;
  const int b0 = (split && edgeChain) ? P.bodyBlocks : 0;
  const int nb = split ? (bodyChain ? P.bodyBlocks : int(gridDim.x) - P.bodyBlocks) : int(gridDim.x);
  const int gtid = (int(blockIdx.x) - b0) * blockDim.x + threadIdx.x, nthr = nb * blockDim.x;
  unsigned long long* const sync = P.sync + ((split && edgeChain) ? 1 : 0);
  bool started = false;
  auto barrier = [&](long long count) {
    if (count == 0) return false;
    if (started) grid_barrier(sync, unsigned(nb), P.timeout);
    started = true;
    return true;
  };
  if (bodyChain) {
    if (barrier(G.nGhost + G.nFilter))
      for (int v = gtid; v < G.nGhost + G.nFilter; v += nthr) adj_ghost_consume_item(G, A, P.ipbar, P, v);
    if (barrier(P.ncell))
      for (int v = gtid; v < P.ncell; v += nthr) adj_ghost_gather_item(G, A, P.ipbar, P, v);
    if (barrier(P.nfs))
      for (int v = gtid; v < P.nfs; v += nthr) adj_filter_item(A, P.fsNodes, P.fsSlots, v);
  }
  if (!edgeChain) return;
  const double stageT = P.roles->stageT[s];
  // each thread's first edge block of the coming phase is read before the barrier in front of it
  const int lane = gtid & 63, e0 = gtid >> 6;
  EdgeBlock eb{};
  auto first = [&](int axis) {
    if (e0 < P.nEdge[axis]) eb = P.edges[axis][e0];
  };
  auto blocks = [&](int axis, auto item) {  // a thread's lane is the same in every block it takes (64 divides nthr)
    for (int q = e0; q < P.nEdge[axis]; q += nthr >> 6) {
      if (q != e0) eb = P.edges[axis][q];
      item();
    }
  };
  first(2);
  for (int axis = 2; axis >= 0; --axis) {  // z, y, then x
    if (barrier(P.nEdge[axis]))
      blocks(axis, [&] {
        adj_edge_item(G, eb, lane & 31, lane >> 5, A, P.edgeVal, axis, stageT, P.fbar, P.lamInflow);
      });
    first(axis > 0 ? axis - 1 : 0);
  }
  if (barrier(P.inletGather ? P.nEdge[0] : 0))
    blocks(0, [&] { adj_inlet_gather_item(G, eb, lane & 31, lane >> 5, A, P.fbar); });
}

// The RK4 combine's adjoint and the RHS inputs: one thread per node.
__global__ void __launch_bounds__(256) k_adj_combine(const __grid_constant__ Grid G, const __grid_constant__ AdjBcParams P,
                                                     int s) {
  const double dtUsed = P.roles->dtUsed;
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < G.N; n += (long long)gridDim.x * blockDim.x)
    adj_prepare_item(G, P.A, s, dtUsed, P.solidMask, P.lam, P.V, n);
}

// Several device-to-device copies in one launch (blockIdx.y: the copy).
struct CopySet {
  const double* src[kMaxCopies];
  double* dst[kMaxCopies];
  long long words[kMaxCopies];
};

__global__ void k_copy_set(CopySet S) {
  const int c = blockIdx.y;
  const double* __restrict__ src = S.src[c];
  double* __restrict__ dst = S.dst[c];
  const long long n = S.words[c];
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x)
    dst[m] = src[m];
}

// Tape copies (blockIdx.y: the copy), sources and set from the control block of the running step.
__global__ void k_tape_copy(const StepCtl* __restrict__ ctl, const __grid_constant__ TapeCopy T) {
  const int c = blockIdx.y;
  const StepCtl& C = *ctl;
  long long set = (long long)C.level + T.levelOffset;
  if (set < 0) return;
  set %= T.nSets;
  const int q = T.q[c], f = T.f[c];
  const double* src;
  switch (T.kind[c]) {
    case TAPE_I: src = C.I[q][f]; break;
    case TAPE_R_SEP:
      if (C.R[q] == C.I[q][0]) return;
      src = C.R[q];
      break;
    case TAPE_O: src = C.O[q][f]; break;
    default: src = T.src[c];
  }
  src += T.srcOff[c];
  double* __restrict__ dst = T.tape + set * T.setWords + T.dstOff[c];
  const long long n = T.words[c];
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x)
    dst[m] = src[m];
}

// Transposed RHS (flux form, nsf_rhs_adjoint_flux.cuh) and the chain rule through the primitive / transport values.
// A block takes 16 (k) x 4 (j) x 4 (i) nodes, one a thread: the RHS adjoints, u, v, w, T and mu of the nodes and a
// one-node halo come into shared memory by asynchronous copies, all in one round trip. Three blocks an SM overlap one's
// copies with another's arithmetic. The other inputs (momenta, rho_E, p) are read at the node itself. Halo nodes outside
// the grid are staged as zeros.
// What bounds it: L2 traffic (about 340 bytes a node, halos included) and the latency of the copies. Measured (64^3, 100
// steps of the backward run from the tape, ms): 32.9 with the term-by-term gather over 19 RHS nodes marching along i,
// 29.0 for the flux form marching along i with asynchronous plane copies, 26.9 with 16 x 8 x 4 nodes and two a thread
// (two blocks of 112 registers), 25.8 now (80 registers).
constexpr int RT_K = 16, RT_J = 4, RT_L = 4, RT_THREADS = RT_K * RT_J * RT_L;
constexpr int RT_ROW = RT_K + 4;                      // a staged row: k0 - 1 at 1, k0 .. k0 + 15 at 2 (16-byte aligned) ..
constexpr int RT_PLANE = (RT_J + 2) * RT_ROW;         // doubles per field and staged plane
constexpr int RT_FIELDS = 10;                         // RHS adjoints 0..4, then u, v, w, T, mu
constexpr int RT_SLOT = RT_FIELDS * RT_PLANE;
constexpr int RT_SMEM = (RT_L + 2) * RT_SLOT * 8;     // bytes: 57,600
constexpr int kAdjRhsBlocks = 3;                      // resident blocks per SM (registers and shared memory)

// 8 or 16 bytes from global to shared memory, asynchronously; zeros if !in.
__device__ __forceinline__ void copy8_async(double* dst, const double* src, bool in) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copy16_async(double* dst, const double* src, int bytes) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(RT_THREADS, kAdjRhsBlocks)
    k_adj_rhs(const Grid* __restrict__ gp, const __grid_constant__ Consts C, AdjPtrs A, const double* __restrict__ lam,
              const double* __restrict__ V) {
  extern __shared__ __align__(16) double sm[];
  const Grid& G = *gp;
  const long long N = G.N, sI = G.sI, sJ = G.sJ;
  const int NI = G.NI, NJ = G.NJ, NK = G.NK;
  const int tilesK = (NK + RT_K - 1) / RT_K;
  const int j0 = (blockIdx.x / tilesK) * RT_J, k0 = (blockIdx.x % tilesK) * RT_K, i0 = blockIdx.y * RT_L;
  const int tid = threadIdx.x;
  {  // ten copies a row and field: eight aligned pairs of the tile's own nodes, the halo node on either side
    constexpr int OPS = RT_K / 2 + 2, ROWS = (RT_L + 2) * (RT_J + 2);
    for (int idx = tid; idx < ROWS * OPS; idx += RT_THREADS) {
      const int row = idx / OPS, op = idx - row * OPS, pl = row / (RT_J + 2), hj = row - pl * (RT_J + 2);
      const int p = i0 - 1 + pl, jj = j0 - 1 + hj;
      const bool rowIn = p >= 0 && p < NI && jj >= 0 && jj < NJ;
      const int kk = op < RT_K / 2 ? k0 + 2 * op : op == RT_K / 2 ? k0 - 1 : k0 + RT_K;
      const bool in = rowIn && kk >= 0 && kk < NK;
      const long long n = in ? p * sI + jj * sJ + kk : 0;
      double* d = sm + pl * RT_SLOT + hj * RT_ROW + (kk - k0) + 2;
      const int bytes = !in ? 0 : kk + 1 < NK ? 16 : 8;  // of a pair
#pragma unroll
      for (int f = 0; f < RT_FIELDS; ++f) {
        // staged fields u, v, w, T, mu are rows 4, 5, 6, 8, 9 of V
        const double* src = (f < 5 ? lam + f * N : V + (f < 8 ? f - 1 : f) * N) + n;
        if (op < RT_K / 2)
          copy16_async(d + f * RT_PLANE, src, bytes);
        else
          copy8_async(d + f * RT_PLANE, src, in);
      }
    }
  }
  const int tx = tid % RT_K, ty = tid / RT_K % RT_J, grp = tid / (RT_K * RT_J);
  const int j = j0 + ty, k = k0 + tx;
  const int c = (ty + 1) * RT_ROW + tx + 2;
  const int i = i0 + grp;
  const bool mine = i < NI && j < NJ && k < NK;
  const long long m = mine ? i * sI + j * sJ + k : 0;
  // the node's filter slot (-1: not filtered), two dependent loads, while the copies travel
  const int fi = mine && G.nFilter > 0 && (G.type[m] & FILTER_BIT) ? G.fidx[m] : -1;
  const bool filt = fi >= 0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (!mine) return;
  const double mom[3] = {A.val[1][m], A.val[2][m], A.val[3][m]}, rE = A.val[4][m], p = V[7 * N + m];
  const double rho = filt ? A.valFpre[2 * fi] : A.valR[m];
  const double* const sC = sm + (grp + 1) * RT_SLOT + c;
  auto lamAt = [&](int e, int di, int dj, int dk) { return sC[di * RT_SLOT + e * RT_PLANE + dj * RT_ROW + dk]; };
  auto valAt = [&](int v, int di, int dj, int dk) { return sC[di * RT_SLOT + (5 + v) * RT_PLANE + dj * RT_ROW + dk]; };
  auto inner = [&](int d, int o) {
    return d == 0 ? i + o >= 1 && i + o <= NI - 2 : d == 1 ? j + o >= 1 && j + o <= NJ - 2 : k + o >= 1 && k + o <= NK - 2;
  };
  auto node = [&](int d) { return inner((d + 1) % 3, 0) && inner((d + 2) % 3, 0); };
  auto face = [&](int d, int o) {
    const int x = d == 0 ? i : d == 1 ? j : k, n = d == 0 ? NI : d == 1 ? NJ : NK;
    return node(d) && x + o >= 0 && x + o < n;
  };
  const adj::Bar bar = adj::rhs_adjoint(C, lamAt, valAt, mom, rE, p, node, inner, face);
  // the adjoints this node adds into (only this thread writes them in this kernel), on their way during the chain rule
  double* const dR = filt ? A.lamFpre + 2 * fi : A.lamR + m;                // density's
  double* const dE = filt ? A.lamFpre + 2 * fi + 1 : A.lamI[4] + m;         // that of rho_E in the primitives
  const double aI1 = A.lamI[1][m], aI2 = A.lamI[2][m], aI3 = A.lamI[3][m], aI4 = A.lamI[4][m], aR = *dR, aE = *dE;
  // chain rule: u = m r1, p = gm1 (rE - (rho+1) K), T = (gamma p - rho) r1, mu = x sqrt(x) sc1/(re (T+sc1)),
  // with r1 = 1/(rho+1), K = |u|^2/2, x = 1 + T
  // the density of the primitives: the stage's density input, or the pre-filter copy at filter nodes
  const double r1 = recip_nr(rho + 1.0);
  const double u = sC[5 * RT_PLANE], v = sC[6 * RT_PLANE], w = sC[7 * RT_PLANE], T = sC[8 * RT_PLANE];
  const double K = 0.5 * (u * u + v * v + w * w);
  double ub = bar.u[0], vb = bar.u[1], wb = bar.u[2], pb = bar.p, Tb = bar.T;
  const double x = 1.0 + T, sx = sqrt_nr(x), den = T + C.sc1;
  Tb += bar.mu * C.sc1 * (1.5 * sx * den - x * sx) * recip_nr(C.re * den * den);
  pb += C.gamma * r1 * Tb;
  double rhob = -r1 * Tb - T * r1 * Tb;
  const double rEb = C.gm1 * pb;
  rhob += -C.gm1 * K * pb;
  const double Kb = -C.gm1 * (rho + 1.0) * pb;
  ub += Kb * u;
  vb += Kb * v;
  wb += Kb * w;
  rhob += -(u * ub + v * vb + w * wb) * r1;
  A.lamI[1][m] = aI1 + (bar.m[0] + r1 * ub);
  A.lamI[2][m] = aI2 + (bar.m[1] + r1 * vb);
  A.lamI[3][m] = aI3 + (bar.m[2] + r1 * wb);
  *dR = aR + rhob;
  if (filt) {
    A.lamI[4][m] = aI4 + bar.rE;
    *dE = aE + rEb;
  } else {
    A.lamI[4][m] = (aI4 + bar.rE) + rEb;
  }
}

// ------------------------------------------------------------------------------- density filter
// k_density_filter: dst = (6 src + 6 neighbours)/12 at interior nodes, dst = src at edge-plane and ghost
// nodes; solid inactive nodes off the edge planes keep their value.
__device__ __forceinline__ int df_kind(uint8_t raw) {  // 2: filtered, 1: copied, 0: untouched
  const uint8_t t = raw & TYPE_MASK;
  return t == FLUID_INTERIOR ? 2 : (t != SOLID_INACTIVE || (raw & EDGE_PLANE_BIT)) ? 1 : 0;
}

__global__ void k_adj_density_filter(const Grid* __restrict__ gp, const double* __restrict__ lamDst,
                                     double* __restrict__ lamSrc) {
  const Grid& G = *gp;
  const long long off[6] = {G.sI, -G.sI, G.sJ, -G.sJ, 1, -1};
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < G.N; m += (long long)gridDim.x * blockDim.x) {
    const int kind = df_kind(G.type[m]);
    double a = kind == 2 ? 0.5 * lamDst[m] : kind == 1 ? lamDst[m] : 0.0;
    for (int d = 0; d < 6; ++d) {
      const long long n = m + off[d];
      if (n < 0 || n >= G.N) continue;
      if (df_kind(G.type[n]) == 2) a += lamDst[n] / 12;
    }
    lamSrc[m] += a;
  }
}

__global__ void k_adj_density_filter_clear(const Grid* __restrict__ gp, double* __restrict__ lamDst) {
  const Grid& G = *gp;
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < G.N; m += (long long)gridDim.x * blockDim.x)
    if (df_kind(G.type[m])) lamDst[m] = 0.0;
}

int blocks_for(long long n, int nSM) {
  const long long b = (n + 255) / 256;
  return int(b < 8 * nSM ? (b > 0 ? b : 1) : 8 * nSM);
}

}  // namespace

// ------------------------------------------------------------------------------------ launchers
void launch_objective(const Grid* dg, const double* nx, double dA, double weight, double* acc, void* stream) {
  k_objective<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(dg, nx, dA, weight, acc);
}

// fpre = the density and rho_E of the filter nodes in buffer `U` (the state at level 0).
__global__ void k_fpre_init(const Grid* __restrict__ gp, const double* __restrict__ rho, const double* __restrict__ rE) {
  const Grid& G = *gp;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < G.nFilter; q += gridDim.x * blockDim.x) {
    G.fpre[2 * q] = rho[G.fnode[q]];
    G.fpre[2 * q + 1] = rE[G.fnode[q]];
  }
}

// The adjoint of that copy: the filter nodes' density / rho_E adjoints gather the fpre adjoints.
__global__ void k_fpre_init_adj(const Grid* __restrict__ gp, const double* __restrict__ lamFpre, double* lamRho,
                                double* lamRE) {
  const Grid& G = *gp;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < G.nFilter; q += gridDim.x * blockDim.x) {
    lamRho[G.fnode[q]] += lamFpre[2 * q];
    lamRE[G.fnode[q]] += lamFpre[2 * q + 1];
  }
}

void launch_fpre_init(const Grid* dg, int nFilter, const double* rho, const double* rE, int nSM, void* stream) {
  if (nFilter > 0) k_fpre_init<<<blocks_for(nFilter, nSM), 256, 0, static_cast<cudaStream_t>(stream)>>>(dg, rho, rE);
}

void launch_fpre_init_adj(const Grid* dg, int nFilter, const double* lamFpre, double* lamRho, double* lamRE, int nSM,
                          void* stream) {
  if (nFilter > 0)
    k_fpre_init_adj<<<blocks_for(nFilter, nSM), 256, 0, static_cast<cudaStream_t>(stream)>>>(dg, lamFpre, lamRho, lamRE);
}

void launch_adj_bc(const Grid& hg, const AdjBcParams& P, int s, int nSM, void* stream) {
  static int perSM = -1;
  if (perSM < 0) {
    int nb = 0;
    perSM = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_adj_bc, kAdjBcThreads, 0) == cudaSuccess ? nb : 0;
  }
  // enough blocks for the largest phase (of each chain when split), all resident (cooperative launch)
  auto blocks_of = [](long long items) { return std::max<long long>(1, (items + kAdjBcThreads - 1) / kAdjBcThreads); };
  const long long bodyItems = std::max<long long>(hg.nGhost + hg.nFilter, std::max(P.ncell, P.nfs));
  const long long edgeItems = 64ll * std::max(P.nEdge[0], std::max(P.nEdge[1], P.nEdge[2]));
  const long long cap = (long long)(perSM > 0 ? perSM : 1) * nSM;
  AdjBcParams Q = P;
  long long want = blocks_of(std::max(bodyItems, edgeItems));
  if (P.bodyBlocks > 0) {  // two chains: blocks for each (the request is a flag; the size is set here)
    const long long nbB = blocks_of(bodyItems), nbE = blocks_of(edgeItems);
    if (nbB + nbE <= cap) {
      Q.bodyBlocks = int(nbB);
      want = nbB + nbE;
    } else {
      Q.bodyBlocks = 0;
    }
  }
  const unsigned blocks = unsigned(want < cap ? want : cap);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kAdjBcThreads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_adj_bc, hg, Q, s);
  k_adj_combine<<<blocks_for(hg.N, nSM), 256, 0, static_cast<cudaStream_t>(stream)>>>(hg, P, s);
}

int adj_kernels_init() {
  return int(cudaFuncSetAttribute(k_adj_rhs, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM));
}

void launch_adj_rhs(const Grid* dg, const Grid& hg, const AdjPtrs& A, const double* lam, const double* V,
                    void* stream) {
  const int tiles = ((hg.NJ + RT_J - 1) / RT_J) * ((hg.NK + RT_K - 1) / RT_K);
  k_adj_rhs<<<dim3(tiles, (hg.NI + RT_L - 1) / RT_L), RT_THREADS, RT_SMEM, static_cast<cudaStream_t>(stream)>>>(
      dg, hg.C, A, lam, V);
}

void launch_copies(const double* const* src, double* const* dst, const long long* words, int count, int nSM,
                   void* stream) {
  if (count <= 0) return;
  CopySet S{};
  long long most = 1;
  for (int c = 0; c < count; ++c) {
    S.src[c] = src[c];
    S.dst[c] = dst[c];
    S.words[c] = words[c];
    most = words[c] > most ? words[c] : most;
  }
  const long long b = (most + 255) / 256, cap = 2LL * nSM;
  k_copy_set<<<dim3(unsigned(b < cap ? b : cap), count), 256, 0, static_cast<cudaStream_t>(stream)>>>(S);
}

void launch_tape_copy(const StepCtl* ctl, const TapeCopy& T, int nSM, void* stream) {
  if (T.n <= 0) return;
  long long most = 1;
  for (int c = 0; c < T.n; ++c) most = T.words[c] > most ? T.words[c] : most;
  const long long b = (most + 255) / 256, cap = 2LL * nSM;
  k_tape_copy<<<dim3(unsigned(b < cap ? b : cap), T.n), 256, 0, static_cast<cudaStream_t>(stream)>>>(ctl, T);
}

void launch_adj_density_filter(const Grid* dg, long long N, const double* lamDstConst, double* lamDst, double* lamSrc,
                               int nSM, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  k_adj_density_filter<<<blocks_for(N, nSM), 256, 0, st>>>(dg, lamDstConst, lamSrc);
  k_adj_density_filter_clear<<<blocks_for(N, nSM), 256, 0, st>>>(dg, lamDst);
}

}  // namespace nsf
