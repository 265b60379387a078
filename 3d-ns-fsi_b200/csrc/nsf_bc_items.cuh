// Per-node boundary work of one stage (solid-node copies, mesh-edge conditions, near-body filter, ghost
// interpolation, filter write-back) and the start and end of a step, as device functions shared by the
// separate kernels and the fused boundary kernel (nsf_kernels.cu) and the whole-step kernel (nsf_step.cu).
#ifndef NSF_BC_ITEMS_CUH
#define NSF_BC_ITEMS_CUH

#include "nsf_device.cuh"
#include "nsf_internal.h"
#include "nsf_physics.cuh"

namespace nsf {

// ----------------------------------------------------------------------------------------------
// Solid-node values the reference's stage buffer still holds from earlier writes (see nsf_device.cuh).
// One solid node q of a grid; the device functions here are shared by the separate kernels and the fused
// boundary kernel (k_bc), which reads fields written earlier in the same launch: those reads bypass L1.
__device__ __forceinline__ void solid_copy_node(const StepCtl* c, int s, int mask, long long n) {
  double v[5];  // every load before the first store: one memory round trip, not one per field
#pragma unroll
  for (int f = 0; f < 5; ++f) v[f] = mask & (1 << f) ? __ldcg((f == 0 ? c->R[s] : c->I[s][f]) + n) : 0.0;
#pragma unroll
  for (int f = 0; f < 5; ++f)
    if (mask & (1 << f)) c->O[s][f][n] = v[f];
}

__device__ __forceinline__ void solid_copy_item(const Grid& G, const StepCtl* c, int s, int mask, int q) {
  solid_copy_node(c, s, mask, G.snode[q]);
}

// Field f at node m as the stage's boundary work reads it after the solid-node copy. For a solid node off
// the mesh faces (solid = true; nothing but the copy writes it in a stage) the value comes from the copy's
// source, so the reader does not wait for the copy; the values are the same either way.
__device__ __forceinline__ double ld_res(const StepCtl* c, int s, int f, long long m, bool solid) {
  const double* from = c->O[s][f];
  if (solid && (c->copyMask[s] & (1 << f))) from = f == 0 ? c->R[s] : c->I[s][f];
  return __ldcg(from + m);  // one load either way: several calls' loads can be in flight together
}

// ----------------------------------------------------------------------------------------------
// Mesh-edge boundary conditions of one axis (both faces; the faces of one axis never read each other's
// nodes). Launched for x, then y, then z: the reference's application order outlet/inlet (x), y-max,
// y-min, z-max, z-min (Mesh.cpp:155-167 after the reversal at Mesh.cpp:70). Each block comes from the
// launch plan's list (member, face, first in-plane coordinates, mask of the nodes it works on).
// periodic_source: the node a periodic face node finally copies -- the opposite interior-plane node, and if
// that node lies on another periodic face (which copied it earlier in the reference's order), that face's
// source, and so on (at most two more hops). The copies are exact, so reading the final source gives the
// value the reference copies; it lets chains of copies run together (nsf_bc_plan.cpp).
// edge_node: one node (thread tx, ty of an edge block) of a mesh-edge boundary condition; adds the stage-4
// dt terms and the NaN check of edge and ghost-typed nodes.
__device__ __forceinline__ void periodic_source(const Grid& G, int axis, int side, int ijk[3]) {
  const int nAx[3] = {G.NI, G.NJ, G.NK};
  ijk[axis] = side == 0 ? nAx[axis] - 2 : 1;
  for (int hop = 0; hop < 2; ++hop) {
    int found = -1;
    for (int e = 0; e < G.nEdge && found < 0; ++e) {
      const int* b = G.eBox[e];
      if (G.eBc[e] == NSF_BC_PERIODIC && ijk[0] >= b[0] && ijk[0] <= b[1] && ijk[1] >= b[2] && ijk[1] <= b[3] &&
          ijk[2] >= b[4] && ijk[2] <= b[5])
        found = e;
    }
    if (found < 0) return;
    const int a = G.eAxis[found];
    ijk[a] = G.eSide[found] == 0 ? nAx[a] - 2 : 1;
  }
}

__device__ __forceinline__ void edge_node(const Grid& G, const StepCtl* c, const EdgeBlock& eb, int tx, int ty, int s,
                                          int axis, DtAcc& dta, int& bad) {
  const Consts& C = G.C;
  const int e = eb.e;
  {
    const int* b = G.eBox[e];
    // in-plane coordinates: (a, bb) = the two axes other than `axis`, in (i, j, k) order
    const int ax1 = axis == 0 ? 1 : 0, ax2 = axis == 2 ? 1 : 2;
    const int a = eb.a0 + ty;
    const int bb = eb.b0 + tx;
    if (a <= b[2 * ax1 + 1] && bb <= b[2 * ax2 + 1] && ((eb.mask >> (ty * 32 + tx)) & 1)) {
      int ijk[3];
      ijk[axis] = b[2 * axis];
      ijk[ax1] = a;
      ijk[ax2] = bb;
      const long long st = axis == 0 ? G.sI : axis == 1 ? G.sJ : 1;
      const long long n = ijk[0] * G.sI + ijk[1] * G.sJ + ijk[2];
      const int side = G.eSide[e], bc = G.eBc[e];
      double* const* O = c->O[s];
      const bool solidSrc = (eb.solidSrc >> (ty * 32 + tx)) & 1;
      auto ld = [&](int f, long long m) { return ld_res(c, s, f, m, solidSrc); };
      const long long a1 = side == 0 ? n + st : n - st, a2 = side == 0 ? n + 2 * st : n - 2 * st;  // Boundary.cpp:74-108
      double cv[5];
      double u = 0, v = 0, w = 0, p = 0, T = 0;
      bool primKnown = false;
      if (bc == NSF_BC_INLET) {  // Boundary.cpp:250-296 with filterInletDensity :142-245
        // extrapolated density of this node and of its in-plane neighbours inside the owned box
        const long long s1 = ax1 == 0 ? G.sI : G.sJ, s2 = ax2 == 1 ? G.sJ : 1;
        // every load first (a neighbour outside the box reads the node's own values, which are not used)
        const bool has[4] = {a < b[2 * ax1 + 1], a > b[2 * ax1], bb < b[2 * ax2 + 1], bb > b[2 * ax2]};
        const long long off[4] = {s1, -s1, s2, -s2};
        double r1[5], r2[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          const long long m = q < 4 && has[q & 3] ? n + off[q & 3] : n;
          r1[q] = ld(0, side == 0 ? m + st : m - st);
          r2[q] = ld(0, side == 0 ? m + 2 * st : m - 2 * st);
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
        const double rho = f;
        double vel = fmin(1., c->stageT[s] / 10.) * C.m0;
        if (G.inflow && axis == 0) vel *= G.inflow[a * G.NKp + bb];  // profile factor (1 in a plain run)
        if (side == 1) vel *= -1;
        u = axis == 0 ? vel : 0;
        v = axis == 1 ? vel : 0;
        w = axis == 2 ? vel : 0;
        T = 0;
        p = (T * (1 + rho) + rho) / C.gamma;
        cons_of(C, u, v, w, p, T, cv);
        primKnown = true;
      } else if (bc == NSF_BC_OUTLET) {  // Boundary.cpp:304-336
        const double rho = 2 * ld(0, a1) - ld(0, a2);
        const double ru = 2 * ld(1, a1) - ld(1, a2);
        const double rv = 2 * ld(2, a1) - ld(2, a2);
        const double rw = 2 * ld(3, a1) - ld(3, a2);
        p = 0;
        u = ru / (1 + rho);
        v = rv / (1 + rho);
        w = rw / (1 + rho);
        T = (C.gamma * p - rho) / (1 + rho);
        cv[0] = rho;
        cv[1] = ru;
        cv[2] = rv;
        cv[3] = rw;
        cv[4] = p / C.gm1 + (1 + rho) / 2 * (u * u + v * v + w * w);
        primKnown = true;
      } else if (bc == BC_SLAB_COPY) {  // an x-slab's periodic x face: already copied by the plane exchange
        for (int f = 0; f < 5; ++f) cv[f] = ld(f, n);
      } else if (bc == NSF_BC_PERIODIC) {  // Boundary.cpp:344-367, opposite index :111-133
        int src[3] = {ijk[0], ijk[1], ijk[2]};
        periodic_source(G, axis, side, src);
        const long long m = src[0] * G.sI + src[1] * G.sJ + src[2];
        for (int f = 0; f < 5; ++f) cv[f] = ld(f, m);
      } else {  // symmetry, Boundary.cpp:377-417: mirror the primitives of the second interior node
        const Prim q = prims_of(C, ld(0, a2), ld(1, a2), ld(2, a2), ld(3, a2), ld(4, a2));
        u = q.u;
        v = q.v;
        w = q.w;
        if (axis == 0) u = -q.u;
        if (axis == 1) v = -q.v;
        if (axis == 2) w = -q.w;
        p = q.p;
        T = q.T;
        cons_of(C, u, v, w, p, T, cv);
        primKnown = true;
      }
      for (int f = 0; f < 5; ++f) O[f][n] = cv[f];
      if (s == 3) {
        const uint8_t t = G.type[n] & TYPE_MASK;
        if (t == FLUID_EDGE || t == FLUID_GHOST) {
          if (primKnown)
            dt_terms_known(C, cv[0], u, v, w, p, T, dta);
          else
            dt_terms_bc(C, cv, dta);
          for (int f = 0; f < 5; ++f) bad |= !isfinite(cv[f]);
        }
      }
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Near-body filter (ImmersedBoundary::filterClosestFluidNodes, Boundary.cpp:618-652). Jacobi: every
// filtered value is computed from unfiltered neighbours; results go to fnew and are written back by
// the ghost pass. The values before the filter go to fpre: the reference does not recompute the primitive
// variables of these nodes after filtering, so the next stage builds their primitives from fpre.
// filter_item: filter node f of a grid (stage-4 dt terms, change norms of rho and rho_E, NaN check).
// filter_node: the same with the slot's constants in hand (its node, fsolid bits and fmeta word).
__device__ __forceinline__ void filter_node(const Grid& G, const StepCtl* c, int s, int f, long long n, unsigned sb,
                                            int meta, DtAcc& dta, double nsum[5], int& bad) {
  double* const* O = c->O[s];
  auto r = [&](long long m, int q) { return ld_res(c, s, 0, m, (sb >> q) & 1); };
  auto e = [&](long long m, int q) { return ld_res(c, s, 4, m, (sb >> q) & 1); };
  const double r0 = r(n, 0), e0 = e(n, 0);
  const double rf =
      (6 * r0 + r(n + G.sI, 1) + r(n - G.sI, 2) + r(n + G.sJ, 3) + r(n - G.sJ, 4) + r(n + 1, 5) + r(n - 1, 6)) / 12;
  const double ef =
      (6 * e0 + e(n + G.sI, 1) + e(n - G.sI, 2) + e(n + G.sJ, 3) + e(n - G.sJ, 4) + e(n + 1, 5) + e(n - 1, 6)) / 12;
  G.fpre[2 * f] = r0;
  G.fpre[2 * f + 1] = e0;
  G.fnew[2 * f] = rf;
  G.fnew[2 * f + 1] = ef;
  // stage 4: the node's dt and change-norm terms, once, from its last slot (a node two bodies filter has
  // two): the final filtered values, and primitives from the values before the node's first filter
  if (s == 3 && (meta & FMETA_LAST)) {
    const int first = meta & ~FMETA_LAST;
    const double p0 = first == f ? r0 : __ldcg(G.fpre + 2 * first);
    const double p4 = first == f ? e0 : __ldcg(G.fpre + 2 * first + 1);
    const Prim q = prims_of_nr(G.C, p0, __ldcg(O[1] + n), __ldcg(O[2] + n), __ldcg(O[3] + n), p4);
    dt_terms_known(G.C, rf, q.u, q.v, q.w, q.p, q.T, dta);
    const double d0 = __ldcg(c->U0[0] + n) - rf, d4 = __ldcg(c->U0[4] + n) - ef;
    nsum[0] += d0 * d0;
    nsum[4] += d4 * d4;
    bad |= !isfinite(rf) || !isfinite(ef);
  }
}

__device__ __forceinline__ void filter_item(const Grid& G, const StepCtl* c, int s, int f, DtAcc& dta, double nsum[5],
                                            int& bad) {
  filter_node(G, c, s, f, G.fnode[f], G.fsolid ? G.fsolid[f] : 0u, G.fmeta ? G.fmeta[f] : (f | FMETA_LAST), dta, nsum,
              bad);
}

// Ghost nodes (Boundary.cpp:432-456): image-point value = cached weights x the 8 surrounding values
// (Neumann weights for rho and rho_E, Dirichlet weights for the momenta, zero weight on ghost corners);
// ghost value = image value with momentum negated (getGhostNodeBCVariables, :777-785). The ghost lists
// are stored sorted by image-point cell, so the lanes of a warp gather overlapping corner sets; every
// corner's five values are loaded before any is used (40 independent loads in flight per ghost) and summed
// in corner order, skipping corners whose two weights are both zero, as the reference's sums do.
// ghost_pass_item: item q of the ghost pass: q < nGhost a ghost, then the filter write-backs (ghosts read
// the filtered values through fnew), then on stage 4 the solid inactive nodes' dt terms (the reference
// never updates their primitive values).
// ghost_node, write_back_node, inactive_node: the three kinds with the item's node in hand; cell(m): the node of
// corner m of ghost q's image-point cell.
template <class Cell>
__device__ __forceinline__ void ghost_node(const Grid& G, const StepCtl* c, int s, int q, long long n, Cell cell,
                                           DtAcc& dta, int& bad) {
  double* const* O = c->O[s];
  const double* w = G.gw + 16 * (long long)q;
  // every load that depends on nothing first, then the filter corners' filtered values: two memory round trips
  double v[8][5], wn[8], wd[8];
  int src[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const long long cn = cell(m);
    src[m] = G.gsrc[8 * (long long)q + m];
    wn[m] = w[m];
    wd[m] = w[8 + m];
#pragma unroll
    for (int f = 0; f < 5; ++f) v[m][f] = __ldcg(O[f] + cn);
  }
#pragma unroll
  for (int m = 0; m < 8; ++m)
    if (src[m] >= 0) {  // a filter corner: the filtered values it sees
      v[m][0] = __ldcg(G.fnew + 2 * src[m]);
      v[m][4] = __ldcg(G.fnew + 2 * src[m] + 1);
    }
  double ip[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    if (wn[m] == 0.0 && wd[m] == 0.0) continue;
    ip[0] += wn[m] * v[m][0];
    ip[4] += wn[m] * v[m][4];
    ip[1] += wd[m] * v[m][1];
    ip[2] += wd[m] * v[m][2];
    ip[3] += wd[m] * v[m][3];
  }
  const double gc[5] = {ip[0], -ip[1], -ip[2], -ip[3], ip[4]};
  for (int f = 0; f < 5; ++f) O[f][n] = gc[f];
  if (s == 3 && G.glast[q]) {  // a node in two bodies' ghost lists: the dt terms of its final values
    dt_terms_bc(G.C, gc, dta);
    for (int f = 0; f < 5; ++f) bad |= !isfinite(gc[f]);
  }
}

__device__ __forceinline__ void write_back_node(const Grid& G, const StepCtl* c, int s, int f, long long n) {
  const double r = __ldcg(G.fnew + 2 * f), e = __ldcg(G.fnew + 2 * f + 1);
  c->O[s][0][n] = r;
  c->O[s][4][n] = e;
}

__device__ __forceinline__ void inactive_node(const Grid& G, const StepCtl* c, int s, int z, long long n, DtAcc& dta) {
  const double* pr = G.iprim + 5 * (long long)z;
  const double r0 = ld_res(c, s, 0, n, true);  // inactive nodes lie off the mesh faces
  if (isnan(pr[0])) {  // periodic copy of a node whose primitives follow its conserved values
    const double v[5] = {r0, ld_res(c, s, 1, n, true), ld_res(c, s, 2, n, true), ld_res(c, s, 3, n, true),
                         ld_res(c, s, 4, n, true)};
    dt_terms_bc(G.C, v, dta);
  } else {
    dta.add(G.C, r0, pr[0], pr[1], pr[2], pr[3], pr[4]);
  }
}

__device__ __forceinline__ void ghost_pass_item(const Grid& G, const StepCtl* c, int s, int q, DtAcc& dta, int& bad) {
  if (q < G.nGhost) {
    const long long* cell = G.gcell + 8 * (long long)q;
    ghost_node(G, c, s, q, G.gnode[q], [&](int m) { return cell[m]; }, dta, bad);
  } else if (q < G.nGhost + G.nFilter) {
    write_back_node(G, c, s, q - G.nGhost, G.fnode[q - G.nGhost]);
  } else {
    const int z = q - G.nGhost - G.nFilter;
    inactive_node(G, c, s, z, G.inode[z], dta);
  }
}

__device__ __forceinline__ int ghost_pass_count(const Grid& G, int s) {
  return G.nGhost + G.nFilter + (s == 3 ? G.nInactive : 0);
}

// ----------------------------------------------------------------------------------------------
// End of step: change norms (Mesh::getNormOfChange, Mesh.cpp:171-178), next dt
// (Solver::updateTimeStepSize, Solver.cpp:80-126), t += dt, ++timeLevel, history row.
// finish_step: t, dt and the time level from the step's dt maxima, by one thread; c may be a shared-memory copy
// of the control block (the whole-step kernel: every block finishes its own copy). history_row: the finished
// step's row. finalize_grid: both, with the reductions of a grid whose partial sums and maxima lie in global
// memory, by every thread of one block; red: 5 x 32 doubles of shared memory.
__device__ inline void finish_step(const Grid& G, StepCtl* c, const double mx[4]) {
  const Consts& C = G.C;
  const double conv = C.convLim / (mx[0] / C.dx + mx[1] / C.dy + mx[2] / C.dz);
  const double visc = C.viscLim / (mx[3] * C.invD2);
  const double tNew = c->t + c->dtUsed;
  double dt = (visc < conv) ? visc : conv;
  if (C.endTime && tNew + dt > C.tEnd) dt = C.tEnd - tNew;
  if (G.dtFrozen && c->level + 1 < (unsigned long long)G.nDtFrozen) dt = G.dtFrozen[c->level + 1];
  c->t = tNew;
  c->dt = dt;
  c->level += 1;
}

// Entry q of the history row (t after the step, dt used, the five norms).
__device__ inline void history_entry(const Grid& G, unsigned long long level, double tNew, double dtUsed,
                                     const double tot[5], int q) {
  const bool kept = (q == 2 && G.C.convHistory != 0) || G.C.convHistory == 2;
  G.hist[7 * (level % MAX_HIST) + q] = q == 0 ? tNew : q == 1 ? dtUsed : kept ? sqrt(G.C.dxdydz * tot[q - 2]) : -1.0;
}

__device__ inline void finalize_grid(Grid* g, double* red) {
  __shared__ double tot[5];
  const int nSlots = g->nNormSlots;
  StepCtl* c = g->ctl;
  double s[5] = {0, 0, 0, 0, 0};
  for (int q = threadIdx.x; q < nSlots; q += blockDim.x)
    for (int f = 0; f < 5; ++f) s[f] += __ldcg(g->normPart + 5 * q + f);
  flush_norms(tot, s, red);
  if (threadIdx.x < 7) history_entry(*g, c->level, c->t + c->dtUsed, c->dtUsed, tot, threadIdx.x);
  __syncthreads();
  if (threadIdx.x != 0) return;
  double mx[4];
  for (int q = 0; q < 4; ++q) mx[q] = __longlong_as_double(static_cast<long long>(atomicAdd(&c->mx[q], 0ull)));
  finish_step(*g, c, mx);
}

// ----------------------------------------------------------------------------------------------
// Start of a step: Simulation::checkStoppingCriterion (end_time), Mesh::checkFilterCondition (Mesh.cpp:85-103),
// the buffer swaps of Mesh.cpp:133-151 expressed as role changes, and per-stage buffer roles. One warp: every
// lane takes the (uniform) decisions, lane f < 5 the roles of field f, so the loads and stores of the five
// fields overlap instead of following one another. c may be a shared-memory copy of the control block;
// keepHist: this warp records the control block of the step (Grid::ctlHist).
__device__ inline void prologue_warp(const Grid& G, StepCtl* c, int lane, bool keepHist) {
  const Consts& C = G.C;
  const double t = c->t, dt = c->dt;
  const unsigned long long level = c->level;
  const int active = C.endTime ? (t < C.tEnd) : 1;
  if (lane == 0) c->active = active;
  if (!active) return;
  int counter = 0;
  for (int q = 0; q < C.nChange; ++q)
    if (t > C.changeT[q]) ++counter;
  int filt = 0;
  if (counter < C.nFilterIv) {
    const unsigned iv = C.filterIv[counter];
    if (iv > 0)
      filt = level < 0xffffffffull ? (static_cast<unsigned>(level) + 1u) % iv == 0 : (level + 1) % iv == 0;
  }
  if (lane < 5) {
    const int f = lane;
    int cons = c->perm[f][0], old = c->perm[f][1];
    const int scr = c->perm[f][2];
    const bool swapRho = filt && f == 0;
    if (swapRho) {  // the filter writes rho into the old buffer, then the two rho buffers trade places
      c->gfSrc = G.bufs[cons][0];
      c->gfDst = G.bufs[old][0];
      const int x = cons;
      cons = old;
      old = x;
    }
    {  // swapConservedVariables
      const int x = cons;
      cons = old;
      old = x;
    }
    // stage 1 of a filter step cannot write the unfiltered density it reads: it writes the scratch buffer
    const int A = swapRho ? scr : cons, B = swapRho ? cons : scr;
    double* const pOld = G.bufs[old][f];
    double* const pA = G.bufs[A][f];
    double* const pB = G.bufs[B][f];
    c->u0Phys[f] = old;
    c->iPhys[0][f] = old;
    c->iPhys[1][f] = A;
    c->iPhys[2][f] = B;
    c->iPhys[3][f] = A;
    if (f == 0) {
      c->rPhys[0] = filt ? cons : old;
      c->rPhys[1] = A;
      c->rPhys[2] = B;
      c->rPhys[3] = A;
      c->R[0] = filt ? G.bufs[cons][0] : pOld;
      c->R[1] = pA;
      c->R[2] = pB;
      c->R[3] = pA;
    }
    c->U0[f] = pOld;
    c->I[0][f] = pOld;
    c->O[0][f] = pA;
    c->I[1][f] = pA;
    c->O[1][f] = pB;
    c->I[2][f] = pB;
    c->O[2][f] = pA;
    c->I[3][f] = pA;
    c->O[3][f] = pB;
    c->perm[f][0] = B;  // roles after the step: final state = B, scratch = A
    c->perm[f][1] = old;
    c->perm[f][2] = A;
  } else if (lane == 5) {
    c->filterNow = filt;
    c->copyMask[0] = filt ? 1 : 0;
    c->copyMask[1] = c->copyMask[2] = c->copyMask[3] = 31;
    c->dtUsed = dt;
    c->stageT[0] = t + dt / 2;
    c->stageT[1] = t + dt / 2;
    c->stageT[2] = t + dt;
    c->stageT[3] = t + dt;
  } else if (lane < 10) {
    c->mx[lane - 6] = 0ull;
  }
  __syncwarp();
  if (keepHist && G.ctlHist && level < (unsigned long long)G.nCtlHist) {
    static_assert(sizeof(StepCtl) % 8 == 0, "copied as 8-byte words");
    const unsigned long long* a = reinterpret_cast<const unsigned long long*>(c);
    unsigned long long* b = reinterpret_cast<unsigned long long*>(G.ctlHist + level);
    for (int q = lane; q < int(sizeof(StepCtl) / 8); q += 32) b[q] = a[q];
  }
}

// Mesh::applyFilter_ifAppropriate body (Mesh.cpp:110-134) at one node (see k_density_filter). Reads through
// L2: the whole-step kernel runs it on values other blocks wrote in the same launch.
__device__ __forceinline__ void density_filter_node(const Grid& G, const StepCtl* c, long long n) {
  const double* src = c->gfSrc;
  double* dst = c->gfDst;
  const long long sI = G.sI, sJ = G.sJ;
  const uint8_t raw = G.type[n], t = raw & TYPE_MASK;
  if (t == FLUID_INTERIOR)
    dst[n] = (6 * __ldcg(src + n) + __ldcg(src + n + sI) + __ldcg(src + n - sI) + __ldcg(src + n + sJ) +
              __ldcg(src + n - sJ) + __ldcg(src + n + 1) + __ldcg(src + n - 1)) / 12;
  else if (t != SOLID_INACTIVE || (raw & EDGE_PLANE_BIT))
    dst[n] = __ldcg(src + n);
}

// A thread's boundary item with its constants resolved (list entry, node, flags), so that running it starts with
// its field reads. The list entry, the node and the flags would each cost a trip to L2 (an acquire of a grid
// barrier empties the SM's L1): the boundary kernel resolves the next level's item before the barrier, the
// whole-step kernel resolves its items once per launch. Node indices are 32-bit: the 20 field
// arrays of 2^31 nodes would take 344 GB.
enum BcItemKind { BC_NONE = 0, BC_SOLID, BC_EDGE, BC_FILTER, BC_GHOST, BC_WRITE_BACK, BC_INACTIVE };
struct BcItem {
  int kind;     // BcItemKind, and above bit 8: edge: reads a solid node (EdgeBlock::solidSrc), filter: fsolid
  int q;        // face, filter slot, ghost or inactive entry
  int n;        // node (edge: first in-plane coordinate)
  int aux;      // edge: second in-plane coordinate; filter: fmeta; ghost: first corner of its cell
};

// Items of level L (0-based, nsf_bc_plan.cpp) of member g in one index range: solid copies (level 0; stage 1
// copies none without a filter step and skips them), edge-block threads (64 per block), filter items, ghost-pass
// items. Each of the member's threads takes every nthr-th index, so items of different kinds run side by side
// rather than one list after another.
__device__ __forceinline__ int bc_level_items(const Grid& G, const BcParams& P, int g, int L) {
  const int M = P.members;
  const int* es = P.edgeStart + L * (M + 1) + g;
  const int* fs = P.itemStart + (L * 2) * (M + 1) + g;
  const int* hs = fs + (M + 1);
  return (L == 0 ? G.nSolid : 0) + 64 * (es[1] - es[0]) + (fs[1] - fs[0]) + (hs[1] - hs[0]);
}

__device__ __forceinline__ BcItem bc_level_item(const Grid& G, const BcParams& P, int g, int L, int v) {
  BcItem it{BC_NONE, 0, 0, 0};
  const int M = P.members;
  const int* es = P.edgeStart + L * (M + 1) + g;
  const int* fs = P.itemStart + (L * 2) * (M + 1) + g;
  const int* hs = fs + (M + 1);
  const int e0 = es[0], f0 = fs[0], h0 = hs[0];
  const int nS = L == 0 ? G.nSolid : 0, nE = 64 * (es[1] - e0), nF = fs[1] - f0, nH = hs[1] - h0;
  if (v < nS) {
    it.kind = BC_SOLID;
    it.n = int(G.snode[v]);
  } else if ((v -= nS) < nE) {
    const EdgeBlock eb = P.edges[e0 + (v >> 6)];
    const int lane = v & 63, axis = G.eAxis[eb.e];
    const int* b = G.eBox[eb.e];
    const int a = eb.a0 + (lane >> 5), bb = eb.b0 + (lane & 31), ax1 = axis == 0 ? 1 : 0, ax2 = axis == 2 ? 1 : 2;
    if (a <= b[2 * ax1 + 1] && bb <= b[2 * ax2 + 1] && ((eb.mask >> lane) & 1))
      it = BcItem{BC_EDGE | int((eb.solidSrc >> lane) & 1) << 8, eb.e, a, bb};
  } else if ((v -= nE) < nF) {
    const int f = P.items[f0 + v];
    it = BcItem{BC_FILTER | int(G.fsolid[f]) << 8, f, int(G.fnode[f]), G.fmeta[f]};
  } else if ((v -= nF) < nH) {
    const int q = P.items[h0 + v];
    if (q < G.nGhost)
      it = BcItem{BC_GHOST, q, int(G.gnode[q]), int(G.gcell[8 * (long long)q])};
    else if (q < G.nGhost + G.nFilter)
      it = BcItem{BC_WRITE_BACK, q - G.nGhost, int(G.fnode[q - G.nGhost]), 0};
    else
      it = BcItem{BC_INACTIVE, q - G.nGhost - G.nFilter, int(G.inode[q - G.nGhost - G.nFilter]), 0};
  }
  return it;
}

// LAST: s == 3; without it the item functions see s <= 2 and drop the dt terms, change norms and NaN check.
template <bool LAST>
__device__ __forceinline__ void bc_run_item(const Grid& G, const StepCtl& cs, int sArg, const BcItem& it, DtAcc& dta,
                                         double (&nsum)[5], int& bad) {
  const int s = LAST ? 3 : min(sArg, 2);
  switch (it.kind & 0xff) {
    case BC_SOLID: {
      const int mask = cs.copyMask[s];
      if (mask) solid_copy_node(&cs, s, mask, it.n);
      break;
    }
    case BC_EDGE: {
      const EdgeBlock eb{0, it.q, it.n, it.aux, 1ull, static_cast<unsigned long long>(it.kind >> 8)};
      edge_node(G, &cs, eb, 0, 0, s, G.eAxis[it.q], dta, bad);
      break;
    }
    case BC_FILTER:
      filter_node(G, &cs, s, it.q, it.n, unsigned(it.kind) >> 8, it.aux, dta, nsum, bad);
      break;
    case BC_GHOST: {  // the corners of an image-point cell: k fastest, i slowest (box_corners)
      const long long c0 = it.aux;
      auto cell = [&](int m) { return c0 + (m >> 2) * G.sI + ((m >> 1) & 1) * G.sJ + (m & 1); };
      ghost_node(G, &cs, s, it.q, it.n, cell, dta, bad);
      break;
    }
    case BC_WRITE_BACK:
      write_back_node(G, &cs, s, it.q, it.n);
      break;
    case BC_INACTIVE:
      if (LAST) inactive_node(G, &cs, s, it.q, it.n, dta);
      break;
    default:
      break;
  }
}

}  // namespace nsf
#endif
