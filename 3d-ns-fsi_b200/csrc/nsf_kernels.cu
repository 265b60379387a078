// CUDA kernels (sm_100a, FP64) of the RK4 time-marching path. Grids up to kStepMaxNodes (nsf_capi.cpp) run whole steps
// in one kernel (nsf_step.cu); of the others one RK4 step (Solver::marchTimeStep, Solver.cpp:130-167) is the launch
// sequence enqueue_step() builds, in which k_bc takes everything between two stage kernels, and the end of the step, in
// one launch; the kernels it stands for run by themselves where a boundary plan is not built or the adjoint's
// recomputation must read the state between them:
//
//   k_prologue            stop criterion, filter decision, buffer roles        (Solver.cpp:133-135)
//   k_density_filter      global 2nd-order density filter, rare              (Mesh.cpp:108-140)
//   4 x { k_stage_ws      fused RHS + primitive recompute + RK4 combine      (Solver.cpp:141-159, 170-507;
//                         TMA-fed, warp-specialised: nsf_stage_ws.cu)
//         k_solid_copy    stale solid-node values, I -> O                    (buffer semantics, see nsf_device.cuh)
//         k_edge_bc x3    outlet/inlet, then y faces, then z faces           (Boundary.cpp:250-417)
//         k_body_filter   near-body filter of rho, rho_E                     (Boundary.cpp:618-652)
//         k_ghost         image-point interpolation with cached weights      (Boundary.cpp:427-457, 655-883) }
//   k_finalize            change norms, next dt, time, history              (Solver.cpp:80-126, 510-530)
//
// Stage 4 also carries the dt maxima, the change norms and the NaN check as block reductions, so no
// kernel re-reads the fields for them.
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cuda_runtime.h>

#include "nsf_bc_items.cuh"
#include "nsf_device.cuh"
#include "nsf_internal.h"
#include "nsf_physics.cuh"

namespace nsf {

// ----------------------------------------------------------------------------------------------
// Start of a step (prologue_warp). Member m = blockIdx.x of the grid array (a single grid: one block).
__global__ void k_prologue(Grid* grids) {
  const Grid& G = grids[blockIdx.x];
  prologue_warp(G, G.ctl, threadIdx.x, true);
}

// Mesh::applyFilter_ifAppropriate body (Mesh.cpp:110-134): interior nodes get the 7-point filter,
// every node of an edge boundary's owned box (whatever its type) and every solid-ghost node is copied,
// the remaining solid inactive nodes are left as they are.
__global__ void k_density_filter(const Grid* __restrict__ grids) {
  const Grid* g = grids + blockIdx.y;
  const StepCtl* c = g->ctl;
  if (!c->active || !c->filterNow) return;
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < g->N; n += (long long)gridDim.x * blockDim.x)
    density_filter_node(*g, c, n);
}

__global__ void k_solid_copy(const Grid* __restrict__ grids, int s) {
  const Grid* g = grids + blockIdx.y;
  const StepCtl* c = g->ctl;
  if (!c->active) return;
  const int mask = c->copyMask[s];
  if (!mask) return;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < g->nSolid; q += gridDim.x * blockDim.x)
    solid_copy_item(*g, c, s, mask, q);
}


__global__ void k_edge_bc(const Grid* __restrict__ grids, const EdgeBlock* __restrict__ blocks, int s, int axis) {
  __shared__ double red[4 * 32];
  const EdgeBlock eb = blocks[blockIdx.x];  // every listed block holds nodes of its face
  const Grid& G = grids[eb.g];
  StepCtl* c = G.ctl;
  if (!c->active) return;
  DtAcc dta;
  int bad = 0;
  edge_node(G, c, eb, threadIdx.x, threadIdx.y, s, axis, dta, bad);
  if (s == 3) {
    flush_dt(c, dta, red);
    if (bad) atomicOr(&c->nonFinite, 1);
  }
}


__global__ void k_body_filter(const Grid* __restrict__ grids, int s) {
  __shared__ double red[5 * 32];
  const Grid& G = grids[blockIdx.y];
  StepCtl* c = G.ctl;
  if (!c->active) return;
  DtAcc dta;
  double nsum[5] = {0, 0, 0, 0, 0};
  int bad = 0;
  // a block past this member's filter nodes never writes its norm slot, which stays zero
  if (int(blockIdx.x * blockDim.x) >= G.nFilter) return;
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < G.nFilter; f += gridDim.x * blockDim.x)
    filter_item(G, c, s, f, dta, nsum, bad);
  if (s == 3) {
    flush_dt(c, dta, red);
    flush_norms(G.normPart + 5 * (G.normSlotFilter + blockIdx.x), nsum, red);
    if (bad) atomicOr(&c->nonFinite, 1);
  }
}


__global__ void k_ghost(const Grid* __restrict__ grids, int s) {
  __shared__ double red[4 * 32];
  const Grid& G = grids[blockIdx.y];
  StepCtl* c = G.ctl;
  if (!c->active) return;
  DtAcc dta;
  int bad = 0;
  const int total = ghost_pass_count(G, s);
  if (int(blockIdx.x * blockDim.x) >= total) return;  // the whole block is past this member's work
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x)
    ghost_pass_item(G, c, s, q, dta, bad);
  if (s == 3) {
    flush_dt(c, dta, red);
    if (bad) atomicOr(&c->nonFinite, 1);
  }
}


__global__ void k_finalize(Grid* grids) {
  __shared__ double red[5 * 32];
  Grid* g = grids + blockIdx.x;
  if (!g->ctl->active) return;
  finalize_grid(g, red);
}

// ----------------------------------------------------------------------------------------------
// Setup: interpolation weights of every ghost node, solved once. For image-point cells whose eight
// nodes are all fluid the weights are those of the reference's nested linear interpolation
// (Boundary.cpp:732-757). Otherwise the reference solves V c = phi with the Vandermonde rows
// [1, x, y, z, xy, xz, yz, xyz] (Neumann rows [0, n, ...] at ghost corners, Boundary.cpp:788-817) and
// evaluates b^T c at the image point; the value is w^T phi with V^T w = b. The system is solved here in
// cell-local scaled coordinates x' = (x - x0)/dx (the bilinear basis is invariant under per-axis affine
// maps; a Neumann row transforms with n'_a = n_a/d_a), which keeps its condition number near 10 instead
// of ~1e6 for the raw coordinates. Gaussian elimination with partial pivoting, in registers, one thread
// per ghost.
__device__ void solve8T(double A[8][8], double b[8]) {
  // solve A^T x = b in place (x returned in b)
  double M[8][8];
  for (int r = 0; r < 8; ++r)
    for (int q = 0; q < 8; ++q) M[r][q] = A[q][r];
  for (int k = 0; k < 8; ++k) {
    int piv = k;
    double best = fabs(M[k][k]);
    for (int r = k + 1; r < 8; ++r)
      if (fabs(M[r][k]) > best) {
        best = fabs(M[r][k]);
        piv = r;
      }
    if (piv != k) {
      for (int q = 0; q < 8; ++q) {
        double t = M[k][q];
        M[k][q] = M[piv][q];
        M[piv][q] = t;
      }
      double t = b[k];
      b[k] = b[piv];
      b[piv] = t;
    }
    for (int r = k + 1; r < 8; ++r) {
      const double l = M[r][k] / M[k][k];
      for (int q = k; q < 8; ++q) M[r][q] -= l * M[k][q];
      b[r] -= l * b[k];
    }
  }
  for (int k = 7; k >= 0; --k) {
    double acc = b[k];
    for (int q = k + 1; q < 8; ++q) acc -= M[k][q] * b[q];
    b[k] = acc / M[k][k];
  }
}

// in: per ghost 8 x (x, y, z) corner points (node position, or body-intercept point for a ghost corner),
// 8 x (nx, ny, nz) unit normals (ghost corners only), 8 flags, image point, lower cell node position.
__global__ void k_ghost_weights(int nGhost, const double* __restrict__ pts, const double* __restrict__ nrm,
                                const uint8_t* __restrict__ flags, const double* __restrict__ ipl,
                                double dx, double dy, double dz, double* __restrict__ wout) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nGhost) return;
  const double* P = pts + 24 * (long long)q;
  const double* Nn = nrm + 24 * (long long)q;
  const uint8_t* fl = flags + 8 * (long long)q;
  const double* L = ipl + 6 * (long long)q;  // image point, lower node position
  const double X = (L[0] - L[3]) / dx, Y = (L[1] - L[4]) / dy, Z = (L[2] - L[5]) / dz;
  double* w = wout + 16 * (long long)q;
  bool anyGhost = false;
  for (int m = 0; m < 8; ++m) anyGhost |= fl[m] != 0;
  if (!anyGhost) {
    // corner m = (di, dj, dk) in asIndexList order: m = 4*di + 2*dj + dk
    for (int m = 0; m < 8; ++m) {
      const int di = m >> 2, dj = (m >> 1) & 1, dk = m & 1;
      const double wv = (di ? X : 1 - X) * (dj ? Y : 1 - Y) * (dk ? Z : 1 - Z);
      w[m] = wv;
      w[8 + m] = wv;
    }
    return;
  }
  for (int set = 0; set < 2; ++set) {  // 0: Neumann rows at ghost corners, 1: Dirichlet everywhere
    double V[8][8], b[8];
    for (int m = 0; m < 8; ++m) {
      const double x = (P[3 * m] - L[3]) / dx, y = (P[3 * m + 1] - L[4]) / dy, z = (P[3 * m + 2] - L[5]) / dz;
      if (set == 0 && fl[m]) {
        const double nx = Nn[3 * m] / (1.0 / dx), ny = Nn[3 * m + 1] / (1.0 / dy), nz = Nn[3 * m + 2] / (1.0 / dz);
        // gradient of the basis in scaled coordinates: d/dx = (1/dx) d/dx'; the row is n . grad
        const double ax = nx / (dx * dx), ay = ny / (dy * dy), az = nz / (dz * dz);
        V[m][0] = 0;
        V[m][1] = ax;
        V[m][2] = ay;
        V[m][3] = az;
        V[m][4] = x * ay + y * ax;
        V[m][5] = x * az + z * ax;
        V[m][6] = y * az + z * ay;
        V[m][7] = x * y * az + x * z * ay + y * z * ax;
      } else {
        V[m][0] = 1;
        V[m][1] = x;
        V[m][2] = y;
        V[m][3] = z;
        V[m][4] = x * y;
        V[m][5] = x * z;
        V[m][6] = y * z;
        V[m][7] = x * y * z;
      }
    }
    b[0] = 1;
    b[1] = X;
    b[2] = Y;
    b[3] = Z;
    b[4] = X * Y;
    b[5] = X * Z;
    b[6] = Y * Z;
    b[7] = X * Y * Z;
    solve8T(V, b);
    for (int m = 0; m < 8; ++m) w[8 * set + m] = fl[m] ? 0.0 : b[m];
  }
}

// Snapshot of the fields a download asks for, packed in the reference's layout (k fastest, no row padding):
// field f goes to out + slot[f] * NI*NJ*NK, or nowhere for slot -1. Conserved fields are the current
// buffers; primitive / transport fields are recomputed from them as the reference holds them, except at
// filtered nodes (values before the last near-body filter) and solid inactive nodes (never updated by the
// reference; k_snapshot_inactive writes their stored values). The buffers are found through the control
// block, so the kernel can be queued behind any number of steps without the host reading it.
__global__ void k_snapshot(const Grid* __restrict__ gp, SnapSlots sl, double* __restrict__ out) {
  const Grid& G = *gp;
  const StepCtl* c = G.ctl;
  const Consts& C = G.C;
  const double* U[5];
  for (int f = 0; f < 5; ++f) U[f] = G.bufs[c->perm[f][0]][f];
  bool prim = false;
#pragma unroll
  for (int f = 5; f < NSF_SNAP_FIELDS; ++f) prim |= sl.slot[f] >= 0;
  const long long NK = G.NK, M = (long long)G.NI * G.NJ * NK;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < M; q += (long long)gridDim.x * blockDim.x) {
    const long long n = (q / NK) * G.NKp + q % NK;
    double v[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      v[f] = U[f][n];
      if (sl.slot[f] >= 0) out[sl.slot[f] * M + q] = v[f];
    }
    if (!prim) continue;
    if (G.type[n] & FILTER_BIT) {
      const int f = G.fidx[n];
      v[0] = G.fpre[2 * f];
      v[4] = G.fpre[2 * f + 1];
    }
    const Prim p = prims_of(C, v[0], v[1], v[2], v[3], v[4]);
    const double pv[7] = {p.u, p.v, p.w, p.p, p.T, p.mu, p.ka};
#pragma unroll
    for (int f = 0; f < 7; ++f)
      if (sl.slot[5 + f] >= 0) out[sl.slot[5 + f] * M + q] = pv[f];
  }
}

// Solid inactive nodes of a snapshot: their stored primitive values, from the list for the time level the
// control block holds (level 0: each node's own initial values; later: the values after the first step).
__global__ void k_snapshot_inactive(const Grid* __restrict__ gp, SnapSlots sl, SnapInactive in,
                                    double* __restrict__ out) {
  const Grid& G = *gp;
  const bool ic = G.ctl->level == 0;
  const long long* nodes = ic ? in.nodesIc : in.nodes;
  const double* p7 = ic ? in.p7Ic : in.p7;
  const int count = ic ? in.countIc : in.count;
  const long long NK = G.NK, M = (long long)G.NI * G.NJ * NK;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
    const long long n = nodes[q], cq = (n / G.NKp) * NK + n % G.NKp;
#pragma unroll
    for (int f = 0; f < 7; ++f)
      if (sl.slot[5 + f] >= 0) out[sl.slot[5 + f] * M + cq] = p7[7 * (long long)q + f];
  }
}

// ----------------------------------------------------------------------------------------------
// Fused boundary kernel: everything a stage does after its stage kernel, in one cooperative launch of
// bcBlocks blocks (a consecutive range of them per member, sized by its work), in the dependency levels of
// nsf_bc_plan.cpp: level 0
// holds the solid-node copies and every edge, filter and ghost-pass item whose inputs are final after the
// stage kernel; each later level reads what earlier levels wrote anywhere in the member's grid, so a barrier
// over the member's blocks separates levels (members share nothing, an ensemble's members do not wait for
// one another, and each member runs only its own levels) and those reads go through L2 (__ldcg in the item
// functions). The member's Grid and control block are copied to shared memory first (every item reads
// them). Stage 4 then flushes the dt maxima, change norms and NaN flag, and the member's last block to
// finish runs the end-of-step finalize. Items wait for memory, not for arithmetic, so the trips to L2 in a row are
// what counts: an item's list entry, node and flags are resolved before the level's barrier (bc_level_item), its
// loads all go out before the first use or store, and consecutive warps of the item range lie on different
// blocks. Measured (us per step): sphere 48^3 148 -> 130, sphere 96^3 408 -> 384, 16 spheres 256x128x128
// 1015 -> 985, the 64-member ensemble 4109 -> 4069 (three resident blocks instead of four: 125, 378, 982, 4096).
// Every block of a member passes every barrier of that member (an
// inactive member's blocks do no work), so the launch is cooperative (all blocks resident).

// Resident blocks of the fused boundary kernel per SM (its registers are capped to fit): the kernel is
// latency-bound, each member's items spread over its blocks' threads.
constexpr int kBcBlocksPerSM = 4;

// LAST: stage 4 (s == 3), the one stage with dt terms, change norms and the NaN check; stages 1-3 run the
// other instantiation, whose item functions see s <= 2 and drop that work and its registers.
template <bool LAST>
__global__ void __launch_bounds__(256, kBcBlocksPerSM) k_bc(Grid* grids, const __grid_constant__ BcParams P, int sArg,
                                                            int fin) {
  const int s = LAST ? 3 : min(sArg, 2);
  __shared__ double red[5 * 32];
  __shared__ __align__(16) unsigned char gsm[sizeof(Grid)];
  __shared__ __align__(16) unsigned char csm[sizeof(StepCtl)];
  __shared__ int gShared;
  const int M = P.members, tid = threadIdx.x;
  if (tid == 0) {  // this block's member: blocks blockStart[g] .. blockStart[g + 1] - 1 work for member g
    int lo = 0, hi = M;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (P.blockStart[mid] <= int(blockIdx.x)) lo = mid; else hi = mid;
    }
    gShared = lo;
  }
  __syncthreads();
  const int g = gShared;
  const int bx = int(blockIdx.x) - P.blockStart[g], nbx = P.blockStart[g + 1] - P.blockStart[g];
  Grid* gp = grids + g;
  StepCtl* c = gp->ctl;  // global: atomics, flags and finalize write here
  {
    static_assert(sizeof(Grid) % 8 == 0 && sizeof(StepCtl) % 8 == 0, "copied as 8-byte words");
    const unsigned long long* a = reinterpret_cast<const unsigned long long*>(gp);
    const unsigned long long* b = reinterpret_cast<const unsigned long long*>(c);
    for (int q = tid; q < int(sizeof(Grid) / 8); q += blockDim.x) reinterpret_cast<unsigned long long*>(gsm)[q] = a[q];
    for (int q = tid; q < int(sizeof(StepCtl) / 8); q += blockDim.x)
      reinterpret_cast<unsigned long long*>(csm)[q] = b[q];
  }
  __syncthreads();
  const Grid& G = *reinterpret_cast<const Grid*>(gsm);
  const StepCtl& cs = *reinterpret_cast<const StepCtl*>(csm);  // read-only copy for the item functions
  const bool active = cs.active != 0;
  // warps are numbered across the member's blocks, so that a short list of items spreads over many SMs
  const int gtid = ((tid >> 5) * nbx + bx) * 32 + (tid & 31), nthr = nbx * int(blockDim.x);
  DtAcc dta;
  double nsum[5] = {0, 0, 0, 0, 0};
  int bad = 0;
  const int levels = P.memberLevels[g];
  int total = 0;
  BcItem item{BC_NONE, 0, 0, 0};  // this thread's next item
  auto resolve = [&](int L) {
    total = bc_level_items(G, P, g, L);
    if (gtid < total) item = bc_level_item(G, P, g, L, gtid);
  };
  if (levels > 0) resolve(0);
  for (int L = 0; L < levels; ++L) {
    if (L > 0) grid_barrier(P.sync + 1 + M + g, unsigned(nbx), &c->timeout);
    if (active)
      for (int v = gtid; v < total;) {
        bc_run_item<LAST>(G, cs, s, item, dta, nsum, bad);
        if ((v += nthr) < total) item = bc_level_item(G, P, g, L, v);
      }
    if (L + 1 < levels) resolve(L + 1);
  }
  if (s == 3) {
    flush_dt(c, dta, red);
    // one norm slot per block (a member has 1 + bcBlocks slots or more when a filter exists)
    if (G.nFilter > 0) flush_norms(gp->normPart + 5 * (G.normSlotFilter + bx), nsum, red);
    if (bad) atomicOr(&c->nonFinite, 1);
  }
  if (fin) {  // the member's last block to get here runs its end-of-step finalize (no waiting)
    __shared__ int last;
    __syncthreads();
    if (tid == 0) {
      const unsigned long long old = atom_add_release(P.sync + 1 + g, 1ull);
      last = (old + 1) % (unsigned long long)nbx == 0;
      if (last) (void)ld_acquire(P.sync + 1 + g);
    }
    __syncthreads();
    if (last && active) finalize_grid(gp, red);
  }
}

static void launch_bc(Grid* dg, int members, const LaunchPlan& L, int s, bool fin, cudaStream_t st) {
  BcParams P{};
  P.edges = L.bcEdges;
  P.edgeStart = L.bcEdgeStart;
  P.items = L.bcItems;
  P.itemStart = L.bcItemStart;
  P.sync = L.bcSync;
  P.blockStart = L.bcBlockStart;
  P.memberLevels = L.bcMemberLevels;
  P.levels = L.bcLevels;
  P.members = members;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(L.bcBlocks));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (s == 3)
    cudaLaunchKernelEx(&cfg, k_bc<true>, dg, P, s, fin ? 1 : 0);
  else
    cudaLaunchKernelEx(&cfg, k_bc<false>, dg, P, s, fin ? 1 : 0);
}

int bc_capacity(int nSM) {
  int nb = 0;
  int nb2 = 0;  // both instantiations run the same plan: the smaller residency bounds it
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bc<true>, 256, 0) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb2, k_bc<false>, 256, 0) != cudaSuccess) return 0;
  nb = nb2 < nb ? nb2 : nb;
  return nb * nSM;
}

// ----------------------------------------------------------------------------------------------
// Host-side launch helpers (called from nsf_capi.cpp).

void edge_blocks(const Grid& G, const uint8_t* type, int g, int axis, std::vector<EdgeBlock>& out) {
  const int ax1 = axis == 0 ? 1 : 0, ax2 = axis == 2 ? 1 : 2;
  // periodic faces whose copies the stage kernel writes: those nodes leave the blocks (z: (a, bb) = (i, j),
  // y: (a, bb) = (i, k))
  const bool fused = type && ((axis == 2 && G.zFused) || (axis == 1 && G.yFused));
  for (int e = 0; e < G.nEdge; ++e) {
    if (G.eAxis[e] != axis) continue;
    const int* b = G.eBox[e];
    const int ks = G.eSide[e] == 0 ? G.NK - 2 : 1;  // the periodic source plane
    const int js = G.eSide[e] == 0 ? G.NJ - 2 : 1;
    for (int a0 = b[2 * ax1]; a0 <= b[2 * ax1 + 1]; a0 += kEdgeRows)
      for (int b0 = b[2 * ax2]; b0 <= b[2 * ax2 + 1]; b0 += 32) {
        unsigned long long mask = ~0ull;
        if (fused && G.eBc[e] == NSF_BC_PERIODIC) {
          mask = 0;
          for (int ty = 0; ty < kEdgeRows; ++ty)
            for (int tx = 0; tx < 32; ++tx) {
              const int a = a0 + ty, bb = b0 + tx;
              if (a > b[2 * ax1 + 1] || bb > b[2 * ax2 + 1]) continue;
              const bool copiedByStage =
                  axis == 2 ? (type[(size_t(a) * G.NJ + bb) * G.NK + ks] & (ZCOPY_UP_BIT | ZCOPY_DOWN_BIT)) != 0
                            : (type[(size_t(a) * G.NJ + js) * G.NK + bb] & YCOPY_BIT) != 0;
              if (!copiedByStage) mask |= 1ull << (ty * 32 + tx);
            }
          if (!mask) continue;
        }
        out.push_back(EdgeBlock{g, e, a0, b0, mask, 0ull});
      }
  }
}

// One RK4 step for `members` grids (dg: device array of them). hg: the grid on the host for a single-grid
// solver (its stage kernel takes the grid by value), or NULL for an ensemble (the ensemble stage kernel
// reads every member from dg). The small kernels carry the member in a grid dimension, their block
// counts in L being the maxima over the members; the edge kernels run the listed blocks of every member.
// lastStage: NULL, or the plan of a partial stage 4 (single grid): stage 4 then runs the stage kernel over
// that plan's items only and the step ends there (no stage-4 boundary conditions, no finalize).
// ev: NULL, or 8 events recorded around the four stage kernels; evExternal: record them as event nodes of
// a graph being captured (cudaEventRecordExternal) rather than as plain stream events.
static int enqueue_impl(Grid* dg, const Grid* hg, int members, const LaunchPlan& L, cudaStream_t st, cudaEvent_t* ev,
                        StepHook* hook = nullptr, const LaunchPlan* lastStage = nullptr, bool evExternal = false) {
  auto record = [&](cudaEvent_t e) {
    if (evExternal)
      cudaEventRecordWithFlags(e, st, cudaEventRecordExternal);
    else
      cudaEventRecord(e, st);
  };
  int launches = 0;
  const unsigned M = unsigned(members);
  // the fused boundary kernel, unless a hook must run between the solid-node copy and the edge conditions
  // (a partial last stage ends before its boundary work, fused or not)
  const bool fused = L.bcBlocks > 0 && (!hook || !hook->wants_before_edges());
  k_prologue<<<M, 32, 0, st>>>(dg);
  ++launches;
  if (hook) hook->after_prologue();
  k_density_filter<<<dim3(L.gfBlocks, M), 256, 0, st>>>(dg);
  ++launches;
  for (int s = 0; s < 4; ++s) {
    if (ev) record(ev[2 * s]);
    if (hook) hook->before_stage(s);
    if (s == 3 && lastStage && hg) {
      if (lastStage->nItems > 0) {
        launch_stage(*hg, *lastStage, s, st);
        ++launches;
      }
      if (hook) hook->before_edges(s);
      return launches;
    }
    if (hg)
      launch_stage(*hg, L, s, st);
    else
      launch_stage_ensemble(dg, L, s, st);
    if (ev) record(ev[2 * s + 1]);
    ++launches;
    if (fused) {
      if (L.bcLevels > 0 || s == 3) {
        launch_bc(dg, members, L, s, s == 3, st);
        ++launches;
      }
      continue;
    }
    if (L.hasSolid) {
      k_solid_copy<<<dim3(L.solidBlocks, M), 256, 0, st>>>(dg, s);
      ++launches;
    }
    if (hook) hook->before_edges(s);
    for (int a = 0; a < 3; ++a)
      if (L.nEdgeBlocks[a] > 0) {
        k_edge_bc<<<L.nEdgeBlocks[a], dim3(32, kEdgeRows), 0, st>>>(dg, L.edgeBlocks[a], s, a);
        ++launches;
      }
    if (L.hasFilter) {
      k_body_filter<<<dim3(L.filterBlocks, M), 256, 0, st>>>(dg, s);
      ++launches;
    }
    if (L.hasGhostWork) {
      k_ghost<<<dim3(L.ghostBlocks, M), 256, 0, st>>>(dg, s);
      ++launches;
    }
  }
  if (!fused) {
    k_finalize<<<M, 256, 0, st>>>(dg);
    ++launches;
  }
  return launches;
}

int enqueue_step_begin(Grid* dg, int members, const LaunchPlan& L, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  k_prologue<<<unsigned(members), 32, 0, st>>>(dg);
  k_density_filter<<<dim3(L.gfBlocks, unsigned(members)), 256, 0, st>>>(dg);
  return 2;
}

int launch_bc_part(Grid* dg, int members, const LaunchPlan& L, int s, bool fin, void* stream) {
  if (L.bcBlocks <= 0 || (L.bcLevels == 0 && !fin)) return 0;
  launch_bc(dg, members, L, s, fin, static_cast<cudaStream_t>(stream));
  return 1;
}

int enqueue_step(Grid* dg, const Grid& hg, const LaunchPlan& L, void* stream) {
  return enqueue_impl(dg, &hg, 1, L, static_cast<cudaStream_t>(stream), nullptr);
}

int enqueue_step_hooked(Grid* dg, const Grid& hg, const LaunchPlan& L, void* stream, StepHook* hook,
                        const LaunchPlan* lastStage) {
  return enqueue_impl(dg, &hg, 1, L, static_cast<cudaStream_t>(stream), nullptr, hook, lastStage);
}

int enqueue_ensemble_step(Grid* dGrids, int members, const LaunchPlan& L, void* stream, void* events) {
  return enqueue_impl(dGrids, nullptr, members, L, static_cast<cudaStream_t>(stream), static_cast<cudaEvent_t*>(events));
}

int enqueue_step_profiled(Grid* dg, const Grid& hg, const LaunchPlan& L, void* stream, void* events, bool inGraph) {
  return enqueue_impl(dg, &hg, 1, L, static_cast<cudaStream_t>(stream), static_cast<cudaEvent_t*>(events), nullptr,
                      nullptr, inGraph);
}

void launch_ghost_weights(int nGhost, const double* pts, const double* nrm, const uint8_t* flags, const double* ipl,
                          double dx, double dy, double dz, double* w, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (nGhost > 0) k_ghost_weights<<<(nGhost + 127) / 128, 128, 0, st>>>(nGhost, pts, nrm, flags, ipl, dx, dy, dz, w);
}

__global__ void k_ctl_out(const StepCtl* __restrict__ ctl, StepCtl* __restrict__ out) {
  const unsigned long long* a = reinterpret_cast<const unsigned long long*>(ctl);
  unsigned long long* b = reinterpret_cast<unsigned long long*>(out);
  for (int q = threadIdx.x; q < int(sizeof(StepCtl) / 8); q += blockDim.x) b[q] = a[q];
}

void launch_ctl_out(const StepCtl* ctl, StepCtl* out, void* stream) {
  k_ctl_out<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(ctl, out);
}

void launch_snapshot(const Grid* dg, const SnapSlots& sl, const SnapInactive& in, double* out, int nSM, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  k_snapshot<<<nSM * 8, 256, 0, st>>>(dg, sl, out);
  bool prim = false;
  for (int f = 5; f < NSF_SNAP_FIELDS; ++f) prim |= sl.slot[f] >= 0;
  const int most = in.count > in.countIc ? in.count : in.countIc;
  if (prim && most > 0) k_snapshot_inactive<<<(most + 255) / 256, 256, 0, st>>>(dg, sl, in, out);
}

// The Newton-Raphson reciprocal and square root next to the IEEE ones, for a check of their error.
__global__ void k_math_selftest(long long n, const double* __restrict__ x, double* __restrict__ out) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const double a = x[q];
    out[4 * q + 0] = recip_nr(a);
    out[4 * q + 1] = 1.0 / a;
    out[4 * q + 2] = sqrt_nr(a);
    out[4 * q + 3] = sqrt(a);
  }
}

int math_selftest(long long n, const double* hostIn, double* hostOut) {
  double *dx = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&dx, (n > 0 ? n : 1) * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&dout, 4 * (n > 0 ? n : 1) * sizeof(double));
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(dx, hostIn, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && n > 0) {
    k_math_selftest<<<int((n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024), 256>>>(n, dx, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(hostOut, dout, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dout);
  return int(e);
}

}  // namespace nsf
