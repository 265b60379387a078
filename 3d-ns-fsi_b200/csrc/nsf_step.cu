// Whole-step kernel for small grids (sm_100a, FP64): any number of RK4 steps in one cooperative launch.
//
// A grid of up to a few hundred thousand nodes gives each of the 148 SMs under two thousand nodes per stage, and
// its fields (20 arrays) lie in the 126 MB L2. What bounds its step is latency: launches, ring fills and the
// plane-by-plane march of the streaming stage kernel (nsf_stage_ws.cu), which walks six planes one after another
// to compute four. Here one block per SM stays resident for the whole call and every phase of a step is spread
// over all its threads:
//
//   start of step    every block takes the same decisions on its own shared copy of the control block
//   density filter   on filter steps only
//   4 x { stage      tiles of TK x TJ columns and L planes: the primitive values of the tile and its halo into
//                    shared memory (one pass over all threads), then the RHS and the RK4 combine, 128 columns x
//                    NT/128 groups of consecutive planes
//         boundary   the dependency levels of nsf_bc_plan.cpp, as in k_bc (nsf_kernels.cu) }
//   end of step      dt maxima and change norms: one partial per block, combined by every block
//
// Phases are separated by a grid barrier (all blocks resident; bounded polls, StepCtl::timeout). Values written
// in the launch are read through L2 (__ldcg). Arithmetic and its order per node are the streaming kernel's and
// k_bc's, so the fields equal theirs bit for bit (ensembles, x-slabs and the adjoint use those kernels).
//
// Measured (us per step: by the launch sequence / by this kernel, one B200): sphere 32^3 101 / 57, sphere 48^3 123 / 71,
// cylinder 161x83x3 188 / 82, walls and a sphere 75x53x61 158 / 131, Taylor-Green 64^3 106 / 102 (the launch sequence
// as it was before this kernel came: 119, 142, 218, 186, 111).
// A step of sphere 48^3 (SM cycles of a block at 1.9 GHz, 141 K in all): four stage phases of 13-15 K (4.3 K the
// staged planes, 9.5 K the RHS: two planes a thread, half of the FP64 rate), four boundary phases of 3-5 K edges
// and 4-6 K ghosts, a barrier about 2.2 K from the last arrival to the release (memory latency), 8 K the end and
// start of the step.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "nsf_bc_items.cuh"
#include "nsf_device.cuh"
#include "nsf_internal.h"
#include "nsf_physics.cuh"

namespace nsf {
namespace {

// Threads per block, one block per SM. Measured at 512 / 384 / 256 threads (128 / 168 / 202 registers; us per step):
// sphere 48^3 85 / 80 / 94, walls 75x53x61 149 / 140 / 171, Taylor-Green 80^3 196 / 171 / 198. With 512 the RHS
// spills, with 256 too few warps hide its latency.
constexpr int NT = 384;
constexpr int NCOL = 128;      // columns of a tile
constexpr int NG = NT / NCOL;  // groups of threads that share a tile's planes
constexpr int NQ = 9;          // end-of-step quantities: four dt maxima, five change-norm sums
constexpr int kStash = 3;      // boundary levels whose first item per thread is kept in shared memory
constexpr int kTileStash = 16;
constexpr size_t kSmemBudget = 200 * 1024;  // staged planes of a tile (227 KB a block less the stash and the copies)

struct StepParams {
  BcParams bc;
  const StageItem* items;  // tiles of block b: items[start[b] .. start[b + 1])
  const int* start;
  double* part;                // [NQ][blocks] end-of-step partials
  int stashOffset;             // bytes from the start of the dynamic shared memory to the item stash
  StepTape tape;
  unsigned long long* sync;    // the grid barrier's arrival counter (see grid_barrier, nsf_physics.cuh)
};

template <int TK_, int TJ_>
struct BT {
  static constexpr int TK = TK_, TJ = TJ_, HK = TK + 2, HJ = TJ + 2, HP = HK * HJ;
  static constexpr int FS = HP, PS = 10 * FS;  // doubles per staged field and plane: u v w p T mu, rho_u .. rho_E
  static constexpr int LMAX = int(kSmemBudget / (PS * 8)) - 2;
  static_assert(TK * TJ == NCOL && LMAX >= NG, "a tile has 128 columns and room for a plane per group");
};

// One tile of stage s (s < 3, or s == 3 with LAST). Called by every thread of the block.
template <class T, bool LAST>
__device__ __forceinline__ void stage_tile(const Grid& G, const StepCtl& c, int s, const StageItem& w, double* sm,
                                           DtAcc& dta, double (&nsum)[5], int& bad) {
  constexpr int TK = T::TK, HK = T::HK, HP = T::HP, FS = T::FS, PS = T::PS;
  const int tid = threadIdx.x;
  const int L = w.i1 - w.i0 + 1;
  const Consts& C = G.C;
  {  // primitive values of the tile and its halo; nodes past the mesh (partial tiles) are left out: no column
     // inside the mesh reads them
    const double* const q0 = c.R[s];
    const double* const q1 = c.I[s][1];
    const double* const q2 = c.I[s][2];
    const double* const q3 = c.I[s][3];
    const double* const q4 = c.I[s][4];
    const ThermoConsts TC{C.gamma, C.gm1, C.muA, C.muRe, C.pf};
    constexpr int U = 4;  // nodes a thread loads before it computes: their loads and reciprocal chains overlap
    const int total = (L + 2) * HP;
#pragma unroll 1
    for (int b0 = tid; b0 < total; b0 += U * NT) {
      double v[U][5];
      int slot[U];  // near-body filter slot, -1 for an unfiltered node, -2 outside the mesh or the tile
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = b0 + u * NT;
        const int pl = idx / HP, r = idx - pl * HP, hj = r / HK, hk = r - hj * HK;
        const int j = w.j0 - 1 + hj, k = w.k0 - 1 + hk;
        const bool in = idx < total && j < G.NJ && k < G.NK;
        slot[u] = in ? -1 : -2;
        if (in) {
          const long long n = (long long)(w.i0 - 1 + pl) * G.sI + (long long)j * G.sJ + k;
          if (G.nFilter > 0) slot[u] = __ldg(G.fidx + n);
          v[u][0] = __ldcg(q0 + n);
          v[u][1] = __ldcg(q1 + n);
          v[u][2] = __ldcg(q2 + n);
          v[u][3] = __ldcg(q3 + n);
          v[u][4] = __ldcg(q4 + n);
        } else {
#pragma unroll
          for (int f = 0; f < 5; ++f) v[u][f] = 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = b0 + u * NT;
        if (slot[u] == -2) continue;
        const int pl = idx / HP, r = idx - pl * HP;
        double rho = v[u][0], rE = v[u][4];
        if (slot[u] >= 0) {  // filtered nodes take their primitive values from before the near-body filter
          rho = __ldcg(G.fpre + 2 * slot[u]);
          rE = __ldcg(G.fpre + 2 * slot[u] + 1);
        }
        const Prim q = prims_of_nr(TC, rho, v[u][1], v[u][2], v[u][3], rE);
        double* d = sm + pl * PS + r;
        d[0 * FS] = q.u;
        d[1 * FS] = q.v;
        d[2 * FS] = q.w;
        d[3 * FS] = q.p;
        d[4 * FS] = q.T;
        d[5 * FS] = q.mu;
        d[6 * FS] = v[u][1];
        d[7 * FS] = v[u][2];
        d[8 * FS] = v[u][3];
        d[9 * FS] = v[u][4];
      }
    }
  }
  __syncthreads();
  const int ct = tid & (NCOL - 1), grp = tid / NCOL;
  const int tx = ct % TK, ty = ct / TK;
  const int cidx = (ty + 1) * HK + (tx + 1);
  const int j = w.j0 + ty, k = w.k0 + tx;
  const int per = (L + NG - 1) / NG, a0 = grp * per, a1 = min(L, a0 + per);
  if (a0 < a1 && j <= G.NJ - 2 && k <= G.NK - 2) {
    constexpr int oN = HK, oU = 1;
    XOwn ownPrev{};
    XNode gm1{}, gm2{};
    double fprev[5] = {0, 0, 0, 0, 0};
    // x-direction quantities of staged plane q (see nsf_stage_ws.cu)
    auto x_part = [&](int q, bool face, XOwn& own, XNode& g, double (&f)[5]) {
      const double* ps = sm + q * PS + cidx;
      own = XOwn{ps[5 * FS], ps[0 * FS], ps[1 * FS], ps[2 * FS], ps[4 * FS]};
      g = x_node(C, ps[6 * FS], ps[7 * FS], ps[8 * FS], ps[9 * FS], own.u, own.v, own.w, ps[3 * FS], own.mu,
                 ps[1 * FS + oN] - ps[1 * FS - oN], ps[0 * FS + oN] - ps[0 * FS - oN],
                 ps[2 * FS + oU] - ps[2 * FS - oU], ps[0 * FS + oU] - ps[0 * FS - oU]);
#pragma unroll
      for (int e = 0; e < 5; ++e) f[e] = 0.0;
      if (face) x_face(C, ownPrev, own, f);
    };
    {
      XOwn own;
      double f[5];
      x_part(a0, false, own, gm2, f);
      ownPrev = own;
      x_part(a0 + 1, true, own, gm1, fprev);
      ownPrev = own;
    }
    long long n = (long long)(w.i0 + a0) * G.sI + (long long)j * G.sJ + k;
    const double inc = (s == 2) ? c.dtUsed : c.dtUsed / 2, dtFactor = c.dtUsed / 6;
#pragma unroll 1
    for (int a = a0; a < a1; ++a, n += G.sI) {
      const uint8_t tc = G.type[n];
      double u0[5], ac[5];
#pragma unroll
      for (int f = 0; f < 5; ++f) u0[f] = __ldcg(c.U0[f] + n);
      if (LAST || s > 0) {
#pragma unroll
        for (int f = 0; f < 5; ++f) ac[f] = __ldcg(G.acc[f] + n);
      }
      XNode g;
      XOwn own;
      double f[5], kk[5];
      x_part(a + 2, true, own, g, f);
      const double* pP = sm + (a + 1) * PS;
      using X = CrossMem<HK, FS>;
      yz_part<HK, FS>(C, pP + 5 * FS, pP, X{pP - PS, cidx}, X{pP, cidx}, X{pP + PS, cidx}, cidx, ownPrev, kk);
#pragma unroll
      for (int e = 0; e < 5; ++e) kk[e] += (g.g[e] - gm2.g[e]) + (f[e] - fprev[e]);
      const bool valid = (tc & TYPE_MASK) == FLUID_INTERIOR;
      double res[5];
      if (!LAST) {
#pragma unroll
        for (int e = 0; e < 5; ++e) {
          if (valid) G.acc[e][n] = s == 0 ? kk[e] : ac[e] + 2 * kk[e];
          res[e] = u0[e] + inc * kk[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < 5; ++e) res[e] = u0[e] + dtFactor * (ac[e] + kk[e]);
        const bool filtered = (tc & FILTER_BIT) != 0;  // rho, rho_E change again in the near-body filter
#pragma unroll
        for (int e = 0; e < 5; ++e) {
          const double d = u0[e] - res[e];
          nsum[e] += (valid && !(filtered && (e == 0 || e == 4))) ? d * d : 0.0;
        }
        bad |= valid && !(isfinite(res[0]) && isfinite(res[1]) && isfinite(res[2]) && isfinite(res[3]) &&
                          isfinite(res[4]));
        if (valid && !filtered) dt_terms(C, res, dta);
      }
      if (valid) {
#pragma unroll
        for (int e = 0; e < 5; ++e) c.O[s][e][n] = res[e];
        if (tc & (ZCOPY_UP_BIT | ZCOPY_DOWN_BIT)) {  // periodic z and y copies, as in nsf_stage_ws.cu
          const long long m = (tc & ZCOPY_UP_BIT) ? n + (G.NK - 2) : n - (G.NK - 2);
#pragma unroll
          for (int e = 0; e < 5; ++e) c.O[s][e][m] = res[e];
        }
        if (tc & YCOPY_BIT) {
          const long long m = j == 1 ? n + (long long)(G.NJ - 2) * G.sJ : n - (long long)(G.NJ - 2) * G.sJ;
#pragma unroll
          for (int e = 0; e < 5; ++e) c.O[s][e][m] = res[e];
        }
      }
      gm2 = gm1;
      gm1 = g;
#pragma unroll
      for (int e = 0; e < 5; ++e) fprev[e] = f[e];
      ownPrev = own;
    }
  }
  __syncthreads();  // the next tile overwrites the staged planes
}

// Grid barrier over all blocks on an arrival counter that only grows: a launch's barrier number q is passed when
// the counter has grown by q times the block count since the launch (target, thread 0's). The arrival is a
// reduction without a return value (release), the poll an acquire load; the block barriers on both sides
// carry that order to the block's other threads. Bounded: the poll limit and the switch that withholds a
// block's arrivals come from the control block (nsf_debug_wait_limit); after a barrier that gave up, the block
// waits for no other (the run is reported invalid, nothing hangs).
struct StepBarrier {
  unsigned long long* S;
  unsigned long long target;  // thread 0's
  int* timeout;               // StepCtl::timeout
  bool dead;
  __device__ __forceinline__ void wait(const StepCtl& cs) {
    __syncthreads();
    if (threadIdx.x == 0) {
      if (!(cs.withhold && blockIdx.x == 0))
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(S) : "memory");
      target += gridDim.x;
      const long long limit = dead ? 0 : (cs.waitLimit > 0 ? cs.waitLimit : kBarrierPolls);
      long long it = 0;
      while (ld_acquire(S) < target) {
        if (++it > limit) {
          atomicExch(timeout, 1);
          dead = true;
          break;
        }
      }
    }
    __syncthreads();
  }
};

// words doubles (a multiple of 2, 16-byte aligned) from src to dst by all blocks; src is read through L2. A call: inlined
// at each of its uses it would cost the stage phases their registers.
__device__ __noinline__ void tape_copy(const double* src, double* dst, long long words, int gtid, int nthr) {
  const double2* a = reinterpret_cast<const double2*>(src);
  double2* b = reinterpret_cast<double2*>(dst);
  const long long n = words / 2;
  constexpr int U = 4;
  for (long long q = gtid; q < n; q += (long long)U * nthr) {
    double2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q + (long long)u * nthr < n) v[u] = __ldcg(a + q + (long long)u * nthr);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q + (long long)u * nthr < n) __stcs(b + q + (long long)u * nthr, v[u]);
  }
}

// TAPE: the steps also record their sets (StepParams::tape): a stage's input right before the stage, which no block
// writes until the stage after it, and the step's result after the end-of-step barrier.
template <class T, bool TAPE>
__global__ void __launch_bounds__(NT, 1) k_step(const __grid_constant__ Grid G0, Grid* gp,
                                                const __grid_constant__ StepParams P, int nsteps) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[NQ][NT / 32];
  __shared__ double tot[NQ];
  __shared__ __align__(16) unsigned char gsm[sizeof(Grid)];
  __shared__ __align__(16) unsigned char csm[sizeof(StepCtl)];
  __shared__ __align__(16) unsigned char tsm[kTileStash * sizeof(StageItem)];
  __shared__ int levelCount[kStash];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  StepCtl* const gc = G0.ctl;
  {
    const unsigned long long* a = reinterpret_cast<const unsigned long long*>(gp);
    const unsigned long long* b = reinterpret_cast<const unsigned long long*>(gc);
    for (int q = tid; q < int(sizeof(Grid) / 8); q += NT) reinterpret_cast<unsigned long long*>(gsm)[q] = a[q];
    for (int q = tid; q < int(sizeof(StepCtl) / 8); q += NT) reinterpret_cast<unsigned long long*>(csm)[q] = b[q];
  }
  __syncthreads();
  const Grid& G = *reinterpret_cast<const Grid*>(gsm);
  StepCtl& cs = *reinterpret_cast<StepCtl*>(csm);
  const int itBegin = P.start[blockIdx.x], nTiles = P.start[blockIdx.x + 1] - itBegin;
  StageItem* const tiles = reinterpret_cast<StageItem*>(tsm);
  if (tid < kTileStash && tid < nTiles) tiles[tid] = P.items[itBegin + tid];
  auto tile = [&](int q) { return q < kTileStash ? tiles[q] : P.items[itBegin + q]; };
  // warps are numbered across the blocks, so that a short list of boundary items spreads over all SMs
  const int gtid = (warp * int(gridDim.x) + int(blockIdx.x)) * 32 + lane, nthr = int(gridDim.x) * NT;
  // every earlier launch left the counter at a multiple of the block count, and the first barrier cannot pass
  // before this block has arrived, so the value at the launch is the counter rounded down to a multiple. (A launch
  // whose barrier gave up may not have; its flag stays until the control block is reset, and the counter with it.)
  StepBarrier bar{P.sync, tid == 0 ? ld_acquire(P.sync) / gridDim.x * gridDim.x : 0ull, &gc->timeout, false};
  auto barrier = [&] { bar.wait(cs); };
  // the first boundary item each thread has in the first kStash levels, resolved once for the whole launch
  BcItem* const stash = reinterpret_cast<BcItem*>(reinterpret_cast<unsigned char*>(sm) + P.stashOffset);
  const int nStash = min(P.bc.levels, kStash);
  for (int L = 0; L < nStash; ++L) {
    const int n = bc_level_items(G, P.bc, 0, L);
    if (tid == 0) levelCount[L] = n;
    stash[L * NT + tid] = gtid < n ? bc_level_item(G, P.bc, 0, L, gtid) : BcItem{BC_NONE, 0, 0, 0};
  }
  __syncthreads();
  auto boundary = [&](auto last, int s, DtAcc& dta, double (&nsum)[5], int& bad) {
    for (int L = 0; L < P.bc.levels; ++L) {
      barrier();
      const bool kept = L < kStash;
      const int total = kept ? levelCount[L] : bc_level_items(G, P.bc, 0, L);
      BcItem it{BC_NONE, 0, 0, 0};
      if (kept)
        it = stash[L * NT + tid];
      else if (gtid < total)
        it = bc_level_item(G, P.bc, 0, L, gtid);
      for (int v = gtid; v < total;) {
        bc_run_item<decltype(last)::value>(G, cs, s, it, dta, nsum, bad);
        if ((v += nthr) < total) it = bc_level_item(G, P.bc, 0, L, v);
      }
    }
  };
  for (int step = 0; step < nsteps; ++step) {
    if (warp == 0) prologue_warp(G, &cs, lane, blockIdx.x == 0);
    __syncthreads();
    if (!cs.active) break;  // the same decision in every block
    if (cs.filterNow) {
      for (long long n = gtid; n < G.N; n += nthr) density_filter_node(G, &cs, n);
      barrier();
    }
    double* const set = TAPE ? P.tape.stage + (long long)(cs.level % (unsigned)P.tape.nSets) * P.tape.setWords : nullptr;
    double* const setEnd = TAPE ? P.tape.result + (long long)(cs.level % (unsigned)P.tape.nSets) * P.tape.setWords : nullptr;
    auto record = [&](int s) {
      double* const base = set + s * P.tape.perStage;
      for (int f = 0; f < 5; ++f) tape_copy(cs.I[s][f], base + f * G.N, G.N, gtid, nthr);
      if (cs.R[s] != cs.I[s][0]) tape_copy(cs.R[s], base + 5 * G.N, G.N, gtid, nthr);
      if (G.nFilter > 0) tape_copy(G.fpre, base + 11 * G.N, 2ll * G.nFilter, gtid, nthr);
    };
    DtAcc dta;
    double nsum[5] = {0, 0, 0, 0, 0};
    int bad = 0;
#pragma unroll 1
    for (int s = 0; s < 3; ++s) {
      if (TAPE) record(s);
      for (int q = 0; q < nTiles; ++q) stage_tile<T, false>(G0, cs, s, tile(q), sm, dta, nsum, bad);
      boundary(std::false_type{}, s, dta, nsum, bad);
      barrier();
    }
    if (TAPE) record(3);
    for (int q = 0; q < nTiles; ++q) stage_tile<T, true>(G0, cs, 3, tile(q), sm, dta, nsum, bad);
    boundary(std::true_type{}, 3, dta, nsum, bad);
    // end of step: this block's partials, then every block combines all of them in the same order
    const double v[NQ] = {dta.sx, dta.sy, dta.sz, dta.nu, nsum[0], nsum[1], nsum[2], nsum[3], nsum[4]};
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double x = q < 4 ? warp_max(v[q]) : warp_sum(v[q]);
      if (lane == 0) red[q][warp] = x;
    }
    if (bad) atomicOr(&gc->nonFinite, 1);
    __syncthreads();
    if (warp < NQ) {
      double x = lane < NT / 32 ? red[warp][lane] : 0.0;
      x = warp < 4 ? warp_max(x) : warp_sum(x);
      if (lane == 0) P.part[warp * gridDim.x + blockIdx.x] = x;
    }
    barrier();
    if (warp < NQ) {
      double x = 0;
      for (int b = lane; b < int(gridDim.x); b += 32) {
        const double y = __ldcg(P.part + warp * gridDim.x + b);
        x = warp < 4 ? fmax(x, y) : x + y;
      }
      x = warp < 4 ? warp_max(x) : warp_sum(x);
      if (lane == 0) tot[warp] = x;
    }
    const unsigned long long level = cs.level;
    const double dtUsed = cs.dtUsed, tNew = cs.t + dtUsed;
    __syncthreads();
    if (blockIdx.x == 0 && tid >= 32 && tid < 39) history_entry(G, level, tNew, dtUsed, tot + 4, tid - 32);
    if (tid < 4) cs.mx[tid] = static_cast<unsigned long long>(__double_as_longlong(tot[tid]));
    if (tid == 0) finish_step(G, &cs, tot);
    if (TAPE)
      for (int f = 0; f < 5; ++f) tape_copy(cs.O[3][f], setEnd + f * G.N, G.N, gtid, nthr);
    __syncthreads();
  }
  if (blockIdx.x == 0) {  // the control block as the next call reads it; the flags other blocks set stay as they are
    constexpr int kNonFinite = int(offsetof(StepCtl, nonFinite) / 4), kTimeout = int(offsetof(StepCtl, timeout) / 4);
    for (int q = tid; q < int(sizeof(StepCtl) / 4); q += NT)
      if (q != kNonFinite && q != kTimeout) reinterpret_cast<int*>(gc)[q] = reinterpret_cast<const int*>(csm)[q];
  }
}

using Cube = BT<16, 8>;  // the general tile
using Thin = BT<4, 32>;  // grids of up to four interior nodes along k

template <class T>
StepShape shape_of() {
  return StepShape{T::TK, T::TJ, T::LMAX, T::HP};
}
const void* kernel_of(int shape, bool tape) {
  if (shape == STEP_TILE_THIN)
    return tape ? reinterpret_cast<const void*>(&k_step<Thin, true>) : reinterpret_cast<const void*>(&k_step<Thin, false>);
  return tape ? reinterpret_cast<const void*>(&k_step<Cube, true>) : reinterpret_cast<const void*>(&k_step<Cube, false>);
}

}  // namespace

StepShape step_shape(int shape) { return shape == STEP_TILE_THIN ? shape_of<Thin>() : shape_of<Cube>(); }

static size_t staged_bytes(int shape, int planes) {
  return (size_t(planes + 2) * 10 * size_t(step_shape(shape).haloNodes) * 8 + 15) / 16 * 16;
}
size_t step_smem_bytes(int shape, int planes, int levels) {
  return staged_bytes(shape, planes) + size_t(std::min(levels, kStash)) * NT * sizeof(BcItem);
}

// The tile shape, the planes per tile and the blocks that run them: the smallest estimated time of one stage. A
// block's tile costs a fixed part (load latency, barriers), one pass of the block over the tile's halo nodes
// per NT of them, and one pass over its planes per NG of them plus the start of the carried x quantities. The weights
// are relative; the choice they make was the fastest of 1 .. 12 planes on each grid measured (us per step at 2 .. 10
// planes by the plane): sphere 48^3 (6 chosen) 85 78 87 93 71 78 81 84 89, walls 75x53x61 (8) 154 146 144 132 138 143 131
// 139 148, Taylor-Green 64^3 (7) 132 121 120 108 115 102 106 112 122, 80^3 (10) 233 195 186 183 170 182 178 179 168;
// sphere 32^3 2 planes, cylinder 161x83x3 4.
StepChoice step_choose(int NI, int NJ, int NK, int nSM) {
  StepChoice best{};
  double bestCost = 1e300;
  for (int shape = 0; shape < 2; ++shape) {
    const StepShape t = step_shape(shape);
    if (shape == STEP_TILE_THIN && NK - 2 > t.tk) continue;
    const int tiles = ((NJ - 2 + t.tj - 1) / t.tj) * ((NK - 2 + t.tk - 1) / t.tk), planes = NI - 2;
    for (int len = 1; len <= std::min(planes, t.maxPlanes); ++len) {
      const int items = tiles * ((planes + len - 1) / len), rounds = (items + nSM - 1) / nSM;
      const int loads = ((len + 2) * t.haloNodes + NT - 1) / NT, passes = (len + NG - 1) / NG;
      const double cost = rounds * (2.0 + 0.35 * loads + 2.0 * passes);
      if (cost < bestCost - 1e-9) {
        bestCost = cost;
        best = StepChoice{shape, len, items};
      }
    }
  }
  return best;
}

// The attribute belongs to the function, not to a handle: it is set to all a block can have, whatever the handle's
// plan takes, so that a handle created later does not take it below what an earlier one launches with.
int step_configure(int shape) {
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  for (bool tape : {false, true}) {
    cudaFuncAttributes a{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, kernel_of(shape, tape));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel_of(shape, tape), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               most - int(a.sharedSizeBytes));
  }
  return int(e);
}

int step_capacity(int shape, size_t smem, int nSM) {
  int nb = 0, nb2 = 0;  // both instantiations run the same plan
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel_of(shape, false), NT, smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb2, kernel_of(shape, true), NT, smem) != cudaSuccess) return 0;
  return std::min(nb, nb2) * nSM;
}

int launch_steps(const Grid& hg, Grid* dg, const LaunchPlan& L, const StepPlan& S, int nsteps, void* stream,
                 const StepTape& tape) {
  StepParams P{};
  P.bc.edges = L.bcEdges;
  P.bc.edgeStart = L.bcEdgeStart;
  P.bc.items = L.bcItems;
  P.bc.itemStart = L.bcItemStart;
  P.bc.levels = L.bcLevels;
  P.bc.members = 1;
  P.items = S.items;
  P.start = S.start;
  P.part = S.part;
  P.sync = S.sync;
  P.stashOffset = int(staged_bytes(S.shape, S.planes));
  P.tape = tape;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(S.blocks));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = S.smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  auto go = [&](auto kernel) { return int(cudaLaunchKernelEx(&cfg, kernel, hg, dg, P, nsteps)); };
  if (S.shape == STEP_TILE_THIN) return tape.stage ? go(k_step<Thin, true>) : go(k_step<Thin, false>);
  return tape.stage ? go(k_step<Cube, true>) : go(k_step<Cube, false>);
}

}  // namespace nsf
