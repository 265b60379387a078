// nsf_step_metrics_noalloc: the end-of-step metrics (the five change norms of
// Solver::storeNormsOfChange, Solver.cpp:510-530 / Mesh.cpp:171-178, and the next dt of
// Solver::updateTimeStepSize, Solver.cpp:80-126) for conserved fields that the CALLER holds in device
// memory, computed without allocating anything.
//
// Who needs it: host frameworks that own every byte of device memory and hand this library only
// pointers (a coupling framework or plugin host that forbids third-party cudaMalloc), code running
// while a CUDA stream is being captured into a graph (a cudaMalloc there would not be part of the
// graph and breaks the replay contract), and real-time loops that must not allocate after start-up.
// The solver handle (nsf_create / nsf_march) allocates its scratch; this entry point does not.
//
// Scratch: the per-block partial results of the two-pass reduction live in one file-scope device array
// of kScratchBytes (8 MiB) that every GPU loading this library holds until the process
// exits. It bounds the grid: up to 29,826,048 nodes (9 doubles per 256 nodes, the densest partials a first pass may
// write); larger grids are rejected with NSF_ERR_ARG. Every partial the final pass reads is written earlier in
// the same call, so nothing has to be cleared between calls. All calls share the array: two calls whose
// kernels overlap on the GPU (different streams, or different host threads) race on it and must be
// serialised by the caller.
//
// What bounds it: HBM, 80 bytes a node (two states of five fields, read once). The first pass runs a fixed number of
// blocks, whose threads stride over the nodes with their sums and maxima in registers, so that the nine block
// reductions come once per block instead of once per 256 nodes and the final pass reads a few thousand partials, not
// one per 256 nodes. Measured at 192^3 (566 MB): 231 us (170 + 69 us of kernels) before, 105 us now (5.4 TB/s). Quotients
// are corrected by their residuals and a block's warps are added in pairs, so that dt and norms are no further from an
// evaluation in 64 bits than by divisions and one partial per 256 nodes (rms over 40 states: 192^3 6.6e-17, 6.8e-17
// before; 8.8e-17 with plain products and the warps one after another, which took 2 us less).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

#include "nsf_internal.h"
#include "nsf_physics.cuh"

namespace {

constexpr size_t kScratchBytes = size_t(8) << 20;
constexpr int kThreads = 256;  // threads per block, and the nodes per partial that bound the grid
constexpr int kQ = 9;          // five squared-difference sums, four maxima
constexpr size_t kMaxPartials = kScratchBytes / (kQ * sizeof(double));
constexpr int kBlocksPerSM = 4;

__device__ __align__(256) double g_metrics_scratch[kScratchBytes / sizeof(double)];

// Device address of g_metrics_scratch and the SM count per device, resolved once per device (host code may not use
// the symbol's host-side name as a device address).
double* g_scratch_addr[64] = {};
int g_sm_count[64] = {};
std::mutex g_scratch_mutex;

struct MetricParams {
  int NI, NJ, NK;
  unsigned N, stride;  // nodes; nodes between two of a thread's (all threads of the grid)
  int sI, sJ, sK;      // the stride as (i, j, k) steps
  double gamma, gm1, sc1, re, vmod;
  double dxdydz, dx, dy, dz, invD2, convLim, viscLim;
};

__device__ __forceinline__ double combine(int q, double a, double b) { return q < 5 ? a + b : fmax(a, b); }

// Block-wide reduction of the nine quantities; the result is valid in thread q < kQ.
__device__ __forceinline__ double block_reduce(const double (&v)[kQ], double (&red)[kQ][kThreads / 32]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    double a = v[q];
    for (int o = 16; o > 0; o >>= 1) a = combine(q, a, __shfl_xor_sync(0xffffffffu, a, o));
    if (lane == 0) red[q][wid] = a;
  }
  __syncthreads();
  static_assert(kThreads == 256, "eight warps, in pairs");
  double a = 0;
  if (threadIdx.x < kQ) {
    const int q = threadIdx.x;
    const double* w = red[q];
    a = combine(q, combine(q, combine(q, w[0], w[1]), combine(q, w[2], w[3])),
                combine(q, combine(q, w[4], w[5]), combine(q, w[6], w[7])));
  }
  return a;
}

// Every node once, grid-stride; one partial per block, quantity-major.
__global__ void __launch_bounds__(kThreads, kBlocksPerSM)
    k_metrics_partial(const __grid_constant__ MetricParams p, const double* __restrict__ old5,
                      const double* __restrict__ new5, const uint8_t* __restrict__ types,
                      double* __restrict__ partial) {
  __shared__ double red[kQ][kThreads / 32];
  double v[kQ] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  unsigned n = blockIdx.x * kThreads + threadIdx.x;
  const unsigned plane = unsigned(p.NJ) * unsigned(p.NK);
  int i = int(n / plane), j = int(n % plane / p.NK), k = int(n % p.NK);
  for (; n < p.N; n += p.stride) {
    const bool interior = types ? (types[n] & nsf::TYPE_MASK) == nsf::FLUID_INTERIOR
                                : (i > 0 && j > 0 && k > 0 && i < p.NI - 1 && j < p.NJ - 1 && k < p.NK - 1);
    double u[5], o[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) u[f] = __ldcs(new5 + size_t(f) * p.N + n);
#pragma unroll
    for (int f = 0; f < 5; ++f) o[f] = interior ? __ldcs(old5 + size_t(f) * p.N + n) : u[f];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const double d = o[f] - u[f];
      v[f] += interior ? d * d : 0.0;
    }
    const double a1 = u[0] + 1.0, r1 = nsf::recip_nr(a1);
    const double uu = u[1] * r1, vv = u[2] * r1, ww = u[3] * r1;
    const double pp = p.gm1 * (u[4] - (u[0] + 1.0) * 0.5 * (uu * uu + vv * vv + ww * ww));
    const double T = (p.gamma * pp - u[0]) * r1;
    const double x = 1.0 + T;
    const double den = p.re * (T + p.sc1);
    const double mu = nsf::quot_nr(x * nsf::sqrt_nr(x) * p.sc1, den, nsf::recip_nr(den));
    const double c = nsf::sqrt_nr(nsf::quot_nr(1.0 + p.gamma * pp, a1, r1));
    v[5] = fmax(v[5], c + fabs(uu));
    v[6] = fmax(v[6], c + fabs(vv));
    v[7] = fmax(v[7], c + fabs(ww));
    v[8] = fmax(v[8], nsf::quot_nr(mu, a1, r1) * p.vmod);
    k += p.sK;
    j += p.sJ;
    i += p.sI;
    if (k >= p.NK) {
      k -= p.NK;
      ++j;
    }
    if (j >= p.NJ) {
      j -= p.NJ;
      ++i;
    }
  }
  const double mine = block_reduce(v, red);
  if (threadIdx.x < kQ) partial[threadIdx.x * gridDim.x + blockIdx.x] = mine;
}

// Combines the blocks' partials in block order (deterministic): out[0..4] = change norms, out[5] = next dt (min of
// the convective and viscous limits; the end_time clip needs t, which the caller holds, so the caller applies it).
// One block.
__global__ void __launch_bounds__(kThreads)
    k_metrics_final(const __grid_constant__ MetricParams p, const double* __restrict__ partial, unsigned blocks,
                    double* __restrict__ out) {
  __shared__ double red[kQ][kThreads / 32];
  __shared__ double tot[kQ];
  double v[kQ];
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    v[q] = 0;
    for (unsigned b = threadIdx.x; b < blocks; b += kThreads) v[q] = combine(q, v[q], partial[q * blocks + b]);
  }
  const double all = block_reduce(v, red);
  if (threadIdx.x < kQ) tot[threadIdx.x] = all;
  __syncthreads();
  if (threadIdx.x < 5) out[threadIdx.x] = sqrt(p.dxdydz * tot[threadIdx.x]);
  if (threadIdx.x == 5) {
    const double conv = p.convLim / (tot[5] / p.dx + tot[6] / p.dy + tot[7] / p.dz);
    const double visc = p.viscLim / (tot[8] * p.invD2);
    out[5] = (visc < conv) ? visc : conv;
  }
}

}  // namespace

extern "C" nsf_status nsf_step_metrics_noalloc(const nsf_config* cfg, const double* d_old, const double* d_new,
                                               const uint8_t* d_types, double* d_out, void* stream) {
  if (!cfg || !d_old || !d_new || !d_out) return NSF_ERR_ARG;
  const long long NI = (long long)cfg->NI, NJ = (long long)cfg->NJ, NK = (long long)cfg->NK;
  if (NI < 3 || NJ < 3 || NK < 3) return NSF_ERR_ARG;
  const long long N = NI * NJ * NK;
  if ((unsigned long long)((N + kThreads - 1) / kThreads) > kMaxPartials) {
    std::fprintf(stderr,
                 "nsf_step_metrics_noalloc: %lld nodes exceed the fixed 8 MiB scratch (at most %llu nodes)\n", N,
                 (unsigned long long)(kMaxPartials * kThreads));
    return NSF_ERR_ARG;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NSF_ERR_CUDA;
  double* scratch = nullptr;
  int sms = 0;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_metrics_scratch) != cudaSuccess || !p) return NSF_ERR_CUDA;
      if (cudaDeviceGetAttribute(&g_sm_count[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return NSF_ERR_CUDA;
      g_scratch_addr[dev] = static_cast<double*>(p);
    }
    scratch = g_scratch_addr[dev];
    sms = g_sm_count[dev];
  }
  // Grid spacing by boundary type (Mesh.cpp:44-49), without building a mesh.
  nsf_config c = *cfg;
  if (c.shipped_case) {
    c.bc[0][0] = NSF_BC_INLET;
    c.bc[1][0] = NSF_BC_SYMMETRY;
    c.bc[2][0] = NSF_BC_PERIODIC;
  }
  const long long n3[3] = {NI, NJ, NK};
  const double L[3] = {c.lx, c.ly, c.lz};
  double d[3];
  for (int a = 0; a < 3; ++a) {
    const int t = c.bc[a][0];
    d[a] = L[a] / double(t == NSF_BC_PERIODIC ? n3[a] - 2 : t == NSF_BC_SYMMETRY ? n3[a] - 3 : n3[a] - 1);
  }
  const unsigned blocks = unsigned(std::min<long long>((N + kThreads - 1) / kThreads, (long long)sms * kBlocksPerSM));
  MetricParams p{};
  p.NI = int(NI);
  p.NJ = int(NJ);
  p.NK = int(NK);
  p.N = unsigned(N);
  p.stride = blocks * kThreads;
  p.sI = int(p.stride / (NJ * NK));
  p.sJ = int(p.stride % (NJ * NK) / NK);
  p.sK = int(p.stride % NK);
  p.gamma = c.gamma;
  p.gm1 = c.gamma - 1;
  p.sc1 = 1 + c.sutherlands_c2 / c.t0;
  p.re = c.re;
  p.vmod = std::fmax(4. / 3, c.gamma / c.pr);
  p.dxdydz = d[0] * d[1] * d[2];
  p.dx = d[0];
  p.dy = d[1];
  p.dz = d[2];
  p.invD2 = 1 / (d[0] * d[0]) + 1 / (d[1] * d[1]) + 1 / (d[2] * d[2]);
  p.convLim = std::fabs(c.conv_stability_limit);
  p.viscLim = std::fabs(c.visc_stability_limit);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  k_metrics_partial<<<blocks, kThreads, 0, st>>>(p, d_old, d_new, d_types, scratch);
  k_metrics_final<<<1, kThreads, 0, st>>>(p, scratch, blocks, d_out);
  return cudaGetLastError() == cudaSuccess ? NSF_OK : NSF_ERR_CUDA;
}
