// The dt-limit terms of a boundary node (dt_terms_known, nsf_physics.cuh) and their evaluation by divisions and square
// roots (DtAcc::add, as the host's initial dt), on the device. Arguments: input file (doubles gamma, re, sc1, vmod, then
// rho, p, T of every node), output file (per node: sound speed and viscous term, by the first, then by the second).
#include <cstdio>
#include <vector>

#include "nsf_device.cuh"
#include "nsf_physics.cuh"

__global__ void terms(nsf::Consts C, const double* in, double* out, int n) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const double rho = in[3 * q], p = in[3 * q + 1], T = in[3 * q + 2];
    nsf::DtAcc a{}, b{};
    nsf::dt_terms_known(C, rho, 0.0, 0.0, 0.0, p, T, a);
    const double x = 1.0 + T;
    b.add(C, rho, 0.0, 0.0, 0.0, p, x * sqrt(x) * C.sc1 / (C.re * (T + C.sc1)));
    out[4 * q] = a.sx;
    out[4 * q + 1] = a.nu;
    out[4 * q + 2] = b.sx;
    out[4 * q + 3] = b.nu;
  }
}

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  std::FILE* f = std::fopen(argv[1], "rb");
  if (!f) return 3;
  std::fseek(f, 0, SEEK_END);
  const long count = std::ftell(f) / 8;
  std::rewind(f);
  std::vector<double> in(count);
  if (count < 7 || std::fread(in.data(), 8, size_t(count), f) != size_t(count)) return 4;
  std::fclose(f);
  const int n = int((count - 4) / 3);
  nsf::Consts C{};
  C.gamma = in[0];
  C.re = C.muRe = in[1];
  C.sc1 = in[2];
  C.muA = C.re / C.sc1;
  C.vmod = in[3];
  std::vector<double> out(4 * size_t(n));
  double *dIn = nullptr, *dOut = nullptr;
  if (cudaMalloc(&dIn, 24 * size_t(n)) != cudaSuccess || cudaMalloc(&dOut, 32 * size_t(n)) != cudaSuccess) return 5;
  if (cudaMemcpy(dIn, in.data() + 4, 24 * size_t(n), cudaMemcpyHostToDevice) != cudaSuccess) return 6;
  terms<<<148, 256>>>(C, dIn, dOut, n);
  if (cudaMemcpy(out.data(), dOut, 32 * size_t(n), cudaMemcpyDeviceToHost) != cudaSuccess) return 7;
  f = std::fopen(argv[2], "wb");
  if (!f || std::fwrite(out.data(), 8, out.size(), f) != out.size()) return 8;
  std::fclose(f);
  return 0;
}
