// Viscosity of the staged primitives (mu_nr, nsf_physics.cuh) and the quotient form x sqrt(x) sc1 / (re (T + sc1)) with
// the kernels' refined reciprocal and square root, on the device. Arguments: input file (doubles re, sc1, then T ...),
// output file (mu_nr of every T, then the quotient form).
#include <cstdio>
#include <vector>

#include "nsf_device.cuh"
#include "nsf_physics.cuh"

struct Coef {
  double muRe, muA;
};

__global__ void viscosity(Coef c, double re, double sc1, const double* T, double* out, int n) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const double t = T[q], x = 1.0 + t;
    out[q] = nsf::mu_nr(c, x, t);
    out[n + q] = x * nsf::sqrt_nr(x) * sc1 * nsf::recip_nr(re * (t + sc1));
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
  if (count < 3 || std::fread(in.data(), 8, size_t(count), f) != size_t(count)) return 4;
  std::fclose(f);
  const int n = int(count - 2);
  const double re = in[0], sc1 = in[1];
  std::vector<double> out(2 * size_t(n));
  double *dT = nullptr, *dOut = nullptr;
  if (cudaMalloc(&dT, size_t(n) * 8) != cudaSuccess || cudaMalloc(&dOut, out.size() * 8) != cudaSuccess) return 5;
  if (cudaMemcpy(dT, in.data() + 2, size_t(n) * 8, cudaMemcpyHostToDevice) != cudaSuccess) return 6;
  viscosity<<<148, 256>>>(Coef{re, re / sc1}, re, sc1, dT, dOut, n);
  if (cudaMemcpy(out.data(), dOut, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 7;
  f = std::fopen(argv[2], "wb");
  if (!f || std::fwrite(out.data(), 8, out.size(), f) != out.size()) return 8;
  std::fclose(f);
  return 0;
}
