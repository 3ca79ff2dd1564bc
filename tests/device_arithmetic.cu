// device_arithmetic.cu -- the device functions that stand in for plain operations, one per element, for
// test_gpu_arithmetic.py. Compiled as the FP64 kernels are.
#include "spx_physics.cuh"

namespace {

enum Op { kQuot, kOverC, kOver2C, kUniform };

__global__ void each(int op, int64_t n, const double* x, const double* y, const uint32_t* u, double* out)
{
   const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= n) return;
   switch (op) {
   case kQuot: out[i] = spx::quot(x[i], y[i]); break;
   case kOverC: out[i] = spx::over_c(x[i]); break;
   case kOver2C: out[i] = spx::over_2c(x[i]); break;
   case kUniform: out[i] = spx::u01d(u[i]); break;
   }
}

// deviates of the 2^32 whose cospi differs from the cosine of the pair
__global__ void cosines(unsigned long long* differ)
{
   unsigned long long mine = 0;
   for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < (1ull << 32); k += (uint64_t)gridDim.x * blockDim.x) {
      const double u = spx::u01d((uint32_t)k);
      double s, c;
      spx::sincos_2pi(u, &s, &c);
      mine += __double_as_longlong(cospi(2.0 * u)) != __double_as_longlong(c);
   }
   if (mine) atomicAdd(differ, mine);
}

}  // namespace

// host arrays of n elements (those the operation reads; the others null); returns a cudaError_t
extern "C" int arithmetic(int op, int64_t n, const double* x, const double* y, const uint32_t* u, double* out)
{
   double *dx = nullptr, *dy = nullptr, *dout = nullptr;
   uint32_t* du = nullptr;
   cudaError_t e = cudaMalloc(&dout, sizeof(double) * n);
   auto up = [&](auto*& d, const auto* h) {
      if (!h || e != cudaSuccess) return;
      e = cudaMalloc(&d, sizeof(*h) * n);
      if (e == cudaSuccess) e = cudaMemcpy(d, h, sizeof(*h) * n, cudaMemcpyHostToDevice);
   };
   up(dx, x);
   up(dy, y);
   up(du, u);
   if (e == cudaSuccess) {
      each<<<(unsigned)((n + 255) / 256), 256>>>(op, n, dx, dy, du, dout);
      e = cudaGetLastError();
   }
   if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(double) * n, cudaMemcpyDeviceToHost);
   cudaFree(dx);
   cudaFree(dy);
   cudaFree(du);
   cudaFree(dout);
   return e;
}

extern "C" int cosines_that_differ(unsigned long long* n)
{
   unsigned long long* d = nullptr;
   cudaError_t e = cudaMalloc(&d, sizeof *d);
   if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof *d);
   if (e == cudaSuccess) {
      cosines<<<152 * 8, 256>>>(d);
      e = cudaGetLastError();
   }
   if (e == cudaSuccess) e = cudaMemcpy(n, d, sizeof *d, cudaMemcpyDeviceToHost);
   cudaFree(d);
   return e;
}
