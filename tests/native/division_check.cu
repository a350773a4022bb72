// Test kernels for the exact integrator's shared-reciprocal quotients and the
// recurrences built on them (simcore_b200/csrc/sc_step.cuh), compiled as that
// unit is (--fmad=false).
#include <cuda_runtime.h>

#include "sc_common.cuh"
#include "sc_pair.cuh"
#include "sc_step.cuh"

using namespace sc;

namespace {

__device__ unsigned long long mix(unsigned long long z) {  // splitmix64 (Vigna)
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}

// Bit 0: recip_rn differs from 1 / b though ok; 1: div_rn from x / b though ok;
// 2: div_by from x / b; 3: ok after recip_rn; 4: ok after div_rn.
__device__ int compare(double x, double b) {
  bool ok = true;
  const double y = recip_rn(b, ok);
  const bool okr = ok;
  const double q = div_rn(x, b, y, ok);
  int r = (okr ? 8 : 0) | (ok ? 16 : 0);
  if (okr && !same(y, 1.0 / b)) r |= 1;
  if (ok && !same(q, x / b)) r |= 2;
  if (!same(div_by(x, b, 1.0 / b), x / b)) r |= 4;
  return r;
}

__global__ void k_given(int n, const double *x, const double *b, int *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = compare(x[i], b[i]);
}

// Operands by their index: random significands, exponents within 2^+-range, every
// other one with its quotient near a midpoint of two doubles.
__global__ void k_random(unsigned long long seed, long long n, int range,
                         unsigned long long *wrong) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned long long u = mix(seed + 2 * i), v = mix(seed + 2 * i + 1), w = mix(u ^ ~v);
    auto make = [&](unsigned long long bits, unsigned long long e) {
      const unsigned long long ex = 1023 - range + e % (2 * range + 1);
      return __longlong_as_double((long long)((bits & 0x800fffffffffffffull) | ex << 52));
    };
    const double b = make(u, w & 0xffff);
    double x = make(v, w >> 16 & 0xffff);
    if (i & 1) {  // x = RN((q + half an ulp of q) b)
      const double q = make(v, 0x7fff & range);
      const double ulp = __longlong_as_double(__double_as_longlong(q) + 1) - q;
      x = fma(q, b, 0.5 * ulp * b);
    }
    if ((compare(x, b) & 7) != 0) ++bad;
  }
  if (bad) atomicAdd(wrong, bad);
}

// One lane's recurrences (io: cz, off, diag, den, inv, up, minors, d, x; 64 each).
__global__ void k_solve(double *io, int trail, int n) {
  __shared__ double s[9 * 64];
  for (int i = threadIdx.x; i < 9 * 64; i += blockDim.x) s[i] = io[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    double *cz = s, *off = s + 64, *diag = s + 128, *den = s + 192, *inv = s + 256, *up = s + 320;
    factor_and_minors(trail != 0, true, cz, off, diag, den, inv, up, s + 384, n);
    if (trail) tridiag_rhs<false>(off, den, inv, up, s + 448, s + 512, n - 1);
    else tridiag_rhs<true>(cz, den, inv, up, s + 448, s + 512, n - 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 9 * 64; i += blockDim.x) io[i] = s[i];
}

}  // namespace

extern "C" int check_given(int n, const double *x, const double *b, int *out) {
  double *dx = nullptr, *db = nullptr;
  int *dout = nullptr;
  cudaMalloc(&dx, sizeof(double) * n);
  cudaMalloc(&db, sizeof(double) * n);
  cudaMalloc(&dout, sizeof(int) * n);
  cudaMemcpy(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k_given<<<(n + 127) / 128, 128>>>(n, dx, db, dout);
  cudaMemcpy(out, dout, sizeof(int) * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(db);
  cudaFree(dout);
  return (int)cudaGetLastError();
}

extern "C" int check_random(unsigned long long seed, long long n, int range,
                            unsigned long long *wrong) {
  unsigned long long *d = nullptr;
  cudaMalloc(&d, sizeof(*d));
  cudaMemset(d, 0, sizeof(*d));
  k_random<<<148 * 8, 256>>>(seed, n, range, d);
  cudaMemcpy(wrong, d, sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}

extern "C" int check_solve(double *io, int trail, int n) {
  double *d = nullptr;
  if (n < 3 || n > 63) return -1;
  cudaMalloc(&d, sizeof(double) * 9 * 64);
  cudaMemcpy(d, io, sizeof(double) * 9 * 64, cudaMemcpyHostToDevice);
  k_solve<<<1, 32>>>(d, trail, n);
  cudaMemcpy(io, d, sizeof(double) * 9 * 64, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
