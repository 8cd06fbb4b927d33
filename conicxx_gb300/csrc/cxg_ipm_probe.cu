// Diagnostic entry of the dense root (cxg_dense_ldlt): the root LDL' and triangular solves of
// the batched kernels (cxg_ipm.cuh) on one given matrix, on one CTA.
#include "cxg_ipm.cuh"

namespace cxg {

template <typename T>
__global__ void __launch_bounds__(256) denseProbeKernel(int nr, int nx, const double* K, const double* b,
                                                         DevSettings st, double* Lout, double* Dout, double* xout,
                                                         long long* cyc, int* flags) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Ctx c;
  __shared__ double scArea[160];
  T* M = reinterpret_cast<T*>(smem);
  const int Tn = rootTiles(nr);
  const int64_t rs = rootSize(nr);
  T* y = M + rs;
  if (threadIdx.x == 0) {
    c.nr = nr;
    c.n = nx;
    c.vb = blockDim.x;
    c.red = scArea;
    c.sc = scArea + 128;
  }
  for (int64_t t = threadIdx.x; t < rs; t += blockDim.x) M[t] = (T)0;
  __syncthreads();
  for (int i = nr + (int)threadIdx.x; i < Tn * kTile; i += blockDim.x) M[rootIdx(nr, i, i)] = (T)1;
  for (int t = threadIdx.x; t < nr * nr; t += blockDim.x) {
    const int i = t % nr, j = t / nr;
    if (i >= j) M[rootIdx(nr, i, j)] = (T)K[t];
  }
  __syncthreads();
  int fail = 0, wrong = 0;
  double mind = 0.0;
  const long long t0 = clock64();
  denseLdlt<T>(c, M, st, fail, wrong, mind);
  const long long t1 = clock64();
  for (int t = threadIdx.x; t < nr * nr; t += blockDim.x) {
    const int i = t % nr, j = t / nr;
    Lout[t] = (i > j) ? (double)M[rootIdx(nr, i, j)] : ((i == j) ? 1.0 : 0.0);
  }
  for (int i = threadIdx.x; i < nr; i += blockDim.x) Dout[i] = (double)M[rootIdx(nr, i, i)];
  for (int i = threadIdx.x; i < Tn * kTile; i += blockDim.x) y[i] = (i < nr) ? (T)b[i] : (T)0;
  __syncthreads();
  const long long t2 = clock64();
  denseSolve<T>(c, M, y);
  const long long t3 = clock64();
  for (int i = threadIdx.x; i < nr; i += blockDim.x) xout[i] = (double)y[i];
  if (threadIdx.x == 0) {
    cyc[0] = t1 - t0;
    cyc[1] = t3 - t2;
    flags[0] = fail;
    flags[1] = wrong;
  }
}

template <typename T>
static cudaError_t probeLaunch(int nr, int nx, const double* K, const double* b, const DevSettings& st, int threads,
                               double* L, double* D, double* x, long long* cyc, int* flags) {
  const size_t smem = (size_t)(rootSize(nr) + (int64_t)rootTiles(nr) * kTile) * sizeof(T);
  cudaError_t e = cudaFuncSetAttribute(denseProbeKernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  denseProbeKernel<T><<<1, threads, smem>>>(nr, nx, K, b, st, L, D, x, cyc, flags);
  return cudaGetLastError();
}

size_t denseProbeSmem(int arith, int nr) {
  const size_t elem = (arith == 1) ? 4 : 8;
  return (size_t)(rootSize(nr) + (int64_t)rootTiles(nr) * kTile) * elem;
}

cudaError_t launchDenseProbe(int arith, int nr, int nx, const double* K, const double* b, const DevSettings& st,
                             int threads, double* L, double* D, double* x, long long* cyc, int* flags) {
  if (arith == 1) return probeLaunch<float>(nr, nx, K, b, st, threads, L, D, x, cyc, flags);
  if (arith == 2) return probeLaunch<df64>(nr, nx, K, b, st, threads, L, D, x, cyc, flags);
  return probeLaunch<double>(nr, nx, K, b, st, threads, L, D, x, cyc, flags);
}

}  // namespace cxg
