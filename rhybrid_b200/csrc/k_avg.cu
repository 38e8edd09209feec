// Definitions of the kernels declared in k_avg.cuh (each declaration there says
// what its kernel does); the template kernels stay in the header.
#include "k_avg.cuh"

namespace rh {

__global__ void k_deposit_gather_avg(GridInfo g, const double* S, double* nSum, double* vSum) {
   RH_CELL_PROLOGUE
   const Sources3 Q = sortedSources(g, i, j, k);
   double v[4];
   v[0] = nSum[n];
   for (int l = 0; l < 3; ++l) v[1 + l] = vSum[l * N + n];
   addSources(g, Q, S, N, v);
   nSum[n] = v[0];
   for (int l = 0; l < 3; ++l) vSum[l * N + n] = v[1 + l];
}

__global__ void __launch_bounds__(2 * GA_CELLS)
k_fast_avg_gather(GridInfo g, FastGeom fg, FastBufs fb, double hiR, double loR, double hiJ, double loJ, double* nSum,
                  double* vSum) {
   RH_GATHER_PROLOGUE
   double* const s0 = (h ? vSum + N : nSum) + n;
   double* const s1 = (h ? vSum + 2 * N : vSum) + n;
   const double2 v = gatherMoments<double>(g, fg, fb, i, j, k, h, n, h ? hiJ : hiR, h ? loJ : loR, hiJ, loJ);
   *s0 += v.x;
   *s1 += v.y;
}

__global__ void k_avg_output(long long N, double* nSum, double* vSum, double q, double dV, double inv, double* nOut,
                             double* vOut) {
   const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (n >= N) return;
   const double a = nSum[n];
   if (nOut) nOut[n] = a / (q * dV) * inv;
   if (vOut)
      for (int l = 0; l < 3; ++l) vOut[3 * n + l] = a > 0 ? vSum[l * N + n] / a : 0.0;
   nSum[n] = 0.0;
   for (int l = 0; l < 3; ++l) vSum[l * N + n] = 0.0;
}

__global__ void k_avgB_output(long long N, double* sumB, double inv, double* out) {
   const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (n >= N) return;
   for (int l = 0; l < 3; ++l) {
      out[3 * n + l] = sumB[l * N + n] * inv;
      sumB[l * N + n] = 0.0;
   }
}

}  // namespace rh
