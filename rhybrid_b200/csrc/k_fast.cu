// Definitions of the kernels declared in k_fast.cuh (each declaration there says
// what its kernel does); the template kernels stay in the header.
#include "k_fast.cuh"

namespace rh {

__global__ void k_mig_large_list(const int* inc, long long nb, unsigned* large, int* nlarge) {
   const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (b < nb && inc[b] > MIG_RANK) large[atomicAdd(nlarge, 1)] = (unsigned)b;
}

__global__ void __launch_bounds__(MIG_LARGE_THREADS) k_mig_order_large(const int* inc, const long long* off,
                                                                        unsigned long long* klist, unsigned* vlist,
                                                                        const unsigned* large, const int* nlarge) {
   __shared__ unsigned long long skey[MIG_LARGE];
   __shared__ unsigned sval[MIG_LARGE];
   const int n = *nlarge;
   for (int q = blockIdx.x; q < n; q += gridDim.x) {
      const unsigned b = large[q];
      const int k = inc[b];
      unsigned long long* const kl = klist + off[b];
      unsigned* const vl = vlist + off[b];
      int m = 1;
      while (m < k) m <<= 1;
      for (int i = threadIdx.x; i < m; i += MIG_LARGE_THREADS) {
         skey[i] = i < k ? kl[i] : ~0ull;
         sval[i] = i < k ? vl[i] : ~0u;
      }
      __syncthreads();
      for (int size = 2; size <= m; size <<= 1) {
         for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < m; i += MIG_LARGE_THREADS) {
               const int j = i ^ stride;
               if (j > i) {
                  const bool up = (i & size) == 0;
                  const unsigned long long ki = skey[i], kj = skey[j];
                  const unsigned vi = sval[i], vj = sval[j];
                  const bool gt = ki > kj || (ki == kj && vi > vj);
                  if (gt == up) {
                     skey[i] = kj; skey[j] = ki;
                     sval[i] = vj; sval[j] = vi;
                  }
               }
            }
            __syncthreads();
         }
      }
      for (int i = threadIdx.x; i < k; i += MIG_LARGE_THREADS) vl[i] = sval[i];
      __syncthreads();
   }
}

__global__ void k_fast_seg_of(GridInfo g, FastGeom fg, const double* aos, const int* pcell, long long n,
                              unsigned* key, unsigned char* lx) {
   const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (p >= n) return;
   const int c = pcell[p];
   const int i = c % g.nx, j = (c / g.nx) % g.ny, k = c / (g.nx * g.ny);
   const double* st = aos + 7 * p;
   const int ux = dualU(i + halfS(st[0], g.dx) - 1, g.nx, g.per[0]);
   const int uy = dualU(j + halfS(st[1], g.dx) - 1, g.ny, g.per[1]);
   const int uz = dualU(k + halfS(st[2], g.dx) - 1, g.nz, g.per[2]);
   const int gs = ux / SEG;
   key[p] = (unsigned)(((long long)uy + (long long)fg.nd[1] * uz) * fg.nseg + gs);
   lx[p] = (unsigned char)(ux - gs * SEG);
}

__global__ void k_sorted_bounds(const unsigned* key, long long n, long long nkeys, long long* first) {
   const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (j > n) return;
   const long long lo = j == 0 ? 0 : (long long)key[j - 1] + 1;
   const long long hi = j == n ? nkeys : (long long)key[j];
   for (long long k = lo; k <= hi; ++k) first[k] = j;
}

__global__ void k_bounds_counts(const long long* first, long long nkeys, int* cnt) {
   const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (k < nkeys) cnt[k] = (int)(first[k + 1] - first[k]);
}

__global__ void k_fast_capacity(long long NS, const int* cnt, const int* extra, long long* cap) {
   const long long d = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (d < NS) {
      const long long c = (long long)cnt[d] + (extra ? extra[d] : 0);
      cap[d] = c + max(32LL, c / 4);
   } else if (d == NS) {
      cap[d] = 0;
   }
}

__global__ void k_fast_scatter_sorted(const double* aos, const unsigned char* lxIn, const unsigned* key,
                                      const unsigned* idx, long long n, const long long* first, SegBuf B,
                                      const long long* base) {
   const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (j >= n) return;
   const unsigned S = key[j];
   const long long slot = base[S] + (j - first[S]);
   const unsigned src = idx[j];
   for (int a = 0; a < 7; ++a) B.a[a][slot] = aos[7LL * src + a];
   B.lx[slot] = lxIn[src];
}

__global__ void k_fast_cell_keys(GridInfo g, FastGeom fg, SegBuf B, const long long* base, const long long* first,
                                 unsigned* key, unsigned long long* slots) {
   const long long S = blockIdx.x;
   const long long row = S / fg.nseg;
   const int gs = (int)(S % fg.nseg);
   const int uy = (int)(row % fg.nd[1]), uz = (int)(row / fg.nd[1]);
   const int c = B.cnt[S];
   for (int r = threadIdx.x; r < c; r += blockDim.x) {
      const long long slot = base[S] + r;
      const int u = gs * SEG + B.lx[slot];
      int ci = dualB(u, g.per[0]) + 1 - halfS(B.a[0][slot], g.dx);
      int cj = dualB(uy, g.per[1]) + 1 - halfS(B.a[1][slot], g.dx);
      int ck = dualB(uz, g.per[2]) + 1 - halfS(B.a[2][slot], g.dx);
      wrapc(ci, g.nx, 1); wrapc(cj, g.ny, 1); wrapc(ck, g.nz, 1);
      key[first[S] + r] = (unsigned)cidx(g, ci, cj, ck);
      slots[first[S] + r] = (unsigned long long)slot;
   }
}

__global__ void k_fast_gather_records(SegBuf B, const unsigned long long* slots, const unsigned* idx, long long n,
                                      double* aos) {
   const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (j >= n) return;
   const unsigned long long slot = slots[idx[j]];
   for (int a = 0; a < 7; ++a) aos[7 * j + a] = B.a[a][slot];
}

__global__ void k_fast_relayout(SegBuf from, const long long* fromBase, SegBuf to, const long long* toBase) {
   const long long S = blockIdx.x;
   const int c = from.cnt[S];
   const long long a0 = fromBase[S], b0 = toBase[S];
   for (int r = threadIdx.x; r < c; r += blockDim.x) {
      for (int e = 0; e < 7; ++e) to.a[e][b0 + r] = from.a[e][a0 + r];
      to.lx[b0 + r] = from.lx[a0 + r];
   }
   if (threadIdx.x == 0) to.cnt[S] = c;
}

__global__ void k_fast_max_abs_w(SegBuf B, const long long* base, unsigned long long* out) {
   __shared__ double sm[32];
   const long long S = blockIdx.x;
   const int c = B.cnt[S];
   double m = 0.0;
   for (int r = threadIdx.x; r < c; r += blockDim.x) m = fmax(m, fabs(B.a[6][base[S] + r]));
   for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
   if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, sm[w]);
      if (m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
   }
}

}  // namespace rh
