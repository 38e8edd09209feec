// Temporal averages of the output populations (WRITE_GRID_TEMPORAL_AVERAGES,
// the reference's default build):
//   every step, each accumulating species adds its CIC charge and current sums
//   (before /dV) to the sums of its output population
//     (particle_accumulator.cpp:148-150, 208-215)
//   at an output step, n_<pop>_ave = sum / (q dV) / count, v_<pop>_ave =
//   current sum / charge sum, cellBAverage = sum / count, and the sums restart
//     (operator_userdata.cpp:155-223)
//
//   k_deposit_gather_avg   exact path: one species' 27 per-source sums added to
//                          its population's sums in the reference's order
//   fast path, right after the step's deposit (the same particles it deposits):
//   k_fast_avg_deposit     one block per row segment over the population's
//                          species' particles that stayed in their segment:
//                          CIC records counting-sorted by dual cell and summed
//                          per (dual cell, corner) as the push kernel does,
//                          out as row partials
//   k_mover_pass           the population's deposits that went through the
//                          mover list (left their segment; or deposited in it
//                          and then removed by a boundary), as exact
//                          fixed-point sums
//   k_fast_avg_gather      per cell, row partials + fixed-point part added to
//                          the sums
//   k_avg_output           the output step's normalisation and restart
#pragma once

#include "rh_device.cuh"
#include "k_particles.cuh"
#include "k_fast.cuh"

namespace rh {

// exact path: v_sum of cell n += this species' contributions, sources in ID order
__global__ void k_deposit_gather_avg(GridInfo g, const double* S, double* nSum, double* vSum);

// fast path: the CIC sums of the species in `mask` (bit s) over the particles of
// FS.st[s].cur (the step's stayers), as row partials in fb.RP / fb.RPB. One block
// per segment, records and sums as in k_fast_push_deposit; a thread's next
// particle is loaded while its chunk is processed. (Both populations of 61 x 83 x
// 70 cells, 4.0e6 ions, with the movers' part and the gather: 274 us; 289 us
// with every chunk's loads waited for and one corner x four moments per thread.)
template <int PER>
__global__ void __launch_bounds__(PD_T, 4)
k_fast_avg_deposit(GridInfo gIn, FastGeom fg, FastSpecies FS, unsigned mask, FastBufs fb) {
   GridInfo g = gIn;
   g.per[0] = PER & 1;
   g.per[1] = (PER >> 1) & 1;
   g.per[2] = (PER >> 2) & 1;
   __shared__ alignas(16) double s_rec[PD_T * PD_REC];
   __shared__ alignas(8) unsigned char s_wd[SEG][PD_VW];   // records per (dual cell, warp)
   __shared__ int s_prefix[FAST_MAX_SPECIES + 1];
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const unsigned below = (1u << lane) - 1u;
   const long long S = blockIdx.x;
   const long long row = S / fg.nseg;
   const int gseg = (int)(S % fg.nseg);
   const int u0 = gseg * SEG, u1 = min(u0 + SEG, fg.nd[0]);
   const int ns = FS.ns;
   const double hdx = 0.5 * g.dx;
   if (tid == 0) {
      int a = 0;
      for (int s = 0; s < ns; ++s) {
         s_prefix[s] = a;
         if ((mask >> s) & 1u) a += FS.st[s].cur.cnt[S];
      }
      s_prefix[ns] = a;
   }
   __syncthreads();
   const int total = s_prefix[ns];
   const int myDual = tid >> 3, myPair = (tid >> 1) & 3, myHalf = tid & 1;
   double a00 = 0.0, a01 = 0.0, a10 = 0.0, a11 = 0.0;
   double next[7] = {};
   int nextRd = 0, nextS = 0;
   auto load = [&](int i) {
      if (i >= total) return;
      int s = 0;
      while (s + 1 < ns && i >= s_prefix[s + 1]) ++s;
      const SegSpecies& SS = FS.st[s];
      const long long slot = SS.base[S] + (i - s_prefix[s]);
#pragma unroll
      for (int a = 0; a < 7; ++a) next[a] = SS.cur.a[a][slot];
      nextRd = SS.cur.lx[slot];
      nextS = s;
   };
   load(tid);
   for (int c0 = 0; c0 < total; c0 += PD_T) {
      const int i = c0 + tid;
      const bool rec = i < total;
      double st[7];
#pragma unroll
      for (int a = 0; a < 7; ++a) st[a] = next[a];
      const int rd = nextRd, s = nextS;
      load(i + PD_T);
      // records counting-sorted by dual cell: chunk, warp, lane order within a dual cell
      const unsigned br = __ballot_sync(0xffffffffu, rec);
      s_wd[lane][warp] = 0;
      __syncwarp();
      int rrank = 0;
      if (rec) {
         const unsigned mm = __match_any_sync(br, rd);
         rrank = __popc(mm & below);
         if (rrank == 0) s_wd[rd][warp] = (unsigned char)__popc(mm);
      }
      __syncthreads();
      const uint2 c8 = *reinterpret_cast<const uint2*>(&s_wd[lane][0]);
      int binD, nrec;
      {
         const int t = (int)(((c8.x * 0x01010101u) >> 24) + ((c8.y * 0x01010101u) >> 24));
         int x = t;
         for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
         }
         binD = x - t;
         nrec = __shfl_sync(0xffffffffu, x, 31);
      }
      const unsigned mlo = warp >= 4 ? 0xffffffffu : (1u << (8 * warp)) - 1u;
      const unsigned mhi = warp <= 4 ? 0u : (1u << (8 * (warp - 4))) - 1u;
      const int before = (int)((((c8.x & mlo) * 0x01010101u) >> 24) + (((c8.y & mhi) * 0x01010101u) >> 24));
      const int recPos = __shfl_sync(0xffffffffu, binD + before, rec ? rd : 0) + rrank;
      const int sumLo = __shfl_sync(0xffffffffu, binD, myDual);
      const int sumHiN = __shfl_sync(0xffffffffu, binD, (myDual + 1) & 31);
      const int sumHi = myDual == SEG - 1 ? nrec : sumHiN;
      if (rec) {
         const double w_x = cicFraction(st[0], g, hdx), w_y = cicFraction(st[1], g, hdx), w_z = cicFraction(st[2], g, hdx);
         writeRecord(s_rec + recPos * PD_REC, w_x, w_y, w_z, st[6] * FS.sp[s].q, st[3], st[4], st[5]);
      }
      __syncthreads();
#pragma unroll 2
      for (int r = sumLo; r < sumHi; ++r) {
         const double2* const rr = reinterpret_cast<const double2*>(s_rec + r * PD_REC);
         const double2 w = rr[myPair], u = rr[4 + myHalf];
         a00 += w.x * u.x;
         a01 += w.x * u.y;
         a10 += w.y * u.x;
         a11 += w.y * u.y;
      }
      // the next chunk's first barrier orders these reads before its record writes
   }
   __syncthreads();
   double* const q = s_rec + myDual * 32 + myPair * 8 + myHalf * 2;
   q[0] = a00; q[1] = a01; q[4] = a10; q[5] = a11;
   __syncthreads();
   segPartialsOut<PD_T>(g, fg, fb.RP, fb.RPB, s_rec, row, gseg, u0, u1);
}

// fast path: row partials + fixed-point part added to the population's sums; the
// host clears the fixed-point sums after it
__global__ void __launch_bounds__(2 * GA_CELLS)
k_fast_avg_gather(GridInfo g, FastGeom fg, FastBufs fb, double hiR, double loR, double hiJ, double loJ, double* nSum,
                  double* vSum);

// output step of one population (operator_userdata.cpp:182-211): n = sum/(q dV)*inv,
// v = current sum / charge sum where the charge sum is positive, else 0; the sums
// restart. Outputs interleaved per cell (ParGrid order), as the ABI's arrays.
__global__ void k_avg_output(long long N, double* nSum, double* vSum, double q, double dV, double inv, double* nOut,
                             double* vOut);

// cellBAverage = cellAverageB * inv, and the sum restarts (operator_userdata.cpp:162-176)
__global__ void k_avgB_output(long long N, double* sumB, double inv, double* out);

}  // namespace rh
