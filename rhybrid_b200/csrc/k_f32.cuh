// FP32 precision form (sm_100a): particles stored as an int32 cell index, FP32
// offsets in the cell (cell units, [0,1)) and FP32 velocities (28 B per
// particle, one macroparticle weight per species), pushed and deposited in FP32
// with FP32 accumulation. The grid fields stay FP64 in HBM; a segment's field
// stencil is staged as FP32 in shared memory, and the moments are handed to the
// FP64 field update after the gather.
//
// The structure is the fast path's (k_fast.cuh): row segments of
// RHGPU_FAST_SEGMENT CIC dual cells, one block per segment and one thread per
// particle, stayers kept in order, deposit records counting-sorted by target
// dual cell and summed per (dual cell, corner) x 4 moments, particles leaving
// their segment deposited as exact fixed-point sums and placed afterwards.
// The arithmetic follows the reference's push (boris.h:64-194) and CIC weights
// (particle_accumulator.cpp:68-110) rewritten in cell units:
//   B = xs B(c) + (1 - xs) B(c - 1) with xs the offset (face2r);
//   w_x = off + 0.5 - s, s = (off >= 0.5) (accumulateCell's x0 shift);
//   drift off += v dt/dx; migration by exactly one cell.
// Deposit weights are geometric weights times w q / (w q of species 0), so the
// FP32 sums stay O(ppc); the gather scales by (w q)_0 / dV in FP64.
#pragma once

#include "rh_device.cuh"
#include "k_fields.cuh"
#include "k_particles.cuh"
#include "k_fast.cuh"
#include "k_diag.cuh"

namespace rh {

struct F32Buf {
   int* cell;        // cell index; the seven arrays are planes of one
   long long plane;  // their distance in elements
   float* o[3];      // offsets in the cell, cell units
   float* v[3];      // velocity [m/s]
   int* cnt;         // particles per segment
};
struct F32Species {
   F32Buf cur, nxt;
   const long long* base;
};
struct F32Set {
   int ns;
   F32Species st[FAST_MAX_SPECIES];
   int accumulate[FAST_MAX_SPECIES];
   int accelerate[FAST_MAX_SPECIES];
   float qm[FAST_MAX_SPECIES];       // q dt / (2 m)
   float wqRel[FAST_MAX_SPECIES];    // (w q)_s / (w q)_0
   float R2obs[FAST_MAX_SPECIES];
   double w[FAST_MAX_SPECIES];       // macroparticle weight
};
struct F32Params {
   float dtdx;        // dt / dx
   float dt;
   float dx;
   float below1;      // largest float below 1
   float maxVi2;
   float GMdt;
   int useIFT, use_ep, use_gravity;
};

// a particle leaving its segment (FP32 form)
struct Mover32 {
   float o[3], v[3];
   int cell;
   int species;
   unsigned long long key;   // (source segment << 32) | index in the source segment
   long long dest;           // destination segment
   int lx;                   // dual x in the destination segment | MOVER_* flags
   int pad;
};

struct F32Bufs {
   float* RP;                  // 4 planes x nrows x nx x 4
   float* RPB;                 // 4 planes x nrows x nseg x 4
   unsigned long long* MMlo;   // N x 4 (shared with the FP64 fast path)
   unsigned long long* MMhi;
   const unsigned char* segInner;   // per segment: an obstacle cell within reach (shared with the fast path)
   Mover32* movers;
   unsigned long long* nmovers;
   long long moverCap;
   double scaleR, scaleJ;
};

__device__ inline int halfSf(float o) { return o < 0.5f ? 0 : 1; }

// the segment's field stencil as FP32 (staged by stageSegRows<float>)
using SegFields32 = SegFieldsT<float>;

// Boris-Buneman push in FP32 (boris.h:64-194 in cell units); o: offsets, v: velocity
__device__ __forceinline__ bool pushF32(const GridInfo& g, const SegFields32& F, float qm, bool accelerate,
                                        const F32Params& pp, int i, int j, int k, int lc, int ly, int lz, float o[3],
                                        float v[3]) {
   bool clamp = false;
   float vx = v[0], vy = v[1], vz = v[2];
   if (accelerate) {
      float B[3], Ue[3], E[3];
      const float xs = o[0], ys = o[1], zs = o[2];
      constexpr int SX = SEG + 2;
      const int at = (2 * lz + ly) * SX + lc;      // bx, bz, ue, ep
      const float* const bx = &F.bx[0][0][0] + at;
      const float* const by = &F.by[0][0][0] + at + lz * SX;
      const float* const bz = &F.bz[0][0][0] + at;
      const float* const ue = &F.ue[0][0][0][0] + at;
      // (fused multiply-adds: the FP32 form is not held to the FP64 operation order)
      B[0] = fmaf(xs, bx[1], (1.0f - xs) * bx[0]);
      B[1] = fmaf(ys, by[SX], (1.0f - ys) * by[0]);
      B[2] = fmaf(zs, bz[2 * SX], (1.0f - zs) * bz[0]);
#pragma unroll
      for (int l = 0; l < 3; ++l) Ue[l] = ue[4 * SX * l];
      E[0] = fmaf(B[1], Ue[2], -(B[2] * Ue[1]));
      E[1] = fmaf(B[2], Ue[0], -(B[0] * Ue[2]));
      E[2] = fmaf(B[0], Ue[1], -(B[1] * Ue[0]));
      if (pp.use_ep) {
         const float* const ep = &F.ep[0][0][0][0] + at;
#pragma unroll
         for (int l = 0; l < 3; ++l) E[l] += ep[4 * SX * l];
      }
      const float dvx = qm * E[0], dvy = qm * E[1], dvz = qm * E[2];
      const float tx = qm * B[0], ty = qm * B[1], tz = qm * B[2];
      const float t2 = fmaf(tx, tx, fmaf(ty, ty, tz * tz));
      const float b2 = 2.0f / (1.0f + t2);
      const float sx = b2 * tx, sy = b2 * ty, sz = b2 * tz;
      const float vmx = vx + dvx, vmy = vy + dvy, vmz = vz + dvz;
      const float v0x = fmaf(-vmz, ty, fmaf(vmy, tz, vmx));
      const float v0y = fmaf(-vmx, tz, fmaf(vmz, tx, vmy));
      const float v0z = fmaf(-vmy, tx, fmaf(vmx, ty, vmz));
      const float vpx = fmaf(-v0z, sy, fmaf(v0y, sz, vmx));
      const float vpy = fmaf(-v0x, sz, fmaf(v0z, sx, vmy));
      const float vpz = fmaf(-v0y, sx, fmaf(v0x, sy, vmz));
      vx = vpx + dvx; vy = vpy + dvy; vz = vpz + dvz;
      if (pp.use_gravity) {
         const float xg = (float)blockOrigin(g.x_min, i, g.dx) + o[0] * pp.dx;
         const float yg = (float)blockOrigin(g.y_min, j, g.dx) + o[1] * pp.dx;
         const float zg = (float)blockOrigin(g.z_min, k, g.dx) + o[2] * pp.dx;
         const float rr = sqrtf(xg * xg + yg * yg + zg * zg);
         const float r3 = rr * rr * rr;
         if (r3 > 0.0f) {
            const float sg = -pp.GMdt / r3;
            vx += sg * xg; vy += sg * yg; vz += sg * zg;
         }
      }
      const float v2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
      if (v2 > pp.maxVi2) {
         const float norm = sqrtf(pp.maxVi2 / v2);
         vx *= norm; vy *= norm; vz *= norm;
         clamp = true;
      }
   }
   v[0] = vx; v[1] = vy; v[2] = vz;
   o[0] = fmaf(pp.dtdx, vx, o[0]);
   o[1] = fmaf(pp.dtdx, vy, o[1]);
   o[2] = fmaf(pp.dtdx, vz, o[2]);
   return clamp;
}

// migration of one offset by exactly one cell; nonzero if it moved further
__device__ inline int migrateAxisF(float& o, int& off, float below1) {
   int st = 0;
   off = 0;
   if (o < 0.0f) {
      o += 1.0f;
      off = -1;
      if (o >= 1.0f) o = below1;
      if (o < 0.0f) st = 1;
   } else if (o >= 1.0f) {
      o -= 1.0f;
      off = 1;
      if (o >= 1.0f) st = 1;
   }
   return st;
}

// CIC weights in cell units (accumulateCell's weights), times wq
__device__ inline void cicWeightsF(const float o[3], float wq, float w8[8]) {
   const float wx = o[0] + 0.5f - (float)halfSf(o[0]);
   const float wy = o[1] + 0.5f - (float)halfSf(o[1]);
   const float wz = o[2] + 0.5f - (float)halfSf(o[2]);
   w8[0] = (1.0f - wx) * (1.0f - wy) * (1.0f - wz) * wq;
   w8[1] = wx * (1.0f - wy) * (1.0f - wz) * wq;
   w8[2] = (1.0f - wx) * wy * (1.0f - wz) * wq;
   w8[3] = wx * wy * (1.0f - wz) * wq;
   w8[4] = (1.0f - wx) * (1.0f - wy) * wz * wq;
   w8[5] = wx * (1.0f - wy) * wz * wq;
   w8[6] = (1.0f - wx) * wy * wz * wq;
   w8[7] = wx * wy * wz * wq;
}

constexpr int REC32 = 12;   // floats per deposit record: w8[8], then 1, v[3] (48 bytes apart: any eight on different banks)

// resident blocks per SM: the kernel waits on its barriers and shared-memory
// round trips, so warps count for more than the few registers that 32 a thread
// spill (Mars run, 9.25e7 ions: 4 blocks 3.63 ms, 5 3.31, 6 3.09, 8 3.05)
constexpr int F32_BLOCKS = 8;
// shared memory of k_f32_push_deposit
// one species' storage at the block's segment: its current and next cell planes
// and the other planes' distances (cell, o[3], v[3])
struct F32At {
   const int* cur;
   int* nxt;
   long long curPlane, nxtPlane;
};
struct F32PushShared {
   alignas(16) float rec[PD_T * REC32];     // deposit records of a chunk; at the end acc[SEG][32]
   float pf[7][PD_T];                       // the next chunk's particles: cell (int bits), o[3], v[3]
   SegFields32 f;                           // field stencil of the segment
   F32At at[FAST_MAX_SPECIES];
   StencilRow rows[SF_MAX_ROWS];
   alignas(8) unsigned char wd[SEG][PD_VW];   // records per (dual cell, group)
   int wcnt[PD_VW];                         // stayers per group
   int first[FAST_MAX_SPECIES + 1];         // first group of each species in the segment
   int cnt[FAST_MAX_SPECIES];               // particles of each species in the segment
   int stay[FAST_MAX_SPECIES];              // stayers of each species up to and with the chunk
};

// this thread's particle of the chunk that starts at group V0 requested into pf
// (cp.async): its species s and index p (p < 0: none)
__device__ __forceinline__ void f32Prefetch(F32PushShared& sh, int V0, int ns, int& s, int& p) {
   const int tid = threadIdx.x, V = V0 + (tid >> 5);
   s = pdSpecies(sh, V, ns);
   p = (V - sh.first[s]) * 32 + (tid & 31);
   if (p >= sh.cnt[s]) {
      p = -1;
   } else {
      const int* q = sh.at[s].cur + p;
      const long long plane = sh.at[s].curPlane;
#pragma unroll
      for (int a = 0; a < 7; ++a, q += plane) cpAsync4(&sh.pf[a][tid], q);
   }
   cpAsyncCommit();
}

// PER: the periodic axes (bit a = axis a), fixed at compile time; the host
// launches the instantiation that matches the grid
// GC: the variant that also counts the per-cell maxVi constraint (grid counters on)
//
// One block per segment, as k_fast_push_deposit: chunks of PD_T particles,
// every species starting at a group of 32, one particle per thread, the next
// chunk copied to shared memory (cp.async) while the current one is processed,
// two barriers per chunk, per-group record counts packed in bytes, a leaving
// particle's mover slot reserved before the second barrier and written after
// the deposit sums.
template <int PER, bool GC>
__global__ void __launch_bounds__(PD_T, F32_BLOCKS)
k_f32_push_deposit(GridInfo gIn, Fields f, FastGeom fg, F32Set FS, F32Params pp, F32Bufs fb, double* cntd,
                   unsigned long long* cntu, unsigned* err) {
   GridInfo g = gIn;
   g.per[0] = PER & 1;
   g.per[1] = (PER >> 1) & 1;
   g.per[2] = (PER >> 2) & 1;
   __shared__ F32PushShared sh;
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const unsigned below = (1u << lane) - 1u;
   const int S = (int)blockIdx.x;
   const int nseg = fg.nseg;
   const int row = S / nseg, gseg = S - row * nseg;
   const int uz = row / fg.nd[1], uy = row - uz * fg.nd[1];
   const int u0 = gseg * SEG, u1 = min(u0 + SEG, fg.nd[0]);
   const int ns = FS.ns;
   const int xs0 = dualB(u0, g.per[0]), ys0 = dualB(uy, g.per[1]), zs0 = dualB(uz, g.per[2]);
   const bool segInner = fb.segInner[S] != 0;   // an obstacle cell within one step of the segment
   // every cell a particle of the segment can be in or reach has its neighbours in y and z
   const bool yzIn = ((PER & 2) || (ys0 >= 2 && ys0 + 2 <= g.ny - 2)) && ((PER & 4) || (zs0 >= 2 && zs0 + 2 <= g.nz - 2));
   // set-up: species (warp 0), segment pointers
   if (warp == 0) {
      const int cnt = lane < ns ? FS.st[lane].cur.cnt[S] : 0;
      const int groups = (cnt + 31) >> 5;
      int x = groups;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
         const int y = __shfl_up_sync(0xffffffffu, x, o);
         if (lane >= o) x += y;
      }
      if (lane <= ns) sh.first[lane] = x - groups;
      if (lane < FAST_MAX_SPECIES) { sh.cnt[lane] = cnt; sh.stay[lane] = 0; }
   }
   if (tid >= 32 && tid < 32 + ns) {
      const F32Species& SS = FS.st[tid - 32];
      const long long b = SS.base[S];
      F32At& A = sh.at[tid - 32];
      A.cur = SS.cur.cell + b;
      A.nxt = SS.nxt.cell + b;
      A.curPlane = SS.cur.plane;
      A.nxtPlane = SS.nxt.plane;
   }
   // (stageSegRows' own barrier publishes the species and the pointers)
   stageSegRows<PD_T>(g, f, pp.use_ep, xs0, ys0, zs0, sh.f, sh.rows);
   __syncthreads();
   const int groups = sh.first[ns];
   int sn = 0, pn = -1;   // the prefetched particle's species and index
   f32Prefetch(sh, 0, ns, sn, pn);
   const int myDual = tid >> 3, myPair = (tid >> 1) & 3, myHalf = tid & 1;
   float a00 = 0.0f, a01 = 0.0f, a10 = 0.0f, a11 = 0.0f;

   for (int V0 = 0; V0 < groups; V0 += PD_VW) {
      float o[3], v[3];
      int cell = 0, duv = 0, dyz = 0, mflags = 0, rrank = 0;
      bool stay = false, rec = false, clamp = false;
      cpAsyncWaitAll();   // this thread's copies of the chunk
      const int s = sn, p = pn;
      if (p >= 0) {
         const int c = __float_as_int(sh.pf[0][tid]);
#pragma unroll
         for (int a = 0; a < 3; ++a) { o[a] = sh.pf[1 + a][tid]; v[a] = sh.pf[4 + a][tid]; }
         const int gx = halfSf(o[0]), gy = halfSf(o[1]), gz = halfSf(o[2]);
         const int ly = 1 - gy, lz = 1 - gz;
         const int cj = ys0 + ly, ck = zs0 + lz;   // not wrapped (periodic axes: up to n)
         const int wj = (PER & 2) && cj >= g.ny ? cj - g.ny : cj, wk = (PER & 4) && ck >= g.nz ? ck - g.nz : ck;
         const int wi = c - g.nx * (wj + g.ny * wk);
         const int lu = dualU(wi + gx - 1, g.nx, g.per[0]) - u0;
         const int lc = lu + 1 - gx, ci = xs0 + lc;
         bool accelerate = FS.accelerate[s] && !pp.useIFT && ((PER & 1) || (unsigned)(ci - 1) < (unsigned)(g.nx - 2));
         if (!yzIn)
            accelerate = accelerate && ((PER & 2) || (unsigned)(cj - 1) < (unsigned)(g.ny - 2)) &&
                         ((PER & 4) || (unsigned)(ck - 1) < (unsigned)(g.nz - 2));
         clamp = pushF32(g, sh.f, FS.qm[s], accelerate, pp, wi, wj, wk, lc, ly, lz, o, v);
         if (GC) gridCountAtomic(f, GC_CELL_MAX_VI, g.N, c, clamp);
         if (isnan(o[0]) || isnan(o[1]) || isnan(o[2])) raiseError(err, RHGPU_DEVERR_NAN_PARTICLE);
         int ox, oy, oz;
         int bad = migrateAxisF(o[0], ox, pp.below1);
         bad |= migrateAxisF(o[1], oy, pp.below1);
         bad |= migrateAxisF(o[2], oz, pp.below1);
         // target cell: inside the box, and with all its neighbours
         int ti = ci + ox, tj = cj + oy, tk = ck + oz;
         bool inside = !bad && ((PER & 1) || (unsigned)ti < (unsigned)g.nx);
         bool all = (PER & 1) || (unsigned)(ti - 1) < (unsigned)(g.nx - 2);
         if (!yzIn) {
            inside = inside && ((PER & 2) || (unsigned)tj < (unsigned)g.ny) && ((PER & 4) || (unsigned)tk < (unsigned)g.nz);
            all = all && ((PER & 2) || (unsigned)(tj - 1) < (unsigned)(g.ny - 2)) &&
                  ((PER & 4) || (unsigned)(tk - 1) < (unsigned)(g.nz - 2));
         }
         bool removed = !inside || !all;
         if (removed) {
            double* const q = removedSums(cntd, S, s);
            atomicAdd(&q[0], FS.w[s]);
            atomicAdd(&q[1], FS.w[s] * ((double)v[0] * v[0] + (double)v[1] * v[1] + (double)v[2] * v[2]));
         }
         if (inside) {
            if (PER & 1) wrapc(ti, g.nx, 1);
            if (PER & 2) wrapc(tj, g.ny, 1);
            if (PER & 4) wrapc(tk, g.nz, 1);
            cell = ti + g.nx * (tj + g.ny * tk);
            // the new dual cell relative to the segment's first, and to its row
            int du = lu + ox + halfSf(o[0]) - gx;
            const int dy = oy + halfSf(o[1]) - gy, dz = oz + halfSf(o[2]) - gz;
            if ((PER & 1) && nseg == 1) {
               if (du < 0) du += fg.nd[0];
               else if (du >= fg.nd[0]) du -= fg.nd[0];
            }
            const bool inSeg = dy == 0 && dz == 0 && (unsigned)du < (unsigned)(u1 - u0);
            duv = du;
            dyz = (dy + 2) | ((dz + 2) << 3);
            if (FS.accumulate[s]) {
               rec = inSeg;   // its CIC weights are formed just before the record is written
               if (!inSeg) mflags = MOVER_DEPOSIT;
            }
            if (segInner && !removed && (f.flags[cell] & RHGPU_FLAG_INNER_PARTICLE)) {
               const float xp = (float)blockOrigin(g.x_min, ti, g.dx) + o[0] * pp.dx;
               const float yp = (float)blockOrigin(g.y_min, tj, g.dx) + o[1] * pp.dx;
               const float zp = (float)blockOrigin(g.z_min, tk, g.dx) + o[2] * pp.dx;
               if (xp * xp + yp * yp + zp * zp < FS.R2obs[s]) {
                  removed = true;
                  double* const q = removedSums(cntd, S, s);
                  atomicAdd(&q[2], FS.w[s]);
                  atomicAdd(&q[3], FS.w[s] * ((double)v[0] * v[0] + (double)v[1] * v[1] + (double)v[2] * v[2]));
               }
            }
            if (!removed) {
               stay = inSeg;
               if (!inSeg) mflags |= MOVER_PLACE;
            }
         }
      }
      if (clamp) atomicAdd(&cntu[CNT_SPECIES_MAXVI + s], 1ull);
      // order of the group's stayers and records: ballots, and its records per dual cell
      const unsigned bs = __ballot_sync(0xffffffffu, stay);
      const unsigned br = __ballot_sync(0xffffffffu, rec);
      if (lane == 0) {
         const int n = __popc(bs);
         sh.wcnt[warp] = n;
         if (n) atomicAdd(&sh.stay[s], n);
      }
      sh.wd[lane][warp] = 0;
      __syncwarp();
      if (rec) {
         const unsigned mm = __match_any_sync(br, duv);
         rrank = __popc(mm & below);
         if (rrank == 0) sh.wd[duv][warp] = (unsigned char)__popc(mm);
      }
      __syncthreads();
      // every shared-memory read of this chunk's particles is done: request the next chunk's
      if (V0 + PD_VW < groups) f32Prefetch(sh, V0 + PD_VW, ns, sn, pn);
      // every warp, per dual cell (lane): the first sorted record of the dual cell (bin)
      const uint2 c8 = *reinterpret_cast<const uint2*>(&sh.wd[lane][0]);
      int binD, nrec;
      {
         const int t = (int)(((c8.x * 0x01010101u) >> 24) + ((c8.y * 0x01010101u) >> 24));
         int x = t;
         for (int q = 1; q < 32; q <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, q);
            if (lane >= q) x += y;
         }
         binD = x - t;
         nrec = __shfl_sync(0xffffffffu, x, 31);
      }
      const int sumLo = __shfl_sync(0xffffffffu, binD, myDual);
      const int sumHiN = __shfl_sync(0xffffffffu, binD, (myDual + 1) & 31);
      const int sumHi = myDual == SEG - 1 ? nrec : sumHiN;
      const int wc = lane < PD_VW ? sh.wcnt[lane] : 0;
      // this group's records start after those of the groups before it, per dual cell
      const unsigned mlo = warp >= 4 ? 0xffffffffu : (1u << (8 * warp)) - 1u;
      const unsigned mhi = warp <= 4 ? 0u : (1u << (8 * (warp - 4))) - 1u;
      const int before = (int)((((c8.x & mlo) * 0x01010101u) >> 24) + (((c8.y & mhi) * 0x01010101u) >> 24));
      const int recPos = __shfl_sync(0xffffffffu, binD + before, rec ? duv : 0) + rrank;
      // next slot of a stayer: the species' stayers up to and with the chunk less those from this group on
      const int vEnd = sh.first[s + 1] - V0;
      const int from = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane >= warp && lane < vEnd ? wc : 0));
      const int slot = sh.stay[s] - from + __popc(bs & below);
      // mover slots reserved now, written after the sums
      const unsigned lm = __ballot_sync(0xffffffffu, mflags != 0);
      unsigned long long mb = 0;
      if (lm && lane == __ffs(lm) - 1) mb = atomicAdd(fb.nmovers, (unsigned long long)__popc(lm));
      if (rec) {
         float w8[8];
         cicWeightsF(o, FS.wqRel[s], w8);
         float4* const r = reinterpret_cast<float4*>(sh.rec + recPos * REC32);
         r[0] = make_float4(w8[0], w8[1], w8[2], w8[3]);
         r[1] = make_float4(w8[4], w8[5], w8[6], w8[7]);
         r[2] = make_float4(1.0f, v[0], v[1], v[2]);
      }
      __syncthreads();
      if (stay) {
         int* q = sh.at[s].nxt + slot;
         const long long plane = sh.at[s].nxtPlane;
         *q = cell;
#pragma unroll
         for (int a = 0; a < 3; ++a) { q += plane; *q = __float_as_int(o[a]); }
#pragma unroll
         for (int a = 0; a < 3; ++a) { q += plane; *q = __float_as_int(v[a]); }
      }
      // ---- this thread's sums, records in list order ----------------------------------------
#pragma unroll 2
      for (int r = sumLo; r < sumHi; ++r) {
         const float2* const rr = reinterpret_cast<const float2*>(sh.rec + r * REC32);
         const float2 w = rr[myPair], u = rr[4 + myHalf];
         a00 = fmaf(w.x, u.x, a00);
         a01 = fmaf(w.x, u.y, a01);
         a10 = fmaf(w.y, u.x, a10);
         a11 = fmaf(w.y, u.y, a11);
      }
      // ---- particles that left the segment -----------------------------------------------
      if (!lm) continue;
      const unsigned long long m0 = __shfl_sync(0xffffffffu, mb, __ffs(lm) - 1);
      if (!mflags) continue;
      const unsigned long long m = m0 + __popc(lm & below);
      if ((long long)m >= fb.moverCap) {
         raiseError(err, RHGPU_DEVERR_CAPACITY);
         continue;
      }
      int vx = u0 + duv, vy = uy + (dyz & 7) - 2, vz = uz + (dyz >> 3) - 2;
      if (PER & 1) wrapc(vx, fg.nd[0], 1);
      if (PER & 2) wrapc(vy, fg.nd[1], 1);
      if (PER & 4) wrapc(vz, fg.nd[2], 1);
      Mover32& M = fb.movers[m];
#pragma unroll
      for (int a = 0; a < 3; ++a) { M.o[a] = o[a]; M.v[a] = v[a]; }
      M.cell = cell;
      M.species = s;
      M.key = ((unsigned long long)S << 32) | (unsigned long long)p;
      const int gd = vx / SEG;
      M.dest = ((long long)vy + (long long)fg.nd[1] * vz) * nseg + gd;
      M.lx = (vx - gd * SEG) | mflags;
      // no barrier here: the next chunk's first barrier orders the reads of rec
      // and wd before their next writes
   }

   __syncthreads();
   if (tid < ns) FS.st[tid].nxt.cnt[S] = sh.stay[tid];
   {
      float* const q = sh.rec + myDual * 32 + myPair * 8 + myHalf * 2;
      q[0] = a00; q[1] = a01; q[4] = a10; q[5] = a11;
   }
   __syncthreads();
   segPartialsOut<PD_T>(g, fg, fb.RP, fb.RPB, sh.rec, row, gseg, u0, u1);
}

// corner o's four deposits of one mover (k_mover_pass): cicWeightsF's products, in its order
__device__ __forceinline__ void moverTerms(const GridInfo&, const F32Set& FS, const Mover32& M, int o, double t[4]) {
   float f[3];
   for (int a = 0; a < 3; ++a) {
      const float w = M.o[a] + 0.5f - (float)halfSf(M.o[a]);
      f[a] = (o >> a) & 1 ? w : 1.0f - w;
   }
   const float w = f[0] * f[1] * f[2] * FS.wqRel[M.species];
   t[0] = (double)w;
   for (int l = 0; l < 3; ++l) t[1 + l] = (double)(w * M.v[l]);
}
__device__ __forceinline__ void placeMover(const F32Species& SS, long long slot, const Mover32& M) {
   SS.nxt.cell[slot] = M.cell;
#pragma unroll
   for (int e = 0; e < 3; ++e) { SS.nxt.o[e][slot] = M.o[e]; SS.nxt.v[e][slot] = M.v[e]; }
}

// cell moments: gatherMoments times (w q)_0 / dV, and the rho clamp
template <bool GC>   // GC: also count the rho clamp per cell (grid counters on)
__global__ void __launch_bounds__(2 * GA_CELLS)
k_f32_gather(GridInfo g, Fields f, FastGeom fg, F32Bufs fb, double hiR, double loR, double hiJ, double loJ,
             double scale, double minRho, unsigned long long* cnt) {
   RH_GATHER_PROLOGUE
   double2 v = gatherMoments<float>(g, fg, fb, i, j, k, h, n, h ? hiJ : hiR, h ? loJ : loR, hiJ, loJ);
   v.x *= scale;
   v.y *= scale;
   const bool clamp = h == 0 && v.x < minRho;
   if (clamp) v.x = minRho;
   countIf(clamp, &cnt[CNT_MIN_CELL_RHO]);
   if (GC) gridCount(f, GC_CELL_MIN_RHOQI, N, n, clamp);
   (h ? f.cellJi + N : f.cellRho)[n] = v.x;
   (h ? f.cellJi + 2 * N : f.cellJi)[n] = v.y;
}

// ---- upload / download / relayout ----------------------------------------------------------
__device__ inline float offsetOf(double x, double rdx, float below1) {
   float o = (float)(x * rdx);
   if (o >= 1.0f) o = below1;
   if (o < 0.0f) o = 0.0f;
   return o;
}
// uploaded records: 7 doubles (cell-local position [m], velocity, weight), or
// the FP32 form's own 6 floats (offsets in the cell in units of dx, velocity)
struct RecordsD {
   const double* a;
   __device__ float off(long long p, int k, double rdx, float below1) const { return offsetOf(a[7 * p + k], rdx, below1); }
   __device__ float vel(long long p, int k) const { return (float)a[7 * p + 3 + k]; }
};
struct RecordsF {
   const float* a;
   __device__ float off(long long p, int k, double, float below1) const {
      float o = a[6 * p + k];
      if (o >= 1.0f) o = below1;
      if (o < 0.0f) o = 0.0f;
      return o;
   }
   __device__ float vel(long long p, int k) const { return a[6 * p + 3 + k]; }
};

// segment and dual x of each uploaded particle, from its FP32 offsets
template <class R>
__global__ void k_f32_seg_of(GridInfo g, FastGeom fg, R rec, const int* pcell, long long n, float below1,
                             unsigned* key) {
   const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (p >= n) return;
   const int c = pcell[p];
   const int i = c % g.nx, j = (c / g.nx) % g.ny, k = c / (g.nx * g.ny);
   const int ux = dualU(i + halfSf(rec.off(p, 0, g.rdx, below1)) - 1, g.nx, g.per[0]);
   const int uy = dualU(j + halfSf(rec.off(p, 1, g.rdx, below1)) - 1, g.ny, g.per[1]);
   const int uz = dualU(k + halfSf(rec.off(p, 2, g.rdx, below1)) - 1, g.nz, g.per[2]);
   key[p] = (unsigned)(((long long)uy + (long long)fg.nd[1] * uz) * fg.nseg + ux / SEG);
}
template <class R>
__global__ void k_f32_scatter_sorted(GridInfo g, R rec, const int* pcell, const unsigned* key,
                                     const unsigned* idx, long long n, const long long* first, F32Buf B,
                                     const long long* base, float below1) {
   const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (j >= n) return;
   const unsigned S = key[j];
   const long long slot = base[S] + (j - first[S]);
   const unsigned src = idx[j];
   B.cell[slot] = pcell[src];
   for (int a = 0; a < 3; ++a) {
      B.o[a][slot] = rec.off(src, a, g.rdx, below1);
      B.v[a][slot] = rec.vel(src, a);
   }
}
__global__ void k_f32_cell_keys(FastGeom fg, F32Buf B, const long long* base, const long long* first, unsigned* key,
                                unsigned long long* slots);
__global__ void k_f32_gather_records(F32Buf B, const unsigned long long* slots, const unsigned* idx, long long n,
                                     double dx, double w, double* aos);
// the FP32 form's own records: 6 floats per particle, offsets and velocity as stored
__global__ void k_f32_gather_records_f32(F32Buf B, const unsigned long long* slots, const unsigned* idx, long long n,
                                         float* rec);
__global__ void k_f32_relayout(F32Buf from, const long long* fromBase, F32Buf to, const long long* toBase);
// min and max |weight| of uploaded particles, grid-stride with one atomic pair per block
// (bit patterns of non-negative doubles order like the values)
__global__ void k_weight_range(const double* aos, long long n, unsigned long long* mn, unsigned long long* mx);
// population log sums of one FP32-form species in FP64 (see k_diag.cuh)
__global__ void __launch_bounds__(DIAG_THREADS)
k_diag_particles_f32(F32Buf B, const long long* base, long long NS, double w, double* part);

// total ion mass density (logCalcParticle, diagnostics.h:223-238) on the FP32
// form: every particle adds its species' w*m to its cell as an exact fixed-point sum
__global__ void k_diag_rhom_f32(F32Buf B, const long long* base, long long NS, double wm, double scale,
                                unsigned long long* lo, unsigned long long* hi);

}  // namespace rh
