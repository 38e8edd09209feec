// Fast path (sm_100a, FP64): fused push + CIC deposit over particles binned
// by row segment. Same per-particle and per-cell arithmetic as the bit-exact
// path (boris.h:64-194, particle_accumulator.cpp:65-333); the deposit sums are
// formed in a different, fixed order, restated bit for bit by the oracle's
// RHO_DEPOSIT_GPU mode (oracle/rh_oracle.c).
//
// Dual cells: the 2x2x2 block of cells whose centres surround a particle
// (base b = c + s - 1 per axis, s = 0 if x < 0.5 dx else 1, the index shift of
// accumulateCell, particle_accumulator.cpp:78-84). Dual index u = b + 1 on a
// non-periodic axis (n + 1 dual cells), b mod n on a periodic one.
//
// Storage (per species, structure of arrays): a dual row (uy, uz) is cut into
// segments of RHGPU_FAST_SEGMENT dual cells along x; segment S = row * nseg + g
// owns the slots [base[S], base[S+1]) (slack included), the first cnt[S] hold
// its particles with their dual x index within the segment (lx, one byte).
// Two buffers per species (current, next) share the layout.
//
//   k_fast_push_deposit  one block per segment, one thread per particle:
//                        push + migration + CIC weights of the new position +
//                        boundary removal (particle_boundary_cond_hybrid.h:112-185).
//                        The field stencil and each chunk of particles are
//                        copied to shared memory with per-thread cp.async, the
//                        next chunk while the current one is processed.
//                        Particles that stay in the segment are written to the
//                        next buffer in order; their deposit records go to
//                        shared memory counting-sorted by target dual cell
//                        (stable) and are summed sequentially per (dual cell,
//                        corner, moment) in FP64, one thread per two corners
//                        and two moments. Particles that leave the segment go
//                        to the mover list.
//   k_mover_pass         the movers' CIC contributions as exact 128-bit
//                        fixed-point sums (order-independent), and their count
//                        per destination
//   k_mig_*              placement of the movers after the stayers of their
//                        destination segment, in (source segment, index) order
//   k_fast_gather        cell moments from the four row partials (+ the segment
//                        boundary partial) + the fixed-point part, then /dV and
//                        the rho clamp (particle_accumulator.cpp:319-333)
#pragma once

#include "rh_device.cuh"
#include "k_fields.cuh"
#include "k_particles.cuh"

namespace rh {

constexpr int FAST_MAX_SPECIES = 8;
constexpr int SEG = RHGPU_FAST_SEGMENT;   // dual cells per segment
struct SegBuf {
   double* a[7];        // x, y, z (cell-local), vx, vy, vz, weight: planes of one array
   long long plane;     // their distance in elements
   unsigned char* lx;   // dual x index within the segment
   int* cnt;            // particles per segment
};
struct SegSpecies {
   SegBuf cur, nxt;
   const long long* base;   // NS+1 slot offsets
};
struct FastSpecies {
   int ns;
   SegSpecies st[FAST_MAX_SPECIES];
   SpeciesDev sp[FAST_MAX_SPECIES];
};
struct FastGeom {
   int nd[3];        // dual cells per axis
   int nseg;         // segments per dual row
   long long nrows;  // dual rows
   long long NS;     // segments
};

// a particle leaving its segment: key orders the arrivals of a destination
// segment, (source segment << 32) | index in the source segment
struct Mover {
   double s[7];
   unsigned long long key;
   long long dest;   // destination segment
   int species;
   int lx;           // dual x in the destination segment | MOVER_* flags
};
constexpr int MOVER_DEPOSIT = 1 << 8;   // deposits its CIC contributions (fixed point)
constexpr int MOVER_PLACE = 1 << 9;     // is stored in the destination segment
constexpr int MOVER_AVG = 1 << 10;      // removed after its in-segment deposit: population averages only

// state of a step's migration, read back by the host once per step
struct MigCtl {
   unsigned long long nm;       // movers of the step (may exceed the list: an error)
   unsigned long long placed;   // list positions given to destinations
   unsigned over;               // bit s: arrivals of species s do not fit some segment
   int maxInc;                  // most arrivals of one destination, where above MIG_RANK
};

struct FastBufs {
   double* RP;                 // row partials: 4 planes x nrows x nx x 4
   double* RPB;                // segment-boundary partials: 4 planes x nrows x nseg x 4
   unsigned long long* MMlo;   // N x 4: a cell's four sums in one 32-byte sector
   unsigned long long* MMhi;   // N x 4
   const unsigned char* segInner;   // per segment: an obstacle (RHGPU_FLAG_INNER_PARTICLE) cell within reach
   Mover* movers;
   unsigned long long* nmovers;
   long long moverCap;
   double scaleR, scaleJ;      // 2^kR, 2^kJ
};

// b in [-n, 2n)
__host__ __device__ inline int dualU(int b, int n, int per) { return per ? (b < 0 ? b + n : (b >= n ? b - n : b)) : b + 1; }
__host__ __device__ inline int dualB(int u, int per) { return per ? u : u - 1; }
__host__ __device__ inline int halfS(double x, double dx) { return (x < (0 + 0.5) * dx) ? 0 : 1; }

// exact 128-bit fixed-point accumulation of v * scale (rounded to an integer, |.| < 2^62)
__device__ inline void add128(unsigned long long* lo, unsigned long long* hi, double v, double scale) {
   const long long iv = __double2ll_rn(v * scale);
   const unsigned long long ulo = (unsigned long long)iv;
   const unsigned long long sext = iv < 0 ? ~0ull : 0ull;
   const unsigned long long old = atomicAdd(lo, ulo);
   const unsigned long long carry = (old + ulo < old) ? 1ull : 0ull;
   const unsigned long long h = sext + carry;
   if (h) atomicAdd(hi, h);
}

__device__ inline double fixedToDouble(unsigned long long lo, unsigned long long hi, double hiScale, double loScale) {
   return __ll2double_rn((long long)hi) * hiScale + __ull2double_rn(lo) * loScale;
}

// cicWeights (particle_accumulator.cpp:68-110) with the divisions by dx done by divDx
__device__ inline void cicWeightsDx(double x, double y, double z, double wq, const GridInfo& g, double w8[8]) {
   const double dx = g.dx;
   int i = (int)floor(divDx(x, g)), j = (int)floor(divDx(y, g)), k = (int)floor(divDx(z, g));
   if (x < (i + 0.5) * dx) { --i; }
   if (y < (j + 0.5) * dx) { --j; }
   if (z < (k + 0.5) * dx) { --k; }
   ++i; ++j; ++k;
   const double x0 = (i - 1 + 0.5) * dx, y0 = (j - 1 + 0.5) * dx, z0 = (k - 1 + 0.5) * dx;
   const double w_x = divDx(x - x0, g), w_y = divDx(y - y0, g), w_z = divDx(z - z0, g);
   w8[0] = (1 - w_x) * (1 - w_y) * (1 - w_z) * wq;
   w8[1] = w_x * (1 - w_y) * (1 - w_z) * wq;
   w8[2] = (1 - w_x) * w_y * (1 - w_z) * wq;
   w8[3] = w_x * w_y * (1 - w_z) * wq;
   w8[4] = (1 - w_x) * (1 - w_y) * w_z * wq;
   w8[5] = w_x * (1 - w_y) * w_z * wq;
   w8[6] = (1 - w_x) * w_y * w_z * wq;
   w8[7] = w_x * w_y * w_z * wq;
}

// cicWeightsDx for a cell-local position in [0, dx), as every particle has
// after its migration: there floor(x / dx) = 0 (x / dx rounds below 1), so the
// dual base of each axis is the half-cell shift alone and the weights are
// those of cicWeightsDx, bit for bit
__device__ inline void cicWeightsLocal(double x, double y, double z, double wq, const GridInfo& g, double w8[8]) {
   const double dx = g.dx;
   const int i = halfS(x, dx), j = halfS(y, dx), k = halfS(z, dx);
   const double x0 = (i - 1 + 0.5) * dx, y0 = (j - 1 + 0.5) * dx, z0 = (k - 1 + 0.5) * dx;
   const double w_x = divDx(x - x0, g), w_y = divDx(y - y0, g), w_z = divDx(z - z0, g);
   w8[0] = (1 - w_x) * (1 - w_y) * (1 - w_z) * wq;
   w8[1] = w_x * (1 - w_y) * (1 - w_z) * wq;
   w8[2] = (1 - w_x) * w_y * (1 - w_z) * wq;
   w8[3] = w_x * w_y * (1 - w_z) * wq;
   w8[4] = (1 - w_x) * (1 - w_y) * w_z * wq;
   w8[5] = w_x * (1 - w_y) * w_z * wq;
   w8[6] = (1 - w_x) * w_y * w_z * wq;
   w8[7] = w_x * w_y * w_z * wq;
}

// the field stencil of one segment's cells in shared memory: local cell
// (lc, ly, lz) = global (xs0 + lc, ys0 + ly, zs0 + lz), lc in [0, SEG],
// ly, lz in {0, 1}; faceB also holds the -x / -y / -z neighbour faces
// (every x-row has the same length, so that one offset serves all but by)
template <class T>
struct SegFieldsT {
   T bx[2][2][SEG + 2];    // [lz][ly][lc + 1]
   T by[2][3][SEG + 2];    // [lz][ly + 1][lc]
   T bz[3][2][SEG + 2];    // [lz + 1][ly][lc]
   T ue[3][2][2][SEG + 2]; // [l][lz][ly][lc]
   T ep[3][2][2][SEG + 2];
};
using SegFields = SegFieldsT<double>;
constexpr int SF_ROWS_B = 4 + 6 + 6;    // x-rows of faceB components in the stencil
constexpr int SF_ROWS_C = 12;           // x-rows of one cell vector field (3 components x 2 x 2)

// one x-row of the stencil: its shared-memory start, length, first global x,
// and the global array, component and (y, z)
template <class T>
__device__ inline T* stencilRow(SegFieldsT<T>& F, const Fields& f, int r, int& len, int& dxs, const double*& arr,
                                int& l, int& dy, int& dz) {
   if (r < 4) {   // faceB x: ly, lz in {0, 1}, lc from -1
      const int lz = r >> 1, ly = r & 1;
      len = SEG + 2; dxs = -1; arr = f.faceB; l = 0; dy = ly; dz = lz;
      return &F.bx[lz][ly][0];
   }
   if (r < 10) {  // faceB y: ly from -1
      const int q = r - 4, lz = q / 3, lyp = q - 3 * lz;
      len = SEG + 1; dxs = 0; arr = f.faceB; l = 1; dy = lyp - 1; dz = lz;
      return &F.by[lz][lyp][0];
   }
   if (r < 16) {  // faceB z: lz from -1
      const int q = r - 10, lzp = q >> 1, ly = q & 1;
      len = SEG + 1; dxs = 0; arr = f.faceB; l = 2; dy = ly; dz = lzp - 1;
      return &F.bz[lzp][ly][0];
   }
   const int q = (r - 16) % SF_ROWS_C, c = q >> 2, lz = (q >> 1) & 1, ly = q & 1;
   len = SEG + 1; dxs = 0; l = c; dy = ly; dz = lz;
   if (r < 16 + SF_ROWS_C) {
      arr = f.cellUe;
      return &F.ue[c][lz][ly][0];
   }
   arr = f.cellEp;
   return &F.ep[c][lz][ly][0];
}

// the stencil in two passes: threads 0..nrows-1 describe one x-row each
// (source row or none outside a non-periodic box in y/z, first global x,
// shared-memory offset), then all threads copy the rows' elements, SF_ROW_W
// slots per row (values 0 outside a non-periodic box; the push accelerates
// only particles of cells with all neighbours, so those are never read); all
// loads of a thread are issued before its shared-memory stores
constexpr int SF_ROW_W = SEG + 2;                               // slots per row (bx rows use all)
constexpr int SF_MAX_ROWS = SF_ROWS_B + 2 * SF_ROWS_C;
struct StencilRow {
   const double* src;   // global x = 0 of the row, or nullptr (zeros)
   int dst;             // element offset of the row in the stencil
   int xs;              // global x of the row's first element
   int len;             // elements of the row
};

template <int NT, class T>
__device__ inline void stageSegRows(const GridInfo& g, const Fields& f, bool useEp, int xs0, int ys0, int zs0,
                                    SegFieldsT<T>& F, StencilRow* rows) {
   const int nrows = SF_ROWS_B + SF_ROWS_C * (useEp ? 2 : 1);
   const int tid = threadIdx.x;
   if (tid < nrows) {
      int len, dxs, l, dy, dz;
      const double* arr;
      T* dst = stencilRow(F, f, tid, len, dxs, arr, l, dy, dz);
      int y = ys0 + dy, z = zs0 + dz;
      if (g.per[1]) { if (y < 0) y += g.ny; else if (y >= g.ny) y -= g.ny; }
      if (g.per[2]) { if (z < 0) z += g.nz; else if (z >= g.nz) z -= g.nz; }
      StencilRow r;
      r.src = (y >= 0 && y < g.ny && z >= 0 && z < g.nz)
                  ? arr + (long long)l * g.N + (long long)g.nx * ((long long)y + (long long)g.ny * z)
                  : nullptr;
      r.dst = (int)(dst - (T*)&F);
      r.xs = xs0 + dxs;
      r.len = len;
      rows[tid] = r;
   }
   __syncthreads();
   constexpr int SF_PER_THREAD = (SF_MAX_ROWS * SF_ROW_W + NT - 1) / NT;
   double v[SF_PER_THREAD];
   int d[SF_PER_THREAD];
#pragma unroll
   for (int k = 0; k < SF_PER_THREAD; ++k) {
      const int e = tid + NT * k;
      const int ri = e / SF_ROW_W, c = e - ri * SF_ROW_W;
      v[k] = 0.0;
      d[k] = -1;
      if (ri >= nrows) continue;
      const StencilRow r = rows[ri];
      if (c >= r.len) continue;
      d[k] = r.dst + c;
      int x = r.xs + c;
      if (g.per[0]) { if (x < 0) x += g.nx; else if (x >= g.nx) x -= g.nx; }
      if (r.src && x >= 0 && x < g.nx) v[k] = r.src[x];
   }
   T* const base = (T*)&F;
#pragma unroll
   for (int k = 0; k < SF_PER_THREAD; ++k)
      if (d[k] >= 0) base[d[k]] = (T)v[k];
}

// x, y, z in [0, dx) over dx, as divDx: the three quotients' range is tested at
// once, by exponent (2^-500 to 2^500; zeros, negative and non-finite values fail it)
__device__ __forceinline__ void divDx3(double x, double y, double z, const GridInfo& g, double q[3]) {
   q[0] = x * g.rdx; q[1] = y * g.rdx; q[2] = z * g.rdx;
   constexpr unsigned LO = (1023u - 500u) << 20, RANGE = 1000u << 20;
   const unsigned e = max(max((unsigned)__double2hiint(q[0]) - LO, (unsigned)__double2hiint(q[1]) - LO),
                          (unsigned)__double2hiint(q[2]) - LO);
   if (e < RANGE) {
      q[0] = fma(fma(-q[0], g.dx, x), g.rdx, q[0]);
      q[1] = fma(fma(-q[1], g.dx, y), g.rdx, q[1]);
      q[2] = fma(fma(-q[2], g.dx, z), g.rdx, q[2]);
   } else {
      q[0] = x / g.dx; q[1] = y / g.dx; q[2] = z / g.dx;
   }
}

// push of one particle with the fields of cell (lc, ly, lz) of the segment's
// staged stencil, the arithmetic and order of the exact path's k_push with its
// divisions by dx as divDx; true if its speed was clamped. (i, j, k) is the
// cell, used by gravity only.
__device__ __forceinline__ bool pushStaged(const GridInfo& g, const SegFields& F, double qm, bool accelerate,
                                           const PushParams& pp, int i, int j, int k, int lc, int ly, int lz, double st[7]) {
   bool clamp = false;
   double vx = st[3], vy = st[4], vz = st[5];
   if (accelerate) {
      constexpr int SX = SEG + 2;
      const int o = (2 * lz + ly) * SX + lc;      // bx, bz, ue, ep
      const double* const bx = &F.bx[0][0][0] + o;
      const double* const by = &F.by[0][0][0] + o + lz * SX;
      const double* const bz = &F.bz[0][0][0] + o;
      const double* const ue = &F.ue[0][0][0][0] + o;
      double B[3], Ue[3], E[3], q[3];
      divDx3(st[0], st[1], st[2], g, q);
      B[0] = q[0] * bx[1] + (1.0 - q[0]) * bx[0];
      B[1] = q[1] * by[SX] + (1.0 - q[1]) * by[0];
      B[2] = q[2] * bz[2 * SX] + (1.0 - q[2]) * bz[0];
#pragma unroll
      for (int l = 0; l < 3; ++l) Ue[l] = ue[4 * SX * l];
      E[0] = B[1] * Ue[2] - B[2] * Ue[1];
      E[1] = B[2] * Ue[0] - B[0] * Ue[2];
      E[2] = B[0] * Ue[1] - B[1] * Ue[0];
      if (pp.use_ep) {
         const double* const ep = &F.ep[0][0][0][0] + o;
#pragma unroll
         for (int l = 0; l < 3; ++l) E[l] += ep[4 * SX * l];
      }
      const double dvx = qm * E[0], dvy = qm * E[1], dvz = qm * E[2];
      const double tx = qm * B[0], ty = qm * B[1], tz = qm * B[2];
      const double t2 = tx * tx + ty * ty + tz * tz;
      const double b2 = 2. / (1. + t2);
      const double sx = b2 * tx, sy = b2 * ty, sz = b2 * tz;
      const double vmx = vx + dvx, vmy = vy + dvy, vmz = vz + dvz;
      const double v0x = vmx + vmy * tz - vmz * ty;
      const double v0y = vmy + vmz * tx - vmx * tz;
      const double v0z = vmz + vmx * ty - vmy * tx;
      const double vpx = vmx + v0y * sz - v0z * sy;
      const double vpy = vmy + v0z * sx - v0x * sz;
      const double vpz = vmz + v0x * sy - v0y * sx;
      vx = vpx + dvx; vy = vpy + dvy; vz = vpz + dvz;
      if (pp.use_gravity) {
         const double xg = st[0] + blockOrigin(g.x_min, i, g.dx), yg = st[1] + blockOrigin(g.y_min, j, g.dx),
                      zg = st[2] + blockOrigin(g.z_min, k, g.dx);
         const double rr = sqrt(sq(xg) + sq(yg) + sq(zg));
         const double r3 = rr * rr * rr;
         if (r3 > 0) {
            const double s = -pp.GMdt / r3;
            vx += s * xg; vy += s * yg; vz += s * zg;
         }
      }
      const double v2 = sq(vx) + sq(vy) + sq(vz);
      if (v2 > pp.maxVi2) {
         const double norm = sqrt(pp.maxVi2 / v2);
         vx *= norm; vy *= norm; vz *= norm;
         clamp = true;
      }
   }
   st[3] = vx; st[4] = vy; st[5] = vz;
   st[0] += g.dt * vx;
   st[1] += g.dt * vy;
   st[2] += g.dt * vz;
   return clamp;
}

// the block's sums per (dual cell, corner, moment), in acc[dual * 32 + corner *
// 4 + moment] -> the segment's row partials (corner ox = 1 of each dual cell
// plus ox = 0 of the next) and, where the first dual cell's partner is in
// another segment, its boundary partial. NT threads.
template <int NT, class T>
__device__ __forceinline__ void segPartialsOut(const GridInfo& g, const FastGeom& fg, T* RP, T* RPB, const T* acc,
                                               long long row, int gseg, int u0, int u1) {
   const int tid = threadIdx.x;
   const int nx = g.nx;
   const long long nrows = fg.nrows;
#pragma unroll
   for (int e = tid; e < SEG * 16; e += NT) {
      const int dl = e >> 4, qq = (e >> 2) & 3, m = e & 3;
      const int lo = u0 + dl;   // the dual cell giving corner ox = 1 to cell x
      if (lo >= u1) continue;
      int x, hi;
      if (g.per[0]) {
         x = lo + 1 == nx ? 0 : lo + 1;
         hi = lo + 1 < u1 ? dl + 1 : (fg.nseg == 1 ? 0 : -1);
      } else {
         x = lo;
         if (x >= nx) continue;
         hi = lo + 1 < u1 ? dl + 1 : -1;
      }
      T v = acc[dl * 32 + ((1 + 2 * qq) << 2) + m];
      if (hi >= 0) v = v + acc[hi * 32 + ((2 * qq) << 2) + m];
      RP[(((long long)qq * nrows + row) * nx + x) * 4 + m] = v;
   }
   // corner ox = 0 of the first dual cell, when the cell's other dual cell is in another segment
   if (tid < 16 && (g.per[0] ? fg.nseg > 1 : gseg >= 1)) {
      const int qq = tid >> 2, m = tid & 3;
      RPB[(((long long)qq * nrows + row) * fg.nseg + gseg) * 4 + m] = acc[((2 * qq) << 2) + m];
   }
}

// one species' storage at the block's segment: its current and next x planes,
// the other planes' distances, and the dual x indices
struct SegAt {
   const double* cur;
   double* nxt;
   long long curPlane, nxtPlane;
   const unsigned char* curLx;
   unsigned char* nxtLx;
};

// k_fast_push_deposit: one thread per particle of a chunk, a warp's 32 particles
// a group of one species
constexpr int PD_T = 256, PD_VW = PD_T / 32;
static_assert(PD_VW == 8, "a dual cell's record counts per group are the bytes of a 64-bit word");
static_assert(SEG * 8 == PD_T, "the deposit sums map (dual cell, corner pair, moment pair) to one thread");
// a deposit record: w8[8], then 1, vx, vy, vz, so that the charge is one more
// product of the same sum; 14 doubles apart, so that the 16-byte accesses of
// eight lanes at any records fall on different banks
constexpr int PD_REC = 14;

// shared memory of k_fast_push_deposit (dynamic: more than the 48 KB static limit)
struct PushDepositShared {
   double rec[PD_T * PD_REC];            // deposit records of a chunk; at the end acc[SEG][32]
   double pf[7][PD_T];                // the next chunk's particles, one plane per component
   SegFields f;                           // field stencil of the segment
   SegAt at[FAST_MAX_SPECIES];
   StencilRow rows[SF_MAX_ROWS];
   alignas(8) unsigned char wd[SEG][PD_VW];   // records per (dual cell, group)
   int wcnt[PD_VW];                       // stayers per group
   int first[FAST_MAX_SPECIES + 1];       // first group of each species in the segment
   int cnt[FAST_MAX_SPECIES];             // particles of each species in the segment
   int stay[FAST_MAX_SPECIES];            // stayers of each species up to and with the chunk
};
constexpr size_t PUSH_DEPOSIT_SMEM = sizeof(PushDepositShared);
static_assert(PD_T * PD_REC >= SEG * 32, "the final sums reuse the records");

// the field stencil requested with cp.async: the stencil rows (see
// stageSegRows) with zeros outside a non-periodic box
template <int PER>
__device__ __forceinline__ void pdStage(const GridInfo& g, const Fields& f, bool useEp, PushDepositShared& sh) {
   const int nrows = SF_ROWS_B + SF_ROWS_C * (useEp ? 2 : 1);
   double* const base = (double*)&sh.f;
   for (int e = threadIdx.x; e < nrows * SF_ROW_W; e += PD_T) {
      const int ri = e / SF_ROW_W, c = e - ri * SF_ROW_W;
      const StencilRow r = sh.rows[ri];
      if (c >= r.len) continue;
      int x = r.xs + c;
      if (PER & 1) { if (x < 0) x += g.nx; else if (x >= g.nx) x -= g.nx; }
      const bool ok = r.src != nullptr && x >= 0 && x < g.nx;
      cpAsync8(base + r.dst + c, ok ? r.src + x : f.faceB, ok ? 8 : 0);
   }
}

// species of group V of the segment (groups past the last one: the last species)
template <class SH>
__device__ __forceinline__ int pdSpecies(const SH& sh, int V, int ns) {
   int s = 0;
   while (s + 1 < ns && V >= sh.first[s + 1]) ++s;
   return s;
}

// this thread's particle of the chunk that starts at group V0 requested into pf
// (its species s, index p and dual x lx; p < 0: none)
__device__ __forceinline__ void pdPrefetch(PushDepositShared& sh, int V0, int ns, int& s, int& p, int& lx) {
   const int tid = threadIdx.x, V = V0 + (tid >> 5);
   s = pdSpecies(sh, V, ns);
   p = (V - sh.first[s]) * 32 + (tid & 31);
   if (p >= sh.cnt[s]) {
      p = -1;
   } else {
      const double* q = sh.at[s].cur + p;
      const long long plane = sh.at[s].curPlane;
#pragma unroll
      for (int a = 0; a < 7; ++a, q += plane) cpAsync8(&sh.pf[a][tid], q, 8);
      lx = sh.at[s].curLx[p];
   }
   cpAsyncCommit();
}

// the CIC fraction of one axis: (x - the dual cell's lower centre) / dx, bit for
// bit that of cicWeightsLocal. The quotient needs no range test: the numerator
// is 0 or at least an ulp of dx / 2, at most dx.
__device__ __forceinline__ double cicFraction(double x, const GridInfo& g, double hdx) {
   const double r = x < hdx ? x + hdx : x - hdx;
   const double q = r * g.rdx;
   return fma(fma(-q, g.dx, r), g.rdx, q);
}

// one deposit record: the eight CIC weights (the products of cicWeightsLocal, in
// its order), then 1 and the velocity
__device__ __forceinline__ void writeRecord(double* rec, double w_x, double w_y, double w_z, double wq, double vx,
                                            double vy, double vz) {
   double2* const r = reinterpret_cast<double2*>(rec);
   r[0] = make_double2((1 - w_x) * (1 - w_y) * (1 - w_z) * wq, w_x * (1 - w_y) * (1 - w_z) * wq);
   r[1] = make_double2((1 - w_x) * w_y * (1 - w_z) * wq, w_x * w_y * (1 - w_z) * wq);
   r[2] = make_double2((1 - w_x) * (1 - w_y) * w_z * wq, w_x * (1 - w_y) * w_z * wq);
   r[3] = make_double2((1 - w_x) * w_y * w_z * wq, w_x * w_y * w_z * wq);
   r[4] = make_double2(1.0, vx);
   r[5] = make_double2(vy, vz);
}

// migration of one axis (migrateAxis); a coordinate inside [0, dx) is told by
// one unsigned comparison of its bits (negative values and NaN compare above)
__device__ __forceinline__ int migrateAxisBits(double& x, int& off, const GridInfo& g, bool& nan) {
   off = 0;
   if ((unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(g.dx)) return 0;
   nan |= isnan(x);
   return migrateAxis(x, off, g.dx, g.dx_below);
}

// EXTRA: the variant with the optional outputs (the removed in-segment deposits
// listed for the population averages, the per-cell maxVi constraint counter);
// the default instantiation carries neither.
// PER: the periodic axes (bit a = axis a), fixed at compile time; the host
// launches the instantiation that matches the grid.
//
// One block per segment; chunks of PD_T particles in storage order, species
// after species, every species starting at a group of 32 so that a warp's
// species is uniform. The particles of chunk k+1 are copied to shared memory
// (cp.async, each thread its own position) while chunk k is processed; per chunk
// two barriers order the records and the stayers. A particle leaving the segment reserves its mover
// slot before the second barrier and is written after the deposit sums, so the
// reservation's round trip overlaps the chunk's remaining work.
//
// It is bound by issue slots and the waits between them at the 32 warps per SM
// that 64 registers and 56 KB of shared memory leave (62 % of cycles issue, 59 %
// of the shared-memory wavefronts), not by memory.
// Mars run, 9.25e7 ions, 120 x 160 x 160 cells: 4.27 ms per step = 2330 GB/s of
// its 104 bytes per ion and cell; 4.33 ms with a pointer per plane; 4.62 ms with
// species packed within a chunk, eleven 8-byte accesses per record and one corner
// x four moments per thread;
// 5.35 ms with two particles per thread at 16 warps per SM.
template <int PER, bool EXTRA>
__global__ void __launch_bounds__(PD_T, 4)
k_fast_push_deposit(GridInfo gIn, Fields f, FastGeom fg, FastSpecies FS, PushParams pp, FastBufs fb,
                    double* cntd, unsigned long long* cntu, unsigned* err) {
   extern __shared__ __align__(16) unsigned char pdSmem[];
   PushDepositShared& sh = *reinterpret_cast<PushDepositShared*>(pdSmem);
   GridInfo g = gIn;
   g.per[0] = PER & 1;
   g.per[1] = (PER >> 1) & 1;
   g.per[2] = (PER >> 2) & 1;
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const unsigned below = (1u << lane) - 1u;
   const int S = (int)blockIdx.x;
   const int nseg = fg.nseg;
   const int row = S / nseg, gseg = S - row * nseg;
   const int uz = row / fg.nd[1], uy = row - uz * fg.nd[1];
   const int u0 = gseg * SEG, u1 = min(u0 + SEG, fg.nd[0]);
   const int ns = FS.ns;
   const double dx = g.dx, hdx = 0.5 * dx;
   const int xs0 = dualB(u0, g.per[0]), ys0 = dualB(uy, g.per[1]), zs0 = dualB(uz, g.per[2]);
   // no obstacle cell within one step of the segment: the obstacle test is skipped
   const bool segInner = fb.segInner[S] != 0;
   // every cell a particle of the segment can be in or reach has its neighbours in y and z
   const bool yzIn = ((PER & 2) || (ys0 >= 2 && ys0 + 2 <= g.ny - 2)) && ((PER & 4) || (zs0 >= 2 && zs0 + 2 <= g.nz - 2));

   // ---- set-up: species (warp 0), segment pointers, stencil rows
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
      const SegSpecies& SS = FS.st[tid - 32];
      const long long b = SS.base[S];
      SegAt& A = sh.at[tid - 32];
      A.cur = SS.cur.a[0] + b;
      A.nxt = SS.nxt.a[0] + b;
      A.curPlane = SS.cur.plane;
      A.nxtPlane = SS.nxt.plane;
      A.curLx = SS.cur.lx + b;
      A.nxtLx = SS.nxt.lx + b;
   }
   if (const int r = PD_T - 1 - tid; r < SF_ROWS_B + SF_ROWS_C * (pp.use_ep ? 2 : 1)) {
      int len, dxs, l, dy, dz;
      const double* arr;
      double* dst = stencilRow(sh.f, f, r, len, dxs, arr, l, dy, dz);
      int y = ys0 + dy, z = zs0 + dz;
      if (PER & 2) { if (y < 0) y += g.ny; else if (y >= g.ny) y -= g.ny; }
      if (PER & 4) { if (z < 0) z += g.nz; else if (z >= g.nz) z -= g.nz; }
      StencilRow sr;
      sr.src = (y >= 0 && y < g.ny && z >= 0 && z < g.nz)
                   ? arr + (long long)l * g.N + (long long)g.nx * ((long long)y + (long long)g.ny * z)
                   : nullptr;
      sr.dst = (int)(dst - (double*)&sh.f);
      sr.xs = xs0 + dxs;
      sr.len = len;
      sh.rows[r] = sr;
   }
   __syncthreads();
   const int groups = sh.first[ns];
   int sn = 0, pn = -1, lxn = 0;   // the prefetched particle's species, index and dual x
   pdPrefetch(sh, 0, ns, sn, pn, lxn);
   pdStage<PER>(g, f, pp.use_ep, sh);
   cpAsyncCommit();
   cpAsyncWaitAll();
   __syncthreads();

   // this thread's sums: two corners of one dual cell, two moments (charge and Jx, or Jy and Jz)
   const int myDual = tid >> 3, myPair = (tid >> 1) & 3, myHalf = tid & 1;
   double a00 = 0.0, a01 = 0.0, a10 = 0.0, a11 = 0.0;

   for (int V0 = 0; V0 < groups; V0 += PD_VW) {
      double st[7];
      int duv = 0, dyz = 0, mflags = 0, rrank = 0;
      bool stay = false, rec = false, clamp = false;
      if (V0 > 0) cpAsyncWaitAll();   // this thread's copies of the chunk
      const int s = sn, p = pn;
      if (p >= 0) {
#pragma unroll
         for (int a = 0; a < 7; ++a) st[a] = sh.pf[a][tid];
         const int lu = lxn;
         const int gx = st[0] < hdx ? 0 : 1, gy = st[1] < hdx ? 0 : 1, gz = st[2] < hdx ? 0 : 1;
         const int lc = lu + 1 - gx, ly = 1 - gy, lz = 1 - gz;
         const int ci = xs0 + lc, cj = ys0 + ly, ck = zs0 + lz;   // not wrapped (periodic axes: up to n)
         bool accelerate = FS.sp[s].accelerate && !pp.useIFT && ((PER & 1) || (unsigned)(ci - 1) < (unsigned)(g.nx - 2));
         if (!yzIn)
            accelerate = accelerate && ((PER & 2) || (unsigned)(cj - 1) < (unsigned)(g.ny - 2)) &&
                         ((PER & 4) || (unsigned)(ck - 1) < (unsigned)(g.nz - 2));
         const int wi = (PER & 1) && ci >= g.nx ? ci - g.nx : ci, wj = (PER & 2) && cj >= g.ny ? cj - g.ny : cj,
                   wk = (PER & 4) && ck >= g.nz ? ck - g.nz : ck;
         clamp = pushStaged(g, sh.f, FS.sp[s].qmideltT2, accelerate, pp, wi, wj, wk, lc, ly, lz, st);
         if (EXTRA) gridCountAtomic(f, GC_CELL_MAX_VI, g.N, cidx(g, wi, wj, wk), clamp);
         int ox, oy, oz;
         bool nan = false;
         int bad = migrateAxisBits(st[0], ox, g, nan);
         bad |= migrateAxisBits(st[1], oy, g, nan);
         bad |= migrateAxisBits(st[2], oz, g, nan);
         if (nan) raiseError(err, RHGPU_DEVERR_NAN_PARTICLE);
         // target cell: inside the box, and with all its neighbours
         const int ti = ci + ox, tj = cj + oy, tk = ck + oz;
         bool inside = !bad && ((PER & 1) || (unsigned)ti < (unsigned)g.nx);
         bool all = (PER & 1) || (unsigned)(ti - 1) < (unsigned)(g.nx - 2);
         if (!yzIn) {
            inside = inside && ((PER & 2) || (unsigned)tj < (unsigned)g.ny) && ((PER & 4) || (unsigned)tk < (unsigned)g.nz);
            all = all && ((PER & 2) || (unsigned)(tj - 1) < (unsigned)(g.ny - 2)) &&
                  ((PER & 4) || (unsigned)(tk - 1) < (unsigned)(g.nz - 2));
         }
         bool removed = !inside || !all;
         if (removed) {
            const double ke = st[6] * (sq(st[3]) + sq(st[4]) + sq(st[5]));
            double* const q = removedSums(cntd, S, s);
            atomicAdd(&q[0], st[6]);
            atomicAdd(&q[1], ke);
         }
         if (inside) {
            // the new dual cell relative to the segment's first, and to its row
            int du = lu + ox + (st[0] < hdx ? 0 : 1) - gx;
            const int dy = oy + (st[1] < hdx ? 0 : 1) - gy, dz = oz + (st[2] < hdx ? 0 : 1) - gz;
            if ((PER & 1) && nseg == 1) {
               if (du < 0) du += fg.nd[0];
               else if (du >= fg.nd[0]) du -= fg.nd[0];
            }
            const bool inSeg = dy == 0 && dz == 0 && (unsigned)du < (unsigned)(u1 - u0);
            duv = du;
            dyz = (dy + 2) | ((dz + 2) << 3);
            if (FS.sp[s].accumulate) {
               rec = inSeg;   // its CIC weights are formed just before the record is written
               if (!inSeg) mflags = MOVER_DEPOSIT;   // deposited by k_mover_pass
            }
            if (segInner && !removed) {
               int xi = ti, xj = tj, xk = tk;
               wrapc(xi, g.nx, g.per[0]); wrapc(xj, g.ny, g.per[1]); wrapc(xk, g.nz, g.per[2]);
               if (f.flags[cidx(g, xi, xj, xk)] & RHGPU_FLAG_INNER_PARTICLE) {
                  const double xp = blockOrigin(g.x_min, xi, dx) + st[0];
                  const double yp = blockOrigin(g.y_min, xj, dx) + st[1];
                  const double zp = blockOrigin(g.z_min, xk, dx) + st[2];
                  if (sq(xp) + sq(yp) + sq(zp) < FS.sp[s].R2obs) {
                     removed = true;
                     const double ke = st[6] * (sq(st[3]) + sq(st[4]) + sq(st[5]));
                     double* const q = removedSums(cntd, S, s);
                     atomicAdd(&q[2], st[6]);
                     atomicAdd(&q[3], ke);
                  }
               }
            }
            if (!removed) {
               stay = inSeg;
               if (!inSeg) mflags |= MOVER_PLACE;
            } else if (EXTRA && rec && pp.avgList) {
               mflags |= MOVER_AVG;   // population averages: its in-segment deposit is listed
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
      if (V0 + PD_VW < groups) pdPrefetch(sh, V0 + PD_VW, ns, sn, pn, lxn);
      // (unconditional: the arithmetic fills the waits of the scan below)
      const double w_x = cicFraction(st[0], g, hdx), w_y = cicFraction(st[1], g, hdx), w_z = cicFraction(st[2], g, hdx);
      // every warp, per dual cell (lane): the first sorted record of the dual cell
      // (bin); the group counts of dual cell `lane` are bytes (each at most 32),
      // byte sums by one multiply per 32-bit half
      const uint2 c8 = *reinterpret_cast<const uint2*>(&sh.wd[lane][0]);
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
         writeRecord(sh.rec + recPos * PD_REC, w_x, w_y, w_z, st[6] * FS.sp[s].q, st[3], st[4], st[5]);
      }
      __syncthreads();
      if (stay) {
         double* q = sh.at[s].nxt + slot;
         const long long plane = sh.at[s].nxtPlane;
#pragma unroll
         for (int a = 0; a < 7; ++a, q += plane) *q = st[a];
         sh.at[s].nxtLx[slot] = (unsigned char)duv;
      }
      // ---- this thread's sums, records in list order ----------------------------------------
#pragma unroll 2
      for (int r = sumLo; r < sumHi; ++r) {
         const double2* const rr = reinterpret_cast<const double2*>(sh.rec + r * PD_REC);
         const double2 w = rr[myPair], u = rr[4 + myHalf];
         a00 += w.x * u.x;
         a01 += w.x * u.y;
         a10 += w.y * u.x;
         a11 += w.y * u.y;
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
      Mover& M = fb.movers[m];
#pragma unroll
      for (int a = 0; a < 7; ++a) M.s[a] = st[a];
      M.key = ((unsigned long long)S << 32) | (unsigned long long)p;
      const int gd = vx / SEG;
      M.dest = ((long long)vy + (long long)fg.nd[1] * vz) * nseg + gd;
      M.species = s;
      M.lx = (vx - gd * SEG) | mflags;
      // no barrier here: the next chunk's first barrier orders the reads of rec
      // and wd before their next writes
   }

   // ---- outputs: stayer counts, row partials, segment-boundary partial ---------------------
   __syncthreads();
   if (tid < ns) FS.st[tid].nxt.cnt[S] = sh.stay[tid];
   {
      double* const q = sh.rec + myDual * 32 + myPair * 8 + myHalf * 2;
      q[0] = a00; q[1] = a01; q[4] = a10; q[5] = a11;
   }
   __syncthreads();
   segPartialsOut<PD_T>(g, fg, fb.RP, fb.RPB, sh.rec, row, gseg, u0, u1);
}

// corner o's four deposits (charge, current) of one mover: the weight products
// of cicWeightsLocal, in its order
__device__ __forceinline__ void moverTerms(const GridInfo& g, const FastSpecies& FS, const Mover& M, int o, double t[4]) {
   const double dx = g.dx, x = M.s[0], y = M.s[1], z = M.s[2];
   const double x0 = (halfS(x, dx) - 1 + 0.5) * dx, y0 = (halfS(y, dx) - 1 + 0.5) * dx, z0 = (halfS(z, dx) - 1 + 0.5) * dx;
   const double w_x = divDx(x - x0, g), w_y = divDx(y - y0, g), w_z = divDx(z - z0, g);
   const double fx = o & 1 ? w_x : 1 - w_x, fy = o & 2 ? w_y : 1 - w_y, fz = o & 4 ? w_z : 1 - w_z;
   t[0] = fx * fy * fz * (M.s[6] * FS.sp[M.species].q);
   for (int l = 0; l < 3; ++l) t[1 + l] = t[0] * M.s[3 + l];
}

// One pass over the movers: the contributions of those whose flags meet `need`
// (species in smask) as exact fixed-point sums into lo / hi, and, with inc, the
// arrivals counted per destination, rank[m] being a mover's place in that count
// (in any order; k_mig_place orders them).
//
// A warp takes four movers, one lane per corner; the 16 x 8 terms go through
// shared memory so that each of four atomics of the warp covers one mover, the
// four sums of a cell on adjacent lanes (one 32-byte sector, two for corners
// adjacent in x). The pass is bound by those returning atomics: one thread per
// mover with its 32 atomics in a row over four planes took 0.30 ms for 2.9e6
// movers of the Mars run and 30-39 us for the few thousand of a 32^3 box, where
// the chain of one thread is all there is.
constexpr int MP_THREADS = 256;
template <class MV, class SET>
__global__ void __launch_bounds__(MP_THREADS)
k_mover_pass(GridInfo g, FastGeom fg, SET FS, const MV* mv, const MigCtl* ctl, long long cap, int need, unsigned smask,
             unsigned long long* lo, unsigned long long* hi, double scaleR, double scaleJ, int* inc, unsigned* rank) {
   __shared__ long long term[MP_THREADS / 32][32][4];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, o = lane & 7;
   const long long nm = (long long)ctl->nm;
   if (nm > cap) return;   // more movers than the list holds: the host ends the step with an error
   const long long step = (long long)gridDim.x * (MP_THREADS / 8);
   for (long long m0 = ((long long)blockIdx.x * (MP_THREADS / 32) + warp) * 4; m0 < nm; m0 += step) {
      const long long m = m0 + (lane >> 3);
      const MV& M = mv[m < nm ? m : m0];
      const int flags = m < nm ? M.lx : 0;
      const int dest = (int)M.dest;
      if (inc && o == 0 && (flags & MOVER_PLACE)) rank[m] = (unsigned)atomicAdd(&inc[M.species * (int)fg.NS + dest], 1);
      int dc = -1;
      if ((flags & need) && ((smask >> M.species) & 1u)) {
         const int row = dest / fg.nseg;
         const int vx = (dest - row * fg.nseg) * SEG + (flags & 0xff);
         const int vz = row / fg.nd[1], vy = row - vz * fg.nd[1];
         int cx = dualB(vx, g.per[0]) + (o & 1), cy = dualB(vy, g.per[1]) + ((o >> 1) & 1), cz = dualB(vz, g.per[2]) + (o >> 2);
         if (wrapc(cx, g.nx, g.per[0]) && wrapc(cy, g.ny, g.per[1]) && wrapc(cz, g.nz, g.per[2])) {
            dc = (int)cidx(g, cx, cy, cz);
            double t[4];
            moverTerms(g, FS, M, o, t);
            term[warp][lane][0] = __double2ll_rn(t[0] * scaleR);
#pragma unroll
            for (int l = 1; l < 4; ++l) term[warp][lane][l] = __double2ll_rn(t[l] * scaleJ);
         }
      }
      __syncwarp();
      unsigned long long old[4];
      long long iv[4], at[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
         const int src = 8 * r + (lane >> 2);
         const int d = __shfl_sync(0xffffffffu, dc, src);
         at[r] = d < 0 ? -1 : 4LL * d + (lane & 3);
         if (d >= 0) {
            iv[r] = term[warp][src][lane & 3];
            old[r] = atomicAdd(&lo[at[r]], (unsigned long long)iv[r]);
         }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
         if (at[r] < 0) continue;
         const unsigned long long h = (iv[r] < 0 ? ~0ull : 0ull) + (old[r] + (unsigned long long)iv[r] < old[r] ? 1ull : 0ull);
         if (h) atomicAdd(&hi[at[r]], h);
      }
      __syncwarp();
   }
}

// Two threads per cell, two moments each (charge and Jx, Jy and Jz): a cell's
// four row partials and fixed-point sums are one vector per thread, consecutive
// over a warp's 16 cells. The fixed-point sums are cleared after the gather by a
// fill (fixedClear), not here: a kernel that reads and writes them in place
// moves the same bytes but took 0.13 to 1.08 ms on the Mars run (3.07e6 cells,
// FP32 and FP64 form), depending on its vector width and resident warps, where
// the gather and the fill together take 0.13 (FP32) and 0.15 (FP64).
constexpr int GA_CELLS = 64;   // cells of a block of 128 threads, consecutive in x
// the blocks of a row and the rows share the launch's x axis: its y axis ends at
// 65535 blocks, and ny may be more
inline dim3 gatherGrid(const GridInfo& g) { return dim3((g.nx + GA_CELLS - 1) / GA_CELLS * g.ny, 1, g.nz); }
#define RH_GATHER_PROLOGUE                                        \
   const int nxb = (g.nx + GA_CELLS - 1) / GA_CELLS;              \
   const int j = (int)blockIdx.x / nxb, k = blockIdx.z;           \
   const int i = ((int)blockIdx.x - j * nxb) * GA_CELLS + (threadIdx.x >> 1); \
   const int h = threadIdx.x & 1;                                 \
   if (i >= g.nx) return;                                         \
   const long long n = cidx(g, i, j, k);                          \
   const long long N = g.N;

template <class T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

// moments 2h and 2h + 1 of cell (i, j, k): the four row partials, each with its
// segment's boundary partial where the cell's other dual cell is in another
// segment, and the fixed-point part (scales hi/lo S0, S1). A cell that no mover
// touched adds +0.0, which changes no sum here (a sum of products started at
// +0.0 is never -0.0).
template <class T, class B>
__device__ __forceinline__ double2 gatherMoments(const GridInfo& g, const FastGeom& fg, const B& fb, int i, int j, int k,
                                                 int h, long long n, double hiS0, double loS0, double hiS1, double loS1) {
   using V = typename Vec2<T>::type;
   const bool bnd = g.per[0] ? (fg.nseg > 1 && i % SEG == 0) : ((i + 1) % SEG == 0);
   const int gb = g.per[0] ? i / SEG : (i + 1) / SEG;
   V r[4], rb[4];
#pragma unroll
   for (int qq = 0; qq < 4; ++qq) {
      const int uyy = dualU(j - (qq & 1), g.ny, g.per[1]);
      const int uzz = dualU(k - (qq >> 1), g.nz, g.per[2]);
      const long long row = (long long)qq * fg.nrows + uyy + (long long)fg.nd[1] * uzz;
      r[qq] = reinterpret_cast<const V*>(fb.RP)[(row * g.nx + i) * 2 + h];
      if (bnd) rb[qq] = reinterpret_cast<const V*>(fb.RPB)[(row * fg.nseg + gb) * 2 + h];
   }
   const ulonglong2 lo = reinterpret_cast<const ulonglong2*>(fb.MMlo)[2 * n + h];
   const ulonglong2 hi = reinterpret_cast<const ulonglong2*>(fb.MMhi)[2 * n + h];
   double2 v = make_double2(0.0, 0.0);
#pragma unroll
   for (int qq = 0; qq < 4; ++qq) {
      if (bnd) { r[qq].x = r[qq].x + rb[qq].x; r[qq].y = r[qq].y + rb[qq].y; }
      v.x = qq == 0 ? (double)r[0].x : v.x + (double)r[qq].x;
      v.y = qq == 0 ? (double)r[0].y : v.y + (double)r[qq].y;
   }
   v.x += fixedToDouble(lo.x, hi.x, hiS0, loS0);
   v.y += fixedToDouble(lo.y, hi.y, hiS1, loS1);
   return v;
}

// destination moments: gatherMoments, then /dV and the rho clamp
template <bool GC>   // GC: also count the rho clamp per cell (grid counters on)
__global__ void __launch_bounds__(2 * GA_CELLS)
k_fast_gather(GridInfo g, Fields f, FastGeom fg, FastBufs fb, double hiR, double loR, double hiJ, double loJ,
              double minRho, unsigned long long* cnt) {
   RH_GATHER_PROLOGUE
   double2 v = gatherMoments<double>(g, fg, fb, i, j, k, h, n, h ? hiJ : hiR, h ? loJ : loR, hiJ, loJ);
   v.x /= g.dV;
   v.y /= g.dV;
   const bool clamp = h == 0 && v.x < minRho;
   if (clamp) v.x = minRho;
   countIf(clamp, &cnt[CNT_MIN_CELL_RHO]);
   if (GC) gridCount(f, GC_CELL_MIN_RHOQI, N, n, clamp);
   (h ? f.cellJi + N : f.cellRho)[n] = v.x;
   (h ? f.cellJi + 2 * N : f.cellJi)[n] = v.y;
}

// ---- mover placement ------------------------------------------------------------------------
// The arrivals of a destination (species, segment) bucket are stored after its
// stayers in the order of their mover keys (source segment, index in it). Each
// bucket's arrivals are listed together (k_mig_buckets gives every bucket a
// stretch of the list, in whatever order the buckets come, and k_mig_list fills
// it), and a mover's place is the number of smaller keys in its bucket, which
// k_mig_place counts, one thread per list position, so that a warp reads the
// same one or two buckets. The three kernels do nothing when the step needs the
// host (no room in a segment, or a bucket above MIG_RANK arrivals), which reads
// MigCtl after it has launched the rest of the step and then relays out, orders
// the large buckets one block each (k_mig_order_large) or, past MIG_LARGE, all
// movers by two radix sorts (by key, then stably by bucket), and places.
// (Counts, a scan over all buckets, a second counting pass, one thread ordering
// each bucket and two host round trips in between took 83-93 us for the 32^3 box
// and 0.26 ms for the Mars run.)
constexpr int MIG_RANK = 256;     // arrivals of a bucket whose order is found by counting
constexpr int MIG_LARGE = 2048;   // arrivals one block orders in shared memory (k_mig_order_large)

// every bucket with arrivals: its stretch of the list (one reservation per
// warp), whether its segment has room, and the size of the buckets above MIG_RANK
template <class SET>
__global__ void k_mig_buckets(SET FS, int NS, const int* inc, long long* off, MigCtl* ctl) {
   const int b = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
   const int k = b < FS.ns * NS ? inc[b] : 0;
   int x = k;
#pragma unroll
   for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
   }
   unsigned long long base = 0;
   if (lane == 31 && x > 0) base = atomicAdd(&ctl->placed, (unsigned long long)x);
   base = __shfl_sync(0xffffffffu, base, 31);
   if (k == 0) return;
   off[b] = (long long)base + (x - k);
   const int s = b / NS, S = b - s * NS;
   if (FS.st[s].base[S] + FS.st[s].nxt.cnt[S] + k > FS.st[s].base[S + 1]) atomicOr(&ctl->over, 1u << s);
   if (k > MIG_RANK) atomicMax(&ctl->maxInc, k);
}
// the step needs the host before its movers can be placed
__device__ __forceinline__ bool migHeld(const MigCtl* ctl, long long cap, int force) {
   return (long long)ctl->nm > cap || (!force && (ctl->over != 0 || ctl->maxInc > MIG_RANK));
}
template <class MV>
__global__ void k_mig_list(const MV* mv, const MigCtl* ctl, long long cap, int force, int NS, const long long* off,
                           const unsigned* rank, unsigned long long* klist, unsigned* vlist) {
   if (migHeld(ctl, cap, force)) return;
   const long long nm = (long long)ctl->nm;
   for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nm; t += (long long)gridDim.x * blockDim.x) {
      if (!(mv[t].lx & MOVER_PLACE)) continue;
      const long long q = off[mv[t].species * NS + (int)mv[t].dest] + rank[t];
      klist[q] = mv[t].key;
      vlist[q] = (unsigned)t;
   }
}
// one mover into a slot of its destination's next buffer
__device__ __forceinline__ void placeMover(const SegSpecies& SS, long long slot, const Mover& M) {
#pragma unroll
   for (int e = 0; e < 7; ++e) SS.nxt.a[e][slot] = M.s[e];
   SS.nxt.lx[slot] = (unsigned char)(M.lx & 0xff);
}
template <class MV, class SET>
__global__ void k_mig_place(SET FS, const MV* mv, const MigCtl* ctl, long long cap, int force, int NS, const int* inc,
                            const long long* off, const unsigned long long* klist, const unsigned* vlist) {
   if (migHeld(ctl, cap, force)) return;
   const long long n = (long long)ctl->placed;
   for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
      const unsigned t = vlist[q];
      const MV& M = mv[t];
      const int S = (int)M.dest, b = M.species * NS + S;
      const int k = inc[b];
      const long long first = off[b];
      long long before = q - first;   // a bucket above MIG_RANK is in order already
      if (k <= MIG_RANK) {
         const unsigned long long key = klist[q];
         before = 0;
         for (int j = 0; j < k; ++j) {
            const unsigned long long kj = klist[first + j];
            before += kj < key || (kj == key && vlist[first + j] < t) ? 1 : 0;
         }
      }
      const auto& SS = FS.st[M.species];
      placeMover(SS, SS.base[S] + SS.nxt.cnt[S] + before, M);
   }
}
// the arrivals added to the segments' counts, and cleared for the next step
template <class SET>
__global__ void k_mig_counts(SET FS, const MigCtl* ctl, long long cap, int force, int NS, int* inc) {
   if (migHeld(ctl, cap, force)) return;
   const int b = blockIdx.x * blockDim.x + threadIdx.x;
   if (b >= FS.ns * NS || inc[b] == 0) return;
   FS.st[b / NS].nxt.cnt[b % NS] += inc[b];
   inc[b] = 0;
}
// whether every species has room for its arrivals (after a relayout)
template <class SET>
__global__ void k_mig_check(SET FS, int NS, const int* inc, MigCtl* ctl) {
   const int b = blockIdx.x * blockDim.x + threadIdx.x;
   if (b >= FS.ns * NS || inc[b] == 0) return;
   const int s = b / NS, S = b - s * NS;
   if (FS.st[s].base[S] + FS.st[s].nxt.cnt[S] + inc[b] > FS.st[s].base[S + 1]) atomicOr(&ctl->over, 1u << s);
}

// the buckets with more than MIG_RANK arrivals, appended to large[] (count in *nlarge)
__global__ void k_mig_large_list(const int* inc, long long nb, unsigned* large, int* nlarge);

// each bucket of large[] (at most MIG_LARGE arrivals) ordered by one block: its
// stretch of the list sorted bitonically by (key, mover index) in shared memory
constexpr int MIG_LARGE_THREADS = 256;
__global__ void __launch_bounds__(MIG_LARGE_THREADS) k_mig_order_large(const int* inc, const long long* off,
                                                                        unsigned long long* klist, unsigned* vlist,
                                                                        const unsigned* large, const int* nlarge);

// the radix order: sort keys of every mover (bucket nb: not placed), and mover
// order[q] to slot q - off[bucket] after its bucket's stayers
template <class MV>
__global__ void k_mig_sort_keys(const MV* mv, long long n, long long NS, long long nb, unsigned long long* key,
                                unsigned* val, unsigned* bkt) {
   const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= n) return;
   key[t] = mv[t].key;
   val[t] = (unsigned)t;
   bkt[t] = (mv[t].lx & MOVER_PLACE) ? (unsigned)((long long)mv[t].species * NS + mv[t].dest) : (unsigned)nb;
}
template <class MV, class SET>
__global__ void k_mig_place_order(SET FS, int NS, long long nb, const MV* mv, const unsigned* order, const unsigned* bkt,
                                  const long long* off, long long n) {
   const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
   if (q >= n) return;
   const long long b = bkt[q];
   if (b >= nb) return;
   const int s = (int)b / NS, S = (int)b - s * NS;
   const auto& SS = FS.st[s];
   placeMover(SS, SS.base[S] + SS.nxt.cnt[S] + (q - off[b]), mv[order[q]]);
}

// ---- upload / download / relayout support -----------------------------------------------------
// segment and dual x (in the segment) of each uploaded particle (records grouped by cell)
__global__ void k_fast_seg_of(GridInfo g, FastGeom fg, const double* aos, const int* pcell, long long n,
                              unsigned* key, unsigned char* lx);
// for keys sorted ascending: first[k] = first position with key >= k, k in [0, nkeys]
// (every k written exactly once, no atomics)
__global__ void k_sorted_bounds(const unsigned* key, long long n, long long nkeys, long long* first);
// counts from the bounds
__global__ void k_bounds_counts(const long long* first, long long nkeys, int* cnt);
// segment capacity with slack: c + max(32, c/4); entry NS is 0 (for the scan's total)
__global__ void k_fast_capacity(long long NS, const int* cnt, const int* extra, long long* cap);
// sorted upload records -> segment slots
__global__ void k_fast_scatter_sorted(const double* aos, const unsigned char* lxIn, const unsigned* key,
                                      const unsigned* idx, long long n, const long long* first, SegBuf B,
                                      const long long* base);
// one block per segment: cell key and slot of every particle, in storage order
__global__ void k_fast_cell_keys(GridInfo g, FastGeom fg, SegBuf B, const long long* base, const long long* first,
                                 unsigned* key, unsigned long long* slots);
__global__ void k_fast_gather_records(SegBuf B, const unsigned long long* slots, const unsigned* idx, long long n,
                                      double* aos);
// one block per segment: copy the particles of a segment to another layout
__global__ void k_fast_relayout(SegBuf from, const long long* fromBase, SegBuf to, const long long* toBase);
// one block per segment: largest |weight|
// (non-negative doubles order like their bit patterns; one atomic per block)
__global__ void k_fast_max_abs_w(SegBuf B, const long long* base, unsigned long long* out);

}  // namespace rh
