// Definitions of the kernels declared in k_fields.cuh (each declaration there says
// what its kernel does); the template kernels stay in the header.
#include "k_fields.cuh"

namespace rh {

__constant__ NeumannTables c_neu;

cudaError_t setNeumannTables(const NeumannTables& t) { return cudaMemcpyToSymbol(c_neu, &t, sizeof t); }

#define RH_C2N(dst, src, off)                                                                  \
   dst[off + n] = 0.125 * (src[off + c000] + src[off + c001] + src[off + c010] + src[off + c100] + \
                           src[off + c011] + src[off + c110] + src[off + c101] + src[off + c111]);

__global__ void k_face2cell(GridInfo g, Fields f) {
   RH_CELL_PROLOGUE
   if (!allNb(g, i, j, k)) return;
   const double* fb = f.faceB;
   f.cellB[0 * N + n] = 0.5 * (fb[0 * N + n] + fb[0 * N + nbr(g, i, j, k, -1, 0, 0)]);
   f.cellB[1 * N + n] = 0.5 * (fb[1 * N + n] + fb[1 * N + nbr(g, i, j, k, 0, -1, 0)]);
   f.cellB[2 * N + n] = 0.5 * (fb[2 * N + n] + fb[2 * N + nbr(g, i, j, k, 0, 0, -1)]);
}

__global__ void k_ext_cell_neumann3(GridInfo g, double* a, const int* ext, int next) {
   const int e = blockIdx.x * blockDim.x + threadIdx.x;
   if (e >= next) return;
   const int c = ext[e];
   int i, j, k;
   extCellIJK(g, c, i, j, k);
   const long long N = g.N, n = c;
   const int m = missingMask(g, i, j, k);
   const signed char* o = c_neu.cellSrc[m];
   const long long s = nbr(g, i, j, k, o[0], o[1], o[2]);
   if (s < 0) return;
   for (int l = 0; l < 3; ++l) a[l * N + n] = a[l * N + s];
}

__global__ void k_cell2node3(GridInfo g, const double* src, double* dst) {
   RH_CELL_PROLOGUE
   if (!plusOk(g, i, j, k)) return;
   const long long c000 = n, c001 = nbr(g, i, j, k, 0, 0, 1), c010 = nbr(g, i, j, k, 0, 1, 0),
                   c100 = nbr(g, i, j, k, 1, 0, 0), c011 = nbr(g, i, j, k, 0, 1, 1),
                   c110 = nbr(g, i, j, k, 1, 1, 0), c101 = nbr(g, i, j, k, 1, 0, 1),
                   c111 = nbr(g, i, j, k, 1, 1, 1);
   for (int l = 0; l < 3; ++l) { RH_C2N(dst, src, l * N) }
}
#undef RH_C2N

__global__ void k_node2cell3(GridInfo g, const double* src, double* dst) {
   RH_CELL_PROLOGUE
   if (!allNb(g, i, j, k)) return;
   const long long a0 = n, a1 = nbr(g, i, j, k, -1, 0, 0), a2 = nbr(g, i, j, k, -1, -1, 0),
                   a3 = nbr(g, i, j, k, 0, -1, 0), a4 = nbr(g, i, j, k, 0, 0, -1),
                   a5 = nbr(g, i, j, k, 0, -1, -1), a6 = nbr(g, i, j, k, -1, 0, -1),
                   a7 = nbr(g, i, j, k, -1, -1, -1);
   for (int l = 0; l < 3; ++l) {
      const long long o = l * N;
      dst[o + n] = 0.125 * (src[o + a0] + src[o + a1] + src[o + a2] + src[o + a3] + src[o + a4] +
                            src[o + a5] + src[o + a6] + src[o + a7]);
   }
}

// the 27 neighbours in the order of the sum, each axis 0, 1, 2 for -1, 0, +1
__device__ constexpr signed char NODE_AVG_ORDER[27][3] = {
   {1,1,1},{1,1,0},{0,1,1},{1,2,1},{2,1,1},{1,0,1},{1,1,2},{0,1,0},{1,0,0},{1,2,0},{2,1,0},
   {0,0,1},{0,2,1},{2,2,1},{2,0,1},{0,1,2},{1,2,2},{2,1,2},{1,0,2},{0,0,2},{0,2,2},{2,0,2},
   {2,2,2},{0,0,0},{0,2,0},{2,0,0},{2,2,0}};

// (61 x 83 x 70 nodes: 47 us with the offsets formed once per node and constant
// coefficients; 180 us with every neighbour's index formed per component and the
// coefficients gathered into an array.)
__global__ void __launch_bounds__(128) k_node_avg(GridInfo g, const double* old, double* out, FieldParams fp) {
   RH_CELL_PROLOGUE
   if (!plusOk(g, i, j, k)) return;
   const double initVal = 1.7976931348623157e308;
   // the three coordinates per axis as index offsets (3 N fits an int), and
   // whether the lower ones exist (the upper ones do)
   const bool lox = xNeg(g, i), loy = yNeg(g, j), loz = zNeg(g, k);
   const int sy = g.nx, sz = g.nx * g.ny;
   const int ox[3] = {i > 0 ? i - 1 : g.nx - 1, i, i + 1 < g.nx ? i + 1 : 0};
   const int oy[3] = {sy * (j > 0 ? j - 1 : g.ny - 1), sy * j, sy * (j + 1 < g.ny ? j + 1 : 0)};
   const int oz[3] = {sz * (k > 0 ? k - 1 : g.nz - 1), sz * k, sz * (k + 1 < g.nz ? k + 1 : 0)};
#pragma unroll 1
   for (int l = 0; l < 3; ++l) {
      const double* const src = old + l * N;
      double v[27];
      bool marked = false;
#pragma unroll
      for (int q = 0; q < 27; ++q) {
         const int X = NODE_AVG_ORDER[q][0], Y = NODE_AVG_ORDER[q][1], Z = NODE_AVG_ORDER[q][2];
         const bool ok = (X > 0 || lox) && (Y > 0 || loy) && (Z > 0 || loz);
         v[q] = ok ? src[ox[X] + oy[Y] + oz[Z]] : ((X == 0 && Y == 0 && Z == 0 && l == 0) ? initVal : 0.0);
         marked = marked || v[q] == initVal;
      }
      double s = 0.0;
      if (!marked) {
#pragma unroll
         for (int q = 0; q < 27; ++q) {
            const double t = fp.gauss[(NODE_AVG_ORDER[q][0] != 1) + (NODE_AVG_ORDER[q][1] != 1) + (NODE_AVG_ORDER[q][2] != 1)] * v[q];
            s = q == 0 ? t : s + t;
         }
      } else {   // marked neighbours are left out, the other coefficients normalised
         double Cs = 0.0;
#pragma unroll
         for (int q = 0; q < 27; ++q) {
            const double c = v[q] == initVal ? 0.0 : fp.gauss[(NODE_AVG_ORDER[q][0] != 1) + (NODE_AVG_ORDER[q][1] != 1) + (NODE_AVG_ORDER[q][2] != 1)];
            Cs = q == 0 ? c : Cs + c;
         }
#pragma unroll
         for (int q = 0; q < 27; ++q) {
            const bool out = v[q] == initVal;
            double c = out ? 0.0 : fp.gauss[(NODE_AVG_ORDER[q][0] != 1) + (NODE_AVG_ORDER[q][1] != 1) + (NODE_AVG_ORDER[q][2] != 1)];
            if (Cs > 0.0) c /= Cs;
            const double t = c * (out ? 0.0 : v[q]);
            s = q == 0 ? t : s + t;
         }
      }
      out[l * N + n] = s;
   }
}

__global__ void k_faraday(GridInfo g, Fields f) {
   RH_CELL_PROLOGUE
   bool doX = true, doY = true, doZ = true;
   if (!allNb(g, i, j, k)) {
      if (!plusOk(g, i, j, k)) return;
      if (!xNeg(g, i)) { doY = doZ = false; }
      if (!yNeg(g, j)) { doX = doZ = false; }
      if (!zNeg(g, k)) { doX = doY = false; }
   }
   const double* E = f.nodeE;
   const double dx = g.dx, dt = g.dt;
   if (doX) {
      const long long s5 = nbr(g, i, j, k, 0, -1, 0), s6 = nbr(g, i, j, k, 0, -1, -1), s7 = nbr(g, i, j, k, 0, 0, -1);
      const double n5y = E[1 * N + s5], n5z = E[2 * N + s5], n6y = E[1 * N + s6], n6z = E[2 * N + s6];
      const double n7y = E[1 * N + s7], n7z = E[2 * N + s7], n8y = E[1 * N + n], n8z = E[2 * N + n];
      const double curlX = 0.5 * (+n5z + n6z - n6y - n7y - n7z - n8z + n8y + n5y) / dx;
      f.faceB[0 * N + n] += dt * curlX;
   }
   if (doY) {
      const long long s3 = nbr(g, i, j, k, -1, 0, -1), s4 = nbr(g, i, j, k, -1, 0, 0), s7 = nbr(g, i, j, k, 0, 0, -1);
      const double n3x = E[0 * N + s3], n3z = E[2 * N + s3], n4x = E[0 * N + s4], n4z = E[2 * N + s4];
      const double n7x = E[0 * N + s7], n7z = E[2 * N + s7], n8x = E[0 * N + n], n8z = E[2 * N + n];
      const double curlY = 0.5 * (-n4x - n8x + n8z + n7z + n7x + n3x - n3z - n4z) / dx;
      f.faceB[1 * N + n] += dt * curlY;
   }
   if (doZ) {
      const long long s1 = nbr(g, i, j, k, -1, -1, 0), s4 = nbr(g, i, j, k, -1, 0, 0), s5 = nbr(g, i, j, k, 0, -1, 0);
      const double n1x = E[0 * N + s1], n1y = E[1 * N + s1], n4x = E[0 * N + s4], n4y = E[1 * N + s4];
      const double n5x = E[0 * N + s5], n5y = E[1 * N + s5], n8x = E[0 * N + n], n8y = E[1 * N + n];
      const double curlZ = 0.5 * (-n1x - n5x - n5y - n8y + n8x + n4x + n4y + n1y) / dx;
      f.faceB[2 * N + n] += dt * curlZ;
   }
}

__global__ void k_ext_bc(GridInfo g, Fields f, FieldParams fp, const int* ext, int next) {
   const int e = blockIdx.x * blockDim.x + threadIdx.x;
   if (e >= next) return;
   const int c = ext[e];
   int i, j, k;
   extCellIJK(g, c, i, j, k);
   const long long N = g.N, n = c;
   const int m = missingMask(g, i, j, k);
   const int wall[6] = {32, 1, 2, 4, 8, 16};  // +x -x +y -y +z -z
   {  // neumannCell(cellB, 3), neumannCell(cellJi, 3), neumannCell(cellRhoQi, 1), setIMFCell
      const signed char* o = c_neu.cellSrc[m];
      const long long s = nbr(g, i, j, k, o[0], o[1], o[2]);
      if (s >= 0) {
         for (int l = 0; l < 3; ++l) f.cellB[l * N + n] = f.cellB[l * N + s];
         for (int l = 0; l < 3; ++l) f.cellJi[l * N + n] = f.cellJi[l * N + s];
         f.cellRho[n] = f.cellRho[s];
      }
      for (int w = 0; w < 6; ++w)
         if ((m & wall[w]) && fp.imfCell[w])
            for (int l = 0; l < 3; ++l) f.cellB[l * N + n] = fp.imf[l];
   }
   {  // neumannFace(faceB), setIMFFace(faceB)
      double v[3];
      bool set[3] = {false, false, false};
      for (int l = 0; l < 3; ++l) {
         if (!c_neu.faceUse[m][l]) continue;
         const signed char* o = c_neu.faceSrc[m][l];
         const long long s = nbr(g, i, j, k, o[0], o[1], o[2]);
         if (s < 0) continue;
         v[l] = f.faceB[l * N + s];
         set[l] = true;
      }
      for (int l = 0; l < 3; ++l) if (set[l]) f.faceB[l * N + n] = v[l];
      for (int w = 0; w < 6; ++w) {
         if ((m & wall[w]) && fp.imfFace[w]) {
            const int axis = w / 2;
            for (int l = 0; l < 3; ++l) if (l != axis) f.faceB[l * N + n] = fp.imf[l];
         }
      }
   }
}

// one layer slot's array a at (x, y) of this thread plus (dx, dy)
struct NodeStencil {
   const double* L;   // cell layer k
   const double* U;   // cell layer k + 1
   int off;
   __device__ __forceinline__ double at(int a, int dx, int dy, int dz) const {
      return (dz ? U : L)[a * (ND_Y + 1) * NT_LX + off + dy * NT_LX + dx];
   }
   // the eight corners' mean in the reference's order
   __device__ __forceinline__ double mean(int a) const {
      return 0.125 * (at(a, 0, 0, 0) + at(a, 0, 0, 1) + at(a, 0, 1, 0) + at(a, 1, 0, 0) + at(a, 0, 1, 1) + at(a, 1, 1, 0) +
                      at(a, 1, 0, 1) + at(a, 1, 1, 1));
   }
};

__device__ __forceinline__ void nodeFromStencil(const GridInfo& g, const Fields& f, const FieldParams& fp,
                                                unsigned long long* cnt, int i, int j, int k, long long n,
                                                const NodeStencil& st, const double avg[3], double eta) {
   const long long N = g.N;
   for (int l = 0; l < 3; ++l) f.cellAvgB[l * N + n] = avg[l] + st.at(l, 0, 0, 0);
   if (!plusOk(g, i, j, k)) return;
   // cell2Node
   double nodeBavg[3];
#pragma unroll
   for (int l = 0; l < 3; ++l) nodeBavg[l] = st.mean(l);
   double rho = st.mean(3);
   double Ji[3];
#pragma unroll
   for (int l = 0; l < 3; ++l) {
      Ji[l] = st.mean(4 + l);
      f.nodeJi[l * N + n] = Ji[l];
   }
   // calcNodeJ (its whistler limiter reads the averaged nodeB and the unclamped nodeRhoQi)
   double Jn[3];
   {
      const double edgeJx1 = -st.at(7 + 2, 0, 0, 0) + st.at(7 + 1, 0, 0, 0) + st.at(7 + 2, 0, 1, 0) - st.at(7 + 1, 0, 0, 1);
      const double edgeJx2 = -st.at(7 + 2, 1, 0, 0) + st.at(7 + 1, 1, 0, 0) + st.at(7 + 2, 1, 1, 0) - st.at(7 + 1, 1, 0, 1);
      const double edgeJy1 = +st.at(7 + 2, 0, 0, 0) + st.at(7 + 0, 0, 0, 1) - st.at(7 + 2, 1, 0, 0) - st.at(7 + 0, 0, 0, 0);
      const double edgeJy2 = +st.at(7 + 2, 0, 1, 0) + st.at(7 + 0, 0, 1, 1) - st.at(7 + 2, 1, 1, 0) - st.at(7 + 0, 0, 1, 0);
      const double edgeJz1 = -st.at(7 + 1, 0, 0, 0) + st.at(7 + 0, 0, 0, 0) + st.at(7 + 1, 1, 0, 0) - st.at(7 + 0, 0, 1, 0);
      const double edgeJz2 = -st.at(7 + 1, 0, 0, 1) + st.at(7 + 0, 0, 0, 1) + st.at(7 + 1, 1, 0, 1) - st.at(7 + 0, 0, 1, 1);
      double d = 1.0;
      double vw = 0.0;
      const double ne = rho / RHGPU_CHARGE_ELEMENTARY;
      const double Btot = sqrt(sq(nodeBavg[0]) + sq(nodeBavg[1]) + sq(nodeBavg[2]));
      if (ne > 0.0 && g.dx > 0.0) {
         vw = 2.0 * Btot * 3.14159265358979323846 / (RHGPU_PERMEABILITY * ne * RHGPU_CHARGE_ELEMENTARY * g.dx);
      }
      const bool lim = vw > fp.maxVw && fp.maxVw > 0.0;
      if (lim) d = vw / fp.maxVw;
      countIf(lim, &cnt[CNT_MAX_VW]);
      gridCount(f, GC_NODE_MAX_VW, N, n, lim);
      const double a = 0.5 / (g.dx * RHGPU_PERMEABILITY * d);
      Jn[0] = (edgeJx1 + edgeJx2) * a;
      Jn[1] = (edgeJy1 + edgeJy2) * a;
      Jn[2] = (edgeJz1 + edgeJz2) * a;
      for (int l = 0; l < 3; ++l) f.nodeJ[l * N + n] = Jn[l];
   }
   // calcNodeUe
   double Ue[3];
   bool rhoClamp = false, ueClamp = false;
   if (f.flags[n] & RHGPU_FLAG_INNER_NODE) {
      for (int l = 0; l < 3; ++l) Ue[l] = fp.obstacleUe[l];
   } else {
      if (rho < fp.minRho) {
         rho = fp.minRho;
         rhoClamp = true;
      }
      for (int l = 0; l < 3; ++l) {
         if (fabs(rho) > 0) {
            if (fp.use_hall) Ue[l] = -(Jn[l] - Ji[l]) / rho;
            else Ue[l] = Ji[l] / rho;
         } else {
            Ue[l] = 0.0;
         }
      }
      const double Ue2 = sq(Ue[0]) + sq(Ue[1]) + sq(Ue[2]);
      if (Ue2 > fp.maxUe2) {
         const double norm = sqrt(fp.maxUe2 / Ue2);
         Ue[0] *= norm; Ue[1] *= norm; Ue[2] *= norm;
         ueClamp = true;
      }
   }
   f.nodeRho[n] = rho;
   countIf(rhoClamp, &cnt[CNT_MIN_NODE_RHO]);
   countIf(ueClamp, &cnt[CNT_MAX_NODE_UE]);
   gridCount(f, GC_CELL_MAX_UE, N, n, ueClamp);
   for (int l = 0; l < 3; ++l) f.nodeUe[l * N + n] = Ue[l];
   // upwindNodeB: the same eight cells as cell2Node (c111 ... c222 = c000 ... c111)
   double xU = -0.5, yU = 0, zU = 0;
   const double U = sqrt(sq(Ue[0]) + sq(Ue[1]) + sq(Ue[2]));
   if (U > 0) {
      const double a = -0.5 / U;
      xU = Ue[0] * a; yU = Ue[1] * a; zU = Ue[2] * a;
   }
   const double w111 = 1 / sqrt(sq(-0.5 - xU) + sq(-0.5 - yU) + sq(-0.5 - zU));
   const double w112 = 1 / sqrt(sq(-0.5 - xU) + sq(-0.5 - yU) + sq(+0.5 - zU));
   const double w121 = 1 / sqrt(sq(-0.5 - xU) + sq(+0.5 - yU) + sq(-0.5 - zU));
   const double w211 = 1 / sqrt(sq(+0.5 - xU) + sq(-0.5 - yU) + sq(-0.5 - zU));
   const double w122 = 1 / sqrt(sq(-0.5 - xU) + sq(+0.5 - yU) + sq(+0.5 - zU));
   const double w221 = 1 / sqrt(sq(+0.5 - xU) + sq(+0.5 - yU) + sq(-0.5 - zU));
   const double w212 = 1 / sqrt(sq(+0.5 - xU) + sq(-0.5 - yU) + sq(+0.5 - zU));
   const double w222 = 1 / sqrt(sq(+0.5 - xU) + sq(+0.5 - yU) + sq(+0.5 - zU));
   const double wsum = w111 + w112 + w121 + w211 + w122 + w221 + w212 + w222;
   double B[3];
   if (wsum > 0) {
      for (int l = 0; l < 3; ++l) {
         B[l] = (w111 * st.at(l, 0, 0, 0) + w112 * st.at(l, 0, 0, 1) + w121 * st.at(l, 0, 1, 0) + w211 * st.at(l, 1, 0, 0) +
                 w122 * st.at(l, 0, 1, 1) + w221 * st.at(l, 1, 1, 0) + w212 * st.at(l, 1, 0, 1) + w222 * st.at(l, 1, 1, 1)) / wsum;
      }
   } else {
      B[0] = B[1] = B[2] = 0.0;
   }
   for (int l = 0; l < 3; ++l) f.nodeB[l * N + n] = B[l];
   // calcNodeE: E = -Ue x B + eta J
   double E[3];
   E[0] = -(Ue[1] * B[2] - Ue[2] * B[1]);
   E[1] = -(Ue[2] * B[0] - Ue[0] * B[2]);
   E[2] = -(Ue[0] * B[1] - Ue[1] * B[0]);
   E[0] += eta * Jn[0];
   E[1] += eta * Jn[1];
   E[2] += eta * Jn[2];
   bool eClamp = false;
   if (fp.maxE2 > 0) {
      const double E2 = sq(E[0]) + sq(E[1]) + sq(E[2]);
      if (E2 > fp.maxE2) {
         const double scaling = sqrt(fp.maxE2 / E2);
         E[0] *= scaling; E[1] *= scaling; E[2] *= scaling;
         eClamp = true;
      }
   }
   countIf(eClamp, &cnt[CNT_MAX_E]);
   gridCount(f, GC_NODE_MAX_E, N, n, eClamp);
   for (int l = 0; l < 3; ++l) f.nodeE[l * N + n] = E[l];
}

__device__ __forceinline__ void ndStage(const GridInfo& g, const Fields& f, double* dst, int i0, int j0, int kz) {
   const long long N = g.N;
   stageLayer<ND_ARR, ND_Y>(
       g,
       [&](int a) {
          return a < 3 ? f.cellB + a * N : a == 3 ? f.cellRho : a < 7 ? f.cellJi + (a - 4) * N : f.faceB + (a - 7) * N;
       },
       f.faceB, dst, i0, j0, kz);
}

__global__ void __launch_bounds__(32 * ND_Y, 3) k_node_fused(GridInfo g, Fields f, FieldParams fp, int nzb, unsigned long long* cnt) {
   extern __shared__ __align__(16) double ndLayers[];
   const int i0 = blockIdx.x * NT_X, j0 = blockIdx.y * ND_Y, k0 = blockIdx.z * nzb;
   const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
   const int nk = min(nzb, g.nz - k0);
   const bool mine = i < g.nx && j < g.ny;
   ndStage(g, f, ndLayers, i0, j0, k0);
   ndStage(g, f, ndLayers + ND_LAYER, i0, j0, k0 + 1);
   cpAsyncCommit();
   if (nk > 1) ndStage(g, f, ndLayers + 2 * ND_LAYER, i0, j0, k0 + 2);
   cpAsyncCommit();
   int a = 0, b = 1;   // slots of layers k and k + 1
   for (int t = 0; t < nk; ++t) {
      const int k = k0 + t;
      const long long n = mine ? cidx(g, i, j, k) : 0;
      // the node's own values, on their way during the wait for the layers
      const double avg[3] = {f.cellAvgB[n], f.cellAvgB[g.N + n], f.cellAvgB[2 * g.N + n]}, eta = f.nodeEta[n];
      cpAsyncWaitGroup<1>();   // cell layers k and k + 1 are in
      __syncthreads();
      NodeStencil st;
      st.L = ndLayers + a * ND_LAYER;
      st.U = ndLayers + b * ND_LAYER;
      st.off = threadIdx.y * NT_LX + threadIdx.x;
      if (mine) nodeFromStencil(g, f, fp, cnt, i, j, k, n, st, avg, eta);
      __syncthreads();         // layer k is read by every thread: its slot takes layer k + 3
      if (t + 2 < nk) ndStage(g, f, ndLayers + a * ND_LAYER, i0, j0, k + 3);
      cpAsyncCommit();
      a = b;
      b = b == 2 ? 0 : b + 1;
   }
}

}  // namespace rh
