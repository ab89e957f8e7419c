// egpu_assembly.cu -- element assembly into the CRS matrix on the device.
//
// Replaces the bulk element loops of HeatSolve (modules/HeatSolve.src:655-985) and
// StressSolve (modules/StressSolve.src:815-1072) for linear isotropic diffusion and
// isotropic elasticity.  Hexahedra: one warp computes four elements on the FP64 matrix
// instruction.  Tetrahedra and triangles: one warp computes one element; lanes < ngauss
// evaluate the geometry of one integration point each (ElementInfo / ElementMetric,
// ElementDescription.src:2586-3320, 6757-6884) into shared memory, then all lanes form the
// element matrix entries.  Entries are added to precomputed CRS positions.  Elements of one
// colour share no node, so the scatter needs no atomics; colours run one after another.
#include <algorithm>
#include <cmath>
#include <vector>

#include "egpu_internal.cuh"
#include "egpu_solve.h"

int egpu_color_elements(int nnodes, int nelem, int nen, const int *elem_nodes, std::vector<int> &color_of);

namespace egpu {

// reference element data: quadrature (Integration.src:281-295, 1446-1486, 84-91) and
// nodal basis (elements.def 808 :606-643, 504 :365-404, 303 :155-185)
template <int CODE>
struct Ref;

template <>
struct Ref<504> {
  static constexpr int NEN = 4, NGP = 4, DIM = 3;
  __device__ static void gp(int t, double &u, double &v, double &w, double &s) {
    const double U[4] = {0.1757281246520584, 0.2445310270213291, 0.5556470949048655, 0.0240937534217468};
    const double V[4] = {0.5656137776620919, 0.0501800797762026, 0.1487681308666864, 0.2354380116950194};
    const double W[4] = {0.2180665126782654, 0.5635595064952189, 0.0350112499848832, 0.1833627308416330};
    u = U[t];
    v = V[t];
    w = W[t];
    s = 0.25 / 6.0;
  }
  __device__ static void basis(double u, double v, double w, double *N, double (*dN)[3]) {
    N[0] = 1.0 - u - v - w;
    N[1] = u;
    N[2] = v;
    N[3] = w;
    const double d[4][3] = {{-1, -1, -1}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int i = 0; i < 3; ++i) dN[p][i] = d[p][i];
  }
};

template <>
struct Ref<303> {
  static constexpr int NEN = 3, NGP = 3, DIM = 2;
  __device__ static void gp(int t, double &u, double &v, double &w, double &s) {
    const double U[3] = {0.16666666666666667, 0.66666666666666667, 0.16666666666666667};
    const double V[3] = {0.16666666666666667, 0.16666666666666667, 0.66666666666666667};
    u = U[t];
    v = V[t];
    w = 0.0;
    s = 0.33333333333333333 / 2.0;
  }
  __device__ static void basis(double u, double v, double, double *N, double (*dN)[3]) {
    N[0] = 1.0 - u - v;
    N[1] = u;
    N[2] = v;
    const double d[3][3] = {{-1, -1, 0}, {1, 0, 0}, {0, 1, 0}};
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int i = 0; i < 3; ++i) dN[p][i] = d[p][i];
  }
};

// geometry of one integration point: dBdx (NEN x 3), detJ*weight.  Returns false for a
// degenerate element (ElementMetric's DetG <= TINY test).
template <int CODE>
__device__ bool gp_geometry(int t, const double (*X)[3], int cdim, double *N, double (*dB)[3], double &s) {
  using R = Ref<CODE>;
  constexpr int NEN = R::NEN, DIM = R::DIM;
  double u, v, w, wt;
  R::gp(t, u, v, w, wt);
  double dN[NEN][3];
  R::basis(u, v, w, N, dN);
  double dx[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double acc = 0.0;
      if (i < DIM)
#pragma unroll
        for (int p = 0; p < NEN; ++p) acc += X[p][c] * dN[p][i];
      dx[c][i] = acc;
    }
  double G[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, GI[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      double acc = 0.0;
      for (int k = 0; k < cdim; ++k) acc += dx[k][i] * dx[k][j];
      G[i][j] = acc;
    }
  double detG;
  if (DIM == 2) {
    detG = G[0][0] * G[1][1] - G[0][1] * G[1][0];
    if (detG <= EGPU_TINY_DP) return false;
    GI[0][0] = G[1][1] / detG;
    GI[0][1] = -G[0][1] / detG;
    GI[1][0] = -G[1][0] / detG;
    GI[1][1] = G[0][0] / detG;
  } else {
    detG = G[0][0] * (G[1][1] * G[2][2] - G[1][2] * G[2][1]) + G[0][1] * (G[1][2] * G[2][0] - G[1][0] * G[2][2]) +
           G[0][2] * (G[1][0] * G[2][1] - G[1][1] * G[2][0]);
    if (detG <= EGPU_TINY_DP) return false;
    const double q = 1.0 / detG;
    GI[0][0] = q * (G[1][1] * G[2][2] - G[2][1] * G[1][2]);
    GI[1][0] = -q * (G[1][0] * G[2][2] - G[2][0] * G[1][2]);
    GI[2][0] = q * (G[1][0] * G[2][1] - G[2][0] * G[1][1]);
    GI[0][1] = -q * (G[0][1] * G[2][2] - G[2][1] * G[0][2]);
    GI[1][1] = q * (G[0][0] * G[2][2] - G[2][0] * G[0][2]);
    GI[2][1] = -q * (G[0][0] * G[2][1] - G[2][0] * G[0][1]);
    GI[0][2] = q * (G[0][1] * G[1][2] - G[1][1] * G[0][2]);
    GI[1][2] = -q * (G[0][0] * G[1][2] - G[1][0] * G[0][2]);
    GI[2][2] = q * (G[0][0] * G[1][1] - G[1][0] * G[0][1]);
  }
  s = sqrt(detG) * wt;
  double L[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      double acc = 0.0;
#pragma unroll
      for (int k = 0; k < DIM; ++k) acc += dx[i][k] * GI[k][j];
      L[i][j] = acc;
    }
#pragma unroll
  for (int p = 0; p < NEN; ++p)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double acc = 0.0;
      if (j < cdim)
#pragma unroll
        for (int k = 0; k < DIM; ++k) acc += dN[p][k] * L[j][k];
      dB[p][j] = acc;
    }
  return true;
}

// FP64 matrix instruction D = A B + D on one 8x8 tile (A 8x4 row-major, B 4x8 column-major):
// lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4) + {0, 1}].
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

constexpr int ASM_WARPS = 8;

// ------------------------------------------------------------------------------------
// Hexahedra (808), four elements per warp.
//
// The element matrix is a contraction over the integration points: with the gradients
// G_t(p, i) = dN_p/dx_i at point t, Poisson's K = sum_(t,i) (w_t G_t(p,i)) G_t(q,i) is an
// 8x24 by 24x8 product, and elasticity's M_ij = sum_t (s_t G_t(p,i)) G_t(q,j) nine 8x8x8
// ones.  Both run on the FP64 matrix instruction, whose fragments put node p = lane / 4 and
// point t = lane % 4 (+ 4) on a lane: the same value is the A operand (times the weight)
// and the B operand, so a lane needs the gradients of one node at two points only, and forms
// them itself from the points' 3x3 geometry factors L_t (gradient = L_t dN/dxi).
//   1. lane = (element, node): node ids, coordinates and material, staged in shared memory
//   2. lane = (element, point): Jacobian, metric, L_t and the weights, into shared memory
//      (all 32 lanes busy; one element per warp left 24 of them idle)
//   3. per element: two gradients per lane, six (Poisson) or eighteen (elasticity) matrix
//      instructions, and the accumulators are exactly the lane's CRS entries (two columns)
// The CRS positions and the values they hold are loaded before step 2, so their latency is
// covered by it.  Elements of a colour share no node, so the preloaded values are current.
constexpr int HEX_EPW = 4;       // elements per warp
constexpr int HEX_XS = 25;       // doubles per element of staged coordinates (24 + 1: no bank conflicts)
constexpr int HEX_LS = 12;       // doubles per point: L (9), weight, load weight, pad

struct HexShared {
  double X[HEX_EPW * HEX_XS];
  double kn[32], ln[32];
  double2 L[32 * HEX_LS / 2];
};

// reference coordinates of node p and point t as sign bits (u, v, w); 1 = +
__device__ __forceinline__ int hex_node_bits(int p) { return ((0x66 >> p) & 1) | (((0xCC >> p) & 1) << 1) | ((p >> 2) << 2); }

// dN_p/dxi at point t (elements.def 808 :606-643, 2-point Gauss per direction)
__device__ __forceinline__ void hex_dN(int p, int t, double &d0, double &d1, double &d2) {
  const double g = 0.57735026918962576451;  // 1/sqrt(3)
  const int pb = hex_node_bits(p), x = pb ^ t;
  const double a = (x & 1) ? 1.0 - g : 1.0 + g, b = (x & 2) ? 1.0 - g : 1.0 + g, c = (x & 4) ? 1.0 - g : 1.0 + g;
  d0 = ((pb & 1) ? 0.125 : -0.125) * b * c;
  d1 = ((pb & 2) ? 0.125 : -0.125) * a * c;
  d2 = ((pb & 4) ? 0.125 : -0.125) * a * b;
}
__device__ __forceinline__ double hex_N(int p, int t) {
  const double g = 0.57735026918962576451;
  const int x = hex_node_bits(p) ^ t;
  const double a = (x & 1) ? 1.0 - g : 1.0 + g, b = (x & 2) ? 1.0 - g : 1.0 + g, c = (x & 4) ? 1.0 - g : 1.0 + g;
  return 0.125 * a * b * c;
}

// step 2 for lane (el, t): L_t = dx GI with GI the inverse metric (ElementMetric), and
// s = sqrt(detG); a degenerate element (DetG <= TINY) gets L = 0, s = 0
__device__ __forceinline__ double hex_point(const double *X, int t, int cdim, double (&L)[3][3]) {
  double dx[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int i = 0; i < 3; ++i) dx[c][i] = 0.0;
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    double d0, d1, d2;
    hex_dN(p, t, d0, d1, d2);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double x = X[3 * p + c];
      dx[c][0] += x * d0;
      dx[c][1] += x * d1;
      dx[c][2] += x * d2;
    }
  }
  double G[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      double acc = dx[0][i] * dx[0][j] + dx[1][i] * dx[1][j];
      if (cdim > 2) acc += dx[2][i] * dx[2][j];
      G[i][j] = acc;
      G[j][i] = acc;
    }
  const double detG = G[0][0] * (G[1][1] * G[2][2] - G[1][2] * G[2][1]) + G[0][1] * (G[1][2] * G[2][0] - G[1][0] * G[2][2]) +
                      G[0][2] * (G[1][0] * G[2][1] - G[1][1] * G[2][0]);
  const bool ok = !(detG <= EGPU_TINY_DP);  // NaN coordinates give NaN, not a missing element
  const double q = ok ? 1.0 / detG : 0.0;
  double GI[3][3];
  GI[0][0] = q * (G[1][1] * G[2][2] - G[2][1] * G[1][2]);
  GI[1][0] = -q * (G[1][0] * G[2][2] - G[2][0] * G[1][2]);
  GI[2][0] = q * (G[1][0] * G[2][1] - G[2][0] * G[1][1]);
  GI[1][1] = q * (G[0][0] * G[2][2] - G[2][0] * G[0][2]);
  GI[2][1] = -q * (G[0][0] * G[2][1] - G[2][0] * G[0][1]);
  GI[2][2] = q * (G[0][0] * G[1][1] - G[1][0] * G[0][1]);
  GI[0][1] = GI[1][0];
  GI[0][2] = GI[2][0];
  GI[1][2] = GI[2][1];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      L[i][j] = i < cdim ? dx[i][0] * GI[0][j] + dx[i][1] * GI[1][j] + dx[i][2] * GI[2][j] : 0.0;
  return ok ? sqrt(detG) : 0.0;
}

// gradient of the lane's node at one point: row i of L_t times dN/dxi; returns the weight
__device__ __forceinline__ double hex_grad(const double2 *L, double d0, double d1, double d2, double (&g)[3]) {
  const double2 l0 = L[0], l1 = L[1], l2 = L[2], l3 = L[3], l4 = L[4];
  g[0] = d0 * l0.x + d1 * l0.y + d2 * l1.x;
  g[1] = d0 * l1.y + d1 * l2.x + d2 * l2.y;
  g[2] = d0 * l3.x + d1 * l3.y + d2 * l4.x;
  return l4.y;
}

__device__ __forceinline__ void hex_store_point(double2 *L, const double (&l)[3][3], double w, double f) {
  L[0] = make_double2(l[0][0], l[0][1]);
  L[1] = make_double2(l[0][2], l[1][0]);
  L[2] = make_double2(l[1][1], l[1][2]);
  L[3] = make_double2(l[2][0], l[2][1]);
  L[4] = make_double2(l[2][2], w);
  L[5] = make_double2(f, 0.0);
}

// Diffusion on 808: K_pq = sum_t s_t k_t dN_q.dN_p, f_p = sum_t s_t (sum_m load_m N_m) N_p
// (DiffuseConvectiveAnisotropic.src:334-344, 515-561, 569-612)
__global__ void __launch_bounds__(ASM_WARPS * 32, 2) k_assemble_poisson_hex(
    int ne, const int *__restrict__ elist, const int *__restrict__ enodes, const double *__restrict__ xyz,
    int cdim, const double *__restrict__ elem_k, const double *__restrict__ nodal_k,
    const double *__restrict__ load, const int *__restrict__ perm, const int *__restrict__ slots,
    double *__restrict__ values, double *__restrict__ rhs) {
  __shared__ __align__(16) HexShared sh_all[ASM_WARPS];
  HexShared &sh = sh_all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * ASM_WARPS + (threadIdx.x >> 5)) * HEX_EPW;
  if (w0 >= ne) return;
  const int el = lane >> 3, nd = lane & 7;
  const bool have = w0 + el < ne;
  const int e = have ? elist[w0 + el] : 0;
  const int node = have ? enodes[(size_t)e * 8 + nd] : 0;
  // this lane's CRS positions (node lane/4's row, two columns) and their present values
  int2 sl[HEX_EPW];
  double2 old[HEX_EPW];
#pragma unroll
  for (int j = 0; j < HEX_EPW; ++j) {
    const int ej = __shfl_sync(0xffffffffu, e, 8 * j);
    sl[j] = w0 + j < ne ? __ldcs(reinterpret_cast<const int2 *>(slots + (size_t)ej * 64) + lane) : make_int2(-1, -1);
  }
  sh.kn[lane] = !have ? 0.0 : elem_k ? elem_k[e] : (nodal_k ? nodal_k[node] : 1.0);
  sh.ln[lane] = have && load ? load[node] : 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) sh.X[el * HEX_XS + 3 * nd + c] = have ? xyz[(size_t)node * 3 + c] : 0.0;
#pragma unroll
  for (int j = 0; j < HEX_EPW; ++j) {
    old[j].x = sl[j].x >= 0 ? values[sl[j].x] : 0.0;
    old[j].y = sl[j].y >= 0 ? values[sl[j].y] : 0.0;
  }
  __syncwarp();
  {
    double L[3][3];
    const double s = hex_point(sh.X + el * HEX_XS, nd, cdim, L);
    double kk = 0.0, ff = 0.0;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const double N = hex_N(p, nd);
      kk += sh.kn[8 * el + p] * N;
      ff += sh.ln[8 * el + p] * N;
    }
    hex_store_point(sh.L + lane * (HEX_LS / 2), L, s * kk, s * ff);
  }
  __syncwarp();
  const int p = lane >> 2, kq = lane & 3;
  double d1[3], d2[3];
  hex_dN(p, kq, d1[0], d1[1], d1[2]);
  hex_dN(p, kq + 4, d2[0], d2[1], d2[2]);
#pragma unroll
  for (int j = 0; j < HEX_EPW; ++j) {
    double g[3], c0 = 0.0, c1 = 0.0;
    double wt = hex_grad(sh.L + (8 * j + kq) * (HEX_LS / 2), d1[0], d1[1], d1[2], g);
#pragma unroll
    for (int i = 0; i < 3; ++i) dmma_8x8x4(c0, c1, wt * g[i], g[i]);
    wt = hex_grad(sh.L + (8 * j + kq + 4) * (HEX_LS / 2), d2[0], d2[1], d2[2], g);
#pragma unroll
    for (int i = 0; i < 3; ++i) dmma_8x8x4(c0, c1, wt * g[i], g[i]);
    if (sl[j].x >= 0) values[sl[j].x] = old[j].x + c0;
    if (sl[j].y >= 0) values[sl[j].y] = old[j].y + c1;
  }
  if (load && have) {
    double F = 0.0;
#pragma unroll
    for (int t = 0; t < 8; ++t) F += sh.L[(8 * el + t) * (HEX_LS / 2) + 5].x * hex_N(nd, t);
    const int r = perm[node];
    if (r >= 0) rhs[r] += F;
  }
}

// Isotropic elasticity on 808 (see k_assemble_elastic for the form of K): the nine 8x8
// matrices M_ij of a node pair end on one lane, which combines them,
//   K_(p,i),(q,j) = c12 M_ij + c44 (M_ji + delta_ij (M_00 + M_11 + M_22)).
__global__ void __launch_bounds__(ASM_WARPS * 32, 2) k_assemble_elastic_hex(
    int ne, const int *__restrict__ elist, const int *__restrict__ enodes, const double *__restrict__ xyz,
    double c12, double c44, double bf0, double bf1, double bf2, const int *__restrict__ perm,
    const int *__restrict__ slots, double *__restrict__ values, double *__restrict__ rhs) {
  __shared__ __align__(16) HexShared sh_all[ASM_WARPS];
  HexShared &sh = sh_all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int w0 = (blockIdx.x * ASM_WARPS + (threadIdx.x >> 5)) * HEX_EPW;
  if (w0 >= ne) return;
  const int el = lane >> 3, nd = lane & 7;
  const bool have = w0 + el < ne;
  const int e = have ? elist[w0 + el] : 0;
  const int node = have ? enodes[(size_t)e * 8 + nd] : 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) sh.X[el * HEX_XS + 3 * nd + c] = have ? xyz[(size_t)node * 3 + c] : 0.0;
  __syncwarp();
  {
    double L[3][3];
    const double s = hex_point(sh.X + el * HEX_XS, nd, 3, L);
    double sn = 0.0;
#pragma unroll
    for (int p = 0; p < 8; ++p) sn += hex_N(p, nd);
    hex_store_point(sh.L + lane * (HEX_LS / 2), L, s, s * sn);
  }
  __syncwarp();
  const int p = lane >> 2, kq = lane & 3;
  double d1[3], d2[3];
  hex_dN(p, kq, d1[0], d1[1], d1[2]);
  hex_dN(p, kq + 4, d2[0], d2[1], d2[2]);
  for (int j = 0; j < HEX_EPW && w0 + j < ne; ++j) {
    const int ej = __shfl_sync(0xffffffffu, e, 8 * j);
    // row (p, i): six consecutive positions, columns (q, q + 1) x 3 DOFs
    const int *sb = slots + (size_t)ej * 576 + 72 * p + 6 * kq;
    int2 sl[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int h = 0; h < 3; ++h) sl[i][h] = __ldcs(reinterpret_cast<const int2 *>(sb + 24 * i) + h);
    double g1[3], g2[3];
    const double w1 = hex_grad(sh.L + (8 * j + kq) * (HEX_LS / 2), d1[0], d1[1], d1[2], g1);
    const double w2 = hex_grad(sh.L + (8 * j + kq + 4) * (HEX_LS / 2), d2[0], d2[1], d2[2], g2);
    double M[3][3][2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        M[i][c][0] = M[i][c][1] = 0.0;
        dmma_8x8x4(M[i][c][0], M[i][c][1], w1 * g1[i], g1[c]);
        dmma_8x8x4(M[i][c][0], M[i][c][1], w2 * g2[i], g2[c]);
      }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      // entry (q, c) of the row sits at 3 q + c of its six
      double old[6];
      int pos[6];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        pos[2 * h] = sl[i][h].x;
        pos[2 * h + 1] = sl[i][h].y;
      }
#pragma unroll
      for (int t = 0; t < 6; ++t) old[t] = pos[t] >= 0 ? values[pos[t]] : 0.0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double tr = M[0][0][q] + M[1][1][q] + M[2][2][q];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double v = c12 * M[i][c][q] + c44 * M[c][i][q];
          if (i == c) v += c44 * tr;
          if (pos[3 * q + c] >= 0) values[pos[3 * q + c]] = old[3 * q + c] + v;
        }
      }
    }
  }
  if (have) {
    double F = 0.0;
#pragma unroll
    for (int t = 0; t < 8; ++t) F += sh.L[(8 * el + t) * (HEX_LS / 2) + 5].x * hex_N(nd, t);
    const int r = perm[node];
    if (r >= 0) {
      rhs[3 * r] += bf0 * F;
      rhs[3 * r + 1] += bf1 * F;
      rhs[3 * r + 2] += bf2 * F;
    }
  }
}


// Diffusion: K_pq = sum_t s_t k_t dN_q.dN_p, f_p = sum_t s_t (sum_m load_m N_m) N_p
// (DiffuseConvectiveAnisotropic.src:334-344, 515-561, 569-612)
template <int CODE>
__global__ void __launch_bounds__(ASM_WARPS * 32, 3) k_assemble_poisson(
    int ne, const int *__restrict__ elist, const int *__restrict__ enodes, const double *__restrict__ xyz,
    int cdim, const double *__restrict__ elem_k, const double *__restrict__ nodal_k,
    const double *__restrict__ load, const int *__restrict__ perm, const int *__restrict__ slots,
    double *__restrict__ values, double *__restrict__ rhs) {
  using R = Ref<CODE>;
  constexpr int NEN = R::NEN, NGP = R::NGP;
  __shared__ double sh_dB[ASM_WARPS][NGP][NEN][3];
  __shared__ double sh_N[ASM_WARPS][NGP][NEN];
  __shared__ double sh_s[ASM_WARPS][NGP], sh_k[ASM_WARPS][NGP], sh_f[ASM_WARPS][NGP];
  // the element's node coordinates and nodal k / load, staged once per warp (lane p holds
  // node p's) instead of in every lane's registers
  __shared__ double sh_X[ASM_WARPS][NEN][3], sh_kn[ASM_WARPS][NEN], sh_ln[ASM_WARPS][NEN];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * ASM_WARPS + wib;
  if (w >= ne) return;
  const int e = elist[w];
  int node = 0;
  if (lane < NEN) {
    node = enodes[(size_t)e * NEN + lane];
    sh_kn[wib][lane] = elem_k ? elem_k[e] : (nodal_k ? nodal_k[node] : 1.0);
    sh_ln[wib][lane] = load ? load[node] : 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) sh_X[wib][lane][c] = xyz[(size_t)node * 3 + c];
  }
  __syncwarp();
  if (lane < NGP) {
    double N[NEN], dB[NEN][3], s;
    const bool ok = gp_geometry<CODE>(lane, sh_X[wib], cdim, N, dB, s);
    double kk = 0.0, ff = 0.0;
#pragma unroll
    for (int p = 0; p < NEN; ++p) {
      kk += sh_kn[wib][p] * N[p];
      ff += sh_ln[wib][p] * N[p];
    }
    sh_s[wib][lane] = ok ? s : 0.0;
    sh_k[wib][lane] = kk;
    sh_f[wib][lane] = ff;
#pragma unroll
    for (int p = 0; p < NEN; ++p) {
      sh_N[wib][lane][p] = N[p];
#pragma unroll
      for (int i = 0; i < 3; ++i) sh_dB[wib][lane][p][i] = dB[p][i];
    }
  }
  __syncwarp();
  const int *sl = slots + (size_t)e * NEN * NEN;
  for (int idx = lane; idx < NEN * NEN; idx += 32) {
    const int p = idx / NEN, q = idx % NEN;
    double K = 0.0;
#pragma unroll
    for (int t = 0; t < NGP; ++t) {
      double A = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) A += sh_k[wib][t] * sh_dB[wib][t][q][i] * sh_dB[wib][t][p][i];
      K += sh_s[wib][t] * A;
    }
    const int slot = sl[idx];
    if (slot >= 0) values[slot] += K;
  }
  if (lane < NEN) {
    double F = 0.0;
#pragma unroll
    for (int t = 0; t < NGP; ++t) F += sh_s[wib][t] * (sh_f[wib][t] * sh_N[wib][t][lane]);
    const int r = perm[node];
    if (r >= 0) rhs[r] += F;
  }
}

// Isotropic elasticity (Stress.src:260-273, 366-439, 476-515): with c12 = E nu/((1+nu)(1-2nu)),
// c44 = E (1/2-nu)/((1+nu)(1-2nu)) the product G_p C B_q collapses to
//   K_(p,i),(q,j) = c12 a_i b_j + c44 (a_j b_i + delta_ij a.b),  a = dN_p/dx, b = dN_q/dx,
// which is already symmetric, so the reference's (K+K^T)/2 leaves it unchanged.
template <int CODE>
__global__ void __launch_bounds__(ASM_WARPS * 32) k_assemble_elastic(
    int ne, const int *__restrict__ elist, const int *__restrict__ enodes, const double *__restrict__ xyz,
    double c12, double c44, double bf0, double bf1, double bf2, const int *__restrict__ perm,
    const int *__restrict__ slots, double *__restrict__ values, double *__restrict__ rhs) {
  using R = Ref<CODE>;
  constexpr int NEN = R::NEN, NGP = R::NGP, ND = 3 * NEN;
  __shared__ double sh_dB[ASM_WARPS][NGP][NEN][3];
  __shared__ double sh_N[ASM_WARPS][NGP][NEN];
  __shared__ double sh_s[ASM_WARPS][NGP], sh_sn[ASM_WARPS][NGP];
  __shared__ double sh_X[ASM_WARPS][NEN][3];  // node coordinates, staged once per warp
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * ASM_WARPS + wib;
  if (w >= ne) return;
  const int e = elist[w];
  int node = 0;
  if (lane < NEN) {
    node = enodes[(size_t)e * NEN + lane];
#pragma unroll
    for (int c = 0; c < 3; ++c) sh_X[wib][lane][c] = xyz[(size_t)node * 3 + c];
  }
  __syncwarp();
  if (lane < NGP) {
    double N[NEN], dB[NEN][3], s;
    const bool ok = gp_geometry<CODE>(lane, sh_X[wib], 3, N, dB, s);
    double sn = 0.0;
#pragma unroll
    for (int p = 0; p < NEN; ++p) sn += N[p];
    sh_s[wib][lane] = ok ? s : 0.0;
    sh_sn[wib][lane] = sn;
#pragma unroll
    for (int p = 0; p < NEN; ++p) {
      sh_N[wib][lane][p] = N[p];
#pragma unroll
      for (int i = 0; i < 3; ++i) sh_dB[wib][lane][p][i] = dB[p][i];
    }
  }
  __syncwarp();
  const int *sl = slots + (size_t)e * ND * ND;
  for (int idx = lane; idx < ND * ND; idx += 32) {
    const int ra = idx / ND, cb = idx % ND;
    const int p = ra / 3, i = ra % 3, q = cb / 3, j = cb % 3;
    double K = 0.0;
#pragma unroll
    for (int t = 0; t < NGP; ++t) {
      const double *a = sh_dB[wib][t][p], *b = sh_dB[wib][t][q];
      double v = c12 * a[i] * b[j] + c44 * a[j] * b[i];
      if (i == j) v += c44 * (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]);
      K += sh_s[wib][t] * v;
    }
    const int slot = sl[idx];
    if (slot >= 0) values[slot] += K;
  }
  int node_of[NEN];
#pragma unroll
  for (int p = 0; p < NEN; ++p) node_of[p] = __shfl_sync(0xffffffffu, node, p);
  if (lane < ND) {
    const int p = lane / 3, i = lane % 3;
    const double bfi = i == 0 ? bf0 : (i == 1 ? bf1 : bf2);
    double F = 0.0;
#pragma unroll
    for (int t = 0; t < NGP; ++t) F += sh_s[wib][t] * ((bfi * sh_sn[wib][t]) * sh_N[wib][t][p]);
    const int r = perm[node_of[p]];
    if (r >= 0) rhs[3 * r + i] += F;
  }
}

// element -> CRS positions: slots[e][a][b] = position of (row(a), col(b)) in Cols,
// found by binary search in the row (rows are sorted, CRS_SortMatrix)
__global__ void k_slot_map(int nelem, int nen, int dofs, const int *__restrict__ enodes,
                           const int *__restrict__ perm, const int *__restrict__ rows,
                           const int *__restrict__ cols, int *__restrict__ slots, int *err) {
  const int nd = nen * dofs;
  const long long total = (long long)nelem * nd;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t / nd), a = (int)(t % nd);
    const int pn = perm[enodes[(size_t)e * nen + a / dofs]];
    int *out = slots + ((size_t)e * nd + a) * nd;
    if (pn < 0) {
      for (int b = 0; b < nd; ++b) out[b] = -1;
      continue;
    }
    const int row = pn * dofs + a % dofs;
    const int beg = rows[row], end = rows[row + 1];
    for (int b = 0; b < nd; ++b) {
      const int qn = perm[enodes[(size_t)e * nen + b / dofs]];
      int pos = -1;
      if (qn >= 0) {
        const int col = qn * dofs + b % dofs;
        int lo = beg, hi = end - 1;
        while (lo <= hi) {
          const int mid = (lo + hi) >> 1;
          const int c = cols[mid];
          if (c == col) {
            pos = mid;
            break;
          }
          if (c < col)
            lo = mid + 1;
          else
            hi = mid - 1;
        }
        if (pos < 0) atomicExch(err, 1);
      }
      out[b] = pos;
    }
  }
}

__global__ void k_fill_zero(double *p, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = 0.0;
}

// DefaultDirichletBCs (DefUtils.src:3530-4031) on the whole matrix in one pass:
// scale without rhs normalisation, constrained rows -> zero row, unit diagonal,
// b = val/D (SolverUtils.src:2465-2473), or symmetric elimination (CRS_SetSymmDirichlet,
// CRSMatrix.src:674-740), then back-scaling.  Eight lanes per row, so a row's values and
// columns are read and written as whole sectors; the right-hand side takes the constrained
// columns' terms in column order, as the reference does.
__global__ void k_dirichlet(int n, const int *__restrict__ rows, const int *__restrict__ cols,
                            const int *__restrict__ diag, double *__restrict__ values, double *__restrict__ rhs,
                            const double *__restrict__ D, const unsigned char *__restrict__ cflag,
                            const double *__restrict__ cval, int symmetric) {
  const int lane = threadIdx.x & 7, sub = threadIdx.x & 24;
  const int stride = (gridDim.x * blockDim.x) >> 3;
  // the four rows of a warp run in step, so the collectives below are whole-warp ones
  for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4; i0 < n; i0 += stride) {
    const int i = i0 + (sub >> 3);
    const bool on = i < n;
    const double di = on ? D[i] : 1.0;
    double bi = on ? rhs[i] * di : 0.0;
    const int beg = on ? rows[i] : 0, end = on ? rows[i + 1] : 0;
    const bool fixed = on && cflag[i];
    const int nch = __reduce_max_sync(0xffffffffu, fixed ? 0 : (end - beg + 7) >> 3);
    if (fixed) {
      const int dg = diag[i];
      for (int k = beg + lane; k < end; k += 8) values[k] = k == dg ? 1.0 / (di * di) : 0.0;
      bi = cval[i] / di;
    }
#pragma unroll 4
    for (int ch = 0; ch < nch; ++ch) {
      const int k = beg + 8 * ch + lane;
      double term = 0.0;
      bool con = false;
      if (!fixed && k < end) {
        const int c = cols[k];
        const double dc = D[c], dd = di * dc;
        double v = values[k] * dd;
        if (symmetric && cflag[c]) {
          con = true;
          term = v * (cval[c] / dc);
          v = 0.0;
        }
        values[k] = v / dd;
      }
      if (symmetric) {
        const unsigned any = __ballot_sync(0xffffffffu, con);
        if (any) {  // constrained neighbours are rare: the terms in column order, row by row
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const double t = __shfl_sync(0xffffffffu, term, sub + q);
            if ((any >> (sub + q)) & 1u) bi = bi - t;
          }
        }
      }
    }
    if (on && lane == 0) rhs[i] = bi / di * 1.0;
  }
}

// ScaleLinearSystem diagonal (SolverUtils.src:6500-6562) of the assembled matrix
__global__ void k_dirichlet_scale_diag(int n, const int *__restrict__ rows, const int *__restrict__ diag,
                                       const double *__restrict__ vals, double *__restrict__ D) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int j = diag[i];
    double d = j >= 0 ? vals[j] : 0.0;
    if (fabs(d) <= EGPU_TINY_DP) {
      double s = 0.0;
      for (int k = rows[i]; k < rows[i + 1]; ++k) s += fabs(vals[k]);
      d = s;
    }
    D[i] = fabs(d) > EGPU_TINY_DP ? 1.0 / sqrt(fabs(d)) : 1.0;
  }
}

__global__ void k_scatter_con(int ncon, const int *__restrict__ con_rows, const double *__restrict__ con_vals,
                              unsigned char *cflag, double *cval, int n, int *err) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ncon; t += gridDim.x * blockDim.x) {
    const int r = con_rows[t] - 1;
    if (r < 0 || r >= n) {
      atomicExch(err, 1);
      continue;
    }
    cflag[r] = 1;
    cval[r] = con_vals ? con_vals[t] : 0.0;
  }
}

}  // namespace egpu

using namespace egpu;

static int grid_of(egpu_ctx *ctx, long long work, int block = 256) {
  long long g = (work + block - 1) / block;
  return (int)std::max(1LL, std::min(g, (long long)ctx->num_sms * 16));
}

extern "C" int egpu_assembly_bind(egpu_mat *A, int nnodes, const double *xyz, int cdim, int nelem, int code,
                                  const int *elem_nodes, const int *perm, int dofs) {
  if (!A || nnodes <= 0 || nelem <= 0 || !xyz || !elem_nodes || !perm) return EGPU_ERR_ARG;
  if (code != 808 && code != 504 && code != 303) return EGPU_ERR_ARG;
  if (dofs != 1 && !(dofs == 3 && code != 303)) return EGPU_ERR_ARG;
  if (cdim != 2 && cdim != 3) return EGPU_ERR_ARG;
  egpu_ctx *ctx = A->ctx;
  cudaSetDevice(ctx->device);
  const int nen = code % 100;
  AssemblyData &S = A->asmb;
  S.nnodes = nnodes;
  S.nelem = nelem;
  S.nen = nen;
  S.code = code;
  S.dofs = dofs;
  S.cdim = cdim;
  std::vector<int> en0((size_t)nelem * nen), p0(nnodes);
  for (size_t k = 0; k < en0.size(); ++k) {
    if (elem_nodes[k] < 1 || elem_nodes[k] > nnodes) return EGPU_ERR_ARG;
    en0[k] = elem_nodes[k] - 1;
  }
  for (int i = 0; i < nnodes; ++i) {
    p0[i] = perm[i] - 1;
    if (p0[i] >= 0 && (long long)(p0[i] + 1) * dofs > A->n) return EGPU_ERR_ARG;
  }
  std::vector<int> color_of;
  const int ncol = egpu_color_elements(nnodes, nelem, nen, elem_nodes, color_of);
  // One launch per colour.  (Groups by row range and colour, so that a range's Values stay in L2 for
  // all its colours, were slower at every size: hex 96^3 693 against 615 us, 128^3 1,591 and
  // 1,362, elasticity 64^3 2,158 and 1,403, tetrahedral elasticity 56^3 3,350 and 3,018, and with
  // elements in random order 4,265 and 1,648 at 64^3: a group is then one or two waves, bound by its own chain.)
  S.color_ptr.assign(ncol + 1, 0);
  for (int e = 0; e < nelem; ++e) S.color_ptr[color_of[e] + 1]++;
  for (int c = 0; c < ncol; ++c) S.color_ptr[c + 1] += S.color_ptr[c];
  std::vector<int> grouped(nelem), fill(S.color_ptr.begin(), S.color_ptr.end() - 1);
  for (int e = 0; e < nelem; ++e) grouped[fill[color_of[e]]++] = e;
  const int nd = nen * dofs;
  EGPU_CUDA_TRY(ctx, S.xyz.alloc((size_t)nnodes * 3));
  EGPU_CUDA_TRY(ctx, S.elem_nodes.alloc(en0.size()));
  EGPU_CUDA_TRY(ctx, S.perm.alloc(nnodes));
  EGPU_CUDA_TRY(ctx, S.color_elems.alloc(nelem));
  EGPU_CUDA_TRY(ctx, S.slots.alloc((size_t)nelem * nd * nd));
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(S.xyz.p, xyz, (size_t)nnodes * 3 * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(S.elem_nodes.p, en0.data(), en0.size() * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(S.perm.p, p0.data(), nnodes * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(S.color_elems.p, grouped.data(), nelem * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  int *err = (int *)(ctx->sync.p + 1);
  EGPU_CUDA_TRY(ctx, cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  k_slot_map<<<grid_of(ctx, (long long)nelem * nd), 256, 0, ctx->stream>>>(nelem, nen, dofs, S.elem_nodes.p, S.perm.p,
                                                                          A->rows.p, A->cols.p, S.slots.p, err);
  ctx->launches++;
  int herr = 0;
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  EGPU_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (herr) {
    egpu_set_error(ctx, "mesh and CRS pattern disagree: an element coupling has no matrix entry");
    return EGPU_ERR_ARG;
  }
  S.bound = true;
  return EGPU_OK;
}

extern "C" int egpu_assemble_poisson(egpu_mat *A, const double *elem_k, const double *nodal_k, const double *load) {
  if (!A || !A->asmb.bound || A->asmb.dofs != 1) return EGPU_ERR_STATE;
  egpu_ctx *ctx = A->ctx;
  cudaSetDevice(ctx->device);
  AssemblyData &S = A->asmb;
  DevBuf<double> dk, dn, dl;
  if (elem_k) {
    EGPU_CUDA_TRY(ctx, dk.alloc(S.nelem));
    EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(dk.p, elem_k, S.nelem * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  }
  if (nodal_k) {
    EGPU_CUDA_TRY(ctx, dn.alloc(S.nnodes));
    EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(dn.p, nodal_k, S.nnodes * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  }
  if (load) {
    EGPU_CUDA_TRY(ctx, dl.alloc(S.nnodes));
    EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(dl.p, load, S.nnodes * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  }
  k_fill_zero<<<grid_of(ctx, A->nnz), 256, 0, ctx->stream>>>(A->values.p, A->nnz);
  k_fill_zero<<<grid_of(ctx, A->n), 256, 0, ctx->stream>>>(A->rhs.p, A->n);
  ctx->launches += 2;
  const int ncol = (int)S.color_ptr.size() - 1;
  for (int c = 0; c < ncol; ++c) {
    const int ne = S.color_ptr[c + 1] - S.color_ptr[c];
    if (!ne) continue;
    const int *el = S.color_elems.p + S.color_ptr[c];
    const int grid = (ne + ASM_WARPS - 1) / ASM_WARPS;
#define EGPU_ASM(CODE)                                                                                       \
  k_assemble_poisson<CODE><<<grid, ASM_WARPS * 32, 0, ctx->stream>>>(ne, el, S.elem_nodes.p, S.xyz.p, S.cdim, \
                                                                     dk.p, dn.p, dl.p, S.perm.p, S.slots.p,    \
                                                                     A->values.p, A->rhs.p)
    if (S.code == 808)
      k_assemble_poisson_hex<<<(ne + ASM_WARPS * HEX_EPW - 1) / (ASM_WARPS * HEX_EPW), ASM_WARPS * 32, 0, ctx->stream>>>(
          ne, el, S.elem_nodes.p, S.xyz.p, S.cdim, dk.p, dn.p, dl.p, S.perm.p, S.slots.p, A->values.p, A->rhs.p);
    else if (S.code == 504)
      EGPU_ASM(504);
    else
      EGPU_ASM(303);
#undef EGPU_ASM
    ctx->launches++;
  }
  EGPU_CUDA_TRY(ctx, cudaGetLastError());
  EGPU_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  A->has_values = true;
  A->has_rhs = true;
  A->ilu_valid = false;
  return EGPU_OK;
}

extern "C" int egpu_assemble_elastic(egpu_mat *A, double young, double poisson, const double *bf) {
  if (!A || !A->asmb.bound || A->asmb.dofs != 3 || !bf) return EGPU_ERR_STATE;
  egpu_ctx *ctx = A->ctx;
  cudaSetDevice(ctx->device);
  AssemblyData &S = A->asmb;
  const double cs = young / ((1 + poisson) * (1 - 2 * poisson));
  const double c12 = poisson * cs, c44 = (0.5 - poisson) * cs;
  k_fill_zero<<<grid_of(ctx, A->nnz), 256, 0, ctx->stream>>>(A->values.p, A->nnz);
  k_fill_zero<<<grid_of(ctx, A->n), 256, 0, ctx->stream>>>(A->rhs.p, A->n);
  ctx->launches += 2;
  const int ncol = (int)S.color_ptr.size() - 1;
  for (int c = 0; c < ncol; ++c) {
    const int ne = S.color_ptr[c + 1] - S.color_ptr[c];
    if (!ne) continue;
    const int *el = S.color_elems.p + S.color_ptr[c];
    const int grid = (ne + ASM_WARPS - 1) / ASM_WARPS;
    if (S.code == 808)
      k_assemble_elastic_hex<<<(ne + ASM_WARPS * HEX_EPW - 1) / (ASM_WARPS * HEX_EPW), ASM_WARPS * 32, 0, ctx->stream>>>(ne, el, S.elem_nodes.p, S.xyz.p, c12, c44, bf[0],
                                                                        bf[1], bf[2], S.perm.p, S.slots.p, A->values.p,
                                                                        A->rhs.p);
    else
      k_assemble_elastic<504><<<grid, ASM_WARPS * 32, 0, ctx->stream>>>(ne, el, S.elem_nodes.p, S.xyz.p, c12, c44, bf[0],
                                                                        bf[1], bf[2], S.perm.p, S.slots.p, A->values.p,
                                                                        A->rhs.p);
    ctx->launches++;
  }
  EGPU_CUDA_TRY(ctx, cudaGetLastError());
  EGPU_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  A->has_values = true;
  A->has_rhs = true;
  A->ilu_valid = false;
  return EGPU_OK;
}

extern "C" int egpu_dirichlet(egpu_mat *A, int ncon, const int *con_rows, const double *con_vals, int symmetric) {
  if (!A || ncon < 0 || (ncon > 0 && !con_rows)) return EGPU_ERR_ARG;
  egpu_ctx *ctx = A->ctx;
  cudaSetDevice(ctx->device);
  const int n = A->n;
  DevBuf<int> dr;
  DevBuf<double> dv, D, cval;
  DevBuf<unsigned char> cflag;
  EGPU_CUDA_TRY(ctx, cflag.alloc(n));
  EGPU_CUDA_TRY(ctx, cval.alloc(n));
  EGPU_CUDA_TRY(ctx, D.alloc(n));
  EGPU_CUDA_TRY(ctx, cudaMemsetAsync(cflag.p, 0, n, ctx->stream));
  int *err = (int *)(ctx->sync.p + 1);
  EGPU_CUDA_TRY(ctx, cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  if (ncon > 0) {
    EGPU_CUDA_TRY(ctx, dr.alloc(ncon));
    EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(dr.p, con_rows, ncon * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    if (con_vals) {
      EGPU_CUDA_TRY(ctx, dv.alloc(ncon));
      EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(dv.p, con_vals, ncon * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    }
    k_scatter_con<<<grid_of(ctx, ncon), 256, 0, ctx->stream>>>(ncon, dr.p, dv.p, cflag.p, cval.p, n, err);
    ctx->launches++;
  }
  // Linear System Dirichlet Scaling defaults to Linear System Scaling = True
  k_dirichlet_scale_diag<<<grid_of(ctx, n), 256, 0, ctx->stream>>>(n, A->rows.p, A->diag.p, A->values.p, D.p);
  k_dirichlet<<<grid_of(ctx, (long long)n * 8), 256, 0, ctx->stream>>>(n, A->rows.p, A->cols.p, A->diag.p, A->values.p, A->rhs.p, D.p,
                                                        cflag.p, cval.p, symmetric);
  ctx->launches += 2;
  int herr = 0;
  EGPU_CUDA_TRY(ctx, cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  EGPU_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (herr) {
    egpu_set_error(ctx, "Dirichlet row index out of range");
    return EGPU_ERR_ARG;
  }
  A->ilu_valid = false;
  return EGPU_OK;
}
