// pg_kernels.cuh -- element-level kernels and their set-up (the rows are in pg_rows.cuh).
//
//   coh_element      one lane per cohesive quadrature point, the lanes of an element together:
//                    opening delta = R sum_n N_n (U+ - U-), the traction-separation law with its
//                    internal-variable update and damage zone, and the element's cohesive blocks
//                    and tractions (src/Utilities.cpp:528-594).  FP64.
//   k_cut_volumetric run once at set-up: the cut elements' volumetric (linear, state-independent)
//                    element matrices from sub-element quadrature with enriched B-matrices
//                    (src/Assembler.cpp:223-274), cached for every later assembly.  FP64.
//   k_general_static run once at set-up: the static image of the rows pg_rows.cuh calls general.
// No atomics anywhere: every row has one owner and sums in a fixed order, so results are
// bit-reproducible from run to run.
#pragma once

#include "pg_device.cuh"

namespace pgd {

template <int N> struct IntC { static constexpr int value = N; };

// Geometry of an affine simplex (tri3 / tet4): physical gradients g[n][d] and the Jacobian
// determinant.  Jac(a,i) = sum_n dN_n/dr_a x_n[i] (Elem::transform_gradients), i.e. x_{a+1} - x_0;
// inverse = adjugate * (1/det) (Utilities::inverse).
template <int DIM, typename T>
__device__ __forceinline__ void simplex_geom(const T (*x)[DIM], T (*g)[DIM], T* J) {
  if (DIM == 2) {
    const T j00 = x[1][0] - x[0][0], j01 = x[1][1] - x[0][1];
    const T j10 = x[2][0] - x[0][0], j11 = x[2][1] - x[0][1];
    const T det = j00 * j11 - j01 * j10;
    const T s = T(1) / det;
    const T i00 = j11 * s, i11 = j00 * s, i01 = (T(-1) * j01) * s, i10 = (T(-1) * j10) * s;
    g[0][0] = -(i00 + i01); g[0][1] = -(i10 + i11);
    g[1][0] = i00; g[1][1] = i10;
    g[2][0] = i01; g[2][1] = i11;
    *J = det;
  } else {
    T a[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int i = 0; i < 3; ++i) a[r][i] = x[r + 1][i] - x[0][i];
    const T det = a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1]) - a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0]) +
                  a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]);
    T R[3][3];
    R[0][0] = a[1][1] * a[2][2] - a[2][1] * a[1][2];
    R[0][1] = T(-1) * (a[0][1] * a[2][2] - a[2][1] * a[0][2]);
    R[0][2] = a[0][1] * a[1][2] - a[1][1] * a[0][2];
    R[1][0] = T(-1) * (a[1][0] * a[2][2] - a[2][0] * a[1][2]);
    R[1][1] = a[0][0] * a[2][2] - a[2][0] * a[0][2];
    R[1][2] = T(-1) * (a[0][0] * a[1][2] - a[1][0] * a[0][2]);
    R[2][0] = a[1][0] * a[2][1] - a[2][0] * a[1][1];
    R[2][1] = T(-1) * (a[0][0] * a[2][1] - a[2][0] * a[0][1]);
    R[2][2] = a[0][0] * a[1][1] - a[1][0] * a[0][1];
    const T s = T(1) / det;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      g[1][i] = R[i][0] * s; g[2][i] = R[i][1] * s; g[3][i] = R[i][2] * s;
      g[0][i] = -(g[1][i] + g[2][i] + g[3][i]);
    }
    *J = det;
  }
}

// sigma = D eps with the linear-elastic zero pattern (LinearElasticIsotropicMaterial::computeStress)
template <int DIM, typename T>
__device__ __forceinline__ void lei_stress(const T* D, const T* e, T* s) {
  if (DIM == 2) {
    s[0] = D[0] * e[0] + D[1] * e[1];
    s[1] = D[3] * e[0] + D[4] * e[1];
    s[2] = D[8] * e[2];
  } else {
    s[0] = D[0] * e[0] + D[1] * e[1] + D[2] * e[2];
    s[1] = D[6] * e[0] + D[7] * e[1] + D[8] * e[2];
    s[2] = D[12] * e[0] + D[13] * e[1] + D[14] * e[2];
    s[3] = D[21] * e[3];
    s[4] = D[28] * e[4];
    s[5] = D[35] * e[5];
  }
}

// Row q of B_a^T D for node gradient ga ("part" of the reference's SmallStrainKFast).
template <int DIM, typename T>
__device__ __forceinline__ void bt_d_row(const T* D, const T* ga, int q, T* part) {
  if (DIM == 2) {
    if (q == 0) { part[0] = ga[0] * D[0] + ga[1] * D[6]; part[1] = ga[0] * D[1] + ga[1] * D[7]; part[2] = ga[0] * D[2] + ga[1] * D[8]; }
    else        { part[0] = ga[1] * D[3] + ga[0] * D[6]; part[1] = ga[1] * D[4] + ga[0] * D[7]; part[2] = ga[1] * D[5] + ga[0] * D[8]; }
  } else {
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      if (q == 0) part[v] = ga[0] * D[0 * 6 + v] + ga[2] * D[4 * 6 + v] + ga[1] * D[5 * 6 + v];
      else if (q == 1) part[v] = ga[1] * D[1 * 6 + v] + ga[2] * D[3 * 6 + v] + ga[0] * D[5 * 6 + v];
      else part[v] = ga[2] * D[2 * 6 + v] + ga[1] * D[3 * 6 + v] + ga[0] * D[4 * 6 + v];
    }
  }
}
// (part . B_b)(:, q2)
template <int DIM, typename T>
__device__ __forceinline__ T part_b(const T* part, const T* gb, int q2) {
  if (DIM == 2) return (q2 == 0) ? part[0] * gb[0] + part[2] * gb[1] : part[1] * gb[1] + part[2] * gb[0];
  if (q2 == 0) return part[0] * gb[0] + part[4] * gb[2] + part[5] * gb[1];
  if (q2 == 1) return part[1] * gb[1] + part[3] * gb[2] + part[5] * gb[0];
  return part[2] * gb[2] + part[3] * gb[1] + part[4] * gb[0];
}
// (B_a^T sigma)[q]
template <int DIM, typename T>
__device__ __forceinline__ T bt_sig(const T* ga, const T* s, int q) {
  if (DIM == 2) return (q == 0) ? ga[0] * s[0] + ga[1] * s[2] : ga[1] * s[1] + ga[0] * s[2];
  if (q == 0) return ga[0] * s[0] + ga[2] * s[4] + ga[1] * s[5];
  if (q == 1) return ga[1] * s[1] + ga[2] * s[3] + ga[0] * s[5];
  return ga[2] * s[2] + ga[1] * s[3] + ga[0] * s[4];
}
// Voigt strain of a set of nodes
template <int DIM, typename T>
__device__ __forceinline__ void add_strain(const T* g, const T* u, T* e) {
  if (DIM == 2) {
    e[0] += g[0] * u[0]; e[1] += g[1] * u[1]; e[2] += g[1] * u[0] + g[0] * u[1];
  } else {
    e[0] += g[0] * u[0]; e[1] += g[1] * u[1]; e[2] += g[2] * u[2];
    e[3] += g[2] * u[1] + g[1] * u[2];
    e[4] += g[2] * u[0] + g[0] * u[2];
    e[5] += g[1] * u[0] + g[0] * u[1];
  }
}

// Weight sum of the reference rules for the uncut parents: tri3 order 3 and tet4 order 3.
__device__ __host__ inline double tri4_wsum() { return ((-0.28125 + 0.260416666666666666666666666666665) + 0.260416666666666666666666666666665) + 0.260416666666666666666666666666665; }
__device__ __host__ inline double tet5_wsum() { return (((-0.8 + 0.45) + 0.45) + 0.45) + 0.45; }

// Point qp of the quad4 2 x 2 Gauss rule (src/quad4.cpp:108-127: the edge points -+1/sqrt(3),
// qp -> (qp % 2, qp / 2), weights 1 x 1) on the bilinear map of the nodes x: the physical
// gradients g of the four shape functions (Jacobian J(a, i) = sum_k dN_k/dr_a x_k[i], its
// inverse by the adjugate, Elem::transform_gradients, src/elem.cpp:115-139) and the weight J W.
__device__ __forceinline__ void quad4_point(const double (*x)[2], int qp, double (*g)[2], double* w) {
  const double kG = 0.57735026918962576450914878050196;
  const double r = (qp % 2) ? kG : -kG, s = (qp / 2) ? kG : -kG;
  const double dN[4][2] = {{-0.25 * (1.0 - s), -0.25 * (1.0 - r)}, {0.25 * (1.0 - s), -0.25 * (1.0 + r)},
                           {0.25 * (1.0 + s), 0.25 * (1.0 + r)}, {-0.25 * (1.0 + s), 0.25 * (1.0 - r)}};
  double J[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) J[a][i] += dN[k][a] * x[k][i];
  const double det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
  const double sc = 1.0 / det;
  const double R[2][2] = {{J[1][1] * sc, (-1.0 * J[0][1]) * sc}, {(-1.0 * J[1][0]) * sc, J[0][0] * sc}};
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int i = 0; i < 2; ++i) g[k][i] = R[i][0] * dN[k][0] + R[i][1] * dN[k][1];
  *w = det * (1.0 * 1.0);
}

// Rows of node la of an uncut element with corner coordinates x, added to blk (row q at blk + q *
// pitch, node b's columns at b * DIM): sum over its points of w (B_la^T D B_b); and its
// macroscale-strain response w (B_la^T D) added to G (DIM x NV).  Simplices have constant gradients,
// so their order-3 points are summed into one weight; quad4 sums its four Gauss points first.
template <int DIM, int NPE>
__device__ __forceinline__ void element_rows(const double (*x)[DIM], int la, const double* D, double* blk, int pitch, double* G) {
  constexpr int NV = (DIM == 2) ? 3 : 6;
  if constexpr (DIM == 2 && NPE == 4) {
    double kb[2][8], gs[2][3];
    for (int q = 0; q < 2; ++q) {
      for (int i = 0; i < 8; ++i) kb[q][i] = 0.0;
      for (int v = 0; v < 3; ++v) gs[q][v] = 0.0;
    }
    for (int qp = 0; qp < 4; ++qp) {
      double g[4][2], w;
      quad4_point(x, qp, g, &w);
      for (int q = 0; q < 2; ++q) {
        double part[3];
        bt_d_row<2, double>(D, g[la], q, part);
        for (int b = 0; b < 4; ++b)
          for (int q2 = 0; q2 < 2; ++q2) kb[q][b * 2 + q2] += w * part_b<2, double>(part, g[b], q2);
        for (int v = 0; v < 3; ++v) gs[q][v] += w * part[v];
      }
    }
    for (int q = 0; q < 2; ++q) {
      for (int i = 0; i < 8; ++i) blk[q * pitch + i] += kb[q][i];
      for (int v = 0; v < 3; ++v) G[q * 3 + v] += gs[q][v];
    }
  } else {
    double g[NPE][DIM], J;
    simplex_geom<DIM, double>(x, g, &J);
    const double wgt = J * ((DIM == 2) ? tri4_wsum() : tet5_wsum());
    for (int q = 0; q < DIM; ++q) {
      double part[NV];
      bt_d_row<DIM, double>(D, g[la], q, part);
      for (int b = 0; b < NPE; ++b)
        for (int q2 = 0; q2 < DIM; ++q2) blk[q * pitch + b * DIM + q2] += wgt * part_b<DIM, double>(part, g[b], q2);
      for (int v = 0; v < NV; ++v) G[q * NV + v] += wgt * part[v];
    }
  }
}

// Set-up: the static image of the general rows, one thread per node: each adjacent element's block
// row (a cut element's from its volumetric matrix K_vol, k_cut_volumetric; an uncut one's formed
// here) added into the node's rows, and its macroscale-strain response into the node's sum, in
// entry order (cut elements first).  A node's image is laid out like its CSR rows: row q at q * (DIM
// x slots), slot s's columns at s * DIM.  stat and stat_g start at zero.
template <int DIM>
__global__ void __launch_bounds__(128) k_general_static(DevProblem P, double* stat, double* stat_g) {
  constexpr int NV = (DIM == 2) ? 3 : 6;
  constexpr int D2 = DIM * DIM;
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= P.n_slow_dn) return;
  const int4 gd = __ldg(&P.gdesc[node]);
  const int pitch = gd.w * DIM;
  double* S = stat + (size_t)__ldg(&P.gnd[2 * node]).x * D2;
  double* Gs = stat_g + (size_t)node * DIM * NV;
  bool bad = false;
  for (int e = 0; e < gd.y; ++e) {
    const int4 ad = __ldg(&P.adesc[gd.x + e]);
    const int4 ax = __ldg(&P.aresd[gd.x + e]);
    const int la = ad.y & 255, mn = ad.y >> 8;
    if (mn == 0) {
      const int nd[4] = {ax.x, ax.y, ax.z, ax.w};
      auto add = [&](auto npe) {
        constexpr int NPE = decltype(npe)::value;
        double x[NPE][DIM], blk[DIM * NPE * DIM];
        for (int n = 0; n < NPE; ++n) load_node<DIM>(P.X, nd[n], x[n]);
        for (int i = 0; i < DIM * NPE * DIM; ++i) blk[i] = 0.0;
        element_rows<DIM, NPE>(x, la, P.Dd + ad.w * 36, blk, NPE * DIM, Gs);
        for (int q = 0; q < DIM; ++q)
          for (int b = 0; b < NPE; ++b)
            for (int d = 0; d < DIM; ++d) S[q * pitch + ((ad.z >> (8 * b)) & 255) * DIM + d] += blk[(q * NPE + b) * DIM + d];
      };
      if (DIM == 2 && P.npe == 4) { if constexpr (DIM == 2) add(IntC<4>{}); }
      else add(IntC<DIM + 1>{});
      continue;
    }
    const int cc = ax.x;
    const double* kr = P.ke + __ldg(&P.ke_off[cc]) + (size_t)la * mn * D2;   // block row la of K_vol
    for (int b = 0; b < mn; ++b) {
      double* o = S + __ldg(&P.adj_slots[ad.z + b]) * DIM;
      for (int q = 0; q < DIM; ++q)
        for (int d = 0; d < DIM; ++d) o[q * pitch + d] += kr[b * D2 + q * DIM + d];
    }
    const double* gm = P.gmac + (size_t)__ldg(&P.re_off[cc]) / DIM * DIM * NV + (size_t)la * DIM * NV;
#pragma unroll
    for (int i = 0; i < DIM * NV; ++i) Gs[i] += gm[i];
  }
  for (int i = 0; i < pitch * DIM; ++i) bad |= !isfinite(S[i]);
  if (bad) atomicOr(P.err, ERR_NONFINITE);
}

// Cohesive elements, one lane per quadrature point (CQ lanes per element: 2 in 2D for CohEdge2, 4
// in 3D for CohTri3 / CohQuad4).  Lane qi forms the opening delta = R sum_n N_n (U+ - U-) of its
// point, runs the traction-separation law with its internal-variable update and damage zone
// (src/Utilities.cpp:528-594, the Material_*Cohesive* files) and forms w R^T D R and w R^T T; the
// lanes then exchange these by shuffles and each writes some of the element's blocks
// B_ab = sum_qp N_a N_b w R^T D R (a, b < nh) and tractions t_a = sum_qp N_a w R^T T (sums in point
// order) to the scratch at kc_off[ce].  The element's stiffness block (n1, n2) is
// sgn * B_{n1 % nh, n2 % nh} and its internal force at n1 is sgn * t_{n1 % nh}, the signs following
// cohesiveKFast / cohesiveInternalForceFast.  Every lane of the warp must call it (valid = false
// for lanes past the last element).
template <int DIM>
struct CohLanes { static constexpr int CQ = (DIM == 2) ? 2 : 4; };

template <int DIM>
__device__ __forceinline__ void coh_element(const DevProblem& P, int ce, int qi, bool valid) {
  constexpr int D2 = DIM * DIM;
  constexpr int CQ = CohLanes<DIM>::CQ;
  const int lane = threadIdx.x & 31, base_lane = lane & ~(CQ - 1);
  int4 d4 = make_int4(0, 0, 0, 0);
  int nh = 0, nq = 0;
  if (valid) {
    d4 = __ldg(&P.cdesc[2 * ce]);
    const int4 e4 = __ldg(&P.cdesc[2 * ce + 1]);
    nh = e4.x;
    nq = min(CQ, e4.y);
  }
  const int q0 = d4.y;
  double W[D2], Tr[DIM];
#pragma unroll
  for (int i = 0; i < D2; ++i) W[i] = 0.0;
#pragma unroll
  for (int i = 0; i < DIM; ++i) Tr[i] = 0.0;
  bool bad = false;
  if (valid && qi < nq) {
    const int* gn = P.coh_gnode + d4.x;   // the element's node ids
    const int cq = q0 + qi;
    const double* N = P.cqp_N + d4.z + qi * nh;
    // (every load below depends on the descriptor alone, except U and the internal variables)
    const int iv = (P.coh.nvar > 0) ? __ldg(&P.cqp_isv[cq]) : 0;
    const double w = __ldg(&P.cqp_wgt[cq]);
    double R[D2];
#pragma unroll
    for (int i = 0; i < D2; ++i) R[i] = __ldg(&P.cqp_R[(size_t)cq * D2 + i]);
    double d0[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) d0[d] = 0.0;
    constexpr int NH = (DIM == 2) ? 2 : 4;   // nodes of a side, at most
    int np[NH], nm[NH];
    double Nn[NH], up[NH][DIM], um[NH][DIM];
#pragma unroll
    for (int n = 0; n < NH; ++n)
      if (n < nh) { nm[n] = __ldg(&gn[n]); np[n] = __ldg(&gn[n + nh]); Nn[n] = __ldg(&N[n]); }
#pragma unroll
    for (int n = 0; n < NH; ++n)
      if (n < nh) { load_node<DIM>(P.U, np[n], up[n]); load_node<DIM>(P.U, nm[n], um[n]); }
#pragma unroll
    for (int n = 0; n < NH; ++n)
      if (n < nh)
#pragma unroll
        for (int d = 0; d < DIM; ++d) d0[d] += Nn[n] * (up[n][d] - um[n][d]);
    double dl[DIM], T[DIM], Dc[D2];
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) s += R[i * DIM + j] * d0[j];
      dl[i] = s;
    }
    double isv[2] = {0.0, 0.0};
    for (int v = 0; v < P.coh.nvar; ++v) isv[v] = P.isv_committed[iv + v];
    uint8_t z;
    coh_law(P.coh, DIM, dl, T, Dc, isv, &z);
    for (int v = 0; v < P.coh.nvar; ++v) P.isv_trial[iv + v] = isv[v];
    P.zone[cq] = z;
    double RtD[D2];
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < DIM; ++j) s += R[j * DIM + i] * Dc[j * DIM + k];
        RtD[i * DIM + k] = s;
      }
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
      for (int l = 0; l < DIM; ++l) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; ++k) s += RtD[i * DIM + k] * R[k * DIM + l];
        W[i * DIM + l] = w * s;
        bad |= !isfinite(s);
      }
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) s += R[j * DIM + i] * T[j];
      Tr[i] = w * s;
      bad |= !isfinite(s);
    }
  }
  // every point's w R^T D R and w R^T T to every lane of the element
  double Wa[CQ][D2], Ta[CQ][DIM];
#pragma unroll
  for (int j = 0; j < CQ; ++j) {
#pragma unroll
    for (int i = 0; i < D2; ++i) Wa[j][i] = __shfl_sync(0xffffffffu, W[i], base_lane + j);
#pragma unroll
    for (int i = 0; i < DIM; ++i) Ta[j][i] = __shfl_sync(0xffffffffu, Tr[i], base_lane + j);
  }
  if (bad) atomicOr(P.err, ERR_NONFINITE);
  if (!valid) return;
  double* out = P.kcoh + d4.w;
  for (int p = qi; p < nh * nh; p += CQ) {
    const int a = p / nh, b = p - a * nh;
    double blk[D2];
#pragma unroll
    for (int i = 0; i < D2; ++i) blk[i] = 0.0;
#pragma unroll
    for (int j = 0; j < CQ; ++j) {
      if (j >= nq) break;
      const double* N = P.cqp_N + d4.z + j * nh;
      const double nn = __ldg(&N[a]) * __ldg(&N[b]);
#pragma unroll
      for (int i = 0; i < D2; ++i) blk[i] += nn * Wa[j][i];
    }
#pragma unroll
    for (int i = 0; i < D2; ++i) out[p * D2 + i] = blk[i];
  }
  for (int a = qi; a < nh; a += CQ) {
    double t[DIM];
#pragma unroll
    for (int i = 0; i < DIM; ++i) t[i] = 0.0;
#pragma unroll
    for (int j = 0; j < CQ; ++j) {
      if (j >= nq) break;
      const double na = __ldg(&P.cqp_N[d4.z + j * nh + a]);
#pragma unroll
      for (int i = 0; i < DIM; ++i) t[i] += na * Ta[j][i];
    }
#pragma unroll
    for (int i = 0; i < DIM; ++i) out[nh * nh * D2 + a * DIM + i] = t[i];
  }
}

// State-independent part of the cut elements, computed once at set-up: the volumetric element
// matrix K_vol = sum over sub-element points of w B_i^T D B_j with the enriched gradients
// (src/Assembler.cpp:223-274; the bulk law is linear, so this block does not change between
// assemblies) and the macroscale-strain response G_i = sum w B_i^T D (R_i = K_vol,i U +
// G_i eps_macro).  One block per cut element, one thread per node pair; the element's gradients,
// weights and materials are staged in shared memory.  Blocks go to the cache in (i, j) block
// order so a block row is contiguous.  FP64.
__host__ __device__ inline int cut_smem_doubles(int nq, int mn, int dim) { return nq * mn * dim + 2 * nq + 3 * 36 + 8; }
template <int DIM>
__global__ void __launch_bounds__(64) k_cut_volumetric(DevProblem P, const int* __restrict__ list, int n_list, double* gmac) {
  constexpr int NV = (DIM == 2) ? 3 : 6;
  extern __shared__ double sm[];
  if ((int)blockIdx.x >= n_list) return;
  const int c = __ldg(&list[blockIdx.x]);
  const int mn = __ldg(&P.cut_node_off[c + 1]) - __ldg(&P.cut_node_off[c]);
  const int q0 = __ldg(&P.cut_qp_off[c]), q1 = __ldg(&P.cut_qp_off[c + 1]);
  const int nq = q1 - q0;
  double* sg = sm;
  double* sw = sg + (size_t)nq * mn * DIM;
  double* smat = sw + nq;
  double* sD = smat + nq;
  const int gbase = __ldg(&P.qp_grad_off[q0]);
  for (int i = threadIdx.x; i < nq * mn * DIM; i += blockDim.x) sg[i] = __ldg(&P.qp_grad[gbase + i]);
  for (int i = threadIdx.x; i < nq; i += blockDim.x) { sw[i] = __ldg(&P.qp_wgt[q0 + i]); smat[i] = (double)__ldg(&P.qp_mat[q0 + i]); }
  for (int i = threadIdx.x; i < 108; i += blockDim.x) sD[i] = __ldg(&P.Dd[i]);
  __syncthreads();
  double* kout = P.ke + __ldg(&P.ke_off[c]);
  bool bad = false;
  for (int p = threadIdx.x; p < mn * mn; p += blockDim.x) {
    const int i = p / mn, j = p - i * mn;
    double kb[DIM][DIM];
#pragma unroll
    for (int x = 0; x < DIM; ++x)
#pragma unroll
      for (int y = 0; y < DIM; ++y) kb[x][y] = 0.0;
    for (int qq = 0; qq < nq; ++qq) {
      const double w = sw[qq];
      const double* D = sD + 36 * (int)smat[qq];
      const double* gi = sg + ((size_t)qq * mn + i) * DIM;
      const double* gj = sg + ((size_t)qq * mn + j) * DIM;
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        double part[NV];
        bt_d_row<DIM, double>(D, gi, q, part);
#pragma unroll
        for (int q2 = 0; q2 < DIM; ++q2) kb[q][q2] += w * part_b<DIM, double>(part, gj, q2);
      }
    }
    double* o = kout + (size_t)p * DIM * DIM;
#pragma unroll
    for (int x = 0; x < DIM; ++x)
#pragma unroll
      for (int y = 0; y < DIM; ++y) { o[x * DIM + y] = kb[x][y]; bad |= !isfinite(kb[x][y]); }
  }
  double* gout = gmac + (size_t)__ldg(&P.re_off[c]) / DIM * DIM * NV;
  for (int i = threadIdx.x; i < mn; i += blockDim.x) {
    double gacc[DIM][NV];
#pragma unroll
    for (int q = 0; q < DIM; ++q)
#pragma unroll
      for (int v = 0; v < NV; ++v) gacc[q][v] = 0.0;
    for (int qq = 0; qq < nq; ++qq) {
      const double* gi = sg + ((size_t)qq * mn + i) * DIM;
      const double* D = sD + 36 * (int)smat[qq];
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        double part[NV];
        bt_d_row<DIM, double>(D, gi, q, part);
#pragma unroll
        for (int v = 0; v < NV; ++v) gacc[q][v] += sw[qq] * part[v];
      }
    }
#pragma unroll
    for (int q = 0; q < DIM; ++q)
#pragma unroll
      for (int v = 0; v < NV; ++v) gout[((size_t)i * DIM + q) * NV + v] = gacc[q][v];
  }
  if (bad) atomicOr(P.err, ERR_NONFINITE);
}

}  // namespace pgd
