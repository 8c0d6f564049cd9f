// pg_rows.cuh -- the rows of the matrix and of the residual.
//
// Every bulk law is linear elastic, so the volumetric part of a row does not depend on the state.
// Two kinds of rows:
//
// Structured rows (the stencil nodes of pg_stencil.cuh whose adjacent elements all have one
// material).  All elements of the uniform grid are one of a few shapes, so the rows of such a node
// are constants of its class and material, summed once per mesh from the shapes' element matrices
// in adjacency order.  Consecutive nodes' rows are one run of the CSR whose values repeat with a
// short period (tri3: a class-0 node's two rows of 18 and a class-1 node's two of 10, 56 values;
// quad4: 36; tet4: 135, taken twice so that the period is even), so
//   write_chunk   a warp writes up to a few hundred consecutive CSR values from the pattern, in
//                 16-byte stores: the matrix is written at memory speed, with nothing read;
//   node_resid    a thread per node multiplies the rows with the displacements of the neighbours
//                 (and adds the macroscale-strain response).
//
// General rows (boundary nodes, nodes of cut elements, enrichment nodes): the set-up sums each
// node's cut and uncut elements' rows into a static image, laid out like its CSR rows
// ([row][neighbour slot][component], k_general_static), and
//   gen_node      a group of lanes per node reads the image once, multiplies it with the
//                 displacements, adds the cohesive blocks and tractions (from the cohesive
//                 elements' pass) and writes the node's rows.
//
// One launch for the cohesive elements and one for all rows.  Forming every element once per tile
// and summing records (the design before) was bound by barriers and shared-memory traffic; a
// 512 x 512 tri3 RVE with 200 fibers (K and R) took 68 us and takes 35, a 64 x 64 linear one 25 and
// 6.1 (one launch instead of two with four events), K and six residuals of 64^3 tet4 503 and 177.
//
// Every value is a sum in a fixed order: results are bit-reproducible, and a residual-only or a
// batched assembly forms the bits of the full single one (multiply-adds are explicit, so none are
// contracted differently from one kernel to the next).
#pragma once

#include "pg_stencil.cuh"

namespace pgd {

// Programmatic dependent launch: k_rows starts while the cohesive elements' kernel before it runs;
// griddepcontrol.wait returns once that grid has completed and its writes are visible.  Only the
// rows of nodes on cohesive elements read them, and only those wait.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" :::); }

constexpr int kRowThreads = 256;     // a block of the row kernels
constexpr int kChunkValues = 960;    // most CSR values of a chunk (30 per lane)

// ---------------------------------------------------------------- structured rows
// Pattern period of an element type (npe: nodes per element).
__host__ __device__ constexpr int pattern_period(int dim, int npe) { return dim == 3 ? 270 : (npe == 4 ? 36 : 56); }
// Doubles of one class's rows in the residual coefficients ([row][slot][component]).
__host__ __device__ constexpr int row_coefs(int dim) { return dim == 3 ? 135 : 36; }

// Chunk: {first CSR value of K_ff, values, first pattern entry, material | 4 when always FP64}.
// The pattern tables hold, per precision and material, the pattern and the pattern shifted by one
// (for chunks that start on an odd value, whose first value is stored by itself), so the 16-byte
// loads and stores are aligned.  The tables are a few KB, read through the L1.
template <int PER>
__device__ __forceinline__ void write_chunk(const DevProblem& P, int4 ch, int lane) {
  const int m = ch.w & 3;
  const int prec = ((P.flags & FLAG_FP32) && !(ch.w & 4)) ? 1 : 0;
  const int odd = ch.x & 1;
  const double* pat = P.pat + ((prec * 3 + m) * 2 + odd) * PER;
  double* dst = P.val[0] + ch.x;
  if (odd && lane == 0) *dst = __ldg(&P.pat[(prec * 3 + m) * 2 * PER + ch.z]);
  const int left = ch.y - odd;
  double2* d2 = reinterpret_cast<double2*>(dst + odd);
  int k = (ch.z + 2 * lane) % PER;
  constexpr int STEP = 64 % PER;
#pragma unroll 4
  for (int e = lane; e < (left >> 1); e += 32) {
    d2[e] = __ldg(reinterpret_cast<const double2*>(pat + k));
    k += STEP;
    if (k >= PER) k -= PER;
  }
  if ((left & 1) && lane == 0) dst[ch.y - 1] = __ldg(&pat[(ch.z + left - 1) % PER]);
}

// Rows of a stencil node times the displacements of its neighbours.
template <class S, int DIM>
__device__ __forceinline__ void stencil_product(const DevProblem& P, const double* __restrict__ c, int nid, double* r) {
  const int sx = P.nx + 1, sxy = sx * (P.ny + 1);
#pragma unroll
  for (int q = 0; q < DIM; ++q) r[q] = 0.0;
#pragma unroll
  for (int s = 0; s < S::NN; ++s) {
    double u[DIM];
    load_node<DIM>(P.U, nid + S::off(s, 0) + S::off(s, 1) * sx + S::off(s, 2) * sxy, u);
#pragma unroll
    for (int q = 0; q < DIM; ++q)
#pragma unroll
      for (int d = 0; d < DIM; ++d) r[q] = __fma_rn(__ldg(&c[(q * S::NN + s) * DIM + d]), u[d], r[q]);
  }
}

// Residual of stencil node v = {node id, first DOF, -, class | material << 4}: its rows' product
// and the macroscale response; CASES: once per strain of a multi-strain pass.
template <int DIM, bool CASES>
__device__ __forceinline__ void node_resid(const DevProblem& P, int4 v) {
  constexpr int NV = (DIM == 2) ? 3 : 6, NC = (DIM == 2) ? 2 : 1;
  const int cls = v.w & 15, m = v.w >> 4;
  const double* c = P.srow + (m * NC + cls) * row_coefs(DIM);
  double r[DIM];
  if constexpr (DIM == 3) stencil_product<Tet4Stencil0, 3>(P, c, v.x, r);
  else if (cls == 0) stencil_product<Tri3Stencil0, 2>(P, c, v.x, r);   // (quad4: the same neighbours)
  else stencil_product<Tri3Stencil1, 2>(P, c, v.x, r);
  const double* g = P.sg + (m * NC + cls) * DIM * NV;
  if constexpr (CASES) {
    for (int k = 0; k < P.n_cases; ++k)
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        double t = r[q];
#pragma unroll
        for (int w = 0; w < NV; ++w) t = __fma_rn(__ldg(&g[q * NV + w]), P.eps_cases[k][w], t);
        P.Pf_cases[(size_t)k * P.n_free + v.y + q] = t;
      }
  } else {
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
      if (P.subscale)
#pragma unroll
        for (int w = 0; w < NV; ++w) r[q] = __fma_rn(__ldg(&g[q * NV + w]), P.eps_macro[w], r[q]);
      P.Pf[v.y + q] = r[q];
    }
  }
}

// ---------------------------------------------------------------- general rows
// Lanes per general node: 2D a lane takes neighbour slots (a pair of columns), 3D columns.
template <int DIM> struct GenLanes { static constexpr int L = (DIM == 2) ? 8 : 16; };

// Where value (row q, column j of the node's rows) goes for a node whose rows or neighbours are
// partly constrained: the row's F or C block, after the columns of the same kind before it.
template <int DIM>
__device__ __forceinline__ double* irregular_dst(const DevProblem& P, int node, int q, int slot, int d) {
  const int4 gd = __ldg(&P.gdesc[node]);
  const int mk = __ldg(&P.dn_nbr_mask[gd.z + slot]), pre = __ldg(&P.nbr_pre[gd.z + slot]);
  const int* rd = P.growd + (size_t)node * 3 * DIM;
  const bool rf = __ldg(&rd[q]) < P.n_free;
  const int before = __popc(mk & ((1 << d) - 1));
  if (mk & (1 << d)) return P.val[rf ? 0 : 2] + __ldg(&rd[DIM + q]) + pre + before;
  return P.val[rf ? 1 : 3] + __ldg(&rd[2 * DIM + q]) + (slot * DIM - pre) + (d - before);
}

// General node `node` (P.gnd[2 node], P.gnd[2 node + 1]: {first static slot, slots | regular << 16,
// first CSR value of K_ff (regular), first DOF (regular)}, {first traction, tractions, -, -}) by a
// group of L lanes, lane g.  T: slots (2D) or columns (3D) of a lane in flight.  JAC: its rows of the matrix; FUNC: its residual entries; CASES: the
// residuals of a multi-strain pass.  COH: a node on a cohesive element (its cohesive blocks and
// tractions come from the cohesive elements' kernel).  Called by whole groups.
template <int DIM, bool COH, bool CASES, bool JAC, int T>
__device__ __forceinline__ void gen_node(const DevProblem& P, int node, bool func) {
  constexpr int L = GenLanes<DIM>::L, D2 = DIM * DIM, NV = (DIM == 2) ? 3 : 6;
  const int g = threadIdx.x % L;
  const unsigned gmask = ((1u << L) - 1u) << ((threadIdx.x & 31) / L * L);
  const int4 a = __ldg(&P.gnd[2 * node]);
  const int nn = a.y & 0xffff;
  const bool regular = (a.y >> 16) != 0;
  const int pitch = nn * DIM;
  const double* S = P.stat + (size_t)a.x * D2;
  double r[DIM];
#pragma unroll
  for (int q = 0; q < DIM; ++q) r[q] = 0.0;
  // T slots (2D) or columns (3D) of a lane at a time: every load that depends on the descriptor
  // alone is issued before the first one is used
  if constexpr (DIM == 2) {
    for (int k0 = g; k0 < nn; k0 += T * L) {
      double b[T][4];
      int id[T], c0[T], c1[T], cl[T];
      double u[T][2];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int k = k0 + t * L;
        if (k >= nn) break;
        const double2 s0 = __ldg(reinterpret_cast<const double2*>(S) + k);
        const double2 s1 = __ldg(reinterpret_cast<const double2*>(S + pitch) + k);
        b[t][0] = s0.x; b[t][1] = s0.y; b[t][2] = s1.x; b[t][3] = s1.y;
        if (func) id[t] = __ldg(&P.stat_node[a.x + k]);
        if constexpr (COH && JAC) { c0[t] = __ldg(&P.gblk_cl[a.x + k]); c1[t] = __ldg(&P.gblk_cl[a.x + k + 1]); }
      }
#pragma unroll
      for (int t = 0; t < T; ++t) {
        if (k0 + t * L >= nn) break;
        if (func) load_node<2>(P.U, id[t], u[t]);
        if constexpr (COH && JAC) cl[t] = (c1[t] > c0[t]) ? __ldg(&P.gcl[c0[t]]) : 0;
      }
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int k = k0 + t * L;
        if (k >= nn) break;
        double* e = b[t];
        if (func) {
          r[0] = __fma_rn(e[1], u[t][1], __fma_rn(e[0], u[t][0], r[0]));
          r[1] = __fma_rn(e[3], u[t][1], __fma_rn(e[2], u[t][0], r[1]));
        }
        if constexpr (!JAC) continue;
        if constexpr (COH) {
          if (c1[t] > c0[t]) dep_wait();
          int c = cl[t];
          for (int j = c0[t]; j < c1[t]; ++j) {
            const int next = (j + 1 < c1[t]) ? __ldg(&P.gcl[j + 1]) : 0;
            const double sgn = (c & 1) ? -1.0 : 1.0;
            const double2* B = reinterpret_cast<const double2*>(P.kcoh + (c >> 1));
            const double2 t0 = B[0], t1 = B[1];
            e[0] = __fma_rn(sgn, t0.x, e[0]);
            e[1] = __fma_rn(sgn, t0.y, e[1]);
            e[2] = __fma_rn(sgn, t1.x, e[2]);
            e[3] = __fma_rn(sgn, t1.y, e[3]);
            c = next;
          }
        }
        if (regular) {
          double* v = P.val[0] + a.z + 2 * k;
          if ((a.z & 1) == 0) {   // (the pitch is even: both rows are aligned, or neither)
            *reinterpret_cast<double2*>(v) = make_double2(e[0], e[1]);
            *reinterpret_cast<double2*>(v + pitch) = make_double2(e[2], e[3]);
          } else {
            v[0] = e[0];
            v[1] = e[1];
            v[pitch] = e[2];
            v[pitch + 1] = e[3];
          }
        } else {
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int d = 0; d < 2; ++d) *irregular_dst<2>(P, node, q, k, d) = e[q * 2 + d];
        }
      }
    }
  } else {
    for (int j0 = g; j0 < pitch; j0 += T * L) {
      double b[T][3], u[T];
      int id[T], c0[T], c1[T], cl[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int j = j0 + t * L;
        if (j >= pitch) break;
#pragma unroll
        for (int q = 0; q < 3; ++q) b[t][q] = __ldg(&S[q * pitch + j]);
        if (func) id[t] = __ldg(&P.stat_node[a.x + j / 3]);
        if constexpr (COH && JAC) { c0[t] = __ldg(&P.gblk_cl[a.x + j / 3]); c1[t] = __ldg(&P.gblk_cl[a.x + j / 3 + 1]); }
      }
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int j = j0 + t * L;
        if (j >= pitch) break;
        if (func) u[t] = __ldg(&P.U[(size_t)id[t] * 3 + j % 3]);
        if constexpr (COH && JAC) cl[t] = (c1[t] > c0[t]) ? __ldg(&P.gcl[c0[t]]) : 0;
      }
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int j = j0 + t * L;
        if (j >= pitch) break;
        if (func) {
#pragma unroll
          for (int q = 0; q < 3; ++q) r[q] = __fma_rn(b[t][q], u[t], r[q]);
        }
        if constexpr (!JAC) continue;
        if constexpr (COH) {
          if (c1[t] > c0[t]) dep_wait();
          int c = cl[t];
          for (int i = c0[t]; i < c1[t]; ++i) {
            const int next = (i + 1 < c1[t]) ? __ldg(&P.gcl[i + 1]) : 0;
            const double sgn = (c & 1) ? -1.0 : 1.0;
            const double* B = P.kcoh + (c >> 1) + j % 3;
#pragma unroll
            for (int q = 0; q < 3; ++q) b[t][q] = __fma_rn(sgn, B[3 * q], b[t][q]);
            c = next;
          }
        }
        if (regular) {
          double* v = P.val[0] + a.z + j;
#pragma unroll
          for (int q = 0; q < 3; ++q) v[q * pitch] = b[t][q];
        } else {
#pragma unroll
          for (int q = 0; q < 3; ++q) *irregular_dst<3>(P, node, q, j / 3, j % 3) = b[t][q];
        }
      }
    }
  }
  if (!func) return;
  double tr[DIM];
#pragma unroll
  for (int q = 0; q < DIM; ++q) tr[q] = 0.0;
  if constexpr (COH) {
    const int4 t = __ldg(&P.gnd[2 * node + 1]);
    dep_wait();
    for (int j = t.x + g; j < t.x + t.y; j += L) {
      const int c = __ldg(&P.gnode_tl[j]);
      const double sgn = (c & 1) ? -1.0 : 1.0;
      const double* tp = P.kcoh + (c >> 1);
#pragma unroll
      for (int q = 0; q < DIM; ++q) tr[q] = __fma_rn(sgn, tp[q], tr[q]);
    }
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
      r[q] = __dadd_rn(r[q], __shfl_xor_sync(gmask, r[q], o));
      if constexpr (COH) tr[q] = __dadd_rn(tr[q], __shfl_xor_sync(gmask, tr[q], o));
    }
  // every lane holds the sums: lane g writes row g (of the cases: one (case, row) per lane in turn)
  const double* G = P.stat_g + (size_t)node * DIM * NV;
  for (int e = g; e < (CASES ? P.n_cases * DIM : DIM); e += L) {
    const int q = e % DIM, k = e / DIM;
    double t = r[0], s = tr[0];
#pragma unroll
    for (int i = 1; i < DIM; ++i)
      if (q == i) { t = r[i]; s = tr[i]; }
    if (CASES || P.subscale)
#pragma unroll
      for (int w = 0; w < NV; ++w) t = __fma_rn(__ldg(&G[q * NV + w]), CASES ? P.eps_cases[k][w] : P.eps_macro[w], t);
    if constexpr (COH) t = __dadd_rn(t, s);
    const int dof = regular ? a.w + q : __ldg(&P.growd[(size_t)node * 3 * DIM + q]);
    double* f = CASES ? P.Pf_cases + (size_t)k * P.n_free : P.Pf;
    double* c = CASES ? P.Pp_cases + (size_t)k * P.n_const : P.Pp;
    if (dof < P.n_free) f[dof] = t;
    else c[dof - P.n_free] = t;
  }
}

// ---------------------------------------------------------------- kernels of one assembly
// The cohesive elements (coh_element's lanes); the rows launched after it may start while it runs.
template <int DIM>
__global__ void __launch_bounds__(128) k_coh_elements(DevProblem P) {
  dep_launch();
  constexpr int CQ = CohLanes<DIM>::CQ;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int ce = t / CQ;
  coh_element<DIM>(P, ce, t % CQ, ce < P.n_coh_el);
}

// A block's work: `part` 0 general nodes without cohesive elements, 1 stencil residuals, 2 general
// nodes on cohesive elements, 3 CSR chunks; item `b` of the part.  The whole block calls it.
template <int DIM, int PER, bool CASES, bool JAC, bool COH>
__device__ __forceinline__ void row_block(const DevProblem& P, int part, int b) {
  constexpr int GN = kRowThreads / GenLanes<DIM>::L;
  // 3D lanes take several columns at once (22 x 18 x 25 cohesive tet4: 22 us with three, 27 with
  // one; 64^3 linear 177 with two, 182 with three); 2D ones take one slot, since a second costs
  // blocks per SM (512 x 512 with 200 fibers: 38 us against 35)
  constexpr int T = (DIM == 2) ? 1 : (COH ? 3 : 2);
  const bool func = CASES || (P.flags & FLAG_FUNC) != 0;
  const int t = threadIdx.x;
  if (part == 0) {
    const int node = b * GN + t / GenLanes<DIM>::L;
    if (node < P.n_gen_plain) gen_node<DIM, false, CASES, JAC, T>(P, node, func);
  } else if (part == 1) {
    const int i = b * kRowThreads + t;
    if (i < P.n_snode) {
      const int4 v = __ldg(&P.snode[i]);
      if (v.x >= 0) node_resid<DIM, CASES>(P, v);   // (-1: padding of a class to whole warps)
    }
  } else if (COH && part == 2) {
    const int node = P.n_gen_plain + b * GN + t / GenLanes<DIM>::L;
    if (node < P.n_slow_dn) gen_node<DIM, true, CASES, JAC, T>(P, node, func);
  } else if (JAC && part == 3) {
    const int c = b * (kRowThreads / 32) + (t >> 5);
    if (c < P.n_chunk) write_chunk<PER>(P, __ldg(&P.chunk[c]), t & 31);
  }
}

// Blocks of the parts of an assembly with these outputs.
struct RowParts {
  int n[4];
  bool mixed;
  unsigned long long share;   // structured blocks / all blocks, rounded up to a multiple of 2^-32
  // The part and block of the part that block `b` of the launch takes.  Without cohesive elements the
  // structured rows' blocks (residuals, then chunks) are spread evenly among the general rows', so
  // that the stores of the one run beside the long chains of loads of the other from beginning to
  // end (64^3 tet4, K and R and five residuals: 177 us against 182 part after part).  With them the
  // parts follow one another, the chunks last: they run when the blocks that wait for the cohesive
  // elements are done waiting (512 x 512 tri3 with 200 fibers: 34.7 us against 35.6 spread, 37.9
  // with the waiting blocks last, 37.4 with the chunks first).
  __host__ __device__ int total() const { return n[0] + n[1] + n[2] + n[3]; }
  void spread() {
    const unsigned long long t = (unsigned long long)total(), s = (unsigned long long)(n[1] + n[3]);
    share = t ? ((s << 32) + t - 1) / t : 0;
    mixed = n[2] == 0;
  }
  __host__ __device__ void pick(int b, int* part, int* item) const {
    if (!mixed) {
      *part = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (*part == k && b >= n[k]) { b -= n[k]; *part = k + 1; }
      *item = b;
      return;
    }
    const int before = (int)((unsigned)b * share >> 32);
    if ((int)(((unsigned)b + 1u) * share >> 32) > before) {
      *part = before < n[1] ? 1 : 3;
      *item = before < n[1] ? before : before - n[1];
    } else {
      const int g = b - before;
      *part = g < n[0] ? 0 : 2;
      *item = g < n[0] ? g : g - n[0];
    }
  }
};
inline RowParts row_parts(const DevProblem& P, bool jac, bool func, bool cases) {
  const int gn = kRowThreads / ((P.dim == 2) ? GenLanes<2>::L : GenLanes<3>::L);
  auto up = [](int n, int per) { return (n + per - 1) / per; };
  RowParts r;
  r.n[0] = up(P.n_gen_plain, gn);
  r.n[1] = (func || cases) ? up(P.n_snode, kRowThreads) : 0;
  r.n[2] = up(P.n_slow_dn - P.n_gen_plain, gn);
  r.n[3] = (jac && !cases) ? up(P.n_chunk, kRowThreads / 32) : 0;
  r.spread();
  return r;
}

// The rows of one assembly (COH: of a mesh with cohesive elements).
template <int DIM, int PER, bool CASES, bool JAC, bool COH>
__global__ void __launch_bounds__(kRowThreads) k_rows(DevProblem P, RowParts parts) {
  int part, item;
  parts.pick(blockIdx.x, &part, &item);
  row_block<DIM, PER, CASES, JAC, COH>(P, part, item);
}

// ---------------------------------------------------------------- set-up
// Shape constants of a mesh from the corners of a cell at the origin, one thread (the shapes depend on
// the cell size alone, and a cell at the mesh's own place would round lo + h): per shape and material
// the element matrix in FP64 and with FP32 products ([(la DIM + q)(NPE DIM) + lb DIM + q2]), and the
// macroscale response w B_la^T D ([(la DIM + q) NV + v]).  Shapes: tri3 2 x cell parity + element in
// the cell, quad4 one, tet4 the tet's place in the hex.
__host__ __device__ constexpr int shape_count(int dim, int npe) { return dim == 3 ? 6 : (npe == 4 ? 1 : 4); }
__host__ __device__ constexpr int shape_doubles(int dim, int npe) {
  return 2 * npe * dim * npe * dim + npe * dim * (dim == 2 ? 3 : 6);
}

// Nodes of tri3 shape s as (di, dj) corner offsets of its cell: the union-jack split of
// generate_mesh (cells with even i + j split along (0,0)-(1,1)); shapes 0-3: {(0,0) (1,0) (1,1)},
// {(0,0) (1,1) (0,1)}, {(0,0) (1,0) (0,1)}, {(1,0) (1,1) (0,1)}, two bits per node.
__host__ __device__ constexpr int tri_corner(int s, int n, int c) {
  constexpr unsigned bits = (0u << 0) | (1u << 2) | (3u << 4) | (0u << 6) | (3u << 8) | (2u << 10) |
                            (0u << 12) | (1u << 14) | (2u << 16) | (1u << 18) | (3u << 20) | (2u << 22);
  return (int)((bits >> (2 * (3 * s + n) + c)) & 1u);
}
// Tet tt of the hex split of a cell: the corner number of its node n (corners n0 (0,0,0), n1
// (1,0,0), n2 (1,1,0), n3 (0,1,0), n4 (0,0,1), n5 (1,0,1), n6 (1,1,1), n7 (0,1,1); tets
// {n0 n2 n3 n6}, {n0 n3 n7 n6}, {n0 n7 n4 n6}, {n0 n5 n6 n4}, {n1 n5 n6 n0}, {n1 n6 n2 n0}), a
// nibble per corner.
__host__ __device__ constexpr int tet_corner(int tt, int n) {
  constexpr unsigned long long lo = 0x4650647067306320ull;   // tets 0-3
  constexpr unsigned hi = 0x02610651u;                      // tets 4-5
  return (int)(((tt < 4 ? (lo >> (16 * tt)) : (unsigned long long)(hi >> (16 * (tt - 4)))) >> (4 * n)) & 15u);
}
__host__ __device__ constexpr int corner_bit(int cn, int d) {
  return d == 0 ? (cn == 1 || cn == 2 || cn == 5 || cn == 6) : (d == 1 ? (cn == 2 || cn == 3 || cn == 6 || cn == 7) : cn >= 4);
}

template <int DIM, int NPE>
__global__ void k_shape_consts(DevProblem P, double h0, double h1, double h2, double* out) {
  constexpr int ND = NPE * DIM, NV = (DIM == 2) ? 3 : 6;
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const double h[3] = {h0, h1, h2};
  for (int sh = 0; sh < shape_count(DIM, NPE); ++sh) {
    double x[NPE][DIM];
    for (int n = 0; n < NPE; ++n)
      for (int d = 0; d < DIM; ++d) {
        int o;
        if (DIM == 3) o = corner_bit(tet_corner(sh, n), d);
        else if (NPE == 4) o = (d == 0) ? (n == 1 || n == 2) : (n >= 2);
        else o = tri_corner(sh, n, d);
        x[n][d] = o ? h[d] : 0.0;
      }
    for (int m = 0; m < 3; ++m) {
      double* ke = out + (size_t)(sh * 3 + m) * shape_doubles(DIM, NPE);
      double* kef = ke + ND * ND;
      double* gm = kef + ND * ND;
      for (int i = 0; i < shape_doubles(DIM, NPE); ++i) ke[i] = 0.0;
      if constexpr (DIM == 2 && NPE == 4) {
        for (int la = 0; la < 4; ++la) element_rows<2, 4>(x, la, P.Dd + 36 * m, ke + la * 2 * ND, ND, gm + la * 2 * NV);
        for (int i = 0; i < ND * ND; ++i) kef[i] = ke[i];   // (quad4 has no FP32 products)
      } else {
        double g[NPE][DIM], J;
        simplex_geom<DIM, double>(x, g, &J);
        const double w = J * ((DIM == 2) ? tri4_wsum() : tet5_wsum());
        double d[DIM == 2 ? 5 : 12];
        float df[DIM == 2 ? 5 : 12], gk[NPE][DIM];
        iso_from<DIM, double>(P.Dd + 36 * m, d);
        for (int i = 0; i < (DIM == 2 ? 5 : 12); ++i) df[i] = (float)d[i];
        for (int n = 0; n < NPE; ++n)
          for (int c = 0; c < DIM; ++c) gk[n][c] = (float)g[n][c];
        const float wk = (float)w;
        for (int la = 0; la < NPE; ++la)
          for (int q = 0; q < DIM; ++q) {
            double part[NV];
            float partf[NV];
            part_iso<DIM, double>(d, g[la], q, part);
            part_iso<DIM, float>(df, gk[la], q, partf);
            for (int v = 0; v < NV; ++v) gm[(la * DIM + q) * NV + v] = w * part[v];
            for (int lb = 0; lb < NPE; ++lb)
              for (int q2 = 0; q2 < DIM; ++q2) {
                const int i = (la * DIM + q) * ND + lb * DIM + q2;
                ke[i] = w * part_b<DIM, double>(part, g[lb], q2);
                // (3D rounds the FP64 entry, 2D forms the product in FP32)
                kef[i] = (DIM == 2) ? (double)(wk * part_b<DIM, float>(partf, gk[lb], q2)) : (double)(float)ke[i];
              }
          }
      }
    }
  }
}

}  // namespace pgd
