// pg_capi.cu -- the C ABI (include/pigfem_b200.h): set-up, device residency, launches.
//
// A pg_ctx owns every device buffer of one problem: geometry, topology, the cut-element
// quadrature tables, the CSR structure and values of the four blocks, the residual, the
// committed and trial internal variables and the cut-element scratch.  The caller owns its
// host arrays; pointers are never retained across calls.
#include "pg_ctx.h"
#include "pg_launch.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

namespace {

int set_err(pg_ctx* c, int code, const std::string& m) { return pg_set_err(c, code, m); }

template <typename T>
int upload(pg_ctx* c, const std::vector<T>& h, const T** out) {
  *out = nullptr;
  if (h.empty()) return 0;
  if (int rc = pg_alloc_stream(c)) return rc;
  void* p = nullptr;
  if (cudaMallocAsync(&p, h.size() * sizeof(T), c->up) != cudaSuccess) return set_err(c, PG_ERR_DEVICE, "device allocation failed");
  pg_track_alloc(c, p, h.size() * sizeof(T));
  // pageable source: the call returns once the data is staged, so `h` may go away afterwards
  if (cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, c->up) != cudaSuccess)
    return set_err(c, PG_ERR_DEVICE, "host-to-device copy failed");
  *out = (const T*)p;
  return 0;
}

template <typename T>
int dalloc(pg_ctx* c, size_t n, T** out) { return pg_dalloc(c, n, out); }

#define PG_TRY(x) do { int _e = (x); if (_e) return _e; } while (0)

// Fixed-order sum of squares in one launch: block b reduces the values [b, b + 1) * kNormBlock with a
// fixed tree into part[b]; the block that finishes last sums the partials in block order and writes
// the root to pinned host memory.  Small systems take one block.  (Two launches, a serial sum over
// 256 partials by one thread and a copy took 17 us for 3,000 rows.)
constexpr int kNormThreads = 512, kNormBlock = 8 * kNormThreads;
__device__ __forceinline__ double block_total(double s, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  s = (threadIdx.x < kNormThreads / 32) ? sh[threadIdx.x] : 0.0;
  if (threadIdx.x < 32)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;   // in thread 0
}
__global__ void __launch_bounds__(kNormThreads) k_norm(const double* __restrict__ x, int n, double* part, unsigned* count, double* out) {
  __shared__ double sh[32];
  __shared__ bool last;
  const long long b0 = (long long)blockIdx.x * kNormBlock;
  double v[8], s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const long long i = b0 + k * kNormThreads + threadIdx.x;
    v[k] = (i < n) ? x[i] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s = __fma_rn(v[k], v[k], s);
  s = block_total(s, sh);
  if (gridDim.x > 1) {
    if (threadIdx.x == 0) {
      part[blockIdx.x] = s;
      __threadfence();
      last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kNormThreads) s += __ldcg(&part[i]);
    s = block_total(s, sh);
    if (threadIdx.x == 0) *count = 0;   // ready for the next call on the stream
  }
  if (threadIdx.x == 0) *out = sqrt(s);
}

// The structured rows' constants (pg_rows.cuh): the shapes' element matrices (k_shape_consts) summed
// over a node's adjacent elements in adjacency order, per class and material.
template <class S, int DIM>
void class_rows(int npe, int cls, int m, const std::vector<double>& shapes, bool f32, double* rows, double* g) {
  const int nd = npe * DIM, nv = DIM == 2 ? 3 : 6;
  for (int i = 0; i < DIM * S::NN * DIM; ++i) rows[i] = 0.0;
  for (int i = 0; g && i < DIM * nv; ++i) g[i] = 0.0;
  for (int a = 0; a < S::NADJ; ++a) {
    const int sub = S::ent(a, 3), la = S::ent(a, 4);
    const int sh = (DIM == 3 || npe == 4) ? sub : 2 * ((cls + S::ent(a, 0) + S::ent(a, 1)) & 1) + sub;
    const double* ke = shapes.data() + (size_t)(sh * 3 + m) * pgd::shape_doubles(DIM, npe);
    const double* gm = ke + 2 * nd * nd;
    if (f32) ke += nd * nd;
    for (int q = 0; q < DIM; ++q) {
      for (int lb = 0; lb < npe; ++lb)
        for (int d = 0; d < DIM; ++d)
          rows[(q * S::NN + S::ent(a, 5 + lb)) * DIM + d] += ke[(la * DIM + q) * nd + lb * DIM + d];
      for (int v = 0; g && v < nv; ++v) g[q * nv + v] += gm[(la * DIM + q) * nv + v];
    }
  }
}
int structured_constants(pg_ctx* c) {
  const pg::Setup& s = c->s;
  const int dim = s.dim, npe = s.npe, nv = dim == 2 ? 3 : 6, nc = dim == 2 ? 2 : 1;
  std::vector<double> shapes((size_t)pgd::shape_count(dim, npe) * 3 * pgd::shape_doubles(dim, npe));
  if ((dim == 2 ? pgl::shape_consts<2>(c, c->P, shapes.data()) : pgl::shape_consts<3>(c, c->P, shapes.data())) != 0)
    return set_err(c, PG_ERR_DEVICE, "structured-row constants failed");
  const int per = pgd::pattern_period(dim, npe), nr = pgd::row_coefs(dim);
  std::vector<double> pat((size_t)2 * 3 * 2 * per), srow((size_t)3 * nc * nr, 0.0), sg((size_t)3 * nc * dim * nv, 0.0);
  for (int prec = 0; prec < 2; ++prec)
    for (int m = 0; m < 3; ++m) {
      double rows[2][135];
      double* g = prec == 0 ? sg.data() + (size_t)m * nc * dim * nv : nullptr;
      int len[2] = {0, 0};
      if (dim == 3) {
        class_rows<pgd::Tet4Stencil0, 3>(4, 0, m, shapes, prec == 1, rows[0], g);
        class_rows<pgd::Tet4Stencil0, 3>(4, 0, m, shapes, prec == 1, rows[1], nullptr);
        len[0] = len[1] = 135;
      } else if (npe == 4) {
        class_rows<pgd::Quad4Stencil0, 2>(4, 0, m, shapes, prec == 1, rows[0], g);
        len[0] = 36;
      } else {
        class_rows<pgd::Tri3Stencil0, 2>(3, 0, m, shapes, prec == 1, rows[0], g);
        class_rows<pgd::Tri3Stencil1, 2>(3, 1, m, shapes, prec == 1, rows[1], g ? g + dim * nv : nullptr);
        len[0] = 36;
        len[1] = 20;
      }
      if (prec == 0)
        for (int cls = 0; cls < nc; ++cls) std::copy(rows[cls], rows[cls] + len[cls], srow.begin() + (size_t)(m * nc + cls) * nr);
      std::vector<double> p(rows[0], rows[0] + len[0]);
      p.insert(p.end(), rows[1], rows[1] + len[1]);
      for (int odd = 0; odd < 2; ++odd)
        for (int i = 0; i < per; ++i) pat[((size_t)(prec * 3 + m) * 2 + odd) * per + i] = p[(i + odd) % per];
    }
  PG_TRY(upload(c, pat, &c->P.pat));
  PG_TRY(upload(c, srow, &c->P.srow));
  PG_TRY(upload(c, sg, &c->P.sg));
  return 0;
}

int launch(pg_ctx* c, double t_frac, int flags) {
  if (c->timing && !c->ev[0])
    for (int i = 0; i < 5; ++i) cudaEventCreateWithFlags(&c->ev[i], cudaEventDefault);
  pgd::DevProblem P = c->P;
  P.U = c->d_U;
  P.flags = flags;
  for (int v = 0; v < 6; ++v) P.eps_macro[v] = c->s.desc.eps_macro[v] * t_frac;
  const int dim = c->s.dim;
  if (dim == 2) pgl::assembly<2>(c, P);
  else pgl::assembly<3>(c, P);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(c, PG_ERR_DEVICE, std::string("launch failed: ") + cudaGetErrorString(e));
  return 0;
}

}  // namespace

int pg_set_err(pg_ctx* c, int code, const std::string& m) {
  if (c) c->err = m;
  return code;
}

int pg_alloc_stream(pg_ctx* c) {
  if (c->up) return 0;
  static bool pool_ready = false;
  if (!pool_ready) {
    // keep freed blocks in the pool for the next context instead of returning them to the driver
    int dev = 0;
    cudaMemPool_t pool;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      uint64_t thr = ~0ull;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    pool_ready = true;
  }
  if (cudaStreamCreateWithFlags(&c->up, cudaStreamNonBlocking) != cudaSuccess)
    return pg_set_err(c, PG_ERR_DEVICE, "allocation stream creation failed");
  return 0;
}

int pg_alloc_sync(pg_ctx* c) {
  if (c->up && cudaStreamSynchronize(c->up) != cudaSuccess) return pg_set_err(c, PG_ERR_DEVICE, "device allocation failed");
  return 0;
}

extern "C" {

static int create_host(const pg_problem_desc* d, pg_ctx** out, bool device_prep, bool device_pattern) {
  if (!d || !out) return PG_ERR_INPUT;
  *out = nullptr;
  pg_ctx* c = new pg_ctx;
  pg::ProblemDesc pd;
  pd.elem_type = d->elem_type;
  for (int i = 0; i < 3; ++i) { pd.n[i] = d->n[i]; pd.lo[i] = d->lo[i]; pd.hi[i] = d->hi[i]; }
  const int dim = (d->elem_type == PG_TET4) ? 3 : 2;
  if (d->n_incl < 0 || (d->n_incl > 0 && !d->incl)) { delete c; return PG_ERR_INPUT; }
  pd.incl.assign(d->incl, d->incl + (size_t)d->n_incl * (dim + 1));
  pd.E_matrix = d->E_matrix; pd.nu_matrix = d->nu_matrix; pd.E_fiber = d->E_fiber; pd.nu_fiber = d->nu_fiber;
  pd.coh_law = d->coh_law;
  for (int i = 0; i < 4; ++i) pd.coh[i] = d->coh[i];
  pd.plane_strain = d->plane_strain; pd.subscale = d->subscale;
  for (int i = 0; i < 6; ++i) pd.eps_macro[i] = d->eps_macro[i];
  pd.app_strain = d->app_strain;
  pd.ply_frac = d->ply_frac;
  for (int i = 0; i < 5; ++i) pd.ply[i] = d->ply[i];
  pg::PrepResult pr;
  if (device_prep) {
    std::string why;
    if (pg::device_prep(pd, pr, why)) { c->err = why; *out = c; return PG_ERR_DEVICE; }
    c->prep_ms = pr.valid ? pr.device_ms : -1.0;
    pr.pattern_on_device = pr.valid && device_pattern;
  }
  int rc = pg::build_setup(pd, c->s, device_prep ? &pr : nullptr);
  if (!rc && pr.pattern_on_device) {
    // the adjacency and the CSR pattern on the device too
    std::string why;
    double ms = 0.0;
    const int r2 = pg::device_pattern(c->s, why, &ms);
    if (r2) { c->err = why; *out = c; return r2 == 10 ? PG_ERR_DEVICE : PG_ERR_INPUT; }
    c->prep_ms += ms;
  }
  if (rc) { c->err = c->s.error; *out = c; return rc == 2 ? PG_ERR_INPUT : (rc == 4 ? PG_ERR_UNSUPPORTED : (rc == 7 ? PG_ERR_JACOBIAN : PG_ERR_GEOMETRY)); }
  c->n_coh_qp = (int)c->s.cqp_wgt.size();
  *out = c;
  return 0;
}

int pg_create_host(const pg_problem_desc* d, pg_ctx** out) { return create_host(d, out, false, false); }

int pg_create_prep_device(const pg_problem_desc* d, int passes, pg_ctx** out) {
  if (!(passes & PG_PREP_NODES)) return create_host(d, out, false, false);
  return create_host(d, out, true, (passes & PG_PREP_PATTERN) != 0);
}

int pg_prep_device_ms(const pg_ctx* c, double* ms) {
  if (!c || !ms) return PG_ERR_INPUT;
  *ms = c->prep_ms;
  return 0;
}

int pg_upload(pg_ctx* c) {
  if (!c) return PG_ERR_INPUT;
  pg::Setup& s = c->s;
  const int dim = s.dim;

  // ---- derived row-ownership tables
  const int n_nodes = s.n_std + s.n_enr;
  std::vector<uint8_t> mask(s.n_dn, 0);
  for (int a = 0; a < s.n_dn; ++a) {
    const int na = s.dn_node[a];
    for (int q = 0; q < dim; ++q) if (s.node_dof[(size_t)na * dim + q] < s.n_free) mask[a] |= (uint8_t)(1 << q);
  }
  // neighbour masks, adjacency slots
  std::vector<uint8_t> nbr_mask(s.dn_nbr.size());
  for (size_t k = 0; k < s.dn_nbr.size(); ++k) nbr_mask[k] = mask[s.dn_nbr[k]];
  std::vector<int> slot32(s.dn_adj.size(), 0), slot_off(s.dn_adj.size(), 0);
  std::vector<uint8_t> slots;
  for (int a = 0; a < s.n_dn; ++a) {
    const int* nb = s.dn_nbr.data() + s.dn_nbr_off[a];
    const int nn = s.dn_nbr_off[a + 1] - s.dn_nbr_off[a];
    if (nn > 255) return set_err(c, PG_ERR_UNSUPPORTED, "a DOF node with more than 255 neighbours");
    for (int k = s.dn_adj_off[a]; k < s.dn_adj_off[a + 1]; ++k) {
      const int e = s.dn_adj[k] >> 5, cc = s.cut_of[e];
      const int* en = cc < 0 ? &s.conn[(size_t)e * s.npe] : &s.cut_nodes[s.cut_node_off[cc]];
      const int mn = cc < 0 ? s.npe : s.cut_node_off[cc + 1] - s.cut_node_off[cc];
      int pos[pgd::kMaxNodesCut];
      if (mn > pgd::kMaxNodesCut) return set_err(c, PG_ERR_UNSUPPORTED, "a cut element with more than 32 nodes");
      slot_off[k] = (int)slots.size();
      for (int lb = 0; lb < mn; ++lb) {
        const int db = s.node_dn[en[lb]];
        pos[lb] = (int)(std::lower_bound(nb, nb + nn, db) - nb);
        if (pos[lb] >= nn || nb[pos[lb]] != db) return set_err(c, PG_ERR_STATE, "internal: adjacency without neighbour slot");
        // an element's nodes need distinct slots
        for (int k2 = 0; k2 < lb; ++k2)
          if (pos[k2] == pos[lb]) return set_err(c, PG_ERR_UNSUPPORTED, "an element holds a node and its periodic image");
        if (cc < 0) slot32[k] |= pos[lb] << (8 * lb);
        else slots.push_back((uint8_t)pos[lb]);
      }
    }
  }
  // Structured rows (pg_rows.cuh): DOF nodes inside the grid whose adjacency, neighbours and row
  // layout match their class table exactly, whose elements are all uncut and of one material and
  // whose neighbour DOFs are all free.  Everything else is general.
  std::vector<int4> stencil;   // {node id, first DOF, first CSR value, class | material << 4}
  std::vector<int4> chunks;
  std::vector<int> fast, slow;
  {
    const int Nx = s.desc.n[0], Ny = s.desc.n[1], Nz = (dim == 3) ? s.desc.n[2] : 0;
    const int sx = Nx + 1, sxy = sx * (Ny + 1);
    const bool quad = s.etype == pg::QUAD4;
    const int per_cell = dim == 3 ? 6 : (quad ? 1 : 2);
    std::vector<char> in_stencil(s.n_dn, 0);
    std::vector<int4> by_node;
    int open_next = -1, open_cls = -1;   // the CSR value and class that continue the open chunk
    const int phase_of[2] = {0, 2 * pgd::Tri3Stencil0::NN * 2};
    for (int a = 0; a < s.n_dn; ++a) {
      const int nid = s.dn_node[a];
      if (nid >= s.n_std) continue;
      const int i = nid % sx, j = (nid / sx) % (Ny + 1), k = nid / sxy;
      if (i < 1 || i > Nx - 1 || j < 1 || j > Ny - 1) continue;
      if (dim == 3 && (k < 1 || k > Nz - 1)) continue;
      const int cls = (dim == 2 && !quad) ? ((i + j) % 2) : 0;
      const int NN = dim == 3 ? pgd::Tet4Stencil0::NN : (cls == 0 ? pgd::Tri3Stencil0::NN : pgd::Tri3Stencil1::NN);
      const int NADJ = dim == 3 ? pgd::Tet4Stencil0::NADJ
                                : (quad ? pgd::Quad4Stencil0::NADJ : (cls == 0 ? pgd::Tri3Stencil0::NADJ : pgd::Tri3Stencil1::NADJ));
      auto off = [&](int q, int d) {
        return dim == 3 ? pgd::Tet4Stencil0::off(q, d) : (cls == 0 ? pgd::Tri3Stencil0::off(q, d) : pgd::Tri3Stencil1::off(q, d));
      };
      auto entv = [&](int q, int cidx) {
        if (dim == 3) return pgd::Tet4Stencil0::ent(q, cidx);
        if (quad) return pgd::Quad4Stencil0::ent(q, cidx);
        return cls == 0 ? pgd::Tri3Stencil0::ent(q, cidx) : pgd::Tri3Stencil1::ent(q, cidx);
      };
      bool ok = (s.dn_nbr_off[a + 1] - s.dn_nbr_off[a]) == NN && (s.dn_adj_off[a + 1] - s.dn_adj_off[a]) == NADJ;
      for (int q = 0; ok && q < NN; ++q) {
        const int nb = s.dn_node[s.dn_nbr[s.dn_nbr_off[a] + q]];
        ok = nb == nid + off(q, 0) + off(q, 1) * sx + off(q, 2) * sxy && mask[s.dn_nbr[s.dn_nbr_off[a] + q]] == (1 << dim) - 1;
      }
      int mat = -1;
      for (int q = 0; ok && q < NADJ; ++q) {
        const int ci = i + entv(q, 0), cj = j + entv(q, 1), ck = k + entv(q, 2);
        const int e = per_cell * ((ck * Ny + cj) * Nx + ci) + entv(q, 3);
        const int entry = s.dn_adj[s.dn_adj_off[a] + q];
        ok = (entry >> 5) == e && (entry & 31) == entv(q, 4) && s.cut_of[e] < 0;
        if (ok && mat < 0) mat = s.elem_mat[e];
        ok = ok && s.elem_mat[e] == mat;
        for (int n = 0; ok && n < s.npe; ++n) {
          const int sl = entv(q, 5 + n);
          ok = s.conn[(size_t)e * s.npe + n] == nid + off(sl, 0) + off(sl, 1) * sx + off(sl, 2) * sxy;
        }
      }
      if (!ok) continue;
      const int g0 = s.node_dof[(size_t)nid * dim];
      for (int q = 0; ok && q < dim; ++q) ok = s.node_dof[(size_t)nid * dim + q] == g0 + q && g0 + q < s.n_free;
      if (!ok) continue;
      const int row0 = s.rp[0][g0], len = dim * NN * dim;
      for (int q = 0; ok && q < dim; ++q)
        ok = s.rp[0][g0 + q] == row0 + q * NN * dim && s.rp[0][g0 + q + 1] - s.rp[0][g0 + q] == NN * dim &&
             s.rp[1][g0 + q + 1] == s.rp[1][g0 + q];
      if (!ok) continue;
      in_stencil[a] = 1;
      by_node.push_back(make_int4(nid, g0, row0, cls | (mat << 4)));
      // the FP32-mixed rows are those two cells from the boundary; the ring next to it stays FP64
      const bool ring = i < 2 || i > Nx - 2 || j < 2 || j > Ny - 2 || (dim == 3 && (k < 2 || k > Nz - 2));
      const int kind = mat | (ring ? 4 : 0);
      if (!chunks.empty() && open_next == row0 && chunks.back().w == kind && chunks.back().y + len <= pgd::kChunkValues &&
          (dim == 3 || quad || open_cls != cls)) {
        chunks.back().y += len;
      } else {
        chunks.push_back(make_int4(row0, len, (dim == 2 && !quad) ? phase_of[cls] : 0, kind));
      }
      open_next = row0 + len;
      open_cls = cls;
    }
    // the residual's nodes by class (each padded to whole warps with node -1), so that a warp's
    // nodes share a class
    for (int cls = 0; cls < 2; ++cls) {
      for (const int4& v : by_node) if ((v.w & 15) == cls) stencil.push_back(v);
      while (stencil.size() % 32) stencil.push_back(make_int4(-1, 0, 0, cls));
    }
    for (const int4& v : by_node) fast.push_back(s.node_dn[v.x]);
    // general nodes: those on no cohesive element first, then by their number of neighbours, so
    // that the lane groups of a warp walk alike rows
    std::vector<char> on_coh(s.n_dn, 0);
    for (int cc = 0; cc < s.ncut; ++cc)
      for (int ce = s.cut_coh_off[cc]; ce < s.cut_coh_off[cc + 1]; ++ce)
        for (int q = s.coh_local_off[ce]; q < s.coh_local_off[ce + 1]; ++q)
          on_coh[s.node_dn[s.cut_nodes[s.cut_node_off[cc] + s.coh_local[q]]]] = 1;
    for (int a = 0; a < s.n_dn; ++a) if (!in_stencil[a]) slow.push_back(a);
    std::stable_sort(slow.begin(), slow.end(), [&](int x, int y) {
      if (on_coh[x] != on_coh[y]) return on_coh[x] < on_coh[y];
      return (s.dn_nbr_off[x + 1] - s.dn_nbr_off[x]) > (s.dn_nbr_off[y + 1] - s.dn_nbr_off[y]);
    });
    c->P.n_gen_plain = 0;
    for (int a : slow) c->P.n_gen_plain += !on_coh[a];
    c->P.nx = Nx;
    c->P.ny = Ny;
  }
  // cut-element scratch layout
  std::vector<long long> ke_off(s.ncut + 1, 0);
  std::vector<int> re_off(s.ncut + 1, 0);
  for (int cc = 0; cc < s.ncut; ++cc) {
    const int nd = (s.cut_node_off[cc + 1] - s.cut_node_off[cc]) * dim;
    ke_off[cc + 1] = ke_off[cc] + (long long)nd * nd;
    re_off[cc + 1] = re_off[cc] + nd;
  }
  c->cut_scratch = ke_off[s.ncut];
  c->n_coh_qp = (int)s.cqp_wgt.size();

  // descriptors of the general rows
  std::vector<int4> gdesc, adesc, gnd;
  int stat_slots = 0;
  std::vector<int> growd;
  std::vector<int4> aresd;   // per entry: uncut {element nodes}, cut {cut element, first node, cohesive place, 0}
  for (int a : slow) {
    const int na = s.dn_node[a];
    gdesc.push_back(make_int4((int)adesc.size(), s.dn_adj_off[a + 1] - s.dn_adj_off[a], s.dn_nbr_off[a],
                              s.dn_nbr_off[a + 1] - s.dn_nbr_off[a]));
    int rows[3][3];
    for (int q = 0; q < dim; ++q) {
      const int gq = s.node_dof[(size_t)na * dim + q];
      const bool rf = gq < s.n_free;
      const int rr = rf ? gq : gq - s.n_free;
      rows[0][q] = gq;
      rows[1][q] = rf ? s.rp[0][rr] : s.rp[2][rr];
      rows[2][q] = rf ? s.rp[1][rr] : s.rp[3][rr];
    }
    for (int t = 0; t < 3; ++t) for (int q = 0; q < dim; ++q) growd.push_back(rows[t][q]);
    {
      // regular: every row and neighbour DOF free, so the rows are one run of K_ff
      const int nn = gdesc.back().w, g0 = rows[0][0];
      bool regular = true;
      for (int k = gdesc.back().z; k < gdesc.back().z + nn; ++k) regular = regular && nbr_mask[k] == (1 << dim) - 1;
      for (int q = 0; regular && q < dim; ++q)
        regular = rows[0][q] == g0 + q && g0 + q < s.n_free && rows[1][q] == rows[1][0] + q * nn * dim &&
                  s.rp[0][g0 + q + 1] - s.rp[0][g0 + q] == nn * dim;
      gnd.push_back(make_int4(stat_slots, nn | (regular ? 1 << 16 : 0), regular ? rows[1][0] : 0, regular ? g0 : 0));
      gnd.push_back(make_int4(0, 0, 0, 0));
      stat_slots += nn;
    }
    // cut elements first, then uncut ones, each in adjacency order
    for (int pass = 0; pass < 2; ++pass)
    for (int k = s.dn_adj_off[a]; k < s.dn_adj_off[a + 1]; ++k) {
      const int e = s.dn_adj[k] >> 5, la = s.dn_adj[k] & 31;
      const int cc = s.cut_of[e];
      if ((cc >= 0) != (pass == 0)) continue;
      if (cc < 0) {
        adesc.push_back(make_int4(e, la, slot32[k], s.elem_mat[e]));
        const int* en = &s.conn[(size_t)e * s.npe];
        aresd.push_back(make_int4(en[0], en[1], en[2], s.npe > 3 ? en[3] : -1));
      } else {
        const int mn = s.cut_node_off[cc + 1] - s.cut_node_off[cc];
        adesc.push_back(make_int4(e, la | (mn << 8), slot_off[k], 0));
        // the row node's place on a cohesive element of this cut element: (element << 5 | position)
        int cpa = -1;
        for (int ce = s.cut_coh_off[cc]; ce < s.cut_coh_off[cc + 1] && cpa < 0; ++ce)
          for (int j = s.coh_local_off[ce]; j < s.coh_local_off[ce + 1]; ++j)
            if (s.coh_local[j] == la) { cpa = ce * 32 + (j - s.coh_local_off[ce]); break; }
        aresd.push_back(make_int4(cc, s.cut_node_off[cc], cpa, 0));
      }
    }
  }

  // ---- device residency
  pgd::DevProblem& P = c->P;
  P.dim = dim; P.npe = s.npe;
  P.ne = s.ne; P.ncut = s.ncut; P.n_dn = s.n_dn;
  P.n_free = s.n_free; P.n_const = s.n_const; P.subscale = s.desc.subscale;
  P.coh.law = s.coh.law; P.coh.nvar = s.coh.nvar; P.coh.sigma_c = s.coh.sigma_c; P.coh.delta_c1 = s.coh.delta_c1;
  P.coh.delta_c2 = s.coh.delta_c2; P.coh.delta_cn = s.coh.delta_cn; P.coh.delta_ct = s.coh.delta_ct; P.coh.q = s.coh.q;
  P.coh.delta_c = s.coh.delta_c; P.coh.beta2 = s.coh.beta2; P.coh.alpha = s.coh.alpha; P.coh.delta_c3 = s.coh.delta_c3;
  {
    std::vector<double> Dh(108);
    for (int m = 0; m < 3; ++m) for (int i = 0; i < 36; ++i) Dh[m * 36 + i] = s.D[m][i];
    PG_TRY(upload(c, Dh, &P.Dd));
  }
  if (!stencil.empty()) PG_TRY(structured_constants(c));
  P.n_snode = (int)stencil.size();
  P.n_chunk = (int)chunks.size();
  PG_TRY(upload(c, stencil, &P.snode));
  PG_TRY(upload(c, chunks, &P.chunk));
  PG_TRY(upload(c, s.X, &P.X));
  PG_TRY(upload(c, s.conn, &P.conn));
  PG_TRY(upload(c, s.elem_mat, &P.emat));
  PG_TRY(upload(c, s.cut_of, &P.cut_of));
  PG_TRY(upload(c, s.node_dof, &P.node_dof));
  PG_TRY(upload(c, s.cut_node_off, &P.cut_node_off));
  PG_TRY(upload(c, s.cut_nodes, &P.cut_nodes));
  // Device quadrature tables: the quadrature points of an affine (tri3 / tet4) sub-element of an
  // affine parent share one gradient set, so they are merged into one point carrying the sum of
  // their weights (w_0 + w_1 + ... in rule order).  K and R change only by rounding.
  {
    std::vector<int> dq_off(1, 0), dq_mat, dg_off(1, 0);
    std::vector<double> dq_w, dg;
    for (int cc = 0; cc < s.ncut; ++cc) {
      int qp = s.cut_qp_off[cc];
      for (int sb = s.cut_sub_off[cc]; sb < s.cut_sub_off[cc + 1]; ++sb) {
        const int st = s.sub_type[sb];
        const int nq = s.sub_qp_off[sb + 1] - s.sub_qp_off[sb];
        if (s.sub_qp_off[sb] != qp) return set_err(c, PG_ERR_STATE, "internal: quadrature offsets out of order");
        // (a quad4 parent's gradients vary from point to point, so its sub-elements never merge)
        const bool affine = (st == pg::SUB_TRI3 || st == pg::SUB_TET4) && s.etype != pg::QUAD4;
        if (affine) {
          double w = 0.0;
          for (int q = 0; q < nq; ++q) w += s.qp_wgt[qp + q];
          dq_w.push_back(w);
          dq_mat.push_back(s.qp_mat[qp]);
          dg.insert(dg.end(), s.qp_grad.begin() + s.qp_grad_off[qp], s.qp_grad.begin() + s.qp_grad_off[qp + 1]);
          dg_off.push_back((int)dg.size());
        } else {
          for (int q = 0; q < nq; ++q) {
            dq_w.push_back(s.qp_wgt[qp + q]);
            dq_mat.push_back(s.qp_mat[qp + q]);
            dg.insert(dg.end(), s.qp_grad.begin() + s.qp_grad_off[qp + q], s.qp_grad.begin() + s.qp_grad_off[qp + q + 1]);
            dg_off.push_back((int)dg.size());
          }
        }
        qp += nq;
      }
      if (qp != s.cut_qp_off[cc + 1]) return set_err(c, PG_ERR_STATE, "internal: quadrature count mismatch");
      dq_off.push_back((int)dq_w.size());
    }
    {
      // size classes: at most 8 points and 8 nodes (one fiber: tri3 + quad4 sub-elements), the rest
      std::vector<int> lists[2];
      for (int cc = 0; cc < s.ncut; ++cc) {
        const int nq = dq_off[cc + 1] - dq_off[cc], mn = s.cut_node_off[cc + 1] - s.cut_node_off[cc];
        const int cls = (nq <= 8 && mn <= 8) ? 0 : 1;
        lists[cls].push_back(cc);
        c->cut_cls_qp[cls] = std::max(c->cut_cls_qp[cls], nq);
        c->cut_cls_nodes[cls] = std::max(c->cut_cls_nodes[cls], mn);
      }
      for (int cls = 0; cls < 2; ++cls) {
        PG_TRY(upload(c, lists[cls], &c->cut_list[cls]));
        c->n_cut_list[cls] = (int)lists[cls].size();
      }
    }
    PG_TRY(upload(c, dq_off, &P.cut_qp_off));
    PG_TRY(upload(c, dq_w, &P.qp_wgt));
    PG_TRY(upload(c, dq_mat, &P.qp_mat));
    PG_TRY(upload(c, dg_off, &P.qp_grad_off));
    PG_TRY(upload(c, dg, &P.qp_grad));
  }
  PG_TRY(upload(c, s.cqp_N, &P.cqp_N));
  PG_TRY(upload(c, s.cqp_R, &P.cqp_R));
  PG_TRY(upload(c, s.cqp_wgt, &P.cqp_wgt));
  PG_TRY(upload(c, s.cqp_isv, &P.cqp_isv));
  PG_TRY(upload(c, ke_off, &P.ke_off));
  PG_TRY(upload(c, re_off, &P.re_off));
  // the cut elements' volumetric blocks: set-up only (reduced into the static rows, then released)
  double* dke = nullptr;
  PG_TRY(dalloc(c, (size_t)ke_off[s.ncut], &dke));
  P.ke = dke;
  PG_TRY(dalloc(c, (size_t)s.n_isv, &c->d_isv_committed));
  PG_TRY(dalloc(c, (size_t)s.n_isv, &c->d_isv_trial));
  P.isv_committed = c->d_isv_committed; P.isv_trial = c->d_isv_trial;
  PG_TRY(dalloc(c, (size_t)c->n_coh_qp, &c->d_zone));
  P.zone = c->d_zone;
  PG_TRY(upload(c, s.dn_node, &P.dn_node));
  PG_TRY(upload(c, nbr_mask, &P.dn_nbr_mask));
  PG_TRY(upload(c, s.dn_adj_off, &P.dn_adj_off));
  PG_TRY(upload(c, s.dn_adj, &P.dn_adj));
  PG_TRY(upload(c, slots, &P.adj_slots));
  c->fast_dn = fast;
  c->slow_dn = slow;
  P.n_slow_dn = (int)slow.size();
  PG_TRY(upload(c, gdesc, &P.gdesc));
  PG_TRY(upload(c, growd, &P.growd));
  PG_TRY(upload(c, adesc, &P.adesc));
  PG_TRY(upload(c, aresd, &P.aresd));
  // cohesive elements: owning cut element, scratch offsets of their blocks, and the cohesive
  // position of every cut-element local node (a node is on at most one cohesive element)
  std::vector<int> kc_off_h, cohpos_h;
  {
    const int n_ce = (int)s.coh_nh.size();
    if ((long long)n_ce * 32 > 2147483647LL) return set_err(c, PG_ERR_UNSUPPORTED, "too many cohesive elements");
    std::vector<int> ce_cut(n_ce), kc_off(n_ce + 1, 0), cohpos(s.cut_nodes.size(), -1);
    for (int cc = 0; cc < s.ncut; ++cc)
      for (int ce = s.cut_coh_off[cc]; ce < s.cut_coh_off[cc + 1]; ++ce) {
        ce_cut[ce] = cc;
        const int nh = s.coh_nh[ce];
        if (2 * nh > 32) return set_err(c, PG_ERR_UNSUPPORTED, "cohesive element with more than 32 nodes");
        kc_off[ce + 1] = kc_off[ce] + nh * nh * dim * dim + nh * dim;
        for (int k = 0; k < 2 * nh; ++k) {
          const int ln = s.coh_local[s.coh_local_off[ce] + k];
          int& slot = cohpos[s.cut_node_off[cc] + ln];
          if (slot >= 0) return set_err(c, PG_ERR_STATE, "internal: a node on two cohesive elements of one cut element");
          slot = ce * 32 + k;
        }
      }
    {
      // node ids of the cohesive elements' local nodes, laid out like coh_local
      std::vector<int> gnode(s.coh_local.size());
      for (int ce = 0; ce < n_ce; ++ce)
        for (int k = s.coh_local_off[ce]; k < s.coh_local_off[ce + 1]; ++k)
          gnode[k] = s.cut_nodes[s.cut_node_off[ce_cut[ce]] + s.coh_local[k]];
      PG_TRY(upload(c, gnode, &P.coh_gnode));
    }
    {
      std::vector<int4> cdesc;
      int o = 0;
      for (int ce = 0; ce < n_ce; ++ce) {
        const int nh = s.coh_nh[ce], nq = s.coh_qp_off[ce + 1] - s.coh_qp_off[ce];
        cdesc.push_back(make_int4(s.coh_local_off[ce], s.coh_qp_off[ce], o, kc_off[ce]));
        cdesc.push_back(make_int4(nh, nq, 0, 0));
        o += nh * nq;
      }
      if (o != (int)s.cqp_N.size()) return set_err(c, PG_ERR_STATE, "internal: cohesive shape-value count mismatch");
      PG_TRY(upload(c, cdesc, &P.cdesc));
    }
    kc_off_h = kc_off;
    cohpos_h = cohpos;
    double* dk;
    PG_TRY(dalloc(c, (size_t)kc_off[n_ce], &dk));
    P.kcoh = dk;
    P.n_coh_el = n_ce;
  }
  // row positions: free DOFs of the earlier neighbours of every neighbour slot
  {
    std::vector<int> pre(s.dn_nbr.size(), 0);
    for (int a = 0; a < s.n_dn; ++a) {
      int acc = 0;
      for (int k = s.dn_nbr_off[a]; k < s.dn_nbr_off[a + 1]; ++k) { pre[k] = acc; acc += __builtin_popcount(nbr_mask[k]); }
    }
    PG_TRY(upload(c, pre, &P.nbr_pre));
  }
  for (int b = 0; b < 4; ++b) {
    // (two more than there are: the solver's copies of value ranges end on 16-byte boundaries)
    PG_TRY(dalloc(c, s.ci[b].size() + 2, &P.val[b]));
  }
  // The values a later assembly can change (PG_KEEP_STATIC, pg_changing_values): every bulk law
  // is linear elastic, so only the entries coupling DOFs of nodes on one cohesive element depend
  // on the state; each block's changing values lie in the rows from the smallest such DOF on.
  {
    int fmin = s.n_free, pmin = s.n_const;
    for (int cc = 0; cc < s.ncut; ++cc)
      for (int ce = s.cut_coh_off[cc]; ce < s.cut_coh_off[cc + 1]; ++ce)
        for (int q = s.coh_local_off[ce]; q < s.coh_local_off[ce + 1]; ++q) {
          const int node = s.cut_nodes[s.cut_node_off[cc] + s.coh_local[q]];
          for (int d = 0; d < dim; ++d) {
            const int dof = s.node_dof[(size_t)node * dim + d];
            if (dof < s.n_free) fmin = std::min(fmin, dof);
            else pmin = std::min(pmin, dof - s.n_free);
          }
        }
    const bool fr = fmin < s.n_free, pr = pmin < s.n_const;
    long long nnz[4];
    for (int b = 0; b < 4; ++b) nnz[b] = (long long)s.ci[b].size();
    c->changing_from[0] = fr ? s.rp[0][fmin] : nnz[0];
    c->changing_from[1] = (fr && pr) ? s.rp[1][fmin] : nnz[1];
    c->changing_from[2] = (fr && pr) ? s.rp[2][pmin] : nnz[2];
    c->changing_from[3] = pr ? s.rp[3][pmin] : nnz[3];
    c->kept_valid = false;
  }
  PG_TRY(dalloc(c, (size_t)s.n_free, &P.Pf));
  PG_TRY(dalloc(c, (size_t)s.n_const, &P.Pp));
  PG_TRY(dalloc(c, (size_t)n_nodes * dim, &c->d_U));
  PG_TRY(dalloc(c, 1, &c->d_err));
  P.err = c->d_err;
  PG_TRY(dalloc(c, 2 + (size_t)s.n_free / kNormBlock + 1, &c->d_red));
  // Static image of the general rows (k_general_static), the node ids of its slots, the cohesive
  // contributions of every slot in adjacency order and the nodes' traction lists
  {
    const int nv = (dim == 2) ? 3 : 6, D2 = dim * dim;
    std::vector<int> stat_node, gblk_cl(1, 0), gcl, tl;
    stat_node.reserve(stat_slots);
    gblk_cl.reserve(stat_slots + 1);
    std::vector<std::vector<int>> bcl;
    for (size_t i = 0; i < slow.size(); ++i) {
      const int4 gd = gdesc[i];
      for (int k = gd.z; k < gd.z + gd.w; ++k) stat_node.push_back(s.dn_node[s.dn_nbr[k]]);
      if ((int)i < P.n_gen_plain) {
        gblk_cl.insert(gblk_cl.end(), gd.w, 0);
        continue;
      }
      bcl.assign(gd.w, std::vector<int>());
      gnd[2 * i + 1].x = (int)tl.size();
      for (int k = gd.x; k < gd.x + gd.y; ++k) {
        const int4 ad = adesc[k], ax = aresd[k];
        const int mn = ad.y >> 8;
        if (mn == 0) continue;   // uncut: in the static image
        const int cpa = ax.z;
        if (cpa < 0) continue;
        const int ce = cpa >> 5, n1 = cpa & 31, nh = s.coh_nh[ce];
        for (int b = 0; b < mn; ++b) {
          const int cpb = cohpos_h[ax.y + b];
          if (cpb < 0 || (cpb >> 5) != ce) continue;
          const int n2 = cpb & 31;
          const int off = kc_off_h[ce] + ((n1 % nh) * nh + (n2 % nh)) * D2;
          const int neg = ((n1 >= nh) == (n2 >= nh)) ? 0 : 1;
          bcl[slots[ad.z + b]].push_back(off * 2 + neg);
        }
        const int toff = kc_off_h[ce] + nh * nh * D2 + (n1 % nh) * dim;
        tl.push_back(toff * 2 + ((n1 >= nh) ? 0 : 1));
      }
      for (int k = 0; k < gd.w; ++k) {
        gcl.insert(gcl.end(), bcl[k].begin(), bcl[k].end());
        gblk_cl.push_back((int)gcl.size());
      }
      gnd[2 * i + 1].y = (int)tl.size() - gnd[2 * i + 1].x;
    }
    for (size_t k = 0; k < aresd.size() && P.n_gen_plain > 0; ++k)
      if ((int)k < gdesc[P.n_gen_plain - 1].x + gdesc[P.n_gen_plain - 1].y && (adesc[k].y >> 8) != 0 && aresd[k].z >= 0)
        return set_err(c, PG_ERR_STATE, "internal: a node on a cohesive element among the plain general nodes");
    PG_TRY(upload(c, gnd, &P.gnd));
    PG_TRY(upload(c, stat_node, &P.stat_node));
    PG_TRY(upload(c, gblk_cl, &P.gblk_cl));
    PG_TRY(upload(c, gcl, &P.gcl));
    PG_TRY(upload(c, tl, &P.gnode_tl));
    double* dst = nullptr;
    double* dsg = nullptr;
    PG_TRY(dalloc(c, (size_t)stat_slots * D2, &dst));
    PG_TRY(dalloc(c, slow.size() * dim * nv, &dsg));
    P.stat = dst;
    P.stat_g = dsg;
    double* dg = nullptr;
    if (s.ncut > 0) {
      PG_TRY(dalloc(c, (size_t)re_off[s.ncut] / dim * dim * nv, &dg));
      P.gmac = dg;
      if (dim == 2) pgl::cut_volumetric<2>(c, P, dg);
      else pgl::cut_volumetric<3>(c, P, dg);
    }
    if (dim == 2) pgl::general_static<2>(c, P, dst, dsg);
    else pgl::general_static<3>(c, P, dst, dsg);
    int herr = 0;
    cudaMemcpyAsync(&herr, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->up);
    if (cudaStreamSynchronize(c->up) != cudaSuccess) return set_err(c, PG_ERR_DEVICE, "general-row set-up kernel failed");
    if (herr) return set_err(c, PG_ERR_NONFINITE, "non-finite stiffness at set-up");
    // the per-element blocks are reduced: give their memory back
    pg_untrack_free(c, dke);
    if (dg) pg_untrack_free(c, dg);
    P.ke = nullptr;
    P.gmac = nullptr;
  }
  return pg_alloc_sync(c);
}

int pg_create(const pg_problem_desc* d, pg_ctx** out) {
  int rc = pg_create_host(d, out);
  if (rc) return rc;
  return pg_upload(*out);
}

int pg_debug_array(const pg_ctx* c, const char* name, int64_t* n, const void** ptr) {
  if (!c || !name || !n || !ptr) return 0;
  const pg::Setup& s = c->s;
  struct { const char* k; const void* p; size_t n; int kind; } tab[] = {
      {"cut_elem", s.cut_elem.data(), s.cut_elem.size(), 1}, {"cut_node_off", s.cut_node_off.data(), s.cut_node_off.size(), 1},
      {"cut_nodes", s.cut_nodes.data(), s.cut_nodes.size(), 1}, {"cut_qp_off", s.cut_qp_off.data(), s.cut_qp_off.size(), 1},
      {"qp_wgt", s.qp_wgt.data(), s.qp_wgt.size(), 2}, {"qp_mat", s.qp_mat.data(), s.qp_mat.size(), 1},
      {"qp_grad_off", s.qp_grad_off.data(), s.qp_grad_off.size(), 1}, {"qp_grad", s.qp_grad.data(), s.qp_grad.size(), 2},
      {"cut_coh_off", s.cut_coh_off.data(), s.cut_coh_off.size(), 1}, {"coh_nh", s.coh_nh.data(), s.coh_nh.size(), 1},
      {"coh_local_off", s.coh_local_off.data(), s.coh_local_off.size(), 1}, {"coh_local", s.coh_local.data(), s.coh_local.size(), 1},
      {"coh_qp_off", s.coh_qp_off.data(), s.coh_qp_off.size(), 1}, {"cqp_N", s.cqp_N.data(), s.cqp_N.size(), 2},
      {"cqp_R", s.cqp_R.data(), s.cqp_R.size(), 2}, {"cqp_wgt", s.cqp_wgt.data(), s.cqp_wgt.size(), 2},
      {"cqp_isv", s.cqp_isv.data(), s.cqp_isv.size(), 1}, {"conn", s.conn.data(), s.conn.size(), 1},
      {"elem_mat", s.elem_mat.data(), s.elem_mat.size(), 1}, {"cut_of", s.cut_of.data(), s.cut_of.size(), 1},
      {"node_detect", s.node_detect.data(), s.node_detect.size(), 1}, {"enr_edge", s.enr_edge.data(), s.enr_edge.size(), 1},
      {"enr_incl", s.enr_incl.data(), s.enr_incl.size(), 1}, {"sub_type", s.sub_type.data(), s.sub_type.size(), 1},
      {"cut_sub_off", s.cut_sub_off.data(), s.cut_sub_off.size(), 1}, {"sub_mat", s.sub_mat.data(), s.sub_mat.size(), 1},
      {"fast_dn", c->fast_dn.data(), c->fast_dn.size(), 1}, {"slow_dn", c->slow_dn.data(), c->slow_dn.size(), 1},
      {"dn_node", s.dn_node.data(), s.dn_node.size(), 1}, {"dn_nbr", s.dn_nbr.data(), s.dn_nbr.size(), 1},
      {"dn_nbr_off", s.dn_nbr_off.data(), s.dn_nbr_off.size(), 1}, {"dn_adj", s.dn_adj.data(), s.dn_adj.size(), 1},
      {"dn_adj_off", s.dn_adj_off.data(), s.dn_adj_off.size(), 1}, {"pcg_shape", c->pcg.shape, 5, 1},
  };
  for (auto& t : tab)
    if (std::strcmp(t.k, name) == 0) { *n = (int64_t)t.n; *ptr = t.p; return t.kind; }
  *n = 0; *ptr = nullptr;
  return 0;
}

int pg_debug_set(pg_ctx* c, const char* name, int64_t value) {
  if (!c || !name) return PG_ERR_INPUT;
  if (std::strcmp(name, "pcg_stage_values") == 0) {
    if (value < 0 || value > 0xffff || c->pcg.grp) return set_err(c, PG_ERR_INPUT, "pcg_stage_values: before the first solve, at most 65535");
    c->pcg.stage_values = (int)value;
    return 0;
  }
  if (std::strcmp(name, "pcg_wait_ms") == 0 || std::strcmp(name, "pcg_missing") == 0) {
    if (value < 0 || value > 10000) return set_err(c, PG_ERR_INPUT, "pg_debug_set: value out of range");
    (name[4] == 'w' ? c->pcg.wait_ms : c->pcg.missing) = (int)value;
    return 0;
  }
  if (std::strcmp(name, "fail_alloc") == 0 || std::strcmp(name, "fail_launch") == 0) {
    (name[5] == 'a' ? c->fail_alloc : c->fail_launch) = (int)value;
    return 0;
  }
  return set_err(c, PG_ERR_INPUT, "pg_debug_set: unknown name");
}

int pg_set_timing(pg_ctx* c, int on) {
  if (!c) return PG_ERR_INPUT;
  c->timing = on != 0;
  return 0;
}

int pg_kernel_times(pg_ctx* c, float* ms) {
  if (!c || !ms || !c->ev[0]) return set_err(c, PG_ERR_STATE, "nothing was launched");
  if (!c->timed_last) return set_err(c, PG_ERR_STATE, "the last assembly ran with timing off (pg_set_timing)");
  if (cudaEventSynchronize(c->ev[4]) != cudaSuccess) return set_err(c, PG_ERR_DEVICE, "event wait failed");
  // [0] cohesive elements, [1] structured rows, [2] general rows, [3] whole assembly
  for (int k = 0; k < 3; ++k) cudaEventElapsedTime(&ms[k], c->ev[k], c->ev[k + 1]);
  cudaEventElapsedTime(&ms[3], c->ev[0], c->ev[4]);
  return 0;
}

void pg_destroy(pg_ctx* c) {
  if (!c) return;
  // work of this context still in flight finishes before its memory goes back to the pool
  cudaStreamSynchronize(c->stream);
  if (c->pcg.stream) cudaStreamSynchronize(c->pcg.stream);
  if (c->pcg.stream) cudaStreamDestroy(c->pcg.stream);
  for (cudaEvent_t e : {c->pcg.ev, c->pcg.evc[0], c->pcg.evc[1]}) if (e) cudaEventDestroy(e);
  if (c->pcg.hflag) cudaFreeHost(c->pcg.hflag);
  if (c->h_norm) cudaFreeHost(c->h_norm);
  for (cudaEvent_t e : c->ev) if (e) cudaEventDestroy(e);
  for (void* p : c->allocs) cudaFreeAsync(p, c->up);
  if (c->up) cudaStreamDestroy(c->up);   // released once the frees have run
  delete c;
}

const char* pg_last_error(const pg_ctx* c) { return c ? c->err.c_str() : "null context"; }

int pg_device_bytes(const pg_ctx* c, int64_t* now, int64_t* peak) {
  if (!c) return PG_ERR_INPUT;
  if (now) *now = (int64_t)c->dev_bytes;
  if (peak) *peak = (int64_t)c->dev_bytes_peak;
  return 0;
}

int pg_get_sizes(const pg_ctx* c, pg_sizes* o) {
  if (!c || !o) return PG_ERR_INPUT;
  const pg::Setup& s = c->s;
  o->dim = s.dim; o->n_nodes = s.n_std + s.n_enr; o->n_std_nodes = s.n_std; o->n_enrich_nodes = s.n_enr;
  o->n_elem = s.ne; o->n_cut_elem = s.ncut; o->n_coh_elem = (int)s.coh_nh.size(); o->n_coh_qp = c->n_coh_qp;
  o->n_free = s.n_free; o->n_const = s.n_const; o->n_isv = s.n_isv;
  for (int b = 0; b < 4; ++b) o->nnz[b] = (int64_t)s.ci[b].size();
  o->cut_scratch_doubles = c->cut_scratch;
  return 0;
}

int pg_get_pattern(const pg_ctx* c, int b, int32_t* rowptr, int32_t* cols) {
  if (!c || b < 0 || b > 3) return PG_ERR_INPUT;
  if (rowptr) std::memcpy(rowptr, c->s.rp[b].data(), c->s.rp[b].size() * sizeof(int32_t));
  if (cols && !c->s.ci[b].empty()) std::memcpy(cols, c->s.ci[b].data(), c->s.ci[b].size() * sizeof(int32_t));
  return 0;
}

int pg_get_nodes(const pg_ctx* c, double* coords, int32_t* node_dofs, double* dirichlet) {
  if (!c) return PG_ERR_INPUT;
  if (coords) std::memcpy(coords, c->s.X.data(), c->s.X.size() * sizeof(double));
  if (node_dofs) std::memcpy(node_dofs, c->s.node_dof.data(), c->s.node_dof.size() * sizeof(int32_t));
  if (dirichlet && !c->s.dirichlet.empty()) std::memcpy(dirichlet, c->s.dirichlet.data(), c->s.dirichlet.size() * sizeof(double));
  return 0;
}

int pg_set_stream(pg_ctx* c, void* stream) {
  if (!c) return PG_ERR_INPUT;
  c->stream = (cudaStream_t)stream;
  return 0;
}

int pg_assemble_device(pg_ctx* c, const double* d_U, double t_frac, int flags) {
  if (!c || !d_U) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (reinterpret_cast<uintptr_t>(d_U) % 16) return set_err(c, PG_ERR_INPUT, "the displacement array must be 16-byte aligned");
  if (!(flags & (PG_FUNC | PG_JAC))) return 0;
  double* keep = c->d_U;
  c->d_U = const_cast<double*>(d_U);
  int rc = launch(c, t_frac, flags);
  c->d_U = keep;
  c->assembled = (rc == 0);
  return rc;
}

int pg_residual_strains(pg_ctx* c, const double* d_U, double t_frac, int n_cases, const double* eps, double* d_Rf,
                        double* d_Rp) {
  if (!c || !d_U || !eps || !d_Rf || n_cases < 1 || n_cases > 6) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (reinterpret_cast<uintptr_t>(d_U) % 16) return set_err(c, PG_ERR_INPUT, "the displacement array must be 16-byte aligned");
  if (!c->s.desc.subscale) return set_err(c, PG_ERR_INPUT, "macroscale strain cases need a subscale (periodic) problem");
  if (c->s.etype == pg::QUAD4) return set_err(c, PG_ERR_UNSUPPORTED, "the multi-strain pass takes tri3 / tet4 meshes (quad4: one residual-only assembly per strain)");
  if (c->s.n_const > 0 && !d_Rp) return set_err(c, PG_ERR_INPUT, "d_Rp is required when the problem has constrained DOFs");
  pgd::DevProblem P = c->P;
  P.U = d_U;
  P.flags = PG_FUNC;
  for (int v = 0; v < 6; ++v) P.eps_macro[v] = 0.0;
  P.n_cases = n_cases;
  for (int k = 0; k < n_cases; ++k)
    for (int v = 0; v < 6; ++v) P.eps_cases[k][v] = eps[k * 6 + v] * t_frac;
  P.Pf_cases = d_Rf;
  P.Pp_cases = d_Rp;
  const int dim = c->s.dim;
  if (dim == 2) pgl::residual_cases<2>(c, P);
  else pgl::residual_cases<3>(c, P);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(c, PG_ERR_DEVICE, std::string("launch failed: ") + cudaGetErrorString(e));
  return 0;
}

int pg_assemble(pg_ctx* c, const double* U, double t_frac, int flags, double* Kff, double* Kfp, double* Kpf, double* Kpp,
                double* Pf, double* Pp) {
  if (!c || !U) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (!(flags & (PG_FUNC | PG_JAC))) return 0;
  const pg::Setup& s = c->s;
  const size_t nU = (size_t)(s.n_std + s.n_enr) * s.dim;
  if (cudaMemcpyAsync(c->d_U, U, nU * sizeof(double), cudaMemcpyHostToDevice, c->stream) != cudaSuccess)
    return set_err(c, PG_ERR_DEVICE, "copy of U failed");
  cudaMemsetAsync(c->d_err, 0, sizeof(int), c->stream);
  PG_TRY(launch(c, t_frac, flags));
  double* outs[4] = {Kff, Kfp, Kpf, Kpp};
  if (flags & PG_JAC) {
    // PG_KEEP_STATIC with the same host arrays and precision as the last full copy: only the
    // values that can have changed since (a suffix of each block) go back
    const bool fp32 = (flags & PG_FP32) != 0;
    bool keep = (flags & PG_KEEP_STATIC) && c->kept_valid && c->kept_fp32 == fp32;
    for (int b = 0; b < 4; ++b) keep = keep && outs[b] == c->kept[b];
    for (int b = 0; b < 4; ++b) {
      if (!outs[b] || s.ci[b].empty()) continue;
      const long long from = keep ? c->changing_from[b] : 0, nnz = (long long)s.ci[b].size();
      if (from < nnz)
        cudaMemcpyAsync(outs[b] + from, c->P.val[b] + from, (size_t)(nnz - from) * sizeof(double), cudaMemcpyDeviceToHost,
                        c->stream);
    }
    if (flags & PG_KEEP_STATIC) {
      for (int b = 0; b < 4; ++b) c->kept[b] = outs[b];
      c->kept_fp32 = fp32;
      c->kept_valid = true;
    } else {
      c->kept_valid = false;
    }
  }
  if (flags & PG_FUNC) {
    if (Pf && s.n_free) cudaMemcpyAsync(Pf, c->P.Pf, (size_t)s.n_free * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (Pp && s.n_const) cudaMemcpyAsync(Pp, c->P.Pp, (size_t)s.n_const * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  }
  int herr = 0;
  cudaMemcpyAsync(&herr, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return set_err(c, PG_ERR_DEVICE, std::string("assembly failed: ") + cudaGetErrorString(e));
  c->assembled = true;
  if (herr) return set_err(c, PG_ERR_NONFINITE, "non-finite value in a cut-element matrix or vector");
  return 0;
}

int pg_changing_values(const pg_ctx* c, int64_t* first) {
  if (!c || !first) return PG_ERR_INPUT;
  for (int b = 0; b < 4; ++b) first[b] = (int64_t)c->changing_from[b];
  return 0;
}

int pg_device_outputs(pg_ctx* c, double** K, double** Pf, double** Pp) {
  if (!c) return PG_ERR_INPUT;
  if (K) for (int b = 0; b < 4; ++b) K[b] = c->P.val[b];
  if (Pf) *Pf = c->P.Pf;
  if (Pp) *Pp = c->P.Pp;
  return 0;
}

int pg_set_isv(pg_ctx* c, const double* v) {
  if (!c || (!v && c->s.n_isv)) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (c->s.n_isv == 0) return 0;
  cudaMemcpyAsync(c->d_isv_committed, v, (size_t)c->s.n_isv * sizeof(double), cudaMemcpyHostToDevice, c->stream);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return set_err(c, PG_ERR_DEVICE, "copy of internal variables failed");
  return 0;
}

int pg_get_isv(const pg_ctx* c, int trial, double* out) {
  if (!c || (!out && c->s.n_isv)) return PG_ERR_INPUT;
  if (!pg_resident(c)) return PG_ERR_STATE;
  if (c->s.n_isv == 0) return 0;
  cudaStreamSynchronize(c->stream);
  cudaMemcpyAsync(out, trial ? c->d_isv_trial : c->d_isv_committed, (size_t)c->s.n_isv * sizeof(double), cudaMemcpyDeviceToHost,
                  c->stream);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return PG_ERR_DEVICE;
  return 0;
}

int pg_commit_isv(pg_ctx* c) {
  if (!c) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (c->s.n_isv == 0) return 0;
  cudaMemcpyAsync(c->d_isv_committed, c->d_isv_trial, (size_t)c->s.n_isv * sizeof(double), cudaMemcpyDeviceToDevice, c->stream);
  return cudaStreamSynchronize(c->stream) == cudaSuccess ? 0 : PG_ERR_DEVICE;
}

int pg_get_damage_zones(const pg_ctx* c, uint8_t* z) {
  if (!c || (!z && c->n_coh_qp)) return PG_ERR_INPUT;
  if (!pg_resident(c)) return PG_ERR_STATE;
  if (!c->n_coh_qp) return 0;
  cudaStreamSynchronize(c->stream);
  cudaMemcpyAsync(z, c->d_zone, (size_t)c->n_coh_qp, cudaMemcpyDeviceToHost, c->stream);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return PG_ERR_DEVICE;
  return 0;
}

int pg_set_macro_strain(pg_ctx* c, const double* eps) {
  if (!c || !eps) return PG_ERR_INPUT;
  if (!c->s.desc.subscale) return set_err(c, PG_ERR_STATE, "the macroscale strain applies to subscale (periodic) problems only");
  for (int v = 0; v < 6; ++v) c->s.desc.eps_macro[v] = (v < (c->s.dim == 2 ? 3 : 6)) ? eps[v] : 0.0;
  return 0;
}

int pg_residual_norm(pg_ctx* c, double* out) {
  if (!c || !out) return PG_ERR_INPUT;
  if (!pg_resident(c)) return set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (!c->h_norm && cudaMallocHost(&c->h_norm, sizeof(double)) != cudaSuccess) {
    cudaGetLastError();   // (reported here; a later call's check is for its own launches)
    c->h_norm = nullptr;
    return set_err(c, PG_ERR_DEVICE, "pinned norm allocation failed");
  }
  const int nb = std::max(1, (int)(((long long)c->s.n_free + kNormBlock - 1) / kNormBlock));
  // (without its own status a launch that failed would leave the last call's value to be returned)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nb);
  cfg.blockDim = dim3(kNormThreads);
  cfg.stream = c->stream;
  const bool fail = c->fail_launch > 0 && --c->fail_launch == 0;
  if (fail || cudaLaunchKernelEx(&cfg, k_norm, (const double*)c->P.Pf, c->s.n_free, c->d_red + 1,
                                 reinterpret_cast<unsigned*>(c->d_red), c->h_norm) != cudaSuccess) {
    cudaGetLastError();
    return set_err(c, PG_ERR_DEVICE, "residual norm: launch failed");
  }
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return set_err(c, PG_ERR_DEVICE, "residual norm failed");
  *out = *c->h_norm;
  return 0;
}

}  // extern "C"
