// pg_launch.cuh -- the launches of one assembly, one set-up pass and one multi-strain residual
// pass for a given dimension.  Instantiated once per dimension (pg_launch2.cu, pg_launch3.cu) so
// the two sets of kernels compile in separate translation units; pg_capi.cu calls them through
// the declarations below.
#pragma once

#include "pg_ctx.h"
#include "pg_rows.cuh"

namespace pgl {

// The kernels of one assembly (cohesive elements, rows) on the context's stream; P is the launch's
// problem view.
template <int DIM>
void assembly(pg_ctx* c, const pgd::DevProblem& P);
// Set-up: the cut elements' volumetric blocks and macroscale-strain responses, on the allocation
// stream.
template <int DIM>
void cut_volumetric(pg_ctx* c, const pgd::DevProblem& P, double* gmac);
// Set-up: the static image of the general rows (k_general_static) on the allocation stream, after
// cut_volumetric.
template <int DIM>
void general_static(pg_ctx* c, const pgd::DevProblem& P, double* stat, double* stat_g);
// The residuals of P.n_cases macroscale strains (pg_residual_strains) on the context's stream.
template <int DIM>
void residual_cases(pg_ctx* c, const pgd::DevProblem& P);
// Set-up: the shape constants (k_shape_consts) into out (host).  0, or 1 when a CUDA call fails.
template <int DIM>
int shape_consts(pg_ctx* c, const pgd::DevProblem& P, double* out);

#ifdef PG_LAUNCH_IMPL
// The rows of one pass; `dependent`: a programmatic dependent launch of the cohesive elements'
// kernel before it (the rows that do not need its output run beside it).
template <int DIM, bool CASES>
void rows(const pgd::DevProblem& P, pgd::RowParts parts, bool dependent, cudaStream_t st) {
  const int blocks = parts.total();
  if (blocks == 0) return;
  parts.spread();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(pgd::kRowThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 1 : 0;
  auto launch = [&](auto per) {
    constexpr int PER = decltype(per)::value;
    const bool coh = P.n_coh_el > 0;
    if constexpr (!CASES) {
      if (P.flags & PG_JAC) {
        if (coh) cudaLaunchKernelEx(&cfg, pgd::k_rows<DIM, PER, false, true, true>, P, parts);
        else cudaLaunchKernelEx(&cfg, pgd::k_rows<DIM, PER, false, true, false>, P, parts);
        return;
      }
    }
    if (coh) cudaLaunchKernelEx(&cfg, pgd::k_rows<DIM, PER, CASES, false, true>, P, parts);
    else cudaLaunchKernelEx(&cfg, pgd::k_rows<DIM, PER, CASES, false, false>, P, parts);
  };
  if (DIM == 2 && P.npe == 4) launch(pgd::IntC<36>{});
  else launch(pgd::IntC<pgd::pattern_period(DIM, DIM + 1)>{});
}

template <int DIM>
bool cohesive(pg_ctx* c, const pgd::DevProblem& P) {
  if (P.n_coh_el == 0) return false;
  const int lanes = pgd::CohLanes<DIM>::CQ;
  pgd::k_coh_elements<DIM><<<(int)(((long long)P.n_coh_el * lanes + 127) / 128), 128, 0, c->stream>>>(P);
  return true;
}

template <int DIM>
void assembly(pg_ctx* c, const pgd::DevProblem& P) {
  const pgd::RowParts all = pgd::row_parts(P, (P.flags & PG_JAC) != 0, (P.flags & PG_FUNC) != 0, false);
  c->timed_last = c->timing;
  if (!c->timing) {
    const bool dep = cohesive<DIM>(c, P);
    rows<DIM, false>(P, all, dep, c->stream);
    return;
  }
  // timed: the kinds of rows one after another, with events between them
  cudaEventRecord(c->ev[0], c->stream);
  cohesive<DIM>(c, P);
  cudaEventRecord(c->ev[1], c->stream);
  rows<DIM, false>(P, {{0, all.n[1], 0, all.n[3]}, false, 0}, false, c->stream);
  cudaEventRecord(c->ev[2], c->stream);
  rows<DIM, false>(P, {{all.n[0], 0, all.n[2], 0}, false, 0}, false, c->stream);
  cudaEventRecord(c->ev[3], c->stream);
  cudaEventRecord(c->ev[4], c->stream);
}

template <int DIM>
void cut_volumetric(pg_ctx* c, const pgd::DevProblem& P, double* gmac) {
  for (int cls = 0; cls < 2; ++cls) {
    const int n = c->n_cut_list[cls];
    if (n == 0) continue;
    const size_t smem = (size_t)pgd::cut_smem_doubles(c->cut_cls_qp[cls], c->cut_cls_nodes[cls], DIM) * sizeof(double);
    cudaFuncSetAttribute(pgd::k_cut_volumetric<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    pgd::k_cut_volumetric<DIM><<<n, 64, smem, c->up>>>(P, c->cut_list[cls], n, gmac);
  }
}

template <int DIM>
void general_static(pg_ctx* c, const pgd::DevProblem& P, double* stat, double* stat_g) {
  if (P.n_slow_dn > 0) pgd::k_general_static<DIM><<<(P.n_slow_dn + 127) / 128, 128, 0, c->up>>>(P, stat, stat_g);
}

template <int DIM>
void residual_cases(pg_ctx* c, const pgd::DevProblem& P) {
  // the cohesive elements once (openings, laws, internal variables, tractions: U only), then the
  // rows, each for every case
  const bool dep = cohesive<DIM>(c, P);
  rows<DIM, true>(P, pgd::row_parts(P, false, true, true), dep, c->stream);
}

template <int DIM>
int shape_consts(pg_ctx* c, const pgd::DevProblem& P, double* out) {
  const pg::ProblemDesc& d = c->s.desc;
  double h[3] = {0.0, 0.0, 0.0};
  for (int i = 0; i < DIM; ++i) h[i] = (d.hi[i] - d.lo[i]) / d.n[i];
  const size_t bytes = (size_t)pgd::shape_count(DIM, P.npe) * 3 * pgd::shape_doubles(DIM, P.npe) * sizeof(double);
  double* dout = nullptr;
  if (cudaMallocAsync(&dout, bytes, c->up) != cudaSuccess) return 1;
  if constexpr (DIM == 2) {
    if (P.npe == 4) pgd::k_shape_consts<2, 4><<<1, 32, 0, c->up>>>(P, h[0], h[1], 0.0, dout);
    else pgd::k_shape_consts<2, 3><<<1, 32, 0, c->up>>>(P, h[0], h[1], 0.0, dout);
  } else {
    pgd::k_shape_consts<3, 4><<<1, 32, 0, c->up>>>(P, h[0], h[1], h[2], dout);
  }
  cudaMemcpyAsync(out, dout, bytes, cudaMemcpyDeviceToHost, c->up);
  cudaFreeAsync(dout, c->up);
  return cudaStreamSynchronize(c->up) != cudaSuccess;
}

#define PG_INSTANTIATE_LAUNCHES(D)                                                     \
  template void assembly<D>(pg_ctx*, const pgd::DevProblem&);                          \
  template void cut_volumetric<D>(pg_ctx*, const pgd::DevProblem&, double*);           \
  template void general_static<D>(pg_ctx*, const pgd::DevProblem&, double*, double*);  \
  template void residual_cases<D>(pg_ctx*, const pgd::DevProblem&);                    \
  template int shape_consts<D>(pg_ctx*, const pgd::DevProblem&, double*);
#endif

}  // namespace pgl
