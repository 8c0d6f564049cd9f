// pg_ctx.h -- the context behind the C ABI's opaque pg_ctx (internal to libpigfem_b200).
//
// A pg_ctx owns every device buffer of one problem: geometry, topology, the cut-element
// quadrature tables, the CSR structure and values of the four blocks, the residual, the
// committed and trial internal variables, the cut-element scratch and the solver workspace.
#pragma once

#include "pg_device.cuh"
#include "pg_setup.h"
#include "../../include/pigfem_b200.h"

#include <string>
#include <vector>

// Workspace of the Jacobi-preconditioned CG on K_ff (pg_solver.cu), allocated on first use.
struct PcgWork {
  int cap_rhs = 0, nb = 0, ng = 0;              // right-hand sides of the buffers, blocks, row groups
  int4* grp = nullptr;                          // row groups of K_ff (pg_solver.cu)
  int* gci = nullptr;                           // their column lists
  int4* chunk = nullptr;                        // chunks of groups: a warp's unit of work
  int* part_of = nullptr;                       // nb + 1: the chunks of each block
  double* dinv = nullptr;                       // n: inverse diagonal of K_ff
  double *r = nullptr, *p = nullptr, *q = nullptr, *xi = nullptr;   // n x cap_rhs each, interleaved
  double* part = nullptr;                       // partial sums: 3 x cap_rhs x nb
  double* sc = nullptr;                         // scalars per rhs (see pg_solver.cu)
  int* flag = nullptr;                          // per rhs: done, iterations; then the solve's words
  unsigned* bar = nullptr;                      // grid barrier arrivals
  int* hflag = nullptr;                         // pinned host copies of flag (two launches in flight)
  cudaStream_t stream = nullptr;
  cudaEvent_t ev = nullptr, evc[2] = {nullptr, nullptr};
  int stage_values = 0;                         // most values of a chunk (pg_debug_set; 0: a stage's)
  int wait_ms = 0, missing = 0;                 // limit of the kernel's waits (0: the default), arrivals its barriers wait for in vain
  int shape[5] = {0, 0, 0, 0, 0};               // blocks, chunks, most chunks of a warp, its ring's stages, chunks read directly
};

struct pg_ctx {
  pg::Setup s;
  std::string err;
  cudaStream_t stream = 0;
  std::vector<void*> allocs;
  std::vector<size_t> alloc_bytes;   // bytes of allocs[i]
  size_t dev_bytes = 0, dev_bytes_peak = 0;   // held now / most held at once (pg_device_bytes)
  pgd::DevProblem P{};
  double* d_U = nullptr;
  double* d_isv_committed = nullptr;
  double* d_isv_trial = nullptr;
  uint8_t* d_zone = nullptr;
  int* d_err = nullptr;
  double* d_red = nullptr;  // residual norm: the count of finished blocks, then their partials
  double* h_norm = nullptr; // its result (pinned host memory the kernel writes)
  long long cut_scratch = 0;   // doubles of the cut elements' set-up blocks (released after set-up)
  int n_coh_qp = 0;
  bool assembled = false;
  bool timed_last = false;   // the last assembly recorded every timing event (pg_kernel_times)
  int fail_alloc = 0;        // the allocation from here on that fails (pg_debug_set; 0: none)
  int fail_launch = 0;       // likewise the residual norm's launch
  double prep_ms = -1.0;   // device time of the preprocessing passes (pg_create_prep_device), -1 if none ran
  // PG_KEEP_STATIC: the first CSR value of each block from which a later assembly can change
  // values (the rows of DOFs of nodes on cohesive elements; nnz when no value can change), and
  // the host arrays (and precision) the last full copy of K went to
  long long changing_from[4] = {0, 0, 0, 0};
  double* kept[4] = {nullptr, nullptr, nullptr, nullptr};
  bool kept_fp32 = false, kept_valid = false;
  std::vector<int> fast_dn, slow_dn;
  const int* cut_list[2] = {nullptr, nullptr};
  int n_cut_list[2] = {0, 0};
  int cut_cls_qp[2] = {1, 1}, cut_cls_nodes[2] = {1, 1};
  bool timing = false;
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};   // start, cohesive, structured, general done, end
  PcgWork pcg;
  // material sensitivity pass (pg_sens.cu): made on its first call
  struct SensWork {
    bool ready = false;
    double* uncut = nullptr;   // per element: NPE x DIM values
    double* cut = nullptr;     // per cut-element node: DIM values
    double* dD = nullptr;      // 2 materials x 5 parameters x 36
    double* g = nullptr;       // the cut elements' point gradients (unmerged)
    int* g_off = nullptr;
    int* pt_off = nullptr;     // a call's point lists
    double* pt_w = nullptr;
    int* pt_g = nullptr;
  } sens;
  double* d_hom = nullptr;  // homogenization partials
  // Device memory comes from the stream-ordered pool on this stream (cudaMallocAsync /
  // cudaFreeAsync): creating and destroying contexts does not synchronise the device, so other
  // contexts' work in flight (the serving loop) keeps running.
  cudaStream_t up = nullptr;
};

// Whether the context's tables are on the device (pg_create, or pg_create_host then pg_upload);
// every entry point that launches work checks it first, so a host-only context gets
// PG_ERR_STATE instead of kernels on null pointers.
inline bool pg_resident(const pg_ctx* c) { return c && c->P.X != nullptr && c->d_err != nullptr; }

// The allocation stream of a context (created on first use).
int pg_alloc_stream(pg_ctx* c);

// Shared helpers of the translation units of the library.
int pg_set_err(pg_ctx* c, int code, const std::string& m);
// Record a device allocation of the context (freed by pg_destroy, or earlier by pg_untrack_free).
inline void pg_track_alloc(pg_ctx* c, void* p, size_t bytes) {
  c->allocs.push_back(p);
  c->alloc_bytes.push_back(bytes);
  c->dev_bytes += bytes;
  if (c->dev_bytes > c->dev_bytes_peak) c->dev_bytes_peak = c->dev_bytes;
}
// Free one tracked allocation early (stream-ordered on the allocation stream).
inline void pg_untrack_free(pg_ctx* c, void* p) {
  for (size_t i = 0; i < c->allocs.size(); ++i)
    if (c->allocs[i] == p) {
      c->dev_bytes -= c->alloc_bytes[i];
      c->allocs.erase(c->allocs.begin() + i);
      c->alloc_bytes.erase(c->alloc_bytes.begin() + i);
      cudaFreeAsync(p, c->up);
      return;
    }
}

// Zero-filled device array of n T on the context's allocation stream; ready for other streams
// after pg_alloc_sync(c).
template <typename T>
int pg_dalloc(pg_ctx* c, size_t n, T** out) {
  *out = nullptr;
  if (n == 0) n = 1;
  if (int rc = pg_alloc_stream(c)) return rc;
  void* p = nullptr;
  const bool fail = c->fail_alloc > 0 && --c->fail_alloc == 0;
  if (fail || cudaMallocAsync(&p, n * sizeof(T), c->up) != cudaSuccess) {
    cudaGetLastError();   // (reported here; a later call's check is for its own launches)
    return pg_set_err(c, PG_ERR_DEVICE, "device allocation failed");
  }
  pg_track_alloc(c, p, n * sizeof(T));
  cudaMemsetAsync(p, 0, n * sizeof(T), c->up);
  *out = (T*)p;
  return 0;
}
int pg_alloc_sync(pg_ctx* c);


