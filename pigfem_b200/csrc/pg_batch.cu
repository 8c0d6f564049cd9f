// pg_batch.cu -- many RVEs in one set of persistent launches, replayed from a CUDA graph.
//
// A batch holds the device descriptors (DevProblem) of n assembled-ready contexts and two work
// lists that cover all of them: blocks of cohesive elements and blocks of rows (pg_rows.cuh's parts:
// general nodes, stencil residuals, CSR chunks), each item {context, part, block, -}.  One assembly
// of the whole batch is two persistent kernels that stride over the lists (the rows a programmatic
// dependent launch of the cohesive elements); the sequence, with the upload of the per-call
// parameters (each context's displacement pointer, flags and macroscale strain) and the read-back
// of the error word, is captured once into a CUDA graph and replayed.  A block copies the
// descriptor of its item's context to shared memory and fills in the call's parameters.  Every CSR
// value and residual entry is formed by the bodies of the single-context launches, so each
// context's results are bitwise those of pg_assemble_device.
//
// The autotuner (pg_batch_tune) times the candidate launch shapes (2 / 4 / 8 / 16 persistent blocks
// per SM) on the batch itself and keeps the fastest.
#include "pg_ctx.h"
#include "pg_rows.cuh"

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace {

struct BatchCall {
  const double* U;
  int flags;
  int pad;
  double eps[6];
};

constexpr int kSMs = 148;

// The item's problem view: the context's descriptor with this call's parameters.  The whole block
// calls it.
__device__ __forceinline__ void load_view(pgd::DevProblem& v, const pgd::DevProblem* items, const BatchCall* call, int i, int* err) {
  static_assert(sizeof(pgd::DevProblem) % sizeof(int) == 0, "copied by words");
  __syncthreads();   // the view of the item before is done with
  const int* src = reinterpret_cast<const int*>(items + i);
  int* dst = reinterpret_cast<int*>(&v);
  for (int k = threadIdx.x; k < (int)(sizeof(pgd::DevProblem) / sizeof(int)); k += blockDim.x) dst[k] = __ldg(&src[k]);
  __syncthreads();
  if (threadIdx.x < 6) v.eps_macro[threadIdx.x] = call[i].eps[threadIdx.x];
  if (threadIdx.x == 6) { v.U = call[i].U; v.flags = call[i].flags; v.err = err; }
  __syncthreads();
}

// item = {context, first cohesive element, -, -}: 256 / CQ cohesive elements
template <int DIM>
__global__ void __launch_bounds__(pgd::kRowThreads) k_batch_coh(const pgd::DevProblem* __restrict__ items, const BatchCall* call,
                                                                const int4* __restrict__ list, int n, int* err) {
  constexpr int CQ = pgd::CohLanes<DIM>::CQ;
  __shared__ pgd::DevProblem view;
  pgd::dep_launch();
  int last = -1;
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    const int4 it = __ldg(&list[c]);
    if (it.x != last) load_view(view, items, call, it.x, err);
    last = it.x;
    const int e = it.y + threadIdx.x / CQ;
    pgd::coh_element<DIM>(view, e, threadIdx.x % CQ, e < view.n_coh_el);
  }
}

// item = {context, part, block of the part, -}
template <int DIM, bool JAC>
__global__ void __launch_bounds__(pgd::kRowThreads) k_batch_rows(const pgd::DevProblem* __restrict__ items, const BatchCall* call,
                                                                 const int4* __restrict__ list, int n, int* err) {
  __shared__ pgd::DevProblem view;
  int last = -1;
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    const int4 it = __ldg(&list[c]);
    if (it.x != last) load_view(view, items, call, it.x, err);
    last = it.x;
    if (it.y == 1 && !(view.flags & pgd::FLAG_FUNC)) continue;
    pgd::row_block<DIM, pgd::pattern_period(DIM, DIM + 1), false, JAC, true>(view, it.y, it.z);
  }
}

}  // namespace

struct pg_batch {
  std::vector<pg_ctx*> ctx;
  int dim = 2;
  pgd::DevProblem* d_items = nullptr;
  BatchCall* d_call = nullptr;
  BatchCall* h_call = nullptr;
  int4 *d_coh = nullptr, *d_rows = nullptr;
  int *d_err = nullptr, *h_err = nullptr;   // OR of the contexts' device errors of the last call, and its pinned copy
  int n_coh = 0, n_sten = 0, n_gen = 0;     // items: cohesive elements, structured rows, general rows
  int mult = 4;   // launch shape (autotuned): persistent blocks per SM
  cudaStream_t stream = nullptr;
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  cudaGraphExec_t exec[2] = {nullptr, nullptr};   // residuals only, with the matrices
  bool launched = false;
  long long n_elem = 0;
  std::string err;
};

namespace {

int berr(pg_batch* b, int code, const std::string& m) {
  if (b) b->err = m;
  return code;
}

void free_lists(pg_batch* b) {
  if (b->d_coh) cudaFree(b->d_coh);
  if (b->d_rows) cudaFree(b->d_rows);
  b->d_coh = b->d_rows = nullptr;
}

void drop_graphs(pg_batch* b) {
  for (auto& e : b->exec)
    if (e) { cudaGraphExecDestroy(e); e = nullptr; }
}

template <typename T>
int upload_vec(pg_batch* b, const std::vector<T>& h, T** d) {
  *d = nullptr;
  if (h.empty()) return 0;
  if (cudaMalloc(d, h.size() * sizeof(T)) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "cudaMalloc failed");
  if (cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
    return berr(b, PG_ERR_DEVICE, "cudaMemcpy failed");
  return 0;
}

// Work lists of the batch.
int build_lists(pg_batch* b) {
  free_lists(b);
  drop_graphs(b);
  // the rows' blocks of all contexts, mixed as in a single assembly
  std::vector<int4> coh, rows;
  const int per = pgd::kRowThreads / ((b->dim == 2) ? pgd::CohLanes<2>::CQ : pgd::CohLanes<3>::CQ);
  std::vector<int4> of[4];
  pgd::RowParts all = {{0, 0, 0, 0}, false, 0};
  for (int i = 0; i < (int)b->ctx.size(); ++i) {
    const pgd::DevProblem& P = b->ctx[i]->P;
    const pgd::RowParts p = pgd::row_parts(P, true, true, false);
    for (int part = 0; part < 4; ++part)
      for (int k = 0; k < p.n[part]; ++k, ++all.n[part]) of[part].push_back(make_int4(i, part, k, 0));
    for (int f = 0; f < P.n_coh_el; f += per) coh.push_back(make_int4(i, f, 0, 0));
  }
  all.spread();
  for (int k = 0; k < all.total(); ++k) {
    int part, item;
    all.pick(k, &part, &item);
    rows.push_back(of[part][item]);
  }
  b->n_sten = all.n[1] + all.n[3];
  b->n_gen = all.n[0] + all.n[2];
  b->n_coh = (int)coh.size();
  int rc = upload_vec(b, coh, &b->d_coh);
  return rc ? rc : upload_vec(b, rows, &b->d_rows);
}

template <int DIM>
void enqueue_dim(pg_batch* b, bool jac) {
  cudaStream_t st = b->stream;
  const int cap = b->mult * kSMs, n_rows = b->n_sten + b->n_gen;
  if (b->n_coh)
    k_batch_coh<DIM><<<std::min(b->n_coh, cap), pgd::kRowThreads, 0, st>>>(b->d_items, b->d_call, b->d_coh, b->n_coh, b->d_err);
  if (!n_rows) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(n_rows, cap));
  cfg.blockDim = dim3(pgd::kRowThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = b->n_coh ? 1 : 0;
  cudaLaunchKernelEx(&cfg, jac ? k_batch_rows<DIM, true> : k_batch_rows<DIM, false>, (const pgd::DevProblem*)b->d_items,
                     (const BatchCall*)b->d_call, (const int4*)b->d_rows, n_rows, b->d_err);
}

void enqueue(pg_batch* b, bool jac) {
  cudaStream_t st = b->stream;
  cudaMemcpyAsync(b->d_call, b->h_call, sizeof(BatchCall) * b->ctx.size(), cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(b->d_err, 0, sizeof(int), st);
  if (b->dim == 2) enqueue_dim<2>(b, jac);
  else enqueue_dim<3>(b, jac);
  cudaMemcpyAsync(b->h_err, b->d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
}

int graph_for(pg_batch* b, bool jac, cudaGraphExec_t* out) {
  cudaGraphExec_t& e = b->exec[jac ? 1 : 0];
  if (!e) {
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
      return berr(b, PG_ERR_DEVICE, "graph capture failed to start");
    enqueue(b, jac);
    if (cudaStreamEndCapture(b->stream, &g) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "graph capture failed");
    const cudaError_t ie = cudaGraphInstantiate(&e, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) { e = nullptr; return berr(b, PG_ERR_DEVICE, "graph instantiation failed"); }
  }
  *out = e;
  return 0;
}

void fill_call(pg_batch* b, const double* const* d_U, const double* t_frac, int flags) {
  for (size_t i = 0; i < b->ctx.size(); ++i) {
    BatchCall& k = b->h_call[i];
    k.U = d_U[i];
    k.flags = flags & (PG_FUNC | PG_JAC | PG_FP32);
    const double tf = t_frac ? t_frac[i] : 1.0;
    for (int v = 0; v < 6; ++v) k.eps[v] = b->ctx[i]->s.desc.eps_macro[v] * tf;
  }
}

}  // namespace

extern "C" {

int pg_batch_create(pg_ctx* const* ctxs, int n, pg_batch** out) {
  if (!ctxs || n < 1 || !out) return PG_ERR_INPUT;
  *out = nullptr;
  pg_batch* b = new pg_batch;
  *out = b;
  b->dim = ctxs[0] ? ctxs[0]->s.dim : 2;
  std::vector<pgd::DevProblem> items(n);
  for (int i = 0; i < n; ++i) {
    pg_ctx* c = ctxs[i];
    if (!c || !c->P.X) return berr(b, PG_ERR_INPUT, "every context must be uploaded (pg_create or pg_upload)");
    if (c->s.dim != b->dim) return berr(b, PG_ERR_INPUT, "a batch holds contexts of one dimension");
    if (c->s.etype == pg::QUAD4) return berr(b, PG_ERR_UNSUPPORTED, "batches take tri3 / tet4 contexts");
    b->ctx.push_back(c);
    items[i] = c->P;
    b->n_elem += c->s.ne;
  }
  if (cudaMalloc(&b->d_items, sizeof(pgd::DevProblem) * n) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "cudaMalloc failed");
  cudaMemcpy(b->d_items, items.data(), sizeof(pgd::DevProblem) * n, cudaMemcpyHostToDevice);
  if (cudaMalloc(&b->d_err, sizeof(int)) != cudaSuccess || cudaMalloc(&b->d_call, sizeof(BatchCall) * n) != cudaSuccess ||
      cudaMallocHost(&b->h_call, sizeof(BatchCall) * n) != cudaSuccess || cudaMallocHost(&b->h_err, sizeof(int)) != cudaSuccess)
    return berr(b, PG_ERR_DEVICE, "call-parameter buffers failed");
  std::memset(b->h_call, 0, sizeof(BatchCall) * n);
  if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess)
    return berr(b, PG_ERR_DEVICE, "stream creation failed");
  cudaEventCreate(&b->t0);
  cudaEventCreate(&b->t1);
  return build_lists(b);
}

int pg_batch_assemble(pg_batch* b, const double* const* d_U, const double* t_frac, int flags) {
  if (!b || !d_U) return PG_ERR_INPUT;
  if (b->launched && cudaEventSynchronize(b->t1) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "previous batch failed");
  for (size_t i = 0; i < b->ctx.size(); ++i) {
    if (!d_U[i]) return berr(b, PG_ERR_INPUT, "missing displacement pointer");
    if (reinterpret_cast<uintptr_t>(d_U[i]) % 16) return berr(b, PG_ERR_INPUT, "displacement arrays must be 16-byte aligned");
  }
  fill_call(b, d_U, t_frac, flags);
  cudaGraphExec_t e;
  if (int rc = graph_for(b, (flags & PG_JAC) != 0, &e)) return rc;
  cudaEventRecord(b->t0, b->stream);
  if (cudaGraphLaunch(e, b->stream) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "graph launch failed");
  cudaEventRecord(b->t1, b->stream);
  b->launched = true;
  for (pg_ctx* c : b->ctx) c->assembled = true;
  return 0;
}

int pg_batch_wait(pg_batch* b, float* ms) {
  if (!b) return PG_ERR_INPUT;
  if (!b->launched) return berr(b, PG_ERR_STATE, "nothing was launched");
  if (cudaEventSynchronize(b->t1) != cudaSuccess) return berr(b, PG_ERR_DEVICE, "batch assembly failed");
  if (ms) cudaEventElapsedTime(ms, b->t0, b->t1);
  const int herr = *b->h_err;
  if (herr) return berr(b, PG_ERR_NONFINITE, "a context of the batch reported a device error (pg_last_error of each context has no detail)");
  return 0;
}

int pg_batch_tune(pg_batch* b, const double* const* d_U, int flags, int reps, int* best) {
  if (!b || !d_U || reps < 1) return PG_ERR_INPUT;
  const int mults[4] = {2, 4, 8, 16};
  float best_ms = 1e30f;
  int bm = b->mult;
  for (int mi = 0; mi < 4; ++mi) {
    b->mult = mults[mi];
    if (int rc = build_lists(b)) return rc;
    float total = 0.0f;
    for (int r = 0; r < reps + 2; ++r) {
      if (int rc = pg_batch_assemble(b, d_U, nullptr, flags)) return rc;
      float ms = 0.0f;
      if (int rc = pg_batch_wait(b, &ms)) return rc;
      if (r >= 2) total += ms;
    }
    if (total < best_ms) { best_ms = total; bm = b->mult; }
  }
  b->mult = bm;
  if (best) { best[0] = pgd::kRowThreads; best[1] = 1; best[2] = bm; }
  return build_lists(b);
}

int pg_batch_info(const pg_batch* b, int64_t* info) {
  if (!b || !info) return PG_ERR_INPUT;
  info[0] = (int64_t)b->ctx.size();
  info[1] = b->n_elem;
  info[2] = pgd::kRowThreads; info[3] = 1; info[4] = b->mult;
  info[5] = b->n_coh; info[6] = b->n_sten; info[7] = b->n_gen;
  return 0;
}

const char* pg_batch_last_error(const pg_batch* b) { return b ? b->err.c_str() : "null batch"; }

void pg_batch_destroy(pg_batch* b) {
  if (!b) return;
  if (b->launched) cudaEventSynchronize(b->t1);
  drop_graphs(b);
  free_lists(b);
  if (b->d_items) cudaFree(b->d_items);
  if (b->d_call) cudaFree(b->d_call);
  if (b->d_err) cudaFree(b->d_err);
  if (b->h_call) cudaFreeHost(b->h_call);
  if (b->h_err) cudaFreeHost(b->h_err);
  for (cudaEvent_t e : {b->t0, b->t1}) if (e) cudaEventDestroy(e);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

}  // extern "C"
