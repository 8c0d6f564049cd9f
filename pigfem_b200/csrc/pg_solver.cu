// pg_solver.cu -- device solvers and outputs on an assembled context.
//
//   pg_pcg_solve   Jacobi-preconditioned conjugate gradients on K_ff for several right-hand sides
//                  at once (the six unit-strain load cases of a homogenization, or one Newton
//                  correction).  FP64 throughout; every inner product is a fixed-order reduction
//                  (block partials over fixed row ranges, then one ordered sum), so a right-hand
//                  side's iterates do not depend on the other right-hand sides solved with it, and
//                  each right-hand side stops updating at its own convergence.  The iterations run
//                  in cooperative launches of one block per SM, one launch ahead of the flags the
//                  host has read.
//   pg_homogenize  volume average of the stress over the volumetric quadrature points
//                  (Problem::homogenize, src/Problem.cpp:471-484, with the stress functor of
//                  include/AssemblerSmallStrainStructural.h:31-60).
#include "pg_ctx.h"
#include "pg_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace {

constexpr int kThreads = 256;         // homogenization
constexpr int kPcgThreads = 512;      // one block per SM: 128 registers a thread for 3 rows x 6 right-hand sides
constexpr int kPcgWarps = kPcgThreads / 32;
constexpr int kMaxRhs = 6;            // right-hand sides of one pass (the unit strains of a 3D homogenization)
constexpr int kRound = 16;            // the host's iteration limit is a multiple of this
// How long a wait inside the kernel lasts before it gives up: other blocks and fetches arrive within
// milliseconds, on a GPU that several processes share within its time slices.
constexpr unsigned long long kWaitNs = 4000000000ull;
// scalar slots per right-hand side in PcgWork::sc
enum { S_RZ = 0, S_BB, S_RELRES, S_NSC };
// word slots after the 2 x NS per-right-hand-side words of PcgWork::flag
enum { F_ACTIVE = 0, F_BAD, F_STUCK, F_N };

// The matrix reaches the product through shared memory: a warp's unit of work is a chunk of up to
// 32 / L consecutive row groups whose values, columns and descriptors fit one stage, fetched by
// bulk copies into the warp's own ring of stages.  A chunk too long for a stage (kDirect) is read
// from global memory.
template <int M> struct PcgShape;
template <> struct PcgShape<2> {   // 2D: 8 groups of two rows, about 2.3 KB
  static constexpr int L = 4, kGroups = 8, kColBytes = 608, kValBytes = 2464, kStages = 4;
};
template <> struct PcgShape<3> {   // 3D: 4 groups of three rows of 45, 5.1 KB
  static constexpr int L = 8, kGroups = 4, kColBytes = 912, kValBytes = 5424, kStages = 2;
};
template <int M>
__host__ __device__ constexpr int pcg_stage_bytes() {
  return PcgShape<M>::kGroups * 16 + PcgShape<M>::kColBytes + PcgShape<M>::kValBytes;
}
template <int M>
constexpr int pcg_smem_bytes() { return kPcgWarps * PcgShape<M>::kStages * (pcg_stage_bytes<M>() + 8); }
static_assert(pcg_stage_bytes<2>() % 16 == 0 && pcg_stage_bytes<3>() % 16 == 0, "bulk copies need 16-byte stages");
static_assert(PcgShape<2>::kColBytes % 16 == 0 && PcgShape<3>::kColBytes % 16 == 0, "16-byte parts");

// word w of a group: row length, rows << 24, kDirect, groups of its chunk from this one on << 28
constexpr unsigned kDirect = 1u << 26;
__host__ __device__ constexpr int grp_len(unsigned w) { return (int)(w & 0xffffffu); }
__host__ __device__ constexpr int grp_rows(unsigned w) { return (int)(w >> 24) & 3; }

struct PcgArgs {
  const int4* grp;        // row groups: {first row, first value, first entry of gci, w}
  const int* gci;         // one column list per group (its rows share it)
  const int4* chunk;      // chunks: {first group, groups, first value, first entry of gci}, and the end
  const int* part_of;     // nb + 1: the chunks of each block
  const double* val;
  int n, ng, nb;
  double rtol;
  const double* b;        // [s][n]
  double* x;              // [s][n]
  double *dinv, *r, *p, *q, *xi;   // r, p, q, xi (the iterates) interleaved by right-hand side: [i * NS + s]
  double* part;           // [2 NS + NS][nb] partial sums
  double* sc;             // [NS][S_NSC]
  int* flag;              // [0, NS) done, [NS, 2 NS) iterations, then F_*
  unsigned* bar;          // arrivals at the grid barriers of this solve
  unsigned long long wait_ns;   // limit of a wait
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// NS adjacent doubles (16-byte pairs when NS is even).  Plain loads: p and q change during the
// kernel, and the grid barrier's acquire makes the other blocks' values visible.
template <int NS>
__device__ __forceinline__ void load_ns(const double* p, size_t i, double* out) {
  if constexpr (NS % 2 == 0) {
    const double2* q = reinterpret_cast<const double2*>(p + i * NS);
#pragma unroll
    for (int j = 0; j < NS / 2; ++j) { const double2 t = q[j]; out[2 * j] = t.x; out[2 * j + 1] = t.y; }
  } else {
#pragma unroll
    for (int j = 0; j < NS; ++j) out[j] = p[i * NS + j];
  }
}
template <int NS>
__device__ __forceinline__ void store_ns(double* p, size_t i, const double* v) {
  if constexpr (NS % 2 == 0) {
    double2* q = reinterpret_cast<double2*>(p + i * NS);
#pragma unroll
    for (int j = 0; j < NS / 2; ++j) q[j] = make_double2(v[2 * j], v[2 * j + 1]);
  } else {
#pragma unroll
    for (int j = 0; j < NS; ++j) p[i * NS + j] = v[j];
  }
}

// Before the first pass of a solve: the inverse diagonal (the matrix changes with every assembly)
// and the initial guess interleaved into p and xi.  A thread per row group.
template <int NS>
__global__ void __launch_bounds__(128) k_pcg_prepare(PcgArgs a) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.ng) return;
  const int4 d = __ldg(&a.grp[g]);
  const int len = grp_len(d.w), m = grp_rows(d.w);
  for (int i = 0; i < m; ++i) {
    const int row = d.x + i;
    // the columns are sorted: the group's rows are its own columns, so the diagonal is found by bisection
    int lo = 0, hi = len;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(&a.gci[d.z + mid]) < row) lo = mid + 1; else hi = mid;
    }
    const double v = (lo < len && __ldg(&a.gci[d.z + lo]) == row) ? __ldg(&a.val[d.y + i * len + lo]) : 0.0;
    if (!(v > 0.0) || !isfinite(v)) { atomicOr(&a.flag[2 * NS + F_BAD], 1); a.dinv[row] = 0.0; }
    else a.dinv[row] = 1.0 / v;
    double xv[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) xv[s] = a.x[(size_t)s * a.n + row];
    store_ns<NS>(a.p, row, xv);
    store_ns<NS>(a.xi, row, xv);
  }
}

// After the last iteration: the solutions into the caller's layout.
template <int NS>
__global__ void __launch_bounds__(128) k_pcg_finish(PcgArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n || a.flag[2 * NS + F_STUCK]) return;   // (out of step: the caller's x stays)
  double xv[NS];
  load_ns<NS>(a.xi, i, xv);
#pragma unroll
  for (int s = 0; s < NS; ++s) a.x[(size_t)s * a.n + i] = xv[s];
}

// Sums of C values over the lanes of a warp, scattered: at each step a lane hands half of its
// values to its partner and keeps the other half, so C values cost about C shuffles instead of
// 5 C.  Every value's additions form the butterfly tree l ^ 16, l ^ 8, ..., whichever lane ends up
// with it, so a value's sum does not depend on C.  Returns the index of the value left in v[0].
template <int C, int O>
__device__ __forceinline__ int scatter_sum(double* v, int lane) {
  if constexpr (O == 0) {
    return 0;
  } else {
    constexpr int H = (C + 1) / 2;
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const double lo = v[i], hi = (i + H < C) ? v[i + H] : v[i];
      const double got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, O);
      v[i] = __dadd_rn(up ? hi : lo, got);
    }
    const int k = scatter_sum<H, O / 2>(v, lane);
    return (up && k + H < C) ? k + H : k;
  }
}

// The block's sums of C per-thread values to part[k * nb + block], in a fixed order.
template <int C>
__device__ __forceinline__ void block_sums(double* v, double (*red)[3 * kMaxRhs], double* part, int nb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = scatter_sum<C, 16>(v, lane);
  red[warp][k] = v[0];   // lanes left with the same value hold the same bits
  __syncthreads();
  if (threadIdx.x < C) {
    double t = red[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < kPcgWarps; ++w) t = __dadd_rn(t, red[w][threadIdx.x]);
    part[threadIdx.x * nb + blockIdx.x] = t;
  }
}

// All blocks of the (cooperative) launch meet: the arrivals of a solve are counted in one word
// that only grows, `target` is its value once every block has arrived.  Bounded in time: false once
// the limit is reached (the caller returns and the host reports it).
__device__ __forceinline__ bool grid_barrier(const PcgArgs& a, unsigned target, int* stuck) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
    auto arrived = [&]() {
      unsigned got;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(a.bar) : "memory");
      return (int)(got - target) >= 0;
    };
    bool in = arrived();
    if (!in) {
      const unsigned long long t0 = now_ns();
      // (a block that gave up arrives nowhere any more: the others need not wait out their limit)
      for (unsigned k = 1; !(in = arrived()); ++k)
        if (k % 64 == 0 && (now_ns() - t0 >= a.wait_ns || *(volatile int*)stuck != 0)) break;
    }
    ok = in;
    if (!in) atomicOr(stuck, 1);
  }
  __syncthreads();
  return ok != 0;
}

// Ordered sums of the blocks' partials of C values: tot[k], the same in every block.
template <int C>
__device__ __forceinline__ void total_sums(const double* part, int nb, double* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = warp; k < C; k += kPcgWarps) {
    double t = 0.0;
    for (int i = lane; i < nb; i += 32) t = __dadd_rn(t, part[k * nb + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
    if (lane == 0) tot[k] = t;
  }
  __syncthreads();
}

// A warp's ring of stages.  The chunks of the warp follow each other through the iterations (the
// matrix does not change), so the first chunks of the next product are fetched while the vectors
// are updated; when all of them fit the ring they are fetched once.
template <int M>
struct PcgRing {
  using S = PcgShape<M>;
  unsigned char* mem;       // the warp's stages
  unsigned bar;             // shared address of the warp's barriers
  const int4* first;        // the warp's first chunk; the following are kPcgWarps apart
  int n;                    // its chunks
  bool resident;
  unsigned issued, used;    // chunks fetched / consumed so far

  __device__ __forceinline__ void issue(const PcgArgs& a) {   // one lane
    const int4 c = __ldg(first + (size_t)(issued % n) * kPcgWarps), e = __ldg(first + (size_t)(issued % n) * kPcgWarps + 1);
    const unsigned st = issued % S::kStages;
    const unsigned full = bar + 8 * st;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(mem + st * pcg_stage_bytes<M>());
    const bool direct = (c.y & 256) != 0;
    const int v0 = c.z & ~1, c0 = c.w & ~3;
    const unsigned gb = (c.y & 255) * 16u;
    const unsigned vb = direct ? 0u : (unsigned)(((e.z + 1) & ~1) - v0) * 8u;
    const unsigned cb = direct ? 0u : (unsigned)(((e.w + 3) & ~3) - c0) * 4u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(gb + vb + cb) : "memory");
    auto copy = [&](unsigned to, const void* from, unsigned bytes) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to),
                   "l"(from), "r"(bytes), "r"(full)
                   : "memory");
    };
    copy(dst, a.grp + c.x, gb);
    if (cb) copy(dst + S::kGroups * 16, a.gci + c0, cb);
    if (vb) copy(dst + S::kGroups * 16 + S::kColBytes, a.val + v0, vb);
  }
  // Waits (bounded in time) for stage st's fetch number `turn`; the whole warp calls it and agrees.
  __device__ __forceinline__ bool wait(const PcgArgs& a, unsigned st, unsigned turn) const {
    auto arrived = [&]() {
      unsigned ok;
      asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                   : "=r"(ok) : "r"(bar + 8 * st), "r"(turn & 1u) : "memory");
      return __all_sync(0xffffffffu, ok) != 0;
    };
    if (arrived()) return true;
    const unsigned long long t0 = now_ns();
    while (!arrived())
      if (__any_sync(0xffffffffu, now_ns() - t0 >= a.wait_ns)) return false;
    return true;
  }
  __device__ __forceinline__ void fill(const PcgArgs& a, int lane) {
    const unsigned upto = resident ? (unsigned)n : used + S::kStages;
    for (; n > 0 && issued < upto; ++issued)
      if (lane == 0) issue(a);
  }
  // The stage in use is done with: fetches the chunk that follows into it.  The copy's writes come
  // after every lane's loads from the stage: each lane's proxy fence orders its own loads before
  // copies, and __syncwarp orders the lanes before the one that issues the copy.  (__syncwarp alone
  // does not: it says nothing about the async proxy, and a copy was seen to start with loads issued
  // but not yet returned.  An mbarrier that all 32 lanes arrive on orders them too, but its arrivals
  // go one by one: 40^3 tet4 with six right-hand sides 114 us per iteration.)
  __device__ __forceinline__ void refill(const PcgArgs& a, int lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    ++used;
    fill(a, lane);
  }
  // Waits for every fetch still in flight (before the block returns).
  __device__ __forceinline__ void drain(const PcgArgs& a) {
    if (resident) { for (unsigned k = 0; used == 0 && k < issued; ++k) wait(a, k, 0); return; }
    for (; used < issued; ++used) wait(a, used % S::kStages, used / S::kStages);
  }
};

// q = A p on the block's rows, L lanes per row group (a node's free DOFs: up to M consecutive rows
// with one column list).  A lane takes the nonzeros lane, lane + L, ... of all the group's rows, so
// a column index and a column's NS values of p are read once for M rows; the lanes' sums are then
// exchanged so that each row ends in its own lane.  A row's products and sums are the same for any
// NS.  pq gets the lane's rows' p.q.  false when a fetch did not arrive.
template <int NS, int M>
__device__ __forceinline__ bool block_product(const PcgArgs& a, PcgRing<M>& ring, double* pq) {
  using S = PcgShape<M>;
  constexpr int L = S::L;
  const int wl = threadIdx.x & 31, lane = wl % L, sub = wl / L;
#pragma unroll
  for (int j = 0; j < NS; ++j) pq[j] = 0.0;
  for (int i = 0; i < ring.n; ++i) {
    const unsigned st = ring.resident ? (unsigned)i : ring.used % S::kStages;
    if (!ring.wait(a, st, ring.resident ? 0u : ring.used / S::kStages)) return false;
    const unsigned char* mem = ring.mem + st * pcg_stage_bytes<M>();
    const int4* sg = reinterpret_cast<const int4*>(mem);
    const int4 d0 = sg[0];
    int4 d = make_int4(0, 0, 0, 0);
    if (sub < (int)((unsigned)d0.w >> 28)) d = sg[sub];
    const int len = grp_len(d.w), m = grp_rows(d.w);
    // the row this lane ends up with, and its own p
    int mine;
    if constexpr (M == 3) mine = (lane & 4) ? 2 : ((lane & 2) ? 1 : 0);
    else mine = (lane & 2) ? 1 : 0;
    const bool writer = (M == 3 ? (lane == 0 || lane == 2 || lane == 4) : (lane == 0 || lane == 2)) && mine < m;
    double own[NS];
    if (writer) load_ns<NS>(a.p, d.x + mine, own);
    double acc[M][NS];
#pragma unroll
    for (int r = 0; r < M; ++r)
#pragma unroll
      for (int j = 0; j < NS; ++j) acc[r][j] = 0.0;
    auto rows = [&](const double* v, const int* ci) {
#pragma unroll 3
      for (int k = lane; k < len; k += L) {
        double av[M], pv[NS];
        load_ns<NS>(a.p, ci[k], pv);
#pragma unroll
        for (int r = 0; r < M; ++r) av[r] = (r < m) ? v[r * len + k] : 0.0;
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll
          for (int j = 0; j < NS; ++j) acc[r][j] = __fma_rn(av[r], pv[j], acc[r][j]);
      }
    };
    if ((unsigned)d0.w & kDirect) {
      rows(a.val + d.y, a.gci + d.z);
    } else {
      const int* sc = reinterpret_cast<const int*>(mem + S::kGroups * 16);
      const double* sv = reinterpret_cast<const double*>(mem + S::kGroups * 16 + S::kColBytes);
      rows(sv + (d.y - (d0.y & ~1)), sc + (d.z - (d0.z & ~3)));
    }
    double qv[NS];
    if constexpr (M == 3) {
      const bool hi = (lane & 4) != 0, odd = (lane & 2) != 0;
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double got0 = __shfl_xor_sync(0xffffffffu, hi ? acc[0][j] : acc[2][j], 4);
        const double x = __dadd_rn(hi ? acc[2][j] : acc[0][j], got0);
        const double y = __dadd_rn(acc[1][j], __shfl_xor_sync(0xffffffffu, acc[1][j], 4));
        const double got = __shfl_xor_sync(0xffffffffu, (hi || odd) ? x : y, 2);
        const double t = __dadd_rn((!hi && odd) ? y : x, got);
        qv[j] = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 1));
      }
    } else {
      const bool hi = (lane & 2) != 0;
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double got = __shfl_xor_sync(0xffffffffu, hi ? acc[0][j] : acc[1][j], 2);
        const double t = __dadd_rn(hi ? acc[1][j] : acc[0][j], got);
        qv[j] = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 1));
      }
    }
    if (!ring.resident) ring.refill(a, wl);   // (the sums above have used every value of the stage)
    if (writer) {
      store_ns<NS>(a.q, d.x + mine, qv);
#pragma unroll
      for (int j = 0; j < NS; ++j) pq[j] = __fma_rn(own[j], qv[j], pq[j]);
    }
  }
  if (ring.resident) ring.used = 1;   // fetched and seen
  return true;
}

// Iterations [it0, it1) of the solve in one cooperative launch, one block per SM, each block owning
// a fixed range of rows with about the same number of nonzeros.  Per iteration three passes over
// the block's rows, separated by grid barriers:
//   q = A p, partial p.q  |  r -= alpha q, partials of r.z and r.r (z = D^-1 r is never stored)
//   |  x += alpha p, p = z + beta p  |
// Every block forms the scalars itself from all blocks' partials, in the same order, so the blocks
// agree on them and on who is done.  `first`: r = b - A x, p = z before the iterations.
// One launch per round instead of five kernels per iteration: a 128 x 128 tri3 RVE with three
// right-hand sides (39,614 rows) takes 11.4 us per iteration (five kernels: 36 us), of which the
// three barriers with their scalars are about 5 us; 40^3 tet4 with six (219,807 rows, 9.7 M
// nonzeros) 66 us (132 us), bound by the latency of the gathers of p (48 bytes
// per lane) at 16 warps per SM.
template <int NS, int M>
__global__ void __launch_bounds__(kPcgThreads, 1) k_pcg_run(PcgArgs a, int first, int it0, int it1, unsigned arrived) {
  __shared__ double red[kPcgWarps][3 * kMaxRhs];
  __shared__ double tot[3 * kMaxRhs];
  __shared__ double rz[kMaxRhs], bb[kMaxRhs], relres[kMaxRhs], step[kMaxRhs], coef[kMaxRhs];
  __shared__ int done[kMaxRhs], iters[kMaxRhs], active, leave;
  const int t = threadIdx.x;
  // Set before this launch (F_STUCK also by a block of this one that gave up already): the launch
  // queued behind one that gave up would wait for arrivals that never came.
  if (t == 0) leave = a.flag[2 * NS + F_BAD] | *(volatile int*)&a.flag[2 * NS + F_STUCK];
  __syncthreads();
  if (leave != 0) return;   // (read once: the whole block leaves or stays)
  extern __shared__ __align__(16) unsigned char stages[];
  const int c0 = __ldg(&a.part_of[blockIdx.x]), c1 = __ldg(&a.part_of[blockIdx.x + 1]);
  int r0 = 0, r1 = 0;
  if (c0 < c1) {
    r0 = __ldg(&a.grp[__ldg(&a.chunk[c0]).x]).x;
    const int4 d = __ldg(&a.grp[__ldg(&a.chunk[c1]).x - 1]);
    r1 = d.x + grp_rows(d.w);
  }
  PcgRing<M> ring;
  {
    using S = PcgShape<M>;
    const int warp = t >> 5;
    ring.mem = stages + (size_t)warp * S::kStages * pcg_stage_bytes<M>();
    unsigned char* bars = stages + (size_t)kPcgWarps * S::kStages * pcg_stage_bytes<M>();
    ring.bar = (unsigned)__cvta_generic_to_shared(bars) + 8u * S::kStages * warp;
    ring.first = a.chunk + c0 + warp;
    ring.n = (c1 - c0 - warp + kPcgWarps - 1) / kPcgWarps;
    if (ring.n < 0) ring.n = 0;
    ring.resident = ring.n <= S::kStages;
    ring.issued = ring.used = 0;
    if ((t & 31) == 0) {
      for (int k = 0; k < S::kStages; ++k)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ring.bar + 8u * k) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    ring.fill(a, t & 31);
  }
  unsigned target = arrived;
  int* stuck = &a.flag[2 * NS + F_STUCK];
  bool fine = true;
  double sum[2 * NS + NS];
  // a barrier or a fetch that gave up: the block waits for its own copies and returns
  auto give_up = [&]() {
    if (!fine) atomicOr(stuck, 1);
    ring.drain(a);
  };
  if (first) {
    fine = block_product<NS, M>(a, ring, sum);
    if (!__syncthreads_and(fine)) { give_up(); return; }   // (and the block's q)
#pragma unroll
    for (int k = 0; k < 3 * NS; ++k) sum[k] = 0.0;
    for (int i = r0 + t; i < r1; i += kPcgThreads) {
      double qv[NS], rv[NS];
      load_ns<NS>(a.q, i, qv);
      const double di = a.dinv[i];
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double bj = a.b[(size_t)j * a.n + i];
        rv[j] = __dsub_rn(bj, qv[j]);
        sum[j] = __fma_rn(rv[j], __dmul_rn(di, rv[j]), sum[j]);
        sum[NS + j] = __fma_rn(rv[j], rv[j], sum[NS + j]);
        sum[2 * NS + j] = __fma_rn(bj, bj, sum[2 * NS + j]);
      }
      store_ns<NS>(a.r, i, rv);
    }
    block_sums<3 * NS>(sum, red, a.part, a.nb);
    if (!grid_barrier(a, target += a.nb, stuck)) { give_up(); return; }
    total_sums<3 * NS>(a.part, a.nb, tot);
    if (t == 0) {
      active = 0;
      for (int j = 0; j < NS; ++j) {
        const double nb2 = sqrt(tot[2 * NS + j]);
        rz[j] = tot[j];
        bb[j] = tot[2 * NS + j];
        relres[j] = nb2 > 0.0 ? sqrt(tot[NS + j]) / nb2 : 0.0;
        done[j] = (nb2 == 0.0) || (relres[j] <= a.rtol);
        iters[j] = 0;
        active += !done[j];
      }
    }
    for (int i = r0 + t; i < r1; i += kPcgThreads) {
      double rv[NS];
      load_ns<NS>(a.r, i, rv);
      const double di = a.dinv[i];
#pragma unroll
      for (int j = 0; j < NS; ++j) rv[j] = __dmul_rn(di, rv[j]);
      store_ns<NS>(a.p, i, rv);
    }
    if (!grid_barrier(a, target += a.nb, stuck)) { give_up(); return; }
  } else {
    if (t < NS) {
      rz[t] = a.sc[t * S_NSC + S_RZ];
      bb[t] = a.sc[t * S_NSC + S_BB];
      relres[t] = a.sc[t * S_NSC + S_RELRES];
      done[t] = a.flag[t];
      iters[t] = a.flag[NS + t];
    }
    if (t == 0) active = a.flag[2 * NS + F_ACTIVE];
    __syncthreads();
  }
  for (int it = it0; it < it1 && active > 0; ++it) {
    fine = block_product<NS, M>(a, ring, sum);
    if (!__syncthreads_and(fine)) { give_up(); return; }
    block_sums<NS>(sum, red, a.part, a.nb);
    if (!grid_barrier(a, target += a.nb, stuck)) { give_up(); return; }
    total_sums<NS>(a.part, a.nb, tot);
    if (t < NS) step[t] = rz[t] / tot[t];
    __syncthreads();
    double al[NS];
    bool act[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      act[j] = !done[j];
      al[j] = act[j] ? step[j] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 2 * NS; ++k) sum[k] = 0.0;
#pragma unroll 2
    for (int i = r0 + t; i < r1; i += kPcgThreads) {
      double qv[NS], rv[NS];
      load_ns<NS>(a.q, i, qv);
      load_ns<NS>(a.r, i, rv);
      const double di = a.dinv[i];
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        if (act[j]) rv[j] = __fma_rn(-al[j], qv[j], rv[j]);
        sum[j] = __fma_rn(rv[j], __dmul_rn(di, rv[j]), sum[j]);
        sum[NS + j] = __fma_rn(rv[j], rv[j], sum[NS + j]);
      }
      store_ns<NS>(a.r, i, rv);
    }
    // (the second set of partials: a block may still be reading the first)
    block_sums<2 * NS>(sum, red, a.part + NS * a.nb, a.nb);
    if (!grid_barrier(a, target += a.nb, stuck)) { give_up(); return; }
    total_sums<2 * NS>(a.part + NS * a.nb, a.nb, tot);
    if (t < NS) {
      coef[t] = tot[t] / rz[t];
      if (!done[t]) {
        rz[t] = tot[t];
        relres[t] = sqrt(tot[NS + t]) / sqrt(bb[t]);
        ++iters[t];
      }
    }
    __syncthreads();
    // x and p, element by element: the vectors are interleaved, so consecutive threads take
    // consecutive words whatever NS is
    constexpr int W = (NS % 2 == 0) ? 2 : 1;
    double* const vx = a.xi + (size_t)r0 * NS;
    double* const vp = a.p + (size_t)r0 * NS;
    const double* const vr = a.r + (size_t)r0 * NS;
    const int nw = (r1 - r0) * (NS / W);
#pragma unroll 4
    for (int e = t; e < nw; e += kPcgThreads) {
      const int row = e / (NS / W), j0 = (e - row * (NS / W)) * W;
      double xv[W], pv[W], rv[W];
      load_ns<W>(vx, e, xv);
      load_ns<W>(vp, e, pv);
      load_ns<W>(vr, e, rv);
      const double di = a.dinv[r0 + row];
#pragma unroll
      for (int j = 0; j < W; ++j)
        if (!done[j0 + j]) {
          xv[j] = __fma_rn(step[j0 + j], pv[j], xv[j]);
          pv[j] = __fma_rn(coef[j0 + j], pv[j], __dmul_rn(di, rv[j]));
        }
      store_ns<W>(vx, e, xv);
      store_ns<W>(vp, e, pv);
    }
    __syncthreads();   // everyone is past reading done
    if (t == 0) {
      int n_act = 0;
      for (int j = 0; j < NS; ++j) {
        if (!done[j] && (relres[j] <= a.rtol || !isfinite(relres[j]))) done[j] = 1;
        n_act += !done[j];
      }
      active = n_act;
    }
    if (!grid_barrier(a, target += a.nb, stuck)) { give_up(); return; }
  }
  ring.drain(a);
  __syncthreads();
  if (blockIdx.x == 0) {
    if (t < NS) {
      a.sc[t * S_NSC + S_RZ] = rz[t];
      a.sc[t * S_NSC + S_BB] = bb[t];
      a.sc[t * S_NSC + S_RELRES] = relres[t];
      a.flag[t] = done[t];
      a.flag[NS + t] = iters[t];
    }
    if (t == 0) a.flag[2 * NS + F_ACTIVE] = active;
  }
}

struct PcgKernels {
  void (*run)(PcgArgs, int, int, int, unsigned);
  void (*prepare)(PcgArgs);
  void (*finish)(PcgArgs);
  int smem;
};
template <int NS>
PcgKernels pcg_kernels(int dim) {
  if (dim == 3) return {k_pcg_run<NS, 3>, k_pcg_prepare<NS>, k_pcg_finish<NS>, pcg_smem_bytes<3>()};
  return {k_pcg_run<NS, 2>, k_pcg_prepare<NS>, k_pcg_finish<NS>, pcg_smem_bytes<2>()};
}

// Row groups and chunks of K_ff: the consecutive rows of one DOF node share one column list.
template <int M>
void pcg_groups(const pg::Setup& s, int stage_values, std::vector<int4>& grp, std::vector<int>& gci, std::vector<int4>& chunk) {
  using S = PcgShape<M>;
  const int val_bytes = stage_values > 0 ? std::min(stage_values * 8, S::kValBytes) : S::kValBytes;
  const int n = s.n_free;
  const std::vector<int>& rp = s.rp[0];
  std::vector<int> owner(n, -1);
  for (int a = 0; a < s.n_dn; ++a)
    for (int q = 0; q < s.dim; ++q) {
      const int g = s.node_dof[(size_t)s.dn_node[a] * s.dim + q];
      if (g < n) owner[g] = a;
    }
  grp.reserve(n / M + 1);
  gci.reserve(s.ci[0].size() / M + 64);
  int open = 0;   // groups of the open chunk
  auto close = [&](bool direct) {
    if (!open) return;
    chunk.back().y = open | (direct ? 256 : 0);
    for (int k = 0; k < open; ++k) {
      int4& d = grp[grp.size() - open + k];
      d.w = (int)((unsigned)d.w | (direct ? kDirect : 0u) | ((unsigned)(open - k) << 28));
    }
    open = 0;
  };
  for (int r = 0; r < n;) {
    const int len = rp[r + 1] - rp[r];
    int m = 1;
    while (m < M && r + m < n && owner[r + m] == owner[r] && owner[r] >= 0 && rp[r + m + 1] - rp[r + m] == len) ++m;
    const int v1 = rp[r + m], c1 = (int)gci.size() + len;
    // (with the 16-byte boundaries the copies start and end on)
    auto fits = [&](int v0, int c0) {
      return (((v1 + 1) & ~1) - (v0 & ~1)) * 8 <= val_bytes && (((c1 + 3) & ~3) - (c0 & ~3)) * 4 <= S::kColBytes;
    };
    if (open == S::kGroups || (open && !fits(chunk.back().z, chunk.back().w))) close(false);
    if (!open) chunk.push_back(make_int4((int)grp.size(), 0, rp[r], (int)gci.size()));
    grp.push_back(make_int4(r, rp[r], (int)gci.size(), len | (m << 24)));
    gci.insert(gci.end(), s.ci[0].begin() + rp[r], s.ci[0].begin() + rp[r + 1]);
    ++open;
    if (open == 1 && !fits(chunk.back().z, chunk.back().w)) close(true);   // longer than a stage: alone, read from global memory
    r += m;
  }
  close(false);
  chunk.push_back(make_int4((int)grp.size(), 0, n ? rp[n] : 0, (int)gci.size()));
}

int pcg_reserve(pg_ctx* c, int nrhs) {
  PcgWork& w = c->pcg;
  const pg::Setup& s = c->s;
  const int n = s.n_free, dim = s.dim;
  // (every part is recorded once it is whole: a call after a failed one builds it again)
  if (!w.stream) {
    cudaStream_t st = nullptr;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    int* h = nullptr;
    bool ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t& e : ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaMallocHost(&h, sizeof(int) * 64) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      for (cudaEvent_t e : ev) if (e) cudaEventDestroy(e);
      if (st) cudaStreamDestroy(st);
      return pg_set_err(c, PG_ERR_DEVICE, "solver stream creation failed");
    }
    w.stream = st;
    w.ev = ev[0];
    w.evc[0] = ev[1];
    w.evc[1] = ev[2];
    w.hflag = h;
  }
  int rc = 0;
  if (!w.grp) {
    std::vector<int4> grp, chunk;
    std::vector<int> gci;
    if (dim == 3) pcg_groups<3>(s, w.stage_values, grp, gci, chunk);
    else pcg_groups<2>(s, w.stage_values, grp, gci, chunk);
    const int ng = (int)grp.size(), nch = (int)chunk.size() - 1;
    // blocks: one per SM (the launch is cooperative), fewer when there are fewer chunks than
    // warps; contiguous chunk ranges of about equal nonzeros plus vector work
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    w.nb = std::max(1, std::min(sms, (nch + kPcgWarps - 1) / kPcgWarps));
    auto weight = [&](int k) { return (double)(chunk[k + 1].z - chunk[k].z) + 16.0 * dim * (chunk[k + 1].x - chunk[k].x); };
    double total = 0.0, acc = 0.0;
    for (int k = 0; k < nch; ++k) total += weight(k);
    std::vector<int> part(w.nb + 1, nch);
    part[0] = 0;
    for (int k = 0, b = 1; k < nch && b < w.nb; ++k) {
      acc += weight(k);
      while (b < w.nb && acc >= total * b / w.nb) part[b++] = k + 1;
    }
    gci.resize((gci.size() + 7) & ~(size_t)3);   // the last chunk's copy ends on a 16-byte boundary
    int4 *d_grp = nullptr, *d_chunk = nullptr;
    int *d_gci = nullptr, *d_part = nullptr;
    double* d_dinv = nullptr;
    unsigned* d_bar = nullptr;
    rc = pg_dalloc(c, grp.size(), &d_grp) | pg_dalloc(c, gci.size(), &d_gci) | pg_dalloc(c, chunk.size(), &d_chunk) |
         pg_dalloc(c, part.size(), &d_part) | pg_dalloc(c, (size_t)n, &d_dinv) | pg_dalloc(c, 1, &d_bar);
    auto copy = [&](void* d, const void* h, size_t bytes) {
      return cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, c->up) != cudaSuccess;
    };
    if (!rc && (copy(d_grp, grp.data(), grp.size() * sizeof(int4)) || copy(d_gci, gci.data(), gci.size() * sizeof(int)) ||
                copy(d_chunk, chunk.data(), chunk.size() * sizeof(int4)) || copy(d_part, part.data(), part.size() * sizeof(int)) ||
                pg_alloc_sync(c)))
      rc = pg_set_err(c, PG_ERR_DEVICE, "solver tables: copy failed");
    if (rc) {
      for (void* p : {(void*)d_grp, (void*)d_gci, (void*)d_chunk, (void*)d_part, (void*)d_dinv, (void*)d_bar})
        if (p) pg_untrack_free(c, p);
      return PG_ERR_DEVICE;
    }
    w.grp = d_grp;
    w.gci = d_gci;
    w.chunk = d_chunk;
    w.part_of = d_part;
    w.dinv = d_dinv;
    w.bar = d_bar;
    w.ng = ng;
    w.shape[0] = w.nb;
    w.shape[1] = nch;
    w.shape[2] = w.shape[4] = 0;
    for (int b = 0; b < w.nb; ++b) w.shape[2] = std::max(w.shape[2], (part[b + 1] - part[b] + kPcgWarps - 1) / kPcgWarps);
    w.shape[3] = dim == 3 ? PcgShape<3>::kStages : PcgShape<2>::kStages;
    for (int k = 0; k < nch; ++k) w.shape[4] += (chunk[k].y & 256) != 0;
  }
  if (w.cap_rhs < nrhs) {
    // (a solve returns with its work done, so the smaller buffers are idle)
    auto drop = [&]() {
      for (double** p : {&w.r, &w.p, &w.q, &w.xi, &w.part, &w.sc}) {
        if (*p) pg_untrack_free(c, *p);
        *p = nullptr;
      }
      if (w.flag) pg_untrack_free(c, w.flag);
      w.flag = nullptr;
      w.cap_rhs = 0;
    };
    drop();
    rc |= pg_dalloc(c, (size_t)n * nrhs, &w.r) | pg_dalloc(c, (size_t)n * nrhs, &w.p) | pg_dalloc(c, (size_t)n * nrhs, &w.q) |
          pg_dalloc(c, (size_t)n * nrhs, &w.xi) | pg_dalloc(c, (size_t)3 * nrhs * w.nb, &w.part) | pg_dalloc(c, (size_t)S_NSC * nrhs, &w.sc) |
          pg_dalloc(c, (size_t)2 * nrhs + F_N, &w.flag);
    if (rc || pg_alloc_sync(c)) {
      drop();
      return PG_ERR_DEVICE;
    }
    w.cap_rhs = nrhs;
  }
  return 0;
}

// Solves for NS = nrhs <= kMaxRhs right-hand sides; *all is cleared when one misses the tolerance.
int pcg_pass(pg_ctx* c, const double* d_b, double* d_x, int nrhs, double rtol, int max_it, int* iters, double* relres,
             bool* all) {
  PcgWork& w = c->pcg;
  const int n = c->s.n_free;
  PcgArgs a{w.grp, w.gci, w.chunk, w.part_of, c->P.val[0], n, w.ng, w.nb, rtol, d_b, d_x,
            w.dinv, w.r, w.p, w.q, w.xi, w.part, w.sc, w.flag, w.bar, w.wait_ms > 0 ? w.wait_ms * 1000000ull : kWaitNs};
  PcgKernels k;
  switch (nrhs) {
    case 1: k = pcg_kernels<1>(c->s.dim); break;
    case 2: k = pcg_kernels<2>(c->s.dim); break;
    case 3: k = pcg_kernels<3>(c->s.dim); break;
    case 4: k = pcg_kernels<4>(c->s.dim); break;
    case 5: k = pcg_kernels<5>(c->s.dim); break;
    default: k = pcg_kernels<6>(c->s.dim); break;
  }
  if (cudaFuncSetAttribute((const void*)k.run, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem) != cudaSuccess)
    return pg_set_err(c, PG_ERR_DEVICE, "solver shared memory request failed");
  const int n_flag = 2 * nrhs + F_N;
  cudaMemsetAsync(w.flag, 0, sizeof(int) * n_flag, w.stream);
  cudaMemsetAsync(w.bar, 0, sizeof(unsigned), w.stream);
  k.prepare<<<(w.ng + 127) / 128, 128, 0, w.stream>>>(a);
  // Launches of `chunk` iterations, one ahead of the flags the host has seen (a launch that finds
  // every right-hand side done returns at once).  Short iterations get longer launches, so the
  // launch and its scalars' reload stay small beside them; long ones keep the default round, so
  // other streams' work gets its turn within a millisecond or two.
  const int limit = (int)std::min<long long>(((long long)max_it + kRound - 1) / kRound * kRound, 2147483647LL / kRound * kRound);
  const int chunk = ((double)c->s.ci[0].size() * (2 + nrhs) < 2e7) ? 8 * kRound : kRound;
  unsigned arrived = 0;
  int it = 0, rc = 0;
  for (int l = 0;; ++l) {
    if (it < limit) {
      int first = l == 0, it0 = it, it1 = std::min(limit, it + chunk);
      void* args[] = {&a, &first, &it0, &it1, &arrived};
      if (cudaLaunchCooperativeKernel((const void*)k.run, dim3(w.nb), dim3(kPcgThreads), args, (size_t)k.smem, w.stream) != cudaSuccess) {
        rc = pg_set_err(c, PG_ERR_DEVICE, "solver launch failed");
        break;
      }
      arrived += (unsigned)(w.nb * (3 * (it1 - it0) + (first ? 2 : 0)));
      if (first) arrived += (unsigned)w.missing;   // (pg_debug_set: none in earnest)
      it = it1;
    }
    cudaMemcpyAsync(w.hflag + 32 * (l & 1), w.flag, sizeof(int) * n_flag, cudaMemcpyDeviceToHost, w.stream);
    cudaEventRecord(w.evc[l & 1], w.stream);
    if (l == 0 && it < limit) continue;
    // the flags of the launch before this one (of this one when it is the last)
    const int look = it < limit ? (l - 1) & 1 : l & 1;
    if (cudaEventSynchronize(w.evc[look]) != cudaSuccess) { rc = pg_set_err(c, PG_ERR_DEVICE, "solver iteration failed"); break; }
    const int* f = w.hflag + 32 * look + 2 * nrhs;
    if (f[F_BAD] || f[F_STUCK] || f[F_ACTIVE] == 0 || it >= limit) break;
  }
  std::vector<double> sc((size_t)S_NSC * nrhs);
  if (!rc) {
    // (a bad diagonal leaves the caller's x as it was: xi still holds it)
    k.finish<<<(n + 127) / 128, 128, 0, w.stream>>>(a);
    cudaMemcpyAsync(sc.data(), w.sc, sizeof(double) * sc.size(), cudaMemcpyDeviceToHost, w.stream);
    cudaMemcpyAsync(w.hflag, w.flag, sizeof(int) * n_flag, cudaMemcpyDeviceToHost, w.stream);
  }
  if (cudaStreamSynchronize(w.stream) != cudaSuccess && !rc) rc = pg_set_err(c, PG_ERR_DEVICE, "solver read-back failed");
  if (rc) return rc;
  const int* f = w.hflag;
  if (f[2 * nrhs + F_BAD]) return pg_set_err(c, PG_ERR_NONFINITE, "K_ff has a non-positive or non-finite diagonal entry");
  if (f[2 * nrhs + F_STUCK]) return pg_set_err(c, PG_ERR_DEVICE, "a wait of the solver ran out");
  for (int s = 0; s < nrhs; ++s) {
    const double rr = sc[(size_t)s * S_NSC + S_RELRES];
    if (iters) iters[s] = f[nrhs + s];
    if (relres) relres[s] = rr;
    *all = *all && f[s] && std::isfinite(rr);
  }
  return 0;
}

// ---------------------------------------------------------------- homogenization
constexpr int kHomBlocks = 2 * 148;

__device__ __forceinline__ void block_sum(double* sh, double v, double* out) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int w = kThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
  __syncthreads();
}

// Per block: sum over a fixed element range of w * sigma (NV entries) and w.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_homogenize(pgd::DevProblem P, const double* U, double* part) {
  constexpr int NPE = DIM + 1;
  constexpr int NV = (DIM == 2) ? 3 : 6;
  __shared__ double sh[kThreads];
  const int chunk = (P.ne + gridDim.x - 1) / gridDim.x;
  const int e0 = min(P.ne, (int)blockIdx.x * chunk), e1 = min(P.ne, e0 + chunk);
  double acc[NV + 1];
#pragma unroll
  for (int v = 0; v <= NV; ++v) acc[v] = 0.0;
  for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const int cc = P.cut_of[e];
    if (DIM == 2 && cc < 0 && P.npe == 4) {
      // uncut quad4: the four Gauss points of its bilinear map
      double x[4][2], u[4][2];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int id = P.conn[(size_t)e * 4 + n];
#pragma unroll
        for (int d = 0; d < 2; ++d) { x[n][d] = P.X[(size_t)id * 2 + d]; u[n][d] = U[(size_t)id * 2 + d]; }
      }
#pragma unroll
      for (int qp = 0; qp < 4; ++qp) {
        double g[4][2], w, eps[3];
        pgd::quad4_point(x, qp, g, &w);
#pragma unroll
        for (int v = 0; v < 3; ++v) eps[v] = P.subscale ? P.eps_macro[v] : 0.0;
#pragma unroll
        for (int n = 0; n < 4; ++n) pgd::add_strain<2, double>(g[n], u[n], eps);
        double sig[3];
        pgd::lei_stress<2, double>(P.Dd + 36 * P.emat[e], eps, sig);
#pragma unroll
        for (int v = 0; v < 3; ++v) acc[v] += w * sig[v];
        acc[NV] += w;
      }
    } else if (cc < 0) {
      double x[NPE][DIM], g[NPE][DIM], J, eps[NV];
      int nd[NPE];
#pragma unroll
      for (int n = 0; n < NPE; ++n) {
        nd[n] = P.conn[(size_t)e * NPE + n];
#pragma unroll
        for (int d = 0; d < DIM; ++d) x[n][d] = P.X[(size_t)nd[n] * DIM + d];
      }
      pgd::simplex_geom<DIM, double>(x, g, &J);
      const double w = J * ((DIM == 2) ? pgd::tri4_wsum() : pgd::tet5_wsum());
#pragma unroll
      for (int v = 0; v < NV; ++v) eps[v] = P.subscale ? P.eps_macro[v] : 0.0;
#pragma unroll
      for (int n = 0; n < NPE; ++n) {
        double u[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d] = U[(size_t)nd[n] * DIM + d];
        pgd::add_strain<DIM, double>(g[n], u, eps);
      }
      double sig[NV];
      pgd::lei_stress<DIM, double>(P.Dd + 36 * P.emat[e], eps, sig);
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] += w * sig[v];
      acc[NV] += w;
    } else {
      const int mn = P.cut_node_off[cc + 1] - P.cut_node_off[cc];
      const int* cn = P.cut_nodes + P.cut_node_off[cc];
      for (int qq = P.cut_qp_off[cc]; qq < P.cut_qp_off[cc + 1]; ++qq) {
        const double* gq = P.qp_grad + P.qp_grad_off[qq];
        double eps[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) eps[v] = P.subscale ? P.eps_macro[v] : 0.0;
        for (int n = 0; n < mn; ++n) {
          double u[DIM], gn[DIM];
#pragma unroll
          for (int d = 0; d < DIM; ++d) { u[d] = U[(size_t)cn[n] * DIM + d]; gn[d] = gq[n * DIM + d]; }
          pgd::add_strain<DIM, double>(gn, u, eps);
        }
        double sig[NV];
        pgd::lei_stress<DIM, double>(P.Dd + 36 * P.qp_mat[qq], eps, sig);
        const double w = P.qp_wgt[qq];
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] += w * sig[v];
        acc[NV] += w;
      }
    }
  }
  for (int v = 0; v <= NV; ++v) block_sum(sh, acc[v], &part[(size_t)v * gridDim.x + blockIdx.x]);
}

__global__ void k_homogenize_final(const double* part, int nb, int nv, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double vol = 0.0;
  for (int i = 0; i < nb; ++i) vol += part[(size_t)nv * nb + i];
  for (int v = 0; v < nv; ++v) {
    double s = 0.0;
    for (int i = 0; i < nb; ++i) s += part[(size_t)v * nb + i];
    out[v] = s / vol;
  }
  out[nv] = vol;
}

}  // namespace

extern "C" {

int pg_pcg_solve(pg_ctx* c, const double* d_b, double* d_x, int nrhs, double rtol, int max_it, int* iters,
                 double* relres) {
  if (!c || !d_b || !d_x || nrhs < 1 || nrhs > 16 || !(rtol > 0.0) || max_it < 1) return PG_ERR_INPUT;
  if (!pg_resident(c)) return pg_set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  if (!c->assembled) return pg_set_err(c, PG_ERR_STATE, "assemble K before solving with it");
  if (c->s.n_free == 0) return pg_set_err(c, PG_ERR_STATE, "no free degrees of freedom");
  if (int rc = pcg_reserve(c, std::min(nrhs, kMaxRhs))) return rc;
  PcgWork& w = c->pcg;
  // order after the assembly on the context's stream
  cudaEventRecord(w.ev, c->stream);
  cudaStreamWaitEvent(w.stream, w.ev, 0);
  bool all = true;
  for (int s = 0; s < nrhs; s += kMaxRhs) {
    const size_t o = (size_t)s * c->s.n_free;
    if (int rc = pcg_pass(c, d_b + o, d_x + o, std::min(kMaxRhs, nrhs - s), rtol, max_it, iters ? iters + s : nullptr,
                          relres ? relres + s : nullptr, &all))
      return rc;
  }
  // later work on the context's stream sees the solution
  cudaEventRecord(w.ev, w.stream);
  cudaStreamWaitEvent(c->stream, w.ev, 0);
  if (!all) return pg_set_err(c, PG_ERR_STATE, "PCG did not reach the tolerance within max_it");
  return 0;
}

int pg_homogenize(pg_ctx* c, const double* d_U, double t_frac, double* out) {
  if (!c || !d_U || !out) return PG_ERR_INPUT;
  if (!pg_resident(c)) return pg_set_err(c, PG_ERR_STATE, "the context has no device residency (pg_upload it first)");
  const int dim = c->s.dim, nv = dim == 2 ? 3 : 6;
  if (!c->d_hom && (pg_dalloc(c, (size_t)(nv + 2) * kHomBlocks + 8, &c->d_hom) || pg_alloc_sync(c))) return PG_ERR_DEVICE;
  pgd::DevProblem P = c->P;
  for (int v = 0; v < 6; ++v) P.eps_macro[v] = c->s.desc.eps_macro[v] * t_frac;
  if (dim == 2) k_homogenize<2><<<kHomBlocks, kThreads, 0, c->stream>>>(P, d_U, c->d_hom);
  else k_homogenize<3><<<kHomBlocks, kThreads, 0, c->stream>>>(P, d_U, c->d_hom);
  double* res = c->d_hom + (size_t)(nv + 1) * kHomBlocks;
  k_homogenize_final<<<1, 32, 0, c->stream>>>(c->d_hom, kHomBlocks, nv, res);
  double h[7];
  cudaMemcpyAsync(h, res, sizeof(double) * (nv + 1), cudaMemcpyDeviceToHost, c->stream);
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return pg_set_err(c, PG_ERR_DEVICE, "homogenization failed");
  std::memcpy(out, h, sizeof(double) * (nv + 1));
  return 0;
}

}  // extern "C"
