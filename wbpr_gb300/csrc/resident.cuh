// Device helpers shared by the solvers that keep a graph, or its vertices, in
// the shared memory of one thread block or of one thread-block cluster.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

#include "resident.h"

namespace wbpr_dev {
namespace {

constexpr int kResThreads = 1024;
constexpr unsigned kFull = 0xffffffffu;

struct ResCtl {
  int bnd[kResMaxCluster + 1];    // first vertex of every block of the cluster
  int abase[kResMaxCluster + 1];  // its first residual arc
  int busy[2];                    // number of the last barrier before which some block had work, by parity
  int stop;                       // number of the barrier after which every block stops: budget exhausted
  int gr;                         // number of the barrier after which every block relabels globally
  int item;                       // the claimed instance of a batch
  int viol;                       // checked build: indices of this block out of range
  unsigned long long sum[8];      // counters
  // times of the solve, kept by the block's first thread: cycle counter and ns
  // at its start, end and length of the last global relabel, length of all
  long long clk0, gr_end, gr_len, gr_all;
  unsigned long long t0;
};

// The checked build (compiled with -DWBPR_CHECKED): an index outside [0, lim) is
// counted, replaced by 0, and the solve returns WBPR_ERR_VERIFY.
#ifdef WBPR_CHECKED
constexpr bool kChecked = true;
#else
constexpr bool kChecked = false;
#endif
__device__ __forceinline__ unsigned within(ResCtl* c, unsigned i, unsigned lim) {
  if (!kChecked || i < lim) return i;
  atomicAdd(&c->viol, 1);
  return 0;
}

__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_map(unsigned a, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

// Shared memory of a block of the cluster (CL) or of this block.  at() gives
// the address of the memory of block `rank`; every block lays it out alike.
template <bool CL>
struct Sh {
  static __device__ __forceinline__ unsigned at(unsigned a0, unsigned rank) { return CL ? cl_map(a0, rank) : a0; }
  static __device__ __forceinline__ int ld(unsigned a) {
    int v;
    if (CL) asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a));
    else asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ void st(unsigned a, int v) {
    if (CL) asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    else asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
  static __device__ __forceinline__ void st16(unsigned a, unsigned v) {
    if (CL) asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory");
    else asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory");
  }
  static __device__ __forceinline__ void add(unsigned a, int v) {
    if (CL) asm volatile("red.relaxed.cluster.shared::cluster.add.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    else asm volatile("red.relaxed.cta.shared.add.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
  static __device__ __forceinline__ void add64(unsigned a, unsigned long long v) {
    if (CL) asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
    else asm volatile("red.relaxed.cta.shared.add.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
  }
  static __device__ __forceinline__ void min(unsigned a, int v) {
    if (CL) asm volatile("red.relaxed.cluster.shared::cluster.min.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    else asm volatile("red.relaxed.cta.shared.min.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
  static __device__ __forceinline__ void sync() {
    if (CL) {
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
      __syncthreads();
    }
  }
};

__device__ __forceinline__ int2 lds64(unsigned a) {
  int2 v;
  asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ unsigned lds32(unsigned a) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ unsigned lds16(unsigned a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}

// Whether any block of the cluster had work since its last call; every call
// is a barrier of the cluster.  `seq` numbers the calls: a warp with work
// posts the number to every block, so nothing has to be cleared.  There are
// two words, because a fast block may post the next number before a slow one
// has read this one (but not the number after it).
template <bool CL>
__device__ __forceinline__ bool any_work(ResCtl* c, unsigned a0, int cs, bool did, int& seq) {
  ++seq;
  if (!CL) return __syncthreads_or(did);
  if (did && (int)(threadIdx.x & 31) < cs)  // uniform over the warp
    Sh<CL>::st(Sh<CL>::at(a0, threadIdx.x & 31) + (unsigned)offsetof(ResCtl, busy) + 4 * (seq & 1), seq);
  Sh<CL>::sync();
  return *(volatile int*)&c->busy[seq & 1] == seq;
}

// Nothing keeps the lanes of a warp together where they need not be: the
// checked build calls this to have them come one after the other.
__device__ __forceinline__ void lanes_apart() {
  if (kChecked) __nanosleep(64 * (threadIdx.x & 31));
}

struct Count {  // of one thread
  unsigned scanned = 0, bfs = 0, pushes = 0, relabels = 0, visits = 0;
};

// Row offset of vertex v (0..n) in combined arc numbering.
__device__ __forceinline__ int row_at(const ResInstance& in, int v) {
  return in.row ? __ldg(in.row + in.vbase + v) : __ldg(in.frow + v) + __ldg(in.rrow + v);
}

// The counters of one solve: warps into the block's words, blocks into the
// first block's.  A barrier.
template <bool CL>
__device__ __forceinline__ void add_up(ResCtl* c, unsigned a0, const Count& ct, int stranded) {
  if (kChecked) __syncthreads();  // every index has been checked
  unsigned long long v[7] = {ct.scanned, ct.bfs, ct.pushes, ct.relabels, ct.visits, (unsigned)stranded,
                             kChecked && threadIdx.x == 0 ? (unsigned)c->viol : 0};
#pragma unroll
  for (int k = 0; k < (kChecked ? 7 : 6); ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(kFull, v[k], o);
    if ((threadIdx.x & 31) == 0 && v[k]) Sh<CL>::add64(Sh<CL>::at(a0, 0) + (unsigned)offsetof(ResCtl, sum) + 8 * k, v[k]);
  }
  Sh<CL>::sync();
}

// The times of a solve, of a global relabel and between the two.
__device__ __forceinline__ void solve_begins(ResCtl* c) {
  if (threadIdx.x != 0) return;
  c->clk0 = clock64();
  c->t0 = gtime();
  c->gr_all = 0;
}
__device__ __forceinline__ void relabel_begins(ResCtl* c) {
  if (threadIdx.x == 0) c->gr_len = -clock64();
}
__device__ __forceinline__ void relabel_ends(ResCtl* c) {
  if (threadIdx.x != 0) return;
  c->gr_end = clock64();
  c->gr_len += c->gr_end;
  c->gr_all += c->gr_len;
}

// Whether the cluster stops (a budget is exhausted) or relabels globally after
// its next barrier, number seq + 1: one lane of the first block decides, and its
// warp posts the number to every block.  (Not a flag: a slow block may read the
// word only after a fast one has reached the barrier after it.  Not every lane
// for its own block: they could read the clock at different times, and blocks
// that decided differently would wait for each other forever.)
template <bool CL>
__device__ __forceinline__ void decide(ResCtl* c, unsigned a0, int rank, int cs, const ResRun& run, int rounds, int since, int seq) {
  if (rank != 0 || threadIdx.x >= 32) return;
  bool stop = false, gr = false;
  lanes_apart();
  if (threadIdx.x == 0) {
    // the cycle counter first (cheaper to read; an SM does over half a cycle per ns)
    const long long now = clock64();
    stop = (run.max_rounds > 0 && rounds >= run.max_rounds) ||
           ((unsigned long long)(now - c->clk0) >= run.budget_ns >> 1 && time_past(c->t0, run.budget_ns));
    gr = since >= 8 && (now - c->gr_end) * 16 >= c->gr_len * run.grp;
  }
  stop = __shfl_sync(kFull, stop, 0);
  gr = __shfl_sync(kFull, gr, 0);
  if ((int)threadIdx.x >= cs) return;
  const unsigned to = Sh<CL>::at(a0, threadIdx.x);
  if (stop) Sh<CL>::st(to + (unsigned)offsetof(ResCtl, stop), seq + 1);
  if (gr) Sh<CL>::st(to + (unsigned)offsetof(ResCtl, gr), seq + 1);
}

// Writes the results of one solve (called by every thread of the cluster
// behind the barrier after which c->sum is complete); `mine`: this block owns
// t, whose excess is `flow`.
__device__ __forceinline__ void report(const ResReport& to, const ResCtl* c, int rank, bool mine, int flow, int err, int rounds, int grs,
                                       int levels) {
  if (threadIdx.x != 0) return;
  const unsigned long long ns = gtime() - c->t0;
  if (kChecked && rank == 0 && c->sum[6]) err = (int)WBPR_ERR_VERIFY;
  if (mine) {
    if (to.out) to.out->flow = flow;
    else *to.flow = err ? -1 : flow;
  }
  if (rank != 0) return;
  if (!to.out) {
    *to.ns = ns;
    *to.rounds = rounds;
    return;
  }
  Stats s{};
  s.arcs_scanned = c->sum[0];
  s.bfs_arcs = c->sum[1];
  s.pushes = c->sum[2];
  s.relabels = c->sum[3];
  s.vertex_visits = c->sum[4];
  s.stranded = (int)c->sum[5];
  s.rounds = rounds;
  s.grs = grs;
  s.bfs_levels = levels;
  s.gr_ns = (unsigned long long)((double)ns * ((double)c->gr_all / (double)(clock64() - c->clk0)));
  s.push_ns = s.round_ns = ns - s.gr_ns;
  to.out->st = s;
  to.out->err = err;
}

// The next instance of a batch for this block or cluster; false when none is
// left.  A barrier: the memory of the last instance is free afterwards.
template <bool CL>
__device__ bool claim(const ResBatch& b, char* sm, ResParams& p, int4* rec) {
  ResCtl* c = (ResCtl*)sm;
  const unsigned rank = CL ? cl_rank() : 0, cs = CL ? cl_size() : 1;
  Sh<CL>::sync();  // every block is done with the last instance (and has started)
  if (rank == 0 && threadIdx.x == 0) {
    const int i = atomicAdd(b.next, 1);
    for (unsigned k = 0; k < cs; ++k) Sh<CL>::st(Sh<CL>::at(sm_addr(sm), k) + (unsigned)offsetof(ResCtl, item), i);
  }
  Sh<CL>::sync();
  const int i = *(volatile int*)&c->item;
  if (i >= b.count) return false;
  const int id = __ldg(b.order + i);
  const ResInst in = b.inst[id];
  p.in = ResInstance{};
  p.in.n = in.n;
  p.in.vbase = in.vbase;
  p.in.s = in.s - in.vbase;
  p.in.t = in.t - in.vbase;
  p.in.mode = kModeFresh;
  p.in.row = b.row;
  p.in.arc = b.arc;
  p.in.arx = b.arx;
  p.in.lab = b.lab;
  p.in.e = b.e;
  p.to = ResReport{nullptr, b.flows + id, b.inst_ns + id, b.inst_rounds + id};
  p.run = b.run;
  p.keep = false;
  p.rec = rec;
  return true;
}

// The launch configuration of `clusters` clusters of `blocks` blocks each, with the whole shared memory of an SM for every block.
template <auto Fn>
cudaError_t cluster_config(int blocks, int clusters, cudaStream_t st, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  static std::mutex mu;
  static bool ready[64] = {false};  // of this kernel, by device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 64 || !ready[dev]) {
      if ((e = cudaFuncSetAttribute((const void*)Fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem)) != cudaSuccess) return e;
      if ((e = cudaFuncSetAttribute((const void*)Fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
      if (dev < 64) ready[dev] = true;
    }
  }
  cfg->gridDim = dim3(blocks * clusters);
  cfg->blockDim = dim3(kResThreads);
  cfg->dynamicSmemBytes = kResSmem;
  cfg->stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = blocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = blocks > 1 ? 1 : 0;  // a block without one is a cluster of its own
  return cudaSuccess;
}
template <auto Fn, class Prm>
cudaError_t launch_cluster(const Prm& p, int blocks, cudaStream_t st, int clusters = 1) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  const cudaError_t e = cluster_config<Fn>(blocks, clusters, st, &cfg, at);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&p};
  return cudaLaunchKernelExC(&cfg, (const void*)Fn, args);
}

}  // namespace
}  // namespace wbpr_dev
