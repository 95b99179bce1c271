// Resident solver: push-relabel with the residual graph in shared memory.
//
// Small graphs are bound by latency, not by bytes: the persistent kernel
// (pr_kernel.cuh) spends 10-20 us on a round or a BFS level of a graph of a
// few thousand vertices, nearly all of it chains of dependent L2 accesses and
// the grid barrier.  Here the whole residual graph sits in the shared memory
// of one block, or of a cluster of 16 (distributed shared memory, the
// hardware's cluster barrier), from its first load to the write-back: 8 bytes
// an arc and 14 a vertex.  The vertices are split over the blocks in order,
// by weight; a block owns its vertices' labels, excess and rows, and reaches
// its neighbours' with remote loads and fire-and-forget remote reductions.
// There are no queues: each step, every warp looks over the state of the
// vertices it owns, which costs one shared-memory load a vertex and needs no
// returning atomic.  A step pushes and relabels in one pass (discharge()), so
// a round has one barrier instead of two.
//
// Measured on GB300, solve time before (persistent kernel, one seed) and now (mean
// of ten seeds where the families' names say no more):
//   GENRMF 4x5 (80 vertices, one block)            1.00 -> 0.11 ms
//   GENRMF 8x16 (1,024 vertices, one block), RCSR  7.69 -> 0.69 ms
//   layered 11x37 (409 vertices, one block), RCSR  1.91 -> 0.13 ms
//   GENRMF 16x40 (10,240 vertices, cluster)        33.8 -> 3.9 ms (one seed)
//   layered 32x256 (8,194 vertices, cluster)       2.96 -> 0.75 ms (one seed)
//   R-MAT scale 13 (230k residual arcs, cluster)   0.70 -> 0.48 ms, RCSR 0.78 -> 0.51
// A round takes 1.0-1.7 us in one block and about 2.2 us in the cluster, a BFS
// level 0.6-0.8 us in one block; what bounds it now is the length of one
// warp's instruction chain through discharge() (about 1,000 cycles) and, in
// the cluster, the block that holds most of the active vertices.
//
// Blocks of 1,024 threads: with 512, a warp looks after twice the vertices one
// after the other (GENRMF 8x16 0.89 against 0.67 ms).  A cluster is always 16
// blocks: the least number that fits is slower (GENRMF 16x40 on 8: 4.9 ms,
// layered 32x256 on 4: 0.85 ms), and a graph that fits one block is slower on
// 16 (GENRMF 8x16: 0.80 ms).
#include "resident.cuh"
#include "resident.h"

namespace wbpr_dev {
namespace {

// BFS levels a block runs between two cluster barriers (the search is
// label-correcting).  GENRMF 16x40: 1 level 4.88, 8 3.76, 32 4.0-5.5 ms;
// layered 32x256 0.85, 0.53, 0.5-0.8 ms.
constexpr int kResBfsLevels = 8;
// Global relabel once the rounds since the last one took this many sixteenths
// of its time, and at least 8 rounds.  In a cluster at 4, 8, 16, 24: GENRMF
// 16x40 9.2, 6.0, 3.8, 3.6 ms, layered 32x256 0.85, 0.93, 0.53, 0.66, R-MAT
// scale 13 0.40, 0.41, 0.48, 0.57.  In one block at 16, 24, 32, 48: GENRMF 8x16
// 0.67, 0.59, 0.58, 0.63 ms, 10x20 1.63, 1.52, 1.45, 1.56, layered 20x100
// 0.34, 0.33, 0.31, 0.29.
constexpr int kResGrShare = 16;
constexpr int kResGrShareBlock = 28;

// The layout of one block's memory and its share of the graph.  The vertices
// are dealt to the groups of 32 slots (a warp looks after a group) in turn, and
// within a group to its four runs of 8 slots in turn: neighbours in vertex
// order, which tend to be active together, fall to different warps, and the
// few vertices of a small graph to as many warps and tiles as there are.
struct Part {
  ResCtl* c;
  int2* rec;               // {residual, head (block << 12 | slot) | twin arc << 16}
  int2* ve;                // {label, excess} by slot
  unsigned* row;           // first arc | arcs << 16, by slot
  unsigned short* ex;      // label a vertex was last expanded with in the running BFS, by slot
  unsigned a0, a_rec, a_ve;  // shared-memory addresses: of the block's memory, of rec, of ve
  int cs, rank;
  unsigned a_row, a_ex;    // of row and ex
  bool big;                // some row of this block is longer than kBigRow
  int groups;              // of 32 slots, the same in every block
  int nv, na;              // vertices and arcs of this block
  int arcs;                // there is room for in every block
  int n;                   // of the instance
  int sv, tv;              // s and t as (block << 12 | slot), -1 for none
  int sl, tl;              // s and t among this block's slots, or -1
  __device__ __forceinline__ int slot(int j) const {
    const int q = j / groups;
    return (j - q * groups) * 32 + (q & 3) * 8 + (q >> 2);
  }
  // the memory of a head's block, the head's {label, excess} and an arc's record there
  template <bool CL>
  __device__ __forceinline__ unsigned mem(unsigned head) const {
    return Sh<CL>::at(a0, within(c, head >> 12, cs));
  }
  __device__ __forceinline__ unsigned ve_in(unsigned m, unsigned head) const { return m + a_ve + 8 * within(c, head & 0xfff, 32 * groups); }
  __device__ __forceinline__ unsigned rec_in(unsigned m, unsigned arc) const { return m + a_rec + 8 * within(c, arc, arcs); }
};

// First vertex of block k: a 32-way search by one warp over the monotone
// weight of the vertices before it.
__device__ __forceinline__ int boundary(const ResInstance& in, int row0, long long total, int k, int cs) {
  const int lane = threadIdx.x & 31;
  const long long target = total * k / cs;
  int lo = 0, hi = in.n;
  while (lo < hi) {
    const int step = (hi - lo + 31) >> 5;
    const int x = lo + lane * step;
    bool below = false;
    if (x < hi) below = (long long)kResVertexBytes * x + (long long)kResArcBytes * (row_at(in, x) - row0) < target;
    const int c = __popc(__ballot_sync(0xffffffffu, below));  // the predicate is monotone
    if (c == 0) break;
    const int nlo = lo + (c - 1) * step + 1;
    hi = min(hi, lo + c * step);
    lo = nlo;
  }
  return lo;
}

__device__ __forceinline__ int owner_of(const ResCtl* c, int cs, int v) {
  int lo = 0, hi = cs;  // the last block whose first vertex is <= v
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (c->bnd[m] <= v) lo = m;
    else hi = m;
  }
  return lo;
}

// Splits the instance over the cluster and lays out the memory; false when a
// block's share does not fit (all blocks agree).
template <bool CL>
__device__ bool setup(const ResInstance& in, char* sm, Part& P) {
  ResCtl* c = (ResCtl*)sm;
  P.c = c;
  P.cs = CL ? (int)cl_size() : 1;
  P.rank = CL ? (int)cl_rank() : 0;
  P.n = in.n;
  const int row0 = row_at(in, 0);
  const int rown = row_at(in, in.n);
  const long long total = (long long)kResVertexBytes * in.n + (long long)kResArcBytes * (rown - row0);
  const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = wid; k <= P.cs; k += nw) {
    const int v = k == 0 ? 0 : (k == P.cs ? in.n : boundary(in, row0, total, k, P.cs));
    if ((threadIdx.x & 31) == 0) {
      c->bnd[k] = v;
      c->abase[k] = row_at(in, v);
    }
  }
  if (threadIdx.x < 8) c->sum[threadIdx.x] = 0;
  if (threadIdx.x == 0) c->busy[0] = c->busy[1] = c->stop = c->gr = c->viol = 0;
  __syncthreads();
  int nvmax = 0, namax = 0;
  for (int k = 0; k < P.cs; ++k) {
    nvmax = max(nvmax, c->bnd[k + 1] - c->bnd[k]);
    namax = max(namax, c->abase[k + 1] - c->abase[k]);
  }
  P.groups = max((int)blockDim.x >> 5, (nvmax + 31) >> 5);
  P.arcs = namax;
  const int slots = 32 * P.groups;
  char* q = sm + ((sizeof(ResCtl) + 15) & ~15u);
  P.rec = (int2*)q;
  q += 8 * (size_t)namax;
  P.ve = (int2*)q;
  q += 8 * (size_t)slots;
  P.row = (unsigned*)q;
  q += 4 * (size_t)slots;
  P.ex = (unsigned short*)q;
  q += 2 * (size_t)slots;
  if (q > sm + kResSmem || slots > kResMaxVertices || namax > kResMaxArcs) return false;
  P.a0 = sm_addr(sm);
  P.a_rec = sm_addr(P.rec) - P.a0;
  P.a_ve = sm_addr(P.ve) - P.a0;
  P.a_row = sm_addr(P.row);
  P.a_ex = sm_addr(P.ex);
  P.nv = c->bnd[P.rank + 1] - c->bnd[P.rank];
  P.na = c->abase[P.rank + 1] - c->abase[P.rank];
  P.sv = P.tv = P.sl = P.tl = -1;
  if (in.s >= 0) {
    const int o = owner_of(c, P.cs, in.s), l = P.slot(in.s - c->bnd[o]);
    P.sv = o << 12 | l;
    if (o == P.rank) P.sl = l;
  }
  {
    const int o = owner_of(c, P.cs, in.t), l = P.slot(in.t - c->bnd[o]);
    P.tv = o << 12 | l;
    if (o == P.rank) P.tl = l;
  }
  return true;
}

constexpr unsigned kBigRow = 128;  // rows longer than this are walked by a whole warp

// The row of entry x of n rows with offsets o: the last j with o[j] <= x.
__device__ __forceinline__ int row_of_entry(const int* o, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(o + mid) <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Reads this block's rows (residuals from the capacities in a fresh solve).
template <bool CL>
__device__ void load(const ResInstance& in, Part& P) {
  const ResCtl* c = P.c;
  const int v0 = c->bnd[P.rank], a0 = c->abase[P.rank];
  const bool fresh = in.mode == kModeFresh;
  bool big = false;
  for (int i = threadIdx.x; i < 32 * P.groups; i += blockDim.x) {
    const int k = P.slot(i);
    P.ve[k] = make_int2(P.n, 0);
    P.row[k] = 0;
    P.ex[k] = 0;
    if (i >= P.nv) continue;
    const int b = row_at(in, v0 + i) - a0, e = row_at(in, v0 + i + 1) - a0;
    P.row[k] = (unsigned)b | (unsigned)(e - b) << 16;
    big |= (unsigned)(e - b) > kBigRow;
    if (in.mode == kModeState) P.ve[k].y = __ldcg(in.e + in.vbase + v0 + i);
  }
  P.big = __syncthreads_or(big);
  if (in.row) {
#pragma unroll 4
    for (int a = threadIdx.x; a < P.na; a += blockDim.x) {
      const int2 r = __ldcg(in.arc + a0 + a), x = __ldg(in.arx + a0 + a);
      const int d = (int)within(P.c, r.x - in.vbase, P.n), o = owner_of(c, P.cs, d);
      const unsigned tw = within(P.c, x.x - c->abase[o], P.arcs);
      P.rec[a] = make_int2(fresh ? x.y : r.y, (int)((unsigned)(o << 12 | P.slot(d - c->bnd[o])) | tw << 16));
    }
    Sh<CL>::sync();
    return;
  }
  Sh<CL>::sync();  // every block's memory may be written from here on
  // RCSR: a thread an entry, which finds its row by search.  (With 8 lanes a row
  // and a warp for one over 128 arcs, a load waited for its longest rows: the sink
  // side of the cut on R-MAT of 16 arcs a vertex, scale 10 0.283 -> 0.084 ms, scale
  // 13 0.233 -> 0.098; the persistent kernel's search takes 0.074 and 0.091.)
  const int f0 = __ldg(in.frow + v0), nf = __ldg(in.frow + v0 + P.nv) - f0, r0 = __ldg(in.rrow + v0);
  for (int k = threadIdx.x; k < P.na; k += blockDim.x) {
    if (k < nf) {
      const int f = f0 + k, v = v0 + row_of_entry(in.frow + v0, P.nv, f);
      int2 r = __ldcg(in.farc + f);
      r.x = (int)within(P.c, r.x, P.n);
      const int o = owner_of(c, P.cs, r.x);
      int2* q = P.rec + within(P.c, f + __ldg(in.rrow + v) - a0, P.arcs);
      q->x = fresh ? __ldg(in.fcap + f) : r.y;
      *(unsigned short*)&q->y = (unsigned short)(o << 12 | P.slot(r.x - c->bnd[o]));  // its twin is written below
    } else {
      const int e = r0 + k - nf, v = v0 + row_of_entry(in.rrow + v0, P.nv, e);
      int2 r = __ldg(in.rarc + e);  // {tail, forward arc}
      r.x = (int)within(P.c, r.x, P.n);
      const int o = owner_of(c, P.cs, r.x), here = (int)within(P.c, e + __ldg(in.frow + v + 1) - a0, P.arcs);
      const unsigned tw = within(P.c, r.y + __ldg(in.rrow + r.x) - c->abase[o], P.arcs);
      P.rec[here] = make_int2(fresh ? 0 : __ldcg(in.fcb + r.y), (int)((unsigned)(o << 12 | P.slot(r.x - c->bnd[o])) | tw << 16));
      Sh<CL>::st16(Sh<CL>::at(P.a0, o) + P.a_rec + 8 * tw + 6, (unsigned)here);
    }
  }
  Sh<CL>::sync();
}

__device__ void write_back(const ResInstance& in, const Part& P) {
  const ResCtl* c = P.c;
  const int v0 = c->bnd[P.rank], a0 = c->abase[P.rank];
  for (int i = threadIdx.x; i < P.nv; i += blockDim.x) {
    const int2 x = P.ve[P.slot(i)];
    in.lab[in.vbase + v0 + i] = x.x;
    if (in.mode != kModeBfsOnly) in.e[in.vbase + v0 + i] = x.y;
  }
  if (in.mode == kModeBfsOnly) return;
  if (in.row) {
    for (int a = threadIdx.x; a < P.na; a += blockDim.x) in.arc[a0 + a].y = P.rec[a].x;
    return;
  }
  const int f0 = __ldg(in.frow + v0), f1 = __ldg(in.frow + v0 + P.nv);
#pragma unroll 4
  for (int f = f0 + threadIdx.x; f < f1; f += blockDim.x) {
    const int v = v0 + row_of_entry(in.frow + v0, P.nv, f);
    const int cf = P.rec[f + __ldg(in.rrow + v) - a0].x;
    in.farc[f].y = cf;
    in.fcb[f] = __ldg(in.fcap + f) - cf;
  }
}

// Expands the vertices in slots u (one per W-lane tile, -1 for none) of label
// l: lowers the labels of the heads (DIR 0: over arcs whose twin has residual).
template <int W, bool CL, int DIR>
__device__ __forceinline__ void bfs_expand(const Part& P, int u, int l, Count& ct) {
  const unsigned lane = threadIdx.x & (W - 1);
  const unsigned row = u >= 0 ? lds32(P.a_row + 4 * u) : 0;
  const unsigned deg = row >> 16, first = row & 0xffff;
  const int nl = l + 1;
  for (unsigned k = lane; k < deg; k += W) {
    const int2 r = lds64(P.rec_in(P.a0, first + k));
    if (DIR == 1 && r.x <= 0) continue;
    const unsigned d = r.y & 0xffff, m = P.mem<CL>(d), al = P.ve_in(m, d);
    const int lv = Sh<CL>::ld(al);
    const int cf = DIR == 0 ? Sh<CL>::ld(P.rec_in(m, (unsigned)r.y >> 16)) : 1;
    if (lv > nl && cf > 0 && (int)d != P.sv) Sh<CL>::min(al, nl);
  }
  if (lane == 0) ct.bfs += deg;
}

// Exact distances to (DIR 0) or from (DIR 1) t over residual arcs, s never
// labelled, n where there is none: label-correcting, `bsub` levels inside a
// block between two cluster barriers.  Returns the levels of the longest run.
template <int W, bool CL, int DIR>
__device__ int bfs_resident(const ResParams& p, Part& P, int& seq, Count& ct) {
  for (int i = threadIdx.x; i < 32 * P.groups; i += blockDim.x) {
    P.ve[i].x = i == P.tl ? 0 : P.n;
    P.ex[i] = (unsigned short)min(P.n, 65535);
  }
  Sh<CL>::sync();
  int levels = 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (;;) {
    bool did = false;
    for (int k = 0; k < p.run.bsub; ++k) {
      bool now = false;
      for (int g = wid; g < P.groups; g += nw) {
        const int i = g * 32 + lane;
        const int l = (int)lds32(P.a0 + P.a_ve + 8 * i);
        const bool open = l < (int)lds16(P.a_ex + 2 * i);
        unsigned mask = __ballot_sync(kFull, open);
        if (!mask) continue;
        now = true;
        if (open) P.ex[i] = (unsigned short)l;
        if (W < 32 && P.big) {
          unsigned big = __ballot_sync(kFull, open && P.row[i] >> 16 > kBigRow);
          mask &= ~big;
          for (; big; big &= big - 1) {
            const int t = __ffs(big) - 1;
            bfs_expand<32, CL, DIR>(P, g * 32 + t, __shfl_sync(kFull, l, t), ct);
          }
        }
        while (mask) {  // the k-th lowest open one goes to tile k
          unsigned m = mask;
#pragma unroll
          for (int j = 0; j < 32 / W; ++j) {
            if (j < lane / W) m &= m - 1;
            mask &= mask - 1;
          }
          const int t = m ? __ffs(m) - 1 : -1;
          const int lt = __shfl_sync(kFull, l, t & 31);
          bfs_expand<W, CL, DIR>(P, t < 0 ? -1 : g * 32 + t, lt, ct);
        }
      }
      did |= now;
      if (k + 1 < p.run.bsub && !__syncthreads_or(now)) break;
    }
    if (!any_work<CL>(P.c, P.a0, P.cs, did, seq)) return levels;
    levels += p.run.bsub;
  }
}

// Push and relabel the active vertices in slots u (one per W-lane tile, -1
// for none; whole warps call it) that hold E.  Other warps and blocks add to a
// vertex's excess meanwhile, so E is what one lane read for all of them: lanes
// that read it each for themselves could see different values, and what they
// push would not be what the vertex loses.  A vertex's own label is the one it had when
// the step began; a head's label may be read before or after that head's
// relabel of the step.  An arc is admissible when the head's label is lower.
// Of the two ends of an arc at most one can push along it in a step, because
// an end only ever raises its label, after its pushes.  The new label is at
// most two above the old one, which keeps it valid against pushes of the same
// step into u that this scan has not seen: they come from labels at most one
// above u's.
template <int W, bool CL>
__device__ __forceinline__ void discharge(const Part& P, int u, int E, Count& ct) {
  const unsigned lane = threadIdx.x & (W - 1);
  lanes_apart();
  if (CL) {  // read again: in a cluster more has come by now (layered 40x300 with the older value 0.886 ms, 0.855 so)
    if (u >= 0 && lane == 0) E = (int)lds32(P.a0 + P.a_ve + 8 * u + 4);
    E = __shfl_sync(kFull, E, 0, W);
  }
  unsigned row = 0;
  int hu = 0;  // no other warp writes it
  if (u >= 0) {
    hu = (int)lds32(P.a0 + P.a_ve + 8 * u);
    row = lds32(P.a_row + 4 * u);
  }
  const unsigned deg = row >> 16, first = row & 0xffff;
  unsigned erem = (unsigned)E, k = 0;
  int mn = kBig;
  constexpr int Q = 2;
  do {
    int2 r[Q];
    unsigned m[Q], room[Q], own = 0;
    int hv[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned i = k + q * W + lane;
      r[q] = make_int2(0, 0);
      if (i < deg && erem > 0) r[q] = lds64(P.rec_in(P.a0, first + i));
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      m[q] = P.mem<CL>(r[q].y & 0xffff);
      hv[q] = kBig;
      if (r[q].x > 0) hv[q] = Sh<CL>::ld(P.ve_in(m[q], r[q].y & 0xffff));
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      room[q] = hv[q] < hu ? (unsigned)r[q].x : 0u;
      own = min(own + room[q], erem);
    }
    if (__any_sync(kFull, own > 0)) {
      // the tile's excess goes to its admissible arcs lane by lane
      unsigned incl = own;
#pragma unroll
      for (int d = 1; d < W; d <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, incl, d, W);
        if ((int)lane >= d) incl = min(incl + y, erem);
      }
      unsigned before = __shfl_up_sync(kFull, incl, 1, W);
      if (lane == 0) before = 0;
      const unsigned total = __shfl_sync(kFull, incl, W - 1, W);
      unsigned left = erem - before;  // what this lane's arcs may take
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int push = (int)min(room[q], left);
        left -= push;
        if (push > 0) {
          Sh<false>::add(P.rec_in(P.a0, first + k + q * W + lane), -push);
          Sh<CL>::add(P.rec_in(m[q], (unsigned)r[q].y >> 16), push);
          Sh<CL>::add(P.ve_in(m[q], r[q].y & 0xffff) + 4, push);
          ++ct.pushes;
        }
        if (r[q].x > push) mn = min(mn, hv[q]);
      }
      erem -= total;
    } else {
#pragma unroll
      for (int q = 0; q < Q; ++q) mn = min(mn, hv[q]);
    }
    k += W * Q;
  } while (__any_sync(kFull, k < deg && erem > 0));
  if (__any_sync(kFull, erem > 0)) {
#pragma unroll
    for (int d = W / 2; d > 0; d >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, d, W));
    if (lane == 0 && erem > 0) {
      P.ve[u].x = min(max(min(mn, hu + 1), hu) + 1, P.n);
      ++ct.relabels;
    }
  }
  if (lane == 0 && u >= 0) {
    ct.scanned += min(k, deg);
    ++ct.visits;
    if (E > (int)erem) Sh<false>::add(P.a0 + P.a_ve + 8 * u + 4, (int)erem - E);
  }
}

// One push / relabel step of this block; whether it had an active vertex.
template <int W, bool CL>
__device__ __forceinline__ bool push_step(const Part& P, Count& ct) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  bool did = false;
  for (int g = wid; g < P.groups; g += nw) {
    const int i = g * 32 + lane;
    const int2 le = lds64(P.a0 + P.a_ve + 8 * i);
    const bool act = le.y > 0 && le.x < P.n && i != P.tl;  // s keeps label n
    unsigned mask = __ballot_sync(kFull, act);
    if (!mask) continue;
    did = true;
    if (W < 32 && P.big) {
      unsigned big = __ballot_sync(kFull, act && P.row[i] >> 16 > kBigRow);
      mask &= ~big;
      for (; big; big &= big - 1) {
        const int t = __ffs(big) - 1;
        discharge<32, CL>(P, g * 32 + t, __shfl_sync(kFull, le.y, t), ct);
      }
    }
    // a tile takes the active ones among its own W slots
    unsigned mine = W == 32 ? mask : mask >> (lane & ~(W - 1)) & ((1u << (W & 31)) - 1u);
    while (__any_sync(kFull, mine)) {
      const int t = __ffs(mine) - 1, E = __shfl_sync(kFull, le.y, t & (W - 1), W);
      discharge<W, CL>(P, mine ? g * 32 + (lane & ~(W - 1)) + t : -1, mine ? E : 0, ct);
      mine &= mine - 1;
    }
  }
  return did;
}

template <int W, bool CL>
__device__ void solve_resident(const ResParams& p, Part& P) {
  const ResInstance& in = p.in;
  Count ct;
  int seq = 0, grs = 0, rounds = 0, since = 0, err = 0, total_levels = 0;
  solve_begins(P.c);
  if (in.mode == kModeBfsOnly) {
    if (in.dir == 0) bfs_resident<W, CL, 0>(p, P, seq, ct);
    else bfs_resident<W, CL, 1>(p, P, seq, ct);
  } else {
    if (in.mode == kModeFresh && P.sl >= 0) {
      // preflow: saturate every residual arc out of s
      const unsigned row = P.row[P.sl];
      for (int k = threadIdx.x; k < (int)(row >> 16); k += blockDim.x) {
        const int a = (row & 0xffff) + k;
        const int2 r = P.rec[a];
        const unsigned d = r.y & 0xffff, m = P.mem<CL>(d);
        if (r.x <= 0 || (int)d == P.sv) continue;
        P.rec[a].x = 0;
        Sh<CL>::add(P.rec_in(m, (unsigned)r.y >> 16), r.x);
        Sh<CL>::add(P.ve_in(m, d) + 4, r.x);
      }
    }
    Sh<CL>::sync();
    bool need_gr = true;
    for (;;) {
      if (need_gr) {
        relabel_begins(P.c);
        total_levels += bfs_resident<W, CL, 0>(p, P, seq, ct);
        relabel_ends(P.c);
        ++grs;
        since = 0;
      }
      const bool did = push_step<W, CL>(P, ct);
      decide<CL>(P.c, P.a0, P.rank, P.cs, p.run, rounds, since, seq);
      // the labels are valid after every step, so no active vertex means a
      // maximum preflow
      if (!any_work<CL>(P.c, P.a0, P.cs, did, seq)) break;
      if (*(volatile int*)&P.c->stop == seq) {
        err = (int)WBPR_ERR_NO_CONVERGENCE;
        break;
      }
      need_gr = *(volatile int*)&P.c->gr == seq;
      ++rounds;
      ++since;
    }
  }
  if (p.keep) write_back(in, P);
  if (kChecked || in.mode != kModeBfsOnly) {
    int str = 0;
    for (int i = threadIdx.x; i < 32 * P.groups; i += blockDim.x)
      str += i != P.sl && i != P.tl && P.ve[i].y > 0 && P.ve[i].x >= P.n;
    add_up<CL>(P.c, P.a0, ct, str);
  }
  report(p.to, P.c, P.rank, in.mode != kModeBfsOnly && P.tl >= 0, P.tl >= 0 ? P.ve[P.tl].y : 0, err, rounds, grs, total_levels);
}

extern __shared__ __align__(16) char res_smem[];

template <int W, bool CL>
__global__ void __launch_bounds__(kResThreads, 1) pr_resident(const __grid_constant__ ResParams p) {
  if (p.gate && (__ldcg(p.gate) | __ldcg(p.gate + 1) | __ldcg(p.gate + 2) | __ldcg(p.gate + 3))) return;
  Part P;
  if (!setup<CL>(p.in, res_smem, P)) {
    if (P.rank == 0 && threadIdx.x == 0) p.to.out->err = kResNoFit;
    return;
  }
  load<CL>(p.in, P);
  solve_resident<W, CL>(p, P);
}

__global__ void __launch_bounds__(kResThreads, 1) pr_resident_batch(const __grid_constant__ ResBatch b) {
  ResParams p;
  while (claim<false>(b, res_smem, p, nullptr)) {
    Part P;
    if (!setup<false>(p.in, res_smem, P)) {  // the host puts no such instance here
      if (threadIdx.x == 0) *p.to.flow = -1;
      continue;
    }
    load<false>(p.in, P);
    solve_resident<8, false>(p, P);
  }
}

}  // namespace

bool resident_one_block(long long n, long long na) {
  const long long slots = 32 * (n > kResThreads ? (n + 31) / 32 : kResThreads / 32);
  return (long long)((sizeof(ResCtl) + 15) & ~15u) + kResArcBytes * na + kResVertexBytes * slots <= kResSmem && slots <= kResMaxVertices &&
         na <= kResMaxArcs;
}

int resident_cluster(long long n, long long na) {
  if (resident_one_block(n, na)) return 1;
  // the blocks' shares are of equal weight, but for one row, and every block has
  // a slot a thread, used or not
  constexpr long long cs = kResMaxCluster, idle = kResVertexBytes * kResThreads;
  const long long w = kResVertexBytes * n + kResArcBytes * na;
  const long long share = (w + w / 32) / cs + (n < cs * kResThreads ? idle - kResVertexBytes * n / cs : 0);
  return share <= kResSmem - kResHeader && n <= cs * kResMaxVertices && na <= cs * kResMaxArcs ? (int)cs : 0;
}

cudaError_t launch_resident(const ResParams& p0, int tile, int cluster, cudaStream_t st) {
  ResParams p = p0;
  p.run.bsub = cluster == 1 ? 1 : kResBfsLevels;
  p.run.grp = cluster == 1 ? kResGrShareBlock : kResGrShare;
  if (cluster == 1) return tile < 32 ? launch_cluster<pr_resident<8, false>>(p, 1, st) : launch_cluster<pr_resident<32, false>>(p, 1, st);
  return tile < 32 ? launch_cluster<pr_resident<8, true>>(p, cluster, st) : launch_cluster<pr_resident<32, true>>(p, cluster, st);
}

cudaError_t launch_resident_batch(const ResBatch& b0, int blocks, cudaStream_t st) {
  ResBatch b = b0;
  b.run.bsub = 1;
  b.run.grp = kResGrShareBlock;
  return launch_cluster<pr_resident_batch>(b, 1, st, blocks);
}

}  // namespace wbpr_dev
