// Hybrid solver: push-relabel with the vertices in a cluster's shared memory.
//
// For sparse graphs of up to 280,000 vertices whose arcs do not fit in shared
// memory.  Labels, excess and the BFS's bookkeeping (12 bytes a vertex, 20 with
// the rows where there is room) live in the distributed shared memory of one
// cluster of 16 blocks; the arcs are 16-byte records in global memory, which
// the 129 MB L2 holds.  A step's chain is then one L2 access (the record, which
// carries the twin's residual too), one remote shared-memory load (the head's
// label) and reductions that nobody waits for, and its barrier is the
// cluster's: about 3 us a round and 1.4 us a BFS level on GENRMF 32x64, where
// the persistent kernel takes 17 and 8 us on up to 304 blocks.  Rounds, labels
// and relabel trigger are those of the resident solver (resident.cu).
//
// The vertices are dealt to the blocks in turn: neighbours in vertex order tend
// to be active together, and with runs of consecutive vertices a BFS wave
// sits in one or two blocks (GENRMF 32x64 80 ms against 54, layered 40x2000
// 8.1 against 2.4 ms).  A warp collects the vertices to work on from all its
// groups before it starts, four at a time: their chains are what a step waits
// for (grid 512x512 34 ms with a chain for every fourth of every group, 17 ms
// with the list).  The twin's residual in the record saves the BFS a second L2
// access an arc (grid 512x512 37 -> 34 ms).
//
// Measured on GB300, persistent kernel and now:
//   GENRMF 32x64 (65,536 vertices)     183  -> 24 ms (mean of ten seeds)
//   GENRMF 40x80 (128,000 vertices)    230  -> 48 ms
//   grid 512x512 (three seeds)         45, 44, 21 -> 17, 17, 10-13 ms
//   grid 200x200                       27.3 -> 6.0 ms
//   layered 100x2500 (250,002)         14.6 -> 3.8-4.8 ms
//   layered 64x512                     6.1  -> 1.1 ms (2.0 ms resident)
// What bounds it: the chain of a step, and on the largest graphs the 16 SMs.
#include "resident.cuh"

namespace wbpr_dev {
namespace {

constexpr int kTile = 8;        // lanes of a row
// BFS levels a block runs between two cluster barriers.  GENRMF 32x64 (before
// the lists) 1, 2, 4, 8: 50.0, 48.0, 52.2, 53.7 ms; grid 512x512 (seeds 1, 3)
// 2, 4: 17.7, 12.6 and 17.1, 12.9 ms.
constexpr int kHybBfsLevels = 4;
// Global relabel once the rounds since the last one took this many sixteenths
// of its time.  16 against 24: GENRMF 32x64 32.7, 29.9 ms; grid 400x400
// 10.7-13.9, 11.3-13.8 ms; layered 40x2000 1.52, 1.51 ms.
constexpr int kHybGrShare = 20;

using Smem = Sh<true>;

// A block's share: `chunk` consecutive vertices.  Four consecutive slots belong
// to a lane, 128 to a group, which one warp looks after; vertices are dealt to
// the groups in turn, and in a group to its four 8-lane tiles in turn.
struct HPart {
  ResCtl* c;
  unsigned a0;                      // shared-memory address of the block's memory
  unsigned a_list, a_lab, a_e, a_ex, a_row;  // offsets from it
  int4* rec;
  int rank, cs, shift;     // cs = 1 << shift blocks
  int groups;
  int n, na;               // vertices and arcs of the instance
  int row0;                // arc number of record 0
  bool rows;               // rows are in shared memory
  int sl, tl;              // s and t among this block's slots, or -1
  int sv, tv;              // s and t as (block << 16 | slot), -1 for none
  __device__ __forceinline__ int slot(int j) const {
    const int q = j / groups;
    return (j - q * groups) * 128 + ((q & 3) * 8 + (q >> 2 & 7)) * 4 + (q >> 5);
  }
  // the vertex in a slot of this block (>= n: the slot is empty)
  __device__ __forceinline__ int vertex(int s) const {
    const int l = s >> 2 & 31, q = (s & 3) * 32 + (l & 7) * 4 + (l >> 3);
    return (q * groups + (s >> 7)) * cs + rank;
  }
  // a head's memory, its slot there, and an arc, in range
  __device__ __forceinline__ unsigned mem(int head) const { return Smem::at(a0, within(c, (unsigned)head >> 16, cs)); }
  __device__ __forceinline__ unsigned at(int head) const { return 4 * within(c, head & 0xffff, 128 * groups); }
  __device__ __forceinline__ int arc(int a) const { return (int)within(c, a, na); }
  __device__ __forceinline__ int code(int v) const { return (v & (cs - 1)) << 16 | slot(v >> shift); }
};

__device__ __forceinline__ int4 lds128(unsigned a) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts128(unsigned a, const int4& v) {
  asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts32(unsigned a, int v) { asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
// A record: {residual, residual of the twin, head (block << 16 | slot), twin}.
// Records are read and changed in L2, where every block sees them.  Moving v
// units along an arc is one 64-bit add in each of the two records: the lower
// word never goes below zero and the upper one never above a capacity, so
// nothing is carried between the words.
__device__ __forceinline__ void move(int4* rec, int a, int v) {  // v out of a's residual, into its twin's
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(rec + a), "l"(((long long)v << 32) - v) : "memory");
}
__device__ __forceinline__ int resid(const int4* rec, int a) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(&rec[a].x) : "memory");
  return v;
}
__device__ __forceinline__ int4 record(const int4* rec, int a) {
  int4 v;
  asm volatile("ld.global.cg.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(rec + a) : "memory");
  return v;
}

// How the vertices are dealt to a cluster of cs blocks.
__device__ void shape(const ResInstance& in, int4* rec, int cs, HPart& P) {
  P.cs = cs;
  P.shift = 31 - __clz(cs);
  P.n = in.n;
  P.rec = rec;
  P.row0 = row_at(in, 0);
  P.na = row_at(in, in.n) - P.row0;
  P.groups = max(kResThreads >> 5, ((in.n + cs - 1) / cs + 127) >> 7);
}

__device__ void setup(const ResInstance& in, int4* rec, char* sm, HPart& P) {
  ResCtl* c = (ResCtl*)sm;
  P.c = c;
  shape(in, rec, (int)cl_size(), P);
  P.rank = (int)cl_rank();
  const unsigned slots = 128 * P.groups;
  P.a0 = sm_addr(sm);
  P.a_list = (sizeof(ResCtl) + 15) & ~15u;
  P.a_lab = P.a_list + kHybListBytes;
  P.a_e = P.a_lab + 4 * slots;
  P.a_ex = P.a_e + 4 * slots;
  P.a_row = P.a_ex + 4 * slots;
  P.rows = P.a_row + kHybRowBytes * slots <= (unsigned)kResSmem;
  P.sv = in.s >= 0 ? P.code(in.s) : -1;
  P.tv = P.code(in.t);
  P.sl = P.sv >= 0 && P.sv >> 16 == P.rank ? P.sv & 0xffff : -1;
  P.tl = P.tv >> 16 == P.rank ? P.tv & 0xffff : -1;
  if (threadIdx.x < 8) c->sum[threadIdx.x] = 0;
  if (threadIdx.x == 0) c->busy[0] = c->busy[1] = c->stop = c->gr = c->viol = 0;
  for (unsigned i = threadIdx.x; i < slots; i += blockDim.x) {
    const int v = P.vertex(i);
    int e = 0, b = 0, d = 0;
    if (v < P.n) {
      if (in.mode == kModeState) e = __ldcg(in.e + in.vbase + v);
      b = row_at(in, v);
      d = row_at(in, v + 1) - b;
    }
    sts32(P.a0 + P.a_lab + 4 * i, P.n);
    sts32(P.a0 + P.a_e + 4 * i, e);
    sts32(P.a0 + P.a_ex + 4 * i, 0);
    if (P.rows) {
      sts32(P.a0 + P.a_row + 8 * i, b - P.row0);
      sts32(P.a0 + P.a_row + 8 * i + 4, d);
    }
  }
}

__device__ __forceinline__ int2 row_of(const ResInstance& in, const HPart& P, int u) {
  if (P.rows) return lds64(P.a0 + P.a_row + 8 * u);
  const int v = P.vertex(u), b = row_at(in, v);
  return make_int2(b - P.row0, row_at(in, v + 1) - b);
}

// Builds the records, every arc by the next of nt threads.
__device__ void build_records(const ResInstance& in, const HPart& P, int tid, int nt) {
  const bool fresh = in.mode == kModeFresh;
  if (in.row) {
    const int na = row_at(in, in.n) - P.row0;
#pragma unroll 4
    for (int a = tid; a < na; a += nt) {
      const int2 r = __ldcg(in.arc + P.row0 + a), x = __ldg(in.arx + P.row0 + a);
      const int other = fresh ? __ldg(&in.arx[x.x].y) : __ldcg(&in.arc[x.x].y);
      P.rec[a] = make_int4(fresh ? x.y : r.y, other, P.code(r.x - in.vbase), x.x - P.row0);
    }
    return;
  }
  // RCSR: reverse entry k of v, {tail, forward arc}, gives both records
  const int m = __ldg(in.rrow + in.n);
  for (int k = tid; k < m; k += nt) {
    int lo = 0, hi = in.n;  // the row of k: the last v with rrow[v] <= k
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(in.rrow + mid) <= k) lo = mid;
      else hi = mid;
    }
    const int2 r = __ldg(in.rarc + k);
    const int here = __ldg(in.frow + lo + 1) + k, fwd = r.y + __ldg(in.rrow + r.x);
    const int cf = fresh ? __ldg(in.fcap + r.y) : __ldcg(&in.farc[r.y].y), cb = fresh ? 0 : __ldcg(in.fcb + r.y);
    P.rec[fwd] = make_int4(cf, cb, P.code(lo), here);
    P.rec[here] = make_int4(cb, cf, P.code(r.x), fwd);
  }
}

__device__ void write_back(const ResInstance& in, const HPart& P) {
  for (int i = threadIdx.x; i < 128 * P.groups; i += blockDim.x) {
    const int v = P.vertex(i);
    if (v >= P.n) continue;
    in.lab[in.vbase + v] = (int)lds32(P.a0 + P.a_lab + 4 * i);
    if (in.mode != kModeBfsOnly) in.e[in.vbase + v] = (int)lds32(P.a0 + P.a_e + 4 * i);
  }
}

// The residuals from the records, every arc by the next of nt threads.
__device__ void write_arcs(const ResInstance& in, const HPart& P, int tid, int nt) {
  if (in.row) {
    const int na = row_at(in, in.n) - P.row0;
#pragma unroll 4
    for (int a = tid; a < na; a += nt) in.arc[P.row0 + a].y = resid(P.rec, a);
    return;
  }
  const int m = __ldg(in.rrow + in.n);
  for (int k = tid; k < m; k += nt) {
    const int2 r = __ldg(in.rarc + k);
    const int cf = resid(P.rec, r.y + __ldg(in.rrow + r.x));
    in.farc[r.y].y = cf;
    in.fcb[r.y] = __ldg(in.fcap + r.y) - cf;
  }
}

// Lowers the label of arc a's head to nl where the arc (DIR 1) or its twin
// (DIR 0) has residual.
template <int DIR>
__device__ __forceinline__ void bfs_arc(const HPart& P, int a, int nl) {
  const int4 r = record(P.rec, P.arc(a));
  if ((DIR == 0 ? r.y : r.x) <= 0 || r.z == P.sv) return;
  const unsigned al = P.mem(r.z) + P.a_lab + P.at(r.z);
  if (Smem::ld(al) > nl) Smem::min(al, nl);
}

// The warp's list of slots to work on in this step; up to 128 more fit while
// it holds at most 128.
struct List {
  unsigned at;  // shared-memory address
  int n = 0;
  __device__ __forceinline__ explicit List(const HPart& P) : at(P.a0 + P.a_list + (threadIdx.x >> 5) * kHybListBytes / (kResThreads / 32)) {}
  // the slots 128 * g + 4 * lane + q whose bit q of `open` is set
  __device__ __forceinline__ void add(int g, unsigned open) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned m = __ballot_sync(kFull, open >> q & 1);
      if (open >> q & 1)
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(at + 2 * (n + __popc(m & ((1u << lane) - 1u)))), "h"((unsigned short)(128 * g + 4 * lane + q)) : "memory");
      n += __popc(m);
    }
  }
  // calls f(slot) for all of them, 32 / W at once (-1 for a tile without one)
  template <int W, class F>
  __device__ __forceinline__ void drain(F f) {
    __syncwarp();
    for (int i = 0; i < n; i += 32 / W) {
      const int k = i + (threadIdx.x & 31) / W;
      f(k < n ? (int)lds16(at + 2 * k) : -1);
    }
    __syncwarp();
    n = 0;
  }
};

template <int W, int DIR>
__device__ __forceinline__ void bfs_expand(const ResInstance& in, const HPart& P, int u, Count& ct) {
  const int lane = threadIdx.x & (W - 1);
  if (u < 0) return;
  const int2 row = row_of(in, P, u);
  const int nl = (int)lds32(P.a0 + P.a_ex + 4 * u) + 1;
  for (int k = lane; k < row.y; k += 2 * W) {
    const int4 r = record(P.rec, P.arc(row.x + k));
    int4 r2 = make_int4(0, 0, P.sv, 0);
    if (k + W < row.y) r2 = record(P.rec, P.arc(row.x + k + W));
    const bool ok = (DIR == 0 ? r.y : r.x) > 0 && r.z != P.sv, ok2 = (DIR == 0 ? r2.y : r2.x) > 0 && r2.z != P.sv;
    const int z2 = ok2 ? r2.z : 0;
    const unsigned al = P.mem(r.z) + P.a_lab + P.at(r.z), al2 = P.mem(z2) + P.a_lab + P.at(z2);
    int l = 0, l2 = 0;
    if (ok) l = Smem::ld(al);
    if (ok2) l2 = Smem::ld(al2);
    if (l > nl) Smem::min(al, nl);
    if (l2 > nl) Smem::min(al2, nl);
  }
  if (lane == 0) ct.bfs += row.y;
}

// Exact distances to (DIR 0) or from (DIR 1) t, as in the resident solver.
// The root's row, which may be the graph's longest, is shared by all blocks.
template <int DIR>
__device__ int bfs_hybrid(const ResParams& p, const HPart& P, int& seq, Count& ct) {
  const ResInstance& in = p.in;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = threadIdx.x; i < 128 * P.groups; i += blockDim.x) {
    sts32(P.a0 + P.a_lab + 4 * i, i == P.tl ? 0 : P.n);
    sts32(P.a0 + P.a_ex + 4 * i, i == P.tl ? 0 : P.n);
  }
  Smem::sync();
  {
    const int b = row_at(in, in.t) - P.row0, e = row_at(in, in.t + 1) - P.row0;
    for (int a = b + P.rank * blockDim.x + threadIdx.x; a < e; a += P.cs * blockDim.x) bfs_arc<DIR>(P, a, 1);
    if (P.tl >= 0 && threadIdx.x == 0) ct.bfs += e - b;
  }
  Smem::sync();
  int levels = 1;
  List list(P);
  for (;;) {
    bool did = false;
    for (int k = 0; k < p.run.bsub; ++k) {
      bool now = false;
      const auto expand = [&](int u) { bfs_expand<kTile, DIR>(in, P, u, ct); };
      for (int g = wid; g < P.groups; g += nw) {
        const unsigned at = 512 * g + 16 * lane;
        const int4 l = lds128(P.a0 + P.a_lab + at), x = lds128(P.a0 + P.a_ex + at);
        const unsigned open = (l.x < x.x) | (l.y < x.y) << 1 | (l.z < x.z) << 2 | (l.w < x.w) << 3;
        if (!__any_sync(kFull, open)) continue;
        now = true;
        if (open)
          sts128(P.a0 + P.a_ex + at, make_int4(min(l.x, x.x), min(l.y, x.y), min(l.z, x.z), min(l.w, x.w)));
        list.add(g, open);
        if (list.n > 128) list.drain<kTile>(expand);
      }
      list.drain<kTile>(expand);
      did |= now;
      if (k + 1 < p.run.bsub && !__syncthreads_or(now)) break;
    }
    if (!any_work<true>(P.c, P.a0, P.cs, did, seq)) return levels;
    levels += p.run.bsub;
  }
}

// Push and relabel, as discharge() of the resident solver (the same argument
// keeps the labels valid, and E is what one lane read); pushes into t are summed by the thread.
template <int W>
__device__ __forceinline__ void discharge(const ResInstance& in, const HPart& P, int u, int& sink, Count& ct) {
  const int lane = threadIdx.x & (W - 1);
  lanes_apart();
  int E = 0, hu = 0;  // (no other warp writes the label)
  int2 row = make_int2(0, 0);
  if (u >= 0) {
    if (lane == 0) E = (int)lds32(P.a0 + P.a_e + 4 * u);
    hu = (int)lds32(P.a0 + P.a_lab + 4 * u);
    row = row_of(in, P, u);
  }
  E = __shfl_sync(kFull, E, 0, W);
  unsigned erem = (unsigned)E;
  int mn = kBig, k = 0;
  constexpr int Q = 2;
  do {
    int4 r[Q];
    unsigned m[Q], room[Q], own = 0;
    int hv[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int i = k + q * W + lane;
      r[q] = make_int4(0, 0, 0, 0);
      if (i < row.y && erem > 0) r[q] = record(P.rec, P.arc(row.x + i));
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      m[q] = P.mem(r[q].z) + P.at(r[q].z);
      hv[q] = kBig;
      if (r[q].x > 0) hv[q] = Smem::ld(m[q] + P.a_lab);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      room[q] = hv[q] < hu ? (unsigned)r[q].x : 0u;
      own = min(own + room[q], erem);
    }
    if (__any_sync(kFull, own > 0)) {
      unsigned incl = own;
#pragma unroll
      for (int d = 1; d < W; d <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, incl, d, W);
        if (lane >= d) incl = min(incl + y, erem);
      }
      unsigned before = __shfl_up_sync(kFull, incl, 1, W);
      if (lane == 0) before = 0;
      const unsigned total = __shfl_sync(kFull, incl, W - 1, W);
      unsigned left = erem - before;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int push = (int)min(room[q], left);
        left -= push;
        if (push > 0) {
          move(P.rec, P.arc(row.x + k + q * W + lane), push);
          move(P.rec, P.arc(r[q].w), -push);
          if (r[q].z == P.tv) sink += push;
          else Smem::add(m[q] + P.a_e, push);
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
  } while (__any_sync(kFull, k < row.y && erem > 0));
  if (__any_sync(kFull, erem > 0)) {
#pragma unroll
    for (int d = W / 2; d > 0; d >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, d, W));
    if (lane == 0 && erem > 0) {
      sts32(P.a0 + P.a_lab + 4 * u, min(max(min(mn, hu + 1), hu) + 1, P.n));
      ++ct.relabels;
    }
  }
  if (lane == 0 && u >= 0) {
    ct.scanned += min(k, row.y);
    ++ct.visits;
    if (E > (int)erem) Sh<false>::add(P.a0 + P.a_e + 4 * u, (int)erem - E);
  }
}

__device__ bool push_step(const ResInstance& in, const HPart& P, Count& ct) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  bool did = false;
  int sink = 0;
  List list(P);
  const auto work = [&](int u) { discharge<kTile>(in, P, u, sink, ct); };
  for (int g = wid; g < P.groups; g += nw) {
    const unsigned at = 512 * g + 16 * lane;
    const int4 e = lds128(P.a0 + P.a_e + at);
    if (!__any_sync(kFull, e.x > 0 || e.y > 0 || e.z > 0 || e.w > 0)) continue;
    const int4 l = lds128(P.a0 + P.a_lab + at);  // s keeps label n
    unsigned act = (e.x > 0 && l.x < P.n) | (e.y > 0 && l.y < P.n) << 1 | (e.z > 0 && l.z < P.n) << 2 | (e.w > 0 && l.w < P.n) << 3;
    if (P.tl >> 2 == 32 * g + lane) act &= ~(1u << (P.tl & 3));
    list.add(g, act);
    did |= list.n > 0;
    if (list.n > 128) list.drain<kTile>(work);
  }
  list.drain<kTile>(work);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sink += __shfl_xor_sync(kFull, sink, o);
  if (lane == 0 && sink) Smem::add(Smem::at(P.a0, (unsigned)P.tv >> 16) + P.a_e + 4 * (P.tv & 0xffff), sink);
  return did;
}

__device__ void solve_hybrid(const ResParams& p, const HPart& P) {
  const ResInstance& in = p.in;
  Count ct;
  int seq = 0, grs = 0, rounds = 0, since = 0, err = 0, total_levels = 0;
  solve_begins(P.c);
  if (in.mode == kModeBfsOnly) {
    if (in.dir == 0) bfs_hybrid<0>(p, P, seq, ct);
    else bfs_hybrid<1>(p, P, seq, ct);
  } else {
    if (in.mode == kModeFresh) {
      // preflow: every residual arc out of s, by all blocks
      const int b = row_at(in, in.s) - P.row0, e = row_at(in, in.s + 1) - P.row0;
      for (int a = b + P.rank * blockDim.x + threadIdx.x; a < e; a += P.cs * blockDim.x) {
        const int4 r = record(P.rec, P.arc(a));
        if (r.x <= 0 || r.z == P.sv) continue;
        move(P.rec, P.arc(a), r.x);
        move(P.rec, P.arc(r.w), -r.x);
        Smem::add(P.mem(r.z) + P.a_e + P.at(r.z), r.x);
      }
      Smem::sync();
    }
    bool need_gr = true;
    for (;;) {
      if (need_gr) {
        relabel_begins(P.c);
        total_levels += bfs_hybrid<0>(p, P, seq, ct);
        relabel_ends(P.c);
        ++grs;
        since = 0;
      }
      const bool did = push_step(in, P, ct);
      decide<true>(P.c, P.a0, P.rank, P.cs, p.run, rounds, since, seq);
      if (!any_work<true>(P.c, P.a0, P.cs, did, seq)) break;
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
    for (int i = threadIdx.x; i < 128 * P.groups; i += blockDim.x)
      str += i != P.sl && i != P.tl && (int)lds32(P.a0 + P.a_e + 4 * i) > 0 && (int)lds32(P.a0 + P.a_lab + 4 * i) >= P.n;
    add_up<true>(P.c, P.a0, ct, str);
  }
  report(p.to, P.c, P.rank, in.mode != kModeBfsOnly && P.tl >= 0, P.tl >= 0 ? (int)lds32(P.a0 + P.a_e + 4 * P.tl) : 0, err, rounds, grs, total_levels);
}

extern __shared__ __align__(16) char hyb_smem[];

// A single solve's records are built, and its residuals written back, by the
// whole GPU in launches of their own: the cluster's 16 SMs took longer over
// them than over a solve of few rounds.  In the cluster and now, on RCSR (whose
// records need a search for the row of each reverse entry) and BCSR16: random
// graphs of 280,000 vertices with 1.7M arcs 1.81 -> 0.72 and 0.99 -> 0.66 ms,
// with 0.4M 1.25 -> 0.81 and 1.04 -> 0.97; sink side of the cut of a 512x512
// grid 1.07 -> 0.66 and 0.79 -> 0.64 ms.  Below 200,000 units nothing changes.
// (In a batch the other SMs have instances of their own.)
constexpr int kArcBlocks = 152 * 8;
__global__ void __launch_bounds__(256) hybrid_load(const __grid_constant__ ResParams p) {
  HPart P;
  shape(p.in, p.rec, kResMaxCluster, P);
  build_records(p.in, P, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void __launch_bounds__(256) hybrid_store(const __grid_constant__ ResParams p) {
  HPart P;
  shape(p.in, p.rec, kResMaxCluster, P);
  write_arcs(p.in, P, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(kResThreads, 1) pr_hybrid(const __grid_constant__ ResParams p) {
  HPart P;
  setup(p.in, p.rec, hyb_smem, P);
  Smem::sync();
  solve_hybrid(p, P);
}

__global__ void __launch_bounds__(kResThreads, 1) pr_hybrid_batch(const __grid_constant__ ResBatch b) {
  ResParams p;
  int4* rec = b.rec + b.rec_stride * (blockIdx.x / cl_size());
  while (claim<true>(b, hyb_smem, p, rec)) {
    HPart P;
    setup(p.in, p.rec, hyb_smem, P);
    build_records(p.in, P, P.rank * blockDim.x + threadIdx.x, P.cs * blockDim.x);
    Smem::sync();
    solve_hybrid(p, P);
  }
}

}  // namespace

cudaError_t launch_hybrid(const ResParams& p0, cudaStream_t st) {
  ResParams p = p0;
  p.run.bsub = kHybBfsLevels;
  p.run.grp = kHybGrShare;
  hybrid_load<<<kArcBlocks, 256, 0, st>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_cluster<pr_hybrid>(p, kResMaxCluster, st);
  if (e == cudaSuccess && p.keep && p.in.mode != kModeBfsOnly) {
    hybrid_store<<<kArcBlocks, 256, 0, st>>>(p);
    e = cudaGetLastError();
  }
  return e;
}

int hybrid_clusters(int blocks) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  if (cluster_config<pr_hybrid_batch>(blocks, 1024, nullptr, &cfg, at) != cudaSuccess) return 0;
  int n = 0, dev = 0, sms = 0;
  if (blocks == 1) {
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
  }
  if (cudaOccupancyMaxActiveClusters(&n, (const void*)pr_hybrid_batch, &cfg) != cudaSuccess) n = 0;
  cudaGetLastError();
  return n;
}

cudaError_t launch_hybrid_batch(const ResBatch& b0, int blocks, int clusters, cudaStream_t st) {
  ResBatch b = b0;
  b.run.bsub = kHybBfsLevels;
  b.run.grp = kHybGrShare;
  return launch_cluster<pr_hybrid_batch>(b, blocks, st, clusters);
}

}  // namespace wbpr_dev
