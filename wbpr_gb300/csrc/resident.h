// The resident solver: a whole solve with the residual graph held in the
// shared memory of one thread block, or of one thread-block cluster.
#pragma once

#include <cuda_runtime.h>

#include "pr_kernel.cuh"

namespace wbpr_dev {

constexpr int kResMaxCluster = 16;      // blocks of a cluster (16: the non-portable maximum)
constexpr int kResMaxVertices = 4096;   // vertices of one block (12 bits of a record's head)
constexpr int kResMaxArcs = 65535;      // residual arcs of one block (16 bits of a record's twin)
constexpr int kResSmem = 227 * 1024;    // shared memory of one block
constexpr int kResVertexBytes = 14;     // label, excess, row, list, expanded label
constexpr int kResArcBytes = 8;         // {residual, head | twin << 16}
constexpr int kResHeader = 2048;        // control words, and slack for alignment
// status of a launch whose partition does not fit (nothing was changed)
constexpr int kResNoFit = -1;

// What one launch reports; written by the launch, no clearing needed.
struct ResOut {
  Stats st;
  int err;
  int flow;
};

// One instance: vertices vbase .. vbase + n - 1 of either layout.
struct ResInstance {
  int n;
  int vbase;   // BCSR16 only: heads are vbase + v, twins are global arc ids
  int s, t;    // local ids; BFS only: t is the root, s the vertex never labelled (or -1)
  int mode;    // Mode
  int dir;     // BFS only: 0 vertices that reach the root, 1 reached from it
  // BCSR16 (row != nullptr)
  const int* row;
  int2* arc;
  const int2* arx;
  // RCSR
  const int* frow;
  int2* farc;
  int* fcb;
  const int* fcap;
  const int* rrow;
  const int2* rarc;
  int* lab;    // labels out
  int* e;      // excess out (state mode: in and out)
};

// Where the results go.
struct ResReport {
  ResOut* out;  // nullptr: the three words below instead (an instance of a batch)
  long long* flow;
  unsigned long long* ns;
  int* rounds;
};

struct ResRun {
  long long max_rounds;
  unsigned long long budget_ns;
  int bsub;   // BFS levels between two cluster barriers
  int grp;    // global relabel when the rounds since the last one took grp / 16 x its time
};

struct ResParams {
  ResInstance in;
  ResReport to;
  ResRun run;
  const int* gate;  // nullptr, or four words that must all be 0: otherwise the launch does nothing
  bool keep;     // write residuals, labels and excess back
  int4* rec;     // hybrid only: one record a residual arc (hybrid.cu)
};

// Instances of a batch, claimed one after the other by the blocks or clusters
// of one launch.
struct ResInst {
  int vbase, n, s, t;  // s and t are global vertex ids
};
struct ResBatch {
  const int* row;
  int2* arc;
  const int2* arx;
  const ResInst* inst;
  const int* order;  // this launch's instances, largest first
  int count;
  int* next;         // claim counter, zero at launch
  int* lab;
  int* e;
  long long* flows;
  unsigned long long* inst_ns;
  int* inst_rounds;
  ResRun run;
  int4* rec;             // hybrid only: `rec_stride` records a cluster
  long long rec_stride;
};

// The hybrid solver: the vertices in the shared memory of a 16-block cluster,
// the arcs as 16-byte records in global memory.
constexpr int kHybVertexBytes = 12;     // label, excess, expanded label
constexpr int kHybRowBytes = 8;         // the row, where there is room for it
constexpr int kHybListBytes = 32 * 512;  // 256 slots a warp
constexpr int kHybBlockVertices = (kResSmem - kResHeader - kHybListBytes) / kHybVertexBytes / 128 * 128;
constexpr int kHybMaxVertices = kResMaxCluster * kHybBlockVertices;

// Whether the hybrid solver should take a graph: n vertices, na residual arcs,
// `longer` of its rows longer than kLightDeg arcs.
// (Sparse graphs, whose many short rounds and levels are what a solve waits
// for: on R-MAT scale 13 one warp's walk of a long row makes it 1.0 ms against
// 0.47 resident, and a large power-law graph has a dozen rounds that need all
// SMs' bandwidth.)
inline bool hybrid_takes(long long n, long long na, long long longer) {
  return n <= kHybMaxVertices && na < 20 * n && longer <= 2 + n / 256;
}
// Above this many vertices and residual arcs a single solve stays with the
// persistent kernel, whose 152 SMs read the arcs faster.  Persistent and hybrid
// at 280,000 vertices, BCSR16 and RCSR: random graphs of 5.3M units 1.28, 1.14
// and 0.75, 1.20 ms, with many terminals of 4.9M 7.9, 7.5 and 8.7, 7.8; below,
// at 3.6M, 530x530 grids with all pixels terminals 10.7, 5.4 and 11.0, 5.8 ms,
// but a random graph (13 rounds, 3 relabels) 0.42, 0.66 and 0.54, 0.72.
constexpr long long kHybMaxUnits = 1 << 22;
cudaError_t launch_hybrid(const ResParams& p, cudaStream_t st);
// Clusters of `blocks` (a power of two) of the hybrid solver that run at once.
int hybrid_clusters(int blocks);
cudaError_t launch_hybrid_batch(const ResBatch& b, int blocks, int clusters, cudaStream_t st);

// The records' build and write-back are most of a hybrid solve of few rounds.
// Once a handle's solve (or its phase 2) has ended there within trial_rounds()
// and without deep searches, the next ones start on the persistent kernel, for so
// many rounds; one that has not ended by then goes over to the hybrid solver with
// the preflow it has, and so do all that follow.  (A trial in a handle's first
// solve too would take 0.44 ms of the 0.67 below, but 1.8 of 0.9 where 76 rounds
// follow.)  A round costs about 14 us more on the persistent kernel; what is saved
// is 0.03 to 0.07 ms per million vertices and residual arcs.  First and next call on
// a handle, persistent kernel alone and by this rule: random graphs of 3.6M units,
// 13 rounds 0.43, 0.42 and 0.67, 0.45 ms; of 2.5M, no way to t, RCSR 0.08, 0.08 and
// 0.20, 0.09; phase 2 of a 512x512 grid 0.32, 0.29 and 0.51, 0.32, of random graphs
// of 3.8M 0.22, 0.21 and 0.68, 0.23.
constexpr long long kHybTrialUnits = 1 << 18;
constexpr long long kHybTrialPhase2 = 1 << 20;  // below, the hybrid solver is never the slower one
inline long long trial_rounds(long long units) { return units >> 18; }

// Above this many vertices and residual arcs a graph that both could take goes
// to the hybrid solver: its vertices are dealt to the blocks one by one, the
// resident solver's in runs.  GENRMF 16x40 (107k units) 3.9 ms resident, 4.7
// hybrid; layered 32x256 (80k) 0.52, 0.49; layered 64x512 (324k) 2.03, 1.10.
constexpr long long kResPreferUnits = 1 << 17;

// The shared-memory solvers walk a row with one warp (resident) or 8 lanes
// (hybrid), the persistent kernel a long one with the whole grid: graphs that
// have a longer row than this, other than a terminal's, are the persistent
// kernel's.  Solves, persistent and shared-memory, one row of so many arcs:
// resident (s -> hub -> d rays -> t) 4,000 0.46, 0.31 ms, 7,000 0.50, 0.43,
// 10,000 0.44, 0.60, 20,000 0.47, 1.15; hybrid (random graphs of 164k to 692k
// units) 4,000 2.2, 1.2; 2.3, 1.4; 2.4, 1.3 ms, 8,000 2.0, 1.2; 2.7, 1.8; 2.6, 1.9,
// 16,000 1.3, 3.3; 2.1, 3.2; 1.5, 3.1; of 1.1M 4,000 1.3, 1.0, 8,000 0.7, 1.2;
// rays of 29,000 0.47, 6.8.  Batches of 8, general kernel and hybrid: 8,000 3.9,
// 2.4; 7.9, 4.8, 16,000 5.4, 6.4; 7.9, 5.8, rays of 10,000 2.8, 4.7.
constexpr int kResLongRow = 8192;
constexpr int kHybLongRow = 8192;
constexpr int kHybLongRowLarge = 4096;  // above kHybLargeUnits
constexpr long long kHybLargeUnits = 1 << 20;
// The same for phase 2 and a search alone (the hybrid's only where the last
// solve's searches had fewer than kHybShallowLevels levels: in deeper ones a row is
// one step of many).  Resident, 4,000 rays 0.14, 0.12 ms and 0.08, 0.08, 7,000 0.14,
// 0.15 and 0.08, 0.11; hybrid, random graphs 2,000 0.17, 0.16 and 0.21, 0.18, 4,000
// 0.18, 0.21 and 0.22, 0.23, 8,000 0.26, 0.47 and 0.32, 0.39, a 220x220 grid with a
// row of 2,400 0.41, 0.22 and 0.44, 0.22.
constexpr int kResLongSearch = 4096;
constexpr int kHybLongSearch = 2048;

// A search expands every arc of every vertex it reaches, the persistent kernel's
// stops at a row's first hit: on dense graphs of the cluster's size that kernel
// takes searches and phase 2.  Cut and phase 2, persistent and cluster: average
// degree 60 (366k units) 0.14, 0.27 and 0.12, 0.22 ms, 120 (363k) 0.13, 0.17 and
// 0.10, 0.25, 400 (401k) 0.10, 0.26 and 0.08, 0.19, 898 (405k) 0.08, 0.07 and 0.16,
// 0.27; 400 (201k) 0.07, 0.06 and 0.19, 0.12, 76 (R-MAT, 159k) 0.09, 0.06 and 0.33,
// 0.17; 30 (372k) 0.07, 0.07 and 0.27, 0.20.
constexpr double kResDenseDegree = 50;
constexpr long long kResDenseUnits = 1 << 18;
// A wide search of few levels needs all SMs' bandwidth: on graphs of the hybrid
// solver's size above so many units a search alone is the persistent kernel's where
// the last solve's searches had fewer levels than this.  Cut, persistent and
// hybrid: random graphs of 3.6M and 3.8M units (12 and 10 levels) 0.40, 0.63 and
// 0.36, 0.63 ms, of 2.6M (9) 0.17, 0.11; grids of 3.6M (34) 0.61, 0.39, (174) 1.5,
// 0.64; 3.5M (10, few vertices reached) 0.25, 0.16.
constexpr long long kHybShallowUnits = 3600000;
constexpr int kHybShallowLevels = 24;

// Lanes of a row in the resident solver: 8 below this average degree, 32 from it
// on.  Means of four seeds, 8 and 32 lanes: random graphs of 1,000 vertices, degree
// 8 0.081, 0.094 ms, 18 0.102, 0.111, 22 0.083, 0.089, 28 0.112, 0.107, 40 0.127,
// 0.113, 80 0.144, 0.113; of 3,000 8 0.166, 0.170, 18 0.136, 0.130, 28 0.178, 0.171,
// 80 0.291, 0.251; R-MAT scale 11 to 13 7 0.264, 0.296; 0.200, 0.175; 0.262, 0.229, 14
// 0.181, 0.161; 0.235, 0.223; 0.370, 0.323, 20 0.199, 0.188; 0.291, 0.269; 0.421,
// 0.396, 27 0.228, 0.206; 0.338, 0.310; 0.505, 0.473.  (Batches have one kernel, of 8
// lanes: most of their instances are sparse.)
constexpr int kResWideDegree = 20;

// Blocks for a graph of n vertices and na residual arcs: 1 where one block holds
// it, kResMaxCluster where the cluster should (a row too long for its block's
// share can still keep it out), or 0.
int resident_cluster(long long n, long long na);
cudaError_t launch_resident(const ResParams& p, int tile, int cluster, cudaStream_t st);
// Whether one block holds the graph (exact).
bool resident_one_block(long long n, long long na);
cudaError_t launch_resident_batch(const ResBatch& b, int blocks, cudaStream_t st);

}  // namespace wbpr_dev
