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

struct ResParams {
  ResInstance in;
  ResOut* out;
  long long max_rounds;
  unsigned long long budget_ns;
  int smem_bytes;
  int bsub;   // BFS levels between two cluster barriers
  int grp;    // global relabel when the rounds since the last one took grp / 16 x its time
};

// Cluster size for a graph of n vertices and na residual arcs: the smallest
// power of two whose shared memory holds it, or 0.
int resident_cluster(long long n, long long na);
cudaError_t launch_resident(const ResParams& p, int tile, int cluster, cudaStream_t st);

}  // namespace wbpr_dev
