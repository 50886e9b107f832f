// Graph-analytics best-effort workloads of the reference: breadth-first search, single-source
// shortest paths, connected components and PageRank on a graph held whole in GPU memory
// (src/workloads/graphcompute.cu, the block-level-preemptible variant graphcompute.tr.cu; the task
// config config/Z.json runs them under a latency-critical DNN).  The graph comes from files in the
// EMOGI "bel" layout the reference reads (read_graph, graphcompute.cu:15-45): <prefix>.col holds the
// row offsets, <prefix>.dst the neighbour ids, <prefix>.val the edge weights of sssp.
//
// The reference drives each algorithm from the host: one or two kernels per iteration, then a copy
// of a `changed` byte and a stream synchronisation, until nothing changed.  Here one `execute` is a
// fixed kernel list - an initialisation kernel and one group of kernels per iteration - and
// convergence is tracked on the device: iteration i runs only if iteration i-1 raised its flag, the
// kernels of the iterations behind the last live one return at once.  The length of the list is
// found when the model is opened, by running the algorithm once.  For that to be exact the
// iterations are race-free: every kernel reads values only an earlier kernel wrote (the reference's
// kernels read distances and component ids other warps are lowering in the same launch, so its
// iteration count depends on timing; the fixed points are the same).  Connected components use
// hooking with shortcuts instead of the reference's plain label propagation, for the same fixed
// point in a handful of iterations.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <string>

#include "blp.cuh"

struct gpx_model;
struct gpx_model_opts;

namespace gpx {

enum GraphAlgo { GW_BFS = 0, GW_SSSP = 1, GW_CC = 2, GW_PAGERANK = 3 };
enum GraphPhase {
    GW_INIT = 0,    // start of a request: result arrays, frontier and iteration flags
    GW_EDGES = 1,   // walks the edge lists of a tile of vertices (a warp takes one list at a time)
    GW_VERTICES = 2 // per-vertex pass after the edge pass (sssp: update; cc: shortcut)
};

constexpr int kGwThreads = 256;
constexpr int kGwEdgeTileVertsMax = 256;  // vertices per tile of an edge pass at most (32 per warp)
constexpr int kGwVertexTileVerts = 1024;  // vertices per tile of a per-vertex pass
constexpr int kGwMaxIters = 16384;        // iteration flags a graph workload has: no run may need more rounds
// ids of a tile's window: started at a multiple of 32 and rounded up, with the zero behind it and the kernel's own
// variables, its copy fits the default 48 KiB
constexpr int kGwWindowMax = (48 * 1024 - 256) / 4 - 1;
static_assert((kGwWindowMax + 31 + 3 + 4) * 4 + 64 <= 48 * 1024, "window too long");
constexpr unsigned kGwInfinity = 0xFFFFFFFFu;  // MYINFINITY, include/workloads/graphcompute.h:14

struct GraphWlParams {
    int algo;
    int phase;
    int iter;             // iteration index; the BFS level
    int tile_verts;       // edge passes: vertices per tile, a multiple of 8 (one warp takes an eighth of them in turn)
    unsigned n;           // vertices
    unsigned src;         // bfs, sssp: source vertex (0, graphcompute.cu:181,344)
    const unsigned long long *row;  // [n + 1] edge offsets (pagerank: of the in-edge lists)
    const unsigned *adj;            // neighbour ids (pagerank: in-neighbours)
    const unsigned *wgt;            // sssp: edge weights
    const unsigned *outdeg;         // pagerank: out-degree of every vertex
    unsigned *a;          // bfs: label; sssp: cost; cc: comp; pagerank: value (float)
    unsigned *b;          // sssp: new cost; cc: offered ids; pagerank: residual (float)
    unsigned *d0, *d1;    // pagerank: delta, read from d<iter & 1>, written to the other
    unsigned char *f0;    // sssp: label (the frontier)
    int *active;          // [kGwMaxIters + 1]: active[i] != 0 <=> iteration i has work
    // pagerank, for graphs ordered for locality (pack_lists): the ids as 16-bit byte offsets into the copy of the
    // window of deltas the tile can reach, at most kGwWindowMax ids long, in blocks of 32 x pack (a lane's
    // ids of a block next to one another, in the order deal_edges gives them), padded with the offset
    // behind the window, where the shared-memory copy holds a zero.
    int many;                       // bfs: with more tiles than CTAs of the form of more registers are resident: their number
    int pack;                       // ids a lane holds per block: 1, 2, 4 or 8; 0 = lists in adj
    const uint16_t *packed;
    const unsigned *blk;            // [n + 1] first block of every vertex
    const uint2 *win;               // [tiles] first id (a multiple of 32) and deltas to copy (of four)
    int win_max;                    // longest copy
    float alpha, tol;     // pagerank (0.85, 0.001: include/workloads/graphcompute.h:85-86)
};

cudaError_t graphwl_launch(const GraphWlParams &p, int grid, const BlpArgs &blp, cudaStream_t s);
int graphwl_plan(GraphWlParams &p, int total_tiles, int sm_count);  // fills many and returns the grid

// "bfs:<prefix>", "sssp:<prefix>", "cc:<prefix>", "pagerank:<prefix>".
bool is_graph_workload(const std::string &name);
int build_graph_workload(gpx_model &m, const std::string &name, const gpx_model_opts &opts);

}  // namespace gpx
