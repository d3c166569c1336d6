// qz_cg.cuh -- host interface of the on-chip node conjugate gradient
// (qz_cg_resident.cu), used by the level solves in qz_amr.cu.
#pragma once
#include "qz_internal.cuh"

namespace qz {

constexpr int CG_FILL = 148;         // chunks a level's CG points are cut into (B200's SMs)
constexpr int CGR_CHUNK_MAX = 1280;  // rows (of four points) a block keeps on chip
constexpr int CGR_CHUNK_MIN = 128;   // smallest chunk, in rows

// One launch of the on-chip solve: chunks [first, first + count) of the plan.
struct CgrRound {
    int first = 0, count = 0;
    int chunk = 0;       // rows of the largest chunk
    bool shared = false; // a node of several chunks: blocks that exchange values
    int cap = 0;         // most iterations of a node
    double points = 0.0; // interior points of its nodes
};

// Whether CG_FILL blocks of the solve are resident together on the simulation's device.
bool cgr_resident(const qz_sim *s);

// Cuts the nodes q with take[q] into chunks and rounds; node_chunk[2q], [2q + 1]
// become the node's chunk range inside its round.  cap[q]: iteration cap.
void cgr_plan(const AmrLevel &L, const std::vector<char> &take, const std::vector<int> &cap,
              long chunk_min, std::vector<AmrChunk> &chunks, std::vector<int> &node_chunk,
              std::vector<CgrRound> &rounds);

// Buffers of the exchange between the rounds' blocks; false where they cannot be had.
bool cgr_reserve(qz_sim *s, const AmrLevel &L, const std::vector<CgrRound> &rounds);

// Queues the rounds (chunks: the plan's on the device) after cgr_reserve.
struct CgrSolve {
    const AmrChunk *chunks;
    const int *node_chunk;
    int *status, *iters;
    double tol, tol2;
    int method;
    const double *thr_node;
    const int *cap_node;
};
int cgr_launch(qz_sim *s, AmrLevel &L, const std::vector<CgrRound> &rounds, const CgrSolve &v);

// Order of a level's interior points.  Brick layout of a level whose nodes' boxes are
// set (before the nodes go to the device); its zeroed masks, to be marked
// (brick_mark); the scan of their row counts (brick_base: first row of every
// brick, then the counts), from which the caller reads the nodes' row ranges; the
// rows themselves.  cg_order_list does all of it for a one-node level with a list.
// A level whose masks (cg_brick_masks is false) or rows find no room is left without an
// order (cg_ordered), and its nodes are solved with their vectors in memory.
void cg_brick_layout(AmrLevel &L);
bool cg_brick_masks(qz_sim *s, AmrLevel &L, unsigned long long **mask);
int cg_brick_scan(qz_sim *s, AmrLevel &L);
int cg_order(qz_sim *s, AmrLevel &L);
int cg_order_list(qz_sim *s, AmrLevel &L);

// Bits of a brick coordinate that the order holds; a level with a longer node (262,144
// points a side and more) gets no order.
constexpr int BRICK_BITS = 16;

#ifdef __CUDACC__
// Marks grid point (x, y, z) of node N in the level's 4^3-point bricks: brick
// coordinates x / 4, y / 4, z / 4 with their bits interleaved, axes that ran out
// of bits left out.
__device__ __forceinline__ void brick_mark(const AmrNode &N, int x, int y, int z,
                                           unsigned long long *mask)
{
    const unsigned c[3] = {(unsigned)x >> 2, (unsigned)y >> 2, (unsigned)z >> 2};
    unsigned m = 0;
    int sh = 0;
    for (int b = 0; b < BRICK_BITS; b++)
        for (int a = 0; a < 3; a++)
            if (b < N.bbits[a])
                m |= ((c[a] >> b) & 1u) << sh++;
    atomicOr(&mask[N.brick_off + (int)m], 1ULL << ((x & 3) | (y & 3) << 2 | (z & 3) << 4));
}
#endif

} // namespace qz
