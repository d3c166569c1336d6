// qz_cg_resident.cu -- the refinement nodes' conjugate gradient with its vectors
// on chip (cg_variant 0 where a node fits).
//
// The node CG (conjugate_gradient.c:322-463) on a refinement node is a few
// hundred iterations over 10^4 to 10^6 points: the data fit in the SMs'
// registers and shared memory, and what bounds an iteration is the chain of
// dependent trips through L2 (sums to every block and back, neighbours' values).
// So here a block of 512 threads keeps its points' r, s, p, A r and pot on chip
// for the whole solve, and an iteration makes one trip:
//
//   * Chronopoulos and Gear's arrangement (1989) of the same iterates: with w = A r
//     and s = A p, both dot products of an iteration (gamma = r.r, delta = w.r)
//     are known together,
//       beta_j  = gamma_j / gamma_{j-1}                      (beta_0 = 0)
//       alpha_j = gamma_j / (delta_j - beta_j gamma_j / alpha_{j-1})
//       s = w + beta s;  p = r + beta p;  pot += alpha p;  r -= alpha s;  w = A r
//   * a block keeps r and s of its ghosts (the points of other blocks next to its
//     own) and advances them with the same expressions, so only w crosses
//     between blocks, published together with the partial sums;
//   * every published double travels as two 64-bit words of 32 data bits and the
//     iteration's 32-bit tag, so a reader knows a value from a stale one by
//     itself: no fence, no flag, no second trip.  A block's two sums are one
//     32-byte store into a line of its own that every block of the node polls.
// Buffers are double by iteration parity: a block writes the words of iteration
// j + 2 only after it has seen every block's sums of j + 1, which each block
// publishes after it has read the words of j.
//
// Points are held in rows of four consecutive x (aligned in the node's grid, holes
// zero), one or two rows a thread: the y and z neighbours of a row are rows, read
// with 16-byte loads, and the x neighbours but two are the row's own registers, so a
// point costs 2.5 shared-memory loads and a sixth of the index arithmetic of six
// single neighbours.  Rows are ordered along a Morton curve of 4^3-point bricks and
// chunks are runs of that order, so that a chunk is compact.
//
// Measured on B200 (conjugate-gradient time): a cube of 43^3 points 2.2 us an iteration,
// 67^3 4.1, 81^3 6.2; the three levels of a 1M-particle sphere (81k, 160k and 301k points,
// 750 iterations) 2.5 ms a step where the kernel with its vectors in memory takes 6.06,
// four levels of two nodes of up to 595k points 15.2 ms where it takes 35.5.  An
// iteration is the sums' trip (0.87 us for 148 blocks with nothing else to do), the ghosts'
// (0.4 us) and the chain of the block's own work; what did not help: pushing sums into
// per-reader inboxes (1.25 us a trip), polling for the ghosts' words before the sums have
// come (the polls hold up the words), one warp waiting for all sums, Ghysels and
// Vanroose's arrangement (3.65 ms: its ghosts' words are waited for at once), one point
// a thread with six index loads (2.5 ms, and 15.3), and every variant with a few spilled
// registers (the blocks' shared memory leaves little L1 for them).
#include <algorithm>
#include <limits.h>
#include <stdio.h>
#include <string.h>

#include "qz_amr_dev.cuh"
#include "qz_cg.cuh"

namespace qz {

#define QZ_PI_D 3.14159265358979323846

typedef unsigned long long u64;

// ---- order of a level's interior points ---------------------------------------------
// Marks a one-node list; *face: it holds a point on the grid's faces, whose neighbours
// by index are not its neighbours in space.
__global__ void k_brick_mark(int n, const int *__restrict__ intr, const AmrNode *__restrict__ nodes,
                             u64 *__restrict__ mask, int *__restrict__ face)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    const AmrNode N = nodes[0];
    int x, y, z;
    grid_coords(N, intr[t], &x, &y, &z);
    if (x == 0 || y == 0 || z == 0 || x >= N.rd[0] || y >= N.rd[1] || z >= N.rd[2])
    {
        *face = 1;
        return;
    }
    brick_mark(N, x, y, z, mask);
}

// One bit a row of the brick (bit 4 q: row q = y + 4 z of the brick holds a point).
__device__ __forceinline__ u64 brick_rows(u64 m)
{
    m |= m >> 1;
    m |= m >> 2;
    return m & 0x1111111111111111ULL;
}

__global__ void k_brick_count(int n, const u64 *__restrict__ mask, int *__restrict__ cnt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n)
        cnt[t] = __popcll(brick_rows(mask[t]));
}

// One thread a row of a brick: the row's place is its brick's first place plus its
// rank in the brick.
__global__ void k_brick_order(long n, int nn, const AmrNode *__restrict__ nodes,
                              const u64 *__restrict__ mask, const int *__restrict__ base,
                              int2 *__restrict__ row, int *__restrict__ pos)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    const int b = (int)(t >> 4), q = (int)(t & 15);
    const u64 m = mask[b];
    const int lanes = (int)((m >> (4 * q)) & 15);
    if (!lanes)
        return;
    int lo = 0, hi = nn - 1; // last node whose bricks start at or before b
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (nodes[mid].brick_off <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    const AmrNode N = nodes[lo];
    int c[3] = {0, 0, 0}, rest = b - N.brick_off;
    for (int i = 0; i < BRICK_BITS; i++)
        for (int a = 0; a < 3; a++)
            if (i < N.bbits[a])
            {
                c[a] |= (rest & 1) << i;
                rest >>= 1;
            }
    const int g = (int)grid_index(N, 4 * c[0], 4 * c[1] + (q & 3), 4 * c[2] + (q >> 2));
    const int at = base[b] + __popcll(brick_rows(m) & ((1ULL << (4 * q)) - 1));
    row[at] = make_int2(g, lanes);
    pos[g] = at;
}

void cg_brick_layout(AmrLevel &L)
{
    long total = 0;
    bool wide = false;
    for (AmrNode &N : L.h)
    {
        int bits = 0;
        for (int a = 0; a < 3; a++)
        {
            N.bbits[a] = 0;
            while ((4L << N.bbits[a]) < N.rd[a] + 1)
                N.bbits[a]++;
            wide = wide || N.bbits[a] > BRICK_BITS;
            bits += N.bbits[a];
        }
        N.brick_off = (int)total;
        total += 1L << bits;
    }
    L.brick_total = wide ? LONG_MAX : total;
    L.cg_ordered = false;
}

// Room for `need` elements and what the tree grows by in a few steps.
static long cgr_room(long need) { return need + need / 4 + 64; }

constexpr long BRICKS_MAX = 1L << 27; // 1 GB of masks

bool cg_brick_masks(qz_sim *s, AmrLevel &L, u64 **mask)
{
    const long nb = L.brick_total;
    if (nb > (s->cgr_bricks > 0 ? s->cgr_bricks : BRICKS_MAX) || !s->brick_mask.ensure(s->mem, nb) ||
        !s->brick_base.ensure(s->mem, 2 * nb + 1))
    {
        cudaGetLastError();
        return false;
    }
    cudaMemsetAsync(s->brick_mask.p, 0, nb * sizeof(u64), s->stream);
    *mask = s->brick_mask.p;
    return true;
}

int cg_brick_scan(qz_sim *s, AmrLevel &L)
{
    const int nb = (int)L.brick_total;
    int *cnt = s->brick_base.p + nb;
    launch(s, QZ_PROF_TREE, 12.0 * nb, k_brick_count, dim3(blocks_for(nb, 256)), dim3(256), nb,
           s->brick_mask.p, cnt);
    return scan_exclusive(s, cnt, s->brick_base.p, nb);
}

int cg_order(qz_sim *s, AmrLevel &L)
{
    if (!L.row.ensure(s->mem, cgr_room(L.row_total)) || !L.pos.ensure(s->mem, cgr_room(L.grid_total)))
    {
        cudaGetLastError();
        return QZ_SUCCESS;
    }
    cudaMemsetAsync(L.pos.p, 0xff, L.grid_total * sizeof(int), s->stream);
    const long n = 16 * L.brick_total;
    launch(s, QZ_PROF_TREE, 1.0 * n + 28.0 * L.row_total, k_brick_order, dim3(blocks_for(n, 256)),
           dim3(256), n, L.nnodes, L.nodes.p, s->brick_mask.p, s->brick_base.p, L.row.p, L.pos.p);
    L.cg_ordered = true;
    return check_cuda(cudaGetLastError(), "conjugate gradient order") ? QZ_SUCCESS : QZ_FAILURE;
}

// A one-node level given by its interior list (the head, a host node); left without an
// order, too, when the list has points on the grid's faces.
int cg_order_list(qz_sim *s, AmrLevel &L)
{
    u64 *mask;
    L.cg_ordered = false;
    if (!cg_brick_masks(s, L, &mask))
        return QZ_SUCCESS;
    const int nb = (int)L.brick_total;
    int *face = s->brick_base.p + 2L * nb;
    cudaMemsetAsync(face, 0, sizeof(int), s->stream);
    launch(s, QZ_PROF_TREE, 12.0 * L.intr_total, k_brick_mark, dim3(blocks_for(L.intr_total, 256)),
           dim3(256), L.intr_total, L.intr.p, L.nodes.p, mask, face);
    if (cg_brick_scan(s, L))
        return QZ_FAILURE;
    int last[3]; // first row of the last brick, its rows, points on the faces
    if (!check_cuda(cudaMemcpyAsync(&last[0], s->brick_base.p + nb - 1, sizeof(int),
                                    cudaMemcpyDeviceToHost, s->stream), "rows") ||
        !check_cuda(cudaMemcpyAsync(&last[1], face - 1, 2 * sizeof(int), cudaMemcpyDeviceToHost,
                                    s->stream), "rows") ||
        !check_cuda(cudaStreamSynchronize(s->stream), "rows"))
        return QZ_FAILURE;
    L.h[0].row_off = 0;
    L.h[0].nrows = L.row_total = last[0] + last[1];
    return last[2] ? QZ_SUCCESS : cg_order(s, L);
}

// ---- the solve --------------------------------------------------------------------------
constexpr int CGR_POLLERS = (CG_FILL + 31) / 32; // warps that poll the blocks' sums
constexpr int CGR_LINE = 16; // words of an L2 line
constexpr int CGR_POLL_LIMIT = 1 << 21;
constexpr int CGR_SMEM = 224 * 1024;
// Ghost half rows a row can ask for: both of its y and z neighbour rows and one of each
// x neighbour.
constexpr int CGR_ROW_GHOSTS = 10;

__device__ __forceinline__ double cgr_value(u64 a, u64 b)
{
    return __longlong_as_double((long long)((a & 0xffffffffULL) | (b << 32)));
}

__device__ __forceinline__ bool cgr_ready(u64 a, u64 b, unsigned tag)
{
    return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// Two doubles (a half row's w, a block's sums) in one 32-byte word group.
__device__ __forceinline__ void cgr_store2(u64 *p, double v, double w, unsigned tag)
{
    const u64 a = (u64)__double_as_longlong(v), b = (u64)__double_as_longlong(w), t = (u64)tag << 32;
    asm volatile("st.relaxed.gpu.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p),
                 "l"((a & 0xffffffffULL) | t), "l"((a >> 32) | t), "l"((b & 0xffffffffULL) | t),
                 "l"((b >> 32) | t)
                 : "memory");
}

__device__ __forceinline__ void cgr_load2(const u64 *p, u64 (&w)[4])
{
    asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(p)
                 : "memory");
}

// Waits for the word group at p (w: its last load); false, and zeros, when it never came.
__device__ __forceinline__ bool cgr_wait2(const u64 *p, u64 (&w)[4], unsigned tag)
{
    int polls = 0;
    while (!cgr_ready(w[0], w[1], tag) || !cgr_ready(w[2], w[3], tag))
    {
        if (++polls > CGR_POLL_LIMIT)
        {
            w[0] = w[1] = w[2] = w[3] = 0;
            return false;
        }
        cgr_load2(p, w);
    }
    return true;
}

// Waits for a block's sums at p, whose top bit carries its failed test; false when they
// never came.
__device__ __forceinline__ bool cgr_wait_sums(const u64 *p, u64 (&w)[4], unsigned tag)
{
    constexpr u64 FB = 1ULL << 63;
    int polls = 0;
    for (;;)
    {
        cgr_load2(p, w);
        if (cgr_ready(w[0] & ~FB, w[1] & ~FB, tag) && cgr_ready(w[2] & ~FB, w[3] & ~FB, tag))
            return true;
        if (++polls > CGR_POLL_LIMIT)
            return false;
    }
}

// Both waits of the solve on words that nothing publishes (they end at their poll limit).
__global__ void k_cgr_wait_probe(const u64 *words, int *out)
{
    u64 w[4];
    cgr_load2(words, w);
    out[0] = cgr_wait2(words, w, 5u) ? 1 : 0;
    out[1] = cgr_wait_sums(words + CGR_LINE, w, 5u) ? 1 : 0;
}

struct CgrArgs {
    const AmrChunk *chunks; // of this launch; begin, end are rows
    int nchunks;
    const int2 *row; // grid index of a row's first point, lanes that hold a point
    const int *pos;  // row that starts at a grid point, or -1
    const AmrNode *nodes;
    const int *node_chunk; // per node: first chunk, end chunk (of this launch)
    const double *d;
    double *pot, *pot_old;
    u64 *halo[2]; // two words a point of a row
    u64 *sums[2]; // four words a chunk of a shared round, CGR_LINE apart
    int *status;  // [0] most iterations of a node, [1] a wait gave up, [2] unconverged nodes
    int *iters;
    double tol, tol2, G;
    int every, max_iter, method;
    const double *thr_node;
    const int *cap_node;
    unsigned tag0;
    int chunk; // rows of the largest chunk
    int gcap;  // ghost rows kept in shared memory; the others in spill
    // scratch of a chunk of a shared round (the others have no ghosts): per ghost row
    // (6 chunk) its row and the lanes asked for; past the first GV a thread the ghost half
    // rows' (10 chunk) words, places and s; r of the ghost rows past gcap
    int2 *grow, *xplace;
    double2 *xs, *spill;
};

// Shared memory of a block, in this order: rows of r (row 0 zero, own, ghosts; lanes
// 0 and 1 of all rows, then lanes 2 and 3, so that 16-byte loads of consecutive rows
// do not conflict), pot at the last failed check of own rows (one row a thread; with two
// it stays in memory and p and pot are here), s and the list of the ghost half rows.
// GV: ghost half rows of a thread with their words in flight together.
template <int NT, int RT, int GV> constexpr long cgr_fixed_bytes()
{
    const long own = (long)RT * NT;
    return 32 * (1 + own) + (RT > 1 ? 64 * own : 32 * own) + 24L * GV * NT;
}
constexpr int CGR_GHOST_BYTES = 32;

// NT threads of RT rows, one block a SM.  With one row everything a thread owns is in
// registers.  Rows past the chunk's end are zeros with zero neighbours, so that the
// loops have no branches and their loads overlap.
template <int NT, int RT, int GV>
__global__ void __launch_bounds__(NT, 1) k_cg_resident(const __grid_constant__ CgrArgs A)
{
    constexpr int CGR_THREADS = NT, CGR_WARPS = NT / 32;
    constexpr bool REG = RT == 1;
    constexpr bool GREG = REG && NT <= 512; // the ghosts' state in registers too
    constexpr int OWN = RT * CGR_THREADS;
    extern __shared__ __align__(16) double2 cgr_dyn[];
    __shared__ double sh_w[2 * CGR_WARPS];
    __shared__ double2 sh_s[CGR_POLLERS];
    __shared__ int sh_f[CGR_WARPS], sh_fs[CGR_POLLERS];
    __shared__ int sh_ng, sh_nv;
    // a wait gave up: for the sums; for a ghost (joins the former before the sums' barrier)
    __shared__ int sh_lost, sh_late;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrow = 1 + OWN + A.gcap;
    double2 *R0 = cgr_dyn, *R1 = R0 + nrow;
    double2 *KP = R1 + nrow;                      // REG: pot at the last failed check
    double2 *KX = KP + 2 * OWN;                   // not REG: p in KP, pot in KX
    double2 *GS = KP + (REG ? 2 : 4) * OWN; // ghost half rows' s
    int2 *EL = reinterpret_cast<int2 *>(GS + GV * NT);
    bool bad = false;
    // chunks past the grid's end are those of nodes of one chunk: no block waits for another
    for (int c = blockIdx.x; c < A.nchunks; c += gridDim.x)
    {
        const AmrChunk C = A.chunks[c];
        const AmrNode N = A.nodes[C.node];
        const int cb = A.node_chunk[2 * C.node], m = A.node_chunk[2 * C.node + 1] - cb;
        const int n = C.end - C.begin;
        const int sy = N.rd[0] + 1, sz = sy * (N.rd[1] + 1);
        const double H = 1.0 / (1 << N.lv), oh2 = 1.0 / (H * H);
        const double rm = 4.0 * A.G * QZ_PI_D * N.mass / (N.ncells * H * H * H);
        double thr = N.nintr * (A.tol * rm) * (A.tol * rm);
        if (A.method == 2)
            thr = thr * (cbrt((double)N.nintr) * cbrt((double)N.nintr));
        if (A.thr_node)
            thr = A.thr_node[C.node];
        const long size = (long)sz * (N.rd[2] + 1);
        int cap = (int)(size < A.max_iter ? size : A.max_iter);
        if (A.cap_node)
        {
            cap = A.cap_node[C.node];
            thr = -1.0; // r.r < -1 never holds: the node runs exactly cap iterations
        }
        int2 *grow = A.grow + 6L * A.chunk * c;
        int2 *xplace = A.xplace + (long)CGR_ROW_GHOSTS * A.chunk * c;
        double2 *xs = A.xs + (long)CGR_ROW_GHOSTS * A.chunk * c;
        double2 *spill = A.spill + 2L * c * (6L * A.chunk > A.gcap ? 6L * A.chunk - A.gcap : 0);
        // ---- neighbours of every own row: rows of R, 16 bits each (y+, y-, z+, z-, x-, x+)
        unsigned nbr[RT][3];
        unsigned lanes[RT]; // lanes that hold a point; from bit 4: those another block reads
        int2 *hash = reinterpret_cast<int2 *>(R0 + 1 + OWN); // (row, ghost); in the ghosts' place
        __syncthreads();
        for (int t = tid; t < A.gcap; t += CGR_THREADS)
            hash[t] = make_int2(-1, 0);
        if (tid == 0)
        {
            sh_ng = sh_nv = sh_lost = sh_late = 0;
            R0[0] = R1[0] = make_double2(0.0, 0.0);
        }
        __syncthreads();
        constexpr unsigned PENDING = 0xffffu;
        constexpr int PROBES = 32;
        auto hash_of = [&](int q) { return (int)__umulhi((unsigned)q * 2654435761u, (unsigned)A.gcap); };
        // neighbour row v of row (g, own lanes) and the lanes of it that the row reads
        auto neighbour = [&](int g, unsigned own, int v, unsigned *need) {
            *need = 0;
            if (own == 0 || (v == 4 && !(own & 1)) || (v == 5 && !(own & 8)))
                return -1;
            const int off[6] = {sy, -sy, sz, -sz, -4, 4};
            const int q = A.pos[g + off[v]];
            if (q < 0)
                return -1;
            const unsigned there = (unsigned)A.row[q].y;
            *need = v == 4 ? there & 8u : v == 5 ? there & 1u : there & own;
            return *need ? q : -1;
        };
#pragma unroll
        for (int u = 0; u < RT; u++)
        {
            const int e = tid + u * CGR_THREADS;
            const int2 me = e < n ? A.row[C.begin + e] : make_int2(0, 0);
            unsigned pk[3] = {0, 0, 0}, pub = 0;
            for (int v = 0; v < 6; v++)
            {
                unsigned need;
                const int q = neighbour(me.x, (unsigned)me.y, v, &need);
                unsigned id = 0;
                bool fresh = false, direct = false;
                int at = 0;
                if (q >= C.begin && q < C.end)
                    id = 1 + q - C.begin;
                else if (q >= 0)
                {
                    pub |= v == 4 ? 1u : v == 5 ? 8u : need;
                    id = PENDING;
                    direct = true; // unless the table takes it
                    at = hash_of(q);
                    for (int t = 0; t < PROBES; t++)
                    {
                        const int k = atomicCAS(&hash[at].x, -1, q);
                        if (k == -1)
                            fresh = true;
                        if (k == -1 || k == q)
                        {
                            direct = false;
                            break;
                        }
                        at = at + 1 < A.gcap ? at + 1 : 0;
                    }
                }
                const unsigned fm = __ballot_sync(0xffffffffu, fresh || direct);
                if (fm)
                {
                    int base = 0;
                    if (lane == 0)
                        base = atomicAdd(&sh_ng, __popc(fm));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (fresh || direct)
                    {
                        const int h = base + __popc(fm & ((1u << lane) - 1));
                        grow[h] = make_int2(q, fresh ? 0 : (int)need);
                        if (fresh)
                            hash[at].y = h;
                        else
                            id = 1 + OWN + h;
                    }
                }
                pk[v >> 1] |= id << (v & 1 ? 16 : 0);
            }
#pragma unroll
            for (int v = 0; v < 3; v++)
                nbr[u][v] = pk[v];
            lanes[u] = (unsigned)me.y | pub << 4;
        }
        __syncthreads();
        const int ng = sh_ng;
#pragma unroll
        for (int u = 0; u < RT; u++)
        {
            if (!(lanes[u] >> 4))
                continue;
            const int2 me = A.row[C.begin + tid + u * CGR_THREADS];
#pragma unroll
            for (int v = 0; v < 6; v++)
            {
                const unsigned sh = v & 1 ? 16 : 0;
                if (((nbr[u][v >> 1] >> sh) & 0xffffu) != PENDING)
                    continue;
                unsigned need;
                const int q = neighbour(me.x, (unsigned)me.y, v, &need);
                int at = hash_of(q);
                while (hash[at].x != q) // it is there: this thread saw it go in
                    at = at + 1 < A.gcap ? at + 1 : 0;
                const int h = hash[at].y;
                atomicOr(&grow[h].y, (int)need);
                nbr[u][v >> 1] = (nbr[u][v >> 1] & ~(0xffffu << sh)) | (unsigned)(1 + OWN + h) << sh;
            }
        }
        __syncthreads(); // the table's memory becomes ghost rows
        const bool spilled = ng > A.gcap; // the same in the whole block
        // ---- start: r = d + (1/H^2) L pot at own points and ghosts
        auto residual = [&](int g) {
            const double *pt = A.pot;
            return A.d[g] + oh2 * (6.0 * pt[g] - pt[g + 1] - pt[g - 1] - pt[g + sy] - pt[g - sy] -
                                   pt[g + sz] - pt[g - sz]);
        };
        double r[RT][4], w[RT][4], sv[RT][4], p[REG ? RT : 1][4], x[REG ? RT : 1][4];
#pragma unroll
        for (int u = 0; u < RT; u++)
        {
            const int e = tid + u * CGR_THREADS;
            const int g = e < n ? A.row[C.begin + e].x : 0;
            double xv[4], old[4];
#pragma unroll
            for (int l = 0; l < 4; l++)
            {
                r[u][l] = w[u][l] = sv[u][l] = 0.0;
                xv[l] = old[l] = 1.0;
                if ((lanes[u] >> l) & 1)
                {
                    r[u][l] = residual(g + l);
                    xv[l] = A.pot[g + l];
                    old[l] = A.pot_old[g + l];
                }
                if constexpr (REG)
                {
                    p[u][l] = 0.0;
                    x[u][l] = xv[l];
                }
            }
            R0[1 + e] = make_double2(r[u][0], r[u][1]);
            R1[1 + e] = make_double2(r[u][2], r[u][3]);
            if constexpr (REG)
            {
                KP[e] = make_double2(old[0], old[1]);
                KP[OWN + e] = make_double2(old[2], old[3]);
            }
            else
            {
                KP[e] = KP[OWN + e] = make_double2(0.0, 0.0);
                KX[e] = make_double2(xv[0], xv[1]);
                KX[OWN + e] = make_double2(xv[2], xv[3]);
            }
        }
        // place of half hf of a ghost row: index from R0 (negative: in spill)
        auto place_of = [&](int h, int hf) {
            return h < A.gcap ? hf * nrow + 1 + OWN + h : -1 - (2 * (h - A.gcap) + hf);
        };
        // the list of ghost half rows: their words and places; those of a warp's ghosts stay
        // together, so that their loads share lines
        for (int h0 = warp * 32; h0 < ng; h0 += CGR_THREADS)
        {
            const int h = h0 + lane;
            const int2 gr = h < ng ? grow[h] : make_int2(0, 0);
            int at = ((gr.y & 3) != 0) + ((gr.y & 12) != 0);
            int sum = at;
            for (int o = 1; o < 32; o <<= 1)
            {
                const int t = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o)
                    sum += t;
            }
            int base = 0;
            if (lane == 31)
                base = atomicAdd(&sh_nv, sum);
            at = __shfl_sync(0xffffffffu, base, 31) + sum - at;
            const int2 row = h < ng ? A.row[gr.x] : make_int2(0, 0);
            for (int hf = 0; hf < 2 && h < ng; hf++)
            {
                const int pl = place_of(h, hf);
                double2 v = make_double2(0.0, 0.0);
                if ((gr.y >> (2 * hf)) & 3)
                {
                    if ((row.y >> (2 * hf)) & 1)
                        v.x = residual(row.x + 2 * hf);
                    if ((row.y >> (2 * hf)) & 2)
                        v.y = residual(row.x + 2 * hf + 1);
                    const int2 en = make_int2(4 * (2 * gr.x + hf), pl);
                    if (at < GV * NT)
                    {
                        EL[at] = en;
                        GS[at] = make_double2(0.0, 0.0);
                    }
                    else
                    {
                        xplace[at] = en;
                        xs[at] = make_double2(0.0, 0.0);
                    }
                    at++;
                }
                (pl >= 0 ? R0[pl] : spill[-1 - pl]) = v;
            }
        }
        __syncthreads();
        const int nv = sh_nv;
        // GREG: words, places and s of this thread's ghost half rows
        int2 gl[GREG ? GV : 1];
        double2 gs[GREG ? GV : 1];
        if constexpr (GREG)
        {
#pragma unroll
            for (int v = 0; v < GV; v++)
            {
                gl[v] = tid + v * NT < nv ? EL[tid + v * NT] : make_int2(0, 0);
                gs[v] = make_double2(0.0, 0.0);
            }
        }
        // w = A r at the own points, then the block's sums of r.r and w.r to every block of
        // the node and w where another block needs it, for iteration j; fail rides on the
        // tags' top bit.  The sums go first: they are waited for first.
        auto stencil = [&](int j, int fail) {
            const unsigned tag = A.tag0 + (unsigned)j;
            double pg = 0.0, pd = 0.0;
            auto rows = [&](auto row0, auto row1) {
#pragma unroll
                for (int u = 0; u < RT; u++)
                {
                    double t[4] = {6.0 * r[u][0] - r[u][1], 6.0 * r[u][1] - r[u][2],
                                   6.0 * r[u][2] - r[u][3], 6.0 * r[u][3] - r[u][2]};
                    t[0] -= row1((int)(nbr[u][2] & 0xffffu)).y;
                    t[1] -= r[u][0];
                    t[2] -= r[u][1];
                    t[3] -= row0((int)(nbr[u][2] >> 16)).x;
#pragma unroll
                    for (int v = 0; v < 4; v++)
                    {
                        const int id = v & 1 ? nbr[u][v >> 1] >> 16 : nbr[u][v >> 1] & 0xffffu;
                        const double2 a = row0(id), b = row1(id);
                        t[0] -= a.x;
                        t[1] -= a.y;
                        t[2] -= b.x;
                        t[3] -= b.y;
                    }
#pragma unroll
                    for (int l = 0; l < 4; l++)
                    {
                        w[u][l] = (lanes[u] >> l) & 1 ? -oh2 * t[l] : 0.0;
                        pg = fma(r[u][l], r[u][l], pg);
                        pd = fma(w[u][l], r[u][l], pd);
                    }
                }
            };
            if (!spilled)
                rows([&](int id) { return R0[id]; }, [&](int id) { return R1[id]; });
            else
            {
                const double2 *S = spill;
                rows([&](int id) { return id < nrow ? R0[id] : S[2 * (id - nrow)]; },
                     [&](int id) { return id < nrow ? R1[id] : S[2 * (id - nrow) + 1]; });
            }
            // lanes 0-15 add the r.r, lanes 16-31 the w.r
            const bool up = lane >= 16;
            double t = (up ? pd : pg) + __shfl_xor_sync(0xffffffffu, up ? pg : pd, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
                t += __shfl_xor_sync(0xffffffffu, t, o);
            fail = __any_sync(0xffffffffu, fail);
            if ((lane & 15) == 0)
            {
                sh_w[warp + (lane >> 4) * CGR_WARPS] = t;
                sh_f[warp] = fail;
            }
            // warp 0 adds the warps' sums and publishes them
            if (warp != 0)
                asm volatile("bar.arrive 1, %0;" ::"n"(CGR_THREADS) : "memory");
            else
            {
                asm volatile("bar.sync 1, %0;" ::"n"(CGR_THREADS) : "memory");
                const int k = lane & 15;
                const double *mine = sh_w + (lane >> 4) * CGR_WARPS;
                t = k < CGR_WARPS ? mine[k] : 0.0;
                fail = k < CGR_WARPS ? sh_f[k] : 0;
                for (int q = k + 16; q < CGR_WARPS; q += 16)
                {
                    t += mine[q];
                    fail |= sh_f[q];
                }
                fail = __any_sync(0xffffffffu, fail);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    t += __shfl_xor_sync(0xffffffffu, t, o);
                const double td = __shfl_sync(0xffffffffu, t, 16);
                if (lane == 0)
                {
                    if (m == 1)
                    {
                        sh_s[0] = make_double2(t, td);
                        sh_fs[0] = fail;
                    }
                    else
                        cgr_store2(A.sums[j & 1] + (long)c * CGR_LINE, t, td,
                                   tag | (fail ? 0x80000000u : 0u));
                }
            }
            u64 *halo = A.halo[j & 1] + 8L * (C.begin + tid);
#pragma unroll
            for (int u = 0; u < RT; u++)
#pragma unroll
                for (int hf = 0; hf < 2; hf++)
                    if ((lanes[u] >> (4 + 2 * hf)) & 3)
                        cgr_store2(halo + 8 * u * CGR_THREADS + 4 * hf, w[u][2 * hf], w[u][2 * hf + 1],
                                   tag);
        };
        stencil(0, 0);
        double inv_g = 0.0, inv_ga = 0.0; // 1 / gamma_{j-1}, 1 / (gamma_{j-1} alpha_{j-1})
        int j = 0, until = A.every;       // updates until the next check
        bool converged = false;
        for (;; j++)
        {
            const unsigned tag = A.tag0 + (unsigned)j;
            const u64 *halo = A.halo[j & 1];
            // ---- the sums of iteration j
            const int pw = warp - 1; // warps 1, 2, .. poll 32 lines each
            if (m > 1 && pw >= 0 && pw * 32 < m)
            {
                double a = 0.0, b = 0.0;
                int f = 0;
                if (pw == 0 && lane == 0 && sh_late)
                    sh_lost = 1;
                if (pw * 32 + lane < m)
                {
                    const u64 *in = A.sums[j & 1] + (long)(cb + pw * 32 + lane) * CGR_LINE;
                    u64 q[4];
                    if (!cgr_wait_sums(in, q, tag))
                        sh_lost = 1;
                    a = cgr_value(q[0], q[1]);
                    b = cgr_value(q[2], q[3]);
                    f = (int)(q[0] >> 63);
                }
                const bool up = lane >= 16;
                double t = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    t += __shfl_xor_sync(0xffffffffu, t, o);
                f = __any_sync(0xffffffffu, f);
                if ((lane & 15) == 0)
                {
                    reinterpret_cast<double *>(sh_s)[2 * pw + (lane >> 4)] = t;
                    sh_fs[pw] = f;
                }
            }
            __syncthreads();
            // the ghosts' w, written just after the sums and loaded after them: polling for
            // them earlier only fills the L2 with loads that hold up the words
            u64 gw[GV][4];
#pragma unroll
            for (int v = 0; v < GV; v++)
                if (tid + v * NT < nv)
                    cgr_load2(halo + (GREG ? gl[GREG ? v : 0] : EL[tid + v * NT]).x, gw[v]);
            double gamma = sh_s[0].x, delta = sh_s[0].y;
            int f = sh_fs[0];
            for (int q = 1; q * 32 < m; q++)
            {
                gamma += sh_s[q].x;
                delta += sh_s[q].y;
                f |= sh_fs[q];
            }
            bad = sh_lost != 0;
            if (bad)
                break;
            // ---- the reference's test after update j, and its cap
            if (until == 0)
            {
                if (!f && (A.method == 1 || gamma < thr))
                {
                    converged = true;
                    break;
                }
#pragma unroll
                for (int u = 0; u < RT; u++)
                {
                    const int e = tid + u * CGR_THREADS;
                    if constexpr (REG)
                    {
                        KP[e] = make_double2(x[u][0], x[u][1]);
                        KP[OWN + e] = make_double2(x[u][2], x[u][3]);
                    }
                    else if (lanes[u] & 15)
                    {
                        const double2 a = KX[e], b = KX[OWN + e];
                        const double xv[4] = {a.x, a.y, b.x, b.y};
                        double *po = A.pot_old + A.row[C.begin + e].x;
#pragma unroll
                        for (int l = 0; l < 4; l++)
                            if ((lanes[u] >> l) & 1)
                                po[l] = xv[l];
                    }
                }
                until = A.every;
            }
            if (j >= cap)
                break;
            // ---- update j + 1
            const double beta = j == 0 ? 0.0 : gamma * inv_g;
            // gamma (gamma / ..): gamma alone squared would leave the range of a double where
            // r.r, whose root is what the caller's units scale, is far from it
            const double alpha = gamma / (delta - gamma * (gamma * inv_ga));
            until--;
            auto ghost = [&](const u64 (&q)[4], double2 &sg, double2 &at) {
                sg.x = fma(beta, sg.x, cgr_value(q[0], q[1]));
                sg.y = fma(beta, sg.y, cgr_value(q[2], q[3]));
                const double2 o = at;
                at = make_double2(fma(-alpha, sg.x, o.x), fma(-alpha, sg.y, o.y));
            };
#pragma unroll
            for (int v = 0; v < GV; v++)
                if (tid + v * NT < nv)
                {
                    const int2 en = GREG ? gl[GREG ? v : 0] : EL[tid + v * NT];
                    if (!cgr_wait2(halo + en.x, gw[v], tag))
                        sh_late = 1;
                    ghost(gw[v], GREG ? gs[GREG ? v : 0] : GS[tid + v * NT],
                          en.y >= 0 ? R0[en.y] : spill[-1 - en.y]);
                }
            // those past the registers' (chunks of a large surface)
            for (int k = tid + GV * NT; k < nv; k += NT)
            {
                const int2 en = xplace[k];
                u64 q[4] = {0, 0, 0, 0};
                if (!cgr_wait2(halo + en.x, q, tag))
                    sh_late = 1;
                ghost(q, xs[k], en.y >= 0 ? R0[en.y] : spill[-1 - en.y]);
            }
#pragma unroll
            for (int u = 0; u < RT; u++)
            {
                const int e = tid + u * CGR_THREADS;
                double pv[4], xv[4];
                if constexpr (!REG)
                {
                    const double2 a = KP[e], b = KP[OWN + e], k = KX[e], q = KX[OWN + e];
                    pv[0] = a.x, pv[1] = a.y, pv[2] = b.x, pv[3] = b.y;
                    xv[0] = k.x, xv[1] = k.y, xv[2] = q.x, xv[3] = q.y;
                }
#pragma unroll
                for (int l = 0; l < 4; l++)
                {
                    double &pl = REG ? p[REG ? u : 0][l] : pv[l];
                    double &xl = REG ? x[REG ? u : 0][l] : xv[l];
                    pl = fma(beta, pl, r[u][l]);
                    sv[u][l] = fma(beta, sv[u][l], w[u][l]);
                    xl = fma(alpha, pl, xl);
                    r[u][l] = fma(-alpha, sv[u][l], r[u][l]);
                }
                R0[1 + e] = make_double2(r[u][0], r[u][1]);
                R1[1 + e] = make_double2(r[u][2], r[u][3]);
                if constexpr (!REG)
                {
                    KP[e] = make_double2(pv[0], pv[1]);
                    KP[OWN + e] = make_double2(pv[2], pv[3]);
                    KX[e] = make_double2(xv[0], xv[1]);
                    KX[OWN + e] = make_double2(xv[2], xv[3]);
                }
            }
            int fail = 0;
            if (until == 0)
            {
#pragma unroll
                for (int u = 0; u < RT; u++)
                {
                    const int e = tid + u * CGR_THREADS;
                    double xv[4], old[4];
                    if constexpr (REG)
                    {
                        const double2 a = KP[e], b = KP[OWN + e];
                        old[0] = a.x, old[1] = a.y, old[2] = b.x, old[3] = b.y;
                    }
                    else
                    {
                        const double2 a = KX[e], b = KX[OWN + e];
                        xv[0] = a.x, xv[1] = a.y, xv[2] = b.x, xv[3] = b.y;
                        const double *po = A.pot_old + (lanes[u] & 15 ? A.row[C.begin + e].x : 0);
#pragma unroll
                        for (int l = 0; l < 4; l++)
                            old[l] = (lanes[u] >> l) & 1 ? po[l] : 1.0;
                    }
#pragma unroll
                    for (int l = 0; l < 4; l++)
                    {
                        // pot / old outside 1 -+ tol2, without the division
                        const double xn = REG ? x[REG ? u : 0][l] : xv[l];
                        if (((lanes[u] >> l) & 1) &&
                            (fabs(xn - old[l]) > A.tol2 * fabs(old[l]) ||
                             (A.method == 1 && fabs(r[u][l]) / rm >= A.tol)))
                            fail = 1;
                    }
                }
            }
            __syncthreads();
            stencil(j + 1, fail);
            // off the chain: while the words travel
            inv_g = 1.0 / gamma;
            inv_ga = inv_g / alpha;
        }
        if (bad)
            break;
#pragma unroll
        for (int u = 0; u < RT; u++)
        {
            const int e = tid + u * CGR_THREADS;
            if (!(lanes[u] & 15))
                continue;
            const int g = A.row[C.begin + e].x;
            double xv[4], old[4];
            const double2 a = (REG ? KP : KX)[e], b = (REG ? KP : KX)[OWN + e];
            const double k[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
            for (int l = 0; l < 4; l++)
            {
                xv[l] = REG ? x[REG ? u : 0][l] : k[l];
                old[l] = k[l];
                if ((lanes[u] >> l) & 1)
                {
                    A.pot[g + l] = xv[l];
                    if constexpr (REG)
                        A.pot_old[g + l] = old[l];
                }
            }
        }
        if (tid == 0 && c == cb)
        {
            A.iters[C.node] = j;
            atomicMax(&A.status[0], j);
            if (converged)
                atomicSub(&A.status[2], 1);
        }
    }
    if (bad && tid == 0)
        atomicOr(&A.status[1], 1);
}

int cgr_wait_probe(qz_sim *s, int out[2])
{
    u64 *w = nullptr; // two lines of words, then the results
    const size_t bytes = (2 * CGR_LINE + 1) * sizeof(u64);
    if (!pool_alloc(s->mem, &w, 2 * CGR_LINE + 1))
    {
        set_error("conjugate gradient wait probe: out of device memory");
        return QZ_FAILURE;
    }
    cudaMemsetAsync(w, 0, bytes, s->stream);
    launch(s, QZ_PROF_OTHER, 0.0, k_cgr_wait_probe, dim3(1), dim3(1), w, (int *)(w + 2 * CGR_LINE));
    const bool ok = check_cuda(cudaMemcpyAsync(out, w + 2 * CGR_LINE, 2 * sizeof(int),
                                               cudaMemcpyDeviceToHost, s->stream), "wait probe") &&
                    check_cuda(cudaStreamSynchronize(s->stream), "wait probe");
    pool_free(s->mem, w);
    if (ok && out[0] && out[1])
        return QZ_SUCCESS;
    if (ok)
        set_error("conjugate gradient: a wait for another block's words gave up");
    return QZ_FAILURE;
}

// ---- host ---------------------------------------------------------------------------------
// Chunks of nodes `set` at size cs.
static long cgr_count(const AmrLevel &L, const std::vector<int> &set, long cs)
{
    long k = 0;
    for (int q : set)
        k += (L.h[q].nrows + cs - 1) / cs;
    return k;
}

// Smallest chunk (a multiple of 8 rows, at least lo) that cuts `set` into CG_FILL
// chunks or fewer, 0 if that is above CGR_CHUNK_MAX.
static long cgr_fit(const AmrLevel &L, const std::vector<int> &set, long lo)
{
    long tot = 0;
    for (int q : set)
        tot += L.h[q].nrows;
    long cs = std::max(lo, ((tot + CG_FILL - 1) / CG_FILL + 7) / 8 * 8);
    while (cs <= CGR_CHUNK_MAX && cgr_count(L, set, cs) > CG_FILL)
        cs += 8;
    return cs <= CGR_CHUNK_MAX ? cs : 0;
}

struct CgrKernel {
    const void *f;
    int threads, rows; // of a block
    long fixed;        // shared memory besides the ghosts'
};
template <int NT, int RT, int GV> static CgrKernel cgr_kernel_of()
{
    return {(const void *)k_cg_resident<NT, RT, GV>, NT, NT * RT, cgr_fixed_bytes<NT, RT, GV>()};
}
// Kernels by the rows a block holds: the fewest threads that hold them, since fewer
// threads have more registers (584 rows with 640 threads 4.53 us an iteration and 608
// 4.03; 1,000 rows with 576 threads of two 6.8 us, with 512 5.3).
static const CgrKernel cgr_kernels[] = {cgr_kernel_of<256, 1, 3>(), cgr_kernel_of<512, 1, 2>(),
                                        cgr_kernel_of<608, 1, 2>(), cgr_kernel_of<512, 2, 3>(),
                                        cgr_kernel_of<576, 2, 2>(), cgr_kernel_of<640, 2, 2>()};
static const CgrKernel &cgr_kernel(long rows)
{
    int k = 0;
    while (cgr_kernels[k].rows < rows)
        k++;
    return cgr_kernels[k];
}

bool cgr_resident(const qz_sim *s)
{
    static PerDevice<bool> of;
    return of.get(s->device, [&] {
        int sms = 0, k = 0;
        bool all = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device) ==
                   cudaSuccess;
        for (const CgrKernel &K : cgr_kernels)
            all = all &&
                  cudaFuncSetAttribute(K.f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       CGR_SMEM) == cudaSuccess &&
                  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, K.f, K.threads, CGR_SMEM) ==
                      cudaSuccess &&
                  (long)k * sms >= CG_FILL;
        cudaGetLastError();
        return all;
    });
}

// Rounds run one after another, the nodes of a round side by side.  Nodes of
// more than one smallest chunk share a round while they fit on chip together (a
// round's length is mostly the trips through L2, whatever its chunks hold).
// Nodes of one chunk need no trip: with many of them they get rounds of
// their own, in which a block solves one after another; a few go along with the
// large nodes unless that would cost those a further row a thread.
void cgr_plan(const AmrLevel &L, const std::vector<char> &take, const std::vector<int> &cap,
              long chunk_min, std::vector<AmrChunk> &chunks, std::vector<int> &node_chunk,
              std::vector<CgrRound> &rounds)
{
    // chunk_min counts points: four to a row
    const long lo = std::min<long>(CGR_CHUNK_MAX,
                                   std::max<long>(CGR_CHUNK_MIN, (chunk_min / 4 + 7) / 8 * 8));
    std::vector<std::vector<int>> sets;
    std::vector<long> size;
    std::vector<int> cur, small;
    long cs = 0;
    for (int q = 0; q < L.nnodes; q++)
    {
        if (!take[q])
            continue;
        if (L.h[q].nrows <= CGR_CHUNK_MIN)
        {
            small.push_back(q);
            continue;
        }
        cur.push_back(q);
        const long fit = cgr_fit(L, cur, lo);
        if (fit)
        {
            cs = fit;
            continue;
        }
        cur.pop_back();
        sets.push_back(cur);
        size.push_back(cs);
        cur.assign(1, q);
        cs = cgr_fit(L, cur, lo);
    }
    if (!cur.empty())
    {
        std::vector<int> all(cur);
        all.insert(all.end(), small.begin(), small.end());
        const long fit = cgr_fit(L, all, lo);
        if (fit && cgr_kernel(fit).rows == cgr_kernel(cs).rows)
        {
            cur.swap(all);
            cs = fit;
            small.clear();
        }
        sets.push_back(cur);
        size.push_back(cs);
    }
    if (!small.empty())
    {
        sets.push_back(small);
        size.push_back(CGR_CHUNK_MIN);
    }
    for (size_t k = 0; k < sets.size(); k++)
    {
        CgrRound R;
        R.first = (int)chunks.size();
        R.chunk = (int)size[k];
        for (int q : sets[k])
        {
            const AmrNode &N = L.h[q];
            node_chunk[2 * q] = (int)chunks.size() - R.first;
            for (int b = N.row_off; b < N.row_off + N.nrows; b += R.chunk)
                chunks.push_back({q, b, std::min(b + R.chunk, N.row_off + N.nrows)});
            node_chunk[2 * q + 1] = (int)chunks.size() - R.first;
            R.shared = R.shared || N.nrows > R.chunk;
            R.cap = std::max(R.cap, cap[q]);
            R.points += N.nintr;
        }
        R.count = (int)chunks.size() - R.first;
        rounds.push_back(R);
    }
}

// Grows buf; new memory starts at zero, which is no iteration's tag.
static bool cgr_words(qz_sim *s, DBuf<u64> &buf, long need)
{
    const long had = buf.cap;
    if (!buf.ensure(s->mem, need))
        return false;
    return buf.cap == had ||
           check_cuda(cudaMemsetAsync(buf.p, 0, buf.cap * sizeof(u64), s->stream), "cg words");
}

static long cgr_halo_words(const AmrLevel &L) { return 8L * std::max(L.row_total, 1); }

bool cgr_reserve(qz_sim *s, const AmrLevel &L, const std::vector<CgrRound> &rounds)
{
    // by the kernels' rows, which a slowly changing tree leaves as they are; a round of
    // one-chunk nodes, whatever their number, exchanges nothing
    long rows = 0;
    for (const CgrRound &R : rounds)
        if (R.shared)
            rows = std::max(rows, (long)cgr_kernel(R.chunk).rows * std::min(CG_FILL, R.count * 2));
    if (rows == 0)
        return true;
    const long halo = cgr_room(2 * cgr_halo_words(L));
    if ((s->cgr_room == 0 || halo <= s->cgr_room) && cgr_words(s, s->cgr_halo, halo) &&
        cgr_words(s, s->cgr_sums, 2L * CGR_LINE * CG_FILL) &&
        s->cgr_list.ensure(s->mem, (6 + CGR_ROW_GHOSTS) * rows) &&
        s->cgr_spill.ensure(s->mem, (2 * CGR_ROW_GHOSTS + 24) * rows))
        return true;
    cudaGetLastError();
    return false;
}

int cgr_launch(qz_sim *s, AmrLevel &L, const std::vector<CgrRound> &rounds, const CgrSolve &v)
{
    if (rounds.empty())
        return QZ_SUCCESS;
    const qz_config &c = s->cfg;
    CgrArgs A;
    memset(&A, 0, sizeof A);
    A.row = L.row.p;
    A.pos = L.pos.p;
    A.nodes = L.nodes.p;
    A.node_chunk = v.node_chunk;
    A.d = L.d;
    A.pot = L.pot;
    A.pot_old = L.pot_old;
    A.status = v.status;
    A.iters = v.iters;
    A.tol = v.tol;
    A.tol2 = v.tol2;
    A.G = c.G;
    A.every = c.check_every > 0 ? c.check_every : 1;
    A.max_iter = c.max_iter;
    A.method = v.method;
    A.thr_node = v.thr_node;
    A.cap_node = v.cap_node;
    const long words = cgr_halo_words(L);
    for (const CgrRound &R : rounds)
    {
        const int blocks = std::min(R.count, CG_FILL);
        // a node of several chunks has all of them resident at once (cgr_plan)
        const CgrKernel &K = cgr_kernel(R.chunk);
        const long rows6 = 6L * R.chunk;
        long gcap = std::min(std::min(rows6, R.chunk + 256L), (CGR_SMEM - K.fixed) / CGR_GHOST_BYTES - 1);
        if (s->cgr_ghosts > 0)
            gcap = std::min<long>(gcap, s->cgr_ghosts);
        const long need = (long)R.cap + 4;
        if (s->cgr_tag < 1 || s->cgr_tag + need >= (1L << 31))
        {
            if (s->cgr_halo.p)
                cudaMemsetAsync(s->cgr_halo.p, 0, s->cgr_halo.cap * sizeof(u64), s->stream);
            if (s->cgr_sums.p)
                cudaMemsetAsync(s->cgr_sums.p, 0, s->cgr_sums.cap * sizeof(u64), s->stream);
            s->cgr_tag = 1;
        }
        A.tag0 = (unsigned)s->cgr_tag;
        s->cgr_tag += need;
        A.chunks = v.chunks + R.first;
        A.nchunks = R.count;
        A.chunk = R.chunk;
        A.gcap = (int)gcap;
        if (R.shared)
        {
            A.halo[0] = s->cgr_halo.p;
            A.halo[1] = s->cgr_halo.p + words;
            A.sums[0] = s->cgr_sums.p;
            A.sums[1] = s->cgr_sums.p + (long)CGR_LINE * CG_FILL;
            A.grow = reinterpret_cast<int2 *>(s->cgr_list.p);
            A.xplace = A.grow + rows6 * R.count;
            A.spill = reinterpret_cast<double2 *>(s->cgr_spill.p);
            A.xs = A.spill + 2 * (rows6 - gcap) * R.count;
        }
        const size_t smem = K.fixed + CGR_GHOST_BYTES * gcap;
        cudaEvent_t eb = nullptr, ee = nullptr;
        if (s->prof)
        {
            eb = prof_event(s);
            ee = prof_event(s);
            cudaEventRecord(eb, s->stream);
        }
        void *args[] = {&A};
        if (!check_cuda(cudaLaunchCooperativeKernel(K.f, dim3(blocks), dim3(K.threads), args, smem,
                                                    s->stream),
                        "on-chip conjugate gradient"))
            return QZ_FAILURE;
        s->stats.kernel_launches++;
        if (s->prof)
        {
            cudaEventRecord(ee, s->stream);
            // d, pot and pot_old in, pot and pot_old out, the order: the iterations stay on chip
            s->prof_pending.push_back({QZ_PROF_CG, 44.0 * R.points, eb, ee});
        }
    }
    return QZ_SUCCESS;
}

} // namespace qz
