// gg_build.cu -- particle permutation, oct-tree construction and moments.
//
// The reference builds its oct-tree by inserting particles one at a time
// (force_treebuild_single, gravity/forcetree.c:152-342) and then computes
// moments with a recursive depth-first pass (force_update_node_recursive,
// forcetree.c:434-942).  Here the tree comes straight from the sorted keys:
// a node is a run of particles sharing a key prefix, so a level-by-level pass
// finds each node's children by binary search on the next 3-bit key digit,
// and children are stored contiguously (first child + count).
//
// Two departures from the reference's node set, neither of which changes a
// force or the interaction count of a target:
//   * chains of single-child nodes are collapsed: a node is stored at the
//     deepest cell that still holds all its particles.  Every node in such a
//     chain has the same mass and centre of mass, and a deeper cell is never
//     opened where a shallower one is not (its len is smaller and its 1.2*len
//     box lies inside the parent's), so the walk uses the same monopole;
//   * a cell with at most `leaf_size` particles is a leaf bucket.  Opening it
//     yields its particles; leaf_size = 1 gives the reference's one-particle
//     leaves.  Cells at the 21-bit key depth with more particles are split
//     into chunks of leaf_size (the reference splits such near-coincident
//     particles at random, forcetree.c:219-231).
// Moments are FP64 sums (mass, mass-weighted position), children summed in
// key order, one depth after the other from the deepest up, with the centre of mass
// falling back to the geometric centre for empty cells (forcetree.c:764-781).
#include <algorithm>

#include "gg_internal.cuh"
#include "gg_kernels.cuh"

#define TB_THREADS 512
#define TB_GROUP 8                      // threads per node when children are looked for
#define TB_NODES (TB_THREADS / TB_GROUP)
#define TB_PER_SM 4                     // blocks per SM that find children: 2,048 threads of 32 registers hide the
                                        // searches' dependent loads
#define TB_MOM_PER_SM 2                 // blocks per SM that form moments (64 registers)

__global__ void k_permute(const unsigned *__restrict__ perm, const GGPart *__restrict__ in, GGPart *__restrict__ out,
                          unsigned *__restrict__ rank, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned src = perm[i];
        if (src >= (unsigned)n) src = 0;   // only after a failed sort, which is reported
        out[i] = in[src];
        rank[src] = (unsigned)i;
    }
}

// deepest common level of two keys (0..21)
__device__ __forceinline__ int common_level(unsigned long long a, unsigned long long b)
{
    unsigned long long x = a ^ b;
    if (x == 0) return GG_MAX_LEVEL;
    int p = 63 - __clzll((long long)x);   // highest differing bit, 0..62
    return GG_MAX_LEVEL - 1 - p / 3;
}

// first index in [lo,hi) with key >= v
__device__ __forceinline__ int lower_bound_key(const unsigned long long *__restrict__ keys, int lo, int hi,
                                               unsigned long long v)
{
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (__ldg(keys + mid) < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// A full-depth cell with more than `leaf` particles is split into at most 8
// equal chunks (which split again at the next depth if still too large), so no
// node ever has more than 8 children.
__device__ __forceinline__ int chunk_size(int cnt, int leaf)
{
    const int n8 = min(8, (cnt + leaf - 1) / leaf);
    return (cnt + n8 - 1) / n8;
}
// every chunk non-empty: ceil(cnt / size) <= 8 chunks of `size` particles (the last may be shorter)
__device__ __forceinline__ int chunk_children(int cnt, int leaf)
{
    const int sz = chunk_size(cnt, leaf);
    return (cnt + sz - 1) / sz;
}

__device__ __forceinline__ unsigned tb_ld_status(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void tb_st_status(unsigned *p, unsigned v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
#define TB_PUBLISHED 0x80000000u

// Barrier of the whole (cooperatively launched) grid: the blocks count up one
// word, and the n-th barrier is passed once n * gridDim.x have arrived.  A wait
// that reaches its limit (some ten seconds: the first one may wait for other
// streams' walks to make room for the whole grid) records GG_EBIT_SORT_TIMEOUT and
// returns false; the block then leaves the kernel, so that later barriers give
// up too and the number of nodes stays zero.
__device__ __forceinline__ bool tb_grid_barrier(const TreeBuf &tb, int which, unsigned &target)
{
    __syncthreads();
    const unsigned extra = (unsigned)tb.wait_extra[which];
    if (gridDim.x + extra == 1) return true;
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        unsigned *const word = tb.barrier + which;
        target += gridDim.x;
        __threadfence();
        atomicAdd(word, 1u);
        int spins = 0;
        while (tb_ld_status(word) < target + extra && ++spins < tb.wait_limit) __nanosleep(20);
        s_ok = spins < tb.wait_limit;
        if (!s_ok) atomicOr(tb.err, GG_EBIT_SORT_TIMEOUT);
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
}

// node k's record and FP64 mass from its sums
__device__ __forceinline__ void tb_finish_node(int k, const TreeBuf &tb, const GGPart *__restrict__ parts,
                                               const GGDomainDev *__restrict__ dom, GGNode *nodes, double M, double sx,
                                               double sy, double sz, float maxsoft, int a, int b)
{
    const int lev = tb.level[k], s = tb.start[k];
    const GGDomainDev d = dom[tb.sys[k]];
    // geometric cell: level `lev` cell containing the node's first particle
    const int gl = lev > GG_MAX_LEVEL ? GG_MAX_LEVEL : lev;
    const double len = ldexp(d.len, -gl);
    double cen[3];
    if (gl == 0) {
        cen[0] = d.center[0]; cen[1] = d.center[1]; cen[2] = d.center[2];
    } else {
        const GGPart p0 = parts[s];
        const double pv[3] = {p0.x, p0.y, p0.z};
        for (int q = 0; q < 3; q++) {
            const unsigned cell = gg_quantize(pv[q], d.corner[q], d.len) >> (GG_MAX_LEVEL - gl);
            cen[q] = d.corner[q] + ((double)cell + 0.5) * len;
        }
    }
    double cx, cy, cz;
    if (M > 0) { cx = sx / M; cy = sy / M; cz = sz / M; }
    else { cx = cen[0]; cy = cen[1]; cz = cen[2]; }
    GGNode nd;
    nd.cx = cx; nd.cy = cy; nd.cz = cz;
    nd.mass = (float)M; nd.len = (float)len; nd.maxsoft = maxsoft;
    nd.gx = (float)(cen[0] - cx); nd.gy = (float)(cen[1] - cy); nd.gz = (float)(cen[2] - cz);
    nd.a = a; nd.b = b; nd.level = lev; nd.parent = tb.parent[k];
    nodes[k] = nd;
    tb.mass64[k] = M;
}

// The tree's nodes in one cooperative launch: roots, then one depth after the
// other.  Every dependence between blocks is a grid barrier (about 1.5 us)
// instead of a kernel boundary, and the loop stops at the tree's own depth.  One
// launch per depth and direction made 57 launches, most of them of empty depths
// in a small tree.  Tree and moments together, B200: 1,000 particles 352 -> 62 us,
// 65,536 430 -> 171, 16.8M 2.02 -> 1.82 ms (in one launch of both, at 64 registers and
// half the threads per SM, 2.34 ms).
//
// One depth: 8 threads per node find the 7 digit boundaries by binary search
// (or the chunk split of a full-depth cell) and the child count; a block
// publishes its children total, adds up the totals of the blocks before it
// (they publish before they wait on anyone) and writes its nodes' children at
// contiguous indices from there.  The last block with nodes sets the next
// depth's range.  A child index at or past the node capacity is not written and
// sets GG_EBIT_NODE_OVERFLOW (the capacity is sized so that it cannot happen).
__global__ void __launch_bounds__(TB_THREADS, TB_PER_SM)
    k_tree_nodes(const unsigned long long *__restrict__ keys, const int *__restrict__ poff, int S, TreeBuf tb, int leaf)
{
    __shared__ int s_sum, s_off, s_tot;
    __shared__ int s_red[TB_THREADS / 32];
    __shared__ int s_nch[TB_NODES];
    __shared__ int s_excl[TB_NODES];
    const int G = gridDim.x, blk = blockIdx.x, tid = threadIdx.x;
    const int gtid = blk * TB_THREADS + tid, gthreads = G * TB_THREADS;
    unsigned target = 0;

    // roots: one per system, geometric level 0 (the domain cube), depth 0
    for (int s = gtid; s < S; s += gthreads) {
        tb.start[s] = poff[s];
        tb.end[s] = poff[s + 1];
        tb.level[s] = 0;
        tb.parent[s] = -1;
        tb.sys[s] = s;
    }
    if (gtid == 0) {
        tb.depth_beg[0] = 0;
        tb.depth_beg[1] = S;
    }
    if (!tb_grid_barrier(tb, 0, target)) return;

    int lb = 0, le = S, depth = 0;
    const int g = tid / TB_GROUP, j = tid % TB_GROUP;
    const int gbase = (tid & 31) & ~(TB_GROUP - 1);
    for (;; depth++) {   // depths 0 .. GG_MAX_DEPTH - 1; the last is all leaves
        const int nl = le - lb;
        const int chunk = max((nl + G - 1) / G, TB_NODES);   // nodes per block: whole passes of the block
        const int cb = lb + blk * chunk, ce = min(le, cb + chunk);
        if (cb < le) {
            const bool one = chunk <= TB_NODES;   // one node per 8 threads: boundaries stay in registers
            if (tid == 0) s_sum = 0;
            __syncthreads();

            // ---- count
            int my = 0, s = 0, e = 0, lev = 0, b = 0, bn = 0, nch = 0;
            for (int base = cb; base < ce; base += TB_NODES) {
                const int k = base + g;
                const bool valid = k < ce;
                s = e = lev = 0;
                if (valid) { s = tb.start[k]; e = tb.end[k]; lev = tb.level[k]; }
                const int cnt = e - s;
                const bool split = valid && cnt > leaf && depth < GG_MAX_DEPTH - 1;
                const bool digit_mode = split && lev < GG_MAX_LEVEL;
                const bool chunk_mode = split && lev >= GG_MAX_LEVEL;
                b = s;
                if (digit_mode && j > 0) {
                    const int shift = 3 * (GG_MAX_LEVEL - (lev + 1));
                    const unsigned long long prefix = keys[s] >> (shift + 3);
                    b = lower_bound_key(keys, s, e, ((prefix << 3) | (unsigned long long)j) << shift);
                }
                if (digit_mode && !one) tb.bnd[(size_t)k * 8 + j] = b;
                const int nb = __shfl_down_sync(0xffffffffu, b, 1, TB_GROUP);
                bn = (j < 7) ? nb : e;
                const unsigned m = __ballot_sync(0xffffffffu, digit_mode && bn > b);
                nch = 0;
                if (digit_mode) nch = __popc((m >> gbase) & 0xFFu);
                else if (chunk_mode) nch = chunk_children(cnt, leaf);
                if (valid && j == 0) {
                    tb.nch[k] = nch;
                    if (!nch) tb.child[k] = -1;
                    my += nch;
                }
            }
            if (my) atomicAdd(&s_sum, my);
            __syncthreads();
            unsigned *const bstat = tb.bstat + (size_t)depth * G;
            if (tid == 0) tb_st_status(bstat + blk, TB_PUBLISHED | (unsigned)s_sum);

            // ---- this block's first child index: the totals of the blocks before it
            int before = 0;
            bool lost = false;
            for (int i = tid; i < blk; i += TB_THREADS) {
                unsigned v = tb_ld_status(bstat + i);
                int spins = 0;
                while (!(v & TB_PUBLISHED)) {
                    if (++spins > tb.wait_limit) {
                        atomicOr(tb.err, GG_EBIT_SORT_TIMEOUT);
                        lost = true;
                        break;
                    }
                    __nanosleep(20);
                    v = tb_ld_status(bstat + i);
                }
                before += (int)(v & ~TB_PUBLISHED);
            }
            before = __reduce_add_sync(0xffffffffu, before);
            if ((tid & 31) == 0) s_red[tid >> 5] = before;
            if (__syncthreads_or(lost)) return;   // without the total the children's places are not known
            if (tid == 0) {
                int off = 0;
                for (int w = 0; w < TB_THREADS / 32; w++) off += s_red[w];
                s_off = off;
                if (ce == le) {   // the last block with nodes: the depth's total is known
                    long long nxt = (long long)le + off + s_sum;
                    if (nxt > tb.cap) {
                        atomicOr(tb.err, GG_EBIT_NODE_OVERFLOW);
                        nxt = tb.cap;
                    }
                    tb.depth_beg[depth + 2] = (int)nxt;
                }
            }
            __syncthreads();   // also orders this block's count-phase stores before the reads below

            // ---- write
            int run = le + s_off;
            if (s_sum != 0) {
                for (int base = cb; base < ce; base += TB_NODES) {
                    const int k = base + g;
                    const bool valid = k < ce;
                    if (!one && valid) {
                        s = tb.start[k];
                        e = tb.end[k];
                        lev = tb.level[k];
                        nch = tb.nch[k];
                    }
                    if (j == 0) s_nch[g] = valid ? nch : 0;
                    __syncthreads();
                    if (tid < 32) {   // exclusive prefix of the TB_NODES = 64 counts, two per lane
                        const int v0 = s_nch[2 * tid], v1 = s_nch[2 * tid + 1];
                        int x = v0 + v1;
                        for (int o = 1; o < 32; o <<= 1) {
                            const int y = __shfl_up_sync(0xffffffffu, x, o);
                            if (tid >= o) x += y;
                        }
                        s_excl[2 * tid] = x - v0 - v1;
                        s_excl[2 * tid + 1] = x - v1;
                        if (tid == 31) s_tot = x;
                    }
                    __syncthreads();
                    if (valid && nch) {
                        const int first = run + s_excl[g], sys = tb.sys[k];
                        if (j == 0) tb.child[k] = first;
                        if (lev >= GG_MAX_LEVEL) {
                            const int csz = chunk_size(e - s, leaf);
                            for (int c = j; c < nch; c += TB_GROUP) {
                                const int idx = first + c;
                                if (idx >= tb.cap) { atomicOr(tb.err, GG_EBIT_NODE_OVERFLOW); continue; }
                                const int cs = s + c * csz, ce2 = min(e, cs + csz);
                                tb.start[idx] = cs; tb.end[idx] = ce2; tb.level[idx] = GG_CHUNK_LEVEL;
                                tb.parent[idx] = k; tb.sys[idx] = sys;
                            }
                        } else {
                            if (!one) {
                                b = tb.bnd[(size_t)k * 8 + j];
                                bn = (j < 7) ? tb.bnd[(size_t)k * 8 + j + 1] : e;
                            }
                            const unsigned gm = 0xFFu << gbase;
                            const unsigned m = __ballot_sync(gm, bn > b);   // the node's 8 threads
                            if (bn > b) {
                                const int idx = first + __popc(m & gm & ((1u << (tid & 31)) - 1u));
                                if (idx >= tb.cap) {
                                    atomicOr(tb.err, GG_EBIT_NODE_OVERFLOW);
                                } else {
                                    tb.start[idx] = b; tb.end[idx] = bn;
                                    tb.level[idx] = common_level(keys[b], keys[bn - 1]);
                                    tb.parent[idx] = k; tb.sys[idx] = sys;
                                }
                            }
                        }
                    }
                    const int tot = s_tot;
                    __syncthreads();
                    run += tot;
                }
            }
        }
        if (!tb_grid_barrier(tb, 0, target)) return;
        lb = le;
        le = __ldcg(tb.depth_beg + depth + 2);
        if (le <= lb || depth + 1 >= GG_MAX_DEPTH) break;   // no nodes at the next depth
    }
    // every node is written; after a wait that gave up or an overflow (its nodes
    // point past the capacity) the number of nodes stays zero
    if (gtid == 0 && !(__ldcg(tb.err) & (GG_EBIT_SORT_TIMEOUT | GG_EBIT_NODE_OVERFLOW))) {
        tb.nnodes[0] = le;
        tb.nnodes[1] = depth;   // the deepest depth: all leaves
    }
}

// Moments, in one cooperative launch: every leaf sums its particles, then one
// depth after the other from the deepest up, an internal node sums its
// children, each in index order in FP64.  Nodes are numbered depth by depth
// with the children of consecutive nodes consecutive, so the lanes of a warp
// read one contiguous stretch of child records (or of particles).
__global__ void __launch_bounds__(TB_THREADS, TB_MOM_PER_SM)
    k_tree_moments(TreeBuf tb, const GGPart *__restrict__ parts, const GGDomainDev *__restrict__ dom, GGNode *nodes)
{
    const int gtid = blockIdx.x * TB_THREADS + threadIdx.x, gthreads = gridDim.x * TB_THREADS;
    __shared__ int s_total;
    if (threadIdx.x == 0) s_total = __ldcg(tb.nnodes);
    __syncthreads();
    const int total = s_total, depth = tb.nnodes[1];
    if (total == 0) return;   // no tree
    unsigned target = 0;
    for (int k = gtid; k < total; k += gthreads) {
        if (tb.child[k] >= 0) continue;
        double M = 0, sx = 0, sy = 0, sz = 0;
        float maxsoft = 0;
        const int s = tb.start[k], e = tb.end[k];
        for (int i = s; i < e; i++) {
            const GGPart p = parts[i];
            const double m = (double)p.m;
            M += m;
            sx += m * p.x; sy += m * p.y; sz += m * p.z;
            maxsoft = fmaxf(maxsoft, p.h);
        }
        tb_finish_node(k, tb, parts, dom, nodes, M, sx, sy, sz, maxsoft, s, -(e - s));
    }
    // internal nodes, deepest first
    for (int d = depth - 1; d >= 0; d--) {
        if (!tb_grid_barrier(tb, 1, target)) {
            if (threadIdx.x == 0) *(volatile int *)tb.nnodes = 0;   // unfinished nodes are not to be read
            return;
        }
        const int db = __ldcg(tb.depth_beg + d), de = __ldcg(tb.depth_beg + d + 1);
        for (int k = db + gtid; k < de; k += gthreads) {
            const int c0 = tb.child[k];
            if (c0 < 0) continue;
            double M = 0, sx = 0, sy = 0, sz = 0;
            float maxsoft = 0;
            const int nc = tb.nch[k];
            for (int c = c0; c < c0 + nc; c++) {   // written by other blocks of this launch: read through L2
                const double m = __ldcg(tb.mass64 + c);
                const double2 xy = __ldcg(reinterpret_cast<const double2 *>(&nodes[c].cx));
                const double z = __ldcg(&nodes[c].cz);
                M += m;
                sx += m * xy.x; sy += m * xy.y; sz += m * z;
                maxsoft = fmaxf(maxsoft, __ldcg(&nodes[c].maxsoft));
            }
            tb_finish_node(k, tb, parts, dom, nodes, M, sx, sy, sz, maxsoft, c0, nc);
        }
    }
}

void gg_launch_permute(const unsigned *perm, const GGPart *in, GGPart *out, unsigned *rank, int n, cudaStream_t st)
{
    int threads = 256, blocks = gg_num_sms() * 8;
    if ((long long)blocks * threads > n) blocks = (n + threads - 1) / threads;
    if (blocks < 1) blocks = 1;
    k_permute<<<blocks, threads, 0, st>>>(perm, in, out, rank, n);
    gg_note_launches(1);
}

// blocks of the node kernel at most (its look-back words are sized for them)
int gg_tree_grid() { return gg_num_sms() * TB_PER_SM; }

gg_status gg_launch_tree(const unsigned long long *keys, const int *poff, int S, int n, int leaf, int cap, TreeBuf tb,
                         const GGPart *parts, const GGDomainDev *dom, GGNode *nodes, cudaStream_t st)
{
    // about 1,024 particles per block: few blocks for a small tree, as a barrier
    // of one block costs nothing (1,000 particles: 53 us in one block, 76 us in
    // two; 65,536: 165 us in 64 blocks, 192 us in 16)
    const long long want = ((long long)n + S + 1023) / 1024;
    const int G = (int)std::min((long long)gg_tree_grid(), want);
    const int Gm = (int)std::min((long long)gg_num_sms() * TB_MOM_PER_SM, want);
    tb.cap = cap;
    GG_CUDA_TRY(cudaMemsetAsync(tb.nnodes, 0, TREE_STATE_WORDS(G) * sizeof(unsigned), st));
    void *args[] = {&keys, &poff, &S, &tb, &leaf};
    GG_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_tree_nodes, dim3(G), dim3(TB_THREADS), args, 0, st));
    void *margs[] = {&tb, &parts, &dom, &nodes};
    GG_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_tree_moments, dim3(Gm), dim3(TB_THREADS), margs, 0, st));
    gg_note_launches(2);
    return GG_OK;
}
