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
#define TB_GIVEN_UP 0x80000000u

// How the blocks of a tree kernel work together.  Each depth (each phase of the
// moments) is cut into parts, at most one per block of the grid, and a block
// takes one part after the other by ticket: all parts of a depth, then those of
// the next.  A part waits only for parts with earlier tickets, which are
// finished or held by a block that runs and whose earlier part is finished: so
// however few blocks find room beside other kernels, the first unfinished part
// can always go on.  (A grid barrier needs every block resident at once: a
// kernel of another stream that holds a single warp slot kept a build of 600,000
// particles from starting.)
//
// `first` (shared memory, thread 0's) is the ticket of the phase's first part, and
// a block's place its ticket less that.  tb_step ends a block's turn at a phase of
// `parts` parts: the part it worked on is counted as finished and its next ticket
// taken; if that is not of this phase, it waits until all parts are finished and
// goes on to the next phase (*moved).  It returns the new place, or -1 after a wait
// that reached its limit (some ten seconds): that one records
// GG_EBIT_SORT_TIMEOUT and marks the word, so that the others leave too; the
// number of nodes stays zero.
__device__ __forceinline__ int tb_step(const TreeBuf &tb, int kernel, int phase, int parts, int &first, int place,
                                       bool *moved)
{
    __shared__ int s_place, s_moved;
    __syncthreads();
    if (gridDim.x + tb.wait_extra[kernel] == 1) {   // one block, one part per phase, nobody to wait for
        *moved = true;
        return 0;
    }
    if (threadIdx.x == 0) {
        unsigned *const word = tb.done + kernel * TREE_PHASES + phase;
        const unsigned want = (unsigned)(parts + tb.wait_extra[kernel]);
        int next = first + place;
        if (place < parts) {
            __threadfence();
            atomicAdd(word, 1u);
            next = (int)atomicAdd(tb.ticket + kernel, 1u);
        }
        unsigned v = tb_ld_status(word);   // in flight together with the ticket
        const bool over = next - first >= parts;
        if (over) first += parts;
        s_place = next - first;
        s_moved = over;
        if (over) {
            int spins = 0;
            while (v < want && ++spins < tb.wait_limit) {   // (the mark ends it)
                __nanosleep(20);
                v = tb_ld_status(word);
            }
            if (v < want) {
                atomicOr(tb.err, GG_EBIT_SORT_TIMEOUT);
                atomicOr(word, TB_GIVEN_UP);
            }
            if (v < want || (v & TB_GIVEN_UP)) s_place = -1;
            __threadfence();
        }
    }
    __syncthreads();
    *moved = s_moved;
    return s_place;
}
// a block's first ticket
__device__ __forceinline__ int tb_first(const TreeBuf &tb, int kernel)
{
    return gridDim.x == 1 ? 0 : (int)atomicAdd(tb.ticket + kernel, 1u);
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

// The tree's nodes in one launch: one depth after the other, down to the tree's
// own depth.  A wait between two depths costs about 1.5 us instead of a kernel
// boundary; one launch per depth and direction made 57 launches, most of them
// of empty depths in a small tree.  Tree and moments together, B200: 1,000
// particles 352 -> 63 us, 65,536 430 -> 176, 16.8M 2.02 -> 1.78 ms (in one launch of
// both, at 64 registers and half the threads per SM, 2.34 ms; with a grid barrier
// instead of the tickets 60 us, 170, 1.81).
//
// One depth: 8 threads per node find the 7 digit boundaries by binary search
// (or the chunk split of a full-depth cell) and the child count; a block
// publishes its part's children total, adds up the totals of the parts before it
// (published before their blocks wait on anyone) and writes its nodes' children at
// contiguous indices from there.  The last part sets the next depth's range.  A
// child index at or past the node capacity is not written and sets
// GG_EBIT_NODE_OVERFLOW (the capacity is sized so that it cannot happen).
__global__ void __launch_bounds__(TB_THREADS, TB_PER_SM)
    k_tree_nodes(const unsigned long long *__restrict__ keys, const int *__restrict__ poff, int S, TreeBuf tb, int leaf)
{
    __shared__ int s_sum, s_off, s_tot;
    __shared__ int s_red[TB_THREADS / 32];
    __shared__ int s_nch[TB_NODES];
    __shared__ int s_excl[TB_NODES];
    const int G = gridDim.x, tid = threadIdx.x;
    const int g = tid / TB_GROUP, j = tid % TB_GROUP;
    const int gbase = (tid & 31) & ~(TB_GROUP - 1);
    int lb = 0, le = S, depth = 0;   // nodes lb to le - 1 of a depth; depths 0 .. GG_MAX_DEPTH - 1, the last all leaves
    __shared__ int s_first;
    if (tid == 0) {
        s_first = 0;
        s_tot = tb_first(tb, 0);
    }
    __syncthreads();
    int blk = s_tot;   // place in the depth
    for (;;) {
        const int nl = le - lb;
        const int chunk = max((nl + G - 1) / G, TB_NODES);   // nodes per part: whole passes of the block
        const int parts = (nl + chunk - 1) / chunk;
        if (blk < parts) {
            const int cb = lb + blk * chunk, ce = min(le, cb + chunk);
            const bool one = chunk <= TB_NODES;   // one node per 8 threads: boundaries stay in registers
            if (depth == 0) {   // roots: one per system, geometric level 0 (the domain cube)
                for (int s = cb + tid; s < ce; s += TB_THREADS) {
                    tb.start[s] = poff[s];
                    tb.end[s] = poff[s + 1];
                    tb.level[s] = 0;
                    tb.parent[s] = -1;
                    tb.sys[s] = s;
                }
                if (tid == 0 && blk == 0) {
                    tb.depth_beg[0] = 0;
                    tb.depth_beg[1] = S;
                }
            }
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

            // ---- this part's first child index: the totals of the parts before it
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
            if (__syncthreads_or(lost)) {   // without the total the children's places are not known
                if (tid == 0) atomicOr(tb.done + depth, TB_GIVEN_UP);
                return;
            }
            if (tid == 0) {
                int off = 0;
                for (int w = 0; w < TB_THREADS / 32; w++) off += s_red[w];
                s_off = off;
                if (ce == le) {   // the last part: the depth's total is known
                    long long nxt = (long long)le + off + s_sum;
                    if (nxt > tb.cap) {
                        atomicOr(tb.err, GG_EBIT_NODE_OVERFLOW);
                        nxt = tb.cap;
                    }
                    tb.depth_beg[depth + 2] = (int)nxt;
                }
            }
            __syncthreads();   // also orders this part's count-phase stores before the reads below

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
        bool moved;
        blk = tb_step(tb, 0, depth, parts, s_first, blk, &moved);
        if (blk < 0) return;
        if (moved) {
            depth++;
            lb = le;
            le = __ldcg(tb.depth_beg + depth + 1);
            if (le <= lb || depth >= GG_MAX_DEPTH) break;   // no nodes at the next depth
        }
    }
    // every node is written; after a wait that gave up or an overflow (its nodes
    // point past the capacity) the number of nodes stays zero
    if (blk == 0 && tid == 0 && !(__ldcg(tb.err) & (GG_EBIT_SORT_TIMEOUT | GG_EBIT_NODE_OVERFLOW))) {
        tb.nnodes[0] = lb;
        tb.nnodes[1] = depth - 1;   // the deepest depth: all leaves
    }
}

// Moments, in one launch: every leaf sums its particles, then one
// depth after the other from the deepest up, an internal node sums its
// children, each in index order in FP64.  Nodes are numbered depth by depth
// with the children of consecutive nodes consecutive, so the lanes of a warp
// read one contiguous stretch of child records (or of particles).
__global__ void __launch_bounds__(TB_THREADS, TB_MOM_PER_SM)
    k_tree_moments(TreeBuf tb, const GGPart *__restrict__ parts, const GGDomainDev *__restrict__ dom, GGNode *nodes)
{
    __shared__ int s_total, s_ticket, s_first;
    if (threadIdx.x == 0) {
        s_first = 0;
        s_total = __ldcg(tb.nnodes);
        s_ticket = tb_first(tb, 1);
    }
    __syncthreads();
    const int depth = tb.nnodes[1];
    int place = s_ticket;
    if (s_total == 0) return;   // no tree
    // phase 0: the leaves of every depth; phase p: the internal nodes of depth `depth - p`
    for (int phase = 0;;) {
        const int kb = phase == 0 ? 0 : tb.depth_beg[depth - phase];
        const int ke = phase == 0 ? s_total : tb.depth_beg[depth - phase + 1];
        const int nparts = min((int)gridDim.x, (ke - kb + TB_THREADS - 1) / TB_THREADS);
        if (place < nparts) {
            for (int k = kb + place * TB_THREADS + threadIdx.x; k < ke; k += nparts * TB_THREADS) {
                const int c0 = tb.child[k];
                if ((c0 < 0) != (phase == 0)) continue;
                double M = 0, sx = 0, sy = 0, sz = 0;
                float maxsoft = 0;
                if (phase == 0) {
                    const int s = tb.start[k], e = tb.end[k];
                    for (int i = s; i < e; i++) {
                        const GGPart p = parts[i];
                        const double m = (double)p.m;
                        M += m;
                        sx += m * p.x; sy += m * p.y; sz += m * p.z;
                        maxsoft = fmaxf(maxsoft, p.h);
                    }
                    tb_finish_node(k, tb, parts, dom, nodes, M, sx, sy, sz, maxsoft, s, -(e - s));
                } else {
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
        } else if (phase == depth) {
            return;
        }
        bool moved;
        place = tb_step(tb, 1, phase, nparts, s_first, place, &moved);
        if (place < 0) {
            if (threadIdx.x == 0) *(volatile int *)tb.nnodes = 0;   // unfinished nodes are not to be read
            return;
        }
        if (moved && phase++ == depth) return;
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
    // about 1,024 particles per block: few blocks for a small tree, as the waits
    // of one block cost nothing (1,000 particles: 53 us in one block, 76 us in
    // two; 65,536: 165 us in 64 blocks, 192 us in 16)
    const long long want = ((long long)n + S + 1023) / 1024;
    const int G = (int)std::min((long long)gg_tree_grid(), want);
    const int Gm = (int)std::min((long long)gg_num_sms() * TB_MOM_PER_SM, want);
    tb.cap = cap;
    GG_CUDA_TRY(cudaMemsetAsync(tb.nnodes, 0, TREE_STATE_WORDS(G) * sizeof(unsigned), st));
    k_tree_nodes<<<G, TB_THREADS, 0, st>>>(keys, poff, S, tb, leaf);
    k_tree_moments<<<Gm, TB_THREADS, 0, st>>>(tb, parts, dom, nodes);
    GG_CUDA_TRY(cudaGetLastError());
    gg_note_launches(2);
    return GG_OK;
}
