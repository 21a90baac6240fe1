// gg_walk.cu -- warp-cooperative tree walk (force_treeevaluate, forcetree.c:1633-2807).
//
// A warp serves one group of up to 64 targets that are consecutive in
// Peano-Hilbert order (two targets per lane; see Targets).  The warp walks the tree once
// for the whole group with an explicit node stack: each round takes up to 64
// nodes, two per lane, and tests them against the group's bounding box with
// the reference's opening rules made conservative over the group
// (distance = from the node's centre of mass to the box, the smallest
// ErrTolForceAcc*OldAcc of the group, the largest target softening):
//   - massless nodes are skipped                         (forcetree.c:2038)
//   - one-particle nodes are always opened               (:2043-2050)
//   - h < maxsoft and r^2 < maxsoft^2 opens              (:2099-2102)
//   - Barnes-Hut pass: len^2 > r^2 theta^2 opens         (:2104-2111)
//   - relative pass: r^2 < (soft+0.6 len)^2 or
//     r^2 < (maxsoft+0.6 len)^2, m len^2 > r^4 aold, or
//     the target inside the 1.2*len box opens           (:2119-2147)
// For a group of one target these are exactly the reference's tests, run in
// FP64 on the FP64 centre of mass (exact mode).  Larger groups run the same
// tests in FP32 on offsets from the group centre, with the box half-widths
// rounded up; a test within FP32 rounding of its threshold may go either way,
// which is far below the margin the group's conservative box adds.  Used nodes and particles are
// appended (ballot + popc compaction) to per-warp shared-memory lists as
// FP32 offsets from the group centre; a "far" list holds entries that are
// Newtonian for every target of the group (no softening branch, no self
// term) and a "near" list holds the rest.  When a list reaches the flush
// threshold every lane evaluates it for its targets in FP32 (cubic-spline
// softening, kernel.h:452-470, with h = max(h_target, h_source),
// forcetree.c:2263-2283); each flush's partial sums are added to the
// per-target totals with Kahan compensation.  Interactions are counted like
// the reference (forcetree.c:2258, :2488): one per used node or particle with
// r^2 > 0 and m > 0.
//
// How the work is arranged on the SM (each part is described where it is):
//   - the next round's node records are staged in shared memory while this
//     round's leaves and flushes run (per-lane cp.async, or bulk copies of
//     runs of consecutive records on an mbarrier);
//   - a round tests up to 64 nodes, two per lane; the opened nodes' children are
//     laid end to end by one scan, and the next round takes them from there; the
//     particles of opened leaves queue as runs and are classified 32 at a time;
//   - the lists are one array per component, evaluated two entries per packed
//     FP32x2 instruction;
//   - the persistent warps take groups in the order the host side planned
//     (most expensive first, from the previous walk's measured cost), and each
//     group records its own cost for the next walk.
#include <climits>

#include "gg_internal.cuh"
#include "gg_kernels.cuh"

#define WALK_THREADS 256
#define WALK_WARPS (WALK_THREADS / 32)
#define FULL 0xffffffffu

int gg_walk_threads() { return WALK_THREADS; }

// Per-warp shared memory, in floats:
//   far list [FAR_ARRAYS][FAR_CAP] | near list [NEAR_ARRAYS][NEAR_CAP] | node stack int[WALK_SSTACK] |
//   node slots GGNode[32 NH] | runs of a window int[32] | queued runs int[2][RUNS] |
//   mbarrier of the node copies (16 bytes)
// The stack spills to the warp's global stack area when it overflows (deep or
// wide traversals only).
#define WALK_SSTACK 512
// Queue of the runs of particles of opened leaves (a ring): its particles are
// taken 32 at a time.  Fewer than 32 particles, so at most 31 runs, wait when a
// round adds its own (up to 32 NH).
#define RUNS 128
// The lists are arrays of one component each ({x, y, z, m}; near: {x, y, z} and
// a softening record of three): lanes append to consecutive words, and a
// flush loads two or four consecutive entries of a component at once.
#define FAR_ARRAYS 4
#define NEAR_ARRAYS 6
// Nodes per lane and round: with two, the round's fixed part (loop, scan,
// windows) is paid once for 64 nodes.  Per 1M clustered walk, groups of 32:
// 2.15e9 -> 2.00e9 warp instructions, 3.07 -> 2.88 ms.
#define NH 2
// A list is evaluated when it holds this many entries (or the configured
// threshold, if smaller).  Between two looks at the thresholds a round appends
// up to 32 NH nodes and a batch of 32 particles.  Longer lists would save some of
// the flushes' fixed part; two blocks' shared memory is all there is.
#define FAR_FLUSH_MAX 96
#define NEAR_FLUSH_MAX 64
#define FAR_CAP (FAR_FLUSH_MAX + 32 * NH + 32)
#define NEAR_CAP (NEAR_FLUSH_MAX + 32 * NH + 32)
#define WALK_WARP_FLOATS \
    (FAR_ARRAYS * FAR_CAP + NEAR_ARRAYS * NEAR_CAP + WALK_SSTACK + NH * 32 * 16 + 32 + 2 * RUNS + 4 + 8)

// ---- staging of node records
// The next round's node records are copied into shared memory, one 64-byte slot
// per lane, while this round's leaves and flushes are processed; no registers
// are held while the copies are in flight.  A lane's slot is refilled only
// after its test of the node in it is complete.  Two ways (gg_config
// .node_staging), measured close to each other:
//  0: each lane copies its own record with cp.async (16-byte pieces through
//     L1, where the top levels of the tree, which every group visits, hit);
//  1: the bulk-copy (TMA) engine, one copy per run of consecutive records.
// (Staging two rounds ahead, in two slots, measured no faster.)
// Slots are 64 bytes apart, so the lanes' i-th 16-byte pieces would meet in two
// of the eight 16-byte bank groups: piece i of slot l lies at piece
// i ^ ((l >> 1) & 3), which spreads every eight lanes over all banks.  (A bulk
// copy writes records as they are.  Four lanes per record, which looks up each
// cache line once instead of four times, measured no faster: the walk is bound by
// instruction issue, and the lanes then have to exchange their node indices.)
__device__ __forceinline__ void stage_lanes(unsigned slot0, const GGNode *nodes, const int (&node)[NH], int k, int lane)
{
    const int swz = (lane >> 1) & 3;
#pragma unroll
    for (int h = 0; h < NH; h++)
        if (32 * h + lane < k) {
            const int4 *src = reinterpret_cast<const int4 *>(nodes + node[h]);
#pragma unroll
            for (int i = 0; i < 4; i++)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(slot0 + 64u * (32 * h + lane) +
                                                                              16u * (i ^ swz)),
                             "l"(src + i)
                             : "memory");
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Bulk copies: the nodes a round pops sit in
// consecutive lanes, and the children of one node are consecutive records, so
// they form a few runs of consecutive records: the first lane of each run
// issues one cp.async.bulk for the whole run.  The copies complete on the
// warp's mbarrier, which lane 0 arms with the round's byte count; the test
// waits on the barrier's phase.  Every wait is bounded: after WALK_WAIT_LIMIT
// polls the warp records GG_EBIT_WALK_TIMEOUT, waits once more (bounded) for
// its copies and leaves the kernel.
#define WALK_WAIT_LIMIT (1 << 20)

__device__ __forceinline__ void stage_nodes(unsigned bar, unsigned slot0, const GGNode *nodes, const int (&node)[NH],
                                            int k, int lane)
{
    // the slots were read by this round's tests, whose values were consumed
    // before the next nodes were known (warp-synchronous): the copies may overwrite them
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(k * 64) : "memory");
    __syncwarp();
#pragma unroll
    for (int h = 0; h < NH; h++) {
        const int kh = min(k - 32 * h, 32);   // nodes of this part
        if (kh <= 0) break;
        const int prev = __shfl_up_sync(FULL, node[h], 1);
        const bool start = lane < kh && (lane == 0 || node[h] != prev + 1);
        const unsigned starts = __ballot_sync(FULL, start);
        if (start) {
            const unsigned later = starts & ~((2u << lane) - 1u);   // run starts after this lane
            const int end = later ? __ffs(later) - 1 : kh;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(slot0 + 64u * (32 * h + lane)), "l"(nodes + node[h]), "r"(64u * (end - lane)), "r"(bar)
                         : "memory");
        }
    }
}

// true once the phase of the given parity has completed; false if the bounded
// wait gave up
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity)
{
    for (int i = 0; i < WALK_WAIT_LIMIT; i++) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// a particle record in one 256-bit load
__device__ __forceinline__ GGPart load_part(const GGPart *p)
{
    GGPart r;
    double mh;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(mh) : "l"(p));
    r.m = __int_as_float(__double2loint(mh));
    r.h = __int_as_float(__double2hiint(mh));
    return r;
}

struct Kahan {
    float s, c;
    __device__ __forceinline__ void add(float x)
    {
        float y = x - c;
        float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// This file is compiled with denormals flushed to zero (-ftz=true): rsqrtf and
// the reciprocals are then single hardware approximations without range
// fix-ups.  An entry goes to the far list only when its squared distance from
// the group's box exceeds FAR_MIN_R2, so every far pair has a normal r^2; near
// pairs are selected, not multiplied, out of the sums when r^2 is zero (and
// r^2 below the smallest normal float is zero here).
#define FAR_MIN_R2 1e-36f

// ---- packed FP32x2 arithmetic (sm_100): one instruction, two IEEE FP32
// operations with round-to-nearest, each exactly the scalar operation
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sel2(bool px, bool py, float2 a, float2 b)
{
    return make_float2(px ? a.x : b.x, py ? a.y : b.y);
}

// component arrays of a list: entry j
__device__ __forceinline__ void list_put(float *list, int j, float4 v)
{
    list[j] = v.x;
    list[FAR_CAP + j] = v.y;
    list[2 * FAR_CAP + j] = v.z;
    list[3 * FAR_CAP + j] = v.w;
}
// near entry j: position, and its softening record (see near_soft)
__device__ __forceinline__ void near_put(float *list, int j, float4 v, float4 soft)
{
    list[j] = v.x;
    list[NEAR_CAP + j] = v.y;
    list[2 * NEAR_CAP + j] = v.z;
    list[3 * NEAR_CAP + j] = soft.x;
    list[4 * NEAR_CAP + j] = soft.y;
    list[5 * NEAR_CAP + j] = soft.z;
}
// A flush takes a whole number of quanta; the last one of a group is filled up
// with massless entries 1e18 away (r^2 is finite and the terms exactly zero).
#define PAD_ENTRY make_float4(1e18f, 1e18f, 1e18f, 0.f)
#define PAD_SOFT make_float4(1.f, 0.f, 0.f, 0.f)

// Cubic-spline softened force and potential factors for u = r/h < 1
// (kernel.h:452-470), without a branch or a per-piece coefficient choice.  The
// outer piece (0.5 <= u < 1) equals the inner polynomial plus a correction
// that vanishes below u = 0.5, written in t = max(u - 0.5, 0):
//   w_force = 32/3 + u^2 (32 u - 38.4)  -  256 t^4 (t^2/6 + t/5 + 1/16) / u^3
//   w_pot   = -2.8 + u^2 (16/3 + u^2 (6.4 u - 9.6))  +  t^5 (-6.4 - 128/15 t) / u
// (the force correction is the mass the outer piece of the density removes,
// divided by u^3; the potential correction integrates u times it from 0.5).
// iu = 1/u is passed in (the caller has it from r^-1).  The corrections are
// multiplied out starting from t, so a zero t stays zero however large iu is.
// Returns w_force, writes w_pot; they are still to be scaled by h^-3 and h^-1.
// Two pairs at a time, in packed FP32x2.
__device__ __forceinline__ float2 spline_wf2(float2 u, float2 iu, float2 *wp)
{
    const float2 u2 = mul2(u, u);
    const float2 um = add2(u, dup2(-0.5f));
    const float2 t = make_float2(fmaxf(um.x, 0.f), fmaxf(um.y, 0.f));
    const float2 t2 = mul2(t, t), t4 = mul2(t2, t2);
    const float2 fin = fma2(u2, fma2(u, dup2(32.f), dup2(-38.4f)), dup2(10.666666666667f));
    const float2 q = mul2(t4, fma2(t, fma2(t, dup2(0.166666666667f), dup2(0.2f)), dup2(0.0625f)));
    const float2 pin = fma2(u2, fma2(u2, fma2(u, dup2(6.4f), dup2(-9.6f)), dup2(5.333333333333f)), dup2(-2.8f));
    *wp = fma2(mul2(mul2(t4, t), fma2(t, dup2(-8.533333333333f), dup2(-6.4f))), iu, pin);
    return fma2(dup2(-256.f), mul2(mul2(mul2(q, iu), iu), iu), fin);
}

// Targets per lane (TPL) and lane parts (SPLIT): the warp's SPLIT parts of
// 32 / SPLIT lanes all hold the same TPL * 32 / SPLIT targets, and each part
// evaluates its share of the list entries.  Groups of up to 32 targets use
// TPL = SPLIT = 2, larger ones TPL = 2, SPLIT = 1.  With two targets per lane a
// load of entries serves both, and the parts load different entries at once:
// half the loads per target of one target per lane, and half the L1 cycles (a
// uniform 128-bit shared-memory load returns 512 bytes to the warp: with one
// target per lane L1 was 82% busy in the far flush).
//
// What bounds the walk is instruction issue.  A packed FP32x2 instruction takes
// two issue slots; counting those twice, 89-94% of all slots are taken (1M
// particles: clustered 63% issue active + half of the FMA pipe's 53%, in groups of
// 64 61% + half of 64%, galaxy 65% + half of 58%).  The far flush alone runs at 15.1
// slots per entry and 32 targets (13 FP32 operations, one rsqrt, a share of the
// loads), the near flush at 43 (49.9 before its softening record was {h^-2, m/h,
// m/h^3}).
template <int TPL>
struct Targets {
    float x[TPL], y[TPL], z[TPL], h[TPL], hinv[TPL];
    bool valid[TPL];
    Kahan ax[TPL], ay[TPL], az[TPL], pot[TPL];
    int self[TPL];   // near entries at r = 0: the target itself or a coincident particle
};

// The per-entry sums of a flush, added to the targets' Kahan totals.
template <int TPL, bool POT>
__device__ __forceinline__ void add_sums(Targets<TPL> &T, const float2 (&px)[TPL], const float2 (&py)[TPL],
                                         const float2 (&pz)[TPL], const float2 (&pp)[TPL])
{
#pragma unroll
    for (int s = 0; s < TPL; s++) {
        if (!POT) {
            T.ax[s].add(px[s].x + px[s].y);
            T.ay[s].add(py[s].x + py[s].y);
            T.az[s].add(pz[s].x + pz[s].y);
        }
        T.pot[s].add(pp[s].x + pp[s].y);
    }
}

// Far list: Newtonian for every target of the group, two entries per packed
// instruction, four per load.  n is a whole number of quanta (4 * SPLIT
// entries).  Each flush keeps one partial sum per entry parity and adds both
// into the Kahan totals.
// POT: the potential-only walk (force_treeevaluate_potential, forcetree.c:3169-3474)
template <int TPL, int SPLIT, bool POT>
__device__ __forceinline__ void flush_far(const float *__restrict__ far, int n, int part, Targets<TPL> &T)
{
    float2 px[TPL], py[TPL], pz[TPL], pp[TPL], nx[TPL], ny[TPL], nz[TPL];
#pragma unroll
    for (int s = 0; s < TPL; s++) {
        px[s] = py[s] = pz[s] = pp[s] = dup2(0.f);
        nx[s] = dup2(-T.x[s]); ny[s] = dup2(-T.y[s]); nz[s] = dup2(-T.z[s]);
    }
    const float4 *X = reinterpret_cast<const float4 *>(far) + part;
    constexpr int c4 = FAR_CAP / 4;
#pragma unroll 1
    for (int q = n / (4 * SPLIT); q > 0; q--, X += SPLIT) {
        const float4 x4 = X[0], y4 = X[c4], z4 = X[2 * c4], m4 = X[3 * c4];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float2 ex = e ? make_float2(x4.z, x4.w) : make_float2(x4.x, x4.y);
            const float2 ey = e ? make_float2(y4.z, y4.w) : make_float2(y4.x, y4.y);
            const float2 ez = e ? make_float2(z4.z, z4.w) : make_float2(z4.x, z4.y);
            const float2 em = e ? make_float2(m4.z, m4.w) : make_float2(m4.x, m4.y);
#pragma unroll
            for (int s = 0; s < TPL; s++) {
                const float2 dx = add2(ex, nx[s]), dy = add2(ey, ny[s]), dz = add2(ez, nz[s]);
                const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                const float2 rinv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                const float2 mr = mul2(em, rinv);
                if (!POT) {
                    const float2 fac = mul2(mul2(mr, rinv), rinv);
                    px[s] = fma2(dx, fac, px[s]);
                    py[s] = fma2(dy, fac, py[s]);
                    pz[s] = fma2(dz, fac, pz[s]);
                }
                pp[s] = fma2(mr, dup2(-1.f), pp[s]);
            }
        }
    }
    add_sums<TPL, POT>(T, px, py, pz, pp);
}

// Near list: entries within the softening of some target of the group.  Most
// of them need the spline for some lanes and the Newtonian form for others
// (both for 85% of entries on the galaxy), so every lane evaluates both
// branch-free and selects, two entries per packed instruction.  r^2 = 0 (the
// target itself, or a coincident particle) contributes nothing and is not
// counted.
// POT: the potential-only walk, which has no r^2 > 0 condition: an r = 0 pair
// adds m w_pot(0) / h like any other (the caller removes the self term).
//
// This form is for groups of one kernel radius h_t (most groups): the pair's
// softening h_g = max(h_t, h_source) and its products are per entry, formed
// when the entry was listed: {h_g^-2, m/h_g, m/h_g^3}.  u^2 = r^2 / h_g^2 and its
// rsqrt give u and 1/u, and force and potential share t^4/u (t and the spline:
// see spline_wf2).
// r^2 = 0 gives u = 1e-18: a finite force factor, times an offset of zero.
// Unrolled by two, so that few warps have two chains in flight: walk of 100
// targets scattered over a galaxy of 500,000 (4 groups) 32.5 -> 32.0 ms, 4.2M galaxy
// 44.7 -> 44.3 ms.  (The far flush unrolled spills: 45.8 ms; so does this one in the
// kernel of cut walks of groups beyond 32, where it stays as it is.)
template <int TPL, int SPLIT, bool POT, int UNROLL>
__device__ __forceinline__ void flush_near(const float *__restrict__ near, int n, int part, Targets<TPL> &T)
{
    float2 px[TPL], py[TPL], pz[TPL], pp[TPL], nx[TPL], ny[TPL], nz[TPL];
#pragma unroll
    for (int s = 0; s < TPL; s++) {
        px[s] = py[s] = pz[s] = pp[s] = dup2(0.f);
        nx[s] = dup2(-T.x[s]); ny[s] = dup2(-T.y[s]); nz[s] = dup2(-T.z[s]);
    }
    const float2 *X = reinterpret_cast<const float2 *>(near) + part;
    constexpr int c2 = NEAR_CAP / 2;
#pragma unroll UNROLL
    for (int q = n / (2 * SPLIT); q > 0; q--, X += SPLIT) {
        const float2 ex = X[0], ey = X[c2], ez = X[2 * c2], h2 = X[3 * c2], mh = X[4 * c2], mh3 = X[5 * c2];
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            const float2 dx = add2(ex, nx[s]), dy = add2(ey, ny[s]), dz = add2(ez, nz[s]);
            const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
            float2 u2 = mul2(r2, h2);
            u2 = make_float2(fmaxf(u2.x, 1e-36f), fmaxf(u2.y, 1e-36f));
            const float2 iu = make_float2(rsqrtf(u2.x), rsqrtf(u2.y));
            const float2 u = mul2(u2, iu), iu2 = mul2(iu, iu);
            // saturated above 1, where the Newtonian form is selected
            const float2 t = make_float2(__saturatef(u.x - 0.5f), __saturatef(u.y - 0.5f));
            const float2 t2 = mul2(t, t), t4u = mul2(mul2(t2, t2), iu);
            const float2 pin =
                fma2(u2, fma2(u2, fma2(u, dup2(6.4f), dup2(-9.6f)), dup2(5.333333333333f)), dup2(-2.8f));
            const float2 wp = fma2(mul2(t4u, t), fma2(t, dup2(-8.533333333333f), dup2(-6.4f)), pin);
            // spline for u = r/h_g < 1 (kernel.h:452-470), Newtonian beyond (:391-398);
            // the two meet at u = 1, where the spline's force factor is 1/u^3
            const bool sx = u.x < 1.f, sy = u.y < 1.f;
            float2 fp = sel2(sx, sy, wp, make_float2(-iu.x, -iu.y));
            if (!POT) {
                const float2 fin = fma2(u2, fma2(u, dup2(32.f), dup2(-38.4f)), dup2(10.666666666667f));
                const float2 out = fma2(t, fma2(t, dup2(-42.666666666667f), dup2(-51.2f)), dup2(-16.f));
                const float2 wf = fma2(mul2(t4u, iu2), out, fin);
                const float2 fac = mul2(mh3, sel2(sx, sy, wf, mul2(iu2, iu)));
                const bool ux = r2.x > 0.f, uy = r2.y > 0.f;
                fp = sel2(ux, uy, fp, dup2(0.f));
                T.self[s] += (ux ? 0 : 1) + (uy ? 0 : 1);
                px[s] = fma2(dx, fac, px[s]);
                py[s] = fma2(dy, fac, py[s]);
                pz[s] = fma2(dz, fac, pz[s]);
            }
            pp[s] = fma2(mh, fp, pp[s]);
        }
    }
    add_sums<TPL, POT>(T, px, py, pz, pp);
}

// The same for groups of several kernel radii, or of one that near_one_radius
// refuses: h_g is formed per pair from the entry's {h_source, 1/h_source, m}, and
// Newtonian pairs have no part of it (any distance whose m/r^3 is an FP32 number).
template <int TPL, int SPLIT, bool POT>
__device__ __forceinline__ void flush_near_mixed(const float *__restrict__ near, int n, int part, Targets<TPL> &T)
{
    float2 px[TPL], py[TPL], pz[TPL], pp[TPL], nx[TPL], ny[TPL], nz[TPL];
#pragma unroll
    for (int s = 0; s < TPL; s++) {
        px[s] = py[s] = pz[s] = pp[s] = dup2(0.f);
        nx[s] = dup2(-T.x[s]); ny[s] = dup2(-T.y[s]); nz[s] = dup2(-T.z[s]);
    }
    const float2 *X = reinterpret_cast<const float2 *>(near) + part;
    constexpr int c2 = NEAR_CAP / 2;
#pragma unroll 1
    for (int q = n / (2 * SPLIT); q > 0; q--, X += SPLIT) {
        const float2 ex = X[0], ey = X[c2], ez = X[2 * c2], hs = X[3 * c2], hsinv = X[4 * c2], em = X[5 * c2];
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            const float2 dx = add2(ex, nx[s]), dy = add2(ey, ny[s]), dz = add2(ez, nz[s]);
            const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
            const float2 hg = make_float2(fmaxf(T.h[s], hs.x), fmaxf(T.h[s], hs.y));
            // 1/h_g: the inverses are rounded alike
            const float2 hinv = make_float2(fminf(T.hinv[s], hsinv.x), fminf(T.hinv[s], hsinv.y));
            // finite at r = 0 when it counts
            const float2 rinv = make_float2(rsqrtf(POT ? fmaxf(r2.x, 1e-30f) : r2.x),
                                            rsqrtf(POT ? fmaxf(r2.y, 1e-30f) : r2.y));
            const float2 u = mul2(mul2(r2, rinv), hinv), iu = mul2(hg, rinv);
            float2 wp;
            const float2 wf = spline_wf2(u, iu, &wp);
            const bool sx = u.x < 1.f, sy = u.y < 1.f;
            const float2 mr = mul2(em, rinv);
            float2 fp = sel2(sx, sy, mul2(mul2(em, wp), hinv), make_float2(-mr.x, -mr.y));
            if (!POT) {
                float2 fac =
                    sel2(sx, sy, mul2(mul2(em, wf), mul2(mul2(hinv, hinv), hinv)), mul2(mr, mul2(rinv, rinv)));
                const bool ux = r2.x > 0.f, uy = r2.y > 0.f;
                fac = sel2(ux, uy, fac, dup2(0.f));
                fp = sel2(ux, uy, fp, dup2(0.f));
                T.self[s] += (ux ? 0 : 1) + (uy ? 0 : 1);
                px[s] = fma2(dx, fac, px[s]);
                py[s] = fma2(dy, fac, py[s]);
                pz[s] = fma2(dz, fac, pz[s]);
            }
            pp[s] = add2(pp[s], fp);
        }
    }
    add_sums<TPL, POT>(T, px, py, pz, pp);
}

// moves the r < 8 entries from m on to the front of a list of NA arrays (m >= 24)
template <int NA, int CAP>
__device__ __forceinline__ void list_shift(float *list, int m, int r, int lane)
{
    __syncwarp();
    if (lane < r) {
#pragma unroll
        for (int a = 0; a < NA; a++) list[a * CAP + lane] = list[a * CAP + m + lane];
    }
    __syncwarp();
}

// Softening record of a near-list entry with kernel radius hsrc and mass m (see
// flush_near).  hone: the group's one kernel radius, negative if it takes the form
// of several.  (A flag beside the radius cost the 16.8M walk 41.15 -> 41.82 ms.)
__device__ __forceinline__ float4 near_soft(float hsrc, float m, float hone)
{
    if (hone >= 0.f) {
        const float hinv = __frcp_rn(fmaxf(hone, hsrc)), mh = m * hinv;
        return make_float4(hinv * hinv, mh, mh * hinv * hinv, 0.f);
    }
    return make_float4(hsrc, hsrc > 0.f ? __frcp_rn(hsrc) : INFINITY, m, 0.f);
}

// Whether the near flush for one kernel radius h > 0 can take a group's
// records {h_g^-2, m/h_g, m/h_g^3}.  It forms Newtonian pairs from them too, by u =
// r/h_g, so the records must be finite, and u, which reaches 4 box half-widths hw
// over h, must have a u^3.  Other groups (unsoftened ones, radii tiny against the
// box or the mass M) take the form that has r and m themselves.
__device__ __forceinline__ bool near_one_radius(float h, float hw, float M)
{
    const float hinv = __frcp_rn(h);   // infinite for h = 0
    return h >= 1e-9f * hw && hinv * hinv < 1e37f && M * hinv * hinv * hinv < 1e37f;
}

__device__ __forceinline__ double warp_min_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(FULL, v, o));
    return v;
}
__device__ __forceinline__ double warp_max_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
    return v;
}
// one target's results: t its place in the target list, pi its sorted particle
template <bool POT>
__device__ __forceinline__ void write_target(const WalkParams &p, int t, int pi, float hinv, double ax, double ay,
                                             double az, double ph, int nint, float tcost)
{
    const unsigned li = p.perm[pi];
    const int o = p.tout ? p.tout[t] : (int)li;
    if (POT) {
        // compute_potential removes the self term m_i kernel(0) / h_i
        // (potential.c:137-145); subtract the FP32 value the walk added
        const float mi = p.parts[pi].m;
        p.pot[o] = ph - (double)((mi * -2.8f) * hinv);
    } else {
        p.acc[3 * (size_t)o] = ax;
        p.acc[3 * (size_t)o + 1] = ay;
        p.acc[3 * (size_t)o + 2] = az;
        if (p.pot) p.pot[o] = ph;
        if (p.oldacc_out) p.oldacc_out[li] = sqrt(ax * ax + ay * ay + az * az);
    }
    if (p.ninter) p.ninter[o] = nint;
    if (p.cost_out) p.cost_out[li] = tcost;
}

// ---- cut walks (see k_walk)
__device__ __forceinline__ int ld_flag(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_flag(int *p, int v)
{
    asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The next sub-walk for a warp that found no group left, or -1.  Sub-walks are
// numbered by cut; a warp takes the next number and waits until that cut is made or
// too few groups are unfinished for it.  All groups are held by running warps by
// then, so the wait ends; it is bounded all the same (some twenty seconds).
#define WALK_TASK_LIMIT (1 << 22)
__device__ __noinline__ int next_task(const WalkParams &p, int ngroups)
{
    const int t = atomicAdd(p.group_counter + WALK_TASK_COUNTER, 1), f = t / FORK_WALKS;
    if (f >= p.fork_max) return -1;
    unsigned ns = 256;
    for (int i = 0; i < WALK_TASK_LIMIT; i++) {
        // is a cut left for this number?  Each unfinished group makes one more at most
        const int *const done = p.group_counter + WALK_DONE_COUNTER, *const cuts = p.group_counter + WALK_FORK_COUNTER;
        bool over = f >= ld_flag(cuts) + (ngroups - ld_flag(done));
        if (over) {   // for certain: the finished groups first, then their cuts
            const int left = ngroups - ld_flag(done);
            __threadfence();
            over = f >= ld_flag(cuts) + left;
        }
        if (ld_flag(p.fork_ready + f)) {
            __threadfence();
            return t;
        }
        if (over) return -1;
        __nanosleep(ns);
        ns = min(2 * ns, 4096u);
    }
    atomicOr(p.err, GG_EBIT_WALK_TIMEOUT);
    return -1;
}

// The sums of a cut walk's parts, added in order, by one warp.
template <bool POT>
__device__ __noinline__ void join_cut(const WalkParams &p, const WalkFork *fork, int group, int lane)
{
    const GGGroup grp = p.groups[group];
    int mycount = 0;
    for (int slot = lane; slot < grp.count; slot += 32) {   // written by other warps of this launch: read through L2
        auto part = [](const double4 *q) {
            const double2 a = __ldcg(reinterpret_cast<const double2 *>(q)),
                          b = __ldcg(reinterpret_cast<const double2 *>(q) + 1);
            return make_double4(a.x, a.y, b.x, b.y);
        };
        double4 a = part(fork->sum0 + slot);
        int nint = __ldcg(fork->nint0 + slot);
        for (int i = 0; i < FORK_WALKS; i++) {
            const double4 q = part(fork->sum[i] + slot);
            a.x += q.x; a.y += q.y; a.z += q.z; a.w += q.w;
            nint += __ldcg(fork->nint[i] + slot);
        }
        const int t = grp.first + slot, pi = p.tlist ? p.tlist[t] : t;
        const float h = p.parts[pi].h;
        write_target<POT>(p, t, pi, h > 0.f ? __frcp_rn(h) : INFINITY, a.x, a.y, a.z, a.w, nint, __ldcg(&fork->cost));
        mycount += nint;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mycount += __shfl_xor_sync(FULL, mycount, o);
    if (lane == 0) atomicAdd(p.interactions, (unsigned long long)mycount);
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += y;
    }
    return v;
}
// F64T: opening tests in FP64 (used for one-target groups, where the tests are
// exactly the reference's); otherwise the tests run in FP32 on FP64-formed
// offsets from the group centre, against a bounding box rounded outwards.
template <int TPL, int SPLIT, bool F64T, bool POT, bool TMA, bool CUT>
__global__ void __launch_bounds__(WALK_THREADS, 2) k_walk(const __grid_constant__ WalkParams p)
{
    extern __shared__ float4 walk_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    constexpr int LP = 32 / SPLIT;   // lanes per part
    constexpr int QUANTUM = 4 * SPLIT;
    const int part = lane / LP;
    const int swz = TMA ? 0 : (lane >> 1) & 3;   // node slot pieces, see stage_lanes
    const int FL = min(p.flush, FAR_FLUSH_MAX), NL = min(p.flush, NEAR_FLUSH_MAX);
    float *far = reinterpret_cast<float *>(walk_smem) + (size_t)warp * WALK_WARP_FLOATS;
    float *near = far + FAR_ARRAYS * FAR_CAP;
    float *rest = near + NEAR_ARRAYS * NEAR_CAP;
    int *sstack = reinterpret_cast<int *>(rest);
    int4 *const nslot = reinterpret_cast<int4 *>(rest + WALK_SSTACK) + 4 * lane;
    const unsigned slot0 = (unsigned)__cvta_generic_to_shared(rest + WALK_SSTACK);
    int *run = reinterpret_cast<int *>(rest + WALK_SSTACK + NH * 32 * 16);   // see expand
    int *qbase = run + 32, *qend = qbase + RUNS;   // queued runs: first particle less its position, end position
    const unsigned bar = (unsigned)__cvta_generic_to_shared(qend + RUNS);
    // state of a cut walk (CUT): kept here, not in registers
    struct CutState { WalkFork *fork; int sub, npend, own, group, tasks, at; };
    CutState &cut = *reinterpret_cast<CutState *>(qend + RUNS + 4);
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (CUT) cut.own = cut.tasks = 0;
    }
    __syncwarp();
    unsigned phase = 0;   // parity of the barrier phase the next wait is for
    constexpr bool tma = TMA;   // node staging by bulk copies (else per-lane cp.async)
    int *gstack = p.stack + (size_t)(blockIdx.x * WALK_WARPS + warp) * p.stack_cap;
    const int ngroups = *p.nnodes ? *p.ngroups : 0;
    const double theta = p.theta;

    for (;;) {
        int g = 0;
        if (!CUT) {
            if (lane == 0) g = atomicAdd(p.group_counter, 1);
            g = __shfl_sync(FULL, g, 0);
            if (g >= ngroups) break;
            if (p.gorder) g = (int)p.gorder[g];
        } else {
            if (lane == 0) {
                if (cut.own && cut.sub < FORK_WALKS) {   // the warp's own next sub-walk
                    cut.sub++;
                    g = cut.group;
                } else if (cut.tasks || (g = atomicAdd(p.group_counter, 1)) >= ngroups) {
                    // groups have run out: sub-walks of cut ones
                    cut.tasks = 1;
                    const int t = next_task(p, ngroups);
                    if (t >= 0) {
                        WalkFork *const fork = p.forks + t / FORK_WALKS;
                        cut.fork = fork;
                        cut.sub = 1 + t % FORK_WALKS;
                        cut.npend = __ldcg(&fork->npend);
                        cut.group = __ldcg(&fork->group);
                        cut.own = 0;
                    }
                    g = t >= 0 ? cut.group : -1;
                } else {
                    if (p.gorder) g = (int)p.gorder[g];
                    cut.fork = nullptr;
                    cut.sub = cut.npend = cut.own = 0;
                    cut.group = g;
                }
            }
            g = __shfl_sync(FULL, g, 0);
            if (g < 0) break;
            __syncwarp();
        }
        const GGGroup grp = p.groups[g];
        const unsigned t_start = (unsigned)clock();
        // Long walks.  A group with far more work than most (a dense centre, a box
        // that reaches into one) would set the length of a walk that has only a few
        // groups per warp.  Once its work (node tests, list entries) reaches
        // p.fork_work the nodes still pending are dealt out to FORK_WALKS sub-walks
        // with sums of their own: tasks of the warps that have run out of groups, or,
        // when the records of cuts are used up, the same warp's next work.  The sums
        // are added in order either way, and whether and where a walk is cut depends on the group, its
        // system's size and the opening criterion alone, so a system's results do not
        // depend on what it is batched with.
        // ---- targets of the group
        Targets<TPL> T;
        double tx[TPL], ty[TPL], tz[TPL];
        double bmin[3] = {INFINITY, INFINITY, INFINITY}, bmax[3] = {-INFINITY, -INFINITY, -INFINITY};
        double aold_min = INFINITY;
        float hmin = INFINITY, hmax = 0.f;
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            int k = s * LP + lane % LP;
            bool v = k < grp.count;
            T.valid[s] = v;
            tx[s] = ty[s] = tz[s] = 0.0;
            T.h[s] = 0.f;
            T.hinv[s] = INFINITY;
            if (v) {
                int t = grp.first + k;
                int pi = p.tlist ? p.tlist[t] : t;
                GGPart q = load_part(p.parts + pi);
                tx[s] = q.x; ty[s] = q.y; tz[s] = q.z;
                T.h[s] = q.h;
                T.hinv[s] = q.h > 0.f ? __frcp_rn(q.h) : INFINITY;
                double oa = p.oldacc_in ? p.oldacc_in[p.perm[pi]] : 0.0;
                aold_min = fmin(aold_min, p.tol * oa);
                hmin = fminf(hmin, q.h);
                hmax = fmaxf(hmax, q.h);
                bmin[0] = fmin(bmin[0], q.x); bmax[0] = fmax(bmax[0], q.x);
                bmin[1] = fmin(bmin[1], q.y); bmax[1] = fmax(bmax[1], q.y);
                bmin[2] = fmin(bmin[2], q.z); bmax[2] = fmax(bmax[2], q.z);
            }
        }
        double cg[3], hw[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            bmin[q] = warp_min_d(bmin[q]);
            bmax[q] = warp_max_d(bmax[q]);
            cg[q] = 0.5 * (bmin[q] + bmax[q]);
            hw[q] = fmax(0.5 * (bmax[q] - bmin[q]), fmax(bmax[q] - cg[q], cg[q] - bmin[q]));
        }
        aold_min = warp_min_d(aold_min);
        if (CUT && lane == 0) {
            const int nt = p.toff[grp.sys + 1] - p.toff[grp.sys];
            // (sub-walks are not cut again; with an OldAcc of 0 every node is opened)
            const bool may = cut.sub == 0 && nt >= FORK_MIN_TARGETS && nt <= FORK_MAX_TARGETS &&
                             (theta > 0.0 || aold_min > 0.0);
            cut.at = !may ? INT_MAX : nt <= FORK_HALF_TARGETS ? p.fork_work / 2 : p.fork_work;
        }
        hmin = (float)warp_min_d((double)hmin);
        hmax = (float)warp_max_d((double)hmax);
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            T.x[s] = (float)(tx[s] - cg[0]);
            T.y[s] = (float)(ty[s] - cg[1]);
            T.z[s] = (float)(tz[s] - cg[2]);
        }
        const double hmaxd = (double)hmax, hmind = (double)hmin;
        const float hwf[3] = {__double2float_ru(hw[0]), __double2float_ru(hw[1]), __double2float_ru(hw[2])};
        const float aoldf = (float)aold_min, thetaf = (float)theta;
        const float hone = hmin == hmax && near_one_radius(hmax, fmaxf(hwf[0], fmaxf(hwf[1], hwf[2])),
                                                           p.nodes[grp.root].mass) ? hmax : -1.f;   // warp-uniform

        // ---- traversal
        // Each round tests up to 32 NH nodes, NH per lane.  The next round's nodes
        // are the last of {node stack, children of this round's opened
        // nodes}; only what is left over goes to the stack, which lives in shared
        // memory (sp entries) on top of a spill area in global memory (gsp
        // entries).  Their records are staged (cp.async) before this round's leaf
        // particles and list flushes are processed, and a batch of particle
        // records is in flight during the tests.  One loop does whatever is due,
        // so that every part appears in the code once (the kernel is large
        // against the instruction cache).
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            T.self[s] = 0;
            T.ax[s] = {0.f, 0.f}; T.ay[s] = {0.f, 0.f}; T.az[s] = {0.f, 0.f}; T.pot[s] = {0.f, 0.f};
        }
        int sp = 0, gsp = 0, nf = 0, nn = 0;
        int qhead = 0, qtail = 0;     // runs of particles in the queue
        int pw = 0, pt = 0;           // positions of the queue's particles: next, end
        int list_far = 0, list_near = 0, tested = 0;   // warp-uniform statistics of this group
        int limit = FL, nlimit = NL;  // the lists are flushed at these lengths; 1 once the traversal is over
        bool overflow = false, timed_out = false;
        int k = 1;                    // nodes staged for the next round
        auto stage = [&](const int (&node)[NH], int kn) {
            if (kn == 0) return;
            if (tma) stage_nodes(bar, slot0, p.nodes, node, kn, lane);   // one barrier phase per staged round
            else stage_lanes(slot0, p.nodes, node, kn, lane);
        };
        {
            int node[NH];
            node[0] = lane == 0 ? grp.root : -1;
            if (CUT && cut.sub > 0) {   // every FORK_WALKS-th pending node: at most FORK_PENDING / FORK_WALKS
                const int sub = cut.sub, m = (cut.npend - sub + FORK_WALKS) / FORK_WALKS;
                for (int i = lane; i < m; i += 32) sstack[i] = __ldcg(cut.fork->pending + sub - 1 + FORK_WALKS * i);
                __syncwarp();
                k = min(m, 32 * NH);
                sp = m - k;
#pragma unroll
                for (int h = 0; h < NH; h++) node[h] = 32 * h + lane < k ? sstack[sp + 32 * h + lane] : -1;
            }
            stage(node, k);
        }
        // appends one entry per lane with `use`: to the far list, or to the near list with its softening
        auto append = [&](bool use, bool isfar, const float4 &e, float h) {
            const unsigned mu = __ballot_sync(FULL, use), mf = __ballot_sync(FULL, use && isfar), mn = mu & ~mf;
            if (use && isfar) list_put(far, nf + __popc(mf & lt_mask), e);
            if (mn) {   // warp-uniform
                if (use && !isfar) near_put(near, nn + __popc(mn & lt_mask), e, near_soft(h, e.w, hone));
                nn += __popc(mn);
                list_near += __popc(mn);
            }
            nf += __popc(mf);
            list_far += __popc(mf);
        };
        // Runs of consecutive indices laid end to end: a run maps its positions q
        // to base + q.  The lane that owns a run's first position in a window of 32
        // has stored its base at run[position] and set its bit; each lane then looks
        // back to the nearest such position.  Returns the index at the lane's
        // position, or -1 before the first run.  (Conversions, population counts
        // and bit searches run at a quarter of the rate of other integer work, in
        // the pipe that the flushes' rsqrt needs: one search per window, instead of
        // counts per bit of the run lengths.)
        auto lookup = [&](unsigned bits, int w) -> int {
            const unsigned starts = __reduce_or_sync(FULL, bits) & (lt_mask | (1u << lane));
            __syncwarp();
            const int index = starts ? run[31 - __clz((int)starts)] + w + lane : -1;
            __syncwarp();   // the next window writes run
            return index;
        };
        // the lane's NH runs of positions beg to end - 1; the window starts at position w
        auto expand = [&](const int (&base)[NH], const int (&beg)[NH], const int (&end)[NH], int w) -> int {
            unsigned bits = 0;
#pragma unroll
            for (int h = 0; h < NH; h++) {
                const int d = max(beg[h] - w, 0);
                if (end[h] > w && d < 32 && end[h] > beg[h]) {
                    run[d] = base[h];
                    bits |= 1u << d;
                }
            }
            return lookup(bits, w);
        };
        for (;;) {
            // ---- full lists: their whole quanta are evaluated, the rest moves to the front
            if (nf >= limit) {
                const int m = nf & ~(QUANTUM - 1);
                __syncwarp();
                flush_far<TPL, SPLIT, POT>(far, m, part, T);
                nf -= m;
                list_shift<FAR_ARRAYS, FAR_CAP>(far, m, nf, lane);
            }
            if (nn >= nlimit) {
                const int m = nn & ~(QUANTUM - 1);
                __syncwarp();
                if (hone >= 0.f) flush_near<TPL, SPLIT, POT, CUT && SPLIT == 1 ? 1 : 2>(near, m, part, T);
                else flush_near_mixed<TPL, SPLIT, POT>(near, m, part, T);
                nn -= m;
                list_shift<NEAR_ARRAYS, NEAR_CAP>(near, m, nn, lane);
            }
            // ---- the next 32 queued particles, one per lane: their records are loaded here and used below
            const bool batch = pt - pw >= 32 || (pt > pw && k == 0);
            GGPart pp;
            bool have = false;
            if (batch) {
                const int m = min(32, pt - pw);
                const bool queued = qhead + lane < qtail;
                const int slot = (qhead + lane) & (RUNS - 1);
                const int end = queued ? qend[slot] - pw : INT_MAX;   // runs are not empty: 32 of them suffice
                int d = __shfl_up_sync(FULL, end, 1);
                if (lane == 0) d = 0;
                unsigned bits = 0;
                if (queued && d < 32) {
                    run[d] = qbase[slot];
                    bits = 1u << d;
                }
                const int i = lookup(bits, pw);
                have = lane < m;
                if (have) pp = load_part(p.parts + i);
                pw += m;
                qhead += __popc(__ballot_sync(FULL, end <= m));
            }
            // ---- a round of node tests
            if (k > 0 && pt - pw < 32) {
                tested += k;
                if (tma) {
                    if (!bar_wait(bar, phase)) {
                        timed_out = true;
                        break;
                    }
                    phase ^= 1u;
                } else {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncwarp();   // other lanes' copies too
                }
                int na[NH], nc[NH], np[NH];
                float4 ent[NH];
                float soft[NH];
                bool used[NH], isfar[NH];
#pragma unroll
                for (int h = 0; h < NH; h++) {
                    na[h] = nc[h] = np[h] = 0;
                    ent[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                    soft[h] = 0.f;
                    used[h] = isfar[h] = false;
                    if (k <= 32 * h) continue;   // warp-uniform
                    GGNode nd;
#pragma unroll
                    for (int i = 0; i < 4; i++) reinterpret_cast<int4 *>(&nd)[i] = nslot[32 * 4 * h + (i ^ swz)];
                    const int nb = nd.b;
                    const float ms = nd.maxsoft, L = nd.len;
                    bool open;
                    if (!F64T) {
                        const float dx = (float)(nd.cx - cg[0]), dy = (float)(nd.cy - cg[1]),
                                    dz = (float)(nd.cz - cg[2]);
                        const float ex = fmaxf(fabsf(dx) - hwf[0], 0.f), ey = fmaxf(fabsf(dy) - hwf[1], 0.f),
                                    ez = fmaxf(fabsf(dz) - hwf[2], 0.f);
                        const float r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                        const float hh = fmaxf(hmax, ms);
                        if (thetaf > 0.f) {
                            open = ((hmin < ms) && (r2 < ms * ms)) || (L * L > r2 * thetaf * thetaf);
                        } else {
                            // r < soft + 0.6 len for the larger of the two softenings, which
                            // also covers r < maxsoft
                            const float a1 = fmaf(0.6f, L, hh);
                            open = (r2 < a1 * a1) | (nd.mass * L * L > r2 * r2 * aoldf) |
                                   ((fabsf(dx + nd.gx) < fmaf(0.6f, L, hwf[0])) &
                                    (fabsf(dy + nd.gy) < fmaf(0.6f, L, hwf[1])) &
                                    (fabsf(dz + nd.gz) < fmaf(0.6f, L, hwf[2])));
                        }
                        ent[h] = make_float4(dx, dy, dz, nd.mass);
                        isfar[h] = (r2 >= hh * hh) && (r2 > FAR_MIN_R2);
                    } else {
                        const double dx = nd.cx - cg[0], dy = nd.cy - cg[1], dz = nd.cz - cg[2];
                        const double ex = fmax(fabs(dx) - hw[0], 0.0), ey = fmax(fabs(dy) - hw[1], 0.0),
                                     ez = fmax(fabs(dz) - hw[2], 0.0);
                        const double r2 = ex * ex + ey * ey + ez * ez;
                        const double msd = (double)ms, Ld = (double)L;
                        open = (hmind < msd) && (r2 < msd * msd);
                        if (!open) {
                            if (theta > 0.0) {
                                open = Ld * Ld > r2 * theta * theta;
                            } else {
                                const double a1 = hmaxd + 0.6 * Ld, a2 = msd + 0.6 * Ld;
                                open = (r2 < a1 * a1) || (r2 < a2 * a2) ||
                                       ((double)nd.mass * Ld * Ld > r2 * r2 * aold_min);
                                if (!open) {
                                    const double gx = fabs(dx + (double)nd.gx), gy = fabs(dy + (double)nd.gy),
                                                 gz = fabs(dz + (double)nd.gz);
                                    open = (gx < 0.6 * Ld + hw[0]) && (gy < 0.6 * Ld + hw[1]) &&
                                           (gz < 0.6 * Ld + hw[2]);
                                }
                            }
                        }
                        ent[h] = make_float4((float)dx, (float)dy, (float)dz, nd.mass);
                        const double hh = fmax(hmaxd, msd);
                        isfar[h] = (r2 >= hh * hh) && (r2 > (double)FAR_MIN_R2);
                    }
                    const bool some = 32 * h + lane < k && nd.mass > 0.f;   // massless nodes are skipped
                    open = open || nb == -1;                                // one particle: always opened
                    used[h] = some && !open;
                    soft[h] = ms;
                    na[h] = nd.a;
                    nc[h] = some && open ? max(nb, 0) : 0;    // children of an opened node
                    np[h] = some && open ? max(-nb, 0) : 0;   // particles of an opened leaf
                }
#pragma unroll
                for (int h = 0; h < NH; h++) append(used[h], isfar[h], ent[h], soft[h]);
                // the opened nodes' children (particles) laid end to end over the warp, from one scan of both counts
                int cl = 0, pl = 0;   // this lane's
#pragma unroll
                for (int h = 0; h < NH; h++) { cl += nc[h]; pl += np[h]; }
                int cend, ctot, pend;
                int ptot;
                if (__any_sync(FULL, pl > 1023)) {   // an unsplit leaf at the depth limit
                    cend = warp_incl_scan(cl, lane);
                    pend = warp_incl_scan(pl, lane);
                    ctot = __shfl_sync(FULL, cend, 31);
                    ptot = __shfl_sync(FULL, pend, 31);
                } else {
                    const int both = warp_incl_scan(cl | (pl << 16), lane), sum = __shfl_sync(FULL, both, 31);
                    cend = both & 0xffff;
                    pend = both >> 16;
                    ctot = sum & 0xffff;
                    ptot = sum >> 16;
                }
                int cbase[NH], cbeg[NH], cfin[NH];
                int c = cend - cl, q = pt + pend - pl;
#pragma unroll
                for (int h = 0; h < NH; h++) {
                    cbase[h] = na[h] - c;
                    cbeg[h] = c;
                    c += nc[h];
                    cfin[h] = c;
                }
                if (ptot > 0) {   // the opened leaves' runs join the queue, in the order of their positions
                    int slot = qtail;
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        const unsigned ml = __ballot_sync(FULL, np[h] > 0);
                        slot += __popc(ml & lt_mask);
                        qtail += __popc(ml);
                    }
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        if (np[h] > 0) {
                            qbase[slot & (RUNS - 1)] = na[h] - q;
                            q += np[h];
                            qend[slot & (RUNS - 1)] = q;
                            slot++;
                        }
                    }
                    pt += ptot;
                }
                if (sp == 0 && ctot == 0 && gsp > 0) {   // refill from the spill area, keeping stack order
                    const int m = min(gsp, WALK_SSTACK / 2);
                    for (int i = lane; i < m; i += 32) sstack[i] = gstack[gsp - m + i];
                    gsp -= m;
                    sp = m;
                }
                __syncwarp();
                k = min(sp + ctot, 32 * NH);
                const int w0 = ctot - k;   // first position taken now; negative: from the stack
                int node[NH];
#pragma unroll
                for (int h = 0; h < NH; h++) {
                    const int w = w0 + 32 * h;
                    node[h] = -1;
                    if (w + 32 > 0 && w < ctot) node[h] = expand(cbase, cbeg, cfin, w);
                    if (w + lane < 0) node[h] = sstack[sp + w + lane];
                }
                sp += min(w0, 0);
                // (only where all children are among the next nodes: then those, in registers, and the
                // stack are all that is pending)
                if (CUT && tested + list_far + 3 * list_near >= cut.at && w0 <= 0 && gsp + sp + k >= 2 * FORK_WALKS &&
                    gsp + sp + k <= FORK_PENDING) {
                    int f = 0;
                    if (lane == 0) f = atomicAdd(p.group_counter + WALK_FORK_COUNTER, 1);
                    f = __shfl_sync(FULL, f, 0);
                    const bool own = f >= p.fork_max;
                    WalkFork *const fork =
                        own ? reinterpret_cast<WalkFork *>(p.own_forks + (size_t)(blockIdx.x * WALK_WARPS + warp) *
                                                                             FORK_OWN_BYTES)
                            : p.forks + f;
                    for (int i = lane; i < gsp; i += 32) fork->pending[i] = gstack[i];
                    for (int i = lane; i < sp; i += 32) fork->pending[gsp + i] = sstack[i];
#pragma unroll
                    for (int h = 0; h < NH; h++)
                        if (32 * h + lane < k) fork->pending[gsp + sp + 32 * h + lane] = node[h];
                    __syncwarp();
                    if (lane == 0) {
                        fork->group = cut.group;
                        fork->npend = gsp + sp + k;
                        cut.fork = fork;
                        cut.npend = gsp + sp + k;
                        cut.own = own;
                        if (!own) {   // the record is complete: tasks may start
                            __threadfence();
                            st_flag(p.fork_ready + f, 1);
                        }
                    }
                    gsp = sp = k = 0;   // the rest of this part: queued particles and lists
                    __syncwarp();
                }
                stage(node, k);
                if (w0 > 0) {   // the other children go to the stack
                    while (sp + w0 > WALK_SSTACK) {   // up to half of it spills to global memory, oldest first (w0 < WALK_SSTACK)
                        const int m = min(sp, WALK_SSTACK / 2);
                        if (gsp + m > p.stack_cap) {
                            overflow = true;
                            break;
                        }
                        for (int i = lane; i < m; i += 32) gstack[gsp + i] = sstack[i];
                        __syncwarp();
                        for (int i = lane; i < sp - m; i += 32) sstack[i] = sstack[m + i];   // sp - m <= m: no overlap
                        __syncwarp();
                        gsp += m;
                        sp -= m;
                    }
                    if (overflow) break;
                    for (int w = 0; w < w0; w += 32) {
                        const int c = expand(cbase, cbeg, cfin, w);
                        if (w + lane < w0) sstack[sp + w + lane] = c;
                    }
                    sp += w0;
                }
                __syncwarp();   // stack and queued runs are read by other lanes next
            } else if (!batch) {
                if (limit == 1) break;
                // the traversal is over: the lists' last, partial quanta are filled with massless entries
                const int fe = (nf + QUANTUM - 1) & ~(QUANTUM - 1), ne = (nn + QUANTUM - 1) & ~(QUANTUM - 1);
                __syncwarp();
                if (nf + lane < fe) list_put(far, nf + lane, PAD_ENTRY);
                if (nn + lane < ne) near_put(near, nn + lane, PAD_ENTRY, PAD_SOFT);
                nf = fe;
                nn = ne;
                limit = nlimit = 1;
                continue;
            }
            if (batch) {   // the batch's particles are classified against the group box
                bool use = false, pfar = false;
                float4 pe = make_float4(0.f, 0.f, 0.f, 0.f);
                float ph = 0.f;
                if (have) {
                    const float dx = (float)(pp.x - cg[0]), dy = (float)(pp.y - cg[1]), dz = (float)(pp.z - cg[2]);
                    const float ex = fmaxf(fabsf(dx) - hwf[0], 0.f), ey = fmaxf(fabsf(dy) - hwf[1], 0.f),
                                ez = fmaxf(fabsf(dz) - hwf[2], 0.f);
                    const float r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                    const float hh = fmaxf(hmax, pp.h);
                    pe = make_float4(dx, dy, dz, pp.m);
                    ph = pp.h;
                    use = pp.m > 0.f;
                    pfar = (r2 >= hh * hh) && (r2 > FAR_MIN_R2);
                }
                append(use, pfar, pe, ph);
            }
        }
        if (!tma) asm volatile("cp.async.wait_all;" ::: "memory");   // no copy into the slot outlives its group
        if (timed_out) {   // copies may still be in flight: wait once more, then leave
            if (lane == 0) {
                atomicOr(p.err, GG_EBIT_WALK_TIMEOUT);
                if (CUT && !cut.tasks) atomicAdd(p.group_counter + WALK_DONE_COUNTER, 1);
            }
            bar_wait(bar, phase);
            return;
        }
        if (overflow) {
            if (tma && !bar_wait(bar, phase)) {   // the copies staged for a round that will not run
                if (lane == 0) {
                    atomicOr(p.err, GG_EBIT_WALK_TIMEOUT);
                    if (CUT && !cut.tasks) atomicAdd(p.group_counter + WALK_DONE_COUNTER, 1);
                }
                return;
            }
            if (tma) phase ^= 1u;
            if (lane == 0) {
                atomicOr(p.err, GG_EBIT_STACK_OVERFLOW);
                if (CUT && !cut.tasks) atomicAdd(p.group_counter + WALK_DONE_COUNTER, 1);
                if (CUT) cut.own = 0;
            }
            __syncwarp();
            continue;   // to the next group
        }
        __syncwarp();   // the next group's entries overwrite the lists

        // ---- results
        // this group's device cycles per target: the cost the next walk orders its groups
        // by (from 32 bits: a walk beyond two seconds only loses its place)
        const float tcost = (float)((unsigned)clock() - t_start) / (float)grp.count;
        int mycount = 0;
#pragma unroll
        for (int s = 0; s < TPL; s++) {
            double ax = 0.0, ay = 0.0, az = 0.0;
            if (!POT) { ax = T.ax[s].value(); ay = T.ay[s].value(); az = T.az[s].value(); }
            double ph = T.pot[s].value();
            int self = T.self[s];
#pragma unroll
            for (int o = LP; o < 32; o <<= 1) {   // the parts' shares of the lists
                if (!POT) {
                    ax += __shfl_xor_sync(FULL, ax, o);
                    ay += __shfl_xor_sync(FULL, ay, o);
                    az += __shfl_xor_sync(FULL, az, o);
                }
                ph += __shfl_xor_sync(FULL, ph, o);
                self += __shfl_xor_sync(FULL, self, o);
            }
            if (!T.valid[s] || (SPLIT > 1 && part != s)) continue;   // part s writes target s
            int nint = list_far + list_near - self;
            const int slot = s * LP + lane % LP;
            if (CUT && cut.fork) {
                WalkFork *const fork = cut.fork;
                const int sub = cut.sub;
                const bool own = cut.own;
                if (own && sub > 0) {   // the sums so far
                    const double4 q = fork->sum0[slot];
                    ax = q.x + ax; ay = q.y + ay; az = q.z + az; ph = q.w + ph;
                    nint += fork->nint0[slot];
                }
                if (!own || sub < FORK_WALKS) {
                    const bool first = own || sub == 0;
                    double4 *const sum = first ? fork->sum0 : fork->sum[sub - 1];
                    int *const cnt = first ? fork->nint0 : fork->nint[sub - 1];
                    sum[slot] = make_double4(ax, ay, az, ph);
                    cnt[slot] = nint;
                    if (sub == 0 && slot == 0) fork->cost = tcost;
                    continue;
                }
            }
            const int tt = grp.first + slot;   // (looked up again: a register less through the walk)
            write_target<POT>(p, tt, p.tlist ? p.tlist[tt] : tt, T.hinv[s], ax, ay, az, ph, nint, tcost);
            mycount += nint;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mycount += __shfl_xor_sync(FULL, mycount, o);
        if (lane == 0) {
            atomicAdd(p.interactions, (unsigned long long)mycount);
            atomicAdd(p.interactions + 1, (unsigned long long)list_far);
            atomicAdd(p.interactions + 2, (unsigned long long)list_near);
            atomicAdd(p.interactions + 3, (unsigned long long)tested);
        }
        if (CUT) {
            __syncwarp();   // also before lane 0 goes on to the next sub-walk
            int last = 0;
            if (lane == 0) {
                if (cut.fork) __threadfence();
                if (cut.fork && !cut.own) last = atomicAdd(p.fork_parts + (cut.fork - p.forks), 1) == FORK_WALKS;
                if (!cut.tasks && (!cut.own || cut.sub == FORK_WALKS))
                    atomicAdd(p.group_counter + WALK_DONE_COUNTER, 1);
                if (last) __threadfence();
            }
            // the last part of a cut walk to finish adds them all up
            if (__shfl_sync(FULL, last, 0)) join_cut<POT>(p, cut.fork, cut.group, lane);
        }
    }
}

template <int TPL, int SPLIT, bool F64T, bool POT, bool TMA, bool CUT>
static void launch_walk_c(const WalkParams &p, int blocks, cudaStream_t st)
{
    const int smem = WALK_WARPS * WALK_WARP_FLOATS * (int)sizeof(float);
    cudaFuncSetAttribute(k_walk<TPL, SPLIT, F64T, POT, TMA, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_walk<TPL, SPLIT, F64T, POT, TMA, CUT><<<blocks, WALK_THREADS, smem, st>>>(p);
    gg_note_launches(1);
}

// Walks that may be cut run a kernel of their own: the state of a cut costs
// registers and about 8% of a short walk (Plummer 300,000 0.59 -> 0.64 ms); it gains
// where few long walks end last (galaxy 300,000 2.4 -> 1.5 ms).
template <int TPL, int SPLIT, bool F64T, bool POT, bool TMA>
static void launch_walk_t(const WalkParams &p, int blocks, cudaStream_t st)
{
    if (!F64T && p.may_fork) launch_walk_c<TPL, SPLIT, F64T, POT, TMA, !F64T>(p, blocks, st);
    else launch_walk_c<TPL, SPLIT, F64T, POT, TMA, false>(p, blocks, st);
}

// The persistent grid is blocks_per_sm (1 or 2) blocks per SM.
void gg_launch_walk(const WalkParams &p, int blocks_per_sm, cudaStream_t st)
{
    const int blocks = gg_num_sms() * blocks_per_sm;
    const bool wide = p.group_size > 32, bulk = p.node_staging == 1;
    if (p.group_size == 1) {   // exact mode: the reference's tests
        if (p.pot_only) launch_walk_t<1, 1, true, true, false>(p, blocks, st);
        else launch_walk_t<1, 1, true, false, false>(p, blocks, st);
    } else if (p.pot_only) {
        if (wide) launch_walk_t<2, 1, false, true, false>(p, blocks, st);
        else launch_walk_t<2, 2, false, true, false>(p, blocks, st);
    } else if (bulk) {
        if (wide) launch_walk_t<2, 1, false, false, true>(p, blocks, st);
        else launch_walk_t<2, 2, false, false, true>(p, blocks, st);
    } else {
        if (wide) launch_walk_t<2, 1, false, false, false>(p, blocks, st);
        else launch_walk_t<2, 2, false, false, false>(p, blocks, st);
    }
}
