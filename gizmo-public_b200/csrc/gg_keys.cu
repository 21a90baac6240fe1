// gg_keys.cu -- root cube per system and 63-bit Peano-Hilbert keys.
//
// domain_findExtent (domain.c:2518-2570): FP64 min/max per axis, cube side
// len = 1.001 * max extent, centre = bbox middle, corner = centre - len/2.
// Keys: domain_double_to_int (domain.c:2504-2513) at 21 bits per dimension,
// then the Peano-Hilbert key (system/peano.c:303-319).  At 21 bits the key is
// exactly the reference's 42-bit key shifted right by 63 bits, because the
// reference's key is built most-significant level first.
#include <algorithm>

#include "gg_internal.cuh"
#include "gg_ph_table.h"
#include "gg_kernels.cuh"

__device__ __forceinline__ int gg_sys_of(const int *__restrict__ poff, int S, int i)
{
    // largest s with poff[s] <= i
    int lo = 0, hi = S - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(poff + mid) <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Root cube of one system from its min/max, with the reference's expressions.
__device__ __forceinline__ GGDomainDev extent_domain(const unsigned long long *mm)
{
    double mn[3], mx[3], len = 0;
    for (int k = 0; k < 3; k++) {
        mn[k] = gg_ordered_to_dbl(~__ldcg(mm + k));
        mx[k] = gg_ordered_to_dbl(__ldcg(mm + 3 + k));
        if (!(mn[k] <= mx[k])) { mn[k] = 0; mx[k] = 0; }   // empty system
    }
    for (int k = 0; k < 3; k++) {
        double e = __dsub_rn(mx[k], mn[k]);
        if (e > len) len = e;
    }
    len = __dmul_rn(len, 1.001);
    if (len <= 0) len = 1.0;   // a single particle or empty system: any cube works
    GGDomainDev d;
    for (int k = 0; k < 3; k++) {
        double mid = __dmul_rn(0.5, __dadd_rn(mn[k], mx[k]));
        d.center[k] = mid;
        d.corner[k] = __dsub_rn(mid, __dmul_rn(0.5, len));
    }
    d.len = len;
    d.pad = 0;
    return d;
}

// Each warp reduces a contiguous chunk of particles, reading it coalesced
// (lane l takes every 32nd record), one system segment at a time, and flushes
// the segment's extremes with 64-bit atomics on an order-preserving encoding:
// order-independent, so the result is exact and deterministic.  mm[8 s ..]:
// system s's complemented min x, y, z, max x, y, z, complemented min h and max h
// (kernel radii are not negative: their bit patterns are ordered), all from
// zero, so that one memset prepares every one.  The block that finishes last
// (`done` counts them) forms the root cubes and the ranges of kernel radii of up to
// ROOTS_ONE_BLOCK systems: one launch instead of three.
// With more systems one block is a serial tail, and a launch over the systems
// forms them.  Keys stage, one block / launch, us: 1 system 17.7 / 20.9, 256 22.1 /
// 23.8, 512 25.0 / 24.2, 4,096 60 / 34, 100,000 888 / 172, 1,000,000 8,557 / 1,287.
#define ROOTS_ONE_BLOCK 256

// root cube and range of kernel radii of system s from its extremes
__device__ __forceinline__ void extent_root(int s, const unsigned long long *mm, unsigned *hmm, GGDomainDev *dom)
{
    dom[s] = extent_domain(mm + 8 * (size_t)s);
    const unsigned long long lo = ~__ldcg(mm + 8 * (size_t)s + 6);
    hmm[2 * s] = lo >> 32 ? 0x7f800000u : (unsigned)lo;   // infinite for an empty system
    hmm[2 * s + 1] = (unsigned)__ldcg(mm + 8 * (size_t)s + 7);
}

__global__ void k_extent_roots(int S, const unsigned long long *mm, unsigned *hmm, GGDomainDev *dom)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < S) extent_root(s, mm, hmm, dom);
}

__global__ void k_extent(const GGPart *__restrict__ rec, int n, const int *__restrict__ poff, int S, int chunk,
                         unsigned long long *mm, unsigned *done, unsigned *hmm, GGDomainDev *dom, int *err)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    bool bad = false;
    for (long long c0 = (long long)warp * chunk; c0 < n; c0 += (long long)nwarps * chunk) {
        const int cb = (int)c0, ce = (int)min((long long)n, c0 + chunk);
        int s = gg_sys_of(poff, S, cb);
        for (int seg = cb; seg < ce; s++) {
            const int se = min(ce, __ldg(poff + s + 1));
            double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
            float hmin = INFINITY, hmax = 0.f;
            for (int i = seg + lane; i < se; i += 32) {
                GGPart p = rec[i];
                double v[3] = {p.x, p.y, p.z};
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (!isfinite(v[k])) bad = true;
                    mn[k] = fmin(mn[k], v[k]);
                    mx[k] = fmax(mx[k], v[k]);
                }
                hmin = fminf(hmin, p.h);
                hmax = fmaxf(hmax, p.h);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    mn[k] = fmin(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
                    mx[k] = fmax(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
                }
                hmin = fminf(hmin, __shfl_xor_sync(0xffffffffu, hmin, o));
                hmax = fmaxf(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
            }
            if (lane < 8 && se > seg) {   // one of the eight extremes each
                unsigned long long v;
                if (lane < 3) v = ~gg_dbl_to_ordered(lane == 0 ? mn[0] : lane == 1 ? mn[1] : mn[2]);
                else if (lane < 6) v = gg_dbl_to_ordered(lane == 3 ? mx[0] : lane == 4 ? mx[1] : mx[2]);
                else if (lane == 6) v = ~(unsigned long long)__float_as_uint(fmaxf(hmin, 0.f));
                else v = __float_as_uint(fmaxf(hmax, 0.f));
                atomicMax(mm + 8 * (size_t)s + lane, v);
            }
            seg = se;
        }
    }
    if (bad) atomicOr(err, GG_EBIT_BAD_INPUT);
    if (S > ROOTS_ONE_BLOCK) return;
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int s = threadIdx.x; s < S; s += blockDim.x) extent_root(s, mm, hmm, dom);
}

// 21 levels: the top one from the one-level table, then ten steps of two
// levels each from the two-level table (half the dependent table reads)
__device__ __forceinline__ unsigned long long gg_ph_key21(unsigned x, unsigned y, unsigned z,
                                                          const unsigned short *tab, const unsigned short *tab2)
{
    const int top = GG_MAX_LEVEL - 1;
    unsigned pix = (((x >> top) & 1u) << 2) | (((y >> top) & 1u) << 1) | ((z >> top) & 1u);
    unsigned e = tab[pix];   // state 0
    unsigned long long key = e & 7u;
    unsigned state = e >> 3;
#pragma unroll
    for (int lev = top - 1; lev > 0; lev -= 2) {
        const unsigned hi = (((x >> lev) & 1u) << 2) | (((y >> lev) & 1u) << 1) | ((z >> lev) & 1u);
        const unsigned lo = (((x >> (lev - 1)) & 1u) << 2) | (((y >> (lev - 1)) & 1u) << 1) | ((z >> (lev - 1)) & 1u);
        e = tab2[state * 64 + ((hi << 3) | lo)];
        key = (key << 6) | (e & 63u);
        state = e >> 6;
    }
    return key;
}

// keys + identity values for the sort; positions must lie in [corner, corner+len)
__global__ void k_keys(const GGPart *__restrict__ rec, int n, const int *__restrict__ poff, int S,
                       const GGDomainDev *__restrict__ dom, unsigned long long *keys, unsigned *vals, int *err)
{
    __shared__ unsigned short tab[GG_PH_NSTATES * 8], tab2[GG_PH_NSTATES * 64];
    for (int i = threadIdx.x; i < GG_PH_NSTATES * 8; i += blockDim.x) tab[i] = GG_PH_TABLE_INIT[i];
    for (int i = threadIdx.x; i < GG_PH_NSTATES * 64; i += blockDim.x) tab2[i] = GG_PH_TABLE2_INIT[i];
    __syncthreads();
    bool bad = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int s = (S == 1) ? 0 : gg_sys_of(poff, S, i);
        GGDomainDev d = dom[s];
        GGPart p = rec[i];
        double v[3] = {p.x, p.y, p.z};
        unsigned q[3];
        for (int k = 0; k < 3; k++) {
            double f = __dadd_rn(__ddiv_rn(__dsub_rn(v[k], d.corner[k]), d.len), 1.0);
            if (!(f >= 1.0 && f < 2.0)) { bad = true; f = fmin(fmax(f, 1.0), 1.9999999999999998); }
            unsigned long long u = (unsigned long long)__double_as_longlong(f);
            q[k] = (unsigned)((u & 0xFFFFFFFFFFFFFull) >> (52 - GG_MAX_LEVEL));
        }
        keys[i] = gg_ph_key21(q[0], q[1], q[2], tab, tab2);
        vals[i] = (unsigned)i;
    }
    if (bad) atomicOr(err, GG_EBIT_BAD_INPUT);
}

// keys of plain (n x 3) FP64 positions in one cube: the kernel-level entry point
__global__ void k_keys_plain(const double *__restrict__ pos, long long n, GGDomainDev d, unsigned long long *keys,
                             int *err)
{
    __shared__ unsigned short tab[GG_PH_NSTATES * 8], tab2[GG_PH_NSTATES * 64];
    for (int i = threadIdx.x; i < GG_PH_NSTATES * 8; i += blockDim.x) tab[i] = GG_PH_TABLE_INIT[i];
    for (int i = threadIdx.x; i < GG_PH_NSTATES * 64; i += blockDim.x) tab2[i] = GG_PH_TABLE2_INIT[i];
    __syncthreads();
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        unsigned q[3];
        for (int k = 0; k < 3; k++) {
            double f = __dadd_rn(__ddiv_rn(__dsub_rn(pos[3 * i + k], d.corner[k]), d.len), 1.0);
            if (!(f >= 1.0 && f < 2.0)) { bad = true; f = fmin(fmax(f, 1.0), 1.9999999999999998); }
            unsigned long long u = (unsigned long long)__double_as_longlong(f);
            q[k] = (unsigned)((u & 0xFFFFFFFFFFFFFull) >> (52 - GG_MAX_LEVEL));
        }
        keys[i] = gg_ph_key21(q[0], q[1], q[2], tab, tab2);
    }
    if (bad && err) atomicOr(err, GG_EBIT_BAD_INPUT);
}

size_t gg_extent_words(int S) { return 8 * (size_t)S + 1; }

void gg_launch_extent(const GGPart *rec, int n, const int *poff, int S, unsigned long long *mm, unsigned *hmm,
                      GGDomainDev *dom, int *err, cudaStream_t st)
{
    cudaMemsetAsync(mm, 0, gg_extent_words(S) * sizeof(*mm), st);
    // particles per warp: small systems spread over the SMs (65,536 particles in
    // chunks of 4,096 used 16 warps, 39 us; in chunks of 128, 5 us), large ones
    // flush to the same few words less often
    int chunk = (n + 2047) / 2048;
    chunk = chunk < 128 ? 128 : chunk > 4096 ? 4096 : (chunk + 31) & ~31;
    const int threads = 256;
    const long long chunks = ((long long)n + chunk - 1) / chunk;
    const int blocks = (int)std::min((long long)gg_num_sms() * 4, (chunks + threads / 32 - 1) / (threads / 32));
    k_extent<<<std::max(blocks, 1), threads, 0, st>>>(rec, n, poff, S, chunk, mm, (unsigned *)(mm + 8 * (size_t)S), hmm, dom,
                                                      err);
    gg_note_launches(1);
    if (S > ROOTS_ONE_BLOCK) {
        k_extent_roots<<<(S + 127) / 128, 128, 0, st>>>(S, mm, hmm, dom);
        gg_note_launches(1);
    }
}

void gg_launch_keys(const GGPart *rec, int n, const int *poff, int S, const GGDomainDev *dom,
                    unsigned long long *keys, unsigned *vals, int *err, cudaStream_t st)
{
    int threads = 256, blocks = gg_num_sms() * 8;
    if ((long long)blocks * threads > n) blocks = (n + threads - 1) / threads;
    if (blocks < 1) blocks = 1;
    k_keys<<<blocks, threads, 0, st>>>(rec, n, poff, S, dom, keys, vals, err);
    gg_note_launches(1);
}

void gg_launch_keys_plain(const double *pos, long long n, const GGDomainDev &d, unsigned long long *keys, int *err,
                          cudaStream_t st)
{
    int threads = 256;
    long long b = (n + threads - 1) / threads;
    int blocks = (int)(b < gg_num_sms() * 8 ? (b < 1 ? 1 : b) : gg_num_sms() * 8);
    k_keys_plain<<<blocks, threads, 0, st>>>(pos, n, d, keys, err);
    gg_note_launches(1);
}
