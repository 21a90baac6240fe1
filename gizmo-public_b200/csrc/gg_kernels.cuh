// gg_kernels.cuh -- launch functions shared between the kernel files and the API.
#pragma once
#include <cstddef>

#include "gg_internal.cuh"

#define GG_SORT_MAX_PASSES 12

// per-node build arrays (device pointers), capacity `cap` nodes
struct TreeBuf {
    int *start, *end, *level, *parent, *sys, *nch, *child;
    int *bnd;          // 8 digit boundaries per node
    double *mass64;    // FP64 node mass (parent sums)
    int *depth_beg;    // GG_MAX_DEPTH + 2 entries
    int *nnodes;       // total nodes, deepest depth (device); zero until the node kernel has written every node, and
                       // again when the moments are given up: whatever reads the nodes takes their number from here
    unsigned *ticket;  // parts handed out: node kernel, moments kernel
    unsigned *done;    // finished parts per depth of the node kernel, per phase of the moments kernel (TREE_PHASES each)
    unsigned *bstat;   // per depth and part: published children totals (GG_MAX_DEPTH x grid)
    int cap;           // node capacity (set by gg_launch_tree)
    int *err;
    int wait_limit;    // polls after which a wait between blocks gives up
    int wait_extra[2]; // parts that the node and the moments kernel's waits count in vain (self-test; else 0)
};

#define TREE_WAIT_LIMIT (1 << 24)
#define TREE_PHASES (GG_MAX_DEPTH + 1)
// TreeBuf's nnodes, ticket, done and bstat lie in one array, cleared before each build
#define TREE_STATE_WORDS(grid) (4 + 2 * TREE_PHASES + (size_t)GG_MAX_DEPTH * (grid))

size_t gg_extent_words(int S);   // 64-bit words of gg_launch_extent's scratch mm
void gg_launch_extent(const GGPart *rec, int n, const int *poff, int S, unsigned long long *mm, unsigned *hmm,
                      GGDomainDev *dom, int *err, cudaStream_t st);
void gg_launch_keys(const GGPart *rec, int n, const int *poff, int S, const GGDomainDev *dom,
                    unsigned long long *keys, unsigned *vals, int *err, cudaStream_t st);
void gg_launch_keys_plain(const double *pos, long long n, const GGDomainDev &d, unsigned long long *keys, int *err,
                          cudaStream_t st);

size_t gg_sort_scratch_bytes(long long n);
int gg_sort_bits();
// Records moved by the last pass of a sort whose values are record indices:
// out[position] = in[value], rank[value] = position.
struct SortGather {
    const GGPart *in;
    GGPart *out;
    unsigned *rank;
};
// gather (nullable): done by the last pass; *gathered says whether it was (no
// pass runs for n <= 1 or no bits).
gg_status gg_sort_pairs_run(unsigned long long *keys, unsigned *vals, long long n, int key_bits, int sys_bits,
                            const int *poff, int S, void *scratch, int *err, cudaStream_t st,
                            const SortGather *gather = nullptr, bool *gathered = nullptr);

void gg_launch_permute(const unsigned *perm, const GGPart *in, GGPart *out, unsigned *rank, int n, cudaStream_t st);
int gg_tree_grid();
gg_status gg_launch_tree(const unsigned long long *keys, const int *poff, int S, int n, int leaf, int cap, TreeBuf tb,
                         const GGPart *parts, const GGDomainDev *dom, GGNode *nodes, cudaStream_t st);

// Long walks are cut (gg_walk.cu) in systems of this range: they have a few groups
// per resident warp, and the longest end last.  Walk ms uncut / cut at tolerance
// 0.0025 in groups of 32 (galaxy, Plummer, clustered): 65,536 0.73 / 0.44, 0.34 /
// 0.30, 0.37 / 0.41; 98,304 0.90 / 0.70, 0.40 / 0.32, 0.51 / 0.45; 200,000 1.88 / 1.12,
// 0.67 / 0.66, 0.67 / 0.69; 300,000 2.69 / 1.55, 0.66 / 0.63, 0.77 / 0.79; 350,000 3.00 /
// 2.98, 0.71 / 0.77, 1.07 / 0.94; 500,000 4.32 / 4.42, 0.85 / 0.92, 1.22 / 1.27.  Beyond
// 300,000 the groups outnumber the warps so far that the longest, started first, end
// with the rest, and the cut's own cost is left (a 10% subset of 4.2M particles, cut:
// 5.7 ms instead of 5.3).  Below 98,304 a cut gains alone, but such systems come in
// batches, whose groups fill the GPU (48 served systems with 65,536 in the range:
// no difference).
#define FORK_MIN_TARGETS 98304
#define FORK_MAX_TARGETS 300000
// Work (node tests, list entries; a softened entry counts three) after which a walk
// is cut at GIZMO's tolerance: about twice a mean group's, or four times in systems
// above FORK_HALF_TARGETS.  Walk ms uncut / cut at 8192 / 16384 / 32768: Plummer
// 65,536 0.34 / 0.31 / 0.35 / 0.35, galaxy 100,000 0.97 / 0.78 / 0.81 / 0.95, galaxy
// 262,144 2.06 / 2.73 / 1.38 / 1.56.  Stricter criteria make every walk longer; the
// work of a cut grows with them (fork_work).
#define FORK_HALF_TARGETS 131072
#define FORK_WORK 16384
#define FORK_WALKS 8        // sub-walks the pending nodes are dealt to
#define FORK_PENDING 2048   // pending nodes at most
#define FORK_RECORDS 512    // cuts whose sub-walks can run as tasks of any warp
// ... in launches of at most this many targets; with more, there is work enough
// for every warp, and each runs its own sub-walks
#define FORK_TASK_TARGETS 400000
// the record of one cut
struct WalkFork {
    int group, npend;
    float cost;
    int pad;
    int pending[FORK_PENDING];
    // per target: acceleration and potential, interactions; of the walk up to the
    // cut, and (not in the records of single warps, which end here) of the sub-walks
    double4 sum0[64];
    int nint0[64];
    double4 sum[FORK_WALKS][64];
    int nint[FORK_WALKS][64];
};
#define FORK_OWN_BYTES offsetof(WalkFork, sum)
// places in WalkParams.group_counter: groups handed out, cuts made, tasks handed out, groups finished
#define WALK_FORK_COUNTER 1
#define WALK_TASK_COUNTER 2
#define WALK_DONE_COUNTER 3
#define WALK_COUNTERS 8     // then, per record: whether it is complete, and how many of its parts are finished

struct WalkParams {
    const GGNode *nodes;
    const int *nnodes;          // 0: there is no complete tree, and nothing is walked
    const GGPart *parts;        // sorted
    const GGGroup *groups;
    const int *ngroups;         // device count
    const int *tlist;           // sorted particle index per target, NULL = identity
    const int *tout;            // output slot per target, NULL = load-order index of the particle
    const unsigned *perm;       // sorted position -> load-order index
    const double *oldacc_in;    // per particle (load order), NULL = 0
    double *oldacc_out;         // per particle (load order), may be NULL
    double tol, theta;
    double *acc;                // 3 per output slot
    double *pot;                // per output slot, may be NULL
    int *ninter;                // per output slot, may be NULL
    unsigned long long *interactions;   // [0] interactions, [1] far / [2] near list entries, [3] nodes tested
    int *group_counter;         // counters, zero at the launch
    const int *toff;            // target offsets per system
    WalkFork *forks;            // fork_max records
    char *own_forks;            // a record of FORK_OWN_BYTES per resident warp
    int fork_max;
    int may_fork;               // some walk of this launch may be cut
    int fork_work;              // ... after this much work (half of it up to FORK_HALF_TARGETS)
    int *fork_ready, *fork_parts;   // per record, zero at the launch
    int *stack;
    int stack_cap;
    int *err;
    int group_size;
    int flush;
    int pot_only;               // potential-only walk: acc and oldacc_out unused, pot required
    const unsigned *gorder;     // order in which groups are handed out, NULL = index order
    float *cost_out;            // per particle (load order): its group's cycles per target, may be NULL
    int node_staging;           // 0: per-lane cp.async, 1: bulk copies (TMA) per run of consecutive nodes
};
void gg_launch_walk(const WalkParams &p, int blocks_per_sm, cudaStream_t st);
int gg_walk_threads();

// groups of `gs` consecutive targets per system; toff[S+1] target offsets per system
void gg_launch_groups(const int *toff, int S, int gs, GGGroup *groups, int *ngroups, int *gscan, cudaStream_t st);
long long gg_max_groups(long long n, int S, int gs);
int gg_target_order_lmax(int S);
// Scratch: gnode one int per particle, gstat gg_group_stat_words(nt) words.
size_t gg_group_stat_words(long long nt);
void gg_launch_groups_tree(int nt, const int *tlist, const int *tscan, const int *toff, int S, int gs,
                           const TreeBuf &tb, const GGDomainDev *order_dom, const unsigned *hmm, int lmax, int *gnode,
                           unsigned *gstat, int maxg, GGGroup *groups, int *ngroups, int *err, cudaStream_t st);
// exclusive scan of n ints (scratch: 2 * (gg_num_sms()*4) ints)
void gg_launch_scan(const int *in, int *out, int n, int *scratch, cudaStream_t st);
// active targets: flags in sorted order -> tlist/tout, and per-system offsets
void gg_launch_active(const int *active, int n_active, const unsigned *rank, int n, int *flag, int *flagscan,
                      int *tlist, int *tout, const int *poff, int S, int *toff, int *scratch, int *err,
                      cudaStream_t st);
int gg_scan_scratch_ints();
// walk groups sorted by the summed previous cost of their targets, most
// expensive first: gorder[0..maxg) (groups past the device count sort last)
gg_status gg_order_groups_by_cost(const GGGroup *groups, const int *ngroups, int maxg, const int *tlist,
                                  const unsigned *perm, const float *cost, unsigned long long *key,
                                  unsigned *gorder, void *sort_scratch, int *err, cudaStream_t st);
// targets reordered by (system, kernel radius), key order kept within a class
gg_status gg_order_targets_by_softening(int nt, const int *tlist_in, const int *tout_in, const GGPart *parts,
                                        const unsigned long long *pkeys, const int *poff, int S,
                                        const GGDomainDev *dom, const unsigned *hmm, unsigned long long *key,
                                        unsigned *val, int *tlist_out, int *tout_out, void *sort_scratch, int *err,
                                        cudaStream_t st);

void gg_launch_direct_records(const GGPart *rec, const int *poff, const int2 *tg, int ntg, double *acc, double *pot,
                              double *mass, cudaStream_t st);
void gg_launch_gather_rows(const double *acc, const double *pot, const int2 *tg, int ntg, double *acc_out,
                           double *pot_out, cudaStream_t st);
void gg_launch_direct(long long n_src, const double *pos, const double *mass, const double *h, long long n_tgt,
                      const int *targets, double *acc, double *pot, cudaStream_t st);

// drift of a resident tree (gg_drift.cu)
void gg_launch_node_kinematics(const GGPart *parts, const unsigned *perm, const double *vel, TreeBuf tb, int *counter,
                               double4 *kin, int n, int ncap, int keep_max, cudaStream_t st);
void gg_launch_set_positions(GGPart *in_rec, GGPart *parts, const unsigned *perm, const double *pos, int n, int *err,
                             cudaStream_t st);
void gg_launch_drift(GGPart *in_rec, GGPart *parts, const unsigned *perm, const double *vel, const int *poff, int S,
                     const double *dts, double dt_all, GGNode *nodes, const double4 *kin, const int *node_sys, const int *nnodes,
                     int n, int ncap, cudaStream_t st);

// FP64 per-system sums {1/2 sum m phi, sum m a} (gg_util.cu)
void gg_launch_energy(const int4 *chunks, int nchunks, const int *sys_first_chunk, int S, const GGPart *rec,
                      const double *acc, const double *pot, double *part, double *out, cudaStream_t st);

// bounded look-back self-test (gg_sort.cu)
gg_status gg_sort_timeout_selftest(cudaStream_t st);
