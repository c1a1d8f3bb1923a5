// internal.h -- host-side engine object shared by the C ABI and the launchers.
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/neci_gpu.h"
#include "engine.cuh"

namespace neci {

enum KernelId {
    K_COMPACT = 0,
    K_REHASH,
    K_BEGIN,   // (no stage of its own any more; the ids are part of the ABI)
    K_SWEEP,
    K_EXPAND,  // (as K_BEGIN)
    K_SPAWN,
    K_CORE,
    K_ANN_PROBE,
    K_ANN_COMPRESS,
    K_ANN_INSERT,
    K_MERGE_STATS,
    K_RDM,
    K_FINAL,
    K_SORT_KEYS,   // sort form of the annihilation: keys, radix passes, grouping
    K_SORT_RADIX,
    K_SORT_GROUP,
    K_NUM
};

// Spawn records and new determinants of a step up to which its annihilation
// takes the kernels of a short list.  Both save launches and
// waits, and both put work into one kernel that the split form has beside the
// merge sweep (compression) or at a better occupancy (placement), so the lines
// are those of the step, in us with the split form and so:
// lookup and compression in one (k_ann_gather): lattice with several couplings
// 1.0e5 records 133 and 118, 2.6e5 266 and 258, 5.2e5 458 and 477; n = 39
// 2.1e5 309 and 290, 4.2e5 496 and 502; n = 24 2.8e5 224 and 216, 5.5e5 365
// and 374; 12-site ring 3.5e5 148 and 144, 6.8e5 235 and 234;
// decision and placement in one (k_ann_new), beside k_ann_gather: ring 1.8e5
// records and 5.9e3 new determinants 97.9 and 93.3; n = 32 replica pair 8.3e4
// and 7.4e3 146 and 142; n = 39 1.0e5 and 1.2e4 177 and 179; n = 24 1.5e5 and
// 1.6e4 135 and 136; n = 64 1.7e5 and 3.6e4 822 and 846; n = 39 2.1e5 and
// 2.4e4 290 and 321.
constexpr long long kGatherSpawns = 350000;
constexpr long long kShortSpawns = 200000;
constexpr long long kShortNew = 12000;

struct Engine {
    neci_gpu_system desc{};
    DevSys sys{};
    DevState st{};
    int device = 0;
    int num_sms = 152;
    // resident blocks per SM of the grid-stride spawn-list kernels (their
    // grids fill the GPU once; the latency-bound hash passes want every warp)
    int occ_probe = 4, occ_compress = 4, occ_insert = 4, occ_place = 8;
    // pass 1 of the annihilation runs inside the spawn kernel (chosen from the
    // last step's spawn rate; see update_fuse_probe)
    bool fuse_probe = false;
    // NECI_OPT_FUSE_PROBE: -1 chosen from the spawn rate, 0 never, 1 always
    int fuse_mode = -1;
    // NECI_OPT_ANNIHILATION: NECI_ANN_HASH or NECI_ANN_SORT
    int ann_mode = NECI_ANN_HASH;
    // tuned launch shapes (neci_gpu_tuning): spawn blocks per SM, radix-pass
    // blocks per SM (DevState::comp_shift holds the table load setting)
    int spawn_occ = 8;
    int sort_bpsm = 2;
    // the last step's spawn list was short: lookup and compression, decision
    // and placement in one kernel each (update_short_list)
    bool gather = true, short_list = true;
    bool stepped = false;  // the context has made a step
    // the contexts of a batch share the GPU: each one's grids are this much
    // smaller (batch_share; 1 outside a batch's capture)
    int share = 1;
    int live_share = 16;  // ... and this much at most (update_live_share)
    int merge_bpsm = 2;  // merge sweep blocks per SM beside the placement (update_merge_blocks)
    bool compact_due = false;  // the last step left more holes than occupied slots
    bool rehash_due = false;   // ... or the walker hash over its load
    int core_seg_lane = kCoreSegmentPerLane;  // NECI_OPT_CORE_SEGMENT
    cudaStream_t stream = nullptr;
    IterParams *d_params = nullptr;
    IterParams *h_params = nullptr;          // pinned
    neci_gpu_iter_stats *h_stats = nullptr;  // the steps' records (pinned; k_final writes them)
    int max_stats = 0;
    // changes with every drop of the step graphs (a batch graph built on them
    // is rebuilt)
    unsigned long long graph_version = 0;
    // a batch graph (neci_gpu_iterate_batch) kept by the batch's first
    // context: every instance's step as one branch, and what it was built for
    cudaGraphExec_t batch_graph = nullptr;
    std::vector<std::pair<const void *, unsigned long long>> batch_key;
    cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
    // the step's two branches after the walker-hash lookup (new determinants;
    // the merge sweep), on stream and side
    cudaStream_t side = nullptr;
    cudaEvent_t branch_ev = nullptr, merge_ev = nullptr;
    cudaEvent_t sweep_ev = nullptr, freed_ev = nullptr;  // around k_rdm_freed, which runs beside the spawn
    std::vector<void *> allocs;
    bool have_ref = false, have_pchb = false;
    // lattices: host copies of TMat2D and the neighbour lists, and the device
    // table of DevSys::lat derived from them
    std::vector<double> h_tmat;
    std::vector<int32_t> h_neighbours;
    LatTab *lat_tab = nullptr;
    ulonglong2 *hash_tab = nullptr;  // device table of DevSys::hash_tab
    double *inv_single = nullptr;  // device table of DevSys::inv_single
    float *inv_single32 = nullptr;
    // CUDA graph of one step per precision (FP64, mixed); `graph` is the one
    // ensure_graph selected for the current parameters
    cudaGraphExec_t graphs[2] = {nullptr, nullptr};
    bool graph_core[2] = {false, false};
    bool graph_fast[2] = {false, false};  // the sweep variant a graph was captured with
    cudaGraphExec_t graph = nullptr;
    // profiling
    bool profiling = false;
    cudaEvent_t ev[2 * K_NUM] = {};
    double kernel_ms[K_NUM] = {};
    long long kernel_launches[K_NUM] = {};
};

// Whether the spawn kernel does pass 1 of the annihilation (the walker-hash
// lookup of every child): lattice systems with the hash annihilation and no
// 2-RDM sampling, as NECI_OPT_FUSE_PROBE (or, by default, the spawn rate) says.
inline bool fused_lookup(const Engine &e) {
    if (e.sys.rdm || e.sys.excitgen != NECI_EXGEN_RS_HUBBARD || e.ann_mode != NECI_ANN_HASH) return false;
    return e.fuse_mode < 0 ? e.fuse_probe : e.fuse_mode == 1;
}

// launchers (kernels.cu)
void launch_begin(Engine &e, cudaStream_t s);
void launch_rehash(Engine &e, cudaStream_t s);
void launch_compact(Engine &e, cudaStream_t s);
void launch_sweep(Engine &e, cudaStream_t s);
// sets the per-kernel launch attributes a context needs (non-zero: failure)
int configure_kernels(Engine &e);
void launch_spawn(Engine &e, cudaStream_t s);
void launch_core(Engine &e, cudaStream_t s);
void launch_ann_probe(Engine &e, cudaStream_t s);
void launch_ann_compress(Engine &e, cudaStream_t s);
void launch_ann_insert(Engine &e, cudaStream_t s, int split);
void launch_ann_gather(Engine &e, cudaStream_t s);
void launch_ann_new(Engine &e, cudaStream_t s, int split);
void launch_merge_stats(Engine &e, cudaStream_t s, int with_core, int split);
void launch_final(Engine &e, cudaStream_t s, int advance_iter, int split);
// packing of the occupied slots for a read of the list
void launch_read_scan(Engine &e, long long n);
void launch_read_pack(Engine &e, long long n, long long t0, long long t1, long long *rows, double *dh, double *odh);
void launch_rdm(Engine &e, cudaStream_t s);
void launch_rdm_freed(Engine &e, cudaStream_t s);

// sort form of the annihilation and core selection (sort_kernels.cu)
constexpr int kSortBins = 256;  // digit values of a radix pass (radix.cuh kRadixBins)
void launch_sort_keys(Engine &e, cudaStream_t s);
int launch_sort_radix(Engine &e, cudaStream_t s);
void launch_sort_group(Engine &e, cudaStream_t s, int lookup, int cur);
int sort_ann_blocks(const Engine &e);
int launch_core_select_sort(Engine &e, unsigned long long *key[2], uint32_t *val[2], uint32_t *counts, int blocks,
                            unsigned long long *n_occ);
void launch_core_select_gather(Engine &e, const uint32_t *slot, long long n, long long *core_dets);

// utility launchers (util_kernels.cu)
void launch_util_hash(Engine &e, const long long *dets, long long n, unsigned long long len, long long *out);
void launch_util_excit_level(Engine &e, const long long *a, const long long *b, long long n, int *out);
void launch_util_helement(Engine &e, const long long *a, const long long *b, long long n, double *out);
void launch_util_gen_excit(Engine &e, const long long *det, long long n, unsigned long long seed, long long iter,
                           long long *child, double *pgen, double *hel);
void launch_upload_fix(Engine &e, long long nrows, int compute_diag);
void launch_collect_holes(Engine &e);
void launch_convert_spawns(Engine &e, long long n);
void launch_all_cand(Engine &e);
void launch_compress_out(Engine &e, long long *out, unsigned long long *n_out);
void launch_core_unmark(Engine &e);
void launch_core_mark(Engine &e, const long long *core_dets, long long n_core);
void launch_core_count(Engine &e, const long long *core_dets, long long n_core, long long *counts);
void launch_core_fill(Engine &e, const long long *core_dets, long long n_core);
// PCHB alias tables; returns a cudaError_t value (0: built), and launches
// nothing when its scratch cannot be allocated
int launch_pchb_build(Engine &e);
void launch_build_jk(Engine &e, double *jrow, double *jkrow, float *jrow32, float *jkrow32);
void launch_build_jkmat(Engine &e, double *jmat, double *kmat);

}  // namespace neci
