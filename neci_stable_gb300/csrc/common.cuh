// common.cuh -- device helpers shared by the step kernels (kernels.cu) and
// the spawn kernel (spawn.cuh): block reductions into the step's counters,
// warp-aggregated appends, and the walker hash (hash_table_lookup,
// AddNewHashDet, RemoveHashDet).
#pragma once

#include "engine.cuh"

namespace neci {

// ---------------------------------------------------------------------------
// Reduction helpers.
// ---------------------------------------------------------------------------
// Modulo 2^64, as a plain sum: three 22-bit parts, whose sums over a warp fit
// 32 bits, by the warp reduction instruction (three of them instead of ten
// shuffles and ten additions).
__device__ inline unsigned long long warp_sum_u(unsigned long long v) {
    const unsigned int a = __reduce_add_sync(0xffffffffu, (unsigned int)v & 0x3FFFFFu);
    const unsigned int b = __reduce_add_sync(0xffffffffu, (unsigned int)(v >> 22) & 0x3FFFFFu);
    const unsigned int c = __reduce_add_sync(0xffffffffu, (unsigned int)(v >> 44));
    return a + ((unsigned long long)b << 22) + ((unsigned long long)c << 44);
}

// Sums of NU counts over the block, one atomic per value.
template <int NU>
struct BlockCounts {
    unsigned long long red[NU][8];
    __device__ inline void warp_part(const unsigned long long (&u)[NU]) {
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const unsigned long long s = warp_sum_u(u[k]);
            if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = s;
        }
    }
    // behind a barrier: one thread per value
    __device__ inline void add(unsigned long long *const (&dst)[NU]) const {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            if ((int)threadIdx.x != k) continue;
            unsigned long long s = 0;
            for (int w = 0; w < nw; ++w) s += red[k][w];
            if (s != 0ull) atomicAdd(dst[k], s);
        }
    }
};
template <int NU>
__device__ inline void block_add_u(const unsigned long long (&u)[NU], unsigned long long *const (&dst)[NU]) {
    __shared__ BlockCounts<NU> counts;
    counts.warp_part(u);
    __syncthreads();
    counts.add(dst);
    __syncthreads();
}

// A sum of doubles that is exact: terms of 2^(52 - Q) up to 2^(80 - Q), all of
// whose bits are units of 2^-Q, are added as 96-bit integers; any other term
// goes to an FP64 sum of the thread's own.  An FP64 addition holds its pipe
// (about one lane per clock per SM) for as long as the SM's schedulers issue
// a hundred integer instructions, and this takes some fifteen.  No bit of a
// term is lost at any size, and a thread's share of 2^31 slots (27 594 terms
// below 2^80 units) stays below 2^95.  `own` is the thread's place in shared
// memory, not a register: the sweeps are short of them, and the atomic is a
// loop, which the compiler cannot turn into a predicated FP64 addition for
// every term.
template <int Q>
struct ExactSum {
    unsigned long long lo = 0;
    unsigned int hi = 0;
    __device__ inline void add(double a, double *own) {
        const long long b = __double_as_longlong(a);
        const unsigned int s = ((unsigned int)(b >> 52) & 0x7FFu) - (unsigned int)(1075 - Q);
        if (s > 27u) {
            if (b << 1) atomicAdd(own, a);
            return;
        }
        const unsigned long long m = ((unsigned long long)b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
        unsigned long long x = m << s;
        unsigned int xh = (unsigned int)((m >> 32) >> (32u - s));
        if (b < 0) {
            x = 0ull - x;
            xh = ~xh + (x == 0ull ? 1u : 0u);
        }
        lo += x;
        hi += xh + (lo < x ? 1u : 0u);
    }
};
struct PlainSum {
    double v = 0.0;
    __device__ inline void add(double a, double *) { v += a; }
};
// The sums every slot adds to, by instance: exact with one run, FP64 with a
// replica pair (twice the accumulators do not fit the registers: merge sweep
// 37 to 43 us at n = 32).  Steps with FP64 sums, and so (us): n = 64 8238 and
// 8134, 6x6 lattice 6945 and 6917, n = 24 793 and 782, n = 39 404 and 396; the
// sweep of 63504 determinants with 3000 walkers each 51 and 40.
template <int LR, int Q>
using SlotSum = typename std::conditional<LR == 1, ExactSum<Q>, PlainSum>::type;
// An amplitude (2^-18 to 2^10) and what a step takes from one or adds to it:
// a death, a rounding, a projected amplitude (2^-26 to 4).  (Units of 2^-64
// and 2^-76 left the core amplitudes of a decaying projection out: 45.2 and
// 44.6 us a step on the 10-site ring.)
constexpr int kUnitAmplitude = 70, kUnitChange = 78;

// NF of them over the block, one FP64 atomic per sum (k: its place among the
// block's; unit: 2^-Q).  The total is rounded at the conversion only.
template <int NF>
struct BlockExact {
    unsigned long long lo[NF][8];
    long long hi[NF][8];
    template <int Q>
    __device__ inline void warp_part(int k, const ExactSum<Q> &f) {
        // parts whose sums over a warp fit 32 bits
        const unsigned int a = __reduce_add_sync(0xffffffffu, (unsigned int)f.lo & 0x3FFFFFu);
        const unsigned int b = __reduce_add_sync(0xffffffffu, (unsigned int)(f.lo >> 22) & 0x3FFFFFu);
        const unsigned int c = __reduce_add_sync(0xffffffffu, (unsigned int)(f.lo >> 44));
        const unsigned int d = __reduce_add_sync(0xffffffffu, f.hi & 0xFFFFu);
        const int e = __reduce_add_sync(0xffffffffu, (int)f.hi >> 16);
        if ((threadIdx.x & 31) == 0) {
            const __int128 t = (__int128)(a + ((unsigned long long)b << 22)) + ((__int128)c << 44) +
                               ((__int128)((long long)d + (long long)e * 65536) << 64);
            lo[k][threadIdx.x >> 5] = (unsigned long long)t;
            hi[k][threadIdx.x >> 5] = (long long)(t >> 64);
        }
    }
    // behind a barrier: thread `by` adds sum k
    __device__ inline void add(int k, unsigned int by, double unit, double *target) const {
        if (threadIdx.x != by) return;
        __int128 t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ((__int128)hi[k][w] << 64) + (__int128)lo[k][w];
        if (t == 0) return;
        const bool neg = t < 0;
        const unsigned __int128 u = neg ? (unsigned __int128)(-t) : (unsigned __int128)t;
        const double v = ((double)(unsigned long long)(u >> 64) * 18446744073709551616.0 + (double)(unsigned long long)u) * unit;
        atomicAdd(target, neg ? -v : v);
    }
};

// Block-wide sums of NV doubles and NU counts into global atomics (one atomic
// per value per block).  The doubles are per run, run-minor (v[2i + run]);
// with one run the odd entries are skipped.  blockDim.x: a power of two from
// 8 NV to 256.
// The FP64 pipe of about one lane per clock per SM is what this costs: it
// ends every block, and in a short kernel the sums of a whole step end it at
// once.  So a value that is zero in the whole block (most are: births,
// aborts, the reference's and its connections' sums in most blocks) takes no
// addition; one warp per value folds the threads' values to 32 (7 full-width
// adds of 256 values); and 8 lanes per value, four values a warp, add those
// (6 adds for four values), instead of 5 shuffle levels each.  12 values of
// 256 threads: 156 FP64 warp instructions before, at most 102 now, 34 with
// four of them non-zero.
// NO more doubles are in the last rows of `red` already (the sweeps' threads
// add to their places there).
template <int NV, int NO, int NU>
__device__ inline void block_add_rows(double (*red)[256], const double (&v)[NV], double *const (&dst)[NV + NO], int L,
                                      const unsigned long long (&u)[NU], unsigned long long *const (&du)[NU]) {
    __shared__ double *to[NV + NO];
    __shared__ unsigned int row[NV + NO];  // the non-zero values, in order
    __shared__ unsigned int live[8];   // the warps' masks of non-zero values
    __shared__ BlockCounts<NU> counts;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    unsigned int mask = 0;
#pragma unroll
    for (int m = 0; m < NV; ++m)
        if ((m & 1) < L) {
            red[m][t] = v[m];
            if ((unsigned long long)__double_as_longlong(v[m]) << 1) mask |= 1u << m;
        }
#pragma unroll
    for (int m = NV; m < NV + NO; ++m)
        if ((unsigned long long)__double_as_longlong(red[m][t]) << 1) mask |= 1u << m;
    if (t == 0) {
#pragma unroll
        for (int m = 0; m < NV + NO; ++m) to[m] = dst[m];
    }
    counts.warp_part(u);
    mask = __reduce_or_sync(0xffffffffu, mask);
    if (lane == 0) live[wid] = mask;
    __syncthreads();
    counts.add(du);
    mask = 0;
    for (int w = 0; w < nw; ++w) mask |= live[w];
    // the k-th non-zero value: warp k mod nw.  Not unrolled: at a short
    // kernel's end this code runs once, its instructions fetched for it.
    unsigned int rest = mask;
#pragma unroll 1
    for (int k = 0; rest; ++k, rest &= rest - 1) {
        if ((k & (nw - 1)) != wid) continue;
        const unsigned int m = __ffs(rest) - 1;
        double s = red[m][lane];
        for (int i = lane + 32; i < (int)blockDim.x; i += 32) s += red[m][i];
        red[m][lane] = s;
        if (lane == 0) row[k] = m;
    }
    __syncthreads();
    const int n = __popc(mask);
    if (wid * 4 < n) {  // four values a warp
        const int k = min(t >> 3, n - 1);
        const double *r = red[row[k]];
        double s = r[t & 7];
#pragma unroll
        for (int i = 8; i < 32; i += 8) s += r[(t & 7) + i];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
        if ((t & 7) == 0 && (t >> 3) < n) atomicAdd(to[row[k]], s);
    }
    __syncthreads();
}
template <int NV, int NU>
__device__ inline void block_add(const double (&v)[NV], double *const (&dst)[NV], int L, const unsigned long long (&u)[NU],
                                 unsigned long long *const (&du)[NU]) {
    __shared__ double red[NV][256];
    block_add_rows<NV, 0, NU>(red, v, dst, L, u, du);
}

// Warp-aggregated append of `want` items: returns this lane's first index.
// Every lane of the warp must call it (all loops that use it run a
// warp-uniform number of times).
__device__ inline unsigned long long warp_append(unsigned long long *counter, unsigned int want) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    unsigned int incl = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const unsigned int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total) base = atomicAdd(counter, (unsigned long long)total);
    base = __shfl_sync(0xffffffffu, base, 31);
    return base + incl - want;
}

// warp_append of at most one item per lane: the positions follow from a
// ballot (the same as warp_append's for want in {0, 1}).
__device__ inline unsigned long long warp_append1(unsigned long long *counter, bool want) {
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int m = __ballot_sync(0xffffffffu, want);
    unsigned long long base = 0;
    if (lane == 31 && m) base = atomicAdd(counter, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 31);
    return base + __popc(m & ((1u << lane) - 1u));
}

__device__ inline void set_err(Control *c, int code) { atomicCAS(&c->err, 0, code); }

__device__ inline void load_rh2(const DevSys &s, int32_t *sh) {
    for (int i = threadIdx.x; i <= s.nbasis; i += blockDim.x) sh[i] = s.random_hash2[i];
    __syncthreads();
}

// Remove slot j from the walker hash (RemoveHashDet, load_balancer.fpp:631).
// The caller counts the tombstone and adds its count to Control::n_tomb once
// per block (one atomic per removal would serialise millions of them per
// step on one address).
__device__ inline void hash_remove(const DevState &st, long long j) {
    const uint32_t b = st.slot_bucket[j];
    st.hash[b] = kTomb;
}

// Look a determinant up: returns slot or -1.
__device__ inline long long hash_find(const DevState &st, const unsigned long long *d, int W, int R,
                                      unsigned long long h, Control *ctl) {
    const unsigned long long mask = st.hash_n - 1;
    unsigned long long b = hash_bucket(h, st.hash_n);
    for (int p = 0; p < kProbeLimit; ++p) {
        const uint32_t e = st.hash[b];
        if (e == kEmpty) return -1;
        if (e != kTomb) {
            const long long slot = (long long)e - 1;
            if (det_eq(d, st.dets + slot * R, W)) return slot;
        }
        b = (b + 1) & mask;
    }
    set_err(ctl, NECI_GPU_ERR_HASH_FULL);
    return -1;
}

// Insert a determinant known to be absent.  Returns 1 if it took a
// tombstone's bucket (the caller takes one off its tombstone count).
__device__ inline int hash_insert(const DevState &st, long long slot, unsigned long long h, Control *ctl) {
    const unsigned long long mask = st.hash_n - 1;
    unsigned long long b = hash_bucket(h, st.hash_n);
    for (int p = 0; p < kProbeLimit; ++p) {
        const uint32_t e = st.hash[b];
        if (e == kEmpty || e == kTomb) {
            if (atomicCAS(&st.hash[b], e, (uint32_t)(slot + 1)) == e) {
                st.slot_bucket[slot] = (uint32_t)b;
                return e == kTomb ? 1 : 0;
            }
            continue;  // lost the race for this bucket: look at it again
        }
        b = (b + 1) & mask;
    }
    set_err(ctl, NECI_GPU_ERR_HASH_FULL);
    return 0;
}

// TestInitiator_explicit (fcimc_helper.F90:1142-1240) without ADI, senior
// initiators or an initiator space.
__device__ inline bool test_initiator(const IterParams &p, bool was, double sgn, bool is_ref, bool core) {
    const bool popInit = abs_bits(sgn) > dbl_bits(p.initiator_walk_no);  // |sgn| > InitiatorWalkNo
    if (!was) return popInit;
    if (!is_ref && !(core && p.t_core_inits) && !popInit) return false;
    return true;
}

}  // namespace neci
