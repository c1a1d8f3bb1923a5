// spawn.cuh -- the spawn attempts of a step (FciMCPar.F90:1600-1745,
// loop_over_walkers): generate_excitation, attempt_create and
// create_particle for every attempt entry the sweep wrote, one attempt per
// thread per round.  Instantiated per precision of the amplitude (one
// translation unit each: spawn_fp64.cu, spawn_fp32.cu), excitation generator
// and number of determinant words.
#pragma once

#include "common.cuh"
#include "excitgen.cuh"
#include "internal.h"

namespace neci {

// ===========================================================================
// k_spawn
// ===========================================================================
template <typename Real>
__device__ inline Real prm(double d, float f) { return sizeof(Real) == 8 ? (Real)d : (Real)f; }

// The rounding of a spawned amplitude of magnitude aq in fixed point, with its
// sign: RealSpawnCutoff rounding (|n| < cutoff -> +-cutoff with probability
// |n|/cutoff) or stochastic_round (lib/util_mod.fpp:182) to an integer
// walker, in integer arithmetic.  Returns 0 for no child.
__device__ inline long long round_amplitude(const IterParams &p, bool negative, unsigned long long aq, Stream &rng) {
    unsigned long long v = aq;
    if (p.t_all_real_coeff) {
        // keep with probability aq / cutoff_q
        if (p.t_real_spawn_cutoff && aq < p.cutoff_q)
            v = __umul64hi(rng.next64(), p.cutoff_q) < aq ? p.cutoff_q : 0ull;
    } else {
        const unsigned long long whole = aq >> 32, frac = aq & 0xFFFFFFFFull;
        v = whole;
        if (frac != 0 && (rng.next64() >> 32) < frac) v += 1;
        v <<= 32;
    }
    return negative ? -(long long)v : (long long)v;
}

// attempt_create_normal (fcimc_pointed_fns.F90:178-494) for one generated
// excitation: the child amplitude -tau H_ij sign(C) / (p_gen AvMCExcits),
// taken as -tau H_ij sign(C) (1/p_gen) (1/AvMCExcits) in precision Real and
// converted to fixed point, then rounded there (round_amplitude).  Returns 0
// for no child.
// In FP64 the product is formed as ((tau H_ij) (1/p_gen)) (1/AvMCExcits)
// and its sign applied afterwards: multiplying by -1, by the walker sign and
// by 1/AvMCExcits = 1 are exact, so the value is the reference order's, with
// two multiplies where it has five; the scaling by 2^32 and the rounding to
// an integer are done on the bits (fixed32_from_double).
template <typename Real>
__device__ inline long long spawn_amplitude(const IterParams &p, Real hel, Real invp, bool neg, Stream &rng, int &ovf,
                                            unsigned long long &aq_out) {
    long long q;
    if (sizeof(Real) == 8) {
        double v = (p.tau * (double)hel) * (double)invp;
        if (!p.av_unit) v = v * p.inv_av;
        int64_t qq;
        if (!fixed32_from_double(v, qq)) { ovf = 1; return 0; }
        q = neg ? qq : -qq;  // -tau H sign(C): positive for a negative parent
    } else {
        const Real ww = neg ? (Real)-1 : (Real)1;
        const Real nsp = -prm<Real>(p.tau, p.f_tau) * hel * ww * invp * prm<Real>(p.inv_av, p.f_inv_av);
        const float sc = (float)nsp * 4294967296.0f;
        if (!(fabsf(sc) < 9.2e18f)) { ovf = 1; return 0; }
        q = __float2ll_rn(sc);
    }
    const unsigned long long aq = (unsigned long long)(q < 0 ? -q : q);
    aq_out = aq;
    return round_amplitude(p, q < 0, aq, rng);
}

// One spawn attempt's parent, unpacked from its 8-byte attempt entry
// (slot | run << 32 | sign bit << 33 | attempt index << 34).
struct Parent {
    unsigned long long d[kMaxWords];
    unsigned long long key;
    unsigned int k;
    int run;
    bool neg, core, pinit;
};
// Words of a CurrentDets row (NIfD + 1): RW where the kernel is instantiated
// for that count, else the system's W.
template <int RW>
__device__ inline int rwords(const DevSys &s) { return RW > 0 ? RW : s.W; }

template <int NW, int RW>
__device__ inline void load_parent(const DevSys &s, const DevState &st, const IterParams &p, unsigned long long w0,
                                   Parent &P) {
    const long long j = (long long)(w0 & 0xFFFFFFFFull);
    P.run = (int)((w0 >> 32) & 1ull);
    P.neg = (w0 >> 33) & 1ull;
    P.k = (unsigned int)(w0 >> 34);
    const long long *r = st.dets + j * s.R;
    NECI_FOR_WORDS(w, nwords<NW>(s)) P.d[w] = (unsigned long long)r[w];
    const long long flags = r[rwords<RW>(s) + s.L];
    P.core = st.n_core > 0 && is_core_flags(flags);
    P.pinit = p.t_trunc_initiator && test_bit(flags, init_flag_bit(P.run));
    // det_key of the row (the words past NW are zero), which the sweep
    // stored for every slot with attempts
    P.key = st.dkey[j];
}

// The stream of an attempt from its entry alone: what the classification of
// an attempt (single or double) needs, without the parent's row.
__device__ inline Stream attempt_stream(const DevState &st, const IterParams &p, unsigned long long w0) {
    const long long j = (long long)(w0 & 0xFFFFFFFFull);
    return Stream(st.dkey[j], p.iter, P_ATTEMPT, (uint32_t)((w0 >> 32) & 1ull), (uint32_t)(w0 >> 34));
}

// Attempt v of the row of all attempts of heavy parents, as an entry: its
// parent is the one noted for its granule or one of the next few (a heavy
// parent has more than kBigAttempts attempts).  The parents with hundreds or
// thousands of attempts so cost one record each, not an entry per attempt
// written and read, and no kernel to write them (that kernel took 19 us of
// 906 per step at n = 24 with 1e7 walkers, and 5 us of an idle step).
__device__ inline unsigned long long heavy_attempt(const DevState &st, unsigned long long v) {
    const unsigned long long n_big = min(st.ctl->n_big >> kBigShift, (unsigned long long)st.max_big);
    const unsigned long long *b = st.big + 3ull * st.big_at[v / kBigGranule], *last = st.big + 3 * n_big - 3;
    while (b < last && v - b[1] >= b[2]) b += 3;
    return b[0] + ((v - b[1]) << 34);
}
// The entry of attempt q: the sweep's n_entry entries come first, then the
// heavy parents' attempts.
__device__ inline unsigned long long attempt_entry(const DevState &st, long long q, const volatile long long &n_entry) {
    return q < n_entry ? st.att[q] : heavy_attempt(st, (unsigned long long)(q - n_entry));
}

// Block-local tau-search log of k_spawn: per TauClass the largest gamma (as
// bits) and the logged count, capped near the reference's threshold.
struct TauAcc {
    unsigned long long g[4];
    unsigned int c[4];
};

// log_spawn_magnitude (tau_search_conventional.F90:138-258): gamma =
// |H_ij| / (p_gen / p_class) of one generated excitation, taken as
// |H_ij| (1/p_gen) p_class in precision Real.  Singles and uniform doubles
// count when gamma > 0, parallel and opposite-spin doubles always.
template <typename Real>
__device__ inline void tau_log(const DevSys &s, const Excit<Real> &e, TauAcc *acc) {
    double g;
    if (sizeof(Real) == 8) g = fabs((double)e.hel) * (double)e.invp * s.tau_fac[e.cls];
    else g = (double)(fabsf((float)e.hel) * (float)e.invp * s.f_tau_fac[e.cls]);
    const unsigned long long b = (unsigned long long)__double_as_longlong(g);
    if (b > acc->g[e.cls]) atomicMax(&acc->g[e.cls], b);
    const bool counts = (e.cls == TC_PAR || e.cls == TC_OPP) || g > 0.0;
    if (counts && acc->c[e.cls] <= kTauCntThreshold) atomicAdd(&acc->c[e.cls], 1u);
}

// Whether a child is a core determinant (is_core_state,
// semi_stoch_procs.F90:547).
template <int NW, int RW>
__device__ inline bool core_child(const DevSys &s, const DevState &st, const unsigned long long *c) {
    const long long hs = hash_find(st, c, nwords<NW>(s), s.R, neci_hash(c, nwords<NW>(s), s.random_hash2), st.ctl);
    return hs >= 0 && is_core_flags(st.dets[hs * s.R + rwords<RW>(s) + s.L]);
}

// A spawned amplitude out of the fixed point's range (spawn_amplitude's ovf),
// as the amplitude of its child.
constexpr long long kOverflow = -0x7FFFFFFFFFFFFFFFll - 1;

// attempt_create for a generated excitation: the tau-search log and the
// rounded fixed-point amplitude.  The reference first filters a core parent's
// core children (the deterministic projection makes those spawns).  Without
// the tau search, which logs the attempts that pass, the filter matters only
// for a child that comes to be, so create_particle applies it: a core
// parent's attempts are the most numerous of a semistochastic run and few of
// them spawn.
template <typename Real, int NW, int RW>
__device__ inline long long attempt_create(const DevSys &s, const DevState &st, const IterParams &p, const Parent &P,
                                           Excit<Real> &e, Stream &rng, TauAcc *tacc) {
    if (!e.ok) return 0;
    if (s.tau_search) {
        if (P.core && core_child<NW, RW>(s, st, e.child)) return 0;
        tau_log<Real>(s, e, tacc);
    }
    int ovf = 0;
    const long long q = spawn_amplitude<Real>(p, e.hel, e.invp, P.neg, rng, ovf, e.aq);
    return ovf ? kOverflow : q;
}

// The attempt of the general lattice generator, as the instance for one
// coupling runs it: out of line and on copies of its own, since it is met once
// in 2^53 draws there.
template <typename Real, int NW, int RW>
__device__ __noinline__ long long create_general(const DevSys &s, const DevState &st, const IterParams &p,
                                                 const unsigned long long w0, const int32_t *sh_neigh, TauAcc *tacc,
                                                 Excit<Real> *e) {
    Parent P;
    load_parent<NW, RW>(s, st, p, w0, P);
    Stream rng(P.key, p.iter, P_ATTEMPT, P.run, P.k);
    gen_rs_hubbard<Real, NW>(s, P.d, sh_neigh, rng, *e);
    return attempt_create<Real, NW, RW>(s, st, p, P, *e, rng, tacc);
}

// The attempt of pick_rs_uniform: finish_single and attempt_create with the
// amplitude's magnitude taken from the step's table.
template <typename Real, int NW, int RW>
__device__ inline long long create_uniform(const DevSys &s, const DevState &st, const IterParams &p, const Parent &P,
                                           int src, int tgt, int cell, const unsigned long long *sh_aq, Excit<Real> &e,
                                           Stream &rng, TauAcc *tacc) {
    NECI_FOR_WORDS(w, nwords<NW>(s)) e.child[w] = P.d[w];
    flip_orb(e.child, src);
    flip_orb(e.child, tgt);
    if (s.tau_search || s.rdm) {
        e.cls = TC_SING;
        e.hel = (Real)fabs(s.lat->t);
        e.invp = (Real)s.lat->invp[cell];
    }
    if (s.tau_search) {
        if (P.core && core_child<NW, RW>(s, st, e.child)) return 0;
        tau_log<Real>(s, e, tacc);
    }
    e.aq = sh_aq[cell];
    if (e.aq == ~0ull) return kOverflow;
    // -tau H sign(C): make_single's parity, the coupling's sign, the parent's
    const bool par = occ_between(P.d, nwords<NW>(s), min(src, tgt), max(src, tgt)) & 1;
    return round_amplitude(p, !(par ^ (s.lat->t < 0.0) ^ P.neg), e.aq, rng);
}

// The unbiasing weight of a spawn's parent for the 2-RDM (the role of
// calc_rdmbiasfac, rdm_general.fpp:1039-1085, for a per-spawn estimator):
// the expected number of non-zero spawns onto a child per attempt is
// p_gen P(nz), where P(nz) is min(1, |n| / RealSpawnCutoff) with real
// coefficients and the cutoff, min(1, |n|) with integer walkers, and 1
// otherwise; the attempts number |C_i| AvMCExcits on average, so
// sign(C_i) / (AvMCExcits p_gen P(nz)) has expectation C_i per child.
// aq is |n| in fixed point before rounding.
__device__ inline double rdm_parent_weight(const IterParams &p, double invp, unsigned long long aq, bool neg) {
    double inv_pnz = 1.0;
    if (p.t_all_real_coeff) {
        if (p.t_real_spawn_cutoff && aq < p.cutoff_q) inv_pnz = (double)p.cutoff_q / (double)aq;
    } else if (aq < (1ull << 32)) {
        inv_pnz = 4294967296.0 / (double)aq;
    }
    const double w = (invp * p.inv_av) * inv_pnz;
    return neg ? -w : w;
}

// create_particle (fcimc_helper.F90:152-308): the child's record, appended
// warp-wide, after the core filter (see attempt_create).
template <typename Real, int NW, int RW>
__device__ inline void create_particle(const DevSys &s, const DevState &st, const IterParams &p, long long qv,
                                       const Parent &P, const Excit<Real> &e) {
    bool rec = qv != 0;
    if (rec && P.core && !s.tau_search && core_child<NW, RW>(s, st, e.child)) rec = false;
    if (rec && qv == kOverflow) {
        set_err(st.ctl, NECI_GPU_ERR_OVERFLOW);
        rec = false;
    }
    const unsigned long long pos = warp_append1(&st.ctl->n_spawned, rec);
    if (!rec) return;
    if (pos >= (unsigned long long)st.max_spawned) {
        set_err(st.ctl, NECI_GPU_ERR_SPAWN_FULL);
        return;
    }
    long long *o = st.spawn + pos * s.R;
    NECI_FOR_WORDS(w, rwords<RW>(s)) o[w] = w < nwords<NW>(s) ? (long long)e.child[w] : 0ll;
    for (int k2 = 0; k2 < s.L; ++k2) o[rwords<RW>(s) + k2] = (k2 == P.run) ? qv : 0ll;
    o[rwords<RW>(s) + s.L] = P.pinit ? (1ll << init_flag_bit(P.run)) : 0ll;
    if (!s.rdm) return;
    // the parent and its unbiased sign for the 2-RDM: sign(C_i) divided
    // by the expected number of non-zero spawns onto this child per unit
    // of |C_i|, AvMCExcits p_gen P(spawn != 0)
    long long *par = st.spawn_par + pos * (rwords<RW>(s) + 1);
    NECI_FOR_WORDS(w, rwords<RW>(s)) par[w] = w < nwords<NW>(s) ? (long long)P.d[w] : 0ll;
    par[rwords<RW>(s)] = double_to_word(rdm_parent_weight(p, (double)e.invp, e.aq, P.neg));
}

// Children of a warp waiting for their record, in shared memory (molecular
// systems).  The append's counter is an atomic whose result the warp waits
// for, and the record and with 2-RDM sampling the parent's weight (an FP64
// division) cost a warp the same for one child as for 32; so the children
// wait until a warp has 32.  A round adds at most 32 doubles and 32 singles
// to fewer than 32.  The kernel with records appended round by round, and so
// (us): n = 64 with 2% of 9.8e7 attempts spawning 4745 and 4242, n = 24 with
// 14% of 9.7e6 540 and 520 (FP32 amplitudes 509 and 481), a replica pair
// with 2-RDM sampling at n = 32 and 5.9e5 attempts 53 and 47.
constexpr int kHeld = 96;
template <int NW>
struct Held {
    unsigned long long d[NW > 0 ? NW : kMaxWords][kHeld];
    long long q[kHeld];
    uint32_t mark[kHeld];  // run | initiator parent << 1 | core parent << 2 | negative parent << 3
};
// ... and with 2-RDM sampling, in dynamic shared memory
struct HeldParent {
    double invp[kHeld];
    unsigned long long aq[kHeld];
    uint32_t slot[kHeld];
};
template <typename Real, int NW>
__device__ inline void hold(const DevSys &s, Held<NW> &h, HeldParent *hp, int &n, long long qv, unsigned long long w0,
                            const Parent &P, const Excit<Real> &e) {
    const unsigned int m = __ballot_sync(0xffffffffu, qv != 0);
    if (qv != 0) {
        const int i = n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
        NECI_FOR_WORDS(w, nwords<NW>(s)) h.d[w][i] = e.child[w];
        h.q[i] = qv;
        h.mark[i] = (uint32_t)P.run | (P.pinit ? 2u : 0u) | (P.core ? 4u : 0u) | (P.neg ? 8u : 0u);
        if (hp) {
            hp->invp[i] = (double)e.invp;
            hp->aq[i] = e.aq;
            hp->slot[i] = (uint32_t)w0;
        }
    }
    n += __popc(m);
}
// create_particle for waiting children first .. first + n - 1 (n <= 32).
template <int NW, int RW>
__device__ inline void write_held(const DevSys &s, const DevState &st, const IterParams &p, const Held<NW> &h,
                                  const HeldParent *hp, int first, int n) {
    const int lane = threadIdx.x & 31, i = first + lane;
    bool rec = lane < n;
    unsigned long long c[kMaxWords];
    NECI_FOR_WORDS(w, nwords<NW>(s)) c[w] = 0ull;
    long long qv = 0;
    uint32_t mark = 0;
    if (rec) {
        NECI_FOR_WORDS(w, nwords<NW>(s)) c[w] = h.d[w][i];
        qv = h.q[i];
        mark = h.mark[i];
        if ((mark & 4u) && !s.tau_search && core_child<NW, RW>(s, st, c)) rec = false;
        if (rec && qv == kOverflow) {
            set_err(st.ctl, NECI_GPU_ERR_OVERFLOW);
            rec = false;
        }
    }
    const unsigned long long pos = warp_append1(&st.ctl->n_spawned, rec);
    if (!rec) return;
    if (pos >= (unsigned long long)st.max_spawned) {
        set_err(st.ctl, NECI_GPU_ERR_SPAWN_FULL);
        return;
    }
    const int run = (int)(mark & 1u);
    long long *o = st.spawn + pos * s.R;
    NECI_FOR_WORDS(w, rwords<RW>(s)) o[w] = w < nwords<NW>(s) ? (long long)c[w] : 0ll;
    for (int k2 = 0; k2 < s.L; ++k2) o[rwords<RW>(s) + k2] = (k2 == run) ? qv : 0ll;
    o[rwords<RW>(s) + s.L] = mark & 2u ? (1ll << init_flag_bit(run)) : 0ll;
    if (!hp) return;
    // (as in create_particle)
    long long *par = st.spawn_par + pos * (rwords<RW>(s) + 1);
    const long long *r = st.dets + (long long)hp->slot[i] * s.R;
    NECI_FOR_WORDS(w, rwords<RW>(s)) par[w] = r[w];
    par[rwords<RW>(s)] = double_to_word(rdm_parent_weight(p, hp->invp[i], hp->aq[i], (mark & 8u) != 0));
}

// Children of a warp waiting for the fused lookup, in shared memory: their
// words, amplitude and marks.  A warp holds fewer than 32 between rounds.
constexpr int kWaiting = 64;
template <int NW>
struct Waiting {
    unsigned long long d[NW > 0 ? NW : kMaxWords][kWaiting];
    long long q[kWaiting];
    uint32_t mark[kWaiting];  // run | initiator parent << 1 | core parent << 2
};

// create_particle with pass 1 of the annihilation done at once, for 32 waiting
// children of a warp (entries first .. first + n - 1): each is looked up in
// the walker hash (hash_table_lookup); one that is occupied takes the found
// branch of AnnihilateSpawnedParts (Annihilation.F90:1000-1140), its
// fixed-point amplitude, record count and initiator bit added to the slot's
// spawn sums (acc, meta), while an absent child becomes a candidate record of
// the compression pass, and a core parent's core child is dropped (the
// deterministic projection makes it).  The sums are integer atomics, so the
// order of the spawns does not matter.  Done when the host chose the fused
// lookup (spawns frequent, never with 2-RDM sampling, which needs every
// record and its parent).  The hash and the two dependent reads of a lookup
// cost a warp the same for one child as for 32, so the children wait until a
// warp has 32: looked up round by round, 13 of 32 lanes had one on the 6x6
// lattice and the lookups took half of the kernel's instructions.
// sums: the block's spawns, their number and |amplitude| per run (n_spawned
// and abs_q of the step), a place per thread in shared memory (64-bit shared
// atomics are compare-and-swap loops, which the lanes of a warp that spawn
// together go through in turn).
template <int NW, int RW>
__device__ inline void look_up(const DevSys &s, const DevState &st, Waiting<NW> &wt, int first, int n,
                               const ulonglong2 *hash_tab, unsigned long long (*sums)[128]) {
    const int lane = threadIdx.x & 31, i = first + lane;
    bool rec = lane < n;
    unsigned long long c[kMaxWords], h = 0;
    NECI_FOR_WORDS(w, nwords<NW>(s)) c[w] = 0ull;
    long long qv = 0;
    uint32_t mark = 0;
    if (rec) {
        NECI_FOR_WORDS(w, nwords<NW>(s)) c[w] = wt.d[w][i];
        qv = wt.q[i];
        mark = wt.mark[i];
        h = s.hash_tab ? hash_by_nibbles<NW>(c, s.W, hash_nibbles(s.nbasis), hash_tab)
                       : neci_hash(c, nwords<NW>(s), s.random_hash2);
        const long long slot = hash_find(st, c, nwords<NW>(s), s.R, h, st.ctl);
        bool drop = (mark & 4u) && slot >= 0 && is_core_flags(st.dets[slot * s.R + rwords<RW>(s) + s.L]);
        if (!drop && qv == kOverflow) {
            set_err(st.ctl, NECI_GPU_ERR_OVERFLOW);
            drop = true;
        }
        if (!drop) {
            const unsigned long long aq = (unsigned long long)(qv < 0 ? -qv : qv);
            sums[0][threadIdx.x] += 1ull;
            sums[1 + (mark & 1u)][threadIdx.x] += aq;
            if (slot >= 0) {
                const long long j = slot * s.L + (mark & 1u);
                atomicAdd((unsigned long long *)&st.acc[j], (unsigned long long)qv);
                atomicAdd(&st.meta[j], 1u);
                if (mark & 2u) atomicOr(&st.meta[j], 0x80000000u);
            }
        }
        rec = !drop && slot < 0;
    }
    const unsigned long long pos = warp_append1(&st.ctl->n_cand, rec);
    if (!rec) return;
    if (pos >= (unsigned long long)st.max_spawned) {
        set_err(st.ctl, NECI_GPU_ERR_SPAWN_FULL);
        return;
    }
    const int run = (int)(mark & 1u);
    long long *o = st.spawn + pos * s.R;
    NECI_FOR_WORDS(w, rwords<RW>(s)) o[w] = w < nwords<NW>(s) ? (long long)c[w] : 0ll;
    for (int k2 = 0; k2 < s.L; ++k2) o[rwords<RW>(s) + k2] = (k2 == run) ? qv : 0ll;
    o[rwords<RW>(s) + s.L] = mark & 2u ? (1ll << init_flag_bit(run)) : 0ll;
    st.cand[pos] = (uint32_t)pos;
    st.cand_h[pos] = h;
}

// One attempt of class CLS (0: double, 1: single) whose parent and stream
// are loaded: the stream stands after its first draw (the singles/doubles
// choice), so the draws are those of the attempt processed inline.
template <typename Real, int GEN, int CLS, int NW, int RW>
__device__ inline void spawn_class(const DevSys &s, const DevState &st, const IterParams &p, bool valid,
                                   unsigned long long w0, const Parent &P, Stream &rng, TauAcc *tacc, Held<NW> &held,
                                   HeldParent *hp, int &n_held) {
    Excit<Real> e;
    e.ok = false;
    long long qv = 0;
    if (valid) {
        if (CLS == 1) gen_uniform_single<Real, NW>(s, P.d, rng, e);
        else if (GEN == NECI_EXGEN_UNIFORM) gen_uniform_double<Real, NW>(s, P.d, rng, e);
        else gen_pchb_double<Real, NW>(s, P.d, rng, e);
        qv = attempt_create<Real, NW, RW>(s, st, p, P, e, rng, tacc);
    }
    hold<Real, NW>(s, held, hp, n_held, qv, w0, P, e);
}

// The parent and stream of a queued attempt: the stream resumes after its
// first draw from the saved second draw.
template <int NW, int RW>
__device__ inline Stream load_queued(const DevSys &s, const DevState &st, const IterParams &p, bool valid,
                                     unsigned long long w0, unsigned long long r1, Parent &P) {
    P.run = 0;
    P.pinit = false;
    P.key = 0;
    P.k = 0;
    if (valid) load_parent<NW, RW>(s, st, p, w0, P);
    Stream rng(P.key, p.iter, P_ATTEMPT, P.run, P.k);
    rng.resume_second(r1);
    return rng;
}

// The spawn attempts (FciMCPar.F90:1600-1745, loop_over_walkers), one
// attempt entry per thread per round; every lane runs the same number of
// rounds, so the record append is warp-wide.  Molecular systems queue their
// attempts by class (single or double) in shared memory and process full
// batches with all lanes: with QD (both classes common, chosen by the host
// from pSingles) both classes are queued; without it the doubles are
// generated at once and only the singles are queued.  Lattice systems
// (singles only) generate every attempt at once.
//
// NW is the number of words that can hold orbitals, ceil(nBasis/64), and RW
// the row's W = nBasis/64 + 1 words (NIfD + 1): one more, always zero, when
// nBasis is a multiple of 64.  Excitations are generated on NW words; the
// determinant key, the records and the row offsets use all RW.  NW = RW = 0
// is the instance for any size, with the counts read from the system.
// Resident blocks of 128 threads per SM the spawn kernel is compiled for:
// its register cap is 65536 / (128 x this).
#ifndef NECI_SPAWN_BLOCKS_PER_SM
#define NECI_SPAWN_BLOCKS_PER_SM 8
#endif

template <typename Real, int GEN, int NW, int RW, bool QD>
__global__ void __launch_bounds__(128, NECI_SPAWN_BLOCKS_PER_SM)
    k_spawn(DevSys s, DevState st, const IterParams *pp, int fuse_probe) {
    // lattice systems only: their singles spawn often enough to fill the
    // lookup's lanes; the molecular instances carry no fused code
    const bool fused = GEN == NECI_EXGEN_RS_HUBBARD && fuse_probe != 0 && !s.rdm;
    extern __shared__ __align__(16) unsigned char sh[];
    // per class: attempt entries and their second draws (at most two
    // rounds' worth are held), and each warp's appends of the round (by
    // round parity)
    __shared__ unsigned long long sq[GEN == NECI_EXGEN_RS_HUBBARD ? 1 : 2][256], sr1[GEN == NECI_EXGEN_RS_HUBBARD ? 1 : 2][256];
    __shared__ int wcnt[2][2][4];
    __shared__ unsigned int ring_tail;
    // the fused lookup of lattice systems: sums per thread, waiting children
    // per warp
    __shared__ Waiting<GEN == NECI_EXGEN_RS_HUBBARD ? NW : 1> waiting[GEN == NECI_EXGEN_RS_HUBBARD ? 4 : 1];
    __shared__ unsigned long long sh_sums[GEN == NECI_EXGEN_RS_HUBBARD ? 3 : 1][128];
    // molecular systems: the warps' children waiting for their records
    __shared__ Held<GEN == NECI_EXGEN_RS_HUBBARD ? 1 : NW> held_all[GEN == NECI_EXGEN_RS_HUBBARD ? 1 : 4];
    __shared__ long long sh_n[2];
    // the lattice instance for one coupling: the pick's bounds, the step's
    // amplitude magnitudes, the sites' neighbours
    constexpr bool uniform = GEN == NECI_EXGEN_RS_HUBBARD && QD;
    __shared__ unsigned long long sh_bound[uniform ? kMaxNeigh * kMaxNeigh : 1], sh_aq[uniform ? kMaxNeigh * kMaxNeigh : 1];
    __shared__ unsigned long long sh_nb8[uniform ? 32 * kMaxWords : 1];
    __shared__ TauAcc tacc;
    // attempts in all; sh_n[0] of them have entries (kept in shared memory:
    // the loops below are short of registers)
    if (threadIdx.x == 0) {
        // a step with more attempts than the list holds (by the sweep's 64-bit
        // count: the heavy parents' part of n_big wraps at 2^36) fails and
        // makes none: the sweep leaves out entries that do not fit, and what
        // lies in their places need not be an entry (a list read packs
        // diagonal elements there)
        const unsigned long long total = st.ctl->n_attempts, entries = st.ctl->n_att;
        const bool stop = halted(st), over = total > (unsigned long long)st.max_att;
        if (over && !stop) set_err(st.ctl, NECI_GPU_ERR_SPAWN_FULL);
        sh_n[0] = (long long)entries;
        sh_n[1] = over || stop ? 0 : (long long)total;
    }
    __syncthreads();
    // a block with no attempts leaves (the grid is sized to the capacity)
    if (sh_n[1] <= (long long)blockIdx.x * blockDim.x) return;
    const IterParams p = *pp;
    // lattice systems: the hash table of the fused lookup, the neighbour lists
    ulonglong2 *sh_hash = reinterpret_cast<ulonglong2 *>(sh);
    int32_t *sh_neigh = reinterpret_cast<int32_t *>(sh_hash + hash_tab_len(s.nbasis));
    if (fused && s.hash_tab)
        for (int i = threadIdx.x; i < hash_tab_len(s.nbasis); i += blockDim.x) sh_hash[i] = s.hash_tab[i];
    if (GEN == NECI_EXGEN_RS_HUBBARD)
        for (int i = threadIdx.x; i < s.nsites * s.max_neigh; i += blockDim.x) sh_neigh[i] = s.neighbours[i];
    if (uniform) {
        // the amplitude depends on the pick's table cell alone: the block
        // takes the magnitudes of its step once
        for (int i = threadIdx.x; i < kMaxNeigh * kMaxNeigh; i += blockDim.x) {
            Stream none(0, 0, 0, 0, 0);
            unsigned long long aq = 0;
            int over = 0;
            (void)spawn_amplitude<Real>(p, (Real)fabs(s.lat->t), (Real)s.lat->invp[i], false, none, over, aq);
            sh_bound[i] = s.lat->bound[i];
            sh_aq[i] = over ? ~0ull : aq;
        }
        for (int i = threadIdx.x; i < s.nsites; i += blockDim.x) {
            unsigned long long b = ~0ull;  // the site's neighbours, a byte each (255: none)
            for (int k = 0; k < s.max_neigh; ++k) {
                const int n = s.neighbours[i * s.max_neigh + k];
                if (n > 0) b = (b & ~(0xFFull << (8 * k))) | ((unsigned long long)(n - 1) << (8 * k));
            }
            sh_nb8[i] = b;
        }
    }
    if (threadIdx.x < 4) {
        tacc.g[threadIdx.x] = 0ull;
        tacc.c[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) ring_tail = 0u;
    if (fused)
        for (int k = 0; k < 3; ++k) sh_sums[k][threadIdx.x] = 0ull;
    __syncthreads();
    const volatile long long &n_entry = sh_n[0];
    const long long nat = sh_n[1];
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long nround = ((nat + stride - 1) / stride) * stride;
    const int nb = blockDim.x;  // 128: four warps
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int qn[2] = {0, 0};  // queue lengths, the same in every thread
    if constexpr (GEN == NECI_EXGEN_RS_HUBBARD) {
        // lattice systems (singles only): one attempt per thread per round.
        // QD marks the instance for one coupling (DevSys::lat).
        Waiting<NW> &wt = waiting[wid];
        int n_wait = 0;  // the warp's waiting children, the same in every lane
        for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nround; q += stride) {
            long long qv = 0;
            Parent P;
            P.run = 0;
            P.pinit = false;
            P.core = false;
            Excit<Real> e;
            e.ok = false;
            if (q < nat) {
                const unsigned long long w0 = attempt_entry(st, q, n_entry);
                load_parent<NW, RW>(s, st, p, w0, P);
                Stream rng(P.key, p.iter, P_ATTEMPT, P.run, P.k);
                if (QD) {
                    int src, tgt, cell;
                    if (!pick_rs_uniform<NW>(s, P.d, sh_nb8, sh_bound, rng, src, tgt, cell)) {
                        Excit<Real> eg;
                        qv = create_general<Real, NW, RW>(s, st, p, w0, sh_neigh, &tacc, &eg);
                        e = eg;
                    } else if (cell >= 0) {
                        qv = create_uniform<Real, NW, RW>(s, st, p, P, src, tgt, cell, sh_aq, e, rng, &tacc);
                    }
                } else {
                    gen_rs_hubbard<Real, NW>(s, P.d, sh_neigh, rng, e);
                    qv = attempt_create<Real, NW, RW>(s, st, p, P, e, rng, &tacc);
                }
            }
            if (!fused) {
                create_particle<Real, NW, RW>(s, st, p, qv, P, e);
                continue;
            }
            const unsigned int m = __ballot_sync(0xffffffffu, qv != 0);
            if (qv != 0) {
                const int i = n_wait + __popc(m & ((1u << lane) - 1u));
                NECI_FOR_WORDS(w, nwords<NW>(s)) wt.d[w][i] = e.child[w];
                wt.q[i] = qv;
                wt.mark[i] = (uint32_t)P.run | (P.pinit ? 2u : 0u) | (P.core ? 4u : 0u);
            }
            n_wait += __popc(m);
            if (n_wait >= 32) {
                __syncwarp();
                n_wait -= 32;
                look_up<NW, RW>(s, st, wt, n_wait, 32, sh_hash, sh_sums);
                __syncwarp();
            }
        }
        if (fused) {
            __syncwarp();
            look_up<NW, RW>(s, st, wt, 0, n_wait, sh_hash, sh_sums);
        }
    }
    // Molecular systems without QD (singles rare or dominant): a round
    // classifies one attempt per thread (gen_exc_sd: r < pSingles is a
    // single; gen_rand_excit: r < pDoubles is a double), generates a double
    // at once, inline, and appends a single to a ring of 512 entries.  The
    // ring's tail only grows (shared atomics); the round's barrier is a
    // __syncthreads_count, which gives every thread the round's appends, so
    // the queue length and head are kept in registers, the same in every
    // thread.  A full batch (or after the last attempt what is left) is read
    // at once and processed: the next round's appends land at least 128 and
    // less than 512 entries past the head, never on an entry being read.
    if constexpr (GEN != NECI_EXGEN_RS_HUBBARD && !QD) {
        unsigned long long *ring = &sq[0][0], *ring_r1 = &sr1[0][0];  // 512 entries each
        Held<NW> &held = held_all[wid];
        HeldParent *hp = s.rdm ? reinterpret_cast<HeldParent *>(sh) + wid : nullptr;
        int n_held = 0;  // the same in every lane of the warp
        unsigned int head = 0;
        int cnt = 0;
        long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
        for (;; q += stride) {
            const bool more = q - threadIdx.x < nround;  // the same in the whole block
            bool single = false;
            unsigned long long w0 = 0, r1 = 0;
            if (more) {
                Parent P;
                P.run = 0;
                P.pinit = false;
                Excit<Real> e;
                e.ok = false;
                long long qv = 0;
                if (q < nat) {
                    w0 = attempt_entry(st, q, n_entry);
                    load_parent<NW, RW>(s, st, p, w0, P);
                    Stream rng(P.key, p.iter, P_ATTEMPT, P.run, P.k);
                    const unsigned long long r0 = rng.next64();
                    single = GEN == NECI_EXGEN_UNIFORM ? !(r0 < s.thr_doubles) : r0 < s.thr_singles;
                    if (single) {
                        r1 = rng.next64();
                    } else {
                        if (GEN == NECI_EXGEN_UNIFORM) gen_uniform_double<Real, NW>(s, P.d, rng, e);
                        else gen_pchb_double<Real, NW>(s, P.d, rng, e);
                        qv = attempt_create<Real, NW, RW>(s, st, p, P, e, rng, &tacc);
                    }
                }
                hold<Real, NW>(s, held, hp, n_held, qv, w0, P, e);
            }
            if (single) {
                const unsigned int t = atomicAdd(&ring_tail, 1u) & 511u;
                ring[t] = w0;
                ring_r1[t] = r1;
            }
            cnt += __syncthreads_count(single);
            const int take = cnt >= nb ? nb : (more ? 0 : cnt);
            if (take) {
                const bool v = (int)threadIdx.x < take;
                const unsigned int i = (head + threadIdx.x) & 511u;
                const unsigned long long a = v ? ring[i] : 0ull, b = v ? ring_r1[i] : 0ull;
                head += (unsigned int)take;
                cnt -= take;
                Parent P;
                Stream rng = load_queued<NW, RW>(s, st, p, v, a, b, P);
                spawn_class<Real, GEN, 1, NW, RW>(s, st, p, v, a, P, rng, &tacc, held, hp, n_held);
            }
            // 32 records at once; after the last attempt what is left
            __syncwarp();
            while (n_held >= (more ? 32 : 1)) {
                const int n = min(n_held, 32);
                n_held -= n;
                write_held<NW, RW>(s, st, p, held, hp, n_held, n);
                __syncwarp();
            }
            if (!more && cnt == 0) break;
        }
    }
    // Molecular systems with QD (both classes common): a round classifies
    // one attempt per thread and queues it by class; full batches of a queue
    // are processed with all lanes, so neither class idles the lanes of the
    // other (half of them after the tau search raises pSingles near 1/2).
    // In the rounds after the last attempt the queues are emptied.  Each
    // class is processed by one call site, so its generator is compiled once.
    //
    // Queue appends: each warp posts its counts per class; after one barrier
    // every thread derives the same queue lengths and its own slot, so no
    // shared counter is read and written in the same round.  A round that
    // drains takes a second barrier (its entries visible) and reads its
    // entries at once; the next round writes only after its own first
    // barrier, by which time every thread has read them.
    if constexpr (GEN != NECI_EXGEN_RS_HUBBARD && QD) {
        Held<NW> &held = held_all[wid];
        HeldParent *hp = s.rdm ? reinterpret_cast<HeldParent *>(sh) + wid : nullptr;
        int n_held = 0;  // the same in every lane of the warp
        long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
        for (int round = 0;; ++round, q += stride) {
            const bool more = q - threadIdx.x < nround;  // the same in the whole block
            const bool valid = more && q < nat;
            int cls = 0;
            unsigned long long w0 = 0, r1 = 0;
            if (valid) {
                w0 = attempt_entry(st, q, n_entry);
                Stream rng = attempt_stream(st, p, w0);
                const unsigned long long r0 = rng.next64();
                r1 = rng.next64();
                cls = (GEN == NECI_EXGEN_UNIFORM ? !(r0 < s.thr_doubles) : r0 < s.thr_singles) ? 1 : 0;
            }
            const bool queued = valid;
            unsigned int m[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                m[c] = __ballot_sync(0xffffffffu, queued && cls == c);
                if (lane == 0) wcnt[round & 1][c][wid] = __popc(m[c]);
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                int before = 0, total = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int x = wcnt[round & 1][c][w];
                    before += w < wid ? x : 0;
                    total += x;
                }
                if (queued && cls == c) {
                    const int pos = qn[c] + before + __popc(m[c] & ((1u << lane) - 1u));
                    sq[c][pos] = w0;
                    sr1[c][pos] = r1;
                }
                qn[c] += total;
            }
            // a full batch, or after the last attempt what is left
            const int t0 = qn[0] >= nb ? nb : (more ? 0 : qn[0]);
            const int t1 = qn[1] >= nb ? nb : (more ? 0 : qn[1]);
            if (t0 || t1) {
                __syncthreads();
                bool v0 = false, v1 = false;
                unsigned long long a0 = 0, b0 = 0, a1 = 0, b1 = 0;
                if (t0) {
                    qn[0] -= t0;
                    v0 = (int)threadIdx.x < t0;
                    if (v0) {
                        a0 = sq[0][qn[0] + threadIdx.x];
                        b0 = sr1[0][qn[0] + threadIdx.x];
                    }
                }
                if (t1) {
                    qn[1] -= t1;
                    v1 = (int)threadIdx.x < t1;
                    if (v1) {
                        a1 = sq[1][qn[1] + threadIdx.x];
                        b1 = sr1[1][qn[1] + threadIdx.x];
                    }
                }
                if (t0) {
                    Parent P;
                    Stream rng = load_queued<NW, RW>(s, st, p, v0, a0, b0, P);
                    spawn_class<Real, GEN, 0, NW, RW>(s, st, p, v0, a0, P, rng, &tacc, held, hp, n_held);
                }
                if (t1) {
                    Parent P;
                    Stream rng = load_queued<NW, RW>(s, st, p, v1, a1, b1, P);
                    spawn_class<Real, GEN, 1, NW, RW>(s, st, p, v1, a1, P, rng, &tacc, held, hp, n_held);
                }
            }
            // 32 records at once; after the last attempt what is left
            __syncwarp();
            while (n_held >= (more ? 32 : 1)) {
                const int n = min(n_held, 32);
                n_held -= n;
                write_held<NW, RW>(s, st, p, held, hp, n_held, n);
                __syncwarp();
            }
            if (!more && qn[0] == 0 && qn[1] == 0) break;
        }
    }
    // n_spawned and abs_q of the spawns created here (otherwise pass 1 counts
    // them)
    if (fused) {
        __syncthreads();
        if (wid < 3) {
            unsigned long long t = 0;
            for (int i = lane; i < 128; i += 32) t += sh_sums[wid][i];
            t = warp_sum_u(t);
            if (lane == 0 && t) atomicAdd(wid == 0 ? &st.ctl->n_spawned : &st.ctl->abs_q[wid - 1], t);
        }
    }
    if (s.tau_search) {
        __syncthreads();
        if (threadIdx.x < 4) {
            if (tacc.g[threadIdx.x]) atomicMax(&st.ctl->tau_gamma[threadIdx.x], tacc.g[threadIdx.x]);
            if (tacc.c[threadIdx.x]) atomicAdd(&st.ctl->tau_cnt[threadIdx.x], (unsigned long long)tacc.c[threadIdx.x]);
        }
    }
}

// Grids are sized to the context's capacity (as in kernels.cu).
// The grid fills spawn_occ blocks per SM (8, the launch bound, unless tuned).
inline int spawn_grid(const Engine &e, int threads) {
    const long long want = e.st.max_spawned / (threads * 4 * e.share) + 1, hi = (long long)e.num_sms * e.spawn_occ;
    return (int)(want < 8 ? 8 : (want > hi ? hi : want));
}

// Doubles are queued like singles when both classes are common: the
// fraction of singles between 0.15 and 0.85 (on GB300, at 0.53 queueing
// both made the spawn kernel 17% faster; with rare singles it is slower).
inline int spawn_queue_doubles(const DevSys &s) {
    const double ps = s.excitgen == NECI_EXGEN_UNIFORM ? 1.0 - s.p_doubles : s.p_singles;
    return ps >= 0.15 && ps <= 0.85 ? 1 : 0;
}

template <typename Real, int GEN, bool QD>
void launch_spawn_words(Engine &e, cudaStream_t s, int grid, size_t shm) {
    const int rw = e.sys.W, nw = (e.sys.nbasis + 63) / 64;
    if (rw == 1) k_spawn<Real, GEN, 1, 1, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
    else if (rw == 2 && nw == 1) k_spawn<Real, GEN, 1, 2, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
    else if (rw == 2) k_spawn<Real, GEN, 2, 2, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
    else if (rw == 3 && nw == 2) k_spawn<Real, GEN, 2, 3, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
    else if (rw == 3) k_spawn<Real, GEN, 3, 3, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
    else k_spawn<Real, GEN, 0, 0, QD><<<grid, 128, shm, s>>>(e.sys, e.st, e.d_params, fused_lookup(e) ? 1 : 0);
}

template <typename Real, int GEN>
void launch_spawn_gen(Engine &e, cudaStream_t s, int grid, size_t shm) {
    const bool qd = GEN == NECI_EXGEN_RS_HUBBARD ? e.sys.lat != nullptr : spawn_queue_doubles(e.sys) != 0;
    if (qd) launch_spawn_words<Real, GEN, true>(e, s, grid, shm);
    else launch_spawn_words<Real, GEN, false>(e, s, grid, shm);
}

// The spawn kernel for amplitudes in precision Real.
template <typename Real>
void launch_spawn_real(Engine &e, cudaStream_t s) {
    const size_t shm = e.sys.excitgen == NECI_EXGEN_RS_HUBBARD
                           ? (size_t)hash_tab_len(e.sys.nbasis) * sizeof(ulonglong2) +
                                 (size_t)(e.sys.nsites * e.sys.max_neigh) * sizeof(int32_t)
                           : (e.sys.rdm ? 4 * sizeof(HeldParent) : 0);
    const int grid = spawn_grid(e, 128);
    if (e.sys.excitgen == NECI_EXGEN_RS_HUBBARD) launch_spawn_gen<Real, NECI_EXGEN_RS_HUBBARD>(e, s, grid, shm);
    else if (e.sys.excitgen == NECI_EXGEN_UNIFORM) launch_spawn_gen<Real, NECI_EXGEN_UNIFORM>(e, s, grid, shm);
    else launch_spawn_gen<Real, NECI_EXGEN_PCHB>(e, s, grid, shm);
}

}  // namespace neci
