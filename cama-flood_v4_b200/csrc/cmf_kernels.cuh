// cmf_kernels.cuh -- sm_100a device code of the CaMa-Flood physics time step (FP64).
//
// One outer step (CMF_PHYSICS_ADVANCE, src/cmf_ctrl_physics_mod.F90:21-153) is
//   k_stage   stage scheme at the start of the step + CFL minimum      (:54-59, :161-210)
//   k_ntdt    NT/DT per member, loop bound of the device-side sub-step loop (:205-206)
//   NT x { k_flux  outflow + dam + bifurcation flux         (CMF_CALC_OUTFLW, CMF_DAMOUT_CALC,
//                                                            CMF_CALC_PTHOUT / CMF_LEVEE_OPT_PTHOUT)
//          k_rate  storage-out gather and outflow limiter rate (LSPAMAT steps 1-2); advances the
//                  sub-step counter and the loop condition
//          k_store rescale + inflow gather + dam balance + CALC_VARS_PRE + CMF_CALC_STONXT +
//                  stage scheme + sub-step diagnostics        (LSPAMAT steps 2-3, :101-135)
//        }
//   k_budget  deterministic budget reduction of every member's last sub-step
// Three grid-wide dependencies per sub-step remain (outflow needs the downstream stage; the rate
// needs the upstream outflows; the inflow needs the downstream and upstream rates), so each
// phase is one kernel and the phases are ordered by the graph.
//
// Arithmetic follows the reference statement by statement, compiled with -fmad=false so no
// multiply-add is fused: x**(-1) is 1/x, x**2 is x*x, x**0.5 is an IEEE square root, the depth
// powers of the flux formulas are correctly rounded (pow_depth) and every other non-integral power
// is pow().  Default-real literals of the reference are promoted float values
// (F(...) below).  All gathers sum in the reference's loop order (ascending upstream sequence);
// there are no atomics on state, so results are independent of block size and timing.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#define CMF_F(x) ((double)(float)(x))

namespace cmf {

// Occupancy of the latency-bound cell kernels: at most kCellThreads threads per block and the
// minimum resident blocks per SM (caps registers at 65536 / (threads x blocks)).  k_flux and
// k_store come in two profiles, one of the dimensions the engine's autotuner searches.  Measured per
// launch (us; 16 members of 298,554 cells | one of 1,997,296): k_flux at 6 blocks 262 | 126, 5 blocks 223 |
// 117, 4 blocks 228 | 120, 3 blocks 263 | 135; k_store at 5 blocks 270 | 130, 4 blocks 268 | 135, 3 blocks
// 309 | 159; k_rate at 8 blocks 90 | 49, 6 blocks 88 | 49, 4 blocks 117 | 64.  Both profiles execute the
// same arithmetic; only the register allocation differs.
constexpr int kFluxMinBlocksWide = 5, kStoreMinBlocksWide = 5;
constexpr int kFluxMinBlocksSmall = 4, kStoreMinBlocksSmall = 4;
constexpr size_t kSmallCellMembers = size_t(1) << 19;   // untuned start: `small` up to this many cell-members
#ifndef CMF_STAGE_MINB
#define CMF_STAGE_MINB 6
#endif
constexpr int kCellThreads = 256;
constexpr int kUpSlots = 4;        // upstream cells per cell held in Net::up_ell

constexpr int kBudgets = 12;       // stopre stonxt stonew rivinf rivout stopre2 stonew2 rivsto fldsto fldare levsto dammiss
// dynamic shared memory of k_store: the last sub-step's budget terms, kBudgets per thread
inline size_t store_smem(int block) { return (size_t)kBudgets * block * sizeof(double); }
constexpr int kNtCap = 10000;      // bound of the device-side sub-step loop
// MemberCtl.err codes (mapped to the ABI's positive statuses by the engine)
constexpr int kErrNtCap = 2;       // DT_MIN non-finite or NT above kNtCap: no sub-step ran
constexpr int kErrNonFinite = 3;   // a sub-step produced a non-finite storage

struct MemberCtl {
    double dt_def;                 // DT at entry (DT_DEF)
    double dt;                     // sub-step DT
    double dt_min;                 // CFL minimum of this outer step
    double nadd;                   // NADD_adp before the current sub-step
    unsigned long long dtmin_bits; // atomicMin target (positive doubles order like their bit patterns)
    int nt;                        // sub-steps of this outer step
    int it;                        // index of the next sub-step
    int err;
    int bar_err;                   // member 0: a bounded wait of the persistent kernel ran out
    double budget[kBudgets];       // last finished sub-step
};

constexpr int kNtHist = 64;       // NT histogram bins (the last one holds NT >= kNtHist-1)

struct LoopCtl {
    int k;            // sub-step counter of the device-side loop (advanced by k_rate)
    int kcur;         // the sub-step the running k_flux/k_rate/k_store work on (set by k_flux)
    int ntmax;        // max NT over members
    int err;
    int split;        // 1 until the first sub-step after a host state upload: D2RIVOUT /= D2RIVOUT_PRE
    long long member_substeps;   // sum over outer steps and members of NT (throughput accounting)
    long long loop_iters;        // sum over outer steps of NTmax (kernel-launch accounting)
    long long outer_steps;
    long long near_int;          // (outer step, member) pairs whose DT_DEF/DT_MIN-0.01 lay within
                                 // 1e-12 (relative) of an integer: NT there hangs on DT_MIN's last bits
    long long nt_hist[kNtHist];  // (outer step, member) pairs by NT
    unsigned bar;                // grid-barrier arrival count of the persistent kernel (zeroed per launch)
};

// Static data shared by all members (device pointers).
struct Net {
    int N, R, L, P, Lp, M;
    const int *__restrict__ next;       // [N] 0-based downstream (river cells)
    const int *__restrict__ up_ptr;     // [N+1] upstream CSR, ascending sequence (I1UPST order)
    const int *__restrict__ up_idx;
    // [kUpSlots][N] the first upstream cells of each cell in I1UPST order, -1 past the last; with
    // more than kUpSlots of them the last slot holds -2 - (CSR position of the kUpSlots-th), and the
    // walk goes on in up_idx.  All slots of a cell are read at once, so the upstream values are
    // gathered one dependent load after the cell's own reads instead of two (pointer, index, value).
    const int *__restrict__ up_ell;
    const int *__restrict__ i2mask;     // [N]
    const double *__restrict__ rivelv, *__restrict__ elevtn, *__restrict__ nxtdst, *__restrict__ rivwth;
    const double *__restrict__ rivhgt, *__restrict__ rivlen, *__restrict__ rivman, *__restrict__ grarea;
    const double *__restrict__ rivstomax, *__restrict__ dwnelv;
    const double *__restrict__ next_rivelv;  // [N] D2RIVELV of the downstream cell (its own at mouths)
    // D2NXTDST**(-1), D2RIVWTH**(-1), D2RIVLEN**(-1) of the outflow formulas, computed once at init
    // (the same correctly rounded reciprocal the reference evaluates every time)
    const double *__restrict__ inv_nxtdst, *__restrict__ inv_rivwth, *__restrict__ inv_rivlen;
    const double *__restrict__ fldstomax, *__restrict__ fldgrd, *__restrict__ fldhgt;   // [L][N]
    // bifurcation paths
    const int *__restrict__ pth_up, *__restrict__ pth_dn;   // [P] 0-based, -1 outside domain
    const int *__restrict__ pth_skip;                        // [P] bit0 plain/LSPAMAT skip, bit1 levee skip, bits 2
                                                             // and 3: a levee fraction below 1 at the ends
    const double *__restrict__ pth_dst, *__restrict__ pth_elv, *__restrict__ pth_wth, *__restrict__ pth_man;
    // the ends of paths: per cell its range of entries (path_ends [N], read where C_PATH is set), the
    // cell's I1P_OUT paths and then its I1P_INF paths, each in list order.  An entry holds the path
    // (x, ~path for I1P_INF) and the cell at its other end (y; -1: not rescaled, -2: the cell is
    // not this path's end), so a path's flow and the rate it may need come one load after the entry.
    const int2 *__restrict__ path_ends;
    const int2 *__restrict__ pend;
    // levee (compact per levee cell)
    const int *__restrict__ lev_id;     // [N] -1 when the cell carries the no-levee sentinels
    const double *__restrict__ levhgt, *__restrict__ levfrc, *__restrict__ bashgt, *__restrict__ levdst;
    const double *__restrict__ levbassto, *__restrict__ levtopsto, *__restrict__ levfilsto;
    // dams
    const int *__restrict__ dam_id;     // [N] compact dam of the cell or -1
    const int *__restrict__ dam_stat;   // [D]
    // what a cell takes part in (CellFlag), and the cells of reservoir operation (I1DAM > 0), which run
    // in warps of their own: one such lane made its whole warp walk the rules' dependent loads and powers
    const unsigned char *__restrict__ cflag;                 // [N]
    const int *__restrict__ dam_cells;                       // kinematic cells first, then the dams
    int ndam_cells;
    // by position in dam_cells: the cell's position [N], its upstream cells that feed a dam's inflow
    // (I1DAM 10 or 11, I1UPST order), and the static factors of the kinematic velocities
    const int *__restrict__ dam_pos, *__restrict__ dam_up_ptr, *__restrict__ dam_up_idx;
    const double *__restrict__ kin_vel, *__restrict__ kin_velf;
    const double *__restrict__ qn, *__restrict__ qf, *__restrict__ qa, *__restrict__ convol;
    const double *__restrict__ emevol, *__restrict__ norvol, *__restrict__ adjvol, *__restrict__ r_volupa;
    double pgrv, pmanfld, pdstmth, pcadp, pminslp, dfrcinc;
    int ladpstp, lfldout, lpthout, ldamout, llevee, ldamh22, ldiag;
    int ldiag_out;   // CMF_DIAG_AVEMAX_OUTPUT after every outer step, fused into its last sub-step
};

enum CellFlag : unsigned {
    C_DAM = 1,                 // I1DAM > 0: outflow by cell_dam
    C_KIN = 2,                 // I1DAM == 10 on a river cell: kinematic outflow upstream of a dam
    C_DAMID = 4,               // a dam's storage stands here
    C_PATH = 8,                // paths in the cell's lists (I1P_OUT, I1P_INF)
    C_LEV = 16,                // levee parameters
    C_END = 32                 // an end of a path (PTH_UPST, PTH_DOWN): the path reads its storage and depths
};

// What the phase kernels keep per cell beside the arrays (State::wet): which of the arrays that are zero
// in most cells hold something.  A clear bit means that they hold +0, so a dry cell neither reads nor
// writes them (about 110 of 540 B per cell and sub-step); the averages' bits are of the running outer step.
enum WetBit : unsigned {
    W_STAGE = 1,               // fldsto, flddph, fldfrc, levsto, levdph
    W_PRE = 2,                 // fldsto_pre
    W_FOUT = 4,                // fldout_pre
    W_AFLD = 8,                // a_fldout has been started (else 0)
    W_AOUT = 16                // a_outflw has parted from a_rivout (else equal: fldout was +0 so far)
};

// Per-member state, member-major [M][N] (paths [M][Lp][P] / [M][P]).
struct State {
    double *rivsto, *fldsto, *levsto, *damsto, *daminf;
    // (river, floodplain) outflow before the LSPAMAT rescale (phase A -> B), and after it where the cell's
    // own rate applies (B -> C): one 16-byte element per neighbour gather
    double2 *raw, *out;
    double2 *dph;                             // (D2RIVDPH, D2RIVDPH_PRE) during the sub-steps of the phase kernels
    unsigned char *wet;                       // WetBit
    double *rivout_pre, *fldout_pre;          // D2RIVOUT_PRE / D2FLDOUT_PRE (== D2RIVOUT / D2FLDOUT after a step)
    double *rivout_cur, *fldout_cur;          // host-set D2RIVOUT / D2FLDOUT while LoopCtl.split
    double *rivdph_pre, *fldsto_pre;
    double *rivdph, *flddph, *fldfrc, *fldare, *sfcelv, *storge, *levdph, *rivvel;
    double *rivinf, *fldinf, *pthout, *outflw, *rate;
    double *pthflw_raw, *pthflw_pre, *pthsum_raw, *pthsum;
    double *runoff;
    // sub-step diagnostics
    double *a_rivout, *a_fldout, *a_outflw, *a_rivvel, *a_pthout, *a_runoff, *a_daminf;
    double *m_storge, *m_outflw, *m_rivdph, *a_pthflw, *a_pthsum;
    // output-interval averages and maxima (D2*_oAVG, D2*_oMAX, D1PTHFLW_oAVG, NADD_out per member)
    double *o_rivout, *o_fldout, *o_outflw, *o_rivvel, *o_pthout, *o_runoff, *o_daminf;
    double *om_storge, *om_outflw, *om_rivdph, *o_pthflw, *o_nadd;
    MemberCtl *ctl;
    LoopCtl *loop;
    double *partials;                         // [M][nblk][kBudgets]
};

__device__ __forceinline__ double dmax(double a, double b) { return (a > b) ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return (a < b) ? a : b; }

// The per-cell code reads and writes a cell through an accessor, so that the same arithmetic runs on
// arrays in global memory (OwnG, the phase kernels) and on state held on the SM (OwnR, the resident
// kernel).  Static maps are indexed by the cell i and read through the read-only path, member state
// by g = m*N + i; `nb` reads a value another cell or path owns.
#define CMF_OWN_STATIC(name) \
    __device__ __forceinline__ double name(int i) const { return __ldg(&n.name[i]); }
#define CMF_OWN_STATE(name) \
    __device__ __forceinline__ double name(size_t g) const { return s.name[g]; }
struct OwnMaps {
    const Net &n;
    CMF_OWN_STATIC(rivelv) CMF_OWN_STATIC(elevtn) CMF_OWN_STATIC(nxtdst) CMF_OWN_STATIC(rivwth)
    CMF_OWN_STATIC(rivhgt) CMF_OWN_STATIC(rivlen) CMF_OWN_STATIC(rivman) CMF_OWN_STATIC(grarea)
    CMF_OWN_STATIC(rivstomax) CMF_OWN_STATIC(inv_nxtdst) CMF_OWN_STATIC(inv_rivwth) CMF_OWN_STATIC(inv_rivlen)
    __device__ __forceinline__ int next(int i) const { return __ldg(&n.next[i]); }
    __device__ __forceinline__ int up_lo(int i) const { return __ldg(&n.up_ptr[i]); }
    __device__ __forceinline__ int up_hi(int i) const { return __ldg(&n.up_ptr[i + 1]); }
    __device__ __forceinline__ int up_slot(int k, int i) const { return __ldg(&n.up_ell[(size_t)k * n.N + i]); }
};
struct LazyRate;
// What phase B leaves of an outflow: a positive one (and a mouth's) is rescaled by its own cell's rate here, and
// its gatherer takes the product; a reverse one keeps its value (not > 0) and is multiplied by the gatherer's
// rate.  Where the own rate takes a positive outflow to zero or below it (the rate of an overdrawn cell, which
// net runoff below zero makes, is negative) the product would pass for a reverse flow: NaN stands there, and
// whose sums come out NaN takes them again from the pairs before the rescale, by their signs (each_by_sign).
__device__ __forceinline__ double2 rescale_own(double rout, double fout, double r, bool mouth) {
    if (rout > 0.0 || mouth) {
        rout = rout * r;
        fout = fout * r;
        if (!(rout > 0.0) && !mouth) rout = __longlong_as_double(0x7ff8000000000000ll);
    }
    return make_double2(rout, fout);
}
struct DownCell {
    double rivelv, rivdph, rivdph_pre;
};
struct OwnG : OwnMaps {
    static constexpr bool kResident = false;
    const State &s;
    unsigned fl, wet;          // the cell's CellFlag and WetBit bits
    __device__ __forceinline__ OwnG(const Net &n_, const State &s_, unsigned fl_ = 0u, unsigned wet_ = 0u)
        : OwnMaps{n_}, s(s_), fl(fl_), wet(wet_) {}
    __device__ __forceinline__ unsigned flags() const { return fl; }
    CMF_OWN_STATE(rivsto) CMF_OWN_STATE(rivout_pre) CMF_OWN_STATE(runoff) CMF_OWN_STATE(a_rivvel) CMF_OWN_STATE(a_rivout)
    CMF_OWN_STATE(a_pthout) CMF_OWN_STATE(m_outflw) CMF_OWN_STATE(m_rivdph) CMF_OWN_STATE(m_storge)
    __device__ __forceinline__ LazyRate rate(size_t g) const;
#define CMF_OWN_SPARSE(name, bit) \
    __device__ __forceinline__ double name(size_t g) const { return (wet & bit) ? s.name[g] : 0.0; }
    CMF_OWN_SPARSE(fldsto, W_STAGE) CMF_OWN_SPARSE(flddph, W_STAGE) CMF_OWN_SPARSE(fldfrc, W_STAGE)
    CMF_OWN_SPARSE(levsto, W_STAGE) CMF_OWN_SPARSE(fldsto_pre, W_PRE) CMF_OWN_SPARSE(fldout_pre, W_FOUT)
    CMF_OWN_SPARSE(a_fldout, W_AFLD)
#undef CMF_OWN_SPARSE
    __device__ __forceinline__ double a_outflw(size_t g) const { return (wet & W_AOUT) ? s.a_outflw[g] : s.a_rivout[g]; }
    __device__ __forceinline__ double rivdph(size_t g) const { return s.dph[g].x; }
    __device__ __forceinline__ double rivdph_pre(size_t g) const { return s.dph[g].y; }
    __device__ __forceinline__ double2 own_raw(size_t g) const { return s.raw[g]; }
    __device__ __forceinline__ double2 own_out(size_t g) const { return s.out[g]; }
    __device__ __forceinline__ double nb(const double *p, size_t g) const { return p[g]; }
    __device__ __forceinline__ DownCell down(size_t base, int i, int j) const {
        const double2 d = s.dph[base + j];
        return {__ldg(&n.next_rivelv[i]), d.x, d.y};
    }
    __device__ __forceinline__ void put_raw(size_t g, int, double rout, double fout) const { s.raw[g] = make_double2(rout, fout); }
    __device__ __forceinline__ void put_rate(size_t g, int i, double rout, double fout, double r) const {
        s.rate[g] = r;
        s.out[g] = rescale_own(rout, fout, r, i >= n.R);
    }
    __device__ __forceinline__ void put_a_rivvel(size_t g, double v) const { s.a_rivvel[g] = v; }
    // an array that holds +0 while `bit` is clear
    __device__ __forceinline__ void put_sparse(unsigned bit, double *p, size_t g, double v) {
        const bool some = __double_as_longlong(v) != 0;
        if (some || (wet & bit)) p[g] = v;
        wet = some ? wet | bit : wet & ~bit;
    }
    // CALC_VARS_PRE (src/cmf_ctrl_physics_mod.F90:254-277)
    __device__ __forceinline__ void put_pre(size_t g, double rout, double fout, double dph, double fld, bool last) {
        s.rivout_pre[g] = rout;
        put_sparse(W_FOUT, s.fldout_pre, g, fout);
        put_sparse(W_PRE, s.fldsto_pre, g, fld);
        if (last) s.rivdph_pre[g] = dph;
    }
    // `dph`: the depth this one replaces (CALC_VARS_PRE's)
    template <class Out>
    __device__ __forceinline__ void put_stage(size_t g, const Out &o, double storge, double dph, bool last) {
        s.rivsto[g] = o.rivsto;
        s.dph[g] = make_double2(o.rivdph, dph);
        const bool some = (__double_as_longlong(o.fldsto) | __double_as_longlong(o.flddph) | __double_as_longlong(o.fldfrc) |
                           __double_as_longlong(o.levsto) | __double_as_longlong(o.levdph)) != 0;
        if (some || (wet & W_STAGE)) {
            s.fldsto[g] = o.fldsto;
            s.flddph[g] = o.flddph;
            s.fldfrc[g] = o.fldfrc;
            if (n.llevee) {
                s.levsto[g] = o.levsto;
                s.levdph[g] = o.levdph;
            }
        }
        wet = some ? wet | W_STAGE : wet & ~W_STAGE;
        if (last) s.rivdph[g] = o.rivdph;
        if (last || (fl & C_END)) s.storge[g] = storge;      // read by the paths at this cell
    }
    // f(rivout, fldout) before the LSPAMAT rescale of every upstream cell, in I1UPST order: the CSR
    // walk, since at k_rate's full occupancy the slot table's 16 B per cell cost more than its saved round
    template <class F>
    __device__ __forceinline__ void each_raw(size_t base, int i, F f) const {
        const int u1 = up_hi(i);
        for (int k = up_lo(i); k < u1; k++) {
            const double2 v = s.raw[base + __ldg(&n.up_idx[k])];
            f(v.x, v.y);
        }
    }
    // f(rivout, fldout) after the rescale (:481-489); next(j) == i, so a reverse flow takes rate_i
    template <class Rate, class F>
    __device__ __forceinline__ void each_out(size_t base, int i, Rate rate_i, F f) const;
    // the same from the pairs before the rescale (see rescale_own)
    template <class F>
    __device__ __forceinline__ void each_by_sign(size_t base, int i, double rate_i, F f) const;
};
// the cell's rate, read only where a reverse flow or a path needs it
struct LazyRate {
    const double *p;
    bool cg;                   // past L1: other CTAs of the same launch wrote it
    __device__ __forceinline__ operator double() const { return cg ? __ldcg(p) : *p; }
};
#undef CMF_OWN_STATIC
#undef CMF_OWN_STATE

// f(j) for every upstream cell j of cell i, in I1UPST order.  The CSR walk past the slots reads four
// indices at once (D8 networks have at most seven upstream cells), each f follows without another
// dependent round.
template <class Own, class F>
__device__ __forceinline__ void for_each_upstream(const Net &n, const Own &w, int i, F f) {
    int slot[kUpSlots];
#pragma unroll
    for (int k = 0; k < kUpSlots; k++) slot[k] = w.up_slot(k, i);
#pragma unroll
    for (int k = 0; k < kUpSlots - 1; k++) {
        if (slot[k] < 0) return;
        f(slot[k]);
    }
    const int last = slot[kUpSlots - 1];
    if (last >= 0) {
        f(last);
    } else if (last < -1) {                       // more than kUpSlots upstream cells
        const int k1 = __ldg(&n.up_ptr[i + 1]);
        for (int k = -2 - last; k < k1; k += 4) {
            int j[4];
#pragma unroll
            for (int e = 0; e < 4; e++) j[e] = k + e < k1 ? __ldg(&n.up_idx[k + e]) : -1;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (j[e] >= 0) f(j[e]);
        }
    }
}
__device__ __forceinline__ LazyRate OwnG::rate(size_t g) const { return {s.rate + g, false}; }
template <class Rate, class F>
__device__ __forceinline__ void rescaled(double2 v, Rate rate_i, F f) {
    if (!(v.x > 0.0) && !(v.x == 0.0 && v.y == 0.0)) {        // zeros stay zeros
        const double r = rate_i;
        v.x = v.x * r;
        v.y = v.y * r;
    }
    f(v.x, v.y);
}
template <class Rate, class F>
__device__ __forceinline__ void OwnG::each_out(size_t base, int i, Rate rate_i, F f) const {
    for_each_upstream(n, *this, i, [&](int j) { rescaled(s.out[base + j], rate_i, f); });
}
// f(rivout, fldout) of one flow by the rate its sign before the rescale names: its own cell's or the gatherer's
template <class F>
__device__ __forceinline__ void by_sign(double2 raw, double own, double below, F f) {
    const double r = raw.x > 0.0 ? own : below;
    f(raw.x * r, raw.y * r);
}
template <class F>
__device__ __forceinline__ void OwnG::each_by_sign(size_t base, int i, double rate_i, F f) const {
    for (int k = up_lo(i); k < up_hi(i); k++) {
        const size_t g = base + __ldg(&n.up_idx[k]);
        by_sign(s.raw[g], s.rate[g], rate_i, f);
    }
}


// x**(-7._JPRB/3._JPRB) and x**(-4._JPRB/3._JPRB) of the local-inertial flux formulas
// (src/cmf_calc_outflw_mod.F90:74,106,133,162; src/cmf_calc_pthout_mod.F90:67;
// src/cmf_ctrl_levee_mod.F90:553,573): pow(x, y) for the
// doubles y nearest -7/3 and -4/3, correctly rounded, for the positive depths these formulas take.
// The exponent is y = -K/3 + d with d its rounding offset (d = -0x1.5555555555555p-53 for K = 7,
// +0x1.5555555555555p-54 for K = 4), so x^y = (x^(-1/3))^K * x^d:
//   c0: single-precision exp2(-log2(x)/3) (a few units of 2^-21) and one step of third order in double,
//     c0 (1 + r/3 + 2 r^2/9), r = 1 - x c0^3, which leaves a few ulp; then one Newton step for the
//     inverse cube root, c = c0 (1 + r/3), with c0^3 formed exactly by Dekker's FMA products (c carried
//     as a double-double, relative error about 2^-100);
//   c^K in double-double (Dekker products; relative error about 2^-100);
//   x^d = 1 + d ln x to first order (|d ln x| < 3e-15, so ln x to single precision suffices).
// The sum is rounded once.  Outside (1e-30, 1e30) the general pow is used.
struct DD {
    double hi, lo;
};
__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = a.hi * b.hi;
    double e = fma(a.hi, b.hi, -p);
    e = e + (a.hi * b.lo + a.lo * b.hi);
    return {p, e};
}

template <int K>
__device__ __forceinline__ double pow_depth(double x) {
    static_assert(K == 7 || K == 4, "exponents -7/3 and -4/3 only");
    constexpr double y = -(double)K / 3.0;
    constexpr double d = (K == 7) ? -0x1.5555555555555p-53 : 0x1.5555555555555p-54;
    if (!(x > 1e-30 && x < 1e30)) return pow(x, y);
    const double s0 = (double)exp2f(__log2f((float)x) * (-1.0f / 3.0f));
    const double rs = fma(-x, s0 * s0 * s0, 1.0);
    const double c0 = fma(s0 * rs, fma(rs, 2.0 / 9.0, 1.0 / 3.0), s0);
    const double p2 = c0 * c0, e2 = fma(c0, c0, -p2);
    const double p3 = p2 * c0, e3 = fma(p2, c0, -p3);
    const double t = fma(x, p3, -1.0);
    const double r = -(t + x * (e3 + e2 * c0));
    const DD c = {c0, c0 * (r * (1.0 / 3.0))};
    const DD c2 = dd_mul(c, c), c4 = dd_mul(c2, c2);
    const DD v = (K == 7) ? dd_mul(dd_mul(c4, c2), c) : c4;
    const double corr = v.hi * (d * (double)logf((float)x));
    return v.hi + (v.lo + corr);
}

// (PGRV*DDPH)**(-0.5) of CALC_ADPSTP (src/cmf_ctrl_physics_mod.F90:193,201), correctly rounded.
// NT is INT(DT_DEF/DT_MIN - 0.01) + 1, so a last-bit change of the minimum can move NT; the
// oracle's glibc pow is correctly rounded for all but rare arguments, and so is this:
//   r0 = rsqrt(x) (within an ulp or two); the residual e = 1 - x r0^2 from exact FMA products
//   (r0^2 = p + pe exactly, x p - 1 rounded once at ~2^-51 magnitude); then one Newton step with
//   its second-order term, x^-1/2 = r0 (1 + e/2 + 3e^2/8 + O(e^3)), added to r0 and rounded once.
// Relative error before the final rounding is about 2^-100.  Outside (1e-300, 1e300) pow is used.
__device__ __forceinline__ double rsqrt_cr(double x) {
    if (!(x > 1e-300 && x < 1e300)) return pow(x, -0.5);
    const double r0 = rsqrt(x);
    const double p = r0 * r0, pe = fma(r0, r0, -p);
    const double t = fma(x, p, -1.0);
    const double e = -(t + x * pe);
    return r0 + r0 * (e * (0.5 + 0.375 * e));
}

// CFL key of one cell, PCADP*DDST*(PGRV*DDPH)**(-0.5) (src/cmf_ctrl_physics_mod.F90:190-202)
__device__ __forceinline__ double cfl_key(double pcadp, double ddst, double pgrv, double rivdph) {
    const double ddph = (rivdph > 0.01) ? rivdph : 0.01;
    return (pcadp * ddst) * rsqrt_cr(pgrv * ddph);
}

// ------------------------------------------------------------------------------------------
// stage schemes (one cell)
// ------------------------------------------------------------------------------------------
struct StageOut {
    double rivsto, fldsto, levsto, rivdph, flddph, fldfrc, fldare, levdph;
};

// The floodplain layers a storage fills, from the channel up: I full layers (0-based layer in use, L: all),
// the storage, width and depth below it, and its gradient.  Layers are read B at a time, one dependent
// round per B layers: two in the phase kernels (four at a time spilled in k_store), one in the resident
// kernel, where the registers of a second layer spilled past its little L1 (298,554 cells: 42.4 us per
// sub-step with two, 38.4 us with one).
struct Filled {
    int I;
    double sfil, wfil, dfil, grd;
};
template <int B>
__device__ __forceinline__ Filled fill_layers(const Net &n, int i, double pstoall, double rsm, double wth, double inc) {
    const int N = n.N, L = n.L;
    Filled f{0, rsm, wth, 0.0, 0.0};
    for (int l0 = 0; l0 < L; l0 += B) {
        double smax[B], grd[B];
#pragma unroll
        for (int e = 0; e < B; e++)
            if (l0 + e < L) {
                smax[e] = __ldg(&n.fldstomax[(size_t)(l0 + e) * N + i]);
                grd[e] = __ldg(&n.fldgrd[(size_t)(l0 + e) * N + i]);
            }
#pragma unroll
        for (int e = 0; e < B; e++) {
            if (l0 + e >= L) break;
            if (!(pstoall > smax[e])) {
                f.I = l0 + e;
                f.grd = grd[e];
                return f;
            }
            f.sfil = smax[e];
            f.wfil = f.wfil + inc;
            f.dfil = f.dfil + grd[e] * inc;
        }
    }
    f.I = L;
    return f;
}

// Stage scheme of one cell: CMF_CALC_FLDSTG_DEF (src/cmf_calc_fldstg_mod.F90:46-97), or with levees
// CMF_LEVEE_FLDSTG (src/cmf_ctrl_levee_mod.F90:301-461).  The default scheme is case 1 of the levee
// scheme for a cell without a levee, but for the bound of the river storage.
struct StageMap {
    double rsm, len, wth;
};
template <class Own>
__device__ __forceinline__ StageMap stage_map(const Own &w, int i) { return {w.rivstomax(i), w.rivlen(i), w.rivwth(i)}; }
template <class Own>
__device__ __forceinline__ StageOut stage(const Net &n, const Own &w, int i, const StageMap &map, double rivsto, double fldsto,
                                          double levsto) {
    StageOut o;
    const int N = n.N, L = n.L;
    const double riv_fld = rivsto + fldsto, pstoall = n.llevee ? riv_fld + levsto : riv_fld;
    const double rsm = map.rsm, len = map.len, wth = map.wth;
    o.levsto = 0.0;
    o.levdph = 0.0;
    if (!(pstoall > rsm)) {                                                         // case 0
        o.rivsto = pstoall;
        o.rivdph = dmax((pstoall / len) / wth, 0.0);
        o.fldsto = 0.0;
        o.flddph = 0.0;
        o.fldfrc = 0.0;
        o.fldare = 0.0;
        return o;
    }
    // read by out-of-bank cells only: the levee parameters and the layer width's quotient
    const int lv = (n.llevee && (w.flags() & C_LEV)) ? __ldg(&n.lev_id[i]) : -1;
    const double grarea = w.grarea(i);
    const double inc = (grarea / len) * n.dfrcinc;
    double lhgt = 0.0, lfrc = 0.0, bhgt = 0.0, ldst = 0.0, ltop = 0.0, lfil = 0.0;
    int lcase = 1;
    if (lv >= 0) {
        const double lbas = __ldg(&n.levbassto[lv]);
        lhgt = __ldg(&n.levhgt[lv]);
        lfrc = __ldg(&n.levfrc[lv]);
        bhgt = __ldg(&n.bashgt[lv]);
        ldst = __ldg(&n.levdst[lv]);
        ltop = __ldg(&n.levtopsto[lv]);
        lfil = __ldg(&n.levfilsto[lv]);
        lcase = pstoall < lbas ? 1 : pstoall < ltop ? 2 : pstoall < lfil ? 3 : 4;
    }
    if (lcase == 1 || lcase == 4) {
        const Filled f = fill_layers<Own::kResident ? 1 : 2>(n, i, pstoall, rsm, wth, inc);
        double wadd;
        if (f.I < L) {
            wadd = -f.wfil + sqrt(f.wfil * f.wfil + ((2.0 * (pstoall - f.sfil)) / len) / f.grd);
            o.flddph = f.dfil + f.grd * wadd;
        } else {
            wadd = 0.0;
            o.flddph = f.dfil + ((pstoall - f.sfil) / f.wfil) / len;
        }
        o.rivsto = rsm + (len * wth) * o.flddph;
        if (!n.llevee) o.rivsto = dmin(o.rivsto, pstoall);
        double frc = ((-wth + f.wfil) + wadd) / (inc * (double)L);
        if (lcase == 1) {
            o.fldsto = dmax(pstoall - o.rivsto, 0.0);
            frc = dmax(frc, 0.0);
            frc = dmin(frc, 1.0);
        } else {
            const double sadd = ((o.flddph - lhgt) * (ldst + wth)) * len;
            o.fldsto = dmax((ltop + sadd) - o.rivsto, 0.0);
            o.levsto = dmax((pstoall - o.rivsto) - o.fldsto, 0.0);
            o.levdph = o.flddph;
        }
        o.fldfrc = frc;
        o.fldare = grarea * frc;
    } else if (lcase == 2) {
        const double sadd = pstoall - __ldg(&n.levbassto[lv]);
        const double wadd = ldst + wth;
        o.flddph = bhgt + (sadd / wadd) / len;
        o.rivsto = rsm + (len * wth) * o.flddph;
        o.fldsto = dmax(pstoall - o.rivsto, 0.0);
        o.fldfrc = lfrc;
        o.fldare = grarea * lfrc;
    } else {                                                                        // case 3
        o.flddph = lhgt;
        o.rivsto = rsm + (len * wth) * o.flddph;
        o.fldsto = dmax(ltop - o.rivsto, 0.0);
        o.levsto = dmax((pstoall - o.rivsto) - o.fldsto, 0.0);
        const int ilev = (int)(lfrc * (double)L) + 1;   // 1-based layer with the levee
        double sfil = ltop, wfil = 0.0, dfil = 0.0, sadd;
        int I = ilev;                                   // 1-based
        while (I <= L) {
            const double fhgt = __ldg(&n.fldhgt[(size_t)(I - 1) * N + i]), fmax = __ldg(&n.fldstomax[(size_t)(I - 1) * N + i]);
            sadd = ((ldst + wth) * (lhgt - fhgt)) * len;
            if (pstoall < fmax + sadd) break;
            sfil = fmax + sadd;
            wfil = inc * (double)I - ldst;
            dfil = fhgt - bhgt;
            I++;
        }
        if (I <= L) {
            const double gr = __ldg(&n.fldgrd[(size_t)(I - 1) * N + i]);
            const double wadd = -wfil + sqrt(wfil * wfil + ((2.0 * (pstoall - sfil)) / len) / gr);
            const double dadd = wadd * gr;
            o.levdph = (bhgt + dfil) + dadd;
            double frc = (wfil + ldst) / (inc * (double)L);
            frc = dmax(frc, 0.0);
            frc = dmin(frc, 1.0);
            o.fldfrc = frc;
            o.fldare = grarea * frc;
        } else {
            const double dadd = ((pstoall - sfil) / wfil) / len;
            o.levdph = (bhgt + dfil) + dadd;
            o.fldfrc = 1.0;
            o.fldare = grarea * 1.0;
        }
    }
    o.rivdph = (o.rivsto / len) / wth;
    return o;
}

// D2FLDARE and D2SFCELV are read by nothing inside the sub-step loop, so the sub-steps write them on
// the last sub-step only (the values the caller observes are the same)
template <class Own>
__device__ __forceinline__ void store_stage(const Net &n, const State &s, Own &w, size_t gi, int i, const StageOut &o,
                                            double dph, bool last) {
    if (last) {
        s.fldare[gi] = o.fldare;
        s.sfcelv[gi] = w.rivelv(i) + o.rivdph;
    }
    w.put_stage(gi, o, n.llevee ? (o.rivsto + o.fldsto) + o.levsto : o.rivsto + o.fldsto, dph, last);
}

// The stage scheme at the top of a step: every array, whatever the host or the emulator left in them
__device__ __forceinline__ void put_full_stage(const Net &n, const State &s, size_t gi, int i, const StageOut &o) {
    s.rivsto[gi] = o.rivsto;
    s.fldsto[gi] = o.fldsto;
    s.rivdph[gi] = o.rivdph;
    s.flddph[gi] = o.flddph;
    s.fldfrc[gi] = o.fldfrc;
    s.fldare[gi] = o.fldare;
    s.sfcelv[gi] = __ldg(&n.rivelv[i]) + o.rivdph;
    if (n.llevee) {
        s.levsto[gi] = o.levsto;
        s.levdph[gi] = o.levdph;
        s.storge[gi] = (o.rivsto + o.fldsto) + o.levsto;
    } else {
        s.storge[gi] = o.rivsto + o.fldsto;
    }
}
// What the sub-steps of the phase kernels keep beside the arrays, from the arrays
__device__ __forceinline__ void begin_cell(const Net &n, const State &s, size_t gi, double rivdph, double fldsto, double flddph,
                                           double fldfrc, double levsto, double levdph) {
    auto some = [](double v) { return __double_as_longlong(v) != 0; };
    unsigned w = 0u;
    if (some(fldsto) || some(flddph) || some(fldfrc) || some(levsto) || some(levdph)) w |= W_STAGE;
    if (some(s.fldsto_pre[gi])) w |= W_PRE;
    if (some(s.fldout_pre[gi])) w |= W_FOUT;
    s.wet[gi] = (unsigned char)w;
    s.dph[gi] = make_double2(rivdph, s.rivdph_pre[gi]);
}

// ------------------------------------------------------------------------------------------
// k_stage: stage scheme at the top of CMF_PHYSICS_ADVANCE + CALC_ADPSTP minimum
// ------------------------------------------------------------------------------------------
// begin: sub-steps of the phase kernels follow in the same step
__global__ void __launch_bounds__(kCellThreads, CMF_STAGE_MINB) k_stage(Net n, State s, int begin) {
    const int m = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double key = 1.0e308;
    if (i < n.N) {
        const size_t gi = (size_t)m * n.N + i;
        const OwnG w(n, s, __ldg(&n.cflag[i]));
        const StageOut o = stage(n, w, i, stage_map(w, i), s.rivsto[gi], s.fldsto[gi], n.llevee ? s.levsto[gi] : 0.0);
        put_full_stage(n, s, gi, i, o);
        if (begin) begin_cell(n, s, gi, o.rivdph, o.fldsto, o.flddph, o.fldfrc, o.levsto, o.levdph);
        if (n.ladpstp && __ldg(&n.i2mask[i]) == 0) key = cfl_key(n.pcadp, (i < n.R) ? __ldg(&n.nxtdst[i]) : n.pdstmth, n.pgrv, o.rivdph);
    }
    if (n.ladpstp) {
        for (int o = 16; o > 0; o >>= 1) key = dmin(key, __shfl_down_sync(0xffffffffu, key, o));
        __shared__ double wmin[32];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
        if (lane == 0) wmin[warp] = key;
        __syncthreads();
        if (warp == 0) {
            double x = lane < nw ? wmin[lane] : 1.0e308;
            for (int o = 16; o > 0; o >>= 1) x = dmin(x, __shfl_down_sync(0xffffffffu, x, o));
            if (lane == 0 && x < 1.0e308) atomicMin(&s.ctl[m].dtmin_bits, (unsigned long long)__double_as_longlong(x));
        }
    }
}

// begin_cell for sub-steps that follow a stage scheme of an earlier call
__global__ void k_begin(Net n, State s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N) return;
    const size_t gi = (size_t)blockIdx.y * n.N + i;
    begin_cell(n, s, gi, s.rivdph[gi], s.fldsto[gi], s.flddph[gi], s.fldfrc[gi], n.llevee ? s.levsto[gi] : 0.0,
               n.llevee ? s.levdph[gi] : 0.0);
}

// ------------------------------------------------------------------------------------------
// k_ntdt: NT and DT per member (src/cmf_ctrl_physics_mod.F90:205-206) and the loop bound
// ------------------------------------------------------------------------------------------
struct NtDt {
    double dt_min, dt;
    int nt;                        // 0: refused (NT cap)
    bool near;                     // DT_DEF/DT_MIN - 0.01 next to an integer
};
__device__ __forceinline__ NtDt calc_ntdt(const Net &n, double dt_def, unsigned long long dtmin_bits) {
    NtDt r{dt_def, dt_def, 1, false};
    if (n.ladpstp) {
        r.dt_min = dmin(dt_def, __longlong_as_double((long long)dtmin_bits));
        const double x = dt_def * (1.0 / r.dt_min) - CMF_F(0.01);
        if (!(x >= 0.0) || x > (double)(kNtCap - 1)) {
            r.nt = 0;              // non-finite or oversized NT: refuse to loop
        } else {
            r.nt = (int)x + 1;
            r.dt = dt_def * (double)(1.0f / (float)r.nt);
            r.near = fabs(x - rint(x)) <= 1e-12 * dmax(x, 1.0);
        }
    }
    return r;
}
__device__ __forceinline__ void put_ntdt(MemberCtl &c, LoopCtl *loop, const NtDt &r) {
    c.dt_min = r.dt_min;
    if (r.nt == 0) c.err = kErrNtCap;
    c.nt = r.nt;
    c.dt = r.dt;
    c.it = 0;
    c.nadd = 0.0;
    atomicAdd((unsigned long long *)&loop->nt_hist[min(r.nt, kNtHist - 1)], 1ull);
}

__global__ void k_ntdt(Net n, State s, cudaGraphConditionalHandle h, int use_cond) {
    __shared__ int smax[32];
    int ntmax = 1;
    long long ntsum = 0, near = 0;
    for (int m = threadIdx.x; m < n.M; m += blockDim.x) {
        MemberCtl &c = s.ctl[m];
        const NtDt r = calc_ntdt(n, c.dt_def, c.dtmin_bits);
        put_ntdt(c, s.loop, r);
        if (n.ladpstp) c.dtmin_bits = (unsigned long long)__double_as_longlong(c.dt_def);
        near += r.near;
        ntmax = max(ntmax, r.nt);
        ntsum += r.nt;
    }
    __shared__ long long ssum[32], snear[32];
    for (int o = 16; o > 0; o >>= 1) {
        ntmax = max(ntmax, __shfl_down_sync(0xffffffffu, ntmax, o));
        ntsum += __shfl_down_sync(0xffffffffu, ntsum, o);
        near += __shfl_down_sync(0xffffffffu, near, o);
    }
    if ((threadIdx.x & 31) == 0) { smax[threadIdx.x >> 5] = ntmax; ssum[threadIdx.x >> 5] = ntsum; snear[threadIdx.x >> 5] = near; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int v = 1;
        long long tot = 0, nr = 0;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) { v = max(v, smax[w]); tot += ssum[w]; nr += snear[w]; }
        v = min(v, kNtCap);
        s.loop->k = 0;
        s.loop->ntmax = v;
        s.loop->near_int += nr;
        s.loop->member_substeps += tot;
        s.loop->loop_iters += v;
        s.loop->outer_steps += 1;
        if (use_cond) cudaGraphSetConditional(h, 1u);
    }
}

// ------------------------------------------------------------------------------------------
// phase A: outflow + dam + bifurcation flux
// ------------------------------------------------------------------------------------------
// CMF_CALC_OUTFLW river/floodplain/mouth discharge and limiter, src/cmf_calc_outflw_mod.F90:44-182
// NADD_adp before sub-step k: the running sum of DT over the sub-steps already done (the same
// additions CMF_DIAG_AVEMAX_ADPSTP performs, so the averages divide by the same value)
__device__ __forceinline__ double nadd_before(int k, double dt) {
    double a = 0.0;
    for (int j = 0; j < k; j++) a = a + dt;
    return a;
}

// Exact shortcuts (the same bits as evaluating every expression):
//  - merge(DOUT, 0, Mask) discards DOUT when Mask is false, so the floodplain flux is evaluated only
//    where its area term passes the mask (most cells carry no floodplain water);
//  - min(a/b, 1) with b > 0 is 1 whenever a >= b (a correctly rounded quotient of a >= b is >= 1),
//    so the limiter rates skip the division in the common case; a NaN a still takes the division.
__device__ __forceinline__ double rate_min1(double a, double b) { return (a >= b) ? 1.0 : dmin(a / b, 1.0); }

// CMF_DIAG_AVEMAX_ADPSTP (src/cmf_calc_diag_mod.F90:104-161) of the sub-step before this one,
// carried into this sub-step's phase A, which reads that sub-step's results anyway: its D2RIVOUT and
// D2FLDOUT are this sub-step's D2*OUT_PRE, its D2RIVDPH and D2STORGE the state it left.  Every addition
// and maximum is the reference's, in its order, so each accumulator holds the bits phase C of that
// sub-step would have stored.  Phase C still forms the last sub-step's terms (and the division by
// NADD), and D2PTHOUT_aAVG, whose per-cell path sum phase A does not see; D2DAMINF_aAVG is
// accumulated by cell_dam and, for the cells without a dam rule, rebuilt on the last sub-step
// (daminf_sum).  The accumulators are read after phase A's own stores: read at its top they would hold
// registers across the outflow arithmetic and spill (measured slower).
__device__ __forceinline__ bool same_bits(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ void diag_carry(const State &s, OwnG &w, size_t gi, double DT, bool first, double rivout,
                                           double fldout, double rivdph, double storge) {
    const double outflw = rivout + fldout;
    const double pro = first ? 0.0 : s.a_rivout[gi], pmo = first ? 0.0 : s.m_outflw[gi];
    const double pmd = first ? 0.0 : s.m_rivdph[gi], pms = first ? 0.0 : s.m_storge[gi];
    // a store is skipped when the sub-step leaves the accumulator's bits unchanged (a zero discharge
    // added to a running sum, a maximum that did not move): the array holds the same bits either way
    auto acc = [&](double prev, double *a, double v) {
        const double x = first ? v * DT : prev + v * DT;
        if (first || !same_bits(x, prev)) a[gi] = x;
    };
    if (!same_bits(outflw, rivout) || (!first && (w.wet & W_AOUT))) {
        const double prev = first ? 0.0 : (w.wet & W_AOUT) ? s.a_outflw[gi] : pro;
        s.a_outflw[gi] = first ? outflw * DT : prev + outflw * DT;
        w.wet |= W_AOUT;
    }
    acc(pro, s.a_rivout, rivout);
    if (__double_as_longlong(fldout) != 0 || (!first && (w.wet & W_AFLD))) {
        const double prev = first ? 0.0 : w.a_fldout(gi);
        s.a_fldout[gi] = first ? fldout * DT : prev + fldout * DT;
        w.wet |= W_AFLD;
    }
    const double mo = dmax(pmo, fabs(outflw));
    const double md = dmax(pmd, rivdph);
    const double ms = dmax(pms, storge);
    if (first || !same_bits(mo, pmo)) s.m_outflw[gi] = mo;
    if (first || !same_bits(md, pmd)) s.m_rivdph[gi] = md;
    if (first || !same_bits(ms, pms)) s.m_storge[gi] = ms;
}

// D2DAMINF_aAVG before the last of `nt` sub-steps: accumulated where a dam rule renews D2DAMINF; elsewhere
// D2DAMINF stays what the host set, and the running sum is rebuilt with the same additions (+0 stays +0)
__device__ __forceinline__ double daminf_sum(const State &s, size_t gi, unsigned flags, double DT, int nt, double dinf) {
    if (nt == 1) return 0.0;
    if (flags & C_DAM) return s.a_daminf[gi];
    if (__double_as_longlong(dinf) == 0) return 0.0;
    double t = dinf * DT;
    for (int k = 1; k < nt - 1; k++) t = t + dinf * DT;
    return t;
}

// D2RIVVEL is observed after the last sub-step; its sub-step average is accumulated in phase A
// (CMF_DIAG_AVEMAX_ADPSTP, src/cmf_calc_diag_mod.F90:104-161)
template <class Own>
__device__ __forceinline__ void vel_average(const Net &n, const State &s, const Own &w, size_t gi, double DT, int nt,
                                            double dt_def, int k, double rvel) {
    const bool first = (k == 0), last = (k == nt - 1);
    if (last) s.rivvel[gi] = rvel;
    if (!n.ldiag) return;
    const double prev = first ? 0.0 : w.a_rivvel(gi);
    double a = first ? rvel * DT : prev + rvel * DT;
    if (last) {
        a = a / (nadd_before(k, DT) + DT);
        if (n.ldiag_out) s.o_rivvel[gi] = s.o_rivvel[gi] + a * dt_def;   // CMF_DIAG_AVEMAX_OUTPUT
        s.a_rivvel[gi] = a;
    } else if (first || !same_bits(a, prev)) {
        w.put_a_rivvel(gi, a);          // unchanged bits (a dry cell adds +0): no store needed
    }
}

// Reservoir operation, CMF_DAMOUT_CALC (src/cmf_ctrl_damout_mod.F90:316-498): the outflow of a cell with
// I1DAM > 0, in place of cell_outflow's (which still forms the cell's diagnostics)
template <class Own>
__device__ __forceinline__ void cell_dam(const Net &n, const State &s, const Own &w, int m, int i, double DT, int nt,
                                         double dt_def, int k) {
    const size_t base = (size_t)m * n.N, gi = base + i;
    double rout = 0.0, fout = 0.0, dinf = w.runoff(gi);
    const int q = __ldg(&n.dam_pos[i]), d = __ldg(&n.dam_id[i]);
    // UPDATE_INFLOW 1b: inflow from the dam's upstream cells, in ascending sequence
    for (int e = __ldg(&n.dam_up_ptr[q]); e < __ldg(&n.dam_up_ptr[q + 1]); e++) {
        const int j = __ldg(&n.dam_up_idx[e]);
        const double fpre = n.lfldout ? w.nb(s.fldout_pre, base + j) : 0.0;
        dinf = (dinf + w.nb(s.rivout_pre, base + j)) + fpre;
    }
    if (n.ldiag && k > 0) {              // the previous sub-step's D2DAMINF joins its average before it is replaced
        const double prev = s.daminf[gi] * DT;
        s.a_daminf[gi] = k == 1 ? prev : s.a_daminf[gi] + prev;
    }
    s.daminf[gi] = dinf;
    if (w.flags() & C_KIN) {
        // UPDATE_INFLOW 1c: kinematic outflow upstream of a dam; (1/n) sqrt(slope) of channel and
        // floodplain are static
        const double p23 = CMF_F(2. / 3.);
        const double dph = w.rivdph(gi), wth = w.rivwth(i);
        const double dvel = __ldg(&n.kin_vel[q]) * pow(dph, p23);
        const double darea = wth * dph;
        rout = dmin(darea * dvel, w.rivsto(gi) / DT);
        const double fdph = w.flddph(gi), fsto = w.fldsto(gi);
        if (fdph > 0.0 || fsto != 0.0) {        // else min(0 * 0, 0) = +0
            const double dvel_f = __ldg(&n.kin_velf[q]) * pow(fdph, p23);
            double dare_f = fsto * w.inv_rivlen(i);
            dare_f = dmax(dare_f - fdph * wth, 0.0);
            fout = dmin(dare_f * dvel_f, fsto / DT);
        }
        vel_average(n, s, w, gi, DT, nt, dt_def, k, dvel);
    }
    if (d >= 0 && __ldg(&n.dam_stat[d]) > 0) {
        const double vol = s.damsto[gi];
        const double qn = __ldg(&n.qn[d]), qf = __ldg(&n.qf[d]), qa = __ldg(&n.qa[d]), con = __ldg(&n.convol[d]), eme = __ldg(&n.emevol[d]);
        double q = 0.0;
        if (n.ldamh22) {
            const double nor = __ldg(&n.norvol[d]);
            if (vol <= nor) q = qn * (vol / con);
            else if (nor < vol && vol <= con) {
                if (qf <= dinf) q = qn * CMF_F(0.5) + ((vol - nor) / (con - nor)) * (qf - qn);
                else { const double r = (vol - nor) / (eme - nor); q = qn * CMF_F(0.5) + (r * r) * (qf - qn); }
            } else if (con < vol && vol < eme) {
                if (qf <= dinf)
                    q = qf + ((dmax(CMF_F(1.) - __ldg(&n.r_volupa[d]) / CMF_F(0.2), 0.0) * (vol - con)) / (eme - con)) * (dinf - qf);
                else { const double r = (vol - nor) / (eme - nor); q = qn * CMF_F(0.5) + (r * r) * (qf - qn); }
            } else q = dmax(dinf, qf);
        } else {
            // the regimes' volume fractions share one quotient and one power: a warp of dams in different
            // regimes walks each once (sqrt, cube and tenth root in turn took 12 us of a sub-step)
            const double adj = __ldg(&n.adjvol[d]);
            const int regime = vol <= con ? 1 : vol <= adj ? 2 : (vol > adj && vol <= eme) ? 3 : vol > eme ? 4 : 0;
            const double lo = regime == 1 ? 0.0 : regime == 2 ? con : adj;
            const double x = (vol - lo) / (regime == 1 ? con : regime == 2 ? adj - con : eme - adj);
            double f = 0.0;
            if (regime == 2 || regime == 3) f = pow(x, regime == 2 ? 3.0 : CMF_F(0.1));
            if (regime == 1) q = qn * sqrt(x);
            else if (regime == 2) q = qn + f * (qa - qn);
            else if (regime == 3) {
                const double t = qa + f * (qf - qa);
                q = dinf >= qf ? dmax(qn + ((vol - con) / (eme - con)) * (dinf - qn), t) : t;
            } else if (regime == 4) q = (dinf >= qf) ? dinf : qf;
        }
        q = dmin(dmin(q, vol / DT), (w.rivsto(gi) + w.fldsto(gi)) / DT);
        q = dmax(q, 0.0);
        rout = q;
        fout = 0.0;
    }
    w.put_raw(gi, i, rout, fout);
}

template <class Own>
__device__ __forceinline__ void cell_outflow(const Net &n, const State &s, Own &w, int m, int i, double DT,
                                             int nt, double dt_def, int k, bool split) {
    const size_t base = (size_t)m * n.N, gi = base + i;
    const double gdt = n.pgrv * DT;
    const double rivelv = w.rivelv(i);
    const double rivdph = w.rivdph(gi), rivdph_pre = w.rivdph_pre(gi);
    const double sfc = rivelv + rivdph;
    const double sfc_pre = rivelv + rivdph_pre;
    const double wth = w.rivwth(i);
    const double inv_wth = w.inv_rivwth(i);
    const double man = w.rivman(i);
    const double rivout_pre = w.rivout_pre(gi);
    const double rivout_old = split ? s.rivout_cur[gi] : rivout_pre;
    const double fldout_pre = w.fldout_pre(gi), fsto = w.fldsto(gi), riv_fld = w.rivsto(gi) + fsto;
    const double storge = n.llevee ? riv_fld + w.levsto(gi) : riv_fld;      // D2STORGE of the stage scheme
    // river cells see the downstream cell's surface; a mouth the boundary elevation, over its own depth
    const bool river = i < n.R;
    double dwn, inv_dst, dsfc = sfc, dsfc_pre = sfc_pre, dflw = rivdph, dflw_pr = rivdph_pre;
    if (river) {
        const DownCell below = w.down(base, i, w.next(i));
        dwn = below.rivelv + below.rivdph;
        inv_dst = w.inv_nxtdst(i);
        dsfc = dmax(sfc, dwn);
        dsfc_pre = dmax(sfc_pre, below.rivelv + below.rivdph_pre);
        dflw = dsfc - rivelv;
        dflw_pr = dsfc_pre - rivelv;
    } else {
        dwn = __ldg(&n.dwnelv[i]);
        inv_dst = 1.0 / n.pdstmth;
    }
    // the floodplain's maps and state, read where a first test passes; the resident kernel knows from the
    // cell's bits that there is water on it and reads them with everything else
    double inv_len = 0.0, fdph = 0.0, elv = 0.0, hgt = 0.0, fsto_pre = 0.0;
    auto read_area = [&] { inv_len = w.inv_rivlen(i); fdph = w.flddph(gi); };
    auto read_flow = [&] { elv = w.elevtn(i); hgt = w.rivhgt(i); fsto_pre = w.fldsto_pre(gi); };
    if constexpr (Own::kResident)
        if (n.lfldout && w.flooded()) {
            read_area();
            read_flow();
        }
    // diagnostics of sub-step k-1: here, so that their sums come with the downstream depth and hold no
    // registers across the flow equations
    if (n.ldiag && k > 0) {
        if constexpr (Own::kResident) w.carry(gi, DT, k == 1, rivout_pre, fldout_pre, rivdph, storge);
        else diag_carry(s, w, gi, DT, k == 1, rivout_pre, fldout_pre, rivdph, storge);
    }
    double dslp = (sfc - dwn) * inv_dst;
    double rout, fout = 0.0, rvel;
    {
        const double dare = dmax(wth * dflw, 1.E-10);
        const double dflw_im = dmax(sqrt(dflw * dflw_pr), 1.E-6);
        const double dout_pr = rivout_pre * inv_wth;
        const double dout = (wth * (dout_pr + (gdt * dflw_im) * dslp))
                          * (1.0 / (1.0 + ((gdt * (man * man)) * fabs(dout_pr)) * pow_depth<7>(dflw_im)));
        const double dvel = rivout_old * (1.0 / dare);
        const bool mask = (dflw_im > CMF_F(1.E-5) && dare > CMF_F(1.E-5));
        rout = mask ? dout : 0.0;
        rvel = mask ? dvel : 0.0;
    }
    if (n.lfldout) {
        // the reference's masks are a double at river cells and a default-real literal at mouths
        const double eps = river ? 1.E-5 : CMF_F(1.E-5);
        // without floodplain water the area is max(-FLDDPH * RIVWTH, 0) = 0: nothing more to read
        if constexpr (!Own::kResident)
            if (fsto != 0.0) read_area();
        const double dare = fsto != 0.0 ? dmax(fsto * inv_len - fdph * wth, 0.0) : 0.0;
        if (dare > eps) {
            if constexpr (!Own::kResident) read_flow();
            dslp = dmax(-0.005, dmin(0.005, dslp));
            const double df = river ? dmax(dsfc - elv, 0.0) : sfc - elv;
            const double df_pr = dsfc_pre - elv;
            const double dflw_im = dmax(sqrt(dmax(df * df_pr, 0.0)), 1.E-6);
            const double flddph_pre = dmax(rivdph_pre - hgt, 0.0);
            const double dare_pr = dmax(fsto_pre * inv_len - flddph_pre * wth, 1.E-6);
            const double dare_im = dmax(sqrt(dare * dare_pr), 1.E-6);
            const double dout_pr = fldout_pre;
            const double dout = (dout_pr + (gdt * dare_im) * dslp)
                * (1.0 / (1.0 + (((gdt * (n.pmanfld * n.pmanfld)) * fabs(dout_pr)) * pow_depth<4>(dflw_im)) * (1.0 / dare_im)));
            fout = (dflw_im > eps) ? dout : 0.0;
            if (!(fout * rout > 0.0)) fout = 0.0;
        }
    }
    if (river) {
        // storage-change limiter (v423), :176-182
        const double dlim = dmax((-rout - fout) * DT, CMF_F(1.E-10));
        const double rate = rate_min1(0.05 * storge, dlim);
        rout = rout * rate;
        fout = fout * rate;
    }
    if (!(w.flags() & C_DAM)) w.put_raw(gi, i, rout, fout);
    if (!(w.flags() & C_KIN)) vel_average(n, s, w, gi, DT, nt, dt_def, k, rvel);
}

// CMF_CALC_PTHOUT (src/cmf_calc_pthout_mod.F90:34-94) / CMF_LEVEE_OPT_PTHOUT (src/cmf_ctrl_levee_mod.F90:508-601)
__device__ __forceinline__ double path_flux(double wth, double pre, double gdt, double dflw_im, double dslp, double man,
                                           bool recip) {
    const double dout_pr = recip ? pre * (1.0 / wth) : pre / wth;
    return (wth * (dout_pr + (gdt * dflw_im) * dslp)) / (1.0 + ((gdt * (man * man)) * fabs(dout_pr)) * pow_depth<7>(dflw_im));
}

// Coherent: values of other cells come past L1, of which the resident kernel has hardly any; the phase
// kernels and k_persist read them through L1, which the launch or the barrier's acquire has emptied
template <bool Coherent>
__device__ __forceinline__ double ld_nb(const double *p, size_t g) { return Coherent ? __ldcg(p + g) : p[g]; }

template <bool Coherent>
__device__ __forceinline__ double2 end_depth(const State &s, size_t g) {
    if constexpr (Coherent) return make_double2(__ldcg(s.rivdph + g), __ldcg(s.rivdph_pre + g));
    else return s.dph[g];
}

// Bifurcation paths by lanes: thread x of the path threads takes level l of path p, 32 / Lp paths per
// warp, the lanes of a path consecutive from lane0 (one thread per path ran its levels' powers one after
// the other, up to 5 times as long as a cell, and in the last blocks of the grid).  With more than 32
// levels a warp takes one path, and lane l its levels l and l + 32.
__host__ __device__ inline int paths_per_warp(int Lp) { return Lp > 0 && Lp <= 32 ? 32 / Lp : 1; }
__host__ __device__ inline int path_threads(int P, int Lp) { return P > 0 ? (P + paths_per_warp(Lp) - 1) / paths_per_warp(Lp) * 32 : 0; }
struct PathLane {
    int p, l, lane0;
    bool on;
};
__device__ __forceinline__ PathLane path_lane(const Net &n, int x) {
    const int ppw = paths_per_warp(n.Lp), lane = x & 31, q = min(lane / n.Lp, ppw), l = lane - q * n.Lp;
    const int p = (x >> 5) * ppw + q;
    return {p, l, q * n.Lp, q < ppw && p < n.P && l < n.Lp};
}
// 0 + v(1) + v(2) + ... over the levels of a path, in their order; v[1] holds the levels past 32
__device__ __forceinline__ double level_sum(int Lp, int lane0, const double (&v)[2]) {
    double sum = 0.0;
    for (int k = 0; k < min(Lp, 32); k++) sum = sum + __shfl_sync(0xffffffffu, v[0], (lane0 + k) & 31);
    for (int k = 32; k < Lp; k++) sum = sum + __shfl_sync(0xffffffffu, v[1], k - 32);
    return sum;
}

// Phase A of one path lane (every lane of the warp calls it): the level's flux, and the limiter on the
// sum over the levels.  Its time is rounds of dependent loads, so there are two: what the lane's own
// indices address, then what the path's ends do, read whether or not the branches below come to need it
// (each read where it is used: five rounds; with path_rescale's two instead of four and the cells' own
// range of path ends, a sub-step of 298,554 cells in the resident kernel 44.4 -> 43.1 us, of 2M cells by
// phase kernels 304 -> 294 us).
template <bool Coherent>
__device__ __forceinline__ void path_outflow(const Net &n, const State &s, int m, const PathLane &t, double DT) {
    const int P = n.P, Lp = n.Lp, p = t.p;
    const size_t base = (size_t)m * n.N, pb = (size_t)m * Lp * P;
    int skip = 3, u = 0, d = 0;
    double dst = 1.0, elv = 0.0, wth = 0.0, man = 0.0, pre = 0.0;
    auto level = [&](int l) {
        const size_t o = (size_t)l * P + p;
        elv = __ldg(&n.pth_elv[o]);
        wth = __ldg(&n.pth_wth[o]);
        man = __ldg(&n.pth_man[l]);
        pre = s.pthflw_pre[pb + o];
    };
    if (t.on) {
        skip = __ldg(&n.pth_skip[p]);
        u = __ldg(&n.pth_up[p]);
        d = __ldg(&n.pth_dn[p]);
        dst = __ldg(&n.pth_dst[p]);
        level(t.l);
    }
    const bool live = t.on && !(n.llevee ? (skip & 2) : (skip & 1));
    double f[2] = {0.0, 0.0}, sto = 0.0;
    if (live) {
        const double gdt = n.pgrv * DT;
        const double eu = __ldg(&n.rivelv[u]), ed = __ldg(&n.rivelv[d]);
        const double2 du = end_depth<Coherent>(s, base + u), dd = end_depth<Coherent>(s, base + d);
        const double stu = ld_nb<Coherent>(s.storge, base + u), std = ld_nb<Coherent>(s.storge, base + d);
        const bool leveed = n.llevee && t.l > 0;
        double lu = 0.0, ld = 0.0;
        if (leveed && (skip & 4)) lu = __ldg(&n.elevtn[u]) + ld_nb<Coherent>(s.levdph, base + u);
        if (leveed && (skip & 8)) ld = __ldg(&n.elevtn[d]) + ld_nb<Coherent>(s.levdph, base + d);
        sto = dmin(stu, std);
        const double su = eu + du.x, sd = ed + dd.x;
        double dslp = (su - sd) / dst;
        dslp = dmax(-0.005, dmin(0.005, dslp));
#pragma unroll 1
        for (int h = 0, l = t.l; l < Lp; h++, l += 32) {
            if (h > 0) {
                level(l);
                if (skip & 4) lu = __ldg(&n.elevtn[u]) + ld_nb<Coherent>(s.levdph, base + u);
                if (skip & 8) ld = __ldg(&n.elevtn[d]) + ld_nb<Coherent>(s.levdph, base + d);
            }
            const bool channel = !n.llevee || l == 0;    // with levees: level 1, the river channel
            double im;
            if (channel) {
                const double spu = eu + du.y, spd = ed + dd.y;
                const double dflw = dmax(dmax(su, sd) - elv, 0.0);
                const double dflw_pr = dmax(dmax(spu, spd) - elv, 0.0);
                im = sqrt(dflw * dflw_pr);
                if (!n.llevee) im = dmax(im, sqrt(dflw * 0.01));
                else if (im <= 0.0) im = dflw;           // semi-implicit depth
            } else {
                double slu = su, sld = sd;
                if (skip & 4) slu = dmin(lu, su);
                if (skip & 8) sld = dmin(ld, sd);
                im = dmax(dmax(slu, sld) - elv, 0.0);
            }
            const double v = im > 1.E-5 ? path_flux(wth, pre, gdt, im, dslp, man, !channel) : 0.0;
            if (h == 0) f[0] = v;
            else f[1] = v;
        }
    }
    double sum = level_sum(Lp, t.lane0, f);
    if (!live) sum = 0.0;
    if (sum != 0.0) {
        const double rate = rate_min1(0.05 * sto, fabs(sum * DT));
        f[0] = f[0] * rate;
        f[1] = f[1] * rate;
        sum = sum * rate;
    }
    if (t.on) {
        s.pthflw_raw[pb + (size_t)t.l * P + p] = f[0];
        if (t.l + 32 < Lp) s.pthflw_raw[pb + (size_t)(t.l + 32) * P + p] = f[1];
        if (t.l == 0) s.pthsum_raw[(size_t)m * P + p] = sum;
    }
}

__device__ __forceinline__ OwnG own_cell(const Net &n, const State &s, int m, int i) {
    return OwnG(n, s, __ldg(&n.cflag[i]), s.wet[(size_t)m * n.N + i]);
}
__device__ __forceinline__ void put_wet(const Net &n, const State &s, int m, int i, unsigned before, unsigned now) {
    if (now != before) s.wet[(size_t)m * n.N + i] = (unsigned char)now;
}
// one cell of phase A
__device__ __forceinline__ void flux_cell(const Net &n, const State &s, int m, int i, double DT, int nt, double dt_def, int k,
                                          bool split) {
    OwnG w = own_cell(n, s, m, i);
    const unsigned before = w.wet;
    cell_outflow(n, s, w, m, i, DT, nt, dt_def, k, split);
    put_wet(n, s, m, i, before, w.wet);
}

// Blocks of phase A: cells, then (path, level) lanes, then dam cells
template <int MinBlocks>
__global__ void __launch_bounds__(kCellThreads, MinBlocks) k_flux(Net n, State s, int ncell_blocks, int npath_blocks) {
    const int m = blockIdx.y;
    const MemberCtl &c = s.ctl[m];
    const int k = s.loop->k;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) s.loop->kcur = k;   // for k_rate and k_store
    if (k >= c.nt) return;
    const double DT = c.dt;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if ((int)blockIdx.x < ncell_blocks) {
        if (x < n.N) flux_cell(n, s, m, x, DT, c.nt, c.dt_def, k, s.loop->split != 0);
    } else if ((int)blockIdx.x < ncell_blocks + npath_blocks) {
        path_outflow<false>(n, s, m, path_lane(n, x - ncell_blocks * (int)blockDim.x), DT);
    } else {
        const int d = x - (ncell_blocks + npath_blocks) * (int)blockDim.x;
        if (d < n.ndam_cells) {
            const int i = __ldg(&n.dam_cells[d]);
            cell_dam(n, s, own_cell(n, s, m, i), m, i, DT, c.nt, c.dt_def, k);
        }
    }
}

// ------------------------------------------------------------------------------------------
// phase B: P2STOOUT and D2RATE, src/cmf_calc_outflw_mod.F90:410-451
// ------------------------------------------------------------------------------------------
template <class Own>
__device__ __forceinline__ void cell_rate(const Net &n, const State &s, const Own &w, int m, int i, double DT) {
    const size_t base = (size_t)m * n.N, gi = base + i;
    const double2 raw = w.own_raw(gi);
    const double rout = raw.x, fout = raw.y;
    double so = dmax(rout, 0.0) + dmax(fout, 0.0);
    w.each_raw(base, i, [&](double rj, double fj) { so = (so + dmax(-rj, 0.0)) + dmax(-fj, 0.0); });
    so = so * DT;
    if (w.flags() & C_PATH) {
        const double *sum = s.pthsum_raw + (size_t)m * n.P;
        const int2 ends = __ldg(&n.path_ends[i]);
        for (int e = ends.x; e < ends.y; e++) {
            const int p = __ldg(&n.pend[e].x);
            const double v = w.nb(sum, p >= 0 ? p : ~p);
            so = so + dmax(p >= 0 ? v : -v, 0.0) * DT;
        }
    }
    const double dout = dmax(so, 1.E-10);
    const double dsto = w.rivsto(gi) + w.fldsto(gi);
    w.put_rate(gi, i, rout, fout, rate_min1(dsto, dout));
}

// advance != 0: block (0,0) also moves the loop counter to the next sub-step and sets the WHILE
// condition (every k_flux block has read the counter; k_rate and k_store read `kcur`)
__global__ void __launch_bounds__(kCellThreads, 6) k_rate(Net n, State s, int advance, cudaGraphConditionalHandle h, int use_cond) {
    const int m = blockIdx.y;
    const MemberCtl &c = s.ctl[m];
    const int k = s.loop->kcur;
    if (advance && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        const int kn = k + 1;
        s.loop->k = kn;
        s.loop->split = 0;
        if (use_cond) cudaGraphSetConditional(h, (kn < s.loop->ntmax && kn < kNtCap) ? 1u : 0u);
    }
    if (k >= c.nt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n.N) cell_rate(n, s, own_cell(n, s, m, i), m, i, c.dt);
}

// ------------------------------------------------------------------------------------------
// phase C: rescale + inflow + dam balance + VARS_PRE + STONXT + stage + diagnostics
// ------------------------------------------------------------------------------------------
template <bool Coherent>
__device__ __forceinline__ double scaled_pathsum(const Net &n, const double *sum_raw, const double *rate_m, int p) {
    const double v = ld_nb<Coherent>(sum_raw, p);
    if (__ldg(&n.pth_skip[p]) & 1) return v;
    return v * ld_nb<Coherent>(rate_m, v >= 0.0 ? __ldg(&n.pth_up[p]) : __ldg(&n.pth_dn[p]));
}

// one path lane in phase C (every lane of the warp calls it): LSPAMAT path rescale (:494-517),
// CALC_VARS_PRE copy, diagnostics
template <bool Coherent>
__device__ __forceinline__ void path_rescale(const Net &n, const State &s, int m, const PathLane &t, double DT, bool first,
                                             bool last, double nadd, double dt_def) {
    const int P = n.P, Lp = n.Lp, p = t.p;
    const size_t base = (size_t)m * n.N, pb = (size_t)m * Lp * P;
    const double *rate_m = s.rate + base;
    double a[2] = {0.0, 0.0};
    if (t.on) {
        // two rounds of loads: the path's own values, then the rates of both ends
        const bool sk = __ldg(&n.pth_skip[p]) & 1, add = n.ldiag && !first;
        const int u = __ldg(&n.pth_up[p]), d = __ldg(&n.pth_dn[p]);
        size_t o = pb + (size_t)t.l * P + p;
        double f = s.pthflw_raw[o], x0 = add ? s.a_pthflw[o] : 0.0;
        const double sum = t.l == 0 ? ld_nb<Coherent>(s.pthsum_raw, (size_t)m * P + p) : 0.0;
        double ru = 1.0, rd = 1.0;
        if (!sk) {
            ru = ld_nb<Coherent>(rate_m, u);
            rd = ld_nb<Coherent>(rate_m, d);
        }
        if (t.l == 0) s.pthsum[(size_t)m * P + p] = sk ? sum : sum * (sum >= 0.0 ? ru : rd);
#pragma unroll 1
        for (int h = 0, l = t.l; l < Lp; h++, l += 32) {
            if (h > 0) {
                o = pb + (size_t)l * P + p;
                f = s.pthflw_raw[o];
                x0 = add ? s.a_pthflw[o] : 0.0;
            }
            if (!sk) f = f * (f >= 0.0 ? ru : rd);
            s.pthflw_pre[o] = f;
            if (n.ldiag) {
                double x = first ? f * DT : x0 + f * DT;
                if (last) {
                    x = x / (nadd + DT);
                    if (n.ldiag_out) s.o_pthflw[o] = s.o_pthflw[o] + x * dt_def;
                }
                s.a_pthflw[o] = x;
                if (h == 0) a[0] = x;
                else a[1] = x;
            }
        }
    }
    if (n.ldiag && last) {
        const double asum = level_sum(Lp, t.lane0, a);
        if (t.on && t.l == 0) s.a_pthsum[(size_t)m * P + p] = asum;
    }
}

// one cell in phase C; `bput(k, v)` receives the last sub-step's budget term k
template <class Own, class BPut>
__device__ __forceinline__ void cell_store(const Net &n, const State &s, Own &w, int m, int i, double DT,
                                           bool first, bool last, double nadd, int nt, double dt_def, BPut bput) {
    const size_t base = (size_t)m * n.N;
    const size_t gi = base + i;
    const double *rate_m = s.rate + base;
    // the cell's own state is read up front, before anything is stored: in the compiler's view a
    // store may alias any later load of another state array and would hold that load back
    const auto rate_i = w.rate(gi);
    const double2 own = w.own_out(gi);
    double rout = own.x, fout = own.y;
    const double runoff = w.runoff(gi);
    const double rivsto0 = w.rivsto(gi), fldsto0 = w.fldsto(gi), rivdph0 = w.rivdph(gi);
    const double frc = w.fldfrc(gi);
    const double levsto = n.llevee ? w.levsto(gi) : 0.0;
    // with registers to spare (the resident kernel) the stage scheme's maps come with the gathers; read
    // where they are used they cost a round of loads of their own
    StageMap map;
    if constexpr (Own::kResident) map = stage_map(w, i);
    // own outflow after the LSPAMAT rescale (:456-473); phase B has done a positive one and a mouth's
    if (i < n.R && !(rout > 0.0)) {
        const double r = w.nb(rate_m, w.next(i));
        rout = rout * r;
        fout = fout * r;
    }
    // inflow from the upstream cells
    double rinf = 0.0, finf = 0.0;
    w.each_out(base, i, rate_i, [&](double rj, double fj) {
        rinf = rinf + rj;
        finf = finf + fj;
    });
    if (rout != rout || rinf != rinf) {            // see rescale_own
        if (i < n.R && rout != rout)
            by_sign(s.raw[gi], rate_i, w.nb(rate_m, w.next(i)), [&](double r, double f) {
                rout = r;
                fout = f;
            });
        rinf = finf = 0.0;
        w.each_by_sign(base, i, rate_i, [&](double rj, double fj) {
            rinf = rinf + rj;
            finf = finf + fj;
        });
    }
    double pout = 0.0;
    const bool has_path = w.flags() & C_PATH;
    if (has_path) {
        const double *sum = s.pthsum_raw + (size_t)m * n.P;
        const int2 ends = __ldg(&n.path_ends[i]);
        for (int e = ends.x; e < ends.y; e++) {
            const int2 t = __ldg(&n.pend[e]);
            const bool up = t.x >= 0;              // this cell is the path's upstream end
            double v = w.nb(sum, up ? t.x : ~t.x);
            if (t.y == -2) {                       // listed at a cell that is not its end
                v = scaled_pathsum<Own::kResident>(n, sum, rate_m, up ? t.x : ~t.x);
            } else if (t.y >= 0) {
                const double far = w.nb(rate_m, t.y);
                v = v * ((v >= 0.0) == up ? (double)rate_i : far);
            }
            pout = up ? pout + v : pout - v;
        }
    }
    // CMF_DAMOUT_WATBAL, src/cmf_ctrl_damout_mod.F90:516-535 (the new dam storage is stored below)
    double dmiss = 0.0, damsto1 = 0.0;
    const bool dam = w.flags() & C_DAMID;
    if (dam) {
        const double inflow = (rinf + finf) + runoff;
        const double outflw = rout + fout;
        const double s0 = s.damsto[gi];
        damsto1 = (s0 + inflow * DT) - outflw * DT;
        dmiss = ((s0 - damsto1) + inflow * DT) - outflw * DT;
    }
    bput(11, dmiss);
    // CMF_CALC_STONXT, src/cmf_calc_stonxt_mod.F90:53-100
    bput(0, rivsto0 + fldsto0);
    bput(3, rinf * DT + finf * DT);
    bput(4, (rout * DT + fout * DT) + pout * DT);
    double rs = (rivsto0 + rinf * DT) - rout * DT;
    double fs = fldsto0;
    if (rs < 0.0) { fs = fs + rs; rs = 0.0; }
    fs = ((fs + finf * DT) - fout * DT) - pout * DT;
    if (fs < 0.0) { rs = dmax(rs + fs, 0.0); fs = 0.0; }
    bput(1, rs + fs);
    const double outflw = rout + fout;
    rs = rs + (runoff * (1.0 - frc)) * DT;       // D2GDWRTN is zero without groundwater delay
    fs = fs + (runoff * frc) * DT;
    bput(2, n.llevee ? (rs + fs) + levsto : rs + fs);
    bput(5, n.llevee ? (rs + fs) + levsto : rs + fs);
    // What the new storage does not change leaves before the stage scheme, so that it holds no registers
    // across it.  CALC_VARS_PRE, src/cmf_ctrl_physics_mod.F90:254-277, and the dam storage:
    w.put_pre(gi, rout, fout, rivdph0, fldsto0, last);
    if (dam) s.damsto[gi] = damsto1;
    if (last) {   // diagnostics read by nothing inside the sub-step loop
        s.rivinf[gi] = rinf;
        s.fldinf[gi] = finf;
        s.pthout[gi] = pout;
        s.outflw[gi] = outflw;
    }
    // CMF_DIAG_AVEMAX_ADPSTP / GETAVE_ADPSTP, src/cmf_calc_diag_mod.F90:104-221.  The sub-steps
    // before the last one are accumulated by the next sub-step's phase A (diag_carry), except
    // D2PTHOUT_aAVG: D2PTHINF is never written by the reference (always 0), and a cell without
    // bifurcation channels adds +0 every sub-step, so its average (and output average) stays at the
    // +0 the arrays were created with; cells with channels accumulate it here every sub-step.
    // CMF_DIAG_AVEMAX_OUTPUT (src/cmf_calc_diag_mod.F90:272-318) on the last sub-step: the output
    // interval accumulates the finished sub-step average times DT_DEF.
    const bool out = last && n.ldiag_out;
    if (n.ldiag && (last || has_path)) {
        const double na = nadd + DT;
        const double ddef = dt_def;
        auto acc = [&](double prev, double *a, double *oa, double v) {
            double x = first ? v * DT : prev + v * DT;
            if (last) x = x / na;
            if (first || last || !same_bits(x, prev)) a[gi] = x;
            if (out) oa[gi] = oa[gi] + x * ddef;
        };
        if (has_path) acc(first ? 0.0 : w.a_pthout(gi), s.a_pthout, s.o_pthout, pout);
        if (last) {
            // every previous accumulator is read before the first of them is stored
            const double pro = first ? 0.0 : w.a_rivout(gi), pfo = first ? 0.0 : w.a_fldout(gi);
            const double pof = first ? 0.0 : w.a_outflw(gi), pmo = first ? 0.0 : w.m_outflw(gi);
            const double dinf = n.ldamout ? s.daminf[gi] : 0.0;
            const double pdi = n.ldamout ? daminf_sum(s, gi, w.flags(), DT, nt, dinf) : 0.0;
            acc(pro, s.a_rivout, s.o_rivout, rout);
            acc(pfo, s.a_fldout, s.o_fldout, fout);
            acc(pof, s.a_outflw, s.o_outflw, outflw);
            // runoff and DT are constant over the outer step: the same running sum of
            // runoff*DT the accumulator would hold, rebuilt in registers on the last sub-step
            const double rdt = runoff * DT;
            double a = rdt;
            for (int k = 1; k < nt; k++) a = a + rdt;
            a = a / na;
            s.a_runoff[gi] = a;
            if (out) s.o_runoff[gi] = s.o_runoff[gi] + a * ddef;
            if (n.ldamout) acc(pdi, s.a_daminf, s.o_daminf, dinf);
            const double mo = dmax(pmo, fabs(outflw));
            s.m_outflw[gi] = mo;
            if (out) s.om_outflw[gi] = dmax(s.om_outflw[gi], fabs(mo));
        }
    }
    // stage scheme, :125
    if constexpr (!Own::kResident) map = stage_map(w, i);
    const StageOut o = stage(n, w, i, map, rs, fs, levsto);
    // CMF_CheckNanB-style probe (src/cmf_utils_mod.F90:807-815) on the new storage: a NaN or
    // infinite runoff or state surfaces as a positive status instead of a silent NaN state
    if (!isfinite((o.rivsto + o.fldsto) + o.levsto)) s.ctl[m].err = kErrNonFinite;
    store_stage(n, s, w, gi, i, o, rivdph0, last);
    bput(6, n.llevee ? (o.rivsto + o.fldsto) + o.levsto : o.rivsto + o.fldsto);
    bput(7, o.rivsto);
    bput(8, o.fldsto);
    bput(9, o.fldare);
    bput(10, o.levsto);
    if (n.ldiag && last) {
        const double pmd = first ? 0.0 : w.m_rivdph(gi), pms = first ? 0.0 : w.m_storge(gi);
        const double stg = n.llevee ? (o.rivsto + o.fldsto) + o.levsto : o.rivsto + o.fldsto;
        const double md = dmax(pmd, o.rivdph), ms = dmax(pms, stg);
        s.m_rivdph[gi] = md;
        s.m_storge[gi] = ms;
        if (out) {
            s.om_rivdph[gi] = dmax(s.om_rivdph[gi], md);
            s.om_storge[gi] = dmax(s.om_storge[gi], ms);
        }
    }
}

template <class BPut>
__device__ __forceinline__ void store_cell(const Net &n, const State &s, int m, int i, double DT, bool first, bool last,
                                           double nadd, int nt, double dt_def, BPut bput) {
    OwnG w = own_cell(n, s, m, i);
    const unsigned before = w.wet;
    cell_store(n, s, w, m, i, DT, first, last, nadd, nt, dt_def, bput);
    put_wet(n, s, m, i, before, w.wet);
}

// Budget partials of the last sub-step (the only one the caller observes), one per warp of 32
// consecutive cells: a fixed butterfly over the warp, so the partials -- and the budgets k_budget
// sums from them in a fixed order -- are the same whatever block size or schedule ran the cells.
// Layout [m][k][warp] for a coalesced final reduction.  Every lane of the warp calls it.
__device__ __forceinline__ void warp_budget_partials(const State &s, int m, int warp, int nwarps, double (&b)[kBudgets]) {
#pragma unroll
    for (int k = 0; k < kBudgets; k++)
        for (int o = 16; o > 0; o >>= 1) b[k] = b[k] + __shfl_down_sync(0xffffffffu, b[k], o);
    if ((threadIdx.x & 31) == 0 && warp < nwarps) {     // warps past the last cell hold no cells
        double *dst = s.partials + (size_t)m * kBudgets * nwarps + warp;
#pragma unroll
        for (int k = 0; k < kBudgets; k++) dst[(size_t)k * nwarps] = b[k];
    }
}
__host__ __device__ inline int budget_warps(int N) { return (N + 31) / 32; }

template <int MinBlocks>
__global__ void __launch_bounds__(kCellThreads, MinBlocks) k_store(Net n, State s, int ncell_blocks) {
    const int m = blockIdx.y;
    const MemberCtl &c = s.ctl[m];
    const int kk = s.loop->kcur;
    const bool active = kk < c.nt;
    if (!active) return;   // uniform per block (blockIdx.y), no barrier is skipped divergently
    const double DT = c.dt;
    const bool first = (kk == 0);
    const bool last = (kk == c.nt - 1);
    const double nadd = last ? nadd_before(kk, DT) : 0.0;   // only the averages of the last sub-step need it
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if ((int)blockIdx.x >= ncell_blocks) {
        path_rescale<false>(n, s, m, path_lane(n, x - ncell_blocks * (int)blockDim.x), DT, first, last, nadd, c.dt_def);
        return;
    }
    // budget terms of the last sub-step go to shared memory where they are computed (dynamic
    // shared memory, kBudgets x blockDim doubles), so they hold no registers across the stage scheme
    extern __shared__ double sbud[];
    double *bt = sbud + threadIdx.x;
    const int bstride = blockDim.x;
    auto bput = [&](int k, double v) { if (last) bt[k * bstride] = v; };
    const int i = x;
    if (last && i >= n.N)
#pragma unroll
        for (int k = 0; k < kBudgets; k++) bt[k * bstride] = 0.0;
    if (i < n.N) store_cell(n, s, m, i, DT, first, last, nadd, c.nt, c.dt_def, bput);
    if (last) {
        double b[kBudgets];
#pragma unroll
        for (int k = 0; k < kBudgets; k++) b[k] = bt[k * bstride];
        warp_budget_partials(s, m, i >> 5, budget_warps(n.N), b);
    }
}

// ------------------------------------------------------------------------------------------
// k_budget: after the sub-step loop, the budgets of every member's last sub-step
// ------------------------------------------------------------------------------------------
// grid (members, kBudgets), kBudgetThreads threads: block (m, k) reduces budget k of member m over
// the warp partials its last sub-step wrote -- thread t sums partials t, t+T, ... in order, then a
// fixed warp tree and a fixed tree over the warps: the same sums whatever the timing
constexpr int kBudgetThreads = 256;
__global__ void __launch_bounds__(kBudgetThreads) k_budget(Net n, State s) {
    const int m = blockIdx.x, k = blockIdx.y;
    if (s.ctl[m].nt < 1) return;                        // refused step (NT cap): no sub-step ran
    const int nw = budget_warps(n.N);
    const double *src = s.partials + ((size_t)m * kBudgets + k) * nw;
    double x = 0.0;
    for (int b = threadIdx.x; b < nw; b += kBudgetThreads) x = x + src[b];
    for (int o = 16; o > 0; o >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, o);
    __shared__ double w[kBudgetThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) w[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int j = 0; j < kBudgetThreads / 32; j++) t = t + w[j];
        s.ctl[m].budget[k] = t;
        if (k == 0 && n.ldiag_out) s.o_nadd[m] = s.o_nadd[m] + s.ctl[m].dt_def;   // NADD_out = NADD_out + DT
    }
}

// CMF_DIAG_GETAVE_OUTPUT (src/cmf_calc_diag_mod.F90:324-356): the output-interval sums divided by
// NADD_out in place (maxima untouched).  Cells on blocks [0, ncell_blocks), path levels after them.
__global__ void k_diag_getave_output(Net n, State s, int ncell_blocks) {
    const int m = blockIdx.y;
    const double na = s.o_nadd[m];
    if ((int)blockIdx.x < ncell_blocks) {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n.N) return;
        const size_t gi = (size_t)m * n.N + i;
        s.o_rivout[gi] = s.o_rivout[gi] / na;
        s.o_fldout[gi] = s.o_fldout[gi] / na;
        s.o_outflw[gi] = s.o_outflw[gi] / na;
        s.o_rivvel[gi] = s.o_rivvel[gi] / na;
        s.o_pthout[gi] = s.o_pthout[gi] / na;
        s.o_runoff[gi] = s.o_runoff[gi] / na;
        if (n.ldamout) s.o_daminf[gi] = s.o_daminf[gi] / na;
    } else {
        const int q = (blockIdx.x - ncell_blocks) * blockDim.x + threadIdx.x;
        const size_t PL = (size_t)n.P * n.Lp;
        if ((size_t)q >= PL) return;
        const size_t o = (size_t)m * PL + q;
        s.o_pthflw[o] = s.o_pthflw[o] / na;
    }
}

// ------------------------------------------------------------------------------------------
// k_outpre: CMF_CALC_OUTPRE (src/cmf_opt_outflw_mod.F90:308-421) -- previous-step discharge by the
// diffusive (Manning) wave, after a storage-only restart and the stage scheme.  Cells on blocks
// [0, ncell_blocks), bifurcation paths on the blocks after them; the downstream surface elevation
// is recomputed from the depth (the same sum the reference stores in D2SFCELV first).
// ------------------------------------------------------------------------------------------
__global__ void k_outpre(Net n, State s, int ncell_blocks) {
    const int m = blockIdx.y;
    const size_t base = (size_t)m * n.N;
    const double p23 = CMF_F(2. / 3.);
    if ((int)blockIdx.x < ncell_blocks) {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n.N) return;
        const size_t gi = base + i;
        const double rivdph = s.rivdph[gi];
        const double sfc = __ldg(&n.rivelv[i]) + rivdph;
        s.sfcelv[gi] = sfc;
        s.rivdph_pre[gi] = rivdph;
        double dslope, dsfcmax, dflw;
        if (i < n.R) {
            const int j = __ldg(&n.next[i]);
            const double sfcj = __ldg(&n.rivelv[j]) + s.rivdph[base + j];
            dsfcmax = dmax(sfc, sfcj);
            dslope = (sfc - sfcj) * (1.0 / __ldg(&n.nxtdst[i]));
            dflw = dsfcmax - __ldg(&n.rivelv[i]);
        } else {
            dsfcmax = sfc;
            dslope = (sfc - __ldg(&n.dwnelv[i])) * (1.0 / n.pdstmth);
            dflw = rivdph;
        }
        const double dslope_f = dmax(-0.005, dmin(0.005, dslope));
        const double darea = __ldg(&n.rivwth[i]) * dflw;
        double rout = 0.0;
        if (darea > CMF_F(1.E-5)) {
            rout = darea * (((1.0 / __ldg(&n.rivman[i])) * pow(dflw, p23)) * sqrt(fabs(dslope)));
            if (dslope < 0.0) rout = -rout;
        }
        const double dflw_f = dmax(dsfcmax - __ldg(&n.elevtn[i]), 0.0);
        double dare_f = s.fldsto[gi] * (1.0 / __ldg(&n.rivlen[i]));
        dare_f = dmax(dare_f - s.flddph[gi] * __ldg(&n.rivwth[i]), 0.0);
        double fout = 0.0;
        if (dare_f > CMF_F(1.E-5)) {
            fout = dare_f * (((1.0 / n.pmanfld) * pow(dflw_f, p23)) * sqrt(fabs(dslope_f)));
            if (dslope_f < 0.0) fout = -fout;
        }
        s.rivout_pre[gi] = rout;
        s.fldout_pre[gi] = n.lfldout ? fout : 0.0;
    } else {
        const int p = (blockIdx.x - ncell_blocks) * blockDim.x + threadIdx.x;
        if (p >= n.P) return;
        const int u = __ldg(&n.pth_up[p]), d = __ldg(&n.pth_dn[p]);
        if (u < 0 || d < 0) return;                    // path leaves the domain
        const size_t pb = (size_t)m * n.Lp * n.P;
        const double su = __ldg(&n.rivelv[u]) + s.rivdph[base + u], sd = __ldg(&n.rivelv[d]) + s.rivdph[base + d];
        const double dslope = (su - sd) * (1.0 / __ldg(&n.pth_dst[p]));
        for (int l = 0; l < n.Lp; l++) {
            const size_t o = (size_t)l * n.P + p;
            const double dflw = dmax(dmax(su, sd) - __ldg(&n.pth_elv[o]), 0.0);
            double f = 0.0;
            if (dflw > CMF_F(1.E-5)) {
                f = (__ldg(&n.pth_wth[o]) * dflw) * (((1.0 / __ldg(&n.pth_man[l])) * pow(dflw, p23)) * sqrt(fabs(dslope)));
                if (dslope < 0.0) f = -f;
            }
            s.pthflw_pre[pb + o] = f;
        }
    }
}

// ------------------------------------------------------------------------------------------
// k_runoff_map: CMF_FORCING_PUT on the device (src/cmf_ctrl_forcing_mod.F90:716-831) for every
// member: the runoff field PBUFF(NXIN,NYIN) of member m is grid[m][NYIN][NXIN] (fp64, or fp32
// promoted exactly).  linterp: ROFF_INTERP over the input matrix (inpx/inpy/inpa [INPN][N]);
// else CONV_RESOL at (inpx, inpy) = (I1SEQX, I1SEQY) with the cell area.  clean applies
// CMF_FORCING_GET's NaN -> RMIS and max(., 0) (:486-494) to every value read.
// ------------------------------------------------------------------------------------------
struct RunoffMap {
    int linterp, nxin, nyin, inpn, clean;
    const int *__restrict__ inpx, *__restrict__ inpy;
    const double *__restrict__ inpa;
    double drofunit;
};

__global__ void k_runoff_map(Net n, State s, RunoffMap r, const double *__restrict__ gridd, const float *__restrict__ gridf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n.N) return;
    const int m = blockIdx.y;
    const size_t g0 = (size_t)m * r.nxin * r.nyin;
    const double rmis = CMF_F(1.E20);
    auto val = [&](int ix, int iy) -> double {
        const size_t k = g0 + (size_t)(iy - 1) * r.nxin + (ix - 1);
        double v = gridd ? gridd[k] : (double)gridf[k];
        if (r.clean) {
            if (isnan(v)) v = rmis;
            v = dmax(v, 0.0);
        }
        return v;
    };
    double out = 0.0;
    if (r.linterp) {
        for (int k = 0; k < r.inpn; k++) {
            const int ix = r.inpx[(size_t)k * n.N + i], iy = r.inpy[(size_t)k * n.N + i];
            if (ix > 0) {
                if (ix > r.nxin || iy > r.nyin || iy < 1) continue;   // the reference logs and skips
                const double v = val(ix, iy);
                if (v != rmis) out = out + (v * r.inpa[(size_t)k * n.N + i]) / r.drofunit;
            }
        }
    } else {
        const double v = val(r.inpx[i], r.inpy[i]);
        if (v != rmis) out = dmax((v * __ldg(&n.grarea[i])) / r.drofunit, 0.0);
    }
    s.runoff[(size_t)m * n.N + i] = out;
}

// k_boundary: CMF_BOUNDARY_UPDATE (src/cmf_ctrl_boundary_mod.F90:267-304): downstream boundary
// elevation D2DWNELV = D2ELEVTN (+ D2MEANSL) (+ D2SEALEV); only the mouths read it.
__global__ void k_boundary(int N, const double *__restrict__ elevtn, const double *__restrict__ meansl,
                           const double *__restrict__ sealev, double *dwnelv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double v = meansl ? elevtn[i] + meansl[i] : elevtn[i];
    if (sealev) v = v + sealev[i];
    dwnelv[i] = v;
}

}  // namespace cmf
