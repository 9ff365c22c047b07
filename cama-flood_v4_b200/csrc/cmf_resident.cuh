// cmf_resident.cuh -- one cooperative launch per outer step (CMF_PHYSICS_ADVANCE,
// src/cmf_ctrl_physics_mod.F90:21-153) that keeps every cell's state on its SM through all sub-steps.
//
// One CTA per SM; warp-tiles of 32 cells of one member are dealt round-robin to the CTAs, so the
// costly tiles near the mouths spread, and stay with one thread each: kResFields doubles of a cell
// live in shared memory, its mostly-zero floodplain and levee state in global memory behind a bit
// that says whether it is zero (dry cells neither read nor write it).  What other cells need goes
// through L2: depth after the stage scheme, the outflow pair before and after the rescale as one
// 16-byte element each (one 32-byte sector per upstream gather instead of three), and the rate.
// The downstream cell's previous depth is the one gathered a sub-step ago, so it is kept, not read.
// The phases of a sub-step are separated by grid barriers, as in the graph of phase kernels, and run
// the same per-cell code (cmf_kernels.cuh) through another accessor: the same bits.
// Bifurcation paths take one lane per (path, level).  Ensembles run in groups of members that fit the
// SMs together, one group after the other.
//
// Why: a sub-step of the phase kernels moves about 530 B per cell through L2 or HBM, and its time is
// dependent rounds of loads in three launches.  Here a phase of a cell is one round: static values and
// neighbours' results, addressed from shared memory.  Measured per sub-step (B200): 298,554 cells with
// channels, levees and dams 38 us (one persistent kernel over global memory 82), 2 x 26,691 cells 20 us (36),
// 10,000 plain cells 12.1 us (21).  What is left: about 1.3 us per barrier, the longest tile of each phase
// (out-of-bank cells with levees, ends of paths), and at full size 16 warps per SM, each at the latency of
// its tile.  A spilled register costs more here than a load of its own: there is little L1 left.
#pragma once
#include "cmf_persist.cuh"

namespace cmf {

enum ResField { F_RIVDPH, F_DPHPRE, F_DWNPRE, F_ROUT, F_FOUT, F_RIVSTO, F_ARIVOUT, F_ARIVVEL, F_MOUTFLW, F_MRIVDPH,
                F_MSTORGE, kResFields };
// a cell's bits: CellFlag (8 bits), then "this array's value of the cell is not +0 and stands in global
// memory" for the arrays that are zero in most cells, then its member within the group (kNoCell: none)
enum ResBit : unsigned { B_FLDSTO = 1 << 8, B_FLDSTOPRE = 1 << 9, B_FLDDPH = 1 << 10, B_FLDFRC = 1 << 11, B_LEVSTO = 1 << 12,
                         B_LEVDPH = 1 << 13, B_AFLDOUT = 1 << 14, B_AOUTFLW = 1 << 15 };
constexpr int kResMemberShift = 16;
constexpr unsigned kNoCell = 0xffffu << kResMemberShift;
// Threads of a CTA at most, and so the registers a thread may have: 16 warps of 128 registers, or, while
// a CTA has no more than kResFewTasks tiles and path tiles, so that a phase is two rounds of warps either
// way, 12 of 168.  Per sub-step, 16 and 12 warps: 10,000 plain cells 12.7 and 12.1 us, 2 x 26,691 cells
// 21.1 and 20.4, 2 x 40,000 (22 tasks) 24.1 and 23.1; 2 x 60,000 (33 tasks) 25.8 and 27.0, 298,554 cells
// 38.2 and 42.7.  Eighteen warps or more spill: 52 us or more at 298,554 cells.
constexpr int kResThreadsMany = 512, kResThreadsFew = 384, kResFewTasks = 2 * (kResThreadsFew / 32);
constexpr int kResMaxGroup = 64;                  // members of one group (their NT/DT sit in shared memory)
// What a cell needs of the network, also on the SM: its index, its downstream cell, its element of the
// exchange arrays, and its upstream cells' range there (first element, count above kResDegShift).  The
// elements are the positions of the upstream CSR, where the upstream cells of a cell are consecutive: a
// phase's gathers start from shared memory instead of a round of index loads.
enum ResInt { I_CELL, I_NEXT, I_ELEM, I_UP, I_BITS, kResInts };
constexpr int kResDegShift = 28;
// Dynamic shared memory of a CTA with `slots` tiles: the fields, then the integers
__host__ __device__ constexpr size_t res_smem(int slots) {
    return (size_t)slots * 32 * (kResFields * sizeof(double) + kResInts * sizeof(int));
}
constexpr int kResMaxSlots = (227 * 1024 - 2560) / (int)res_smem(1);   // 2 KB stay for the static part

struct ResArgs {
    int tpm;                    // 32-cell tiles per member
    int group;                  // members per group
    int slots;                  // tiles of a CTA
    int selftest;               // 1: only run a barrier whose count can never complete (timeout check)
    unsigned long long wait_ns; // bound of every device-side wait
    int edges;                  // elements per member of raw and out
    int cells;                  // entries of `order`
    const int *order;           // cells in the order they are dealt to the tiles (-1: none)
    const int *xpos;            // [N] a cell's element (-1: no cell gathers it)
    double2 *raw, *out;         // [group * edges] outflow pairs before and after the rescale
    double *terms;              // [kBudgets][group * tpm * 32] budget terms of the last sub-step
};

struct OwnR : OwnMaps {
    static constexpr bool kResident = true;
    const State &s;
    double *f;                  // this cell's fields, `stride` doubles apart
    int stride;
    unsigned &bits;
    int nxt, x, up;             // downstream cell, element, upstream range
    double2 *raw, *out;         // the member's elements
    bool first_step, waiting;   // waiting: phase B of a dam cell
    __device__ __forceinline__ OwnR(const Net &n_, const State &s_, double *f_, int stride_, const int *ints, unsigned &b_,
                                    const ResArgs &a, int ml, bool first, bool phase_b = false)
        : OwnMaps{n_}, s(s_), f(f_), stride(stride_), bits(b_), nxt(ints[I_NEXT * stride_]), x(ints[I_ELEM * stride_]),
          up(ints[I_UP * stride_]), raw(a.raw + (size_t)ml * a.edges), out(a.out + (size_t)ml * a.edges), first_step(first), waiting(phase_b && (b_ & C_DAM)) {}
    __device__ __forceinline__ int next(int) const { return nxt; }
    __device__ __forceinline__ unsigned flags() const { return bits; }
    __device__ __forceinline__ double get(int k) const { return f[k * stride]; }
    __device__ __forceinline__ void put(int k, double v) const { f[k * stride] = v; }
    __device__ __forceinline__ double sparse(unsigned bit, const double *p, size_t g) const { return (bits & bit) ? p[g] : 0.0; }
    __device__ __forceinline__ void put_sparse(unsigned bit, double *p, size_t g, double v) const {
        if (__double_as_longlong(v) != 0) {
            p[g] = v;
            bits |= bit;
        } else {
            bits &= ~bit;
        }
    }
    __device__ __forceinline__ double rivsto(size_t) const { return get(F_RIVSTO); }
    __device__ __forceinline__ double fldsto(size_t g) const { return sparse(B_FLDSTO, s.fldsto, g); }
    __device__ __forceinline__ double levsto(size_t g) const { return sparse(B_LEVSTO, s.levsto, g); }
    __device__ __forceinline__ bool flooded() const { return bits & B_FLDSTO; }
    __device__ __forceinline__ double rivdph(size_t) const { return get(F_RIVDPH); }
    __device__ __forceinline__ double rivdph_pre(size_t) const { return get(F_DPHPRE); }
    __device__ __forceinline__ double rivout_pre(size_t) const { return get(F_ROUT); }
    __device__ __forceinline__ double fldout_pre(size_t) const { return get(F_FOUT); }
    __device__ __forceinline__ double fldsto_pre(size_t g) const { return sparse(B_FLDSTOPRE, s.fldsto_pre, g); }
    __device__ __forceinline__ double flddph(size_t g) const { return sparse(B_FLDDPH, s.flddph, g); }
    __device__ __forceinline__ double fldfrc(size_t g) const { return sparse(B_FLDFRC, s.fldfrc, g); }
    __device__ __forceinline__ double runoff(size_t g) const { return s.runoff[g]; }
    // (F_ROUT, F_FOUT): the last sub-step's outflow until phase A, then before the rescale, and from
    // phase B on after it unless the flow is reverse.  A dam cell's outflow comes from a task of its own
    // in phase A, while the task of its diagnostics still reads the pair of the last sub-step, so it waits
    // in the phase kernels' arrays for phase B
    __device__ __forceinline__ double2 own_raw(size_t g) const { return waiting ? s.raw[g] : own_out(g); }
    __device__ __forceinline__ double2 own_out(size_t) const { return make_double2(get(F_ROUT), get(F_FOUT)); }
    __device__ __forceinline__ LazyRate rate(size_t g) const { return {s.rate + g, true}; }
    __device__ __forceinline__ double a_rivvel(size_t) const { return get(F_ARIVVEL); }
    __device__ __forceinline__ double a_rivout(size_t) const { return get(F_ARIVOUT); }
    __device__ __forceinline__ double a_fldout(size_t g) const { return sparse(B_AFLDOUT, s.a_fldout, g); }
    // the running sum of rivout + fldout is that of rivout while fldout was +0 in every sub-step so far
    __device__ __forceinline__ double a_outflw(size_t g) const { return (bits & B_AOUTFLW) ? s.a_outflw[g] : get(F_ARIVOUT); }
    __device__ __forceinline__ double a_pthout(size_t g) const { return s.a_pthout[g]; }
    __device__ __forceinline__ double m_outflw(size_t) const { return get(F_MOUTFLW); }
    __device__ __forceinline__ double m_rivdph(size_t) const { return get(F_MRIVDPH); }
    __device__ __forceinline__ double m_storge(size_t) const { return get(F_MSTORGE); }
    // values of other CTAs' cells: past L1, which may hold an older sub-step's line
    __device__ __forceinline__ double nb(const double *p, size_t g) const { return __ldcg(p + g); }
    __device__ __forceinline__ DownCell down(size_t base, int i, int j) const {
        const double d = __ldcg(s.rivdph + base + j);
        const double pre = first_step ? __ldcg(s.rivdph_pre + base + j) : get(F_DWNPRE);
        put(F_DWNPRE, d);
        return {__ldg(&n.next_rivelv[i]), d, pre};
    }
    __device__ __forceinline__ void put_raw(size_t g, int, double rout, double fout) const {
        if (bits & C_DAM) {      // see own_raw
            s.raw[g] = make_double2(rout, fout);
        } else {
            put(F_ROUT, rout);
            put(F_FOUT, fout);
        }
        if (x >= 0) raw[x] = make_double2(rout, fout);
    }
    __device__ __forceinline__ void put_rate(size_t g, int i, double rout, double fout, double r) const {
        s.rate[g] = r;
        const double2 v = rescale_own(rout, fout, r, i >= n.R);
        if (v.x != v.x) s.raw[g] = make_double2(rout, fout);       // for this cell's phase C
        put(F_ROUT, v.x);
        put(F_FOUT, v.y);
        if (x >= 0) out[x] = v;
    }
    __device__ __forceinline__ void put_a_rivvel(size_t, double v) const { put(F_ARIVVEL, v); }
    __device__ __forceinline__ void put_pre(size_t g, double rout, double fout, double dph, double fld, bool) const {
        put(F_ROUT, rout);
        put(F_FOUT, fout);
        put(F_DPHPRE, dph);
        put_sparse(B_FLDSTOPRE, s.fldsto_pre, g, fld);
        if (bits & C_DAM) {      // read by the dam cells downstream
            s.rivout_pre[g] = rout;
            s.fldout_pre[g] = fout;
        }
        if (bits & C_END) s.rivdph_pre[g] = dph;
    }
    template <class Out>
    __device__ __forceinline__ void put_stage(size_t g, const Out &o, double sto, double, bool) const {
        put(F_RIVSTO, o.rivsto);
        put(F_RIVDPH, o.rivdph);
        s.rivdph[g] = o.rivdph;
        put_sparse(B_FLDSTO, s.fldsto, g, o.fldsto);
        put_sparse(B_FLDDPH, s.flddph, g, o.flddph);
        put_sparse(B_FLDFRC, s.fldfrc, g, o.fldfrc);
        if (n.llevee) {
            put_sparse(B_LEVSTO, s.levsto, g, o.levsto);
            put_sparse(B_LEVDPH, s.levdph, g, o.levdph);
        }
        if (bits & C_END) {      // read by the paths at this cell
            s.storge[g] = sto;
            if (n.llevee) s.levdph[g] = o.levdph;
        }
    }
    template <class F>
    __device__ __forceinline__ void each_pair(const double2 *m, F fn) const {
        const int deg = (unsigned)up >> kResDegShift;
        const double2 *p = m + (up & ((1 << kResDegShift) - 1));
        for (int e = 0; e < deg; e += 4) {
            double2 v[4];
#pragma unroll
            for (int b = 0; b < 4; b++)
                if (e + b < deg) v[b] = __ldcg(p + e + b);
#pragma unroll
            for (int b = 0; b < 4; b++)
                if (e + b < deg) fn(v[b].x, v[b].y);
        }
    }
    template <class F>
    __device__ __forceinline__ void each_raw(size_t, int, F fn) const { each_pair(raw, fn); }
    template <class Rate, class F>
    __device__ __forceinline__ void each_out(size_t, int, Rate rate_i, F fn) const {
        each_pair(out, [&](double rj, double fj) { rescaled(make_double2(rj, fj), rate_i, fn); });
    }
    template <class F>
    __device__ __forceinline__ void each_by_sign(size_t base, int, double rate_i, F fn) const {
        const int first = up & ((1 << kResDegShift) - 1), end = first + (int)((unsigned)up >> kResDegShift);
        for (int e = first; e < end; e++) by_sign(__ldcg(raw + e), __ldcg(s.rate + base + __ldg(&n.up_idx[e])), rate_i, fn);
    }
    // the previous sub-step's averages and maxima (diag_carry with the sums held on the SM)
    __device__ __forceinline__ void carry(size_t g, double DT, bool first, double rout, double fout, double dph, double sto) const {
        const double outflw = rout + fout;
        const double pro = first ? 0.0 : get(F_ARIVOUT);
        if (same_bits(outflw, rout) && (first || !(bits & B_AOUTFLW))) {
            bits &= ~B_AOUTFLW;
        } else {
            const double prev = first ? 0.0 : a_outflw(g);
            s.a_outflw[g] = first ? outflw * DT : prev + outflw * DT;
            bits |= B_AOUTFLW;
        }
        put(F_ARIVOUT, first ? rout * DT : pro + rout * DT);
        if (__double_as_longlong(fout) != 0 || (bits & B_AFLDOUT)) {
            const double prev = first ? 0.0 : a_fldout(g);
            put_sparse(B_AFLDOUT, s.a_fldout, g, first ? fout * DT : prev + fout * DT);
        }
        put(F_MOUTFLW, dmax(first ? 0.0 : get(F_MOUTFLW), fabs(outflw)));
        put(F_MRIVDPH, dmax(first ? 0.0 : get(F_MRIVDPH), dph));
        put(F_MSTORGE, dmax(first ? 0.0 : get(F_MSTORGE), sto));
    }
};

template <int Threads>
__global__ void __launch_bounds__(Threads, 1) k_resident(Net n, State s, ResArgs a) {
    extern __shared__ double fields[];
    __shared__ int sflag, s_nt[kResMaxGroup], s_ntmax, s_q[3], s_nd, s_dam[kResMaxSlots];
    __shared__ double s_dt[kResMaxGroup], s_bud[kBudgetThreads / 32];
    __shared__ unsigned long long s_min[kResMaxGroup];
    const unsigned G = gridDim.x, b = blockIdx.x;
    const int tid = threadIdx.x, nw = blockDim.x >> 5, warp = tid >> 5, lane = tid & 31;
    GridBar gb{&s.loop->bar, &s.ctl[0].bar_err, G, 0u, a.wait_ns, &sflag};
    if (a.selftest) {           // the count target includes one arrival that never comes
        gb.nblocks = G + 1;
        gb.sync();
        return;
    }
    const int N = n.N, tpm = a.tpm, slots = a.slots, stride = slots * 32;
    int *s_int = reinterpret_cast<int *>(fields + (size_t)kResFields * stride);    // [kResInts][slots * 32]
    int *s_cell = s_int + I_CELL * stride;
    unsigned *s_bits = reinterpret_cast<unsigned *>(s_int + I_BITS * stride);
    const bool split = s.loop->split != 0;
    const int ptpm = path_threads(n.P, n.Lp) >> 5;       // path tiles (warps) per member
    if (tid < 3) s_q[tid] = 0;
    // the warps of a CTA take its tiles from a counter per phase: a tile's state is in shared memory, so
    // any warp can run it, and the long tiles (dams, path ends, paths), which come first, do not hold
    // back the ones behind them
    auto next = [&](int phase) -> int {
        int q = 0;
        if (lane == 0) q = atomicAdd(&s_q[phase], 1);
        return __shfl_sync(0xffffffffu, q, 0);
    };
    int gntmax = 1;             // CTA 0, thread 0: the step's counters over all groups
    long long ntsum = 0, near = 0;

    for (int m0 = 0; m0 < n.M; m0 += a.group) {
        const int mg = min(a.group, n.M - m0), T = mg * tpm, PT = mg * ptpm;
        const int npath = PT > (int)b ? (PT - 1 - (int)b) / (int)G + 1 : 0;      // this CTA's path tiles
        const size_t nterm = (size_t)a.group * tpm * 32;
        // ---- stage scheme at the top of the step + CALC_ADPSTP minimum (k_stage)
        for (int ml = tid; ml < mg; ml += blockDim.x) s_min[ml] = ~0ull;
        if (tid == 0) {
            s_ntmax = 1;
            s_nd = 0;
        }
        __syncthreads();
#pragma unroll 1
        for (int c = warp; c < slots; c += nw) {
            const int t = c * (int)G + (int)b, slot = c * 32 + lane;
            double key = 1.0e308;
            unsigned bits = kNoCell;
            const int ml = t < T ? t / tpm : 0, e = (t - ml * tpm) * 32 + lane;
            const int i = t < T && e < a.cells ? __ldg(&a.order[e]) : -1;
            if (i >= 0) {
                const int m = m0 + ml;
                const size_t gi = (size_t)m * N + i;
                s_cell[slot] = i;
                s_int[I_NEXT * stride + slot] = __ldg(&n.next[i]);
                s_int[I_ELEM * stride + slot] = __ldg(&a.xpos[i]);
                const int u0 = __ldg(&n.up_ptr[i]);
                s_int[I_UP * stride + slot] = u0 | (__ldg(&n.up_ptr[i + 1]) - u0) << kResDegShift;
                bits = __ldg(&n.cflag[i]) | (unsigned)ml << kResMemberShift;
                OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, ml, true);
                const StageOut o = stage(n, w, i, stage_map(w, i), s.rivsto[gi], s.fldsto[gi], n.llevee ? s.levsto[gi] : 0.0);
                store_stage(n, s, w, gi, i, o, 0.0, true);
                w.put(F_ROUT, s.rivout_pre[gi]);
                w.put(F_FOUT, s.fldout_pre[gi]);
                w.put(F_DPHPRE, s.rivdph_pre[gi]);
                if (__double_as_longlong(s.fldsto_pre[gi]) != 0) bits |= B_FLDSTOPRE;
                if (n.ladpstp && __ldg(&n.i2mask[i]) == 0) key = cfl_key(n.pcadp, (i < n.R) ? __ldg(&n.nxtdst[i]) : n.pdstmth, n.pgrv, o.rivdph);
            }
            s_bits[slot] = bits;
            if (__any_sync(0xffffffffu, bits < kNoCell && (bits & C_DAM)) && lane == 0) s_dam[atomicAdd(&s_nd, 1)] = c;
            if (n.ladpstp && t < T) {
                for (int o = 16; o > 0; o >>= 1) key = dmin(key, __shfl_down_sync(0xffffffffu, key, o));
                if (lane == 0 && key < 1.0e308) atomicMin(&s_min[ml], (unsigned long long)__double_as_longlong(key));
            }
        }
        __syncthreads();
        if (n.ladpstp)
            for (int ml = tid; ml < mg; ml += blockDim.x)
                if (s_min[ml] != ~0ull) atomicMin(&s.ctl[m0 + ml].dtmin_bits, s_min[ml]);
        if (!gb.sync()) return;
        // ---- NT/DT: every CTA derives them from the minimum, CTA 0 keeps the books
        for (int ml = tid; ml < mg; ml += blockDim.x) {
            MemberCtl &c = s.ctl[m0 + ml];
            const NtDt r = calc_ntdt(n, c.dt_def, __ldcg(&c.dtmin_bits));
            s_nt[ml] = r.nt;
            s_dt[ml] = r.dt;
            atomicMax(&s_ntmax, r.nt);
            if (b == 0) {
                put_ntdt(c, s.loop, r);
                s_min[ml] = r.near;
            }
        }
        __syncthreads();
        const int ntmax = min(s_ntmax, kNtCap);
        if (b == 0 && tid == 0) {
            gntmax = max(gntmax, ntmax);
            for (int k = 0; k < mg; k++) {
                ntsum += s_nt[k];
                near += (long long)s_min[k];
            }
        }

        for (int k = 0; k < ntmax; k++) {
            // ---- phase A: reservoir operation, bifurcation flux, outflow
            const int nd = s_nd;
            for (int q; (q = next(0)) < nd + npath + slots;) {
                if (q < nd) {
                    const int slot = s_dam[q] * 32 + lane;
                    unsigned bits = s_bits[slot];
                    const int ml = bits >> kResMemberShift;
                    if (bits >= kNoCell || !(bits & C_DAM) || k >= s_nt[ml]) continue;
                    const int i = s_cell[slot], m = m0 + ml;
                    OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, ml, k == 0);
                    cell_dam(n, s, w, m, i, s_dt[ml], s_nt[ml], s.ctl[m].dt_def, k);
                } else if (q < nd + npath) {
                    const int t = (q - nd) * (int)G + (int)b, ml = t / ptpm;
                    if (k >= s_nt[ml]) continue;             // uniform over the warp
                    path_outflow<true>(n, s, m0 + ml, path_lane(n, (t - ml * ptpm) * 32 + lane), s_dt[ml]);
                } else {
                    const int slot = (q - nd - npath) * 32 + lane;
                    unsigned bits = s_bits[slot];
                    const int ml = bits >> kResMemberShift;
                    if (bits >= kNoCell || k >= s_nt[ml]) continue;
                    const int i = s_cell[slot], m = m0 + ml;
                    OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, ml, k == 0);
                    cell_outflow(n, s, w, m, i, s_dt[ml], s_nt[ml], s.ctl[m].dt_def, k, split && k == 0);
                    s_bits[slot] = bits;
                }
            }
            if (!gb.sync()) return;
            if (tid == 0) s_q[0] = 0;
            // ---- phase B: storage-out gather and rate
            for (int q; (q = next(1)) < slots;) {
                const int slot = q * 32 + lane;
                unsigned bits = s_bits[slot];
                const int ml = bits >> kResMemberShift;
                if (bits >= kNoCell || k >= s_nt[ml]) continue;
                const int i = s_cell[slot];
                OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, ml, k == 0, true);
                cell_rate(n, s, w, m0 + ml, i, s_dt[ml]);
            }
            if (!gb.sync()) return;
            if (tid == 0) s_q[1] = 0;
            // ---- phase C: rescale, inflow, STONXT, stage scheme; path rescale
            for (int q; (q = next(2)) < slots + npath;) {
                if (q < slots) {
                    const int slot = q * 32 + lane;
                    unsigned bits = s_bits[slot];
                    const int ml = bits >> kResMemberShift;
                    if (bits >= kNoCell || k >= s_nt[ml]) continue;
                    const int i = s_cell[slot], m = m0 + ml, nt = s_nt[ml];
                    const double DT = s_dt[ml];
                    const bool last = k == nt - 1;
                    const double nadd = last ? nadd_before(k, DT) : 0.0;
                    // the last sub-step's budget terms go out by cell: they are summed below in the
                    // sequence's order, whatever order the tiles have
                    double *term = a.terms + (size_t)ml * tpm * 32 + i;
                    auto bput = [&](int j, double v) { if (last) term[j * nterm] = v; };
                    OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, ml, k == 0);
                    cell_store(n, s, w, m, i, DT, k == 0, last, nadd, nt, s.ctl[m].dt_def, bput);
                    s_bits[slot] = bits;
                } else {
                    const int t = (q - slots) * (int)G + (int)b, ml = t / ptpm, nt = s_nt[ml];
                    if (k >= nt) continue;
                    const double DT = s_dt[ml];
                    const bool last = k == nt - 1;
                    const double nadd = last ? nadd_before(k, DT) : 0.0, ddef = s.ctl[m0 + ml].dt_def;
                    path_rescale<true>(n, s, m0 + ml, path_lane(n, (t - ml * ptpm) * 32 + lane), DT, k == 0, last, nadd, ddef);
                }
            }
            if (!gb.sync()) return;
            if (tid == 0) s_q[2] = 0;
        }
        // ---- the state the caller observes, from the SM to its arrays
#pragma unroll 1
        for (int c = warp; c < slots; c += nw) {
            const int slot = c * 32 + lane;
            unsigned bits = s_bits[slot];
            if (bits >= kNoCell) continue;
            const size_t gi = (size_t)(m0 + (bits >> kResMemberShift)) * N + s_cell[slot];
            OwnR w(n, s, fields + slot, stride, s_int + slot, bits, a, 0, false);
            s.rivsto[gi] = w.get(F_RIVSTO);
            s.rivout_pre[gi] = w.get(F_ROUT);
            s.fldout_pre[gi] = w.get(F_FOUT);
            s.rivdph_pre[gi] = w.get(F_DPHPRE);
            const double riv_fld = w.rivsto(gi) + w.fldsto(gi);
            s.storge[gi] = n.llevee ? riv_fld + w.levsto(gi) : riv_fld;
            if (!(bits & B_FLDSTO)) s.fldsto[gi] = 0.0;
            if (!(bits & B_FLDSTOPRE)) s.fldsto_pre[gi] = 0.0;
            if (!(bits & B_FLDDPH)) s.flddph[gi] = 0.0;
            if (!(bits & B_FLDFRC)) s.fldfrc[gi] = 0.0;
            if (n.llevee) {
                if (!(bits & B_LEVSTO)) s.levsto[gi] = 0.0;
                if (!(bits & B_LEVDPH)) s.levdph[gi] = 0.0;
            }
        }
        // ---- budgets of every member's last sub-step: k_store's partials per warp of 32 consecutive
        // cells, then k_budget's tree
        const int nwarp = budget_warps(N);
        for (int t = warp * (int)G + (int)b; t < mg * nwarp; t += nw * (int)G) {
            const int ml = t / nwarp, tile = t - ml * nwarp, i = tile * 32 + lane;
            if (s_nt[ml] < 1) continue;
            const double *src = a.terms + (size_t)ml * tpm * 32 + i;
            double *part = s.partials + (size_t)(m0 + ml) * kBudgets * nwarp + tile;
#pragma unroll
            for (int q = 0; q < kBudgets; q++) {
                double x = i < N ? __ldcg(src + q * nterm) : 0.0;
                for (int o = 16; o > 0; o >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, o);
                if (lane == 0) part[(size_t)q * nwarp] = x;
            }
        }
        if (!gb.sync()) return;
        for (int r = b; r < mg * kBudgets; r += G) {
            const int ml = r / kBudgets, q = r % kBudgets;
            if (s_nt[ml] < 1) continue;
            const double *part = s.partials + ((size_t)(m0 + ml) * kBudgets + q) * nwarp;
            for (int v = warp; v < kBudgetThreads / 32; v += nw) {
                double x = 0.0;
                for (int e = v * 32 + lane; e < nwarp; e += kBudgetThreads) x = x + __ldcg(part + e);
                for (int o = 16; o > 0; o >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, o);
                if (lane == 0) s_bud[v] = x;
            }
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int j = 0; j < kBudgetThreads / 32; j++) t = t + s_bud[j];
                s.ctl[m0 + ml].budget[q] = t;
                if (q == 0 && n.ldiag_out) s.o_nadd[m0 + ml] = s.o_nadd[m0 + ml] + s.ctl[m0 + ml].dt_def;
            }
            __syncthreads();
        }
        // every CTA has read the minima (barriers ago): the next step's start from DT again
        if (b == 0 && n.ladpstp)
            for (int ml = tid; ml < mg; ml += blockDim.x)
                s.ctl[m0 + ml].dtmin_bits = (unsigned long long)__double_as_longlong(s.ctl[m0 + ml].dt_def);
        __syncthreads();        // s_nt, s_min and the fields are reused by the next group
    }
    if (b == 0 && tid == 0) {
        s.loop->ntmax = gntmax;
        s.loop->near_int += near;
        s.loop->member_substeps += ntsum;
        s.loop->loop_iters += gntmax;
        s.loop->outer_steps += 1;
        s.loop->split = 0;
    }
}

}  // namespace cmf
