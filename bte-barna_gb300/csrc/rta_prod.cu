// rta_prod.cu - production mode of the RTA particle loop.
//
// Draws come from counter-based Philox4x32-10 streams keyed by (seed,
// particle); mode distributions and Lambert rows are sampled through alias
// tables; positions and times are doubles, or on the grid path 64-bit
// integers of a finer resolution (fixed_walk.cuh); tallies are reduced by
// FP64 atomics.  Three kernels:
//   rta_prod_general  any convex-box geometry, the flight logic of
//                     rta_flight.cuh (one evolparticle step per pass);
//   rta_prod_grid     boxes that tile an axis-aligned grid: a persistent
//                     kernel whose warps refill idle lanes with new particles
//                     and that walks cells by exit times, with a per-lane
//                     pending tally flushed when the (box, bin) key changes;
//   rta_prod_poly     the grid kernel's loop over any convex boxes, exit
//                     times taken against each box's border lines.
#include "kernels.h"
#include "prod_common.cuh"
#include "rta_steady.cuh"

namespace bte {

// Any convex-box geometry, the flight logic of rta_flight.cuh, one
// evolparticle step per loop pass.  Warps are persistent
// and a lane whose particle has finished takes the next one from a global
// counter (one atomic per warp), so lanes stay busy while particles of very
// different lifetimes run out; each particle keeps its own Philox stream,
// so its trajectory does not depend on the lane.
__global__ void __launch_bounds__(128) rta_prod_general(DevTables T, double* tally,
                                                        unsigned long long* counters, int* err,
                                                        unsigned long long* work) {
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const long long total = T.pend - T.pbegin;
    ProdPolicy pol;
    pol.g.init(0, 0);
    pol.out = tally;
    pol.ntally = 0;
    Particle p;
    p.pos = v2(0., 0.);
    p.mode = 0;
    p.sign = 1;
    p.t = 0.;
    p.box = 0;
    p.mo = 0;
    V2 v = v2(0., 0.);
    double dt = 0., time = 0.;
    int nudges = 0, guard = 0, fate = FATE_LOST;
    long long nev = 0, pid = -1;
    bool active = false, done = false, need_flight = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (idle) {
            unsigned long long base = 0;
            const int leader = __ffs(idle) - 1;
            if (lane == leader) base = atomicAdd(work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                const long long mine = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (mine < total) {
                    pid = T.pbegin + mine;
                    pol.g.init(T.seed, (uint64_t)pid);
                    const int e = generate(T, pol, pid, p);
                    if (e) {
                        record_error(err, e, pid);
                    } else {
                        active = true;
                        need_flight = true;
                        time = 0.;
                        nudges = 0;
                        nev = 0;
                    }
                } else {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (!active) continue;
        if (need_flight) {  // draw the next free flight
            if (!(time < T.maxtime)) {
                active = false;
                continue;
            }
            const int k = p.mode;
            if (++nev > T.flight_cap || T.w[p.mo + k] == 0.) {
                record_error(err, nev > T.flight_cap ? E_LIMIT : E_VALUE, pid);
                active = false;
                continue;
            }
            v = v2(T.vxc[k], T.vyc[k]);
            dt = pol.flight(T, p.mo + k);
            c.events++;
            if (time + dt > T.maxtime) dt = T.maxtime - time + 1.0e-8;
            guard = 0;
            fate = FATE_LOST;
            need_flight = false;
        }
        if (!almost_equal(dt, 0.)) {
            int e = ++guard > FLIGHT_CAP ? E_LIMIT : 0;
            if (!e) e = evolparticle(T, pol, p, v, dt, c, nudges, fate);
            if (e) {
                record_error(err, e, pid);
                active = false;
                continue;
            }
        }
        if (almost_equal(dt, 0.)) {  // the flight is over
            if (p.mode == 0) {       // absorbed
                active = false;
                continue;
            }
            time = p.t;
            need_flight = true;
        }
    }
    c.tallies += pol.ntally;
    flush_counters_p<13>(c, counters);
}

// Generation 0: 1 per slot whose first draw picks a gradient generator.
__global__ void steady_select_prod(SteadyArgs A, unsigned long long seed, unsigned* flags) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < A.n; s += stride) {
        Philox g;
        g.init(seed, steady_stream(0, s));
        flags[s] = steady_gen_type(A, g.uniform()) == 1 ? 1u : 0u;
    }
}

// One generation: each slot's one flight, one evolparticle step per loop
// pass, with persistent warps whose finished lanes take the next slot.
__global__ void __launch_bounds__(128) rta_steady_prod(DevTables T, SteadyArgs A, double* tally,
                                                       unsigned long long* counters, int* err) {
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    ProdPolicy pol;
    pol.g.init(0, 0);
    pol.out = tally;
    pol.ntally = 0;
    Particle p;
    p.pos = v2(0., 0.);
    p.mode = 0;
    p.sign = 1;
    p.t = 0.;
    p.box = 0;
    p.mo = 0;
    V2 v = v2(0., 0.);
    double dt = 0.;
    int nudges = 0, guard = 0, fate = FATE_LOST;
    long long slot = -1;
    bool active = false, done = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (idle) {
            unsigned long long base = 0;
            const int leader = __ffs(idle) - 1;
            if (lane == leader) base = atomicAdd(A.work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                slot = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (slot < A.n) {
                    pol.g.init(T.seed, steady_stream(A.gen, slot));
                    const int e = steady_begin(T, A, pol, slot, c, p, v, dt);
                    if (e) {
                        record_error(err, e, slot);
                        A.flag[slot] = 0;
                    } else {
                        active = true;
                        fate = FATE_LOST;
                        guard = 0;
                        nudges = 0;
                    }
                } else {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (!active) continue;
        if (!almost_equal(dt, 0.)) {
            int e = ++guard > FLIGHT_CAP ? E_LIMIT : 0;
            if (!e) e = evolparticle<ProdPolicy, true>(T, pol, p, v, dt, c, nudges, fate);
            if (e) {
                record_error(err, e, slot);
                A.flag[slot] = 0;
                active = false;
                continue;
            }
        }
        if (almost_equal(dt, 0.)) {  // the flight is over
            if (fate == FATE_LOST) c.lost++;
            steady_emit(A, slot, fate, p);
            active = false;
        }
    }
    c.tallies += pol.ntally;
    flush_counters_p<13>(c, counters);
}

void launch_steady_prod(const DevTables& T, const SteadyArgs& A, double* tally,
                        unsigned long long* counters, int* err, unsigned* select_flags, int nsm,
                        cudaStream_t s) {
    if (A.n <= 0) return;
    long long blocks = (A.n + 127) / 128;
    if (select_flags) {
        const long long cap = (long long)nsm * 16;
        if (blocks > cap) blocks = cap;
        steady_select_prod<<<unsigned(blocks), 128, 0, s>>>(A, T.seed, select_flags);
        return;
    }
    const long long cap = (long long)nsm * 4;  // resident blocks of the persistent kernel (128 registers)
    if (blocks > cap) blocks = cap;
    cudaMemsetAsync(A.work, 0, sizeof(unsigned long long), s);
    rta_steady_prod<<<unsigned(blocks), 128, 0, s>>>(T, A, tally, counters, err);
}

void launch_prod_general(const DevTables& T, double* tally, unsigned long long* counters,
                         int* err, unsigned long long* work, int nsm, cudaStream_t s) {
    const long long n = T.pend - T.pbegin;
    if (n <= 0) return;
    long long blocks = (n + 127) / 128;
    const long long cap = (long long)nsm * 3;  // resident blocks (145 registers x 128 threads)
    if (blocks > cap) blocks = cap;
    rta_prod_general<<<unsigned(blocks), 128, 0, s>>>(T, tally, counters, err, work);
}

// ------------------------------------------------------------------ grid path

struct GridParticle {
    double x, y;   // generated position, nm
    int i, j;      // cell
    int mode;
    int sign;
    int box;
    int mo;        // material offset (material * n)
};

// Pending tally of one lane.  Inside one (box, time bin) key the particle
// moves continuously, so the key's contributions telescope: time spent =
// r0 - r, r the time left to the bin's end, and the velocity-weighted sums
// are the displacement x - x0, y - y0 (sum of v * dt over the segments).
// Nothing is accumulated per segment; when the key changes the three
// differences go out as FP64 atomics, with the particle sign applied to the
// sign bit.
struct Pending {
    int key;
    unsigned flushes;
    double r0, x0, y0;
    __device__ __forceinline__ void start(int k, double r, double x, double y) {
        key = k;
        r0 = r;
        x0 = x;
        y0 = y;
    }
    __device__ __forceinline__ void flush(double* tally, unsigned long long signbit, double r, double x,
                                          double y) {
        if (key >= 0) {
            double* b = tally + 3ll * key;
            atomicAdd(b + 0, __longlong_as_double(__double_as_longlong(r0 - r) ^ signbit));
            atomicAdd(b + 1, __longlong_as_double(__double_as_longlong(x - x0) ^ signbit));
            atomicAdd(b + 2, __longlong_as_double(__double_as_longlong(y - y0) ^ signbit));
            flushes++;
        }
        key = -1;
    }
};

// Generate particle `pid` on the grid.  Returns 0 or an error code.
__device__ int grid_generate(const DevTables& T, const DevGrid& G, const int2* boxcell, Philox& g,
                             long long pid, GridParticle& p) {
    int box;
    if (T.source == 0) {
        (void)g.uniform();  // generator-type draw of Init_generator
        const double where = g.uniform();
        int gi = lower_bound_d(T.wall_cum, T.ngen, where);
        if (gi >= T.ngen) gi = T.ngen - 1;
        const WallGenDev W = T.walls[gi];
        const double u = g.uniform();
        p.x = W.p1.x + u * W.nd.x;
        p.y = W.p1.y + u * W.nd.y;
        box = W.box;
        p.sign = W.sign;
        const long long o = (long long)gi * T.n;
        p.mode = alias_draw(g, T.gen_prob + o, T.gen_alt + o, T.n);
    } else {
        int lo = 0, hi = T.ngen;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(T.init_first + mid) <= pid) lo = mid; else hi = mid;
        }
        box = __ldg(T.init_box + lo);
        const int2 ij = __ldg(boxcell + box);
        const double x0 = __ldg(G.gx + ij.x), x1 = __ldg(G.gx + ij.x + 1);
        const double y0 = __ldg(G.gy + ij.y), y1 = __ldg(G.gy + ij.y + 1);
        p.x = x0 + g.uniform() * (x1 - x0);
        p.y = y0 + g.uniform() * (y1 - y0);
        p.sign = __ldg(T.init_sign + lo);
        const long long o = (long long)lo * T.n;
        p.mode = alias_draw(g, T.gen_prob + o, T.gen_alt + o, T.n);
    }
    const int2 ij = __ldg(boxcell + box);
    p.i = ij.x;
    p.j = ij.y;
    p.box = box;
    p.mo = mat_off(T, box);
    return 0;
}

// One lane carries one particle; each pass of the loop advances every active
// lane by exactly one segment, which ends at the first of: the end of the
// free flight, the next cell line, the next time-bin border (the last one is
// maxtime).  Positions and times are 64-bit integers (fixed_walk.cuh): the
// particle's cell, the distance (ax, ay) to the cell's borders ahead of it,
// and the pending tally as time and signed displacement since its (box, bin)
// key opened, so a segment is two exit times, two products and a few
// subtractions on the integer units.  In doubles the same segment held the
// SM's two FP64 lanes for 200 cycles a pass and bounded the kernel at 75 %
// busy; now the FP64 pipe only turns the three pending sums into doubles
// (17 cycles each), and the kernel is bound by instruction issue: 2e6
// particles of the porous transient (36864 modes, 2422 cells, 200 bins) take
// 106-111 ms instead of 144-152, the 1e6-particle ribbon 3.06 instead of 4.78.
// Of 32 lanes 20 are active (57 % of the passes end in a draw, the others in a
// flush, and a warp issues both), 456 instructions a pass, 62 % of the issue
// slots taken.  A lane
// flushes at most once per pass; a sum of zero (a mode without velocity) adds
// nothing and is not sent.  The tally is left in the walk's units (ticks, and
// position units), which the reader scales by powers of two.
// Idle lanes take new particles from a global counter, one atomic per warp.
// The random words of a pass come from one Philox block per lane
// (pass_block); a flight that ends at a void wall or by scattering draws
// its next mode in one block for both cases (Lambert row or post-scattering
// alias table) and draws the next flight length there.
//
// ADJ selects the two passes of the adjoint (ADJ = 0 is the plain kernel),
// which need no tally.  Their FP64 sums bound them (84 % of the pipe in pass
// 2) while every component of the functional was converted and weighted: a
// functional of one component, 1e6 particles: 4.2 and 7.0 ms, now 3.3 and 4.0.
// 1 forward: accumulates each particle's contribution to a linear functional
//   Phi = sum W[box][bin][q] tally[box][bin][q] (W in the walk's units);
// 2 adjoint: replays every particle from its Philox counter (the same draws
//   as pass 1) and adds likelihood-ratio terms, each weighted by the
//   particle's future contribution R = Phi_total - Phi so far:
//   free flight of mode k, dt = tau_k e:  d log f / d tau_k = (e - 1) / tau_k
//   post-scattering draw of mode k (p_k ~ C_k / tau_k): -1 / tau_k on tau_k,
//     plus p_i / tau_i on every tau_i (summed once on the host from sum R)
//   specularity draw at a void wall:       1 / p (specular) or -1 / (1 - p)
// CHECK: the checked variant (BTE_FLAG_CHECKS): every table, tally and grid
// index is tested before use; a violation stops the particle with E_CHECK.
// The checks draw nothing, so the trajectories are the plain variant's.
// A particle that stops with an error leaves its pending sums: the run fails.
template <bool SMEM_TALLY, int MINB, int ADJ, bool CHECK = false>
__global__ void __launch_bounds__(256, MINB) rta_prod_grid(DevTables T, GridArgs A, double* gtally,
                                                     unsigned long long* counters, int* err,
                                                     unsigned long long* work, AdjArgs adj) {
    extern __shared__ double stally[];
    const int nk3 = 3 * T.nboxes * T.nbins;
    double* tally = gtally;
    if (T.ncopies > 1) tally = gtally += (long long)(blockIdx.x % T.ncopies) * T.group_stride;
    if (SMEM_TALLY) {
        for (int k = threadIdx.x; k < nk3; k += blockDim.x) stally[k] = 0.;
        __syncthreads();
        tally = stally;
    }
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const long long total = T.pend - T.pbegin;
    const FixScale& F = A.fx;
    const int last_bin = T.nbins - 1, last_part = (1 << F.sub) - 1;
    const int row = A.G.ny + 2;  // cells of a column of the padded map
    // a particle's flights fit 32 bits: a larger cap is never met
    const uint32_t cap = T.flight_cap < 0xffffffffll ? uint32_t(T.flight_cap) : 0xffffffffu;
    // specular draw on the integer pipe: u32 < p 2^32 (p >= 1: always)
    const unsigned long long spec_thr =
        T.specularity >= 1.0 ? (1ull << 32)
                             : (T.specularity > 0. ? (unsigned long long)(T.specularity * 4294967296.0) : 0ull);
    const double score_spec = 1.0 / T.specularity, score_diff = -1.0 / (1.0 - T.specularity);
    const uint64_t* binw = bin_ticks(T);
    // the particle: mode, box and its column, line and place in the padded
    // map, material offset, time bin and which of its 2^sub parts
    int mode = 0, box = 0, ci = 0, cj = 0, cell = 0, mo = 0, bin = 0, part = 0;
    uint64_t flip = 0;  // FIX_DOWN for a particle of negative sign
    ModeFix mv = {0, 0, ~0ull, ~0ull};
    uint64_t ax = 0, ay = 0;
    // ticks left in the free flight (96 bits) and to the end of the bin part
    uint64_t dt_lo = 0, rb = 0;
    uint32_t dt_hi = 0;
    uint64_t pt = 0;  // pending: ticks, and displacement times the sign
    int64_t px = 0, py = 0;
    long long pid = -1;
    uint32_t nev = 0, npass = 0;
    double* tgrp = tally;  // the tally of the particle's replica group
    bool active = false, done = lane >= A.lanes;
    // adjoint state: Phi so far (pass 1) or still to come (pass 2), pending score terms
    double phi_run = 0., spec_score = 0.;
    double sum_r = 0., g_p = 0., phi_all = 0.;
    long long slot = 0;
    int pend_kind = 0;
    // the particle stops with an error
    auto stop = [&](int e) {
        record_error(err, e, pid);
        active = false;
        done = true;
    };
    // x plus or minus the functional's part of the pending sums: one conversion
    // and one FMA for each component that has a weight at all (a loop: as three
    // conditions they were predicated, and held the FP64 lanes all the same).
    auto weighted = [&](double x, bool minus) -> double {
        const double* Wk = adj.W + 3ll * (box * T.nbins + bin);
        const long long t = (flip != 0) != minus ? -(long long)pt : (long long)pt;
#pragma unroll 1
        for (int m = adj.comps; m; m &= m - 1) {
            const int q = __ffs(m) - 1;
            const long long d = q == 1 ? px : py;
            x = fma(__ldg(Wk + q), double(q == 0 ? t : minus ? -d : d), x);
        }
        return x;
    };
    // A new free flight of the current mode from one random word:
    // dt = -tau ln u (FP32 log), u = (k + 1/2) 2^-23 from 23 bits, never 0
    // or 1; its velocities stay in registers for the segments that follow.
    // Where a direction turns, the border ahead is the other one.
    auto new_flight = [&](uint32_t word) {
        if (CHECK && (mode < 0 || mode >= T.n || mo < 0)) {
            stop(E_CHECK);
            return;
        }
        const ModeFix m = A.mf[mode];
        const double tau_k = __ldg(T.tau + mo + mode);
        const float ef = -logf((float(word >> 9) + 0.5f) * 0x1p-23f);
        if ((m.vx ^ mv.vx) & FIX_DOWN) ax = __ldg(A.wxf + ci) - ax;
        if ((m.vy ^ mv.vy) & FIX_DOWN) ay = __ldg(A.wyf + cj) - ay;
        mv = m;
        dt_lo = fix_flight(ef, tau_k, F.kt, dt_hi);
        c.events++;
        if (ADJ == 2) {
            // future contribution from here: what the flushes left of Phi_total
            // less the pending part
            const double R = weighted(phi_run, true);
            // the flight's (e - 1) / tau and, for a mode from a
            // post-scattering draw, that draw's -1 / tau (the 1 / tau of all a
            // mode's flights: the reader's)
            const double gk = (widen_pos(ef) - ((pend_kind & 1) ? 2.0 : 1.0)) * R;
            if (pend_kind & 1) sum_r += R;
            if (pend_kind & 2) g_p += spec_score * R;
            pend_kind = 0;
            atomicAdd(adj.g_tau + mode, gk);
        }
        // zero rate or runaway particle
        const long long tau_b = __double_as_longlong(tau_k);  // (its sign without the FP64 lanes)
        if (++nev > cap || tau_b <= 0) stop(tau_b > 0 ? E_LIMIT : E_VALUE);
    };
    for (;;) {
        // refill idle lanes of the warp with new particles; a lane is done when
        // the counter has run out or its particle stopped with an error
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (__popc(idle) >= A.refill || !__any_sync(0xffffffffu, active)) {
            unsigned long long base = 0;
            const int leader = idle ? __ffs(idle) - 1 : 0;
            if (idle && lane == leader) base = atomicAdd(work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                const long long mine = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (mine < total) {
                    pid = T.pbegin + mine;
                    tgrp = T.ngroups > 1 ? tally + (long long)(pid % T.ngroups) * T.group_stride : tally;
                    Philox g;
                    g.init(T.seed, (uint64_t)pid);
                    GridParticle p;
                    int e = grid_generate(T, A.G, A.boxcell, g, pid, p);
                    if (CHECK && !e &&
                        (p.box < 0 || p.box >= T.nboxes || p.i < 0 || p.i >= A.G.nx || p.j < 0 || p.j >= A.G.ny))
                        e = E_CHECK;
                    if (e) {
                        stop(e);
                    } else {
                        active = true;
                        mode = p.mode;
                        box = p.box;
                        mo = p.mo;
                        ci = p.i;
                        cj = p.j;
                        cell = (ci + 1) * row + cj + 1;
                        flip = p.sign < 0 ? FIX_DOWN : 0;
                        nev = npass = 0;
                        if (ADJ) {
                            slot = mine;
                            phi_run = ADJ == 2 ? adj.phi_total[mine] : 0.;
                            pend_kind = 0;
                        }
                        bin = part = 0;
                        rb = __ldg(binw);
                        pt = 0;
                        px = py = 0;
                        // the distances as for a flight towards larger
                        // coordinates; the flight turns them where it goes
                        mv.vx = mv.vy = 0;
                        const long long dx = A.gxf[ci + 1] - fix_round(p.x - F.x0, F.kx);
                        const long long dy = A.gyf[cj + 1] - fix_round(p.y - F.y0, F.kx);
                        const long long wx = A.wxf[ci], wy = A.wyf[cj];
                        ax = dx < 0 ? 0 : dx > wx ? wx : dx;
                        ay = dy < 0 ? 0 : dy > wy ? wy : dy;
                        new_flight(g.next32());  // the first flight, from the generation stream
                    }
                } else {
                    done = true;
                }
            }
            if (__all_sync(0xffffffffu, !active)) {
                // a lane whose first flight already failed leaves others to refill
                if (__all_sync(0xffffffffu, done)) break;
                continue;
            }
        }
        if (active) {
            // this pass's random words (used at its end); computed ahead of
            // the segment, with which it shares no data
            const uint4 rr = pass_block(npass++, (uint64_t)pid, T.seed);
            // the mode a scattering at the end of this segment would draw: its
            // table read runs under the segment's arithmetic (1e4 particles
            // 0.51 -> 0.48 ms, 1e6 3.13 -> 3.06; the 64-register variant
            // reads it in place: 114.5 ms there, 116.6 ahead)
            constexpr bool AHEAD = MINB < 4;
            int cand = mode;
            if (AHEAD && !T.ballistic) {
                const int k = int(mulhi32(rr.y, uint32_t(T.n)));
                const int2 e = __ldg(T.resample + mo + k);
                cand = float(rr.z >> 8) * 0x1p-24f < __int_as_float(e.x) ? k : e.y;
            }
            if (CHECK && (ci < 0 || ci >= A.G.nx || cj < 0 || cj >= A.G.ny || box < 0 || box >= T.nboxes || bin < 0 ||
                          bin > last_bin)) {
                stop(E_CHECK);
                continue;
            }
            const FixSeg q = fix_segment(ax, ay, mv, dt_lo, dt_hi, rb);
            const bool border = q.cross_x || q.cross_y;
            const bool downx = (long long)mv.vx < 0, downy = (long long)mv.vy < 0;
            // what lies across the border
            const int step = q.cross_x ? (downx ? -row : row) : (downy ? -1 : 1);
            int nb = box;
            if (border) nb = __ldg(A.map + cell + step);
            ax -= q.dx;
            ay -= q.dy;
            const int64_t fx = (int64_t)(mv.vx ^ flip) >> 63, fy = (int64_t)(mv.vy ^ flip) >> 63;
            px += ((int64_t)q.dx ^ fx) - fx;
            py += ((int64_t)q.dy ^ fy) - fy;
            pt += q.seg;
            rb -= q.seg;
            dt_hi -= dt_lo < q.seg ? 1u : 0u;
            dt_lo -= q.seg;
            // spectral decomposition: the segment's time per mode at selected boxes
            if (ADJ == 0 && T.spec_loc) {
                const int loc = __ldg(T.spec_loc + box);
                if (loc >= 0) {
                    const double ds = double((long long)q.seg);
                    atomicAdd(T.spec + (long long)(loc * T.nbins + bin) * T.n + mode, flip ? -ds : ds);
                }
            }
            const bool reflect = nb == -1;              // void: reflection, a new flight follows
            const bool leave = border && !reflect;      // into the next cell or a reservoir
            if (CHECK && (box * T.nbins + bin >= T.nboxes * T.nbins || nb >= T.nboxes)) {
                stop(E_CHECK);
                continue;
            }
            if (leave || q.bin_end) {
                if (ADJ) {
                    phi_run = weighted(phi_run, ADJ == 2);
                } else {
                    double* b = tgrp + 3ll * (box * T.nbins + bin);
                    if (pt) atomicAdd(b + 0, double(flip ? -(long long)pt : (long long)pt));
                    if (px) atomicAdd(b + 1, double((long long)px));
                    if (py) atomicAdd(b + 2, double((long long)py));
                }
                if (leave || part == last_part) c.tallies++;
                pt = 0;
                px = py = 0;
                if (leave) {
                    if (nb >= 0) {
                        box = nb;
                        cell += step;
                        if (q.cross_x) {
                            ci += downx ? -1 : 1;
                            ax = __ldg(A.wxf + ci);
                        } else {
                            cj += downy ? -1 : 1;
                            ay = __ldg(A.wyf + cj);
                        }
                        c.crossings++;
                    } else {
                        c.absorbed++;
                        active = false;
                    }
                } else {
                    if (part == last_part) {
                        part = 0;
                        active = ++bin <= last_bin;
                    } else {  // (no pass of the draws)
                        ++part;
                        --npass;
                    }
                    if (active) rb = __ldg(binw + bin);
                }
                if (ADJ == 1 && !active) {
                    adj.phi_total[slot] = phi_run;
                    phi_all += phi_run;
                }
            } else {
                // the next mode: a Lambert row at a void wall (or the mirror
                // mode on a specular draw), the post-scattering table after a
                // scattering (none for ballistic runs)
                float pr = 2.f;  // keep whatever the acceptance word
                int keep = mode, alt = mode;
                if (reflect) {
                    // (selects, not an indexed parameter array, which would live in local memory)
                    const int cls = q.cross_x ? (downx ? A.cls[1] : A.cls[0]) : (downy ? A.cls[3] : A.cls[2]);
                    if (cls < 0 || (CHECK && cls >= T.nclass)) {
                        stop(cls < 0 ? E_GEOM : E_CHECK);
                        continue;
                    }
                    const long long r = (long long)cls * T.n + mode;
                    int mirror_mode = -1;
                    if (spec_thr) {
                        const bool spec = rr.w < spec_thr;
                        if (ADJ == 2) {
                            spec_score = spec ? score_spec : score_diff;
                            pend_kind |= 2;
                        }
                        if (spec && T.mirror) mirror_mode = __ldg(T.mirror + r);
                    }
                    if (mirror_mode >= 0) {
                        c.specular++;
                        keep = mirror_mode;
                    } else {
                        const LambertRow lr = lambert_row(T, r);
                        if (lr.len == 0) {
                            stop(E_GEOM);
                            continue;
                        }
                        const int4 e = __ldg(T.lalias + lr.off + mulhi32(rr.y, lr.len));
                        pr = __int_as_float(e.x);
                        keep = e.y;
                        alt = e.z;
                    }
                    c.wall_hits++;
                } else if (!T.ballistic) {
                    if (AHEAD) {
                        keep = alt = cand;
                    } else {
                        keep = int(mulhi32(rr.y, uint32_t(T.n)));
                        const int2 e = __ldg(T.resample + mo + keep);
                        pr = __int_as_float(e.x);
                        alt = e.y;
                    }
                    if (ADJ == 2) pend_kind |= 1;
                }
                const float acc = float(rr.z >> 8) * 0x1p-24f;
                mode = acc < pr ? keep : alt;
                new_flight(rr.x);
            }
        }
    }
    if (ADJ) {
        for (int o = 16; o > 0; o >>= 1) {
            sum_r += __shfl_down_sync(0xffffffffu, sum_r, o);
            g_p += __shfl_down_sync(0xffffffffu, g_p, o);
            phi_all += __shfl_down_sync(0xffffffffu, phi_all, o);
        }
        if (lane == 0) {
            atomicAdd(adj.g_scalar + 0, g_p);
            atomicAdd(adj.g_scalar + 1, sum_r);
            atomicAdd(adj.g_scalar + 2, phi_all);
        }
    }
    flush_counters_p<8>(c, counters);  // no periodic boxes on the grid path
    if (SMEM_TALLY) {
        __syncthreads();
        for (int k = threadIdx.x; k < nk3; k += blockDim.x) {
            const double v = stally[k];
            if (v != 0.) atomicAdd(gtally + k, v);
        }
    }
}

// The integer tables of a run's scales: every mode's velocity record, the
// grid lines and the widths between them (fixed_walk.cuh).
__global__ void fix_tables(FixScale f, const ModeVel* mv, int n, ModeFix* mf, DevGrid G, long long* gxf,
                           long long* gyf, long long* wxf, long long* wyf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    auto line = [&](const double* g, int k, double o) { return fix_round(g[k] - o, f.kx); };
    if (i < n) {
        ModeFix m;
        fix_velocity(mv[i].vx, f, m.vx, m.rx);
        fix_velocity(mv[i].vy, f, m.vy, m.ry);
        mf[i] = m;
    }
    if (i <= G.nx) gxf[i] = line(G.gx, i, f.x0);
    if (i <= G.ny) gyf[i] = line(G.gy, i, f.y0);
    if (i < G.nx) wxf[i] = line(G.gx, i + 1, f.x0) - line(G.gx, i, f.x0);
    if (i < G.ny) wyf[i] = line(G.gy, i + 1, f.y0) - line(G.gy, i, f.y0);
}

void launch_fix_tables(const FixScale& f, const ModeVel* mv, int n, ModeFix* mf, const DevGrid& G, long long* gxf,
                       long long* gyf, long long* wxf, long long* wyf, cudaStream_t s) {
    const int g = G.nx > G.ny ? G.nx + 1 : G.ny + 1, m = n > g ? n : g;
    fix_tables<<<(m + 255) / 256, 256, 0, s>>>(f, mv, n, mf, G, gxf, gyf, wxf, wyf);
}

// The copies of a tally summed into the first, in ps and nm.
__global__ void gather_tally_k(double* t, long long n, int ncopies, double st, double sx) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double v = t[i];
        for (int k = 1; k < ncopies; ++k) v += t[i + k * n];
        t[i] = v * (i % 3 == 0 ? st : sx);
    }
}
void launch_gather_tally(double* tally, long long n, int ncopies, const FixScale& f, int nsm, cudaStream_t s) {
    long long b = (n + 255) / 256;
    if (b > nsm * 8ll) b = nsm * 8ll;
    gather_tally_k<<<unsigned(b), 256, 0, s>>>(tally, n, ncopies, f.per_tick(), f.per_unit());
}

// ------------------------------------------------------------ polygon path

// Production loop of geometries that are not a grid: the grid kernel's
// organisation (persistent warps refilling idle lanes, one segment per lane
// per pass, time left in the bin, telescoping pending tally, one Philox block
// per pass, one mode-redraw block) with the convex box's border lines in
// place of cell lines.  A segment ends at the flight end, the bin border or
// the first border line the flight leaves through (n.v > 0, exit time
// (c - n.x) / n.v, compared without divisions); across that border the
// piece holding the exit point names the neighbour: a box (the flight goes
// on there), a reservoir (absorbed), a periodic box (translated as
// geometry_2d::translate does, the flight goes on) or none (a void wall:
// Lambert or specular redraw).  The reference's handling of corners and ties
// between borders, which has measure zero, is not repeated here.  A flight
// that runs more than POLY_SEG_CAP segments stops the run with E_LIMIT.
constexpr uint32_t POLY_SEG_CAP = 1u << 20;
__global__ void __launch_bounds__(256) rta_prod_poly(DevTables T, PolyArgs A, double* tally,
                                                      unsigned long long* counters, int* err,
                                                      unsigned long long* work) {
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const long long total = T.pend - T.pbegin;
    const int last_bin = T.nbins - 1;
    const unsigned long long spec_thr =
        T.specularity >= 1.0 ? (1ull << 32)
                             : (T.specularity > 0. ? (unsigned long long)(T.specularity * 4294967296.0) : 0ull);
    Pending pd;
    pd.key = -1;
    pd.flushes = 0;
    pd.r0 = pd.x0 = pd.y0 = 0.;
    ProdPolicy pol;  // generation and translation draws
    pol.g.init(0, 0);
    pol.out = tally;
    pol.ntally = 0;
    Particle p;
    p.pos = v2(0., 0.);
    p.mode = p.box = p.mo = 0;
    p.sign = 1;
    p.t = 0.;
    ModeVel mv = {0., 0., 0., 0.};
    const double* binw = T.timegrid + T.ntime;
    double dt = 0., rb = 0.;
    long long pid = -1, nev = 0;
    uint32_t npass = 0, nseg = 0;
    int bin = 0;
    unsigned long long signbit = 0;
    bool active = false, done = false;
    auto new_flight = [&](uint32_t word) -> bool {
        const int k = p.mode;
        mv = A.mv[k];
        const float ef = -logf((float(word >> 9) + 0.5f) * 0x1p-23f);
        dt = widen_pos(ef) * __ldg(T.tau + p.mo + k);
        c.events++;
        nseg = 0;
        if (ob(dt) <= 0 || ++nev > T.flight_cap) {  // zero rate or runaway particle
            record_error(err, ob(dt) > 0 ? E_LIMIT : E_VALUE, pid);
            active = false;
            done = true;
            pd.flush(tally, signbit, rb, p.pos.x, p.pos.y);
            return false;
        }
        return true;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (idle) {
            unsigned long long base = 0;
            const int leader = __ffs(idle) - 1;
            if (lane == leader) base = atomicAdd(work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                const long long mine = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (mine < total) {
                    pid = T.pbegin + mine;
                    pol.g.init(T.seed, (uint64_t)pid);
                    const int e = generate(T, pol, pid, p);
                    if (e) {
                        record_error(err, e, pid);
                        done = true;
                    } else {
                        active = true;
                        nev = 0;
                        npass = 0;
                        bin = 0;
                        rb = __ldg(binw);
                        signbit = p.sign < 0 ? 0x8000000000000000ull : 0ull;
                        pd.start(p.box * T.nbins, rb, p.pos.x, p.pos.y);
                        new_flight(pol.g.next32());  // the first flight, from the generation stream
                    }
                } else {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (!active) continue;
        const uint4 rr = pass_block(npass++, (uint64_t)pid, T.seed);
        if (++nseg > POLY_SEG_CAP) {  // a flight that keeps meeting borders without advancing
            record_error(err, E_LIMIT, pid);
            active = false;
            done = true;
            continue;
        }
        // the first border line the flight leaves through: smallest
        // num / den over the borders with den = n.v > 0, num = c - n.x >= 0
        const GBox& B = T.boxes[p.box];
        int best = -1;
        double te = HUGE_VAL;
        // an axis-aligned rectangle: the cell-line test of the grid kernel,
        // the line ahead in x and in y (a zero velocity component has
        // 1/v = +inf and never exits), the nearer one first on ties
        PolyRect R;
        R.kx1 = -1;
        if (A.rect) R = A.rect[p.box];
        const bool rectb = R.kx1 >= 0;
        bool xfirst = false;
        double xw = 0., yw = 0.;
        int side_nb = -2, side_fl = 0, side_cls = 0;  // what lies across the exit side
        if (rectb) {
            const bool upx = ob(mv.ivx) >= 0, upy = ob(mv.ivy) >= 0;
            xw = upx ? R.x1 : R.x0;
            yw = upy ? R.y1 : R.y0;
            long long bx = ob((xw - p.pos.x) * mv.ivx), by = ob((yw - p.pos.y) * mv.ivy);
            bx = bx > 0 ? bx : 0;
            by = by > 0 ? by : 0;
            // a strip spanning the period never exits through those sides:
            // its flight wraps (below) instead of translating side by side
            if (R.perx) bx = ob(HUGE_VAL);
            if (R.pery) by = ob(HUGE_VAL);
            xfirst = bx <= by;
            best = xfirst ? (upx ? R.kx1 : R.kx0) : (upy ? R.ky1 : R.ky0);
            side_nb = xfirst ? (upx ? R.nx1 : R.nx0) : (upy ? R.ny1 : R.ny0);
            side_fl = xfirst ? (upx ? R.fx1 : R.fx0) : (upy ? R.fy1 : R.fy0);
            side_cls = xfirst ? (upx ? R.cx1 : R.cx0) : (upy ? R.cy1 : R.cy0);
            te = obd(xfirst ? bx : by);
        } else if (A.inv_den) {
            // 1 / den from the table of the border's normal class: one
            // multiplication per border, compared as integers (both >= 0)
            const double* inv = A.inv_den + p.mode;
            for (int k = 0; k < B.nborders; ++k) {
                const PolyBorder& L = A.pb[B.border_off + k];
                const double iv = __ldg(inv + (long long)L.cls * T.n);
                double num = L.c - (L.nx * p.pos.x + L.ny * p.pos.y);
                num = num > 0. ? num : 0.;
                const double tk = num * iv;
                if (iv > 0. && ob(tk) < ob(te)) {
                    best = k;
                    te = tk;
                }
            }
        } else {
            double bnum = 0., bden = 1.;
            for (int k = 0; k < B.nborders; ++k) {
                const PolyBorder& L = A.pb[B.border_off + k];
                const double den = L.nx * mv.vx + L.ny * mv.vy;
                if (!(den > 0.)) continue;
                double num = L.c - (L.nx * p.pos.x + L.ny * p.pos.y);
                num = num > 0. ? num : 0.;
                if (best < 0 || num * bden < bnum * den) {
                    best = k;
                    bnum = num;
                    bden = den;
                }
            }
            te = best >= 0 ? bnum / bden : HUGE_VAL;
        }
        // time bins that end before the flight end and the exit border are
        // closed here, without a pass each: advance to the bin end, flush
        // the pending tally, open the next bin (two FMAs per bin instead of
        // a new exit-time search).  The last bin is left to the pass below.
        {
            long long lim0 = ob(te) < ob(dt) ? ob(te) : ob(dt);
            while (ob(rb) < lim0 && bin < last_bin) {
                const double adv = ob(rb) > 0 ? rb : 0.;
                const double xb = fma(adv, mv.vx, p.pos.x);
                const double yb = fma(adv, mv.vy, p.pos.y);
                if (T.spec_loc) {
                    const int loc = __ldg(T.spec_loc + p.box);
                    if (loc >= 0)
                        atomicAdd(T.spec + (long long)(loc * T.nbins + bin) * T.n + p.mode, p.sign < 0 ? -adv : adv);
                }
                double* b = tally + 3ll * pd.key;
                atomicAdd(b + 0, __longlong_as_double(__double_as_longlong(pd.r0) ^ signbit));
                atomicAdd(b + 1, __longlong_as_double(__double_as_longlong(xb - pd.x0) ^ signbit));
                atomicAdd(b + 2, __longlong_as_double(__double_as_longlong(yb - pd.y0) ^ signbit));
                pd.flushes++;
                dt -= adv;
                te -= adv;
                p.pos = v2(xb, yb);
                ++bin;
                rb = __ldg(binw + bin);
                pd.start(p.box * T.nbins + bin, rb, xb, yb);
                lim0 = ob(te) < ob(dt) ? ob(te) : ob(dt);
            }
        }
        long long te_b = ob(te);
        long long tb_b = ob(rb);
        tb_b = tb_b > 0 ? tb_b : 0;
        const long long dt_b = ob(dt);
        const long long lim_b = te_b < tb_b ? te_b : tb_b;
        const bool flight_end = !(dt_b > lim_b);
        const long long seg_b = flight_end ? dt_b : lim_b;
        const bool wall = !flight_end && te_b <= tb_b;
        const bool bin_end = tb_b <= seg_b;
        const double seg = obd(seg_b);
        double r1 = rb - seg;
        double nx = fma(seg, mv.vx, p.pos.x);
        double ny = fma(seg, mv.vy, p.pos.y);
        dt -= seg;
        if (bin_end) r1 = 0.;
        if (rectb && (R.perx | R.pery)) {
            // the translations the flight made in a strip spanning the
            // period: back into the box by whole periods, the pending
            // tally's start shifted alike (its displacement is the flight's)
            if (R.perx && (nx >= R.x1 || nx < R.x0)) {
                const double W = R.x1 - R.x0, k = floor((nx - R.x0) / W);
                nx -= k * W;
                pd.x0 -= k * W;
                c.translations += (unsigned)fabs(k);
            }
            if (R.pery && (ny >= R.y1 || ny < R.y0)) {
                const double H = R.y1 - R.y0, k = floor((ny - R.y0) / H);
                ny -= k * H;
                pd.y0 -= k * H;
                c.translations += (unsigned)fabs(k);
            }
        }
        // what lies across the exit border
        int target = -1, cls = 0, dmm_t = -1, tflags = 0;
        if (wall && rectb && side_nb != -2) {
            // a side that is void or one neighbour: no piece lookup
            if (xfirst) nx = xw;
            else ny = yw;
            target = side_nb;
            tflags = side_fl;
            cls = side_cls;
        } else if (wall) {
            const PolyBorder& L = A.pb[B.border_off + best];
            cls = L.cls;
            // onto the border line
            double sx;
            if (rectb) {
                if (xfirst) {
                    nx = xw;
                    sx = (ny - L.py) * L.uy;
                } else {
                    ny = yw;
                    sx = (nx - L.px) * L.ux;
                }
            } else {
                const double off = L.nx * nx + L.ny * ny - L.c;
                nx -= off * L.nx;
                ny -= off * L.ny;
                sx = (nx - L.px) * L.ux + (ny - L.py) * L.uy;
            }
            for (int j = 0; j < L.npieces; ++j) {
                const PolyPiece pc = A.pieces[L.piece_off + j];
                if (sx >= pc.s0 && sx <= pc.s1) {
                    target = pc.box;
                    dmm_t = pc.pad;
                    break;
                }
            }
            if (target >= 0) tflags = (T.boxes[target].reservoir ? 1 : 0) | (T.boxes[target].tto >= 0 ? 2 : 0);
        }
        // a contact between crystals (change_material_diffuse,
        // src/RTA_MC2D.cpp:871-964): the interface's table re-emits the
        // particle on either side (Diffuse_mismatch_distribution::reemit,
        // src/sampling.cpp:831-902: p uniform between the first and the last
        // cumulative value of the incident mode's entries, the first entry
        // not below p); the flight ends there.  Without entries the particle
        // crosses in its mode, as the reference's 'X'.
        const bool iface = wall && target >= 0 && dmm_t >= 0 && A.dmm_row;
        bool dmm_back = false;
        int dmm_mode = -1;
        if (iface) {
            const long long* row = A.dmm_row + (long long)dmm_t * (T.n + 1);
            const long long e0 = __ldg(row + p.mode), e1 = __ldg(row + p.mode + 1);
            if (e1 > e0) {
                const double lo = A.dmm_ent[e0].cum, hi = A.dmm_ent[e1 - 1].cum;
                const double u = double((((unsigned long long)rr.y << 32) | rr.z) >> 11) * 0x1p-53;
                const double pp = u * (hi - lo) + lo;
                long long a = e0, b = e1 - 1;
                while (a < b) {
                    const long long mid = (a + b) >> 1;
                    if (A.dmm_ent[mid].cum >= pp) b = mid;
                    else a = mid + 1;
                }
                const DmmEnt en = A.dmm_ent[a];
                dmm_mode = en.out;
                dmm_back = en.side == 0;
            } else {  // no entries: across with the index kept within the crystal
                c.quirks++;
                dmm_mode = dmm_same_index(T, p.mode, T.box_mat[p.box], T.box_mat[target]);
                if (dmm_mode < 0) {
                    record_error(err, E_VALUE, pid);
                    active = false;
                    done = true;
                    continue;
                }
            }
            c.ifc_hits++;
            if (!dmm_back) c.ifc_trans++;
        }
        if (T.spec_loc) {
            const int loc = __ldg(T.spec_loc + p.box);
            if (loc >= 0) {
                const double ds = rb - r1;
                atomicAdd(T.spec + (long long)(loc * T.nbins + bin) * T.n + p.mode, p.sign < 0 ? -ds : ds);
            }
        }
        const double d0 = pd.r0 - r1, d1 = nx - pd.x0, d2 = ny - pd.y0;
        rb = r1;
        p.pos = v2(nx, ny);
        const bool cross = wall && target >= 0 && !dmm_back;
        const bool absorbed = cross && (tflags & 1);
        const bool periodic = cross && !absorbed && (tflags & 2);
        const bool move = cross && !absorbed;
        const bool reflect = wall && target < 0;
        const bool last = bin_end && bin == last_bin;
        if (move || absorbed || bin_end) {
            double* b = tally + 3ll * pd.key;
            atomicAdd(b + 0, __longlong_as_double(__double_as_longlong(d0) ^ signbit));
            atomicAdd(b + 1, __longlong_as_double(__double_as_longlong(d1) ^ signbit));
            atomicAdd(b + 2, __longlong_as_double(__double_as_longlong(d2) ^ signbit));
            pd.flushes++;
            pd.key = -1;
        }
        if (absorbed || last) {
            if (absorbed) c.absorbed++;
            active = false;
            continue;
        }
        if (bin_end) {
            ++bin;
            rb = __ldg(binw + bin);
        }
        if (move) {
            int nb = target;
            if (periodic) {  // translated into the target of the periodic box
                V2 rf;
                const int e = translate<ProdPolicy, true>(T, pol, target, p.pos, v2(mv.vx, mv.vy), nb, rf);
                if (e) {
                    record_error(err, e, pid);
                    active = false;
                    done = true;
                    continue;
                }
                p.pos = rf;
                c.translations++;
            }
            p.box = nb;
            p.mo = mat_off(T, nb);
            c.crossings++;
        }
        if (move || bin_end) pd.start(p.box * T.nbins + bin, rb, p.pos.x, p.pos.y);
        if (iface) {  // a new flight in the re-emitted mode
            if (dmm_mode >= 0) p.mode = dmm_mode;
            if (!new_flight(rr.x)) continue;
        } else if (reflect || flight_end) {
            const int k = p.mode;
            int nm = k;
            if (reflect || !T.ballistic) {
                float pr = 0.f;
                int keep = k, alt = k;
                if (reflect) {
                    int mirror_mode = -1;
                    if (spec_thr && (unsigned long long)rr.w < spec_thr && T.mirror)
                        mirror_mode = __ldg(T.mirror + (long long)cls * T.n + k);
                    if (mirror_mode >= 0) {
                        c.specular++;
                        pr = 2.f;
                        keep = mirror_mode;
                    } else {
                        const LambertRow lr = lambert_row(T, (long long)cls * T.n + k);
                        if (lr.len == 0) {
                            record_error(err, E_GEOM, pid);
                            active = false;
                            done = true;
                            continue;
                        }
                        const int4 e = __ldg(T.lalias + lr.off + mulhi32(rr.y, lr.len));
                        pr = __int_as_float(e.x);
                        keep = e.y;
                        alt = e.z;
                    }
                    c.wall_hits++;
                } else {
                    const int j = int(mulhi32(rr.y, uint32_t(T.n)));
                    const int2 e = __ldg(T.resample + p.mo + j);
                    pr = __int_as_float(e.x);
                    keep = j;
                    alt = e.y;
                }
                const float acc = float(rr.z >> 8) * 0x1p-24f;
                nm = acc < pr ? keep : alt;
            }
            p.mode = nm;
            if (!new_flight(rr.x)) continue;
        }
    }
    c.tallies = pd.flushes;
    flush_counters_p<13>(c, counters);
}

bool launch_prod_poly(const DevTables& T, const PolyArgs& A, double* tally, unsigned long long* counters,
                      int* err, unsigned long long* work, int nsm, cudaStream_t s) {
    const long long n = T.pend - T.pbegin;
    if (n <= 0) return true;
    int maxb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, rta_prod_poly, 256, 0);
    if (maxb < 1) return false;
    long long blocks = (long long)nsm * maxb;
    const long long need = (n + 255) / 256;
    if (blocks > need) blocks = need;
    rta_prod_poly<<<unsigned(blocks), 256, 0, s>>>(T, A, tally, counters, err, work);
    return true;
}

// One steady-state generation on convex boxes, the polygon kernel's segment
// walk: each slot's one flight runs box to box by exit times against the
// border lines (one box visit per pass, tallied at its end as the reference's
// periodic process_segment does) until it scatters inside a box (phi +=
// sign), reaches a void wall (redrawn and carried over), enters a reservoir
// (absorbed) or a periodic box (translated, the flight goes on).  With
// crystals (PA.dmm_row), a contact between crystals re-emits the particle
// and carries it over as a void wall does.
__global__ void __launch_bounds__(128) rta_steady_poly(DevTables T, SteadyArgs A, PolyArgs PA, double* tally,
                                                       unsigned long long* counters, int* err) {
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    ProdPolicy pol;
    pol.g.init(0, 0);
    pol.out = tally;
    pol.ntally = 0;
    Particle p;
    p.pos = v2(0., 0.);
    p.mode = p.box = p.mo = 0;
    p.sign = 1;
    p.t = 0.;
    V2 v = v2(0., 0.);
    double dt = 0.;
    long long slot = -1;
    uint32_t nseg = 0;
    bool active = false, done = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (idle) {
            unsigned long long base = 0;
            const int leader = __ffs(idle) - 1;
            if (lane == leader) base = atomicAdd(A.work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                slot = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (slot < A.n) {
                    pol.g.init(T.seed, steady_stream(A.gen, slot));
                    const int e = steady_begin(T, A, pol, slot, c, p, v, dt);
                    if (e) {
                        record_error(err, e, slot);
                        A.flag[slot] = 0;
                    } else {
                        active = true;
                        nseg = 0;
                        if (PA.dmm_row) {
                            // carried over across an interface into a
                            // reservoir (absorbed) or a periodic box
                            // (translated), as the next evolparticle call
                            // does (src/RTA_MC2D.cpp:1449-1467)
                            const GBox& B0 = T.boxes[p.box];
                            if (B0.reservoir) {
                                c.absorbed++;
                                steady_emit(A, slot, FATE_ABSORBED, p);
                                active = false;
                            } else if (B0.tto >= 0) {
                                V2 rf;
                                int nb = p.box;
                                const int e2 = translate<ProdPolicy, true>(T, pol, p.box, p.pos, v, nb, rf);
                                if (e2) {
                                    record_error(err, e2, slot);
                                    A.flag[slot] = 0;
                                    active = false;
                                } else {
                                    p.pos = rf;
                                    p.box = nb;
                                    p.mo = mat_off(T, nb);
                                    c.translations++;
                                }
                            }
                        }
                    }
                } else {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (!active) continue;
        if (++nseg > POLY_SEG_CAP) {
            record_error(err, E_LIMIT, slot);
            A.flag[slot] = 0;
            active = false;
            continue;
        }
        const GBox& B = T.boxes[p.box];
        int best = -1;
        double bnum = 0., bden = 1.;
        for (int k = 0; k < B.nborders; ++k) {
            const PolyBorder& L = PA.pb[B.border_off + k];
            const double den = L.nx * v.x + L.ny * v.y;
            if (!(den > 0.)) continue;
            double num = L.c - (L.nx * p.pos.x + L.ny * p.pos.y);
            num = num > 0. ? num : 0.;
            if (best < 0 || num * bden < bnum * den) {
                best = k;
                bnum = num;
                bden = den;
            }
        }
        const double te = best >= 0 ? bnum / bden : HUGE_VAL;
        const bool wall = dt > te;
        const double seg = wall ? te : dt;
        double nx = fma(seg, v.x, p.pos.x);
        double ny = fma(seg, v.y, p.pos.y);
        dt -= seg;
        int target = -1, cls = 0, dmm_t = -1;
        if (wall) {
            const PolyBorder& L = PA.pb[B.border_off + best];
            cls = L.cls;
            const double off = L.nx * nx + L.ny * ny - L.c;
            nx -= off * L.nx;
            ny -= off * L.ny;
            const double sx = (nx - L.px) * L.ux + (ny - L.py) * L.uy;
            for (int j = 0; j < L.npieces; ++j) {
                const PolyPiece pc = PA.pieces[L.piece_off + j];
                if (sx >= pc.s0 && sx <= pc.s1) {
                    target = pc.box;
                    dmm_t = pc.pad;
                    break;
                }
            }
        }
        pol.tally_dt(T, p.box, seg, p.sign, v, p.mode);
        p.pos = v2(nx, ny);
        int fate = -1;
        if (!wall) {  // scattering inside the box
            fate = FATE_SCATTER;
            c.scattered++;
        } else if (target < 0) {  // void wall: the new mode, carried to the next generation
            int nm = -1;
            if (T.specularity > 0. && pol.u() < T.specularity) {
                const int mm = T.mirror ? T.mirror[cls * T.n + p.mode] : -1;
                if (mm >= 0) {
                    nm = mm;
                    c.specular++;
                }
            }
            if (nm < 0) nm = pol.bounce(T, cls, p.mode);
            if (nm < 0) {
                record_error(err, E_GEOM, slot);
                A.flag[slot] = 0;
                active = false;
                continue;
            }
            p.mode = nm;
            c.wall_hits++;
            fate = FATE_BOUNCE;
        } else if (dmm_t >= 0 && PA.dmm_row) {
            // a contact between crystals (change_material_diffuse in the
            // periodic evolparticle, src/RTA_MC2D.cpp:1672-1689, 1751-1779):
            // the interface's table re-emits the particle on either side
            // (Diffuse_mismatch_distribution::reemit, src/sampling.cpp:
            // 831-902) and it joins the next generation; an incident mode
            // without entries crosses in its mode, as the reference's 'X'
            const long long* row = PA.dmm_row + (long long)dmm_t * (T.n + 1);
            const long long e0 = __ldg(row + p.mode), e1 = __ldg(row + p.mode + 1);
            bool across = true;
            if (e1 > e0) {
                const double lo = PA.dmm_ent[e0].cum, hi = PA.dmm_ent[e1 - 1].cum;
                const double pp = pol.u() * (hi - lo) + lo;
                long long a = e0, b = e1 - 1;
                while (a < b) {
                    const long long mid = (a + b) >> 1;
                    if (PA.dmm_ent[mid].cum >= pp) b = mid;
                    else a = mid + 1;
                }
                const DmmEnt en = PA.dmm_ent[a];
                p.mode = en.out;
                across = en.side != 0;
            } else {  // no entries: across with the index kept within the crystal
                c.quirks++;
                const int k = dmm_same_index(T, p.mode, T.box_mat[p.box], T.box_mat[target]);
                if (k < 0) {
                    record_error(err, E_VALUE, slot);
                    A.flag[slot] = 0;
                    active = false;
                    continue;
                }
                p.mode = k;
            }
            c.ifc_hits++;
            if (across) {
                c.ifc_trans++;
                p.box = target;
                p.mo = mat_off(T, target);
            }
            fate = FATE_BOUNCE;
        } else if (T.boxes[target].reservoir) {
            c.absorbed++;
            fate = FATE_ABSORBED;
        } else {
            int nb = target;
            if (T.boxes[target].tto >= 0) {
                V2 rf;
                const int e = translate<ProdPolicy, true>(T, pol, target, p.pos, v, nb, rf);
                if (e) {
                    record_error(err, e, slot);
                    A.flag[slot] = 0;
                    active = false;
                    continue;
                }
                p.pos = rf;
                c.translations++;
            }
            p.box = nb;
            p.mo = mat_off(T, nb);
            c.crossings++;
        }
        if (fate >= 0) {
            steady_emit(A, slot, fate, p);
            active = false;
        }
    }
    c.tallies += pol.ntally;
    flush_counters_p<13>(c, counters);
}

bool launch_steady_poly(const DevTables& T, const SteadyArgs& A, const PolyArgs& PA, double* tally,
                        unsigned long long* counters, int* err, int nsm, cudaStream_t s) {
    if (A.n <= 0) return true;
    int maxb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, rta_steady_poly, 128, 0);
    if (maxb < 1) return false;
    long long blocks = (long long)nsm * maxb;
    const long long need = (A.n + 127) / 128;
    if (blocks > need) blocks = need;
    cudaMemsetAsync(A.work, 0, sizeof(unsigned long long), s);
    rta_steady_poly<<<unsigned(blocks), 128, 0, s>>>(T, A, PA, tally, counters, err);
    return true;
}

bool launch_prod_grid(const DevTables& T, const GridArgs& A0, double* tally,
                      unsigned long long* counters, int* err, unsigned long long* work,
                      const ProdTuning& tune, int nsm, cudaStream_t s, int adj_pass,
                      const AdjArgs* adj) {
    const long long n = T.pend - T.pbegin;
    if (n <= 0) return true;
    GridArgs A = A0;
    A.lanes = 32;
    const size_t smem = size_t(3) * T.nboxes * T.nbins * sizeof(double);
    // the adjoint passes run with the tally in global memory
    const bool use_smem = tune.smem_tally != 0 && smem <= 200 * 1024 && adj_pass == 0 && T.ngroups <= 1;
    // residency variants: 4 blocks of 256 threads per SM (64 registers), 3 (79
    // registers) or 2 (no register cap); the shared-memory tally allows one
    // block per SM.  Four hide the table reads better once every lane carries
    // several particles in turn (2e6 on 36864 modes: 112.6 ms against 115.0
    // with three; 4e6 on 6144 modes 17.2 against 16.9), three leave fewer lanes
    // idle at the end of a short run (1e6: 3.03 ms against 3.17).
    const bool tuned = tune.block_threads > 0 || tune.blocks_per_sm > 0 || use_smem;
    if (!tuned && !T.checks)
        A.lanes = particle_lanes(n, nsm);
    const bool small = A.lanes < 32;
    const int threads = tune.block_threads > 0 ? tune.block_threads : small ? 64 : 256;
    if (threads > 256 || threads % 32) return false;
    const bool long_run = n >= 8ll * 1024 * nsm;
    int bps = tune.blocks_per_sm > 0 ? tune.blocks_per_sm : (use_smem ? 1 : long_run ? 4 : 3);
    const AdjArgs none{};
    const AdjArgs& aa = adj ? *adj : none;
    if (T.checks && adj_pass == 0) {  // the checked variant, at its own residency
        int maxb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, rta_prod_grid<false, 2, 0, true>, 256, 0);
        if (maxb < 1) return false;
        long long blocks = (long long)nsm * (maxb < 2 ? maxb : 2);
        const long long need = (n + 255) / 256;
        if (blocks > need) blocks = need;
        rta_prod_grid<false, 2, 0, true><<<unsigned(blocks), 256, 0, s>>>(T, A, tally, counters, err, work, aa);
        return true;
    }
    const void* fn;
    if (use_smem) {
        fn = reinterpret_cast<const void*>(rta_prod_grid<true, 1, 0>);
        if (cudaFuncSetAttribute(rta_prod_grid<true, 1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(smem)) != cudaSuccess)
            return false;
    } else if (adj_pass == 1) {
        fn = reinterpret_cast<const void*>(rta_prod_grid<false, 3, 1>);
    } else if (adj_pass == 2) {
        fn = reinterpret_cast<const void*>(rta_prod_grid<false, 3, 2>);
    } else if (threads * bps > 768) {  // the register cap follows the resident threads
        fn = reinterpret_cast<const void*>(rta_prod_grid<false, 4, 0>);
    } else if (threads * bps > 512) {
        fn = reinterpret_cast<const void*>(rta_prod_grid<false, 3, 0>);
    } else {
        fn = reinterpret_cast<const void*>(rta_prod_grid<false, 2, 0>);
    }
    int maxb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, fn, threads, use_smem ? smem : 0);
    if (maxb < 1) return false;
    if (bps > maxb) bps = maxb;
    long long blocks = (long long)nsm * (small ? maxb : bps);
    const long long per = threads / 32 * A.lanes, need = (n + per - 1) / per;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    const unsigned nb = unsigned(blocks);
    if (use_smem)
        rta_prod_grid<true, 1, 0><<<nb, threads, smem, s>>>(T, A, tally, counters, err, work, aa);
    else if (adj_pass == 1)
        rta_prod_grid<false, 3, 1><<<nb, threads, 0, s>>>(T, A, tally, counters, err, work, aa);
    else if (adj_pass == 2)
        rta_prod_grid<false, 3, 2><<<nb, threads, 0, s>>>(T, A, tally, counters, err, work, aa);
    else if (fn == reinterpret_cast<const void*>(rta_prod_grid<false, 4, 0>))
        rta_prod_grid<false, 4, 0><<<nb, threads, 0, s>>>(T, A, tally, counters, err, work, aa);
    else if (fn == reinterpret_cast<const void*>(rta_prod_grid<false, 3, 0>))
        rta_prod_grid<false, 3, 0><<<nb, threads, 0, s>>>(T, A, tally, counters, err, work, aa);
    else
        rta_prod_grid<false, 2, 0><<<nb, threads, 0, s>>>(T, A, tally, counters, err, work, aa);
    return true;
}

}  // namespace bte
