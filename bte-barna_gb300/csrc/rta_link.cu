// rta_link.cu - the integer walk (fixed_walk.cuh) over axis-aligned
// rectangular boxes that do not tile a grid one to one, or have periodic
// boxes or interfaces between crystals: the boxes are cut into the cells of
// the lines through all their edges, and each side of each cell names what
// lies across it (build_link_grid).  The draws, events and tallies are those
// of the convex-polygon kernels (rta_prod.cu), which take every other shape.
#include "prod_common.cuh"
#include "rta_steady.cuh"

namespace bte {
namespace {

constexpr uint32_t LINK_SEG_CAP = 1u << 20;  // borders met by one flight before E_LIMIT (as POLY_SEG_CAP)

// Where a particle is: the cell it is in (column, row) and how far the cell's
// borders ahead of it are, for the directions of `mv`.
struct CellPos {
    int ci, cj;
    uint64_t ax, ay;
};

// The cell of box b that holds (x, y), seen towards larger coordinates.
__device__ __forceinline__ void locate(const LinkArgs& A, int b, V2 p, CellPos& c) {
    const int4 r = __ldg(A.range + b);
    const int64_t x = fix_round(p.x - A.fx.x0, A.fx.kx), y = fix_round(p.y - A.fx.y0, A.fx.kx);
    c.ci = r.x;
    c.cj = r.z;
    while (c.ci + 1 < r.y && x >= __ldg(A.gxf + c.ci + 1)) ++c.ci;
    while (c.cj + 1 < r.w && y >= __ldg(A.gyf + c.cj + 1)) ++c.cj;
    const int64_t wx = __ldg(A.wxf + c.ci), wy = __ldg(A.wyf + c.cj);
    const int64_t dx = __ldg(A.gxf + c.ci + 1) - x, dy = __ldg(A.gyf + c.cj + 1) - y;
    c.ax = dx < 0 ? 0 : dx > wx ? wx : dx;
    c.ay = dy < 0 ? 0 : dy > wy ? wy : dy;
}

// The distances of a particle that takes the directions of `to` after `from`.
__device__ __forceinline__ void turn(const LinkArgs& A, CellPos& c, const ModeFix& from, const ModeFix& to) {
    if ((to.vx ^ from.vx) & FIX_DOWN) c.ax = __ldg(A.wxf + c.ci) - c.ax;
    if ((to.vy ^ from.vy) & FIX_DOWN) c.ay = __ldg(A.wyf + c.cj) - c.ay;
}

// The position in nm.
__device__ __forceinline__ V2 position(const LinkArgs& A, const CellPos& c, const ModeFix& m) {
    const bool dx = m.vx & FIX_DOWN, dy = m.vy & FIX_DOWN;
    const long long x = dx ? (long long)__ldg(A.gxf + c.ci) + (long long)c.ax : (long long)__ldg(A.gxf + c.ci + 1) - (long long)c.ax;
    const long long y = dy ? (long long)__ldg(A.gyf + c.cj) + (long long)c.ay : (long long)__ldg(A.gyf + c.cj + 1) - (long long)c.ay;
    return v2(double(x) * A.fx.per_unit() + A.fx.x0, double(y) * A.fx.per_unit() + A.fx.y0);
}

// geometry_2d::translate out of the periodic box `from` (its candidates fill
// local memory, which the walk itself does without).
__device__ __noinline__ int translate_at_corner(const DevTables& T, Philox& g, int from, V2 p, V2 v, int& nb, V2& rf) {
    ProdPolicy pol;
    pol.g = g;
    pol.out = nullptr;
    pol.ntally = 0;
    const int e = translate<ProdPolicy, true>(T, pol, from, p, v, nb, rf);
    g = pol.g;
    return e;
}

// Takes a particle that stands on the side `s` of its cell across it: into the
// neighbour, or through a periodic box onto the far line.  CORNER: within
// 2e-6 nm of an end of that side the translation asks geometry_2d::translate,
// whose candidates then include the neighbour beyond that end.  Returns 0 or
// an error code.
template <bool CORNER>
__device__ __forceinline__ int enter(const DevTables& T, const LinkArgs& A, Philox& g, const LinkEntry& k, int s,
                                     const ModeFix& m, int mode, CellPos& c, int& box) {
    if (CORNER && (k.flags & LK_TRANSLATE)) {
        const uint64_t along = s < 2 ? c.ay : c.ax, w = s < 2 ? __ldg(A.wyf + c.cj) : __ldg(A.wxf + c.ci);
        if (along < A.margin || w - along < A.margin) {
            V2 rf;
            int nb = box;
            // on the line that is crossed
            CellPos at = c;
            (s < 2 ? at.ax : at.ay) = 0;
            const int e = translate_at_corner(T, g, __ldg(A.pbox + 4 * (c.ci * A.ny + c.cj) + s), position(A, at, m),
                                              v2(T.vxc[mode], T.vyc[mode]), nb, rf);
            if (e) return e;
            box = nb;
            locate(A, nb, rf, c);
            ModeFix up = {0, 0, 0, 0};
            turn(A, c, up, m);
            return 0;
        }
    }
    box = k.box;
    const int ci = k.cell / A.ny;
    c.cj = k.cell - ci * A.ny;
    c.ci = ci;
    if (s < 2) c.ax = __ldg(A.wxf + ci);
    else c.ay = __ldg(A.wyf + c.cj);
    return 0;
}

__device__ __forceinline__ LinkEntry load_link(const LinkArgs& A, const CellPos& c, int s) {
    const int4 e = __ldg(A.side + 4 * (c.ci * A.ny + c.cj) + s);
    return LinkEntry{e.x, e.y, e.z, e.w};
}

// Whole widths w in r, r < 2^62: by a single-precision quotient, which is off
// by one or two at most below 2^22.
__device__ __forceinline__ uint64_t whole_widths(uint64_t r, uint64_t w) {
    if ((r >> 22) >= w) return r / w;
    uint32_t n = uint32_t(__fdividef(__ull2float_rz(r), __ull2float_ru(w)));
    while (n * w > r) --n;
    while ((n + 1) * w <= r) ++n;
    return n;
}

// A contact between crystals (change_material_diffuse,
// src/RTA_MC2D.cpp:871-964): the interface's table re-emits the particle on
// either side (Diffuse_mismatch_distribution::reemit, src/sampling.cpp:
// 831-902: p uniform between the first and the last cumulative value of the
// incident mode's entries, the first entry not below p); without entries it
// crosses with its index kept within the crystal, as the reference's 'X'.
// u: the uniform draw.  Returns 0 or an error code.
template <class U>
__device__ __forceinline__ int reemit(const DevTables& T, const LinkArgs& A, int table, int from, int to, U&& u, int& mode,
                                      bool& across, Counters& c) {
    const long long* row = A.dmm_row + (long long)table * (T.n + 1);
    const long long e0 = __ldg(row + mode), e1 = __ldg(row + mode + 1);
    across = true;
    if (e1 > e0) {
        const double lo = A.dmm_ent[e0].cum, hi = A.dmm_ent[e1 - 1].cum;
        const double pp = u() * (hi - lo) + lo;
        long long a = e0, b = e1 - 1;
        while (a < b) {
            const long long mid = (a + b) >> 1;
            if (A.dmm_ent[mid].cum >= pp) b = mid;
            else a = mid + 1;
        }
        const DmmEnt en = A.dmm_ent[a];
        mode = en.out;
        across = en.side != 0;
    } else {
        c.quirks++;
        const int k = dmm_same_index(T, mode, T.box_mat[from], T.box_mat[to]);
        if (k < 0) return E_VALUE;
        mode = k;
    }
    c.ifc_hits++;
    if (across) c.ifc_trans++;
    return 0;
}

// Generation of particle `pid` (rta_flight.cuh), out of line: its FP64
// geometry would cost the walk 34 registers.
__device__ __noinline__ int link_generate(const DevTables& T, long long pid, Philox& g, Particle& p) {
    ProdPolicy pol;
    pol.g.init(T.seed, (uint64_t)pid);
    pol.out = nullptr;
    pol.ntally = 0;
    const int e = generate(T, pol, pid, p);
    g = pol.g;
    return e;
}

// The transient loop of rta_prod_grid over linked cells.  What differs:
// - a pass of the draws ends with a flight or at a border of a box, as in the
//   polygon kernel, so the Philox counter stands still at a time-bin border
//   and at a line inside a box;
// - a border may lead through a periodic box (enter) or to another crystal
//   (reemit);
// - a box that spans the period (A.per) is not left through those sides: the
//   flight wraps by whole widths, each counted as a translation, and the
//   pending displacement goes on.
// In doubles the polygon kernel took 160 registers (one block of 256 threads
// per SM) and 42 to 124 FP64 operations per event.  GB300: periodic bar
// (2e6 particles, 10 strips, 100 bins) 10.1 -> 1.45 ms, two-crystal ribbon (3e5
// particles) 1.79 -> 0.70 ms, of 2e3 particles 0.17.
template <bool CORNER>
__global__ void __launch_bounds__(256, 2) rta_prod_link(const __grid_constant__ DevTables T,
                                                        const __grid_constant__ LinkArgs A, double* gtally,
                                                        unsigned long long* counters, int* err,
                                                        unsigned long long* work) {
    double* tally = gtally;
    if (T.ncopies > 1) tally += (long long)(blockIdx.x % T.ncopies) * T.group_stride;
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const long long total = T.pend - T.pbegin;
    const FixScale& F = A.fx;
    const int last_bin = T.nbins - 1, last_part = (1 << F.sub) - 1;
    const uint32_t cap = T.flight_cap < 0xffffffffll ? uint32_t(T.flight_cap) : 0xffffffffu;
    const unsigned long long spec_thr =
        T.specularity >= 1.0 ? (1ull << 32)
                             : (T.specularity > 0. ? (unsigned long long)(T.specularity * 4294967296.0) : 0ull);
    const uint64_t* binw = bin_ticks(T);
    Philox g;  // generation and translation draws
    g.init(0, 0);
    int mode = 0, box = 0, mo = 0, bin = 0, part = 0, per = 0;
    uint64_t flip = 0;
    ModeFix mv = {0, 0, ~0ull, ~0ull};
    CellPos cp = {0, 0, 0, 0};
    uint64_t dt_lo = 0, rb = 0, pt = 0;
    uint32_t dt_hi = 0, nev = 0, npass = 0, nseg = 0;
    int64_t px = 0, py = 0;
    long long pid = -1;
    bool active = false, done = lane >= A.lanes;
    auto stop = [&](int e) {
        record_error(err, e, pid);
        active = false;
        done = true;
    };
    auto new_flight = [&](uint32_t word) {
        const ModeFix m = A.mf[mode];
        const float ef = -logf((float(word >> 9) + 0.5f) * 0x1p-23f);
        const double tau_k = __ldg(T.tau + mo + mode);
        turn(A, cp, mv, m);
        mv = m;
        dt_lo = fix_flight(ef, tau_k, F.kt, dt_hi);
        nseg = 0;
        c.events++;
        const long long tau_b = __double_as_longlong(tau_k);  // (its sign without the FP64 lanes)
        if (++nev > cap || tau_b <= 0) stop(tau_b > 0 ? E_LIMIT : E_VALUE);
    };
    for (;;) {
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
                    Particle p;
                    const int e = link_generate(T, pid, g, p);
                    if (e) {
                        stop(e);
                    } else {
                        active = true;
                        mode = p.mode;
                        box = p.box;
                        mo = p.mo;
                        flip = p.sign < 0 ? FIX_DOWN : 0;
                        nev = npass = 0;
                        bin = part = 0;
                        rb = __ldg(binw);
                        pt = 0;
                        px = py = 0;
                        mv.vx = mv.vy = 0;
                        locate(A, box, p.pos, cp);
                        per = __ldg(A.per + box);
                        new_flight(g.next32());  // the first flight, from the generation stream
                    }
                } else {
                    done = true;
                }
            }
            if (__all_sync(0xffffffffu, !active)) {
                if (__all_sync(0xffffffffu, done)) break;
                continue;
            }
        }
        if (active) {
            const uint4 rr = pass_block(npass, (uint64_t)pid, T.seed);
            int cand = mode;  // the mode a scattering would draw, read ahead as in rta_prod_grid
            if (!T.ballistic) {
                const int j = int(mulhi32(rr.y, uint32_t(T.n)));
                const int2 e = __ldg(T.resample + mo + j);
                cand = float(rr.z >> 8) * 0x1p-24f < __int_as_float(e.x) ? j : e.y;
            }
            ModeFix m = mv;
            if (per & 1) m.rx = ~0ull;
            if (per & 2) m.ry = ~0ull;
            const FixSeg q = fix_segment(cp.ax, cp.ay, m, dt_lo, dt_hi, rb);
            const bool border = q.cross_x || q.cross_y;
            const bool downx = (long long)mv.vx < 0, downy = (long long)mv.vy < 0;
            const int s = q.cross_x ? (downx ? 1 : 0) : (downy ? 3 : 2);
            LinkEntry k = {0, box, 0, 0};
            if (border) k = load_link(A, cp, s);
            if ((per & 1) && q.dx >= cp.ax) {  // whole periods inside the box
                const uint64_t W = __ldg(A.wxf + cp.ci), r = q.dx - cp.ax;
                const uint64_t n = whole_widths(r, W);
                cp.ax = W - (r - n * W);
                c.translations += unsigned(n) + 1;
            } else {
                cp.ax -= q.dx;
            }
            if ((per & 2) && q.dy >= cp.ay) {
                const uint64_t W = __ldg(A.wyf + cp.cj), r = q.dy - cp.ay;
                const uint64_t n = whole_widths(r, W);
                cp.ay = W - (r - n * W);
                c.translations += unsigned(n) + 1;
            } else {
                cp.ay -= q.dy;
            }
            const int64_t fx = (int64_t)(mv.vx ^ flip) >> 63, fy = (int64_t)(mv.vy ^ flip) >> 63;
            px += ((int64_t)q.dx ^ fx) - fx;
            py += ((int64_t)q.dy ^ fy) - fy;
            pt += q.seg;
            rb -= q.seg;
            dt_hi -= dt_lo < q.seg ? 1u : 0u;
            dt_lo -= q.seg;
            if (T.spec_loc) {
                const int loc = __ldg(T.spec_loc + box);
                if (loc >= 0) {
                    const double ds = double((long long)q.seg);
                    atomicAdd(T.spec + (long long)(loc * T.nbins + bin) * T.n + mode, flip ? -ds : ds);
                }
            }
            if (border && (k.flags & LK_INNER)) {  // a line inside the box
                enter<false>(T, A, g, k, s, mv, mode, cp, box);
                continue;
            }
            if (!q.bin_end) {
                ++npass;
                if (border && ++nseg > LINK_SEG_CAP) {
                    stop(E_LIMIT);
                    continue;
                }
            }
            const bool reflect = border && (k.flags & LK_VOID);
            bool leave = border && !reflect, iface = false;
            const int incident = mode;
            if (leave && (k.flags >> 8)) {
                iface = true;
                const int e = reemit(T, A, (k.flags >> 8) - 1, box, k.box,
                                     [&] { return double((((unsigned long long)rr.y << 32) | rr.z) >> 11) * 0x1p-53; }, mode,
                                     leave, c);
                if (e) {
                    stop(e);
                    continue;
                }
            }
            if (leave || q.bin_end) {
                double* b = tally + 3ll * (box * T.nbins + bin);
                if (pt) atomicAdd(b + 0, double(flip ? -(long long)pt : (long long)pt));
                if (px) atomicAdd(b + 1, double((long long)px));
                if (py) atomicAdd(b + 2, double((long long)py));
                if (leave || part == last_part) c.tallies++;
                pt = 0;
                px = py = 0;
                if (leave) {
                    if (k.flags & LK_RESERVOIR) {
                        c.absorbed++;
                        active = false;
                    } else {
                        if (k.flags & LK_TRANSLATE) c.translations++;
                        // (with the incident flight's velocity; a re-emitted mode turns below)
                        const int e = enter<CORNER>(T, A, g, k, s, mv, incident, cp, box);
                        if (e) {
                            stop(e);
                            continue;
                        }
                        mo = mat_off(T, box);
                        per = __ldg(A.per + box);
                        c.crossings++;
                    }
                } else {
                    if (part == last_part) {
                        part = 0;
                        active = ++bin <= last_bin;
                    } else {
                        ++part;
                    }
                    if (active) rb = __ldg(binw + bin);
                }
            }
            if (active && iface) {
                new_flight(rr.x);  // in the re-emitted mode
            } else if (reflect || q.flight_end) {
                float pr = 2.f;  // keep whatever the acceptance word
                int keep = mode, alt = mode;
                if (reflect) {
                    const long long r = (long long)k.cls * T.n + mode;
                    int mirror_mode = -1;
                    if (rr.w < spec_thr && T.mirror) mirror_mode = __ldg(T.mirror + r);
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
                } else {
                    keep = alt = cand;
                }
                const float acc = float(rr.z >> 8) * 0x1p-24f;
                mode = acc < pr ? keep : alt;
                new_flight(rr.x);
            }
        }
    }
    flush_counters_p<13>(c, counters);
}

// One steady-state slot's particle and its flight's length in ps (out of line,
// as link_generate).
__device__ __noinline__ int link_begin(const DevTables& T, const SteadyArgs& S, long long slot, Philox& g, Counters& c,
                                       Particle& p, double& dt) {
    ProdPolicy pol;
    pol.g.init(T.seed, steady_stream(S.gen, slot));
    pol.out = nullptr;
    pol.ntally = 0;
    V2 v;
    const int e = steady_begin(T, S, pol, slot, c, p, v, dt);
    g = pol.g;
    return e;
}

// A mode's velocities with time in units of 2^k ticks: as large as a flight of
// `dt` ps needs to fit one piece and the faster component allows, so that a
// slow mode's long flight takes as few pieces as a fast one's.  (The flight
// keeps 2^-59 of its length.)
__device__ __forceinline__ int slow_down(ModeFix& m, double dt, int kt) {
    const uint64_t vx = m.vx & ~FIX_DOWN, vy = m.vy & ~FIX_DOWN, v = vx > vy ? vx : vy;
    int k = v ? __clzll((long long)v) - 1 : 34;  // (without velocity: 96 bits of ticks into few pieces)
    const int need = int((dbits(dt) >> 52) & 0x7ff) - 1023 + kt - 59;
    k = k > 34 ? 34 : k;
    k = k > need ? need : k;
    k = k < 0 ? 0 : k;
    m.vx = (vx << k) | (m.vx & FIX_DOWN);
    m.vy = (vy << k) | (m.vy & FIX_DOWN);
    if (vx) m.rx -= uint64_t(k);  // the exponent in its low bits
    if (vy) m.ry -= uint64_t(k);
    return k;
}

// One steady-state generation over linked cells: the flights, draws and
// outcomes of rta_steady_poly, a box visit tallied when it ends.  A flight is
// walked in pieces below 2^60 of its time units.  Where the particle is in a
// row of cells that a translation closes to a period and the rest of its
// flight crosses that period twice or more before it leaves the row, the whole
// periods are taken at once: every box of the row gets its share of their
// time and displacement.  Flights that run along the periodic direction cross
// hundreds of boxes, one after the other on one lane, and were what a
// generation waited for (3.6e6 crossings of 3.6e5 flights: 30 ms in doubles for a
// ribbon of 2e5 particles, 42 generations, now 1.25).
__global__ void __launch_bounds__(128, 4) rta_steady_link(const __grid_constant__ DevTables T,
                                                          const __grid_constant__ SteadyArgs S,
                                                          const __grid_constant__ LinkArgs A, double* gtally,
                                                          unsigned long long* counters, int* err) {
    double* tally = gtally + (long long)(blockIdx.x % T.ncopies) * T.group_stride;
    Counters c = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const FixScale& F = A.fx;
    constexpr uint64_t PIECE = 1ull << 60;
    Philox g;
    g.init(0, 0);
    Particle p;
    p.mode = p.box = p.mo = 0;
    p.sign = 1;
    uint64_t flip = 0;
    ModeFix mv = {0, 0, ~0ull, ~0ull};
    CellPos cp = {0, 0, 0, 0};
    uint64_t dt_lo = 0, pt = 0;
    uint32_t dt_hi = 0, nseg = 0;
    int64_t px = 0, py = 0;
    double unit = 1.;  // ticks per time unit of the flight
    long long slot = -1;
    bool active = false, done = lane >= A.lanes;
    auto fail = [&](int e) {
        record_error(err, e, slot);
        S.flag[slot] = 0;
        active = false;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active && !done);
        if (__popc(idle) >= A.refill || !__any_sync(0xffffffffu, active)) {
            unsigned long long base = 0;
            const int leader = idle ? __ffs(idle) - 1 : 0;
            if (idle && lane == leader) base = atomicAdd(S.work, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && !done) {
                slot = (long long)base + __popc(idle & ((1u << lane) - 1u));
                if (slot < S.n) {
                    double dt = 0.;
                    Particle np;
                    const int e = link_begin(T, S, slot, g, c, np, dt);
                    p = np;
                    if (e) {
                        fail(e);
                    } else {
                        active = true;
                        nseg = 0;
                        if (A.dmm_row) {
                            // carried over across an interface into a
                            // reservoir (absorbed) or a periodic box
                            // (translated), as the next evolparticle call
                            // does (src/RTA_MC2D.cpp:1449-1467)
                            const GBox& B0 = T.boxes[p.box];
                            if (B0.reservoir) {
                                c.absorbed++;
                                steady_emit(S, slot, FATE_ABSORBED, p);
                                active = false;
                            } else if (B0.tto >= 0) {
                                V2 rf;
                                int nb = p.box;
                                const int e2 = translate_at_corner(T, g, p.box, p.pos,
                                                                   v2(T.vxc[p.mode], T.vyc[p.mode]), nb, rf);
                                if (e2) {
                                    fail(e2);
                                } else {
                                    p.pos = rf;
                                    p.box = nb;
                                    p.mo = mat_off(T, nb);
                                    c.translations++;
                                }
                            }
                        }
                        if (active) {
                            flip = p.sign < 0 ? FIX_DOWN : 0;
                            pt = 0;
                            px = py = 0;
                            locate(A, p.box, p.pos, cp);
                            mv.vx = mv.vy = 0;
                            ModeFix m = A.mf[p.mode];
                            const int k = slow_down(m, dt, F.kt);
                            turn(A, cp, mv, m);
                            mv = m;
                            unit = bitsd(uint64_t(1023 + k) << 52);
                            dt_lo = fix_ticks(dt, F.kt - k, dt_hi);
                        }
                    }
                } else {
                    done = true;
                }
            }
            if (__all_sync(0xffffffffu, !active)) {
                if (__all_sync(0xffffffffu, done)) break;
                continue;
            }
        }
        if (!active) continue;
        if (++nseg > LINK_SEG_CAP) {
            fail(E_LIMIT);
            continue;
        }
        const FixSeg q = fix_segment(cp.ax, cp.ay, mv, dt_lo, dt_hi, PIECE);
        const bool border = q.cross_x || q.cross_y;
        const bool downx = (long long)mv.vx < 0, downy = (long long)mv.vy < 0;
        const int64_t fx = (int64_t)(mv.vx ^ flip) >> 63, fy = (int64_t)(mv.vy ^ flip) >> 63;
        if (border && !T.spec_loc) {  // whole periods at once
            const int4 cy = __ldg(A.cycle + cp.ci * A.ny + cp.cj);
            const int first = q.cross_x ? cy.x : cy.z, last = q.cross_x ? cy.y : cy.w;
            if (first >= 0) {
                const long long* line = q.cross_x ? A.gxf : A.gyf;
                const uint64_t P = uint64_t(line[last + 1] - line[first]);
                const uint64_t along = (q.cross_x ? mv.vx : mv.vy) & ~FIX_DOWN, ra = q.cross_x ? mv.rx : mv.ry;
                const uint64_t across = (q.cross_x ? mv.vy : mv.vx) & ~FIX_DOWN, rb = q.cross_x ? mv.ry : mv.rx;
                uint64_t& beside = q.cross_x ? cp.ay : cp.ax;
                uint64_t n = 0, o = 0;  // periods, and how far sideways
                double time = 0.;
                for (;;) {
                    const uint64_t out = fix_exit(beside, rb);
                    uint64_t lim = dt_hi || dt_lo > PIECE ? PIECE : dt_lo;
                    lim = out < lim ? out : lim;
                    const uint64_t D = mulhi_low2(lim, along);
                    if (D < 2 * P) break;
                    const uint64_t w = whole_widths(D, P) - 1, t = fix_exit(w * P, ra);
                    uint64_t d = mulhi_low2(t, across);
                    d = d < beside ? d : beside;
                    beside -= d;
                    o += d;
                    dt_hi -= dt_lo < t ? 1u : 0u;
                    dt_lo -= t;
                    time += double((long long)t);
                    n += w;
                }
                if (n) {
                    const double perP = 1.0 / double((long long)P);
                    const double dt_s = (flip ? -unit : unit) * time;
                    const double o_s = ((q.cross_x ? fy : fx) ? -1. : 1.) * double((long long)o);
                    const double a_s = ((q.cross_x ? fx : fy) ? -1. : 1.) * double((long long)n);
                    for (int k = first; k <= last; ++k) {
                        const int cell = q.cross_x ? k * A.ny + cp.cj : cp.ci * A.ny + k;
                        const double w = double(line[k + 1] - line[k]), f = w * perP;
                        double* b = tally + 3ll * __ldg(A.cellbox + cell);
                        atomicAdd(b, dt_s * f);
                        atomicAdd(b + (q.cross_x ? 1 : 2), a_s * w);
                        atomicAdd(b + (q.cross_x ? 2 : 1), o_s * f);
                        if (!(__ldg(&A.side[4 * cell + (q.cross_x ? 0 : 2)].z) & LK_INNER)) c.crossings += unsigned(n);
                    }
                    c.translations += unsigned(n);
                    continue;
                }
            }
        }
        const int s = q.cross_x ? (downx ? 1 : 0) : (downy ? 3 : 2);
        LinkEntry k = {0, 0, 0, 0};
        if (border) k = load_link(A, cp, s);
        cp.ax -= q.dx;
        cp.ay -= q.dy;
        px += ((int64_t)q.dx ^ fx) - fx;
        py += ((int64_t)q.dy ^ fy) - fy;
        pt += q.seg;
        dt_hi -= dt_lo < q.seg ? 1u : 0u;
        dt_lo -= q.seg;
        if (border && (k.flags & LK_INNER)) {
            int b = p.box;
            enter<false>(T, A, g, k, s, mv, p.mode, cp, b);
            continue;
        }
        {  // the box visit ends, or a piece of the flight (the sums hold a few)
            double* b = tally + 3ll * p.box;
            const double t = double((long long)pt) * unit, ts = flip ? -t : t;
            if (pt) atomicAdd(b + 0, ts);
            if (px) atomicAdd(b + 1, double((long long)px));
            if (py) atomicAdd(b + 2, double((long long)py));
            const int loc = T.spec_loc ? __ldg(T.spec_loc + p.box) : -1;
            if (loc >= 0) {
                const long long o = (long long)loc * T.n + p.mode;
                atomicAdd(T.spec + o, ts * F.per_tick());
                if (!q.bin_end) atomicAdd(T.spec_cnt + o, (unsigned long long)(long long)p.sign);
            }
            pt = 0;
            px = py = 0;
        }
        if (q.bin_end) continue;
        int fate = -1;
        if (q.flight_end) {  // scattering inside the box
            fate = FATE_SCATTER;
            c.scattered++;
        } else if (k.flags & LK_VOID) {  // void wall: the new mode, carried to the next generation
            ProdPolicy pol;
            pol.g = g;
            int nm = -1;
            if (T.specularity > 0. && pol.u() < T.specularity) {
                const int mm = T.mirror ? T.mirror[k.cls * T.n + p.mode] : -1;
                if (mm >= 0) {
                    nm = mm;
                    c.specular++;
                }
            }
            if (nm < 0) nm = pol.bounce(T, k.cls, p.mode);
            if (nm < 0) {
                fail(E_GEOM);
                continue;
            }
            p.pos = position(A, cp, mv);
            p.mode = nm;
            c.wall_hits++;
            fate = FATE_BOUNCE;
        } else if (k.flags >> 8) {
            // a contact between crystals: re-emitted, and on to the next
            // generation as at a void wall
            const int target = (k.flags & LK_TRANSLATE) ? __ldg(A.pbox + 4 * (cp.ci * A.ny + cp.cj) + s) : k.box;
            ProdPolicy pol;
            pol.g = g;
            bool across = true;
            p.pos = position(A, cp, mv);
            const int e = reemit(T, A, (k.flags >> 8) - 1, p.box, target, [&] { return pol.u(); }, p.mode, across, c);
            if (e) {
                fail(e);
                continue;
            }
            if (across) {
                p.box = target;
                p.mo = mat_off(T, target);
            }
            fate = FATE_BOUNCE;
        } else if (k.flags & LK_RESERVOIR) {
            c.absorbed++;
            fate = FATE_ABSORBED;
        } else {
            if (k.flags & LK_TRANSLATE) c.translations++;
            const int e = enter<true>(T, A, g, k, s, mv, p.mode, cp, p.box);
            if (e) {
                fail(e);
                continue;
            }
            p.mo = mat_off(T, p.box);
            c.crossings++;
        }
        if (fate >= 0) {
            steady_emit(S, slot, fate, p);
            active = false;
        }
    }
    flush_counters_p<13>(c, counters);
}

}  // namespace

bool launch_steady_link(const DevTables& T, const SteadyArgs& S, const LinkArgs& A0, double* tally,
                        unsigned long long* counters, int* err, int nsm, cudaStream_t s) {
    if (S.n <= 0) return true;
    LinkArgs A = A0;
    A.lanes = particle_lanes(S.n, nsm);
    const int threads = A.lanes < 32 ? 64 : 128;
    int maxb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, rta_steady_link, threads, 0);
    if (maxb < 1) return false;
    long long blocks = (long long)nsm * maxb;
    const long long per = threads / 32 * A.lanes, need = (S.n + per - 1) / per;
    if (blocks > need) blocks = need;
    cudaMemsetAsync(S.work, 0, sizeof(unsigned long long), s);
    rta_steady_link<<<unsigned(blocks), unsigned(threads), 0, s>>>(T, S, A, tally, counters, err);
    return true;
}

bool launch_prod_link(const DevTables& T, const LinkArgs& A0, double* tally, unsigned long long* counters, int* err,
                      unsigned long long* work, int nsm, cudaStream_t s) {
    const long long n = T.pend - T.pbegin;
    if (n <= 0) return true;
    LinkArgs A = A0;
    A.lanes = particle_lanes(n, nsm);
    int maxb = 0;
    // two blocks of 256 threads per SM: with three (80 registers, spills) the
    // bar takes 1.96 ms instead of 1.85, the crystals 0.82 instead of 0.77
    const void* f = A.pbox ? (const void*)rta_prod_link<true> : (const void*)rta_prod_link<false>;
    const int threads = A.lanes < 32 ? 64 : 256;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&maxb, f, threads, 0);
    if (maxb < 1) return false;
    long long blocks = (long long)nsm * maxb;
    const long long per = threads / 32 * A.lanes, need = (n + per - 1) / per;
    if (blocks > need) blocks = need;
    void* args[] = {(void*)&T, (void*)&A, &tally, &counters, &err, &work};
    return cudaLaunchKernel(f, dim3(unsigned(blocks)), dim3(unsigned(threads)), args, 0, s) == cudaSuccess;
}

}  // namespace bte
