// fixed_walk.cuh - positions and times of the grid walk as 64-bit integers.
//
// GB300 has two FP64 lanes per SM: a double-precision warp instruction (an
// addition, an FMA or any conversion from or to double) holds them for 17
// cycles however many of its lanes are active, where a 32-bit integer
// instruction takes 0.6 (measured).  The walk of a particle over an
// axis-aligned grid needs only differences, comparisons and products with a
// velocity or its reciprocal, so it runs on the integer units:
//
//   position  (x - x0) 2^kx   with the domain below 2^62 (2^55 at least)
//   time      t 2^kt          with a time bin below 2^61
//
// A step of the last place is 2^-60 of a time bin, and of the domain's longer
// side 2^-61 where a bin is short against a flight across it, 2^-55 where it is
// eight such flights.  Sums and differences are exact here.  What is not, beside
// doubles (2^-53 of the coordinate, rounded to nearest at every segment):
// - a product loses up to two units, always towards zero;
// - near the domain's origin, and along a side much shorter than the other, a
//   double resolves finer than its ulp at the domain's end, the unit does not;
// - a velocity component keeps 63 bits of the fastest mode's, so one below
//   about 2^-9 of it has fewer than 53 of its own, and one below two units per
//   2^64 ticks is zero: over a bin that is less than the unit either way.
// Scales are powers of two, so a tally leaves as the double nearest to its
// integer sum times 2^-kx or 2^-kt.
//
// tests/test_fixed_walk_cpu.py bounds every segment against exact rational
// arithmetic; tests/test_fixed_walk_doubles_cpu.py compares what whole particles
// leave in their (cell, bin) entries with the same walk in doubles.  Root mean
// square errors there, integers and doubles: ribbon 1000 x 100 nm, bins of 10 ps
// 6e-16 and 6e-14 of the bin, 5e-18 and 1e-16 of the length, 3e-17 and 5e-15 of
// the width; 1500 x 20 nm, 20 ps 7e-16 and 2e-15, 2e-17 and 5e-17, 4e-17 and
// 2e-16.  (With a domain below 2^58 the latter's integers had 1e-14, 3e-16 and
// 7e-16.)  Where a bin is longer than a flight across a domain thirty times as
// long as wide, the integers' errors come out up to twice the doubles'.
#pragma once

#include "bte_device.cuh"

namespace bte {

// The scales of one run (choose_scale).  A time bin longer than 2^3 flights
// of the fastest mode across the domain is walked in 2^sub equal parts, so
// that a displacement always fits.
struct FixScale {
    double x0, y0;   // origin of the positions
    int kx, kt;      // units per nm: 2^kx; ticks per ps: 2^kt
    int sub;
    int pad;
    BTE_HD double per_unit() const { return bitsd(uint64_t(1023 - kx) << 52); }  // nm
    BTE_HD double per_tick() const { return bitsd(uint64_t(1023 - kt) << 52); }  // ps
};

// One mode: per component the speed in position units per 2^64 ticks, with
// the direction (1: towards smaller coordinates) in the top bit, and the
// reciprocal that turns a distance into ticks: with a = floor(log2 speed),
// floor((2^(64+a) - 1) / speed) down to 58 bits and 64 - a in the low six.
struct __align__(32) ModeFix {
    unsigned long long vx, vy, rx, ry;
};
constexpr uint64_t FIX_DOWN = 0x8000000000000000ULL;

BTE_HD uint32_t lo32(uint64_t x) { return uint32_t(x); }
BTE_HD uint32_t hi32(uint64_t x) { return uint32_t(x >> 32); }

// floor(a b / 2^64), or up to two less: the product of the low halves and the
// carry of the middle ones are left out.
BTE_HD uint64_t mulhi_low2(uint64_t a, uint64_t b) {
    return uint64_t(hi32(a)) * hi32(b) + mulhi32(hi32(a), lo32(b)) + mulhi32(lo32(a), hi32(b));
}

// Upper 32 bits of (hi : lo) << s, s in [0, 31].
BTE_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return uint32_t((((uint64_t(hi) << 32) | lo) << s) >> 32);
#endif
}

BTE_HD int log2_floor(uint64_t x) {  // x != 0
#if defined(__CUDA_ARCH__)
    return 63 - __clzll((long long)x);
#else
    return 63 - __builtin_clzll(x);
#endif
}

constexpr uint64_t FIX_NEVER = 0x7fffffffffffffffULL;

// Ticks a flight needs for `dist` units at the speed whose reciprocal is `r`
// (FIX_NEVER and above: not within any time bin).  dist = 0 counts as 1, so
// that a speed of zero (r = ~0) never arrives.
BTE_HD uint64_t fix_exit(uint64_t dist, uint64_t r) {
    const uint32_t sh = lo32(r) & 63u, s = sh & 31u;
    uint32_t h = hi32(dist), l = lo32(dist) | 1u, over = 0;
    if (sh & 32u) {
        over = h;
        h = l;
        l = 0;
    }
    over |= shl_hi(h, 0u, s);  // bits pushed out: at least 2^63 ticks
    const uint64_t d = (uint64_t(shl_hi(l, h, s)) << 32) | (l << s);
    const uint64_t t = mulhi_low2(d, r);
    return over ? FIX_NEVER : t;
}

// The segment of one pass.  A flight of dt ticks (dt_hi 2^64 + dt_lo) with the
// cell's border ahead of it (in its direction) ax and ay units away ends at
// the first of the flight's end, the border in x or y, and the end of the
// time bin, rb ticks away; (dx, dy) is how far it goes.
struct FixSeg {
    uint64_t seg, dx, dy;
    bool flight_end, cross_x, cross_y, bin_end;  // exactly one
};
BTE_HD FixSeg fix_segment(uint64_t ax, uint64_t ay, const ModeFix& m, uint64_t dt_lo, uint32_t dt_hi, uint64_t rb) {
    FixSeg q;
    const uint64_t tx = fix_exit(ax, m.rx), ty = fix_exit(ay, m.ry);
    const bool xfirst = tx <= ty;
    const uint64_t te = xfirst ? tx : ty;
    const bool border = te <= rb;
    const uint64_t lim = border ? te : rb;
    q.flight_end = dt_hi == 0 && dt_lo <= lim;
    q.seg = q.flight_end ? dt_lo : lim;
    q.bin_end = !q.flight_end && !border;
    q.cross_x = !q.flight_end && border && xfirst;
    q.cross_y = !q.flight_end && border && !xfirst;
    q.dx = mulhi_low2(q.seg, m.vx & ~FIX_DOWN);
    q.dy = mulhi_low2(q.seg, m.vy & ~FIX_DOWN);
    if (q.cross_x) q.dx = ax;
    if (q.cross_y) q.dy = ay;
    return q;
}

// tau * e ticks of a flight, e a positive normal float and tau a double > 0:
// the exact 77-bit product of the mantissas, truncated to a tick, as 96 bits
// (a flight beyond 2^95 ticks never ends).  Returns the low 64 bits.
BTE_HD uint64_t fix_flight(float e, double tau, int kt, uint32_t& hi) {
#if defined(__CUDA_ARCH__)
    const uint32_t eb = __float_as_uint(e);
#else
    uint32_t eb;
    __builtin_memcpy(&eb, &e, 4);
#endif
    const uint64_t tb = dbits(tau);
    const uint32_t me = (eb & 0x7fffffu) | 0x800000u;
    const uint32_t mh = (hi32(tb) & 0xfffffu) | 0x100000u;
    // product (2^75 .. 2^77), its top 64 bits: p 2^-13
    const uint64_t pl = uint64_t(me) * lo32(tb), ph = uint64_t(me) * mh;
    const uint64_t p = (ph << 19) + (pl >> 13);
    // dt = p 2^(13 + (Ee - 150) + (Et - 1075) + kt)
    const int x = int((eb >> 23) & 0xffu) + int((hi32(tb) >> 20) & 0x7ffu) + kt - 1212;
    if (x <= 0) {
        hi = 0;
        return x > -64 ? p >> (-x) : 0;
    }
    hi = x < 32 ? uint32_t(p >> (64 - x)) : 0xffffffffu;
    return x < 32 ? p << x : 0;
}

// t ps (a positive double) in ticks, truncated, as 96 bits; beyond them it
// never ends.  Returns the low 64.
BTE_HD uint64_t fix_ticks(double t, int kt, uint32_t& hi) {
    const uint64_t b = dbits(t), m = (b & 0xfffffffffffffULL) | 0x10000000000000ULL;
    const int x = int((b >> 52) & 0x7ff) - 1075 + kt;
    if (x <= 0) {
        hi = 0;
        return x > -64 ? m >> (-x) : 0;
    }
    hi = x < 12 ? 0 : x < 44 ? uint32_t(m >> (64 - x)) : 0xffffffffu;
    return x < 64 ? m << x : 0;
}

// v 2^k to the nearest integer.
BTE_HD int64_t fix_round(double v, int k) {
    const double s = bitsd(uint64_t(1023 + k) << 52);
#if defined(__CUDA_ARCH__)
    return __double2ll_rn(v * s);
#else
    return __builtin_llrint(v * s);
#endif
}

// Velocity v (nm/ps) and its reciprocal in the scales of a run.  A speed
// below two units per 2^64 ticks (a quarter of a unit in a time bin) counts
// as zero.  The reciprocal is never above the exact one, so a border
// is never overrun.
BTE_HD void fix_velocity(double v, const FixScale& f, unsigned long long& fv, unsigned long long& fr) {
    // 2^(64 + kx - kt) may leave the range of one factor: two exact ones
    const int64_t q = fix_round(v * bitsd(uint64_t(1023 + f.kx) << 52), 64 - f.kt);
    const uint64_t a = uint64_t(q < 0 ? -q : q);
    if (a < 2) {
        fv = 0;
        fr = ~0ull;
        return;
    }
    const int n = log2_floor(a);
    const unsigned __int128 num = (((unsigned __int128)1) << (64 + n)) - 1;
    fv = a | (q < 0 ? FIX_DOWN : 0);
    fr = (((unsigned long long)(num / a) - 63ull) & ~63ull) | (unsigned long long)(64 - n);
}

}  // namespace bte
