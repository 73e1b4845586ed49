// prod_common.cuh - what the production kernels share: error and event
// counters, the draws of a pass, alias sampling and the FP64 policy.
#pragma once

#include "kernels.h"

namespace bte {

__device__ __forceinline__ void record_error(int* err, int e, long long pid) {
    if (atomicCAS(err, 0, e) == 0) {
        err[1] = int(pid & 0x7fffffff);
        err[2] = int(pid >> 31);
    }
}

// Warp-reduced counters: the first NC of (events, wall hits, crossings,
// absorbed, specular, nudges, quirks, tally updates, translations,
// steady-state scatters, steady-state drops, interface hits, interface
// transmissions).
template <int NC = 11>
__device__ __forceinline__ void flush_counters_p(const Counters& c, unsigned long long* out) {
    unsigned long long v[13] = {c.events, c.wall_hits, c.crossings, c.absorbed,
                                c.specular, c.nudges, c.quirks, c.tallies, c.translations,
                                c.scattered, c.lost, c.ifc_hits, c.ifc_trans};
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        unsigned long long x = v[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(out + i, x);
    }
}

// Alias draw over n slots: slot from the high bits of one word, acceptance
// from 24 bits of another.
__device__ __forceinline__ int alias_draw(Philox& g, const float* prob, const int* alt, int n) {
    const int j = int(mulhi32(g.next32(), uint32_t(n)));
    const float a = float(g.next32() >> 8) * 0x1p-24f;
    return a < __ldg(prob + j) ? j : __ldg(alt + j);
}

// The Lambert row of (class, mode) r: its first entry and length, packed as
// 36 and 28 bits in one word.
struct LambertRow {
    uint64_t off;
    uint32_t len;
};
__device__ __forceinline__ LambertRow lambert_row(const DevTables& T, long long r) {
    const uint64_t w = __ldg(T.lrow + r);
    return LambertRow{w & 0xfffffffffull, uint32_t(w >> 36)};
}

struct ProdPolicy {
    Philox g;
    double* out;
    unsigned long long ntally;

    __device__ double u() { return g.uniform(); }
    __device__ int choose(int n) { return uniform_below(g, uint32_t(n)); }
    __device__ double flight(const DevTables& T, int k) {
        return double(-logf(g.uniformf())) * __ldg(T.tau + k);  // k: material offset + mode
    }
    __device__ int resample(const DevTables& T, int mo) {
        const int j = int(mulhi32(g.next32(), uint32_t(T.n)));
        const float a = float(g.next32() >> 8) * 0x1p-24f;
        const int2 e = __ldg(T.resample + mo + j);
        return a < __int_as_float(e.x) ? j : e.y;
    }
    __device__ int gen_mode(const DevTables& T, int gi) {
        const long long o = (long long)gi * T.n;
        const int j = alias_draw(g, T.gen_prob + o, T.gen_alt + o, T.n);
        return j;
    }
    __device__ int bounce(const DevTables& T, int cls, int mode) {
        const LambertRow r = lambert_row(T, (long long)cls * T.n + mode);
        if (r.len == 0) return -1;
        const int4 e = __ldg(T.lalias + r.off + mulhi32(g.next32(), r.len));
        const float acc = float(g.next32() >> 8) * 0x1p-24f;
        return acc < __int_as_float(e.x) ? e.y : e.z;
    }
    __device__ int dist(const double*, const float* prob, const int* alt, int n) {
        return alias_draw(g, prob, alt, n);
    }
    // process_segment (periodic), src/RTA_MC2D.cpp:784-834
    __device__ int tally_dt(const DevTables& T, int box, double d, int sign, V2 v, int mode) {
        const double contr = double(sign) * d;
        double* base = out + 3ll * box;
        atomicAdd(base + 0, contr);
        atomicAdd(base + 1, v.x * contr);
        atomicAdd(base + 2, v.y * contr);
        const int loc = T.spec_loc ? __ldg(T.spec_loc + box) : -1;
        if (loc >= 0) {
            const long long o = (long long)loc * T.n + mode;
            atomicAdd(T.spec + o, contr);
            atomicAdd(T.spec_cnt + o, (unsigned long long)(long long)sign);
        }
        ntally++;
        return 0;
    }
    __device__ int tally(const DevTables& T, int box, double t0, double t1, int sign, V2 v, int mode) {
        const int loc = T.spec_loc ? __ldg(T.spec_loc + box) : -1;
        int sb = int(t0 * T.inv_dt), eb = int(t1 * T.inv_dt);
        const int last = T.nbins - 1;
        sb = sb < 0 ? 0 : (sb > last ? last : sb);
        eb = eb < 0 ? 0 : (eb > last ? last : eb);
        const double* g = T.timegrid;
        for (int i = sb; i <= eb; ++i) {
            const double lo = fmax(g[i] - t0, 0.);
            const double hi = fmin(g[i + 1] - t0, t1 - t0);
            const double contr = double(sign) * fmax(hi - lo, 0.);
            if (contr != 0.) {
                double* base = out + 3ll * ((long long)box * T.nbins + i);
                atomicAdd(base + 0, contr);
                atomicAdd(base + 1, v.x * contr);
                atomicAdd(base + 2, v.y * contr);
                if (loc >= 0) atomicAdd(T.spec + (long long)(loc * T.nbins + i) * T.n + mode, contr);
                ntally++;
            }
        }
        return 0;
    }
};

// Order of non-negative doubles (and +inf, and NaN above +inf) through their
// bit patterns as signed 64-bit integers, on the integer pipe: a negative
// operand keeps the sign bit and stays below every non-negative one.
__device__ __forceinline__ long long ob(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double obd(long long b) { return __longlong_as_double(b); }

// float -> double for a positive normal float, by moving its exponent and
// mantissa fields (integer pipe).
__device__ __forceinline__ double widen_pos(float f) {
    const unsigned fb = __float_as_uint(f);
    const unsigned long long e = ((fb >> 23) & 0xffu) + (1023u - 127u);
    return __longlong_as_double((long long)((e << 52) | ((unsigned long long)(fb & 0x7fffffu) << 29)));
}

// Ticks of the time bins (of each of their 2^sub parts), after the grid's
// points and widths.
__device__ __forceinline__ const uint64_t* bin_ticks(const DevTables& T) {
    return reinterpret_cast<const uint64_t*>(T.timegrid + 2 * T.ntime - 1);
}

// The draws of one loop pass: Philox4x32-10 block (pass, 2^30, particle)
// under the run's seed, a counter range the particle's generation draws
// (counter words from 0) never reach.  Every active lane computes one block
// per pass at the same point of the loop, so the generator runs with the
// whole warp instead of once per call site that finds its queue empty.
// x: the free flight, y and z: the alias draw (slot, acceptance), w: the
// specular test.
__device__ __forceinline__ uint4 pass_block(uint32_t pass, uint64_t pid, uint64_t seed) {
    Philox q;
    q.init(seed, pid);
    q.c0 = pass;
    q.c1 = 0x40000000u;
    q.block();
    return make_uint4(q.b0, q.b1, q.b2, q.b3);
}

}  // namespace bte
