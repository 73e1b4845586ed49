// spectral.cu - the spectral outputs of the last run (bte_get_spectral):
// the per-mode time tally at the selected boxes, contracted on the device
// with every mode's Gamma pdf over the omega ticks (src/RTA_MC2D.cpp:719-766),
// scaled and integrated in time (:2350-2420; steady :2729-2830).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ctx.hpp"

namespace bte {
namespace {

constexpr int SPEC_K = 128;      // modes of one block of the contraction
constexpr int SPEC_T = 128;      // its ticks, one per thread
constexpr std::size_t PDF_BYTES = std::size_t(64) << 20;

// Gamma pdf of mode k0 + k (shape w^2 / sigma, scale sigma / w: gamma_pdf,
// :61-63) at every tick; 0 where it is negligible or sigma is 0 (a NaN).
// par: per mode {shape, scale, lgamma(shape), log(scale)}.
// FP64 logarithms and exponentials bound it: 32 us for 1536 modes at 200 ticks,
// once for all the locations of a crystal.
__global__ void spec_pdf(const double4* par, const double* om, int k0, int nk, const double* ticks, int nw,
                         double* pdf) {
    const long long total = (long long)nk * nw;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < total;
         j += (long long)gridDim.x * blockDim.x) {
        const int k = int(j / nw), i = int(j - (long long)k * nw);
        const double4 p = par[k0 + k];
        double g = 0.;
        if (om[k0 + k] > 0.) {
            const double x = ticks[i] / p.y;
            const double lp = (p.x - 1.0) * log(x) - x - p.z - p.w;
            if (lp > -700.) g = exp(lp);
        }
        pdf[j] = g;
    }
}

// out[q][bin][tick] += sum over modes of {1, vx, vy}[q] time[bin][mode]
// pdf[mode][tick], for the modes [k0, k0 + nk).  A block takes one bin, 128
// ticks and 128 modes, whose weighted times it first puts in shared memory;
// blocks over the modes add with FP64 atomics.  Bound by three FMAs per term on
// the two FP64 lanes of an SM, so a warp passes over the modes whose pdf is
// zero at all its 32 ticks (more than half of them): 133 us per location of 40
// bins, 1536 modes and 200 ticks, now 55.  (The host loops took 42 ms for three.)
__global__ void __launch_bounds__(SPEC_T) spec_contract(const double* time, double unit, long long tstride, int nbins,
                                                         const double* vx, const double* vy, int k0, int nk,
                                                         const double* pdf, int nw, double* out) {
    __shared__ double w[3][SPEC_K];
    const int b = blockIdx.y, i = blockIdx.x * SPEC_T + threadIdx.x;
    const int c0 = blockIdx.z * SPEC_K, n = min(SPEC_K, nk - c0);
    if (int(threadIdx.x) < n) {
        const int k = k0 + c0 + threadIdx.x;
        const double t = time[(long long)b * tstride + k] * unit;
        w[0][threadIdx.x] = t;
        w[1][threadIdx.x] = vx[k] * t;
        w[2][threadIdx.x] = vy[k] * t;
    }
    __syncthreads();
    double s[3] = {0., 0., 0.};
    const double* col = pdf + (long long)c0 * nw + i;
    for (int k4 = 0; k4 < n; k4 += 4) {
        double g[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) g[j] = i < nw && k4 + j < n ? col[(long long)(k4 + j) * nw] : 0.;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!__any_sync(0xffffffffu, __double2hiint(g[j]) | __double2loint(g[j]))) continue;
            const double t = w[0][k4 + j];
            if (t == 0.) continue;  // (the same for the whole block)
            s[0] += t * g[j];
            s[1] += w[1][k4 + j] * g[j];
            s[2] += w[2][k4 + j] * g[j];
        }
    }
    if (i >= nw) return;
    for (int q = 0; q < 3; ++q)
        if (s[q] != 0.) atomicAdd(out + ((long long)q * nbins + b) * nw + i, s[q]);
}

// fd_qmesh: per bin and q point the sum over branches of time / omega
// (transient, :757) or of signed segments / omega (steady, :829).
__global__ void spec_fdq(const double* time, double unit, const long long* counts, long long tstride, int nbins,
                         const double* om, int nq, int nb, double* out) {
    const long long total = (long long)nbins * nq;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < total;
         j += (long long)gridDim.x * blockDim.x) {
        const int b = int(j / nq), q = int(j - (long long)b * nq);
        double s = 0.;
        for (int a = 0; a < nb; ++a) {
            const int k = q * nb + a;
            const double f = counts ? double(counts[k]) : time[(long long)b * tstride + k] * unit;
            if (f != 0. && om[k] > 0.) s += f / om[k];
        }
        out[j] = s;
    }
}

// The four arrays of a location: v[bin][i] times `scale`, summed over the bins
// so far (integrate), divided by `div`; one thread per i, eight bins read ahead,
// a warp per block so that the divisions spread over the SMs (as four launches of
// 128 threads a block 80 us per location, now 20).
struct SpecFinish {
    double scale[4], div[4];
    int n[4];
};
__global__ void __launch_bounds__(32) spec_finish(double* v, int nbins, int nw, SpecFinish f, int integrate) {
    const int q = blockIdx.y, n = f.n[q], i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double scale = f.scale[q], div = f.div[q];
    v += (long long)q * nbins * nw;
    double run = 0.;
    for (int b0 = 0; b0 < nbins; b0 += 8) {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = b0 + j < nbins ? v[(long long)(b0 + j) * n + i] * scale : 0.;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            run = integrate ? run + x[j] : x[j];
            if (b0 + j < nbins) v[(long long)(b0 + j) * n + i] = div == 1.0 ? run : run / div;
        }
    }
}

}  // namespace

// Device buffers and the host values they were filled from, kept with the
// context (sized for its largest location set so far).
struct SpectralState {
    DBuf par, om, vx, vy, ticks, pdf, out;
    Pinned host;
    std::vector<double> hpar;
    int crystal = -2;           // whose parameters are on the device,
    long long version = -1;     // of which tables
};

void destroy_spectral(bte_ctx* c) {
    delete c->spectral;
    c->spectral = nullptr;
}

}  // namespace bte

using bte::Error;

extern "C" bte_status bte_get_spectral(bte_ctx* c, bte_spectral_result* out) {
    using namespace bte;
    if (!c || !out) return BTE_ERR_INPUT;
    try {
        if (!c->spec_valid) throw Error(BTE_ERR_STATE, "no run with spectral locations yet");
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        const HostGeometry& g = c->geom;
        const std::size_t n = c->modes.n();  // global modes (the crystals' one after the other)
        const std::size_t nloc = c->spec_boxes.size(), nbins = std::size_t(c->spec_nbins);
        const std::size_t nw = std::size_t(c->spec_nomega);
        // each location's crystal (the reference takes the location's
        // material's grid, :1987-2048): its modes and their first global index
        auto crystal_of = [&](std::size_t l) -> int {
            return c->ncrys > 0 ? g.mat[std::size_t(c->spec_boxes[l])] : -1;
        };
        auto modes_of = [&](int k) -> const HostModes& { return k >= 0 ? c->crys[std::size_t(k)] : c->modes; };
        const HostModes& m0 = modes_of(nloc > 0 ? crystal_of(0) : -1);
        const std::size_t nq = std::size_t(m0.nq);
        for (std::size_t l = 1; l < nloc; ++l) {
            const HostModes& ml = modes_of(crystal_of(l));
            if (ml.nq != m0.nq || ml.grid[0] != m0.grid[0] || ml.grid[1] != m0.grid[1])
                throw Error(BTE_ERR_INPUT, "spectral locations in crystals of different q grids");
        }
        out->nloc = int32_t(nloc);
        out->nbins = int32_t(nbins);
        out->nomega = int32_t(nw);
        out->nq = int32_t(nq);
        const double hbar = 1.054571726e-34;
        const bool steady = c->spec_steady;
        cudaStream_t s = c->stream;
        if (!c->spectral) c->spectral = new SpectralState();
        SpectralState& S = *c->spectral;
        const bool want_w = out->dT_omega || out->jx_omega || out->jy_omega;
        // per location three arrays [bin][tick] and one [bin][q]
        const std::size_t per = nbins * (3 * nw + nq);
        const bool compute = nloc > 0 && (want_w || out->fd_q);
        if (compute) {
            S.out.alloc(nloc * per * sizeof(double));
            ck(cudaMemsetAsync(S.out.p, 0, nloc * per * sizeof(double), s), "memset");
        }
        int pdf_of = -2;  // the crystal whose whole pdf is in S.pdf
        for (std::size_t l = 0; l < nloc; ++l) {
            const int kc = crystal_of(l);
            const HostModes& m = modes_of(kc);
            const std::size_t off = kc >= 0 ? c->crys_off[std::size_t(kc)] : 0, nk = m.n();
            // omega ticks of the location's crystal: LinSpaced(nomega, 0,
            // max omega) + delta/2 (:2041-2045)
            double maxw = 0.;
            for (double w : m.omega) maxw = std::max(maxw, w);
            std::vector<double> grid(nw);
            for (std::size_t i = 0; i < nw; ++i)
                grid[i] = (nw > 1 ? maxw * double(i) / double(nw - 1) : 0.) + 0.5 * maxw / double(nw);
            if (out->omega) std::copy(grid.begin(), grid.end(), out->omega + l * nw);
            if (!compute) continue;
            if (S.crystal != kc || S.version != c->tables_version) {
                sync(c);  // (an earlier location's kernels may still read them)
                S.version = -1;  // (until all of them are there)
                const std::vector<double> sig = mode_sigmas(m);
                S.hpar.assign(4 * nk, 0.);
                for (std::size_t k = 0; k < nk; ++k) {
                    const double w = m.omega[k];
                    if (!(w > 0.)) continue;
                    const double kk = w * w / sig[k], th = sig[k] / w;
                    double* p = S.hpar.data() + 4 * k;
                    p[0] = kk;
                    p[1] = th;
                    p[2] = std::lgamma(kk);
                    p[3] = std::log(th);
                }
                S.par.upload(S.hpar, s);
                S.om.upload(m.omega, s);
                S.vx.upload(m.vxc, s);
                S.vy.upload(m.vyc, s);
                sync(c);
                S.crystal = kc;
                S.version = c->tables_version;
            }
            double* o = S.out.as<double>() + l * per;
            const double* time = c->d_spec.as<double>() + l * nbins * n + off;
            if (want_w) {
                if (pdf_of != kc) {
                    S.ticks.upload(grid, s);
                    sync(c);
                }
                // (at most 65535 blocks over the modes)
                const int chunk = int(std::max<std::size_t>(
                    1, std::min({nk, PDF_BYTES / (nw * sizeof(double)), std::size_t(65535) * SPEC_K})));
                S.pdf.alloc(std::size_t(chunk) * nw * sizeof(double));
                for (std::size_t k0 = 0; k0 < nk; k0 += std::size_t(chunk)) {
                    const int kn = int(std::min(std::size_t(chunk), nk - k0));
                    const long long cells = (long long)kn * (long long)nw;
                    if (pdf_of != kc)
                        spec_pdf<<<unsigned(std::min<long long>((cells + 255) / 256, 8ll * c->nsm)), 256, 0, s>>>(
                            S.par.as<double4>(), S.om.as<double>(), int(k0), kn, S.ticks.as<double>(), int(nw),
                            S.pdf.as<double>());
                    for (std::size_t b0 = 0; b0 < nbins; b0 += 32768) {  // (grid limit in y)
                        const unsigned bn = unsigned(std::min<std::size_t>(32768, nbins - b0));
                        spec_contract<<<dim3(unsigned((nw + SPEC_T - 1) / SPEC_T), bn, unsigned((kn + SPEC_K - 1) / SPEC_K)),
                                        SPEC_T, 0, s>>>(time + b0 * n, c->spec_unit, (long long)n, int(nbins), S.vx.as<double>(),
                                                        S.vy.as<double>(), int(k0), kn, S.pdf.as<double>(), int(nw),
                                                        o + b0 * nw);
                    }
                }
                pdf_of = std::size_t(chunk) == nk ? kc : -2;
            }
            if (out->fd_q)
                spec_fdq<<<unsigned(std::min<std::size_t>((nbins * nq + 255) / 256, std::size_t(8 * c->nsm))), 256, 0, s>>>(
                    time, c->spec_unit, steady ? c->d_speccnt.as<long long>() + l * n + off : nullptr, (long long)n,
                    int(nbins), S.om.as<double>(), int(nq), m.nb, o + 3 * nbins * nw);
            // scaling (:2350-2376) and integration in time (:2386-2413)
            const int box = c->spec_boxes[l];
            const double tb = box_thickness(c, box);
            const double vcorr = tb / m.c;
            const double vbox = g.boxes[std::size_t(box)].area * tb;
            const double cv = calc_cv(m, box_T0(c, box, c->spec_T0));
            const double Eeff = c->spec_Eeff;
            const double sdT = Eeff / vbox, sj = Eeff * 1e12 * 1e9 * 1e9 / vbox;
            const double sq = Eeff * vcorr * double(nq) / (vbox * 1.0e+12 * hbar);
            SpecFinish f{{sdT, sj, sj, sq}, {cv / vcorr, 1.0, 1.0, 1.0}, {}};
            for (int q = 0; q < 4; ++q) f.n[q] = q < 3 ? (want_w ? int(nw) : 0) : (out->fd_q ? int(nq) : 0);
            const std::size_t widest = std::max(nw, nq);
            spec_finish<<<dim3(unsigned((widest + 31) / 32), 4), 32, 0, s>>>(o, int(nbins), int(nw), f, steady ? 0 : 1);
            ck(cudaGetLastError(), "spectral launch");
        }
        const std::size_t raw_vals = nloc * nbins * n, cnt_vals = nloc * n;
        const std::size_t out_bytes = compute ? nloc * per * sizeof(double) : 0;
        const bool cnt = out->counts && steady;
        S.host.reserve(out_bytes + (out->raw ? raw_vals * sizeof(double) : 0) + (cnt ? cnt_vals * sizeof(long long) : 0) + 16);
        char* h = static_cast<char*>(S.host.p);
        char* h_raw = h + out_bytes;
        char* h_cnt = h_raw + (out->raw ? raw_vals * sizeof(double) : 0);
        if (compute) ck(cudaMemcpyAsync(h, S.out.p, out_bytes, cudaMemcpyDeviceToHost, s), "d2h");
        if (out->raw) ck(cudaMemcpyAsync(h_raw, c->d_spec.p, raw_vals * sizeof(double), cudaMemcpyDeviceToHost, s), "d2h");
        if (cnt) ck(cudaMemcpyAsync(h_cnt, c->d_speccnt.p, cnt_vals * sizeof(long long), cudaMemcpyDeviceToHost, s), "d2h");
        sync(c);
        for (std::size_t l = 0; l < nloc && compute; ++l) {
            const double* o = reinterpret_cast<const double*>(h) + l * per;
            double* dst[4] = {out->dT_omega, out->jx_omega, out->jy_omega, out->fd_q};
            for (int q = 0; q < 4; ++q) {
                const std::size_t len = nbins * (q < 3 ? nw : nq);
                if (dst[q]) std::memcpy(dst[q] + l * len, o + std::size_t(q) * nbins * nw, len * sizeof(double));
            }
        }
        if (out->raw) {
            const double* r = reinterpret_cast<const double*>(h_raw);
            for (std::size_t i = 0; i < raw_vals; ++i) out->raw[i] = r[i] * c->spec_unit;
        }
        out->steady = steady ? 1 : 0;
        if (cnt) {
            const long long* r = reinterpret_cast<const long long*>(h_cnt);
            for (std::size_t i = 0; i < cnt_vals; ++i) out->counts[i] = double(r[i]);
        }
        if (out->q1bz) {
            // q points in Cartesian coordinates, reduced coordinates wrapped
            // to [-1/2, 1/2) (a Gamma-centred n1 x n2 grid, iq = i n2 + j)
            const HostModes& m = m0;
            const int n1 = m.grid[0] > 0 ? m.grid[0] : 1, n2 = m.grid[1] > 0 ? m.grid[1] : 1;
            for (std::size_t iq = 0; iq < nq; ++iq) {
                const int i = int(iq) / n2, j = int(iq) % n2;
                const int ii = (i + n1 / 2) % n1 - n1 / 2, jj = (j + n2 / 2) % n2 - n2 / 2;
                out->q1bz[2 * iq + 0] = ii * m.dq[0] + jj * m.dq[3];
                out->q1bz[2 * iq + 1] = ii * m.dq[1] + jj * m.dq[4];
            }
        }
        return BTE_OK;
    } catch (const Error& e) {
        c->err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        c->err = e.what();
        return BTE_ERR_CUDA;
    }
}
