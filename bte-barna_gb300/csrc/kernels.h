// kernels.h - launch wrappers of the particle-loop kernels (host side).
#pragma once

#include <cuda_runtime.h>

#include "fixed_walk.cuh"
#include "rta_flight.cuh"

namespace bte {

// Grid description of the axis-aligned fast path (production mode).
struct DevGrid {
    int nx, ny;
    const double* gx;   // nx + 1 grid lines
    const double* gy;   // ny + 1 grid lines
    const int* cell;    // [nx*ny] box id, -1 void, -2 - b reservoir box b
};

struct ProdTuning {
    int block_threads;
    int blocks_per_sm;
    int smem_tally;
    int particles_per_thread;  // accepted; every lane carries one
};

// (`work` is a zeroed particle counter)
void launch_replay(const DevTables& T, unsigned long long* ex, unsigned long long* counters,
                   int* err, unsigned long long* work, int nsm, cudaStream_t s);
void launch_mode_eps(const double* vx, const double* vy, int n, V2* eps, cudaStream_t s);

// General convex-box production kernel (any geometry); `work` is a zeroed
// particle counter.
void launch_prod_general(const DevTables& T, double* tally, unsigned long long* counters,
                         int* err, unsigned long long* work, int nsm, cudaStream_t s);

// One generation of the periodic / gradient steady state (rta_steady.cuh).
// With `select_flags` set, only the generation-0 pre-pass runs: it writes 1
// per slot whose first draw picks a gradient generator.
struct SteadyArgs;
void launch_steady_replay(const DevTables& T, const SteadyArgs& A, unsigned long long* ex,
                          unsigned long long* counters, int* err, unsigned* select_flags, int nsm,
                          cudaStream_t s);
void launch_steady_prod(const DevTables& T, const SteadyArgs& A, double* tally,
                        unsigned long long* counters, int* err, unsigned* select_flags, int nsm,
                        cudaStream_t s);

// Per-mode velocity record of the grid path.
struct __align__(32) ModeVel {
    double vx, vy;    // get_v velocities, nm/ps
    double ivx, ivy;  // their inverses (+inf where the component is 0)
};

// Grid-path kernel parameters beyond the tables.
struct GridArgs {
    DevGrid G;
    const int2* boxcell;     // box -> (i, j)
    const ModeVel* mv;       // per mode velocities and inverses
    FixScale fx;             // the run's integer units,
    const ModeFix* mf;       //   the modes' velocities in them
    const long long* gxf;    //   the grid lines
    const long long* gyf;
    const unsigned long long* wxf;  // and the widths between them
    const unsigned long long* wyf;
    const int* map;          // the cells with a void rim: [nx + 2][ny + 2], as G.cell
    int lanes;               // lanes of a warp that take particles (set by the launch)
    int refill;              // idle lanes of a warp before new particles are generated
    int cls[4];              // normal classes of the +x, -x, +y, -y walls (-1: none)
};

// Convex-polygon production path: every border as the line n.x = c (n its
// outward unit normal) with its start p, unit direction u, its wall class,
// and the pieces of it that touch a neighbour box, as intervals of the
// arc length s = (x - p).u.
struct PolyBorder {
    double nx, ny, c;
    double px, py, ux, uy;
    int piece_off, npieces, cls, pad;
};
struct PolyPiece {
    double s0, s1;  // the interval of s, widened by 1e-9 at both ends
    int box, pad;   // pad: the mismatch table of the contact (-1: same crystal)
};
// An axis-aligned rectangular box of the polygon path: its lines and the
// box's own indices of its +x, -x, +y, -y borders (kx1 = -1: not such a
// box, the general border search applies); across each side the
// neighbour box when one piece covers the whole side (-1: a void side,
// -2: look the side's pieces up), that box's flags (1: reservoir, 2:
// periodic) and the side's wall class.
struct PolyRect {
    double x0, x1, y0, y1;
    int kx1, kx0, ky1, ky0;
    int nx1, nx0, ny1, ny0;
    int fx1, fx0, fy1, fy0;
    int cx1, cx0, cy1, cy0;
    // 1: the box's +x and -x sides lead through periodic boxes that
    // translate by its width back into the box itself (a strip spanning
    // the period in x); likewise in y
    int perx, pery;
};
struct PolyArgs {
    const PolyBorder* pb;     // [global border index]
    const PolyPiece* pieces;
    const ModeVel* mv;
    // 1 / (n.v) per border normal class and mode ([nclass][n], -1 where the
    // flight does not leave through such a border); null: divide per pass
    const double* inv_den;
    const PolyRect* rect;     // [box] or null
    // diffuse mismatch interfaces between crystals: a piece whose pad is
    // t >= 0 leads through table t; its rows for global mode K are
    // dmm_row[t * (n + 1) + K .. + 1] into dmm_ent
    const long long* dmm_row;
    const DmmEnt* dmm_ent;
};

// Linked cells of axis-aligned boxes (rta_link.cu, build_link_grid): in the
// run's integer units the lines, widths and mode velocities, and per cell and
// side (+x, -x, +y, -y) what lies across it.
struct LinkEntry {
    int cell, box, flags, cls;  // LK_*; above bit 8 the mismatch table + 1 of an interface
};
constexpr int LK_VOID = 1, LK_RESERVOIR = 2, LK_TRANSLATE = 4, LK_INNER = 8;
struct LinkArgs {
    FixScale fx;
    const ModeFix* mf;
    const long long* gxf;
    const long long* gyf;
    const unsigned long long* wxf;
    const unsigned long long* wyf;
    int ny, refill;
    int lanes;                   // lanes of a warp that take particles (set by the launch)
    const int4* side;            // [cell = i ny + j][4] LinkEntry
    const int4* range;           // [box] columns [x, y) and rows [z, w)
    const unsigned char* per;    // [box] 1: spans the period in x, 2: in y
    const int* cellbox;          // [cell] its box
    const int4* cycle;           // [cell] columns of its x period, rows of its y period (-1: none)
    const int* pbox;             // [cell][4] the periodic box across a side (null: none that is entered)
    unsigned long long margin;   // 2e-6 nm
    const long long* dmm_row;
    const DmmEnt* dmm_ent;
};
bool launch_steady_link(const DevTables& T, const SteadyArgs& S, const LinkArgs& A, double* tally,
                        unsigned long long* counters, int* err, int nsm, cudaStream_t s);
bool launch_prod_link(const DevTables& T, const LinkArgs& A, double* tally, unsigned long long* counters, int* err,
                      unsigned long long* work, int nsm, cudaStream_t s);

// Adjoint passes of the grid kernel: the functional's weights per tally
// value, each particle's total contribution (slot = particle - first),
// per-mode gradient accumulators and {d/dp, sum of R over post-scattering
// draws, sum of Phi}.
struct AdjArgs {
    const double* W;      // [nboxes * nbins][3]
    double* phi_total;    // [particles]
    double* g_tau;        // [nmodes], times tau
    double* g_scalar;     // [3]
    int comps;            // bit q: W has a component q that is not zero
};

// Lanes of a warp that take particles, of a run of n.
// A run too small to fill the GPU is bound by the passes of its longest
// particles, and a pass takes as long as its warp's branches together: the
// particles are spread over one lane of up to 16 warps per SM, then over
// as few lanes of 8 warps as hold them.  Kernel times of 1e3, 2e3, 1e4 and
// 3e4 particles with all lanes in use 0.126, 0.62, 0.64 and 0.65 ms, so
// 0.089, 0.35, 0.48 and 0.56 on a ribbon (16 warps at 1e4: 0.55; 4: 0.54).
inline int particle_lanes(long long n, int nsm) {
    if (n <= 16ll * nsm) return 1;
    const long long l = (n + 8ll * nsm - 1) / (8ll * nsm);
    return l < 32 ? int(l) : 32;
}

// Axis-aligned grid production kernel (persistent, warp-refilled work).
// adj_pass 1 / 2 runs the forward / adjoint pass of the adjoint with `adj`
// (no tally).  The tally comes out in the units of A.fx.
// Returns false when the tuning cannot be honoured (e.g. smem too small).
// Production kernel of geometries that are not a grid: exit times from the
// convex box's border lines, neighbours from the border pieces.
bool launch_prod_poly(const DevTables& T, const PolyArgs& A, double* tally, unsigned long long* counters,
                      int* err, unsigned long long* work, int nsm, cudaStream_t s);
bool launch_steady_poly(const DevTables& T, const SteadyArgs& A, const PolyArgs& PA, double* tally,
                        unsigned long long* counters, int* err, int nsm, cudaStream_t s);

bool launch_prod_grid(const DevTables& T, const GridArgs& A, double* tally,
                      unsigned long long* counters, int* err, unsigned long long* work,
                      const ProdTuning& tune, int nsm, cudaStream_t s, int adj_pass = 0,
                      const AdjArgs* adj = nullptr);

// The integer tables of the scales f: mf[n] from mv, the lines and widths from G.
void launch_fix_tables(const FixScale& f, const ModeVel* mv, int n, ModeFix* mf, const DevGrid& G, long long* gxf,
                       long long* gyf, long long* wxf, long long* wyf, cudaStream_t s);
// The copies of a grid-kernel tally of n sums added into the first and turned
// from the walk's units into ps and nm.
void launch_gather_tally(double* tally, long long n, int ncopies, const FixScale& f, int nsm, cudaStream_t s);

// Kernel arguments of a context already prepared for one set of run
// parameters (see prepared_grid_run in capi.cu).
struct PreparedRun {
    DevTables T;
    GridArgs A;
    double Eeff, energy, maxtime, step;
    int nboxes, nbins, ntime;
    cudaStream_t stream;
    cudaEvent_t ev0, ev1;
    int device, nsm;
    ProdTuning tune;
};

}  // namespace bte
