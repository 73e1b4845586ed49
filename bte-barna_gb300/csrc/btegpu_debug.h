/* btegpu_debug.h - host-only views of the engine's tables, exported for the
 * CPU test suite (no GPU needed).  Not part of the public ABI. */
#ifndef BTEGPU_DEBUG_H
#define BTEGPU_DEBUG_H

#include "../../include/btegpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Per box: nborders, (p1x p1y p2x p2y npx npy) per border, ncontacts,
 * (id npx npy) per contact, centre x, y, area.  Returns the count written
 * (or needed when above cap), -1 on error. */
long long btegpu_debug_geometry(const bte_geometry* g, double* out, long long cap);

/* 1 when the boxes tile an axis-aligned grid (fast path), 0 if not. */
int btegpu_debug_grid(const bte_geometry* g, int* nx, int* ny);

/* Lambert-table entries per wall-normal class; returns the total. */
long long btegpu_debug_lambert(const bte_mode_table* m, const bte_geometry* g,
                               long long* nnz_per_class, int maxclass);

/* One properties.msgpack.bin frame; returns its byte count. */
long long btegpu_debug_frame(double time, double Eeff, const double* temps, const int* H, int nboxes,
                             int nmodes, char* out, long long cap);

/* The linked cells of a geometry (build_link_grid): returns their number, 0
 * where the boxes cannot be linked, minus the number needed when above cap.
 * lines: the x lines, then the y lines; out: nx, ny, then per cell four rows
 * (+x, -x, +y, -y) of cell, box, flags, and the cell's four period limits. */
long long btegpu_debug_links(const bte_geometry* g, double* lines, int* out, long long cap);

/* The integer walk of the grid kernel (fixed_walk.cuh), on the host: one
 * particle from (px, py) through free flights k of tau[k] e[k] ps at
 * (vx[k], vy[k]) over the cells of the lines gx[0..nx], gy[0..ny], nbins time
 * bins of `step` ps, until it leaves the grid or the bins end.  Per segment
 * five values: flight, kind (1 / 2: crosses a line in x / y, 4: flight ends,
 * 8: part of a bin ends), x, y, ticks; scales: kx, kt, sub.  Returns the
 * number of segments. */
long long btegpu_debug_fixwalk(const double* gx, int nx, const double* gy, int ny, double vmax, double step,
                               int nbins, double px, double py, long long nflights, const float* e,
                               const double* tau, const double* vx, const double* vy, int* scales, long long* out,
                               long long cap);

/* What a buffer is kept by (Keyed, ctx.hpp): n updates to keys[i], whose fill
 * fails where fails[i]; filled[i]: whether the fill ran.  Returns whether the
 * buffer counts as filled at the end. */
int btegpu_debug_keyed(const int* keys, const int* fails, int n, int* filled);

/* The host build of bte_log. */
int btegpu_debug_log(const double* x, double* y, long long n);

#ifdef __cplusplus
}
#endif

#endif
