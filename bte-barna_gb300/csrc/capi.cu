// capi.cu - the C ABI of include/btegpu.h: context, device tables, run
// orchestration and the post-processing of src/RTA_MC2D.cpp:2326-2435.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <tuple>
#include <string>
#include <thread>
#include <vector>

#include "../../include/btegpu.h"
#include "btegpu_debug.h"
#include "kernels.h"
#include "tables.hpp"
#include "ctx.hpp"
#include "frames.hpp"

using bte::Error;

namespace {

thread_local std::string g_create_error;

}  // namespace

using bte::ck;
using bte::DBuf;
using bte::hw_threads;

namespace bte {

void sync(bte_ctx* c) { ck(cudaStreamSynchronize(c->stream), "cudaStreamSynchronize"); }

void ensure_static(bte_ctx* c) {
    const bte::HostModes& m = c->modes;
    const bte::HostGeometry& g = c->geom;
    const std::size_t n = m.n();
    if (!c->modes_dev) {
        // rates of every material, [nmat][n] (one set without materials)
        const std::vector<double>& wall = c->nmat > 0 ? c->mat_w : m.w;
        std::vector<double> tau(wall.size());
        for (std::size_t k = 0; k < wall.size(); ++k) tau[k] = wall[k] > 0. ? 1.0 / wall[k] : 0.;
        std::vector<bte::ModeVel> mv(n);
        for (std::size_t k = 0; k < n; ++k) {
            mv[k].vx = m.vxc[k];
            mv[k].vy = m.vyc[k];
            mv[k].ivx = m.vxc[k] != 0. ? 1.0 / m.vxc[k] : HUGE_VAL;
            mv[k].ivy = m.vyc[k] != 0. ? 1.0 / m.vyc[k] : HUGE_VAL;
        }
        c->d_vxc.upload(m.vxc, c->stream);
        c->d_vyc.upload(m.vyc, c->stream);
        c->d_w.upload(wall, c->stream);
        c->d_tau.upload(tau, c->stream);
        c->d_mv.upload(mv, c->stream);
        c->d_mf.alloc(n * sizeof(bte::ModeFix));
        c->d_eps.alloc(n * sizeof(bte::V2));
        bte::launch_mode_eps(c->d_vxc.as<double>(), c->d_vyc.as<double>(), int(n), c->d_eps.as<bte::V2>(), c->stream);
        c->vmax = 0.;
        for (std::size_t k = 0; k < n; ++k) c->vmax = std::max({c->vmax, std::fabs(m.vxc[k]), std::fabs(m.vyc[k])});
        c->fix_dev = false;
        sync(c);
        c->modes_dev = true;
    }
    if (!c->geom_dev) {
        c->d_boxes.upload(g.boxes, c->stream);
        c->d_hull.upload(g.hull, c->stream);
        c->d_borders.upload(g.borders, c->stream);
        c->d_contacts.upload(g.contacts, c->stream);
        c->d_cseg.upload(g.contact_seg, c->stream);
        c->d_transl.upload(g.translation, c->stream);
        {
            std::vector<bte::RectKey> rk(g.boxes.size());
            for (std::size_t b = 0; b < rk.size(); ++b) rk[b] = bte::rect_key(g, b);
            c->d_rkey.upload(rk, c->stream);
            sync(c);
        }
        c->d_boxmat.upload(g.mat, c->stream);
        {
            const bte::TranslationFast tf = bte::build_translation_fast(g);
            c->have_tfast = !tf.iv.empty();
            if (c->have_tfast) {
                c->d_tfast.upload(tf.iv, c->stream);
                c->d_tfast_rng.upload(tf.rng, c->stream);
                c->d_tfast_u.upload(tf.u, c->stream);
            }
        }
        c->link = bte::build_link_grid(g);
        const std::vector<double>& gx = g.rect_grid ? g.gx : c->link.gx;
        const std::vector<double>& gy = g.rect_grid ? g.gy : c->link.gy;
        if (g.rect_grid || c->link.ok) {
            c->d_gx.upload(gx, c->stream);
            c->d_gy.upload(gy, c->stream);
            for (bte::DBuf* d : {&c->d_gxf, &c->d_wxf}) d->alloc(gx.size() * sizeof(long long));
            for (bte::DBuf* d : {&c->d_gyf, &c->d_wyf}) d->alloc(gy.size() * sizeof(long long));
            c->fix_dev = false;
        }
        if (g.rect_grid) {
            c->d_gcell.upload(g.gcell, c->stream);
            std::vector<int2> bc(g.boxes.size(), make_int2(-1, -1));
            for (int i = 0; i < g.gnx; ++i)
                for (int j = 0; j < g.gny; ++j) {
                    int v = g.gcell[std::size_t(i) * g.gny + j];
                    int b = v >= 0 ? v : (v <= -2 ? -2 - v : -1);
                    if (b >= 0) bc[std::size_t(b)] = make_int2(i, j);
                }
            c->d_boxcell.upload(bc, c->stream);
            std::vector<int> map(std::size_t(g.gnx + 2) * std::size_t(g.gny + 2), -1);
            for (int i = 0; i < g.gnx; ++i)
                for (int j = 0; j < g.gny; ++j)
                    map[std::size_t(i + 1) * std::size_t(g.gny + 2) + std::size_t(j + 1)] =
                        g.gcell[std::size_t(i) * g.gny + j];
            c->d_map.upload(map, c->stream);
            sync(c);
        }
        {
            // border lines and neighbour pieces of the convex-polygon path
            // (transient boxes off a grid, every steady-state geometry):
            // a segment contact of box a lies on the border of a whose
            // outward normal is the contact's normal; its ends give the
            // interval of arc length that leads into the neighbour
            std::vector<bte::PolyBorder> pb(g.borders.size());
            std::vector<bte::PolyPiece> pieces;
            for (std::size_t a = 0; a < g.boxes.size(); ++a) {
                const bte::GBox& bx = g.boxes[a];
                for (int k = 0; k < bx.nborders; ++k) {
                    const std::size_t gb = std::size_t(bx.border_off + k);
                    const bte::GBorder& br = g.borders[gb];
                    bte::PolyBorder& P = pb[gb];
                    const double len = std::hypot(br.p2.x - br.p1.x, br.p2.y - br.p1.y);
                    P.nx = br.np.x;
                    P.ny = br.np.y;
                    P.c = br.np.x * br.p1.x + br.np.y * br.p1.y;
                    P.px = br.p1.x;
                    P.py = br.p1.y;
                    P.ux = len > 0. ? (br.p2.x - br.p1.x) / len : 0.;
                    P.uy = len > 0. ? (br.p2.y - br.p1.y) / len : 0.;
                    P.cls = br.ncls;
                    P.piece_off = int(pieces.size());
                    for (int i = 0; i < bx.ncontacts; ++i) {
                        const std::size_t ci = std::size_t(bx.contact_off + i);
                        const bte::GBorder& cb = g.contact_borders[ci];
                        if (cb.p1.x == cb.p2.x && cb.p1.y == cb.p2.y) continue;  // point contact
                        const bte::GContact& gc = g.contacts[ci];
                        if (std::fabs(gc.np.x - br.np.x) > 1e-9 || std::fabs(gc.np.y - br.np.y) > 1e-9) continue;
                        const double d1 = br.np.x * cb.p1.x + br.np.y * cb.p1.y - P.c;
                        const double d2 = br.np.x * cb.p2.x + br.np.y * cb.p2.y - P.c;
                        if (std::fabs(d1) > 1e-6 || std::fabs(d2) > 1e-6) continue;  // on another line
                        double s0 = (cb.p1.x - P.px) * P.ux + (cb.p1.y - P.py) * P.uy;
                        double s1 = (cb.p2.x - P.px) * P.ux + (cb.p2.y - P.py) * P.uy;
                        if (s0 > s1) std::swap(s0, s1);
                        pieces.push_back(bte::PolyPiece{s0 - 1.0e-9, s1 + 1.0e-9, gc.id, -1});
                    }
                    P.npieces = int(pieces.size()) - P.piece_off;
                }
            }
            if (pieces.empty()) pieces.push_back(bte::PolyPiece{0., 0., -1, -1});
            c->d_pborders.upload(pb, c->stream);
            c->d_ppieces.upload(pieces, c->stream);
            c->pieces_host = pieces;
            c->pborders_host = pb;
            c->dmm_dev = false;
            // axis-aligned rectangles: four borders with normals +x, -x, +y, -y
            std::vector<bte::PolyRect> rect(g.boxes.size());
            for (std::size_t a = 0; a < g.boxes.size(); ++a) {
                const bte::GBox& bx = g.boxes[a];
                bte::PolyRect R{0., 0., 0., 0., -1, -1, -1, -1, -2, -2, -2, -2, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
                int k4[4] = {-1, -1, -1, -1};
                double c4[4] = {0., 0., 0., 0.};
                bool ok = bx.nborders == 4;
                for (int k = 0; ok && k < 4; ++k) {
                    const bte::PolyBorder& P = pb[std::size_t(bx.border_off + k)];
                    const int side = P.nx == 1. && P.ny == 0. ? 0 : P.nx == -1. && P.ny == 0. ? 1
                                   : P.nx == 0. && P.ny == 1. ? 2 : P.nx == 0. && P.ny == -1. ? 3 : -1;
                    if (side < 0 || k4[side] >= 0) ok = false;
                    else {
                        k4[side] = k;
                        c4[side] = P.c;
                    }
                }
                if (ok) {
                    R.x0 = -c4[1];
                    R.x1 = c4[0];
                    R.y0 = -c4[3];
                    R.y1 = c4[2];
                    R.kx1 = k4[0];
                    R.kx0 = k4[1];
                    R.ky1 = k4[2];
                    R.ky0 = k4[3];
                    if (!(R.x0 < R.x1 && R.y0 < R.y1)) R.kx1 = -1;
                    // what lies across each whole side
                    int nbs[4], fls[4], cls[4];
                    for (int sd = 0; sd < 4; ++sd) {
                        const bte::PolyBorder& P = pb[std::size_t(bx.border_off + k4[sd])];
                        const double len = sd < 2 ? R.y1 - R.y0 : R.x1 - R.x0;
                        cls[sd] = P.cls;
                        fls[sd] = 0;
                        if (P.npieces == 0) {
                            nbs[sd] = -1;
                        } else if (P.npieces == 1 && pieces[std::size_t(P.piece_off)].s0 <= 0. &&
                                   pieces[std::size_t(P.piece_off)].s1 >= len) {
                            const int nb = pieces[std::size_t(P.piece_off)].box;
                            nbs[sd] = nb;
                            fls[sd] = (g.reservoir[std::size_t(nb)] ? 1 : 0) | (g.tto[std::size_t(nb)] >= 0 ? 2 : 0);
                            // a contact between crystals takes the piece lookup (its table)
                            if (g.mat[std::size_t(nb)] != g.mat[a]) nbs[sd] = -2;
                        } else {
                            nbs[sd] = -2;
                        }
                    }
                    R.nx1 = nbs[0];
                    R.nx0 = nbs[1];
                    R.ny1 = nbs[2];
                    R.ny0 = nbs[3];
                    R.fx1 = fls[0];
                    R.fx0 = fls[1];
                    R.fy1 = fls[2];
                    R.fy0 = fls[3];
                    R.cx1 = cls[0];
                    R.cx0 = cls[1];
                    R.cy1 = cls[2];
                    R.cy0 = cls[3];
                    // a strip spanning the period: the periodic box across
                    // one side translates by the box's extent onto the
                    // periodic box across the other side, whose whole side
                    // this box is (geometry_2d::translate lands there)
                    auto self_periodic = [&](int hi, int lo, double ext, bool along_x) {
                        if (hi < 0 || lo < 0 || !(fls[along_x ? 0 : 2] & 2) || !(fls[along_x ? 1 : 3] & 2)) return 0;
                        const bte::V2 th = g.translation[std::size_t(hi)], tl = g.translation[std::size_t(lo)];
                        const bool ok = g.tto[std::size_t(hi)] == lo && g.tto[std::size_t(lo)] == hi &&
                                        (along_x ? (th.x == -ext && th.y == 0. && tl.x == ext && tl.y == 0.)
                                                 : (th.y == -ext && th.x == 0. && tl.y == ext && tl.x == 0.));
                        return ok ? 1 : 0;
                    };
                    if (R.kx1 >= 0) {
                        R.perx = self_periodic(R.nx1, R.nx0, R.x1 - R.x0, true);
                        R.pery = self_periodic(R.ny1, R.ny0, R.y1 - R.y0, false);
                    }
                }
                rect[a] = R;
            }
            c->d_prect.upload(rect, c->stream);
            if (c->link.ok) {
                bte::LinkGrid& L = c->link;
                std::vector<unsigned char> per(g.boxes.size());
                for (std::size_t a = 0; a < per.size(); ++a) {
                    const int* r = L.range.data() + 4 * a;
                    per[a] = (unsigned char)((rect[a].kx1 >= 0 && rect[a].perx ? 1 : 0) |
                                             (rect[a].kx1 >= 0 && rect[a].pery ? 2 : 0));
                    // (a wrap by the box's width needs it to be one cell there)
                    if (((per[a] & 1) && r[1] - r[0] != 1) || ((per[a] & 2) && r[3] - r[2] != 1)) L.ok = false;
                }
                c->link_corner = false;
                std::vector<int> pbox(L.side.size(), -1);
                for (std::size_t k = 0; k < pbox.size(); ++k) {
                    if (!(L.side[k].flags & bte::LINK_TRANSLATE)) continue;
                    // the periodic box itself: the cell across the side
                    const int cell = int(k / 4), sd = int(k % 4), i = cell / L.ny, j = cell % L.ny;
                    const int pi = i + (sd == 0) - (sd == 1), pj = j + (sd == 2) - (sd == 3);
                    for (std::size_t b = 0; b < g.boxes.size(); ++b) {
                        const int* r = L.range.data() + 4 * b;
                        if (pi >= r[0] && pi < r[1] && pj >= r[2] && pj < r[3]) pbox[k] = int(b);
                        // a box that spans this period wraps instead
                        if (i >= r[0] && i < r[1] && j >= r[2] && j < r[3] && !(per[b] & (sd < 2 ? 1 : 2)))
                            c->link_corner = true;
                    }
                }
                c->d_lrange.upload(L.range, c->stream);
                c->d_lper.upload(per, c->stream);
                c->d_lcycle.upload(L.cycle, c->stream);
                c->d_lpbox.upload(pbox, c->stream);
                c->d_lbox.upload(L.box, c->stream);
                c->d_lside.upload(L.side, c->stream);  // (interfaces: filled in with their tables)
                sync(c);
            }
        }
        sync(c);
        c->geom_dev = true;
    }
    if (!c->lambert_dev) {
        bte::LambertTable L;
        std::vector<int> mir;
        if (c->ncrys > 0) {  // each crystal's rows over its own modes, then offset
            std::vector<bte::LambertTable> Ls;
            std::vector<std::vector<int>> ms;
            for (const bte::HostModes& cm : c->crys) {
                Ls.push_back(bte::build_lambert(cm, g, hw_threads()));
                ms.push_back(bte::build_mirror(cm, g));
            }
            L = bte::merge_lambert(Ls, c->crys, c->crys_off);
            mir = bte::merge_mirror(ms, c->crys, c->crys_off, L.nclass);
        } else {
            L = bte::build_lambert(m, g, hw_threads());
            mir = bte::build_mirror(m, g);
        }
        c->nclass = L.nclass;
        c->d_row_ptr.upload(L.row_ptr, c->stream);
        std::vector<unsigned long long> lrow(std::size_t(L.nclass) * m.n());
        for (int k = 0; k < L.nclass; ++k)
            for (std::size_t j = 0; j < m.n(); ++j) {
                const long long* r = L.row_ptr.data() + std::size_t(k) * (m.n() + 1) + j;
                if (r[0] >> 36 || (r[1] - r[0]) >> 28) throw Error(BTE_ERR_INPUT, "Lambert table too large");
                lrow[std::size_t(k) * m.n() + j] = (unsigned long long)r[0] | ((unsigned long long)(r[1] - r[0]) << 36);
            }
        c->d_lrow.upload(lrow, c->stream);
        c->d_lcol.upload(L.col, c->stream);
        c->d_lcdf.upload(L.cdf, c->stream);
        c->d_lalias.upload(L.alias, c->stream);
        c->have_mirror = std::any_of(mir.begin(), mir.end(), [](int x) { return x >= 0; });
        c->d_mirror.upload(mir, c->stream);
        // exit times of the convex-polygon path without a division: 1 / (n.v)
        // per border normal and mode, -1 where such a border is not left
        // (n.v <= 0); only for tables of at most 256 MB
        const std::size_t n = m.n(), ncl = g.normals.size();
        c->d_invden.release();
        if (ncl > 0 && ncl * n * sizeof(double) <= (std::size_t(256) << 20)) {
            std::vector<double> inv(ncl * n);
            for (std::size_t k = 0; k < ncl; ++k)
                for (std::size_t j = 0; j < n; ++j) {
                    const double den = g.normals[k].x * m.vxc[j] + g.normals[k].y * m.vyc[j];
                    inv[k * n + j] = den > 0. ? 1.0 / den : -1.0;
                }
            c->d_invden.upload(inv, c->stream);
        }
        sync(c);
        c->lambert_dev = true;
        if (c->verbose)
            std::printf("#Diffusive table: %d wall normals, %zu entries\n", L.nclass, L.col.size());
    }
    if (c->ncrys > 0 && !c->dmm_dev) {
        // one mismatch table per (crystal A, crystal B, contact normal) over
        // the contacts from a box that is neither a reservoir nor periodic to
        // a box of another crystal, at the Teq of the first such box
        std::map<std::tuple<int, int, double, double>, int> tab_of;
        std::vector<long long> rows;
        std::vector<bte::DmmEnt> ents;
        const std::size_t ntot = m.n();
        for (std::size_t a = 0; a < g.boxes.size(); ++a) {
            if (g.reservoir[a] || g.tto[a] >= 0) continue;
            const bte::GBox& B = g.boxes[a];
            for (int i = 0; i < B.ncontacts; ++i) {
                const std::size_t ci = std::size_t(B.contact_off + i);
                const int b = g.contacts[ci].id;
                const int ma = g.mat[a], mb = g.mat[std::size_t(b)];
                if (ma == mb) continue;
                const bte::V2 nw = g.contact_borders[ci].np;
                const auto key = std::make_tuple(ma, mb, nw.x, nw.y);
                if (tab_of.count(key)) continue;
                const bte::HostModes& A = c->crys[std::size_t(ma)];
                const bte::HostModes& Bm = c->crys[std::size_t(mb)];
                const bte::DmmTable D = bte::build_dmm_table(
                    A, c->crys_off[std::size_t(ma)], Bm, c->crys_off[std::size_t(mb)], ntot, nw,
                    A.V * bte::crystal_thickness(c, ma) / A.c, Bm.V * bte::crystal_thickness(c, mb) / Bm.c,
                    g.Teq[a], hw_threads());
                tab_of[key] = int(tab_of.size());
                const long long base = (long long)ents.size();
                for (std::size_t K = 0; K <= ntot; ++K) rows.push_back(base + D.row[K]);
                for (std::size_t e = 0; e < D.out.size(); ++e) ents.push_back(bte::DmmEnt{D.cum[e], D.out[e], D.side[e]});
            }
        }
        // each piece that leads into another crystal names its table
        std::vector<bte::PolyPiece>& pcs = c->pieces_host;
        for (std::size_t a = 0; a < g.boxes.size(); ++a) {
            if (g.reservoir[a] || g.tto[a] >= 0) continue;
            const bte::GBox& B = g.boxes[a];
            for (int i = 0; i < B.ncontacts; ++i) {
                const std::size_t ci = std::size_t(B.contact_off + i);
                const int b = g.contacts[ci].id;
                if (g.mat[a] == g.mat[std::size_t(b)]) continue;
                const bte::V2 nw = g.contact_borders[ci].np;
                const int t = tab_of.at(std::make_tuple(g.mat[a], g.mat[std::size_t(b)], nw.x, nw.y));
                for (int k = 0; k < B.nborders; ++k) {
                    const bte::PolyBorder& P = c->pborders_host[std::size_t(B.border_off + k)];
                    for (int j = 0; j < P.npieces; ++j) {
                        bte::PolyPiece& pc = pcs[std::size_t(P.piece_off + j)];
                        if (pc.box == b) pc.pad = t;
                    }
                }
            }
        }
        // the same tables per contact, for the evolparticle-faithful kernels
        std::vector<int> cdmm(g.contacts.size(), -1);
        for (std::size_t a = 0; a < g.boxes.size(); ++a) {
            if (g.reservoir[a] || g.tto[a] >= 0) continue;
            const bte::GBox& B = g.boxes[a];
            for (int i = 0; i < B.ncontacts; ++i) {
                const std::size_t ci = std::size_t(B.contact_off + i);
                const int b = g.contacts[ci].id;
                if (g.mat[a] == g.mat[std::size_t(b)]) continue;
                const bte::V2 nw = g.contact_borders[ci].np;
                cdmm[ci] = tab_of.at(std::make_tuple(g.mat[a], g.mat[std::size_t(b)], nw.x, nw.y));
            }
        }
        std::vector<int> coff;
        for (int k = 0; k <= c->ncrys; ++k)
            coff.push_back(k < c->ncrys ? int(c->crys_off[std::size_t(k)]) : int(m.n()));
        if (cdmm.empty()) cdmm.push_back(-1);
        if (rows.empty()) rows.push_back(0);
        if (ents.empty()) ents.push_back(bte::DmmEnt{0., 0, 0});
        c->d_dmm_row.upload(rows, c->stream);
        c->d_dmm_ent.upload(ents, c->stream);
        c->d_cdmm.upload(cdmm, c->stream);
        c->d_crysoff.upload(coff, c->stream);
        c->d_ppieces.upload(pcs, c->stream);
        std::vector<bte::LinkSide> side = c->link.side;
        for (bte::LinkSide& k : side)
            if (k.flags >> 8) k.flags = (k.flags & 255) | ((cdmm[std::size_t((k.flags >> 8) - 1)] + 1) << 8);
        if (c->link.ok) c->d_lside.upload(side, c->stream);
        c->ndmm = int(tab_of.size());
        sync(c);
        c->dmm_dev = true;
    }
}

void ensure_resample(bte_ctx* c, double T0) {
    if (c->nmat > 0) T0 = -2.0;  // one table per material, at the material's T0
    if (c->resample_T0 == T0) return;
    std::vector<double> cdf;
    std::vector<bte::Alias> al;
    if (c->nmat > 0) {
        const std::size_t n = c->modes.n(), nmat = std::size_t(c->nmat);
        cdf.resize(nmat * n);
        al.resize(nmat * n);
        bte::host_parallel(nmat, hw_threads(), [&](std::size_t k) {
            bte::HostModes mm = c->modes;
            std::vector<double> ck;
            std::vector<bte::Alias> ak;
            mm.w.assign(c->mat_w.begin() + std::ptrdiff_t(k * n), c->mat_w.begin() + std::ptrdiff_t((k + 1) * n));
            bte::build_resample(mm, c->mat_T0[k], ck, ak);
            std::copy(ck.begin(), ck.end(), cdf.begin() + std::ptrdiff_t(k * n));
            std::copy(ak.begin(), ak.end(), al.begin() + std::ptrdiff_t(k * n));
        });
    } else {
        bte::build_resample(c->modes, T0, cdf, al);
    }
    static_assert(sizeof(bte::Alias) == sizeof(int2) && offsetof(bte::Alias, alt) == 4, "an alias slot is an int2");
    c->resample_T0 = -1;  // (until all of it is there)
    c->d_rcdf.upload(cdf, c->stream);
    c->d_resample.upload(al, c->stream);
    sync(c);
    c->resample_T0 = T0;
}

}  // namespace bte

namespace {
// Header of a run's device buffer: 16 counters, the work counter at 128, four
// error words at RUN_ERR; the tally follows.
constexpr std::size_t RUN_ERR = 136, RUN_HEAD = 256;
using bte::ensure_resample;
using bte::ensure_static;
using bte::sync;

// Per-material budgets of a walls-source run: wall w of material m is drawn
// with probability share[m] E_w / E_m (energy-weighted when no shares).
void apply_shares(bte_ctx* c, bool upload) {
    if (c->mat_share.empty()) {
        c->shares_dirty = false;
        return;
    }
    c->shares_dirty = true;  // (until the weights are there)
    const std::size_t nm = c->mat_share.size();
    c->mat_energy.assign(nm, 0.);
    for (auto& W : c->gens.walls) {
        const std::size_t k = std::size_t(c->geom.mat[std::size_t(W.box)]);
        if (k >= nm) throw Error(BTE_ERR_INPUT, "box material without loaded rates (bte_load_materials)");
        c->mat_energy[k] += W.energy;
    }
    for (std::size_t k = 0; k < nm; ++k)
        if (c->mat_share[k] > 0. && !(c->mat_energy[k] > 0.))
            throw Error(BTE_ERR_INPUT, "a material with a particle share has no isothermal wall");
    double cum = 0.;
    for (std::size_t i = 0; i < c->gens.walls.size(); ++i) {
        const auto& W = c->gens.walls[i];
        const std::size_t k = std::size_t(c->geom.mat[std::size_t(W.box)]);
        cum += c->mat_share[k] * W.energy / c->mat_energy[k];
        c->gens.wall_cum[i] = cum;
    }
    if (upload) {
        c->d_wcum.upload(c->gens.wall_cum, c->stream);
        sync(c);
    }
    c->shares_dirty = false;
}

void ensure_generators(bte_ctx* c, const bte_rta_params* p) {
    if (c->gen_key_source == p->source) {
        if (p->source == BTE_SOURCE_WALLS && c->shares_dirty) apply_shares(c, true);
        if (p->source == BTE_SOURCE_INITIAL &&
            (c->gen_key_n != p->nparticles || c->gen_key_seed != p->seed)) {
            c->gen_key_n = -1;  // (until the counts are there)
            c->gen_Eeff = bte::initial_counts(c->gens, p->nparticles, p->seed);
            c->d_ifirst.upload(c->gens.init_first, c->stream);
            sync(c);
            c->gen_key_n = p->nparticles;
            c->gen_key_seed = p->seed;
        }
        return;
    }
    bte::Generators gens;  // (a failure up to here leaves the present ones)
    if (c->ncrys > 0) {
        // each crystal's generators, rows over the concatenated modes
        std::vector<bte::Generators> G;
        for (int k = 0; k < c->ncrys; ++k) {
            const bte::GenEmbed e{k, c->crys_off[std::size_t(k)], c->modes.n(), bte::crystal_thickness(c, k)};
            G.push_back(p->source == BTE_SOURCE_WALLS
                            ? bte::build_wall_generators(c->crys[std::size_t(k)], c->geom, false, &e)
                            : bte::build_initial_generators(c->crys[std::size_t(k)], c->geom, &e));
        }
        gens = bte::merge_generators(G, p->source == BTE_SOURCE_WALLS, true);
    } else if (p->source == BTE_SOURCE_WALLS) {
        gens = bte::build_wall_generators(c->modes, c->geom);
    } else {
        if (!c->mat_share.empty()) throw Error(BTE_ERR_INPUT, "particle shares need the walls source");
        gens = bte::build_initial_generators(c->modes, c->geom);
    }
    c->gen_key_source = -1;  // (until all of them are there)
    c->gens = std::move(gens);
    if (p->source == BTE_SOURCE_INITIAL) c->gen_Eeff = bte::initial_counts(c->gens, p->nparticles, p->seed);
    else if (c->ncrys == 0) apply_shares(c, false);
    std::vector<float> prob(c->gens.alias.size());
    std::vector<int> alt(c->gens.alias.size());
    const std::size_t chunk = std::size_t(1) << 20;
    bte::host_parallel((prob.size() + chunk - 1) / chunk, hw_threads(), [&](std::size_t b) {
        for (std::size_t i = b * chunk; i < std::min(prob.size(), (b + 1) * chunk); ++i) {
            prob[i] = c->gens.alias[i].prob;
            alt[i] = c->gens.alias[i].alt;
        }
    });
    c->d_gcdf.upload(c->gens.cdf, c->stream);
    c->d_gprob.upload(prob, c->stream);
    c->d_galt.upload(alt, c->stream);
    std::vector<bte::WallGenDev> wd;
    for (auto& W : c->gens.walls) {
        bte::WallGenDev d;
        d.p1 = W.p1;
        d.nd = W.nd;
        d.sa = W.sa;
        d.sb = W.sb;
        d.box = W.box;
        d.sign = W.sign;
        wd.push_back(d);
    }
    c->d_walls.upload(wd, c->stream);
    c->d_wcum.upload(c->gens.wall_cum, c->stream);
    c->d_ifirst.upload(c->gens.init_first, c->stream);
    c->d_ibox.upload(c->gens.init_box, c->stream);
    c->d_isign.upload(c->gens.init_sign, c->stream);
    sync(c);
    c->gen_key_source = p->source;
    c->gen_key_n = p->nparticles;
    c->gen_key_seed = p->seed;
}

bte_status fail(bte_ctx* c, const Error& e) {
    c->err = e.what();
    return e.code;
}

void validate(const bte_rta_params* p) {
    if (!p) throw Error(BTE_ERR_INPUT, "null parameters");
    if (!(p->dt > 0.) || !(p->maxtime > 0.) || !std::isfinite(p->dt) || !std::isfinite(p->maxtime))
        throw Error(BTE_ERR_INPUT, "time dt and maxtime must be positive");
    if (p->maxtime / p->dt > 1.0e7) throw Error(BTE_ERR_INPUT, "too many time bins");
    if (p->nparticles < 1) throw Error(BTE_ERR_INPUT, "particles N must be >= 1");
    if (p->mode != BTE_MODE_REPLAY && p->mode != BTE_MODE_PRODUCTION)
        throw Error(BTE_ERR_INPUT, "unknown mode");
    if (p->source != BTE_SOURCE_WALLS && p->source != BTE_SOURCE_INITIAL)
        throw Error(BTE_ERR_INPUT, "unknown particle source");
    if (!(p->specularity >= 0. && p->specularity <= 1.))
        throw Error(BTE_ERR_INPUT, "specularity must lie in [0, 1]");
    if (!(p->T0 > 0.)) throw Error(BTE_ERR_INPUT, "T0 must be positive");
}

}  // namespace

namespace bte {
// Validation and tables of one RTA run (shared by bte_rta_run and
// bte_rta_adjoint).
void prepare_run(bte_ctx* c, const bte_rta_params* p) {
    validate(p);
    if (!c->have_modes || !c->have_geom)
        throw Error(BTE_ERR_STATE, "load the mode table and the geometry before running");
    ck(cudaSetDevice(c->device), "cudaSetDevice");
    if (c->ncrys > 0) {
        // crystals joined by mismatch interfaces: every crystal at the run's T0
        if (c->mat_T0.empty() || c->mat_T0[0] != p->T0) {
            c->mat_T0.assign(std::size_t(c->ncrys), p->T0);
            c->resample_T0 = -1;
        }
    }
    for (std::size_t b = 0; b < c->geom.boxes.size(); ++b) {
        if (c->geom.mat[b] >= std::max(c->nmat, 1))
            throw Error(BTE_ERR_INPUT, "box material without loaded rates (bte_load_materials)");
        const double T0b = bte::box_T0(c, int(b), p->T0);
        if (c->nmat > 0 && c->ncrys == 0) {  // a particle keeps its material: materials must not touch
            const bte::GBox& B = c->geom.boxes[b];
            for (int i = 0; i < B.ncontacts; ++i) {
                const int o = c->geom.contacts[std::size_t(B.contact_off + i)].id;
                if (c->geom.mat[std::size_t(o)] != c->geom.mat[b])
                    throw Error(BTE_ERR_INPUT, "boxes of different materials touch");
            }
            if (c->geom.tto[b] >= 0 && c->geom.mat[std::size_t(c->geom.tto[b])] != c->geom.mat[b])
                throw Error(BTE_ERR_INPUT, "a periodic box maps to another material");
        }
        if (!c->geom.reservoir[b] && !bte::almost_equal(c->geom.Teq[b], T0b) && c->geom.Teq[b] != T0b)
            throw Error(BTE_ERR_INPUT, "Tref in xml is different from provided T0");
    }
    ensure_static(c);
    if (p->specularity > 0. && !c->have_mirror)
        throw Error(BTE_ERR_INPUT, "specular walls need an axis-aligned q grid with mirror images");
    ensure_resample(c, p->T0);
    ensure_generators(c, p);
}
}  // namespace bte

namespace {

// Per box: 1 / V_box times the energy (and flux) factor, the temperature per
// energy density, and the reference temperature.
struct BoxPost {
    double e, j, t, T0;
};
struct PostArgs {
    const double* tally;     // [ncopies][box][bin][3]
    int ncopies;
    long long stride;        // doubles from one copy to the next
    double unit_t, unit_x;   // of the raw sums
    int nboxes, nbins, integrate;
    const BoxPost* box;
    double* raw[3];          // outputs [box][bin], null: not asked for
    double* post[3];
};

// The outputs of a production run from its tally (src/RTA_MC2D.cpp:2336-2435):
// the copies summed, per box the energy and flux factors, and for a walls
// source the sum over the time bins so far.  One warp per box and quantity
// takes 32 bins at a time; the running sum is a warp scan.  The host took
// 2 ms for it on the 1e6-particle ribbon's 5200 keys and 25 ms on the sweep's
// 333 000 with eight groups (copying every group's tally back first).
__global__ void __launch_bounds__(128) post_tally(PostArgs a) {
    const int w = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int b = w / 3, q = w % 3;
    if (b >= a.nboxes || !(a.raw[q] || a.post[q])) return;
    const BoxPost f = a.box[b];
    const double unit = q == 0 ? a.unit_t : a.unit_x, fac = q == 0 ? f.e : f.j;
    double carry = 0.;
    for (int i0 = 0; i0 < a.nbins; i0 += 32) {
        const int i = i0 + lane;
        const long long k = (long long)b * a.nbins + i;
        double v = 0.;
        if (i < a.nbins)
            for (int c = 0; c < a.ncopies; ++c) v += a.tally[c * a.stride + 3 * k + q];
        v *= unit;
        if (a.raw[q] && i < a.nbins) a.raw[q][k] = v;
        if (!a.post[q]) continue;
        v *= fac;
        if (a.integrate) {
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            v += carry;
            carry = __shfl_sync(0xffffffffu, v, 31);
        }
        if (i < a.nbins) a.post[q][k] = q == 0 ? v * f.t + f.T0 : v;
    }
}

}  // namespace

namespace bte {
// C_v per material (per crystal: over its own modes, q points and cell),
// cached while the tables and temperatures stay.
const std::vector<double>& heat_capacities(bte_ctx* c, double T0) {
    std::vector<double> T0s(std::size_t(std::max(c->nmat, 1)));
    for (std::size_t k = 0; k < T0s.size(); ++k) T0s[k] = c->nmat > 0 ? c->mat_T0[k] : T0;
    if (c->cv_version != c->tables_version || c->cv_T0s != T0s) {
        c->cv_cache.resize(T0s.size());
        for (std::size_t k = 0; k < T0s.size(); ++k)
            c->cv_cache[k] = bte::calc_cv(c->ncrys > 0 ? c->crys[k] : c->modes, T0s[k]);
        c->cv_T0s = T0s;
        c->cv_version = c->tables_version;
    }
    return c->cv_cache;
}

// The outputs `out` asks for, formed on the device from the tally at
// `tally` and read back with `head` bytes of the run's header in front of
// them (into *hdr): one launch, one copy, one synchronisation.
void device_post(bte_ctx* c, const bte_rta_params* p, int nbx, int nbins, double Eeff, double step,
                 const double* tally, int ncopies, PostUnits u, std::size_t head, bte_rta_result* out) {
    const HostGeometry& g = c->geom;
    const std::size_t nk = std::size_t(nbx) * std::size_t(nbins);
    const bool initial = p->source != BTE_SOURCE_WALLS;
    const bool shares = !c->mat_share.empty() && !initial;
    const std::vector<double>* cvm = out->temperature ? &heat_capacities(c, p->T0) : nullptr;
    std::vector<double> bp(std::size_t(nbx) * 4);
    for (int b = 0; b < nbx; ++b) {
        const std::size_t m = std::size_t(c->nmat > 0 ? g.mat[std::size_t(b)] : 0);
        // Eeff_m = E_m / (share_m N) per material with shares
        double E = Eeff;
        if (shares) E = c->mat_share[m] > 0. ? c->mat_energy[m] / (c->mat_share[m] * double(p->nparticles)) : 0.;
        if (initial) E /= step;  // relaxation of an initial deviation: bin averages
        const double thick = box_thickness(c, b), vbox = g.boxes[std::size_t(b)].area * thick;
        const double vcorr = thick / (c->ncrys > 0 ? c->crys[m].c : c->modes.c);
        double* f = bp.data() + std::size_t(b) * 4;
        f[0] = E / vbox;
        f[1] = E * 1e12 * 1e9 * 1e9 / vbox;
        f[2] = cvm ? vcorr / (*cvm)[m] : 0.;
        f[3] = box_T0(c, b, p->T0);
    }
    c->boxpost.update(std::move(bp), [&](const std::vector<double>& v) { c->d_boxpost.upload(v, c->stream); });
    PostArgs a{};
    a.tally = tally;
    a.ncopies = ncopies;
    a.stride = (long long)(nk * 3);
    a.unit_t = u.t;
    a.unit_x = u.x;
    a.nboxes = nbx;
    a.nbins = nbins;
    a.integrate = initial ? 0 : 1;
    a.box = c->d_boxpost.as<BoxPost>();
    double* host[6] = {out->gz, out->gz_jx, out->gz_jy, out->temperature, out->jx, out->jy};
    std::size_t n = 0;
    for (int q = 0; q < 6; ++q)
        if (host[q]) ++n;
    const std::size_t bytes = head + n * nk * sizeof(double);
    c->d_out.alloc(bytes);
    c->h_out.reserve(bytes);
    double* d = reinterpret_cast<double*>(c->d_out.as<char>() + head);
    for (int q = 0, k = 0; q < 6; ++q)
        if (host[q]) (q < 3 ? a.raw[q] : a.post[q - 3]) = d + nk * std::size_t(k++);
    if (n) post_tally<<<unsigned((3 * nbx + 3) / 4), 128, 0, c->stream>>>(a);
    ck(cudaGetLastError(), "post-processing launch");
    char* h = static_cast<char*>(c->h_out.p);
    if (head) ck(cudaMemcpyAsync(h, c->d_run.p, head, cudaMemcpyDeviceToHost, c->stream), "d2h");
    if (n) ck(cudaMemcpyAsync(h + head, d, n * nk * sizeof(double), cudaMemcpyDeviceToHost, c->stream), "d2h");
    sync(c);
    if (head && *reinterpret_cast<const int*>(h + RUN_ERR) != 0) return;  // the run failed
    const double* r = reinterpret_cast<const double*>(h + head);
    for (int q = 0, k = 0; q < 6; ++q)
        if (host[q]) std::memcpy(host[q], r + nk * std::size_t(k++), nk * sizeof(double));
}

// The post-processing of a replay run's raw tallies on the host
// (src/RTA_MC2D.cpp:2336-2435): / V_box, x Eeff (per material with shares),
// the flux factor, the time integration of a walls source (or bin averages
// of an initial deviation) and T = gz / (C_v / vcorr) + T0.
void rta_post(bte_ctx* c, const bte_rta_params* p, int nbx, int nbins, double Eeff, double step,
              std::vector<double>& gz, std::vector<double>& jx, std::vector<double>& jy, bte_rta_result* out) {
    const bte::HostModes& m = c->modes;
    const bte::HostGeometry& g = c->geom;
    const std::size_t nk = std::size_t(nbx) * std::size_t(nbins);
    // only the tallies an output needs: gz for the temperature, jx, jy
    const bool need_gz = out->temperature != nullptr, need_jx = out->jx != nullptr, need_jy = out->jy != nullptr;
    auto each = [&](auto&& f) {
        if (need_gz) f(gz);
        if (need_jx) f(jx);
        if (need_jy) f(jy);
    };
    // post-processing, src/RTA_MC2D.cpp:2336-2435
    each([&](std::vector<double>& v) {
        for (int ir = 0; ir < nbx; ++ir) {
            const double vbox = g.boxes[std::size_t(ir)].area * bte::box_thickness(c, ir);
            for (int i = 0; i < nbins; ++i) v[std::size_t(ir) * nbins + i] /= vbox;
        }
    });
    if (!c->mat_share.empty() && p->source == BTE_SOURCE_WALLS) {
        // Eeff_m = E_m / (share_m N) per material
        for (int ir = 0; ir < nbx; ++ir) {
            const std::size_t k = std::size_t(g.mat[std::size_t(ir)]);
            const double Em = c->mat_share[k] > 0. ? c->mat_energy[k] / (c->mat_share[k] * double(p->nparticles)) : 0.;
            for (int i = 0; i < nbins; ++i) {
                const std::size_t q = std::size_t(ir) * nbins + i;
                if (need_gz) gz[q] *= Em;
                if (need_jx) jx[q] *= Em * 1e12 * 1e9 * 1e9;
                if (need_jy) jy[q] *= Em * 1e12 * 1e9 * 1e9;
            }
        }
    } else {
        if (need_gz)
            for (auto& x : gz) x *= Eeff;
        if (need_jx)
            for (auto& x : jx) x *= Eeff * 1e12 * 1e9 * 1e9;
        if (need_jy)
            for (auto& x : jy) x *= Eeff * 1e12 * 1e9 * 1e9;
    }
    if (p->source == BTE_SOURCE_WALLS) {
        // step response: integrate in time
        each([&](std::vector<double>& v) {
            for (int ir = 0; ir < nbx; ++ir)
                for (int i = 1; i < nbins; ++i) {
                    const std::size_t k = std::size_t(ir) * nbins + i;
                    v[k] += v[k - 1];
                }
        });
    } else {
        // relaxation of an initial deviation: bin averages
        each([&](std::vector<double>& v) {
            for (std::size_t k = 0; k < nk; ++k) v[k] /= step;
        });
    }
    if (out->temperature) {
        const std::vector<double>& cvm = heat_capacities(c, p->T0);
        for (int ir = 0; ir < nbx; ++ir) {
            const std::size_t mk = std::size_t(c->nmat > 0 ? g.mat[std::size_t(ir)] : 0);
            const double cv = cvm[mk];
            const double vcorr = bte::box_thickness(c, ir) / (c->ncrys > 0 ? c->crys[mk].c : m.c);
            const double T0b = bte::box_T0(c, ir, p->T0);
            for (int i = 0; i < nbins; ++i) {
                const std::size_t k = std::size_t(ir) * nbins + i;
                out->temperature[k] = gz[k] / (cv / vcorr) + T0b;
            }
        }
    }
    if (out->jx) std::copy(jx.begin(), jx.end(), out->jx);
    if (out->jy) std::copy(jy.begin(), jy.end(), out->jy);
}
}  // namespace bte

extern "C" {

int32_t bte_version(void) { return BTEGPU_VERSION; }

bte_status bte_create(bte_ctx** out, const bte_device_opts* opts) {
    if (!out) return BTE_ERR_INPUT;
    *out = nullptr;
    try {
        std::unique_ptr<bte_ctx> c(new bte_ctx());
        c->device = opts ? opts->device : 0;
        c->verbose = opts ? opts->verbose : 0;
        int ndev = 0;
        ck(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
        if (c->device < 0 || c->device >= ndev) throw Error(BTE_ERR_INPUT, "no such CUDA device");
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        ck(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->device), "attribute");
        ck(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), "cudaStreamCreate");
        ck(cudaEventCreate(&c->ev0), "cudaEventCreate");
        ck(cudaEventCreate(&c->ev1), "cudaEventCreate");
        *out = c.release();
        return BTE_OK;
    } catch (const Error& e) {
        g_create_error = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_create_error = e.what();
        return BTE_ERR_CUDA;
    }
}

bte_status bte_destroy(bte_ctx* c) {
    if (!c) return BTE_OK;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    cudaStream_t s = c->stream;
    bte::destroy_berta(c);
    bte::destroy_steady(c);
    bte::destroy_spectral(c);
    delete c;
    if (s) cudaStreamDestroy(s);
    return BTE_OK;
}

bte_status bte_last_error(const bte_ctx* c, char* buf, size_t size) {
    if (!buf || size == 0) return BTE_ERR_INPUT;
    const std::string& m = c ? c->err : g_create_error;
    std::snprintf(buf, size, "%s", m.c_str());
    return BTE_OK;
}

bte_status bte_set_tuning(bte_ctx* c, const bte_tuning* t) {
    if (!c) return BTE_ERR_INPUT;
    if (!t) {
        c->tune = bte::ProdTuning{0, 0, 0, 0};
        return BTE_OK;
    }
    if (t->block_threads < 0 || t->block_threads > 256 || (t->block_threads % 32) != 0) {
        c->err = "block_threads must be a multiple of 32 in [32, 256] (0 = default)";
        return BTE_ERR_INPUT;
    }
    c->tune.block_threads = t->block_threads;
    c->tune.blocks_per_sm = t->blocks_per_sm;
    c->tune.smem_tally = t->smem_tally;
    if (t->particles_per_thread < 0 || t->particles_per_thread > 2) {
        c->err = "particles_per_thread must be 1 or 2 (0 = default)";
        return BTE_ERR_INPUT;
    }
    c->tune.particles_per_thread = t->particles_per_thread;
    return BTE_OK;
}

bte_status bte_load_modes(bte_ctx* c, const bte_mode_table* mt) {
    if (!c) return BTE_ERR_INPUT;
    c->group_valid = false;
    try {
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        c->modes = bte::build_modes(mt);
        c->have_modes = true;
        c->tables_version++;
        c->spec_valid = false;
        bte::reset_propagators(c);
        c->ncrys = 0;
        c->crys.clear();
        c->crys_off.clear();
        c->crys_thick.clear();
        c->dmm_dev = false;
        c->nmat = 0;  // materials are rate sets over one table
        c->mat_w.clear();
        c->mat_T0.clear();
        c->modes_dev = false;
        c->lambert_dev = false;
        c->resample_T0 = -1;
        c->gen_key_source = -1;
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    }
}

bte_status bte_load_geometry(bte_ctx* c, const bte_geometry* g) {
    if (!c) return BTE_ERR_INPUT;
    c->group_valid = false;
    try {
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        bte::HostGeometry ng = bte::build_geometry(g);
        // the Lambert wall table depends on the geometry only through its
        // distinct wall normals: keep it when they are the same
        const bool same_normals = c->have_geom && ng.normals.size() == c->geom.normals.size() &&
                                  std::equal(ng.normals.begin(), ng.normals.end(), c->geom.normals.begin(),
                                             [](const bte::V2& a, const bte::V2& b) {
                                                 return a.x == b.x && a.y == b.y;
                                             });
        c->geom = std::move(ng);
        c->have_geom = true;
        c->tables_version++;
        c->spec_valid = false;
        c->geom_dev = false;
        c->dmm_dev = false;
        if (!same_normals) c->lambert_dev = false;
        c->gen_key_source = -1;
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    }
}

bte_status bte_load_mode_tables(bte_ctx* c, int32_t ntables, const bte_mode_table* tables,
                                const double* thickness) {
    if (!c) return BTE_ERR_INPUT;
    c->group_valid = false;
    try {
        if (ntables < 1 || !tables) throw Error(BTE_ERR_INPUT, "no mode tables");
        std::vector<double> th;
        if (thickness)
            for (int k = 0; k < ntables; ++k) {
                if (!(thickness[k] > 0.) || !std::isfinite(thickness[k]))
                    throw Error(BTE_ERR_INPUT, "crystal thickness must be > 0");
                th.push_back(thickness[k]);
            }
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        std::vector<bte::HostModes> crys;
        for (int k = 0; k < ntables; ++k) crys.push_back(bte::build_modes(&tables[k]));
        std::vector<std::size_t> off;
        bte::HostModes all = bte::concat_modes(crys, off);
        if (all.n() > (std::size_t(1) << 30)) throw Error(BTE_ERR_INPUT, "too many modes");
        // the materials machinery with one rate set per crystal, each masked
        // to its crystal's modes (zero rate, so zero weight, elsewhere)
        const std::size_t n = all.n();
        std::vector<double> mw(std::size_t(ntables) * n, 0.);
        for (int k = 0; k < ntables; ++k)
            for (std::size_t j = 0; j < crys[std::size_t(k)].n(); ++j)
                mw[std::size_t(k) * n + off[std::size_t(k)] + j] = crys[std::size_t(k)].w[j];
        c->modes = std::move(all);
        c->crys = std::move(crys);
        c->crys_off = std::move(off);
        c->crys_thick = std::move(th);
        c->ncrys = ntables;
        c->have_modes = true;
        c->tables_version++;
        c->spec_valid = false;
        bte::reset_propagators(c);
        c->nmat = ntables;
        c->mat_w = std::move(mw);
        c->mat_T0.clear();  // set to each run's T0
        c->mat_share.clear();
        c->modes_dev = false;
        c->lambert_dev = false;
        c->dmm_dev = false;
        c->resample_T0 = -1;
        c->gen_key_source = -1;
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    }
}

bte_status bte_interface_table(const bte_mode_table* A, const bte_mode_table* B, double nx, double ny,
                               double thickness_a, double thickness_b, double Tref, int64_t* first,
                               int64_t* nentries, int32_t* side, int32_t* mode, double* cum) {
    try {
        if (!A || !B || !first || !nentries || !(thickness_a > 0.) || !(thickness_b > 0.) || !(Tref > 0.))
            return BTE_ERR_INPUT;
        const bte::HostModes a = bte::build_modes(A), b = bte::build_modes(B);
        const std::size_t na = a.n();
        const bte::DmmTable D = bte::build_dmm_table(a, 0, b, na, na + b.n(), bte::v2(nx, ny),
                                                     a.V * thickness_a / a.c, b.V * thickness_b / b.c, Tref,
                                                     hw_threads());
        for (std::size_t i = 0; i <= na; ++i) first[i] = D.row[i];
        *nentries = (int64_t)D.out.size();
        if (side && mode && cum)
            for (std::size_t e = 0; e < D.out.size(); ++e) {
                side[e] = D.side[e];
                mode[e] = D.side[e] == 0 ? D.out[e] : int32_t(std::size_t(D.out[e]) - na);
                cum[e] = D.cum[e];
            }
        return BTE_OK;
    } catch (const Error& e) {
        g_create_error = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_create_error = e.what();
        return BTE_ERR_INPUT;
    }
}

bte_status bte_load_materials(bte_ctx* c, int32_t nmat, const double* w, const double* T0,
                              const double* share) {
    if (!c) return BTE_ERR_INPUT;
    c->group_valid = false;
    try {
        if (c->ncrys > 0) throw Error(BTE_ERR_STATE, "rate sets are for one mode table; crystals carry their own rates");
        if (nmat < 0 || (nmat > 0 && (!w || !T0))) throw Error(BTE_ERR_INPUT, "bad material arrays");
        if (share && nmat > 0) {
            double sum = 0.;
            for (int k = 0; k < nmat; ++k) {
                if (!(share[k] >= 0.) || !std::isfinite(share[k])) throw Error(BTE_ERR_INPUT, "bad share");
                sum += share[k];
            }
            if (std::fabs(sum - 1.0) > 1e-9) throw Error(BTE_ERR_INPUT, "material shares must sum to 1");
        }
        if (nmat > 0 && !c->have_modes) throw Error(BTE_ERR_STATE, "load the mode table first");
        const std::size_t n = c->modes.n();
        for (int k = 0; k < nmat; ++k) {
            if (!(T0[k] > 0.) || !std::isfinite(T0[k])) throw Error(BTE_ERR_INPUT, "material T0 must be > 0");
            for (std::size_t i = 0; i < n; ++i)
                if (!std::isfinite(w[size_t(k) * n + i]) || w[size_t(k) * n + i] < 0.)
                    throw Error(BTE_ERR_VALUE, "non-finite or negative material rate");
        }
        const bool same_rates = nmat > 0 && nmat == c->nmat &&
                                std::equal(w, w + size_t(nmat) * n, c->mat_w.begin()) &&
                                std::equal(T0, T0 + nmat, c->mat_T0.begin());
        if (same_rates && share && !c->mat_share.empty()) {
            // only the particle budgets change: reweight the walls
            c->mat_share.assign(share, share + nmat);
            c->shares_dirty = true;
            return BTE_OK;
        }
        // (the spectral outputs are formed with the run's materials)
        if (!same_rates && (nmat > 0 || c->nmat > 0)) c->spec_valid = false;
        c->nmat = nmat;
        c->mat_w.assign(w ? w : nullptr, w ? w + size_t(nmat) * n : nullptr);
        c->mat_T0.assign(T0 ? T0 : nullptr, T0 ? T0 + nmat : nullptr);
        c->mat_share.assign(share && nmat > 0 ? share : nullptr, share && nmat > 0 ? share + nmat : nullptr);
        c->gen_key_source = -1;  // wall weights depend on the shares
        c->modes_dev = false;    // rates and lifetimes
        c->geom_dev = false;     // box materials
        c->resample_T0 = -1;     // post-scattering tables
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    }
}

bte_status bte_set_spectral(bte_ctx* c, int32_t nloc, const int32_t* boxes, int32_t nomega) {
    if (!c) return BTE_ERR_INPUT;
    try {
        if (nloc < 0 || (nloc > 0 && (!boxes || nomega < 1)))
            throw Error(BTE_ERR_INPUT, "spectral locations need boxes and ticks >= 1");
        if (nloc > 0 && !c->have_geom) throw Error(BTE_ERR_STATE, "load the geometry first");
        for (int i = 0; i < nloc; ++i) {
            if (boxes[i] < 0 || boxes[i] >= int(c->geom.boxes.size()))
                throw Error(BTE_ERR_INPUT, "spectral location is not a box");
            for (int j = 0; j < i; ++j)
                if (boxes[j] == boxes[i]) throw Error(BTE_ERR_INPUT, "repeated spectral location");
        }
        c->spec_boxes.assign(boxes ? boxes : nullptr, boxes ? boxes + nloc : nullptr);
        c->spec_nomega = nloc > 0 ? nomega : 0;
        c->spec_valid = false;
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    }
}

bte_status bte_set_groups(bte_ctx* c, int32_t ngroups) {
    if (!c) return BTE_ERR_INPUT;
    if (ngroups < 0 || ngroups > 4096) {
        c->err = "ngroups must be in [0, 4096]";
        return BTE_ERR_INPUT;
    }
    c->ngroups = ngroups;
    c->group_valid = false;
    return BTE_OK;
}

bte_status bte_get_group_result(bte_ctx* c, int32_t group, bte_rta_result* out) {
    if (!c || !out) return BTE_ERR_INPUT;
    if (!c->group_valid) {
        c->err = "no run with replica groups since the last bte_set_groups";
        return BTE_ERR_STATE;
    }
    if (group < 0 || group >= c->group_n) {
        c->err = "group index out of range";
        return BTE_ERR_INPUT;
    }
    try {
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        const std::size_t nk = std::size_t(c->group_nbx) * std::size_t(c->group_nbins);
        // the group holds 1/G of the run's particles: x G estimates the whole run
        const double G = double(c->group_n);
        out->nboxes = c->group_nbx;
        out->nbins = c->group_nbins;
        out->Eeff = c->group_Eeff;
        out->energy_rate = c->gens.total_energy;
        out->events = out->wall_hits = out->crossings = out->absorbed = 0;
        out->specular_hits = out->tally_updates = out->translations = 0;
        out->kernel_ms = 0.;
        const double* tally = reinterpret_cast<const double*>(c->d_run.as<char>() + RUN_HEAD) + std::size_t(group) * nk * 3;
        bte::device_post(c, &c->group_params, c->group_nbx, c->group_nbins, c->group_Eeff, c->group_step, tally, 1,
                         bte::PostUnits{c->group_units.t * G, c->group_units.x * G}, 0, out);
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    } catch (const std::exception& e) {
        c->err = e.what();
        return BTE_ERR_INPUT;
    }
}

bte_status bte_query_sizes(const bte_ctx* c, const bte_rta_params* p, int32_t* nboxes,
                           int32_t* nbins, int64_t* nmodes) {
    if (!c || !p) return BTE_ERR_INPUT;
    if (nboxes) *nboxes = int32_t(c->geom.boxes.size());
    if (nbins) *nbins = p->dt > 0 ? int32_t(std::floor(p->maxtime / p->dt + 1.0e-6)) : 0;
    if (nmodes) *nmodes = int64_t(c->modes.n());
    return BTE_OK;
}

bte_status bte_rta_run(bte_ctx* c, const bte_rta_params* p, bte_rta_result* out) {
    if (!c || !out) return BTE_ERR_INPUT;
    try {
        bte::prepare_run(c, p);
        const bte::HostModes& m = c->modes;
        const bte::HostGeometry& g = c->geom;
        // time grid, src/RTA_MC2D.cpp:2118-2124
        const std::size_t ntime = std::size_t(std::floor(p->maxtime / p->dt + 1.0e-6)) + 1;
        if (ntime < 2) throw Error(BTE_ERR_INPUT, "maxtime shorter than one time bin");
        const double maxtime = double(ntime - 1) * p->dt;
        const double step = (maxtime - 0.0) / double(ntime - 1);
        const bool replay = p->mode == BTE_MODE_REPLAY;
        const bool grid_run = !replay && g.rect_grid && c->ncrys == 0;
        // linked cells, unless particles start inside a periodic box or a
        // reservoir (an initial deviation there), which the cells do not model
        bool link_run = !replay && !grid_run && c->link.ok && !(p->flags & BTE_FLAG_GENERAL);
        if (p->source == BTE_SOURCE_INITIAL)
            for (int b : c->gens.init_box)
                if (g.tto[std::size_t(b)] >= 0 || g.reservoir[std::size_t(b)]) link_run = false;
        bte::GridArgs A{};
        bte::LinkArgs LA{};
        if (grid_run) bte::prepare_fixed(c, step, A);
        if (link_run) {
            bte::prepare_link(c, step, LA);
            A.fx = LA.fx;
        }
        bte::upload_time_grid(c, int(ntime), maxtime, step, A.fx.kt - A.fx.sub);
        const int nbins = int(ntime - 1);
        const int nbx = int(g.boxes.size());
        const std::size_t nk = std::size_t(nbx) * std::size_t(nbins);
        c->group_valid = false;
        if (c->ngroups > 1 && !grid_run)  // (no other kernel knows the groups)
            throw Error(BTE_ERR_INPUT, "replica groups need production mode on boxes of one mode table that tile a grid");
        const int ngroups = c->ngroups > 1 ? c->ngroups : 1;
        const std::size_t tally_bytes =
            replay ? nk * 6 * sizeof(unsigned long long) : nk * 3 * sizeof(double) * std::size_t(ngroups);
        // Eeff (src/RTA_MC2D.cpp:2177) and the particle range
        double Eeff;
        long long total;
        if (p->source == BTE_SOURCE_WALLS) {
            Eeff = c->gens.total_energy / double(p->nparticles);
            total = p->nparticles;
        } else {
            Eeff = c->gen_Eeff;
            total = c->gens.init_first.back();
        }
        long long pbeg = std::max<long long>(0, p->particle_begin);
        long long pend = p->particle_end > 0 ? std::min<long long>(p->particle_end, total) : total;
        if (pend < pbeg) pend = pbeg;

        // A small tally is hit by all SMs at few places (the cells next to the
        // reservoirs, the first bins), and reductions on one address serialise
        // in L2: 1.25e5 B took 4.25 ms with one copy, 3.54 with two, 3.41 with
        // four, 3.38 with eight (1e6 particles, 5200 keys; 2e5 particles, 1080
        // keys: 1.17, 0.75, 0.58, 0.53), and of that 1 % less with 32; a periodic
        // bar of 14 boxes (2e6 particles, 1400 keys) 1.79 with eight, 1.45 with
        // 32.  A run too small to fill the GPU takes four (2e4 particles: 658 us
        // with one, 628 with four, 634 with 32).  Copies beyond 16 MB in all only
        // fill L2 (11.6 MB: 118.0 ms with one, 118.8 with eight).
        int ncopies = 1;
        if ((grid_run || link_run) && ngroups == 1)
            ncopies = int(std::clamp<std::size_t>((std::size_t(16) << 20) / tally_bytes, 1,
                                                  bte::particle_lanes(pend - pbeg, c->nsm) < 32 ? 4 : 32));
        const std::size_t run_bytes = RUN_HEAD + tally_bytes * std::size_t(ncopies);
        c->d_run.alloc(run_bytes);
        ck(cudaMemsetAsync(c->d_run.p, 0, run_bytes, c->stream), "memset");
        char* base = c->d_run.as<char>();
        auto* counters = reinterpret_cast<unsigned long long*>(base);
        auto* work = reinterpret_cast<unsigned long long*>(base + 128);
        auto* err = reinterpret_cast<int*>(base + RUN_ERR);
        auto* tally = reinterpret_cast<double*>(base + RUN_HEAD);

        bte::DevTables T{};
        T.n = int(m.n());
        T.nb = m.nb;
        T.vxc = c->d_vxc.as<double>();
        T.vyc = c->d_vyc.as<double>();
        T.w = c->d_w.as<double>();
        T.tau = c->d_tau.as<double>();
        T.resample_cdf = c->d_rcdf.as<double>();
        T.resample = c->d_resample.as<int2>();
        T.nboxes = nbx;
        T.boxes = c->d_boxes.as<bte::GBox>();
        T.hull = c->d_hull.as<bte::V2>();
        T.borders = c->d_borders.as<bte::GBorder>();
        T.contacts = c->d_contacts.as<bte::GContact>();
        T.cseg = c->d_cseg.as<bte::V2>();
        T.translation = c->d_transl.as<bte::V2>();
        T.tfast = c->have_tfast ? c->d_tfast.as<bte::TransFast>() : nullptr;
        T.tfast_rng = c->d_tfast_rng.as<int2>();
        T.tfast_u = c->d_tfast_u.as<bte::V2>();
        T.nclass = c->nclass;
        T.row_ptr = c->d_row_ptr.as<long long>();
        T.lcol = c->d_lcol.as<int>();
        T.lcdf = c->d_lcdf.as<double>();
        T.lrow = c->d_lrow.as<unsigned long long>();
        T.lalias = c->d_lalias.as<int4>();
        T.mirror = c->have_mirror ? c->d_mirror.as<int>() : nullptr;
        T.box_mat = c->nmat > 0 ? c->d_boxmat.as<int>() : nullptr;
        bte::set_crystal_tables(c, T);
        T.rkey = c->d_rkey.as<bte::RectKey>();
        T.eps = c->d_eps.as<bte::V2>();
        T.ntime = int(ntime);
        T.timegrid = c->d_time.as<double>();
        T.maxtime = maxtime;
        T.inv_dt = 1.0 / step;
        T.source = p->source;
        T.ngen = p->source == BTE_SOURCE_WALLS ? int(c->gens.walls.size()) : int(c->gens.init_box.size());
        T.gen_cdf = c->d_gcdf.as<double>();
        T.gen_prob = c->d_gprob.as<float>();
        T.gen_alt = c->d_galt.as<int>();
        T.walls = c->d_walls.as<bte::WallGenDev>();
        T.wall_cum = c->d_wcum.as<double>();
        T.init_first = c->d_ifirst.as<long long>();
        T.init_box = c->d_ibox.as<int>();
        T.init_sign = c->d_isign.as<int>();
        T.seed = p->seed;
        T.flight_cap = p->flight_cap > 0 ? p->flight_cap : bte::EVENT_CAP;
        T.checks = (p->flags & BTE_FLAG_CHECKS) ? 1 : 0;
        T.ballistic = p->ballistic;
        T.specularity = p->specularity;
        T.pbegin = pbeg;
        T.pend = pend;
        T.nbins = nbins;
        T.ngroups = ngroups;
        T.group_stride = (long long)(nk * 3);
        T.ncopies = ncopies;
        // spectral decomposition: per-mode time at the selected boxes
        c->spec_valid = false;
        const std::size_t nloc = c->spec_boxes.size();
        const std::size_t spec_vals = nloc * std::size_t(nbins) * m.n();
        if (nloc > 0) {
            bte::upload_spectral_locations(c);
            const std::size_t bytes = spec_vals * (replay ? 2 * sizeof(unsigned long long) : sizeof(double));
            c->d_spec.alloc(bytes);
            ck(cudaMemsetAsync(c->d_spec.p, 0, bytes, c->stream), "memset");
            T.spec_loc = c->d_specloc.as<int>();
            T.spec = c->d_spec.as<double>();
            T.spec_ex = c->d_spec.as<unsigned long long>();
        }

        bte::PostUnits units;
        ck(cudaEventRecord(c->ev0, c->stream), "cudaEventRecord");
        if (replay) {
            bte::launch_replay(T, reinterpret_cast<unsigned long long*>(tally), counters, err, work, c->nsm, c->stream);
        } else if (grid_run) {
            if (!bte::launch_prod_grid(T, A, tally, counters, err, work, c->tune, c->nsm, c->stream))
                throw Error(BTE_ERR_INPUT, "tuning not supported by the grid kernel");
        } else if (link_run) {
            if (!bte::launch_prod_link(T, LA, tally, counters, err, work, c->nsm, c->stream))
                throw Error(BTE_ERR_CUDA, "linked-cell kernel does not fit on the device");
        } else if (p->flags & BTE_FLAG_GENERAL) {
            bte::launch_prod_general(T, tally, counters, err, work, c->nsm, c->stream);
        } else {
            const bte::PolyArgs PA{c->d_pborders.as<bte::PolyBorder>(), c->d_ppieces.as<bte::PolyPiece>(),
                                  c->d_mv.as<bte::ModeVel>(), c->d_invden.as<double>(),
                                  c->d_prect.as<bte::PolyRect>(),
                                  c->ncrys > 0 ? c->d_dmm_row.as<long long>() : nullptr,
                                  c->ncrys > 0 ? c->d_dmm_ent.as<bte::DmmEnt>() : nullptr};
            if (!bte::launch_prod_poly(T, PA, tally, counters, err, work, c->nsm, c->stream))
                throw Error(BTE_ERR_CUDA, "polygon kernel does not fit on the device");
        }
        ck(cudaGetLastError(), "kernel launch");
        ck(cudaEventRecord(c->ev1, c->stream), "cudaEventRecord");
        std::vector<unsigned long long> hex;
        if (replay) {
            hex.resize(nk * 6);
            ck(cudaMemcpyAsync(hex.data(), tally, tally_bytes, cudaMemcpyDeviceToHost, c->stream), "d2h");
            c->h_out.reserve(RUN_HEAD);
            ck(cudaMemcpyAsync(c->h_out.p, base, RUN_HEAD, cudaMemcpyDeviceToHost, c->stream), "d2h");
            sync(c);
        } else {
            // the outputs' sum over replica groups or copies, in their order
            if (grid_run || link_run) units = bte::PostUnits{A.fx.per_tick(), A.fx.per_unit()};
            bte::device_post(c, p, nbx, nbins, Eeff, step, tally, ngroups > 1 ? ngroups : ncopies, units, RUN_HEAD, out);
        }
        unsigned long long hc[16];
        int herr[4];
        std::memcpy(hc, c->h_out.p, sizeof hc);
        std::memcpy(herr, static_cast<const char*>(c->h_out.p) + RUN_ERR, sizeof herr);
        float ms = 0;
        ck(cudaEventElapsedTime(&ms, c->ev0, c->ev1), "cudaEventElapsedTime");
        out->kernel_ms = ms;
        if (herr[0] != 0) {
            const long long pid = (long long)herr[1] | ((long long)herr[2] << 31);
            char msg[160];
            std::snprintf(msg, sizeof msg, "particle %lld: %s", pid,
                          herr[0] == BTE_ERR_VALUE ? "invalid scattering rate"
                          : herr[0] == BTE_ERR_LIMIT ? "iteration cap reached"
                          : herr[0] == BTE_ERR_CHECK ? "index check failed"
                                                      : "geometry error");
            throw Error(bte_status(herr[0]), msg);
        }
        if (nloc > 0) {  // the tally stays on the device for bte_get_spectral
            if (replay) bte::spec_from_exact(c, spec_vals);
            c->spec_unit = grid_run || link_run ? A.fx.per_tick() : 1.;
            c->spec_nbins = nbins;
            c->spec_T0 = p->T0;
            c->spec_Eeff = Eeff;
            c->spec_steady = false;
            c->spec_valid = true;
        }
        if (ngroups > 1) {  // the groups' tallies stay on the device
            c->group_n = ngroups;
            c->group_nbx = nbx;
            c->group_nbins = nbins;
            c->group_Eeff = Eeff;
            c->group_step = step;
            c->group_params = *p;
            c->group_units = units;
            c->group_valid = true;
        }
        if (replay) {  // raw tallies
            std::vector<double> gz(nk), jx(nk), jy(nk);
            for (std::size_t k = 0; k < nk; ++k) {
                double* dst[3] = {&gz[k], &jx[k], &jy[k]};
                for (int q = 0; q < 3; ++q) {
                    const unsigned long long hi = hex[6 * k + 2 * q], lo = hex[6 * k + 2 * q + 1];
                    const __int128 v = (__int128)(((unsigned __int128)hi << 64) | lo);
                    *dst[q] = double(v) / bte::FIX_SCALE;
                }
            }
            if (out->exact) std::memcpy(out->exact, hex.data(), nk * 6 * sizeof(long long));
            if (out->gz) std::copy(gz.begin(), gz.end(), out->gz);
            if (out->gz_jx) std::copy(jx.begin(), jx.end(), out->gz_jx);
            if (out->gz_jy) std::copy(jy.begin(), jy.end(), out->gz_jy);
            bte::rta_post(c, p, nbx, nbins, Eeff, step, gz, jx, jy, out);
        }
        out->nboxes = nbx;
        out->nbins = nbins;
        out->Eeff = Eeff;
        out->energy_rate = c->gens.total_energy;
        out->events = (int64_t)hc[0];
        out->wall_hits = (int64_t)hc[1];
        out->crossings = (int64_t)hc[2];
        out->absorbed = (int64_t)hc[3];
        out->specular_hits = (int64_t)hc[4];
        out->tally_updates = (int64_t)hc[7];
        out->translations = (int64_t)hc[8];
        out->interface_hits = (int64_t)hc[11];
        out->interface_transmissions = (int64_t)hc[12];
        return BTE_OK;
    } catch (const Error& e) {
        return fail(c, e);
    } catch (const std::exception& e) {
        c->err = e.what();
        return BTE_ERR_CUDA;
    }
}

// ------------------------------------------------------------------ debug
// Host-only views of the tables for the CPU tests (no GPU needed).

long long btegpu_debug_geometry(const bte_geometry* gm, double* out, long long cap) {
    try {
        bte::HostGeometry g = bte::build_geometry(gm);
        long long k = 0;
        auto put = [&](double x) {
            if (k < cap) out[k] = x;
            k++;
        };
        for (std::size_t b = 0; b < g.boxes.size(); ++b) {
            const bte::GBox& B = g.boxes[b];
            put(double(B.nborders));
            for (int i = 0; i < B.nborders; ++i) {
                const bte::GBorder& br = g.borders[std::size_t(B.border_off + i)];
                put(br.p1.x); put(br.p1.y); put(br.p2.x); put(br.p2.y);
                put(br.np.x); put(br.np.y);
            }
            put(double(B.ncontacts));
            for (int i = 0; i < B.ncontacts; ++i) {
                const bte::GContact& ct = g.contacts[std::size_t(B.contact_off + i)];
                put(double(ct.id)); put(ct.np.x); put(ct.np.y);
            }
            put(B.center.x); put(B.center.y); put(B.area);
        }
        return k;
    } catch (const std::exception&) {
        return -1;
    }
}

int btegpu_debug_grid(const bte_geometry* gm, int* nx, int* ny) {
    try {
        bte::HostGeometry g = bte::build_geometry(gm);
        *nx = g.gnx;
        *ny = g.gny;
        return g.rect_grid ? 1 : 0;
    } catch (const std::exception&) {
        return -1;
    }
}

long long btegpu_debug_lambert(const bte_mode_table* mt, const bte_geometry* gm, long long* nnz_per_class,
                               int maxclass) {
    try {
        bte::HostModes m = bte::build_modes(mt);
        bte::HostGeometry g = bte::build_geometry(gm);
        bte::LambertTable L = bte::build_lambert(m, g, hw_threads());
        const std::size_t n = m.n();
        for (int c = 0; c < L.nclass && c < maxclass; ++c)
            nnz_per_class[c] = L.row_ptr[std::size_t(c) * (n + 1) + n] - L.row_ptr[std::size_t(c) * (n + 1)];
        return (long long)L.col.size();
    } catch (const std::exception&) {
        return -1;
    }
}

long long btegpu_debug_frame(double time, double Eeff, const double* temps, const int* H, int nboxes,
                             int nmodes, char* out, long long cap) {
    std::vector<double> t(temps, temps + nboxes);
    const std::string f = bte::berta_frame(time, Eeff, t, H, std::size_t(nboxes), std::size_t(nmodes));
    if ((long long)f.size() <= cap) std::memcpy(out, f.data(), f.size());
    return (long long)f.size();
}

long long btegpu_debug_links(const bte_geometry* gm, double* lines, int* out, long long cap) {
    try {
        const bte::LinkGrid L = bte::build_link_grid(bte::build_geometry(gm));
        if (!L.ok) return 0;
        const long long n = (long long)L.nx * L.ny;
        if (cap < n) return -n;
        out[0] = L.nx;
        out[1] = L.ny;
        std::copy(L.gx.begin(), L.gx.end(), lines);
        std::copy(L.gy.begin(), L.gy.end(), lines + L.gx.size());
        for (long long k = 0; k < 4 * n; ++k) {
            out[2 + 4 * k] = L.side[std::size_t(k)].cell;
            out[3 + 4 * k] = L.side[std::size_t(k)].box;
            out[4 + 4 * k] = L.side[std::size_t(k)].flags;
            out[5 + 4 * k] = L.cycle[std::size_t(k)];
        }
        return n;
    } catch (const std::exception&) {
        return 0;
    }
}

long long btegpu_debug_fixwalk(const double* gx, int nx, const double* gy, int ny, double vmax, double step,
                               int nbins, double px, double py, long long nflights, const float* e,
                               const double* tau, const double* vx, const double* vy, int* scales, long long* out,
                               long long cap) {
    const bte::FixScale f = bte::choose_scale(gx[0], gx[nx], gy[0], gy[ny], vmax, step);
    scales[0] = f.kx;
    scales[1] = f.kt;
    scales[2] = f.sub;
    auto line = [&](const double* g, int k, double o) { return bte::fix_round(g[k] - o, f.kx); };
    int i = 0, j = 0;
    while (i + 1 < nx && px >= gx[i + 1]) ++i;
    while (j + 1 < ny && py >= gy[j + 1]) ++j;
    int64_t x = bte::fix_round(px - f.x0, f.kx), y = bte::fix_round(py - f.y0, f.kx);
    const uint64_t w = uint64_t(bte::fix_round(step, f.kt - f.sub));
    uint64_t rb = w;
    long long part = 0, m = 0;
    for (long long k = 0; k < nflights; ++k) {
        bte::ModeFix v;
        bte::fix_velocity(vx[k], f, v.vx, v.rx);
        bte::fix_velocity(vy[k], f, v.vy, v.ry);
        const bool ux = !(v.vx & bte::FIX_DOWN), uy = !(v.vy & bte::FIX_DOWN);
        uint32_t hi;
        uint64_t lo = bte::fix_flight(e[k], tau[k], f.kt, hi);
        for (;;) {
            const uint64_t ax = uint64_t(ux ? line(gx, i + 1, f.x0) - x : x - line(gx, i, f.x0));
            const uint64_t ay = uint64_t(uy ? line(gy, j + 1, f.y0) - y : y - line(gy, j, f.y0));
            const bte::FixSeg q = bte::fix_segment(ax, ay, v, lo, hi, rb);
            hi -= lo < q.seg ? 1u : 0u;
            lo -= q.seg;
            rb -= q.seg;
            x += ux ? int64_t(q.dx) : -int64_t(q.dx);
            y += uy ? int64_t(q.dy) : -int64_t(q.dy);
            const int kind = (q.cross_x ? 1 : 0) | (q.cross_y ? 2 : 0) | (q.flight_end ? 4 : 0) | (q.bin_end ? 8 : 0);
            if (m < cap) {
                long long* o = out + 5 * m;
                o[0] = k;
                o[1] = kind;
                o[2] = x;
                o[3] = y;
                o[4] = (long long)q.seg;
            }
            ++m;
            if (q.bin_end) {
                if (++part >= ((long long)nbins << f.sub)) return m;
                rb = w;
            }
            if (q.cross_x) i += ux ? 1 : -1;
            if (q.cross_y) j += uy ? 1 : -1;
            if (i < 0 || j < 0 || i >= nx || j >= ny) return m;
            if (q.flight_end) break;
        }
    }
    return m;
}

int btegpu_debug_keyed(const int* keys, const int* fails, int n, int* filled) {
    bte::Keyed<int> k;
    for (int i = 0; i < n; ++i) {
        filled[i] = 0;
        try {
            k.update(keys[i], [&](int) {
                filled[i] = 1;
                if (fails[i]) throw Error(BTE_ERR_CUDA, "fill");
            });
        } catch (const Error&) {
        }
    }
    return k.valid ? 1 : 0;
}

int btegpu_debug_log(const double* x, double* y, long long n) {
    for (long long i = 0; i < n; ++i) y[i] = bte::bte_log(x[i]);
    return 0;
}

}  // extern "C"

// ------------------------------------------------------------------ prepared runs
// Read-only view of a context whose tables an earlier bte_rta_run built for
// the same parameters: fills the kernel arguments without allocating or
// uploading anything.  Used by the allocation-free entry point (noalloc.cu).
namespace bte {

bte_status prepared_grid_run(bte_ctx* c, const bte_rta_params* p, PreparedRun* r, std::string* why) {
    if (!c || !p || !r) {
        *why = "null argument";
        return BTE_ERR_INPUT;
    }
    if (p->mode != BTE_MODE_PRODUCTION) {
        *why = "the allocation-free run is the production grid kernel: mode must be BTE_MODE_PRODUCTION";
        return BTE_ERR_INPUT;
    }
    if (!(p->dt > 0.) || !(p->maxtime > 0.) || p->nparticles < 1 ||
        !(p->specularity >= 0. && p->specularity <= 1.) || !(p->T0 > 0.)) {
        *why = "invalid run parameters";
        return BTE_ERR_INPUT;
    }
    if (!c->have_modes || !c->have_geom || !c->modes_dev || !c->geom_dev || !c->lambert_dev) {
        *why = "context not prepared: load the tables and run bte_rta_run once with these parameters";
        return BTE_ERR_STATE;
    }
    const HostGeometry& g = c->geom;
    const HostModes& m = c->modes;
    if (!g.rect_grid) {
        *why = "the allocation-free run needs boxes that tile an axis-aligned grid";
        return BTE_ERR_INPUT;
    }
    if (c->ncrys > 0 && c->ndmm > 0) {  // (the grid kernel knows no interfaces)
        *why = "the allocation-free run takes no interfaces between crystals";
        return BTE_ERR_INPUT;
    }
    if (c->resample_T0 != (c->nmat > 0 ? -2.0 : p->T0) || c->gen_key_source != p->source ||
        (p->source == BTE_SOURCE_INITIAL &&
         (c->gen_key_n != p->nparticles || c->gen_key_seed != p->seed))) {
        *why = "context prepared for other parameters: run bte_rta_run once with this T0, source "
               "(and, for the initial source, N and seed) first";
        return BTE_ERR_STATE;
    }
    if (p->specularity > 0. && !c->have_mirror) {
        *why = "specular walls need an axis-aligned q grid with mirror images";
        return BTE_ERR_INPUT;
    }
    const std::size_t ntime = std::size_t(std::floor(p->maxtime / p->dt + 1.0e-6)) + 1;
    if (ntime < 2) {
        *why = "maxtime shorter than one time bin";
        return BTE_ERR_INPUT;
    }
    r->ntime = int(ntime);
    r->nbins = int(ntime - 1);
    r->maxtime = double(ntime - 1) * p->dt;
    r->step = (r->maxtime - 0.0) / double(ntime - 1);
    r->nboxes = int(g.boxes.size());
    long long total;
    if (p->source == BTE_SOURCE_WALLS) {
        r->Eeff = c->gens.total_energy / double(p->nparticles);
        total = p->nparticles;
    } else {
        r->Eeff = c->gen_Eeff;
        total = c->gens.init_first.back();
    }
    r->energy = c->gens.total_energy;
    long long pbeg = std::max<long long>(0, p->particle_begin);
    long long pend = p->particle_end > 0 ? std::min<long long>(p->particle_end, total) : total;
    if (pend < pbeg) pend = pbeg;
    DevTables& T = r->T;
    T = DevTables{};
    T.n = int(m.n());
    T.nb = m.nb;
    T.vxc = c->d_vxc.as<double>();
    T.vyc = c->d_vyc.as<double>();
    T.w = c->d_w.as<double>();
    T.tau = c->d_tau.as<double>();
    T.resample_cdf = c->d_rcdf.as<double>();
    T.resample = c->d_resample.as<int2>();
    T.nboxes = r->nboxes;
    T.boxes = c->d_boxes.as<GBox>();
    T.hull = c->d_hull.as<V2>();
    T.borders = c->d_borders.as<GBorder>();
    T.contacts = c->d_contacts.as<GContact>();
    T.cseg = c->d_cseg.as<V2>();
    T.translation = c->d_transl.as<V2>();
    T.tfast = c->have_tfast ? c->d_tfast.as<TransFast>() : nullptr;
    T.tfast_rng = c->d_tfast_rng.as<int2>();
    T.tfast_u = c->d_tfast_u.as<V2>();
    T.nclass = c->nclass;
    T.row_ptr = c->d_row_ptr.as<long long>();
    T.lcol = c->d_lcol.as<int>();
    T.lcdf = c->d_lcdf.as<double>();
    T.lrow = c->d_lrow.as<unsigned long long>();
    T.lalias = c->d_lalias.as<int4>();
    T.mirror = c->have_mirror ? c->d_mirror.as<int>() : nullptr;
    T.box_mat = c->nmat > 0 ? c->d_boxmat.as<int>() : nullptr;
    set_crystal_tables(c, T);
    T.rkey = c->d_rkey.as<bte::RectKey>();
    T.eps = c->d_eps.as<bte::V2>();
    T.ntime = r->ntime;
    T.timegrid = nullptr;  // set by the caller
    T.maxtime = r->maxtime;
    T.inv_dt = 1.0 / r->step;
    T.source = p->source;
    T.ngen = p->source == BTE_SOURCE_WALLS ? int(c->gens.walls.size()) : int(c->gens.init_box.size());
    T.gen_cdf = c->d_gcdf.as<double>();
    T.gen_prob = c->d_gprob.as<float>();
    T.gen_alt = c->d_galt.as<int>();
    T.walls = c->d_walls.as<WallGenDev>();
    T.wall_cum = c->d_wcum.as<double>();
    T.init_first = c->d_ifirst.as<long long>();
    T.init_box = c->d_ibox.as<int>();
    T.init_sign = c->d_isign.as<int>();
    T.seed = p->seed;
    T.flight_cap = p->flight_cap > 0 ? p->flight_cap : EVENT_CAP;
    T.checks = (p->flags & BTE_FLAG_CHECKS) ? 1 : 0;
    T.ballistic = p->ballistic;
    T.specularity = p->specularity;
    T.pbegin = pbeg;
    T.pend = pend;
    T.nbins = r->nbins;
    r->A = GridArgs{};
    try {
        ck(cudaSetDevice(c->device), "cudaSetDevice");
        prepare_fixed(c, r->step, r->A);
    } catch (const Error& e) {
        *why = e.what();
        return e.code;
    }
    r->stream = c->stream;
    r->ev0 = c->ev0;
    r->ev1 = c->ev1;
    r->device = c->device;
    r->nsm = c->nsm;
    r->tune = c->tune;
    return BTE_OK;
}

// Scales of the integer walk (fixed_walk.cuh): a bin below 2^61 ticks, the
// domain below 2^62 units, and the fastest velocity below 2^63 units per
// 2^64 ticks, which costs the positions at most seven bits once a bin (or its
// 2^sub parts) is no longer than eight flights across the domain.  A part's end
// is a pass and a flush like a bin's.  It has not been seen to cost what the
// walk in doubles did, which took any bin in one piece: 3e5 particles, bins of 4
// ns, a ribbon of 1000 x 100 nm 5.2 ms (in doubles 7.8), 100 x 100 nm 0.49 (2.7),
// 20 x 20 nm 0.24 (2.5), a closed pore of 200 x 100 nm at bins of 1 ns 3.0 (12.1),
// a periodic bar of 20 x 40 nm 0.43 (3.3).
FixScale choose_scale(double x0, double x1, double y0, double y1, double vmax, double step) {
    FixScale f{};
    f.x0 = x0;
    f.y0 = y0;
    const double ext = std::max(x1 - x0, y1 - y0);
    double w = step * (1.0 + 0x1p-20);  // no bin is longer (they differ by rounding)
    while (vmax * w > 8.0 * ext && f.sub < 24) {
        w *= 0.5;
        ++f.sub;
    }
    f.kt = 60 - std::ilogb(w);
    f.kx = 61 - std::ilogb(ext);
    if (vmax > 0.) f.kx = std::min(f.kx, f.kt - 2 - std::ilogb(vmax));
    return f;
}

void fix_on_device(bte_ctx* c, const FixScale& f);

void prepare_fixed(bte_ctx* c, double step, GridArgs& A) {
    const HostGeometry& g = c->geom;
    A.G.nx = g.gnx;
    A.G.ny = g.gny;
    A.G.gx = c->d_gx.as<double>();
    A.G.gy = c->d_gy.as<double>();
    A.G.cell = c->d_gcell.as<int>();
    A.boxcell = c->d_boxcell.as<int2>();
    A.mv = c->d_mv.as<ModeVel>();
    A.mf = c->d_mf.as<ModeFix>();
    A.gxf = c->d_gxf.as<long long>();
    A.gyf = c->d_gyf.as<long long>();
    A.wxf = c->d_wxf.as<unsigned long long>();
    A.wyf = c->d_wyf.as<unsigned long long>();
    A.map = c->d_map.as<int>();
    A.fx = choose_scale(g.gx.front(), g.gx.back(), g.gy.front(), g.gy.back(), c->vmax, step);
    const V2 want[4] = {v2(1, 0), v2(-1, 0), v2(0, 1), v2(0, -1)};
    for (int w = 0; w < 4; ++w) {
        A.cls[w] = -1;
        for (std::size_t k = 0; k < g.normals.size(); ++k)
            if (g.normals[k].x == want[w].x && g.normals[k].y == want[w].y) A.cls[w] = int(k);
    }
    // Generating a particle is a long divergent block with FP64 draws: where
    // particles are absorbed soon (walls), a warp waits for four idle lanes
    // (1e6 particles, 61 flights each: 3.36 ms with one, 3.19 two, 3.14 four,
    // 3.27 eight); an initial deviation keeps its particles to the end (1800
    // flights each: 112.1 ms with one, 114.6 four).
    A.refill = c->gen_key_source == BTE_SOURCE_WALLS ? 4 : 1;
    fix_on_device(c, A.fx);
}

void prepare_link(bte_ctx* c, double step, LinkArgs& A) {
    const LinkGrid& L = c->link;
    A.mf = c->d_mf.as<ModeFix>();
    A.gxf = c->d_gxf.as<long long>();
    A.gyf = c->d_gyf.as<long long>();
    A.wxf = c->d_wxf.as<unsigned long long>();
    A.wyf = c->d_wyf.as<unsigned long long>();
    A.ny = L.ny;
    A.side = c->d_lside.as<int4>();
    A.range = c->d_lrange.as<int4>();
    A.per = c->d_lper.as<unsigned char>();
    A.cellbox = c->d_lbox.as<int>();
    A.cycle = c->d_lcycle.as<int4>();
    A.pbox = c->link_corner ? c->d_lpbox.as<int>() : nullptr;
    A.dmm_row = c->d_dmm_row.as<long long>();
    A.dmm_ent = c->d_dmm_ent.as<DmmEnt>();
    // (as in prepare_fixed; generation on convex boxes costs more: the bar's
    // particles live five flights, 3.63 ms with one idle lane, 2.17 four, 1.89
    // eight, 1.84 sixteen; the crystals' 25, 1.07, 0.80, 0.77, 0.82)
    A.refill = c->gen_key_source == BTE_SOURCE_WALLS ? 8 : 1;
    A.fx = choose_scale(L.gx.front(), L.gx.back(), L.gy.front(), L.gy.back(), c->vmax, step);
    A.margin = (unsigned long long)std::llrint(std::ldexp(2.0e-6, A.fx.kx));
    fix_on_device(c, A.fx);
}

// The integer tables for the scales f, unless they are on the device already.
void fix_on_device(bte_ctx* c, const FixScale& f) {
    const bool rect = c->geom.rect_grid;
    DevGrid G{};
    G.nx = rect ? c->geom.gnx : c->link.nx;
    G.ny = rect ? c->geom.gny : c->link.ny;
    G.gx = c->d_gx.as<double>();
    G.gy = c->d_gy.as<double>();
    if (c->fix_dev && c->fix.x0 == f.x0 && c->fix.y0 == f.y0 && c->fix.kx == f.kx && c->fix.kt == f.kt) return;
    launch_fix_tables(f, c->d_mv.as<ModeVel>(), int(c->modes.n()), c->d_mf.as<ModeFix>(), G, c->d_gxf.as<long long>(),
                      c->d_gyf.as<long long>(), c->d_wxf.as<long long>(), c->d_wyf.as<long long>(), c->stream);
    ck(cudaGetLastError(), "integer tables launch");
    c->fix = f;
    c->fix_dev = true;
}

void upload_time_grid(bte_ctx* c, int ntime, double maxtime, double step, int tick_exp) {
    c->time.update(TimeKey{ntime, tick_exp, maxtime, step}, [&](const TimeKey&) {
        c->h_time = time_grid_with_widths(ntime, maxtime, step, tick_exp);  // (stays until the copy is done)
        c->d_time.upload(c->h_time, c->stream);
    });
}

std::vector<double> time_grid_with_widths(int ntime, double maxtime, double step, int tick_exp) {
    std::vector<double> g(std::size_t(3 * ntime - 2));
    for (int i = 0; i < ntime; ++i) g[std::size_t(i)] = (i == ntime - 1) ? maxtime : 0.0 + double(i) * step;
    for (int i = 0; i + 1 < ntime; ++i) {
        const double w = g[std::size_t(i + 1)] - g[std::size_t(i)];
        g[std::size_t(ntime + i)] = w;
        g[std::size_t(2 * ntime - 1 + i)] = bitsd(uint64_t(std::llrint(std::ldexp(w, tick_exp))));
    }
    return g;
}

void upload_spectral_locations(bte_ctx* c) {
    std::vector<int>& loc = c->h_specloc;  // (stays until the copy is done)
    loc.assign(c->geom.boxes.size(), -1);
    for (std::size_t i = 0; i < c->spec_boxes.size(); ++i) {
        const std::size_t b = std::size_t(c->spec_boxes[i]);  // (of the geometry of bte_set_spectral)
        if (b >= loc.size()) throw Error(BTE_ERR_INPUT, "spectral location is not a box of the loaded geometry");
        loc[b] = int(i);
    }
    c->d_specloc.upload(loc, c->stream);
}

// A replay run's 128-bit per-mode tally in c->d_spec, replaced by its values
// as doubles.
void spec_from_exact(bte_ctx* c, std::size_t vals) {
    std::vector<unsigned long long> h(2 * vals);
    std::vector<double> v(vals);
    ck(cudaMemcpyAsync(h.data(), c->d_spec.p, h.size() * sizeof(h[0]), cudaMemcpyDeviceToHost, c->stream), "d2h");
    sync(c);
    for (std::size_t i = 0; i < vals; ++i)
        v[i] = double((__int128)(((unsigned __int128)h[2 * i] << 64) | h[2 * i + 1])) / FIX_SCALE;
    c->d_spec.upload(v, c->stream);
    sync(c);
}

void fill_static_tables(bte_ctx* c, DevTables& T) {
    T.n = int(c->modes.n());
    T.nb = c->modes.nb;
    T.vxc = c->d_vxc.as<double>();
    T.vyc = c->d_vyc.as<double>();
    T.w = c->d_w.as<double>();
    T.tau = c->d_tau.as<double>();
    T.resample_cdf = c->d_rcdf.as<double>();
    T.resample = c->d_resample.as<int2>();
    T.nboxes = int(c->geom.boxes.size());
    T.boxes = c->d_boxes.as<GBox>();
    T.hull = c->d_hull.as<V2>();
    T.borders = c->d_borders.as<GBorder>();
    T.contacts = c->d_contacts.as<GContact>();
    T.cseg = c->d_cseg.as<V2>();
    T.translation = c->d_transl.as<V2>();
    T.tfast = c->have_tfast ? c->d_tfast.as<TransFast>() : nullptr;
    T.tfast_rng = c->d_tfast_rng.as<int2>();
    T.tfast_u = c->d_tfast_u.as<V2>();
    T.nclass = c->nclass;
    T.row_ptr = c->d_row_ptr.as<long long>();
    T.lcol = c->d_lcol.as<int>();
    T.lcdf = c->d_lcdf.as<double>();
    T.lrow = c->d_lrow.as<unsigned long long>();
    T.lalias = c->d_lalias.as<int4>();
    T.mirror = c->have_mirror ? c->d_mirror.as<int>() : nullptr;
    T.box_mat = c->nmat > 0 ? c->d_boxmat.as<int>() : nullptr;
    set_crystal_tables(c, T);
    T.rkey = c->d_rkey.as<bte::RectKey>();
    T.eps = c->d_eps.as<bte::V2>();
}

// The interface tables of crystals joined by mismatch interfaces (null
// with one crystal).
void set_crystal_tables(const bte_ctx* c, DevTables& T) {
    const bool crys = c->ncrys > 0 && c->dmm_dev;
    T.contact_dmm = crys ? c->d_cdmm.as<int>() : nullptr;
    T.dmm_row = crys ? c->d_dmm_row.as<long long>() : nullptr;
    T.dmm_ent = crys ? c->d_dmm_ent.as<DmmEnt>() : nullptr;
    T.crys_off = crys ? c->d_crysoff.as<int>() : nullptr;
}

double crystal_thickness(const bte_ctx* c, int k) {
    return c->crys_thick.empty() ? c->geom.thickness : c->crys_thick[std::size_t(k)];
}

double box_thickness(const bte_ctx* c, int b) {
    return c->ncrys > 0 ? crystal_thickness(c, c->geom.mat[std::size_t(b)]) : c->geom.thickness;
}

double box_T0(const bte_ctx* c, int b, double T0) {
    return c->nmat > 0 ? c->mat_T0[std::size_t(c->geom.mat[std::size_t(b)])] : T0;
}

void set_ctx_error(bte_ctx* c, const std::string& m) {
    if (c) c->err = m;
}

}  // namespace bte
