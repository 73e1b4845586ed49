"""The linked cells that the production kernels walk on rectangular boxes off
a grid (build_link_grid) against the boxes themselves: what a point just
across each side of each cell lies in, translated where that is a periodic
box."""
import numpy as np
import pytest

import btegpu
import synth

VOID, RESERVOIR, TRANSLATE, INNER = 1, 2, 4, 8


def _offset_blocks():
    """Two reservoirs over a row of blocks whose edges do not line up."""
    b = [synth._rect(0, 0, 10, 6), synth._rect(10, 0, 25, 6), synth._rect(0, 6, 16, 9), synth._rect(16, 6, 25, 9),
         synth._rect(-2, -3, 27, 0), synth._rect(0, 9, 25, 12)]
    return synth._pack(b, [300.0] * 4 + [301.0, 299.0], [300.0] * 4 + [301.0, 299.0], [0] * 4 + [1, 1], 0.335)


def _crystals():
    g = synth.ribbon_geometry(200.0, 50.0, 10)
    g["material"] = np.array([0] * 5 + [1] * 5 + [0, 1], dtype=np.int32)
    return g


GEOMS = {"bar": synth.periodic_bar_geometry(), "layered": synth.layered_bar_geometry(),
         "cell": synth.periodic_cell_geometry(37.5, 20.3, 3, 2), "ribbon": synth.periodic_ribbon_geometry(45.5, 57.3, 3, 3),
         "pulse": synth.pulse_geometry(), "blocks": _offset_blocks(), "crystals": _crystals(),
         "pore": synth.grid_geometry(200.0, 100.0, 10, 5, pore_center=(100.0, 50.0), pore_diameter=50.0)}


@pytest.mark.parametrize("name", sorted(GEOMS))
def test_links_name_what_lies_across(name):
    g = GEOMS[name]
    gx, gy, side, cycle = btegpu.debug_links(g)
    v = np.asarray(g["vertices"]).reshape(-1, 4, 2)
    lo, hi = v.min(axis=1), v.max(axis=1)
    tto = np.asarray(g.get("translate_to", np.full(len(v), -1)))
    tr = np.asarray(g.get("translation", np.zeros((len(v), 2))))
    mat = np.asarray(g.get("material", np.zeros(len(v), dtype=int)))

    def box_of(p):
        hit = np.flatnonzero(((lo < p) & (p < hi)).all(axis=1))
        return int(hit[0]) if hit.size else -1

    nx, ny, eps, seen = len(gx) - 1, len(gy) - 1, 1e-6, 0
    for i in range(nx):
        for j in range(ny):
            mid = np.array([(gx[i] + gx[i + 1]) / 2, (gy[j] + gy[j + 1]) / 2])
            a = box_of(mid)
            if a < 0 or g["reservoir"][a] or tto[a] >= 0:
                continue
            for s, (ex, ey) in enumerate(((1, 0), (-1, 0), (0, 1), (0, -1))):
                p = mid.copy()
                if ex:
                    p[0] = (gx[i + 1] if ex > 0 else gx[i]) + ex * eps
                else:
                    p[1] = (gy[j + 1] if ey > 0 else gy[j]) + ey * eps
                b, (cell, box, flags) = box_of(p), side[i * ny + j][s]
                seen += 1
                if b < 0:
                    assert flags == VOID
                    continue
                assert (flags >> 8 != 0) == (mat[a] != mat[b])
                kind = flags & 255
                if b == a:
                    assert kind == INNER
                elif g["reservoir"][b]:
                    assert kind == RESERVOIR and box == b
                    continue
                elif tto[b] >= 0:
                    assert kind == TRANSLATE
                    p = p + tr[b]
                    b = box_of(p)
                else:
                    assert kind == 0
                ci, cj = divmod(int(cell), ny)
                assert box == b and gx[ci] < p[0] < gx[ci + 1] and gy[cj] < p[1] < gy[cj + 1]
            # a period leads back to its first cell through the last one's side
            for ax in (0, 1):
                f, l = cycle[i * ny + j][2 * ax:2 * ax + 2]
                if f < 0:
                    continue
                c = (l * ny + j) if ax == 0 else (i * ny + l)
                back = side[c][2 * ax]
                assert f <= (i, j)[ax] <= l and back[2] & 255 == TRANSLATE
                assert back[0] == ((f * ny + j) if ax == 0 else (i * ny + f))
    assert seen > 4
    want = {"bar": (True, False), "cell": (True, True), "ribbon": (True, False), "pulse": (True, True)}.get(name)
    if want:
        assert ((cycle[:, 0] >= 0).any(), (cycle[:, 2] >= 0).any()) == want


def test_other_shapes_are_not_linked():
    """A box that is no rectangle, and a translation that lands between boxes."""
    g = synth.periodic_bar_geometry()
    tri = dict(g, npoints=np.array([3] + list(g["npoints"][1:]), dtype=np.int32),
               vertices=np.concatenate([g["vertices"][:6], g["vertices"][8:]]))
    assert btegpu.debug_links(tri) is None
    off = dict(g, translation=np.asarray(g["translation"]) * 0.9)
    assert btegpu.debug_links(off) is None
