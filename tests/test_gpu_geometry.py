"""GPU voxelizer parity: the packed geometry and boundary list equal the binary64
restatement of src/geometry/voxelize.ts + wall-links.ts bit for bit, with the
halfway fractions of linkFractions: false and with measured link fractions
(triangle-bins.ts), on the reference's own test meshes and on the benchmark
bodies."""
import numpy as np
import pytest

from oracle import oracle as O
from pocketwind_gb300 import meshes
from tests.shapes import box

pytestmark = pytest.mark.gpu


def _both(body, supports, layout, floor, link_fractions=False):
    from pocketwind_gb300.geometry import voxelize
    g = voxelize(body, supports, layout, floor, link_fractions=link_fractions)
    r = O.voxelize(body.positions, None if supports is None else supports.positions, layout, floor,
                   link_fractions=link_fractions)
    return g, r


CASES = [
    ("icosphere r20", lambda: (meshes.icosphere((32, 32, 32), 20), None), (64, 64, 64), False),
    ("cube 8000", lambda: (box([20.2] * 3, [40.2] * 3), None), (64, 64, 64), False),
    ("open cube", lambda: (box([20.2] * 3, [40.2] * 3, True), None), (64, 64, 64), False),
    ("thin plate", lambda: (box([20.2] * 3, [20.5, 40.2, 40.2]), None), (64, 64, 64), False),
    ("body and support", lambda: (box([20.2] * 3, [24.2] * 3), box([22.2, 22.2, 18.2], [26.2, 26.2, 22.2])),
     (64, 64, 64), False),
    ("floor corners", lambda: (box([20.25] * 3, [24.25] * 3), box([30.25] * 3, [34.25] * 3)), (64, 64, 64), True),
    ("sphere case 96x48x48", lambda: (meshes.icosphere((24, 24, 24), 6, 4), None), (96, 48, 48), False),
    ("vehicle case 128x64x64", lambda: (meshes.vehicle_case_mesh(128, 64), None), (128, 64, 64), True),
    ("ahmed preset with stilts", lambda: meshes.place_mesh(meshes.ahmed_mesh(), 128, 64, 64, 48, True,
                                                           meshes.stilts_mesh()), (128, 64, 64), True),
    ("empty tunnel", lambda: (meshes.Mesh(np.zeros(0, np.float32), 0), None), (16, 8, 8), True),
]


@pytest.mark.parametrize("measure", [False, True], ids=["halfway", "measured"])
@pytest.mark.parametrize("name,make,layout,floor", CASES, ids=[c[0] for c in CASES])
def test_voxelizer_bit_exact(name, make, layout, floor, measure):
    body, supports = make()
    g, r = _both(body, supports, layout, floor, measure)
    assert np.array_equal(g.geometry, r.geometry)
    assert g.missed_links == r.missed_links
    assert np.array_equal(g.boundary_cells, r.boundary_cells)
    assert (g.solid_cells, g.frontal_cells, g.watertight) == (r.solid_cells, r.frontal_cells, r.watertight)
    assert g.blockage == r.blockage


def test_voxelizer_rejects_invalid_inputs():
    from pocketwind_gb300._lib import RangeError
    from pocketwind_gb300.geometry import voxelize
    mesh = box([20] * 3, [24] * 3)
    with pytest.raises(RangeError):
        voxelize(mesh, None, (1, 64, 64), False)
    bad = mesh.positions.copy()
    bad[0] = np.nan
    with pytest.raises(RangeError):
        voxelize(mesh, meshes.Mesh(bad, mesh.triangle_count), (64, 64, 64), False)


def test_winding_invariance_on_gpu():
    from pocketwind_gb300.geometry import voxelize
    mesh = box([20] * 3, [24] * 3)
    rev = mesh.positions.reshape(-1, 3, 3)[:, [0, 2, 1], :].reshape(-1).copy()
    a = voxelize(mesh, None, (64, 64, 64), False)
    b = voxelize(meshes.Mesh(rev, mesh.triangle_count), None, (64, 64, 64), False)
    assert a.solid_cells == 64 and np.array_equal(a.geometry, b.geometry)


# triangle counts around the warp's 32 (few triangles: their pixels split over many
# warps), boxes of many pixels and of none, a grid that is odd in every direction
@pytest.mark.parametrize("floor", [False, True])
@pytest.mark.parametrize("name,make", [
    ("12 large", lambda: box([3.2, 4.7, 2.9], [30.1, 25.3, 19.8])),
    ("20", lambda: meshes.icosphere((15.3, 14.1, 11.2), 8.7, 0)),
    ("32", lambda: meshes.icosphere((15.3, 14.1, 11.2), 8.7, 0, 4)),
    ("35", lambda: meshes.icosphere((15.3, 14.1, 11.2), 8.7, 0, 5)),
    ("1280", lambda: meshes.icosphere((15.3, 14.1, 11.2), 8.7, 3)),
    ("outside", lambda: box([-9.5, -3.5, 30.2], [60.5, 2.5, 44.1])),
])
def test_voxelizer_triangle_groups(name, make, floor):
    g, r = _both(make(), None, (37, 29, 23), floor)
    assert np.array_equal(g.geometry, r.geometry)
    assert np.array_equal(g.boundary_cells, r.boundary_cells)
    assert (g.solid_cells, g.frontal_cells, g.watertight) == (r.solid_cells, r.frontal_cells, r.watertight)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 8, -1])
def test_voxelizer_rejects_non_finite_body(value, at):
    from pocketwind_gb300._lib import RangeError
    from pocketwind_gb300.geometry import voxelize
    bad = meshes.icosphere((16, 16, 16), 8, 1).positions.copy()
    bad[at] = value
    with pytest.raises(RangeError):
        voxelize(bad, None, (32, 32, 32), False)


# measured fractions: bins of many triangles (several queue flushes a link), of few,
# a body across the periodic y seam, one without supports' triangles
@pytest.mark.parametrize("name,make,layout,floor", [
    ("dense", lambda: (meshes.icosphere((15.3, 14.1, 11.2), 3.3, 4), None), (37, 29, 23), False),
    ("coarse", lambda: (box([3.2, 4.7, 2.9], [30.1, 25.3, 19.8]), None), (37, 29, 23), True),
    ("seam", lambda: (meshes.icosphere((15.3, 0.4, 11.2), 4.6, 3), None), (37, 29, 23), False),
    ("supports", lambda: (meshes.icosphere((15.3, 14.1, 11.2), 4.6, 3), box([13, 12, 0.6], [17, 16, 8.2])),
     (37, 29, 23), True),
    ("no support triangles", lambda: (meshes.icosphere((15.3, 14.1, 11.2), 4.6, 2),
                                      meshes.Mesh(np.zeros(0, np.float32), 0)), (37, 29, 23), False),
])
def test_link_fraction_groups(name, make, layout, floor):
    body, supports = make()
    g, r = _both(body, supports, layout, floor, True)
    assert np.array_equal(g.geometry, r.geometry)
    assert g.missed_links == r.missed_links


# a triangle before the body's wall that the link from cell (5, 0, 0) meets just outside its
# third corner, where the reference's test still takes it: u = -1e-9 (a hair above -EPS) and
# v = 1 + 2e-9, whose sum is 1 + EPS
@pytest.mark.parametrize("corners", [
    ("-0x1.423ffap+0", "-0x1.22637ep+0", "0x1.00b2c6p+0", "0x1.cab6a2p+0", "-0x1.198ab4p-32", "0x1.69798ap-31"),
    ("-0x1.bcebdcp+0", "-0x1.6ac0b6p+0", "0x1.074d3ep+0", "0x1.d44fd8p+0", "-0x1.86066ep-31", "0x1.c55f76p-32"),
    ("-0x1.fd449ep+0", "-0x1.148588p+0", "0x1.546bfep+0", "0x1.7b9e2ap+0", "-0x1.6a982cp-31", "0x1.bacb88p-32"),
])
def test_link_fraction_at_a_corner(corners):
    yz = [float.fromhex(c) for c in corners]
    tri = np.array([[5.25, yz[0], yz[1]], [5.25, yz[2], yz[3]], [5.25, yz[4], yz[5]]], np.float32)
    body = box([5.4, -2.3, -2.3], [8.6, 3.3, 3.3])
    mesh = meshes.Mesh(np.concatenate([body.positions, tri.reshape(-1)]), body.triangle_count + 1)
    g, r = _both(mesh, None, (14, 9, 10), False, True)
    n = 14 * 9 * 10
    first = int(r.geometry[n + 5])
    assert r.geometry[2 * n:].view(np.float32)[first] == 0.25  # the link that meets the triangle
    assert np.array_equal(g.geometry, r.geometry)
    assert g.missed_links == r.missed_links


def _boxes(*corners):
    parts = [box(lo, hi) for lo, hi in corners]
    return np.concatenate([p.positions for p in parts]), sum(p.triangle_count for p in parts)


# a few large triangles in a fine mesh: their groups of 32 hold more pixels than a warp
# takes on its own, first, last, both, and in the supports
@pytest.mark.parametrize("floor", [False, True])
@pytest.mark.parametrize("where", ["first", "last", "both", "supports"])
def test_voxelizer_large_triangles_in_a_fine_mesh(where, floor):
    layout = (96, 70, 81)
    fine = meshes.icosphere((30.3, 33.1, 45.2), 17.7, 6)
    plate = _boxes(([2.3, 1.4, 3.2], [93.1, 68.3, 7.9]), ([50.2, 4.1, 12.3], [91.7, 64.4, 77.3]))
    parts = {"first": [plate, fine], "last": [fine, plate], "both": [plate, fine, plate], "supports": [fine]}[where]
    pos = np.concatenate([p[0] if isinstance(p, tuple) else p.positions for p in parts])
    sup = None
    if where == "supports":
        sup = meshes.Mesh(np.concatenate([plate[0], meshes.icosphere((60.3, 33.1, 45.2), 15, 6).positions]), 0)
        sup.triangle_count = sup.positions.size // 9
    g, r = _both(meshes.Mesh(pos, pos.size // 9), sup, layout, floor)
    assert np.array_equal(g.geometry, r.geometry)
    assert np.array_equal(g.boundary_cells, r.boundary_cells)
    assert (g.solid_cells, g.frontal_cells, g.watertight) == (r.solid_cells, r.frontal_cells, r.watertight)


def test_large_triangles_do_not_hold_up_a_fine_mesh():
    """12 triangles that span the grid, in a mesh of 82,000: less than four times the fine mesh's
    time (a warp a group took 30 times it)."""
    import time
    from pocketwind_gb300.geometry import voxelize
    layout = (256, 128, 128)
    fine = meshes.icosphere((64.3, 64.2, 63.9), 25.0, 6).positions
    both = np.concatenate([fine, box([0.3, 0.2, 0.4], [254.1, 126.3, 126.2]).positions])
    best = []
    for mesh in (fine, both):
        times = []
        for _ in range(8):
            t = time.perf_counter()
            voxelize(mesh, None, layout, False)
            times.append(time.perf_counter() - t)
        best.append(min(times))
    assert best[1] < 4 * best[0], best
