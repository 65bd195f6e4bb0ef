"""The device remesher (include/luna_remesh.h) and the sweep's tiles cut on the device.

The remesher clips each cell on the GPU with the host builder's code and assembles faces and lists in the host
builder's order, so its arrays equal ``build_mesh``'s bit for bit. A mesh given in device memory has its sweep tiles
cut on the device; the step's results do not depend on the tiling, so a step on it equals, bit for bit, the step on
the same mesh given in host memory (tiles cut on the host). A moving step with the remesh on the device equals the
moving step with the host remesh, bit for bit.
"""
import ctypes
import dataclasses
import os

import numpy as np
import pytest
from conftest import jittered_mesh, voronoi_invariants

from luna_cpp_b200 import hydro
from luna_cpp_b200.mesh import build_mesh, jittered_points
from luna_cpp_b200.problems import point_blast, rough_state
from luna_cpp_b200.remesh import Remesher

pytestmark = pytest.mark.gpu

FIELDS = ("owner", "neighbour", "cell_face_start", "cell_face", "area", "face_centroid", "centroid", "volume", "positions")


# LUNA_MESH_DUAL=0 in the environment switches the host builder's 3D cells to face loops while the device keeps plane
# triples: the two then agree to round-off (the same faces and lists; areas, centroids and volumes to 1e-12), not bit for
# bit.
HOST_FACE_LOOPS = os.environ.get("LUNA_MESH_DUAL") == "0"


def assert_same_mesh(host, dev):
    assert (dev.n_cells, dev.n_faces, dev.inconsistent) == (host.n_cells, host.n_faces, host.inconsistent)
    for f in FIELDS:
        a, b = np.ascontiguousarray(getattr(host, f)), np.ascontiguousarray(getattr(dev, f))
        assert a.shape == b.shape, f
        if HOST_FACE_LOOPS and host.dim == 3 and a.dtype.kind == "f":
            assert np.max(np.abs(a - b)) <= 1e-12 * max(np.max(np.abs(a)), 1e-300), f
        else:
            assert a.tobytes() == b.tobytes(), f


def cases():
    rng = np.random.default_rng(7)
    yield "jittered 16^3", jittered_points((16, 16, 16), jitter=0.1, seed=1), (1.0, 1.0, 1.0)
    yield "uniform random 1500", rng.random((1500, 3)), (1.0, 1.0, 1.0)
    box = (1.0, 0.8, 1.2)
    yield "random, box 1 x 0.8 x 1.2", rng.random((1200, 3)) * np.array(box), box
    yield "jittered, outside the box", jittered_points((10, 10, 10), jitter=0.1, seed=3) + np.array([1.0, -2.0, 0.5]), (1.0, 1.0, 1.0)
    yield "2D jittered 40^2", jittered_points((40, 40), jitter=0.1, seed=1), (1.0, 1.0)
    yield "2D uniform random 2000", rng.random((2000, 2)), (1.0, 1.0)


@pytest.mark.parametrize("name,points,box", list(cases()), ids=[c[0] for c in cases()])
def test_device_mesh_equals_host_builder(cuda, name, points, box):
    host = build_mesh(points, box=box)
    r = Remesher(len(box), box)
    dev = r.build(points).to_host()
    assert_same_mesh(host, dev)
    voronoi_invariants(dev)
    r.close()


def lane_cases():
    """What the eight-lane cells meet at their limits: a last block with one cell, more cells than one chunk holds
    (2^17), images at equal distances, a blob whose balls hold more images than a search keeps and whose rim cells have
    more planes than a lane cell, a box of unequal buckets."""
    rng = np.random.default_rng(11)
    yield "9^3 + 8 random", np.vstack([jittered_points((9, 9, 9), jitter=0.1, seed=2), rng.random((8, 3))]), (1.0, 1.0, 1.0)
    yield "131081 random", rng.random((131081, 3)), (1.0, 1.0, 1.0)
    yield "regular 12^3", jittered_points((12, 12, 12), jitter=0.0, seed=1), (1.0, 1.0, 1.0)
    blob = rng.random((4000, 3))
    blob[:800] = 0.35 + 0.3 * blob[:800]
    yield "blob", blob, (1.0, 1.0, 1.0)
    # a peak of density: balls with more images than any of a search's five holds
    peak = rng.random((6000, 3))
    peak[:3000] = (0.5 + 0.05 * rng.standard_normal((3000, 3))) % 1.0
    yield "peak", peak, (1.0, 1.0, 1.0)


@pytest.mark.parametrize("name,points,box", list(lane_cases()), ids=[c[0] for c in lane_cases()])
def test_cells_by_lanes_equal_host_builder(cuda, name, points, box):
    r = Remesher(3, box)
    assert_same_mesh(build_mesh(points, box=box), r.build(points).to_host())
    left = r.one_thread_cells()  # (131,081 random points: one wave of threads, all of them)
    assert {"9^3 + 8 random": left < 50, "131081 random": left == len(points), "regular 12^3": left == 0}.get(name, 0 < left < len(points)), left
    r.close()


@pytest.mark.parametrize("cells,box,lattice", [((40, 40, 40), (1.0, 1.0, 1.0), True), ((39, 40, 41), (1.0, 1.0, 1.0), False),
                                               ((48, 45, 50), (0.96, 0.9, 1.5), True)])
def test_lattice_cells_take_one_thread(cuda, cells, box, lattice):
    """A rectangular lattice of 64,000 cells or more is built by one thread a cell, a smaller one and one with a
    thousandth of jitter by lanes, which finish every cell; the meshes are the host builder's."""
    rng = np.random.default_rng(8)
    r = Remesher(3, box)
    h = np.array(box) / np.array(cells)
    points = (np.stack(np.meshgrid(*[np.arange(n) for n in cells], indexing="ij"), -1).reshape(-1, 3) + 0.5) * h
    assert_same_mesh(build_mesh(points, box=box), r.build(points).to_host())
    assert r.one_thread_cells() == (len(points) if lattice else 0)
    points += 1e-3 * h * rng.uniform(-1, 1, points.shape)
    assert_same_mesh(build_mesh(points, box=box), r.build(points).to_host())
    assert r.one_thread_cells() == 0
    r.close()


@pytest.mark.parametrize("n,share", [(2000, None), (40000, None), (63999, None), (64000, 1), (151552, 1), (151553, None)])
def test_cells_of_random_points_by_count(cuda, n, share):
    """The lanes leave about half of the cells of random points to one thread each (of 2,000 and of 40,000 points spread
    over the warps); between 64,000 and one wave of threads all cells take one thread. The meshes are the host builder's."""
    points = np.random.default_rng(n).random((n, 3))
    r = Remesher(3, (1.0, 1.0, 1.0))
    assert_same_mesh(build_mesh(points), r.build(points).to_host())
    assert r.one_thread_cells() == n if share else 0.2 * n < r.one_thread_cells() < 0.8 * n
    r.close()


def test_remesher_reuse_grows_and_shrinks(cuda):
    """One remesher, meshes of different sizes in turn (its buffers are kept and grown)."""
    r = Remesher(3, (1.0, 1.0, 1.0))
    for nx in (8, 14, 6, 14):
        pts = jittered_points((nx,) * 3, jitter=0.1, seed=nx)
        assert_same_mesh(build_mesh(pts), r.build(pts).to_host())
    assert r.device_bytes() > 0
    r.close()


def test_remesher_errors_are_status_codes(cuda):
    r = Remesher(3, (1.0, 1.0, 1.0))
    with pytest.raises(hydro.LunaError) as e:  # two points: each cell reaches its own images
        r.build(np.array([[0.5, 0.5, 0.5], [0.1, 0.1, 0.1]]))
    assert e.value.status == 1
    pts = jittered_points((6, 6, 6), jitter=0.1, seed=1)
    pts[3, 1] = np.nan
    with pytest.raises(hydro.LunaError) as e:
        r.build(pts)
    assert e.value.status == 1
    # still usable after an error
    good = jittered_points((6, 6, 6), jitter=0.1, seed=1)
    assert_same_mesh(build_mesh(good), r.build(good).to_host())
    r.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32", "grad16"])
def test_static_step_on_device_tiles_equals_host_tiles(cuda, precision):
    """The same mesh given in host memory (tiles cut on the host, greedily) and in device memory (tiles cut on the
    device, fixed Morton chunks): five static steps give the same bits."""
    mesh = jittered_mesh(20)
    r = Remesher(3, mesh.box)
    dmesh = r.build(mesh.positions)
    q0 = point_blast(mesh)
    a = hydro.FiniteVolume(mesh, precision=precision)
    b = hydro.FiniteVolume(dmesh, precision=precision)
    a.set_state(q0)
    b.set_state(q0)
    for _ in range(5):
        dt = a.time_step(0.3)
        assert b.time_step(0.3) == dt
        a.step(dt)
        b.step(dt)
    assert np.array_equal(a.get_state(), b.get_state())
    assert np.array_equal(a.gradients(), b.gradients())
    a.close()
    b.close()
    r.close()


class OnDevice:
    """A host mesh's arrays in device memory, as a caller with a mesh builder of its own on the device has them."""

    def __init__(self, mesh):
        import torch

        self.dim, self.n_cells, self.n_faces, self.box = mesh.dim, mesh.n_cells, mesh.n_faces, mesh.box
        self.desc = hydro.mesh_desc(mesh, [])
        self.arrays = {f: torch.tensor(np.ascontiguousarray(getattr(mesh, f)), device="cuda") for f in FIELDS}
        for f, x in self.arrays.items():
            setattr(self.desc, f, x.data_ptr())
        self.desc.on_device = 1


def shrunk(mesh, side):
    """The mesh at `side` times its size, in the middle of one cell of the Morton keys' upper half. Lists, areas, volumes and
    centroids are the mesh's; the separations across its seam are not periodic any more, so a step on it is arithmetic and
    not physics, the same for every tiling."""
    corner = 0.5 + np.array([2.0 ** -11, 2.0 ** -12, 2.0 ** -12]) - 0.5 * side
    return dataclasses.replace(mesh, positions=corner + side * mesh.positions, centroid=side * mesh.centroid,
                               face_centroid=side * mesh.face_centroid, area=side ** 2 * mesh.area, volume=side ** 3 * mesh.volume)


@pytest.mark.parametrize("nx", [10, 17])
def test_device_tiles_of_cells_far_below_the_box(cuda, nx):
    """Cells that share one upper Morton key, in random order (17^3: 128 of them in index order have more distinct
    neighbours than the small table; 10^3: nearly all the others): the device cuts such a mesh by the whole key, the step
    has the host tiles' bits, and a solver goes from one cut to the other with its mesh."""
    points = jittered_points((nx,) * 3, jitter=0.1, seed=2)
    wide = build_mesh(points[np.random.default_rng(3).permutation(len(points))])
    tiny = shrunk(wide, 1e-4)
    q0 = rough_state(tiny.n_cells) * tiny.volume[:, None]
    a, b = hydro.FiniteVolume(tiny), hydro.FiniteVolume(OnDevice(tiny))
    assert a.tiles()["cut"] == "host" and b.tiles()["cut"] == "device, wide"
    # the cut tried first is the one that the mesh before asked for
    for mesh, cut in ((wide, "device, wide"), (wide, "device"), (tiny, "device, wide"), (tiny, "device, wide")):
        b.set_mesh(OnDevice(mesh))
        assert b.tiles()["cut"] == cut
    assert b.tiles()["second"] == 0  # the cut by the whole key keeps neighbours together
    a.set_state(q0)
    b.set_state(q0)
    for _ in range(2):
        dt = a.time_step(0.1)
        assert b.time_step(0.1) == dt
        a.step(dt)
        b.step(dt)
    assert np.all(np.isfinite(a.get_state())) and np.array_equal(a.get_state(), b.get_state())
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "single", "grad16"])
@pytest.mark.parametrize("cells", [(31, 29, 27), (153, 131)])
def test_device_tiles_with_one_thread_a_cell(cuda, cells, precision):
    """Past the sizes that take several threads a cell (18,944): three steps on the device's tiles have the bits of the host's."""
    box = tuple(c / cells[0] for c in cells)
    r = Remesher(len(cells), box)
    dmesh = r.build(jittered_points(cells, side=box, jitter=0.3, seed=4))
    mesh = dmesh.to_host()
    q0 = rough_state(mesh.n_cells, dim=mesh.dim) * mesh.volume[:, None]
    a, b = hydro.FiniteVolume(mesh, precision=precision), hydro.FiniteVolume(dmesh, precision=precision)
    assert a.tiles()["cut"] == "host" and b.tiles()["cut"] == "device"
    a.set_state(q0)
    b.set_state(q0)
    for _ in range(3):
        dt = a.time_step(0.3)
        assert b.time_step(0.3) == dt
        a.step(dt)
        b.step(dt)
    assert np.array_equal(a.get_state(), b.get_state())
    for x in (a, b, r):
        x.close()


@pytest.mark.parametrize("precision", ["fp64", "grad32"])
@pytest.mark.parametrize("faces,side", [(700, 24), (1400, 24), (700, 160)])
def test_device_tiles_past_the_first_launch(cuda, faces, side, precision):
    """A cell of many faces on a device mesh: its tile stages more than the 640 cells of the first launch (and, with 1,400
    faces, more than 48 KB of them in the derivatives' sweeps too) and goes to the second one, with the geometry read
    through the faces. Steps, adjoint and tangent have the bits of the host's tiles, with several threads a cell and (160^2
    cells around it) with one."""
    from test_gpu_parity import ring_mesh

    mesh = ring_mesh(faces, side)
    assert (mesh.n_cells > 18944) == (side == 160)
    q0 = rough_state(mesh.n_cells, dim=2) * mesh.volume[:, None]
    a, b = hydro.FiniteVolume(mesh, precision=precision), hydro.FiniteVolume(OnDevice(mesh), precision=precision)
    assert b.tiles()["cut"] == "device" and b.tiles()["second"] > 0 and b.tiles()["rows"] > max(640, faces)
    a.set_state(q0)
    b.set_state(q0)
    for _ in range(2):
        dt = a.time_step(0.3)
        assert b.time_step(0.3) == dt
        a.step(dt)
        b.step(dt)
    assert np.array_equal(a.get_state(), b.get_state())
    if precision == "fp64":
        bars = np.random.default_rng(2).standard_normal(q0.shape)
        assert np.array_equal(a.step_adjoint(dt, bars), b.step_adjoint(dt, bars))
        assert np.array_equal(a.step_tangent(dt, bars * q0), b.step_tangent(dt, bars * q0))
    a.close()
    b.close()


@pytest.mark.parametrize("dim", [3, 2])
def test_moving_step_with_device_remesh_equals_host_remesh(cuda, dim):
    """Moving steps (the t^n fluxes, the drift on the 2^-30 grid, the remesh, the t^n+1 fluxes) with the generators and
    the mesh kept on the device against the same steps with the host remesh: the same dt, positions and state, bit for
    bit; mass and energy conserved to round-off."""
    step = 2.0 ** -30
    nx = 12 if dim == 3 else 40
    pts = np.round(jittered_points((nx,) * dim, jitter=0.1, seed=1) / step) * step
    mesh = build_mesh(pts, box=(1.0,) * dim)
    q0 = point_blast(mesh, radius_cells=2.5)
    host = hydro.FiniteVolume(mesh, motion="moving")
    dev = hydro.FiniteVolume(mesh, motion="moving")
    host.set_state(q0)
    dev.set_state(q0)
    r = Remesher(dim, mesh.box)
    lib = hydro.lib()
    for _ in range(4):
        dt = host.time_step(0.3)
        assert dev.time_step(0.3) == dt
        mh = host.step_moving(dt, lambda p: build_mesh(p, box=(1.0,) * dim))
        # dev.step_moving_device(dt, r) in its three calls, the new mesh checked before the hydro takes it
        ptr = r.points_buffer(dev.n)
        hydro.check(lib.luna_fv_step_moving_begin(dev.handle, dt, ptr, 1))
        md = r.build_device(ptr, dev.n)
        assert_same_mesh(mh, md.to_host())
        hydro.check(lib.luna_fv_step_moving_end(dev.handle, ctypes.byref(md.desc)))
    dt = host.time_step(0.3)
    assert dev.time_step(0.3) == dt
    host.step_moving(dt, lambda p: build_mesh(p, box=(1.0,) * dim))
    dev.step_moving_device(dt, r)
    qh, qd = host.get_state(), dev.get_state()
    assert np.array_equal(qh, qd)
    assert abs(qd[:, 0].sum() - q0[:, 0].sum()) / q0[:, 0].sum() < 1e-14
    assert abs(qd[:, -1].sum() - q0[:, -1].sum()) / q0[:, -1].sum() < 1e-14
    host.close()
    dev.close()
    r.close()


def test_device_mesh_64cubed_equals_host_builder(cuda):
    """A 64^3 jittered mesh (262,144 cells, 2.1 M faces): the device build equals the host build."""
    pts = jittered_points((64, 64, 64), jitter=0.1, seed=1)
    r = Remesher(3, (1.0, 1.0, 1.0))
    assert_same_mesh(build_mesh(pts), r.build(pts).to_host())
    r.close()
