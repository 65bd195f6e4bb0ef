"""Small versions of the cases that the library is timed by (perf/cases.py), through the same calls, against values that do
not come from it: ``exact`` (plain torch in 64 bits) for the static steps, the derivatives, the lines and the training step,
the CPU oracle and the conserved sums for the moving runs."""
import numpy as np
import pytest

from luna_cpp_b200.mesh import build_mesh
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def static(cells, problem, **kw):
    nx, ny, nz = (list(cells) + [0])[:3]
    return dict(kind="static", nx=nx, ny=ny, nz=nz, problem=problem, precision="fp64", riemann="hllc", steps=3, limiter="plain") | kw


# What the tolerance of perf/cases.py leaves open, against 64 bits. The float policies: a float face flux is off by a few
# 2^-24 of the state's fluxes, of which a step takes about a third of a cell's content (3 steps: below 1e-6); a binary16
# slope by 2^-11, which moves the face states of the shear layer's two rows of cells by that share of the jump (below 1e-4 of
# the whole state). The learned limiter on a few thousand cells: BF16 features and weights move a factor by about 2^-8, a
# face state by that share of the variation across half a cell (0.3 x 2 pi / 16 / 2 of the state), and 3 steps take a third of
# it each: below 2e-4.
COARSE = {"fp32": 1e-6, "single": 1e-6, "grad32": 1e-6, "grad16": 1e-4}

CASES = {
    "blast": static((14, 13, 15), "blast"),
    "wave, one thread a cell": static((29, 27, 26), "wave", riemann="hll"),
    "shear in 2D": static((60, 51), "shear"),
    "acoustic, single": static((17, 16, 15), "acoustic", precision="single"),
    "wave, fp32": static((28, 27, 26), "wave", precision="fp32"),
    "wave, grad32": static((15, 14, 16), "wave", precision="grad32"),
    "shear, grad16": static((60, 51), "shear", precision="grad16"),
    "learned": static((16, 15, 14), "wave", limiter="learned"),
    "learned in 2D": static((60, 51), "wave", limiter="learned"),
    "rollout": dict(kind="rollout", nx=50, ny=43, nz=0, problem="wave", steps=5, every=2),
    "rollout in 3D": dict(kind="rollout", nx=13, ny=12, nz=14, problem="wave", steps=3, every=2),
    "jacobian": dict(kind="jacobian", nx=16, ny=13, nz=15, problem="wave", riemann="hllc"),
    "jacobian, hll": dict(kind="jacobian", nx=61, ny=47, nz=0, problem="wave", riemann="hll"),
    "lines, outflow": dict(kind="lines", cells=257, lines=3, steps=60, walls="outflow"),
    "lines, periodic": dict(kind="lines", cells=100, lines=5, steps=60, walls="periodic"),
    "lines, reflective": dict(kind="lines", cells=124, lines=2, steps=60, walls="reflective"),
    "train": dict(kind="train", rows=3001),
}


@pytest.mark.parametrize("name", CASES)
def test_case_against_64_bits(cuda, name):
    import torch
    from perf import cases

    case = CASES[name]
    got, want = cases.run(cases.prepare(case, 5)), cases.exact(case, 5)
    tol = cases.tolerance(case)["rel"]
    if case["kind"] == "static":
        tol = 2e-4 if case["limiter"] == "learned" else COARSE.get(case["precision"], tol)
    for key, w in want.items():
        g, w = (torch.as_tensor(x, dtype=torch.float64, device="cuda").reshape(-1) for x in (got[key], w))
        assert float((g - w).norm() / w.norm()) <= tol, key


@pytest.mark.parametrize("cells,problem,precision", [((14, 13, 12), "wave", "single"), ((30, 28, 27), "wave", "single"),
                                                     ((150, 131), "wave", "fp32"), ((40, 33), "wave", "fp32"),
                                                     ((14, 13, 12), "wave", "fp64"), ((40, 33), "wave", "fp64"),
                                                     ((30, 28, 27), "blast", "fp64"), ((30, 28, 27), "blast", "single"),
                                                     ((41, 40, 41), "wave", "single")])
def test_moving_case_against_the_oracle(cuda, cells, problem, precision):
    """The moving run, remeshed on the device, against the oracle's with the host's meshes, on either side of the sizes that
    take several threads a cell and (41 x 40 x 41) of those whose generators are sampled: in double the same generators and the
    state to round-off; with a float Riemann solve the generators to two steps of their grid and every field to 1e-5 of its
    largest entry (a few 2^-24 of the fluxes, two passes and two steps of it). The float blast's cells are not compared:
    across its front a pressure a rounding from zero decides whether a face takes its cell's state. Mass, momentum and energy
    are the start's, the cells fill the box."""
    from perf import cases

    nx, ny, nz = (list(cells) + [0])[:3]
    case = dict(kind="moving", nx=nx, ny=ny, nz=nz, problem=problem, precision=precision, steps=2)
    s = cases.prepare(case, 3)
    got = cases.run(s)
    q0 = s["q0"].cpu().numpy()
    points, box = cases._points(case, 3)
    ora = O.OracleFV(build_mesh(points, box=box), moving=True, precision={"fp64": "double", "fp32": "riemann32"}.get(precision, precision))
    ora.set_state(q0)
    for dt in got["dt"]:
        assert abs(ora.time_step(cases.COURANT) - dt) <= (1e-13 if precision == "fp64" else 1e-5) * dt
        mesh = ora.step_moving(dt, lambda p: build_mesh(p, box=box))
    q, want = got["q"].cpu().numpy(), ora.get_state()
    positions, volume = got["positions"].cpu().numpy(), got["volume"].cpu().numpy()
    apart = np.abs((positions - mesh.positions + 0.5 * np.array(box)) % np.array(box) - 0.5 * np.array(box))
    if precision == "fp64":
        assert np.array_equal(positions, mesh.positions) and np.array_equal(volume, mesh.volume)
        assert np.max(np.abs(q - want) / np.abs(want).max(0)) < 1e-12
    else:
        assert apart.max() <= 2 * cases.GRID * max(box)
        assert problem == "blast" or np.max(np.abs(q - want) / np.abs(want).max(0)) < 1e-5
    size = np.abs(q0).sum(0)
    size[1:-1] = np.abs(q).sum(0)[1:-1].max()
    # double sums over the faces of what one cell loses and another gains: a few 2^-53 of what passed through
    assert np.all(np.abs(q.sum(0) - q0.sum(0)) <= 1e-13 * size)
    assert abs(volume.sum() / np.prod(box) - 1) < 1e-12
