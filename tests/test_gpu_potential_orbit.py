"""FP64 potentials and far fields with the two-orbit rule (csrc/potential_orbit.cuh) against the oracle, run on a B200.

Point counts around the 32-point thread rows and the 64-point blocks, element counts around the staged tile of 32
and the four warps that share it, offset classes 2, 1 and 0 (k R = 0.3, 0.8, 3), complex wavenumbers, points
on and next to the surface, directions that are not unit vectors, and the same rule with its points in
another order, which takes the general kernels.  Tolerance 1e-12 relative Frobenius norm as for the other FP64
paths; next to the surface the sums cancel (electric potential), so those cases state 1e-11.
"""

import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPERATORS = ["potential.laplace.single_layer", "potential.laplace.double_layer", "potential.helmholtz.single_layer",
             "potential.helmholtz.double_layer", "potential.modified_helmholtz.single_layer",
             "potential.modified_helmholtz.double_layer", "far_field.helmholtz.single_layer",
             "far_field.helmholtz.double_layer", "potential.maxwell.electric_field",
             "potential.maxwell.magnetic_field", "far_field.maxwell.electric_field",
             "far_field.maxwell.magnetic_field"]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _space(path, level, support=None):
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space

    grid = ellipsoid(level, 1.0, 0.9, 1.1)
    kind = ("RWG", 0) if "maxwell" in path else ("P", 1) if level else ("DP", 0)
    if support is not None:
        kind = ("DP", 0)
    return function_space(grid, *kind, support_elements=support)


def _points(path, count, rng, radius=2.0):
    p = rng.standard_normal((3, count))
    p /= np.linalg.norm(p, axis=0)
    return p if path.startswith("far_field") else p * (radius * rng.uniform(0.7, 1.5, count))


def _run(path, space, points, k, oracle, tol):
    from bempp_cuda import operators
    from cases import oracle_potential

    obj = operators
    for part in path.split("."):
        obj = getattr(obj, part)
    op = obj(space, points) if "laplace" in path else obj(space, points, k)
    rng = np.random.default_rng(2)
    c = rng.standard_normal(space.global_dof_count) + 1j * rng.standard_normal(space.global_dof_count)
    got = op.evaluate_device(c).cpu().numpy()
    ref = oracle_potential(oracle, op, space, c)
    assert rel_fro(got, ref) < tol
    return got, op, c


@pytest.mark.parametrize("count", [1, 33, 129])
@pytest.mark.parametrize("path", OPERATORS)
def test_point_and_class_edges(oracle, path, count):
    space = _space(path, 2)
    from bempp_cuda.device import device_grid

    radius = device_grid(space.grid).radius
    for kr in (0.3, 0.8, 3.0):
        points = _points(path, count, np.random.default_rng(count))
        _run(path, space, points, kr / radius, oracle, 1e-12)
        if path.startswith("potential.helmholtz") or path.startswith("potential.maxwell"):
            _run(path, space, points, (1.0 + 0.7j) * kr / radius, oracle, 1e-12)


@pytest.mark.parametrize("elements", [1, 3, 31, 33, 65])
def test_element_edges(oracle, elements):
    for path in ("potential.helmholtz.double_layer", "far_field.helmholtz.single_layer"):
        space = _space(path, 2, support=np.arange(7, 7 + elements))
        _run(path, space, _points(path, 40, np.random.default_rng(1)), 2.0, oracle, 1e-12)


@pytest.mark.parametrize("path", [p for p in OPERATORS if p.startswith("potential")])
def test_next_to_the_surface(oracle, path):
    space = _space(path, 3)
    grid = space.grid
    points = np.concatenate([grid.centroids[:5].T + 1e-3 * grid.normals[:5].T, 0.2 * np.eye(3)], axis=1)
    _run(path, space, points, 2.0, oracle, 1e-11)


def test_directions_beyond_the_unit_sphere(oracle):
    path = "far_field.helmholtz.single_layer"
    space = _space(path, 2)
    points = 9.0 * _points(path, 20, np.random.default_rng(4))
    _run(path, space, points, 1.5, oracle, 1e-12)


@pytest.mark.parametrize("path", OPERATORS)
def test_rule_in_another_order(oracle, path, monkeypatch):
    from bempp_cuda import assembly

    space = _space(path, 2)
    points = _points(path, 50, np.random.default_rng(6))
    got, op, c = _run(path, space, points, 1.5, oracle, 1e-12)
    pts, wts = assembly.regular_rule(4)
    order = [3, 1, 2, 0, 4, 5]
    rule = (np.ascontiguousarray(pts[order]), np.ascontiguousarray(wts[order]))
    monkeypatch.setattr(assembly, "regular_rule", lambda o: rule)
    assert rel_fro(op.evaluate_device(c).cpu().numpy(), got) < 1e-12


@pytest.mark.parametrize("path", [p for p in OPERATORS if p.startswith("potential") and "laplace" not in p])
def test_at_a_centroid(oracle, path):
    """Points on a centroid and so close to one that the squared distance is a subnormal number."""
    from bempp_cuda.grid import Grid
    from bempp_cuda.shapes import sphere_arrays
    from bempp_cuda.space import function_space

    vertices, elements = sphere_arrays(0)
    vertices = 3.0 * np.round(vertices) - 1.0  # the face at (3, 0, 0), (0, 3, 0), (0, 0, 3) moves to the centroid 0
    space = function_space(Grid(vertices, elements), *(("RWG", 0) if "maxwell" in path else ("P", 1)))
    points = np.array([[0.0, 1e-160, 1e-160], [0.0, 0.0, -1e-161], [0.0, 0.0, 0.0]])
    for k in (0.1,) if "modified" in path else (0.1, 0.1 + 0.06j):
        got, _, _ = _run(path, space, points, k, oracle, 1e-12)
        assert np.isfinite(got).all()
