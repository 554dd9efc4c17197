"""The regular-pair sweeps on the two-orbit rule (csrc/orbit_pair.cuh, p1.cuh, p1_points.cuh, rwg.cuh, dp0_sym.cuh,
p1_mixed.cuh), run on a B200.

Offset classes 2, 1 and 0 with real and complex wavenumbers against the oracle; two sheets a thousandth of an element
apart, whose distances the expanded square would lose (they are differenced); grids around the row blocks of
one, of a few and of 32 rows; and the 6-point rule with its points in another order, which takes the points form or
the general kernels (FP64 for a mixed operator).  FP64 1e-12, mixed 1e-6 as the other tests; the nearly touching sheets 1e-10: the
sheets' coordinates differ in their last digits, eps / 1e-3 of the gap.
"""

import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPERATORS = [("laplace", "single_layer", "DP", 0), ("laplace", "double_layer", "P", 1),
             ("laplace", "hypersingular", "P", 1), ("helmholtz", "single_layer", "DP", 0),
             ("helmholtz", "adjoint_double_layer", "DP", 0), ("helmholtz", "single_layer", "P", 1),
             ("helmholtz", "double_layer", "P", 1), ("helmholtz", "adjoint_double_layer", "P", 1),
             ("helmholtz", "hypersingular", "P", 1), ("modified_helmholtz", "double_layer", "DP", 0),
             ("modified_helmholtz", "adjoint_double_layer", "P", 1), ("modified_helmholtz", "hypersingular", "P", 1),
             ("maxwell", "electric_field", "RWG", 0), ("maxwell", "magnetic_field", "RWG", 0)]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _operator(equation, name, kind, degree, grid, k, **kw):
    from bempp_cuda import operators
    from bempp_cuda.space import function_space

    domain = function_space(grid, kind, degree)
    dual = function_space(grid, "SNC", 0) if kind == "RWG" else domain
    factory = getattr(getattr(operators.boundary, equation), name)
    extra = () if equation == "laplace" else (k,)
    return factory(domain, domain, dual, *extra, **kw), domain, dual


def _check(oracle, case, grid, k, tol, **kw):
    from bempp_cuda.quadrature import SingularPairs, triangle_rule

    op, domain, dual = _operator(*case, grid, k, **kw)
    d = op.descriptor
    qp, qw = triangle_rule(4)
    rule = SingularPairs(grid, 4, dual.support, domain.support).arrays()
    ref = oracle.assemble_dense(d.kernel_type, d.assembly_type, d.options, d.is_complex, domain, dual, qp, qw, rule)
    got = op.weak_form().A
    assert rel_fro(got, ref) < tol
    return got


@pytest.mark.parametrize("case", OPERATORS)
def test_offset_classes(oracle, case):
    from bempp_cuda.device import device_grid
    from bempp_cuda.shapes import ellipsoid

    grid = ellipsoid(2, 1.0, 0.8, 1.2)
    bound = 2.0 * device_grid(grid).radius
    for theta in (0.4, 0.9, 2.5):
        _check(oracle, case, grid, theta / bound, 1e-12)
        if case[0] in ("helmholtz", "maxwell"):
            _check(oracle, case, grid, (1.0 + 0.8j) * theta / bound, 1e-12)


def _sheets(gap):
    """Two parallel triangulated squares ``gap`` apart, the second shifted in its plane."""
    from bempp_cuda.grid import Grid

    n = 4
    x, y = np.meshgrid(np.linspace(0, 1, n + 1), np.linspace(0, 1, n + 1), indexing="ij")
    a = np.stack([x.ravel(), y.ravel(), np.zeros(x.size)])
    b = a + np.array([[0.03], [0.05], [gap]])
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    p = (i * (n + 1) + j).ravel()
    e = np.concatenate([np.stack([p, p + n + 1, p + 1]), np.stack([p + n + 1, p + n + 2, p + 1])], axis=1)
    return Grid(np.concatenate([a, b], axis=1), np.concatenate([e, e + a.shape[1]], axis=1))


@pytest.mark.parametrize("case", OPERATORS)
def test_nearly_touching_sheets(oracle, case):
    _check(oracle, case, _sheets(2.5e-4), 1.3, 1e-10)


@pytest.mark.parametrize("level", [0, 1, 3])
@pytest.mark.parametrize("case", [OPERATORS[0], OPERATORS[5], OPERATORS[6], OPERATORS[12]])
def test_row_blocks(oracle, case, level):
    from bempp_cuda.shapes import ellipsoid

    _check(oracle, case, ellipsoid(level, 1.0, 0.8, 1.2), 1.0, 1e-12)
    if case[2] == "P" or level > 0:
        _check(oracle, case, ellipsoid(level, 1.0, 0.8, 1.2), 1.0, 1e-6, device_interface="cuda_mixed")


@pytest.mark.parametrize("interface", ["cuda", "cuda_mixed"])
@pytest.mark.parametrize("case", OPERATORS)
def test_rule_in_another_order(case, interface, monkeypatch):
    from bempp_cuda import assembly
    from bempp_cuda.shapes import ellipsoid

    grid = ellipsoid(2, 1.0, 0.8, 1.2)
    ref = _operator(*case, grid, 1.2)[0].weak_form().A
    pts, wts = assembly.regular_rule(4)
    order = [4, 1, 2, 3, 0, 5]
    rule = (np.ascontiguousarray(pts[order]), np.ascontiguousarray(wts[order]))
    monkeypatch.setattr(assembly, "regular_rule", lambda o: rule)
    got = _operator(*case, grid, 1.2, device_interface=interface)[0].weak_form().A
    assert rel_fro(got, ref) < 1e-12


def _octahedron():
    """Eight triangles with vertices at +-1 on the axes (dyadic coordinates)."""
    from bempp_cuda.grid import Grid
    from bempp_cuda.shapes import sphere_arrays

    vertices, elements = sphere_arrays(0)
    return Grid(np.round(vertices), elements)


def _midpoint_refined(grid):
    """Every triangle in four by its edge midpoints, left in its plane: the central one has its parent's centroid."""
    from bempp_cuda.grid import Grid

    v, e = np.asarray(grid.vertices), np.asarray(grid.elements)
    a, b, c = (v[:, e[i]] for i in range(3))
    ab, bc, ca = 0.5 * (a + b), 0.5 * (b + c), 0.5 * (c + a)
    corners = np.concatenate([np.stack(t) for t in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))], axis=2)
    points, index = np.unique(corners.transpose(0, 2, 1).reshape(-1, 3), axis=0, return_inverse=True)
    return Grid(np.ascontiguousarray(points.T), np.ascontiguousarray(index.reshape(3, -1)))


COMMON = [c for c in OPERATORS if c[2] in ("P", "RWG") and c[0] != "laplace"] + [
    ("modified_helmholtz", "single_layer", "P", 1), ("modified_helmholtz", "double_layer", "P", 1)]


def _united(a, b):
    """Both triangulations in one grid (the oracle takes one), no vertex shared."""
    from bempp_cuda.grid import Grid

    return Grid(np.concatenate([a.vertices, b.vertices], axis=1),
                np.concatenate([a.elements, b.elements + a.vertices.shape[1]], axis=1))


@pytest.mark.parametrize("case", COMMON)
def test_common_centroids(oracle, case):
    """Trial and test elements of two grids with the same centroid: r_c = 0, and no two of their points meet."""
    from bempp_cuda import operators
    from bempp_cuda.device import device_grid
    from bempp_cuda.space import function_space
    from cases import oracle_dense

    equation, name, kind, degree = case
    coarse = _octahedron()
    fine = _midpoint_refined(coarse)
    both, nc = _united(coarse, fine), coarse.number_of_elements
    test_kind = "SNC" if kind == "RWG" else kind
    domain, dual = function_space(coarse, kind, degree), function_space(fine, test_kind, degree)
    domain1 = function_space(both, kind, degree, support_elements=np.arange(nc))
    dual1 = function_space(both, test_kind, degree, support_elements=np.arange(nc, both.number_of_elements))
    bound = device_grid(coarse).radius + device_grid(fine).radius
    factory = getattr(getattr(operators.boundary, equation), name)
    for theta in (0.4, 0.9, 2.5):  # offset classes 2, 1, 0
        for k in (theta / bound,) if equation == "modified_helmholtz" else (theta / bound, (1.0 + 0.8j) * theta / bound):
            got = factory(domain, domain, dual, k).weak_form().A
            op = factory(domain1, domain1, dual1, k)
            ref = oracle_dense(oracle, op, domain1, dual1)
            assert np.isfinite(ref).all() and np.isfinite(got).all()
            assert rel_fro(got, ref) < 1e-12
            assert rel_fro(op.weak_form().A, ref) < 1e-12


@pytest.mark.parametrize("name", ["double_layer", "adjoint_double_layer"])
@pytest.mark.parametrize("k", [1e-310 + 0.9j, 1e-30 + 0.9j])
def test_nearly_imaginary_wavenumber(oracle, name, k):
    """A real part too small to divide by."""
    from bempp_cuda.shapes import ellipsoid

    _check(oracle, ("helmholtz", name, "DP", 0), ellipsoid(2, 1.0, 0.8, 1.2), k, 1e-12)


STRETCHED = {"flat": lambda: _ellipsoid(1.0, 1.0, 0.01), "thin": lambda: _ellipsoid(1.0, 0.03, 0.03),
             "sheets": lambda: _sheets(1e-2), "crossing": lambda: _united(_octahedron(), _midpoint_refined(_octahedron()))}


def _ellipsoid(a, b, c):
    from bempp_cuda.shapes import ellipsoid

    return ellipsoid(3, a, b, c)


@pytest.mark.parametrize("mesh", list(STRETCHED))
@pytest.mark.parametrize("case", OPERATORS)
def test_mixed_with_near_elements(oracle, case, mesh):
    """Elements that share no vertex and lie closer than their size: distances by differenced coordinates, which lose
    size / distance of FP32's digits where the expanded square loses its square.  1e-6 as elsewhere; the crossing
    triangulations lie in one plane, their points 0.02 apart at a size of 1.4, so the double layers' normal terms are
    6e-8 * 70 = 4e-6 of their distances instead of zero."""
    grid = STRETCHED[mesh]()
    tol = 4e-6 if mesh == "crossing" else 1e-6
    for k in (1.3,) if case[0] in ("laplace", "modified_helmholtz") else (1.3, 6.0, 1.3 + 0.5j):
        _check(oracle, case, grid, k, tol, device_interface="cuda_mixed")
