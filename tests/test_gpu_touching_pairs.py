"""The touching-pair kernels on the Sauter-Schwab rules (csrc/singular_duffy.cuh) against the flat-table kernels of
bemppcuda_assemble_singular on the same pairs (B200).

Every operator, real and complex wavenumbers in the offset classes 2, 1 and 0, meshes whose pairs take a warp each
(32 elements) and eight lanes each (2048), a space on part of the grid, and both vertex-adjacent orders with and without
mirroring; blocks into the caller's array; other orders, which take the tables, against the oracle.  The two differ in the order of 512 - 1536 terms: 1e-13 of the matrix norm.  The normal terms of the double
layers and the triple products of the magnetic field cancel between neighbours: the tables difference coordinates,
eps / h (2e-15 of the element size h = 0.06 at 2048 elements), and the result is smaller than the terms by the angle
between neighbours, about h, so each term carries 3e-14 and entries of neighbouring signs more: 1e-12.
"""

import numpy as np
import pytest

from conftest import rel_fro

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [("laplace", "single_layer", "DP", 0), ("laplace", "double_layer", "P", 1), ("laplace", "hypersingular", "P", 1),
         ("laplace", "adjoint_double_layer", "DP", 0), ("helmholtz", "single_layer", "P", 1),
         ("helmholtz", "double_layer", "DP", 0), ("helmholtz", "double_layer", "P", 1),
         ("helmholtz", "adjoint_double_layer", "P", 1), ("helmholtz", "hypersingular", "P", 1),
         ("modified_helmholtz", "single_layer", "DP", 0), ("modified_helmholtz", "double_layer", "P", 1),
         ("modified_helmholtz", "hypersingular", "DP", 1), ("maxwell", "electric_field", "RWG", 0),
         ("maxwell", "magnetic_field", "RWG", 0), ("combined", "", "DP", 0)]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _descriptor(equation, name, domain, dual, k):
    from bempp_cuda import operators

    if equation == "combined":
        k = complex(k)
        return operators.OperatorDescriptor("helmholtz_combined_field_boundary", [k.real, k.imag, k.imag, -k.real],
                                            "helmholtz_combined_field", "default_scalar", "double", True, None, 1)
    factory = getattr(getattr(operators.boundary, equation), name)
    return (factory(domain, domain, dual) if equation == "laplace" else factory(domain, domain, dual, k)).descriptor


def _flat(lib):
    return lambda args, order, stream: lib.bemppcuda_assemble_singular(args, stream)


class _Library(object):
    def __init__(self, lib):
        self._lib = lib
        self.bemppcuda_assemble_singular_duffy = _flat(lib)

    def __getattr__(self, name):
        return getattr(self._lib, name)


def _matrix(descriptor, domain, dual, **kw):
    from bempp_cuda import operators
    from bempp_cuda.assembly import result_dtype, singular_into_dense

    out = torch.zeros((dual.global_dof_count, domain.global_dof_count), dtype=result_dtype(descriptor), device="cuda")
    return singular_into_dense(out, descriptor, domain, dual, operators.Parameters(), **kw)


@pytest.mark.parametrize("equation,name,kind,degree", CASES)
@pytest.mark.parametrize("level", [1, 4])
def test_equals_flat_tables(equation, name, kind, degree, level, monkeypatch):
    from bempp_cuda import _lib
    from bempp_cuda.device import device_grid
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space

    grid = ellipsoid(level, 1.0, 0.8, 1.2)
    support = None if kind in ("P", "RWG") else np.arange(grid.number_of_elements - 5)
    domain = function_space(grid, kind, degree, support_elements=support)
    dual = function_space(grid, "SNC", 0) if kind == "RWG" else domain
    bound = 2.0 * device_grid(grid).radius
    tol = 1e-12 if "double" in name or name == "magnetic_field" or equation == "combined" else 1e-13
    shift = -0.5 if equation == "combined" else 0.0
    real = equation in ("laplace", "modified_helmholtz")
    lib = _lib.load()
    for theta in (0.3, 0.7, 2.5):
        for k in [theta / bound] if real else [theta / bound, (1.0 + 0.6j) * theta / bound]:
            d = _descriptor(equation, name, domain, dual, k)
            got = _matrix(d, domain, dual, diag_shift=shift)
            pairs = _matrix(d, domain, dual, diag_shift=shift, mirror=False)
            with monkeypatch.context() as m:
                m.setattr(_lib, "load", lambda: _Library(lib))
                ref = _matrix(d, domain, dual, diag_shift=shift, mirror=False)
            norm = torch.linalg.vector_norm(ref)
            assert float(torch.linalg.vector_norm(got - ref) / norm) < tol
            assert float(torch.linalg.vector_norm(pairs - ref) / norm) < tol


def test_coincident_double_layer_is_zero():
    """Both points of a coincident pair lie in one plane."""
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space

    space = function_space(ellipsoid(3, 1.0, 0.8, 1.2), "DP", 0)
    a = _matrix(_descriptor("helmholtz", "double_layer", space, space, 2.0), space, space)
    assert float(a.diagonal().abs().max()) == 0.0


@pytest.mark.parametrize("order", [3, 5])
@pytest.mark.parametrize("case", [("laplace", "single_layer", "DP", 0), ("helmholtz", "double_layer", "DP", 0),
                                  ("helmholtz", "single_layer", "P", 1), ("laplace", "hypersingular", "P", 1)])
def test_other_orders_take_the_tables(oracle, case, order):
    """A singular order other than 4 goes through the flat tables, vertex-adjacent pairs once for both orders or each on
    its own: against the oracle at that order, 1e-12 as the other FP64 paths."""
    from bempp_cuda import operators
    from bempp_cuda.assembly import result_dtype, singular_into_dense
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space
    from cases import oracle_dense

    equation, name, kind, degree = case
    space = function_space(ellipsoid(2, 1.0, 0.8, 1.2), kind, degree)
    parameters = operators.Parameters()
    parameters.quadrature.singular = order
    factory = getattr(getattr(operators.boundary, equation), name)
    op = factory(space, space, space, *(() if equation == "laplace" else (1.5,)), parameters=parameters)
    ref = oracle_dense(oracle, op, space, space)
    assert rel_fro(op.weak_form().A, ref) < 1e-12
    parts = []
    for mirror in (True, False):
        out = torch.zeros(ref.shape, dtype=result_dtype(op.descriptor), device="cuda")
        parts.append(singular_into_dense(out, op.descriptor, space, space, parameters, mirror=mirror))
    assert float(torch.linalg.vector_norm(parts[0] - parts[1]) / np.linalg.norm(ref)) < 1e-12


def _values(equation, name, kind, degree, structured):
    """The pairs' blocks in the caller's array instead of a matrix, added to the ones that are there; and the pairs."""
    from bempp_cuda import _lib
    from bempp_cuda.assembly import _set_params, kernel_ids, result_dtype
    from bempp_cuda.device import current_stream, device_grid, device_singular_rule, device_space
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space

    grid = ellipsoid(2, 1.0, 0.8, 1.2)
    domain = function_space(grid, kind, degree)
    dual = function_space(grid, "SNC", 0) if kind == "RWG" else domain
    d = _descriptor(equation, name, domain, dual, 1.5)
    rule = device_singular_rule(grid, 4, dual.support, domain.support)
    args = _lib.SingularArgs()
    args.kernel, args.assembly = kernel_ids(d)
    args.is_complex = 1 if d.is_complex else 0
    _set_params(args, d.options)
    args.grid, args.test, args.trial = (device_grid(grid).record(), device_space(dual).record(),
                                        device_space(domain).record())
    rule.fill(args)
    args.phase_radius = 1.0001 * 2.0 * device_grid(grid).radius
    shapes = (device_space(dual).nshape, device_space(domain).nshape)
    values = torch.ones((rule.npairs,) + shapes, dtype=result_dtype(d), device="cuda")
    args.values = values.data_ptr()
    lib = _lib.load()
    _lib.check(lib.bemppcuda_assemble_singular_duffy(args, 4, current_stream()) if structured
               else lib.bemppcuda_assemble_singular(args, current_stream()))
    return values - 1.0, rule


@pytest.mark.parametrize("equation,name,kind,degree", [CASES[1], CASES[5], CASES[8], CASES[12], CASES[13]])
def test_values_per_pair(equation, name, kind, degree):
    got, ref = (_values(equation, name, kind, degree, structured)[0] for structured in (True, False))
    assert float(torch.linalg.vector_norm(ref)) > 0.0
    tol = 1e-12 if "double" in name or name == "magnetic_field" else 1e-13
    # (adding to one loses eps per value)
    assert float((got - ref).abs().max()) < tol * float(ref.abs().max()) + 4e-16


@pytest.mark.parametrize("equation,name,kind,degree", [CASES[6], CASES[13]])
def test_coincident_blocks_in_one_plane_are_zero(equation, name, kind, degree):
    """Double layers and the magnetic field of an element with itself."""
    got, rule = _values(equation, name, kind, degree, True)
    assert float(got[rule.test_elements == rule.trial_elements].abs().max()) == 0.0
    assert float(got.abs().max()) > 0.0
