"""Performance cases: the calls a boundary-element program spends its GPU time in.

A case is a closed triangle surface (a smoothly deformed ellipsoid of 8 n^2 elements) and one call of
the public interface on it: the weak form of a boundary operator, a potential or far field at a set of
points, a batch of small problems with their products, a GMRES solve, or a far-field objective with its
shape gradient.  ``listed`` holds the cases that are reported, ``draw`` gives more of the same ranges.

``exact`` restates every case in plain torch, in 64 bits, from the same meshes: the 6-point triangle
rule for separated elements, the Sauter-Schwab rules (S. Sauter, C. Schwab, "Boundary Element Methods",
Springer 2011, section 5.2) for touching ones.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bempp-cl_b200"))

from bempp_cuda import linalg, operators, shape_gradient  # noqa: E402
from bempp_cuda.batch import BatchAssembler  # noqa: E402
from bempp_cuda.grid import Grid  # noqa: E402
from bempp_cuda.grid_function import GridFunction, device_callable  # noqa: E402
from bempp_cuda.space import function_space  # noqa: E402

# ------------------------------------------------------------------------------------------- the cases


def _operator(equation, operator, space, n, k=0.0, k_imag=0.0, interface="cuda"):
    return {"kind": "operator", "equation": equation, "operator": operator, "space": space, "n": n, "k": k,
            "k_imag": k_imag, "interface": interface}


def _potential(equation, operator, space, n, points, k=0.0, k_imag=0.0, interface="cuda", far=False):
    return dict(_operator(equation, operator, space, n, k, k_imag, interface), kind="potential", points=points, far=far)


def _named(name, case):
    return dict(case, name=name)


def listed():
    return [
        # the first solve of a capacitance or a test problem: all latency
        _named("laplace_dp0_128", _operator("laplace", "single_layer", "DP0", 4)),
        # exterior scattering at a large size, the combined field in mixed precision: the headline workload
        _named("combined_dp0_mixed_32768", _operator("helmholtz", "combined_field", "DP0", 64, 10.0,
                                                     interface="cuda_mixed")),
        # the same equation in double precision on a mesh whose size fits no tile
        _named("combined_dp0_16200", _operator("helmholtz", "combined_field", "DP0", 45, 8.0)),
        # sound-hard scattering (Burton-Miller): the hypersingular operator on continuous functions
        _named("hypersingular_p1_8192", _operator("helmholtz", "hypersingular", "P1", 32, 5.0)),
        # its double layer in mixed precision, odd size
        _named("double_p1_mixed_10952", _operator("helmholtz", "double_layer", "P1", 37, 6.0,
                                                  interface="cuda_mixed")),
        # an absorbing medium: complex wavenumber
        _named("single_p1_damped_7688", _operator("helmholtz", "single_layer", "P1", 31, 5.0, 0.5)),
        # electromagnetic scattering: the electric field operator on RWG functions
        _named("electric_rwg_2048", _operator("maxwell", "electric_field", "RWG", 16, 2.0)),
        # the scattered pressure on a slice of the domain
        _named("potential_p1_10000", _potential("helmholtz", "single_layer", "P1", 32, 10000, 5.0)),
        # the scattered electric field on a slice, odd sizes
        _named("potential_electric_4999", _potential("maxwell", "electric_field", "RWG", 23, 4999, 4.0)),
        # a bistatic radar cross section: the electric far field
        _named("far_electric_3600", _potential("maxwell", "electric_field", "RWG", 32, 3600, 5.0, far=True)),
        # a sweep over 24 small scatterers and wavenumbers with 8 incident waves each
        _named("batch_24", {"kind": "batch", "count": 24, "n_least": 4, "n_most": 22, "precision": "fp64",
                            "kernel": "helmholtz_single_layer"}),
        # a shape-optimisation step: objective, two GMRES solves, gradient by vertices and wavenumber
        _named("gradient_2048", {"kind": "gradient", "n": 16, "k": 4.0, "directions": 32, "solver": "gmres"}),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["operator"] * 6 + ["potential"] * 4 + ["batch", "solve", "gradient"])
    k = round(rng.uniform(1.0, 8.0), 3)
    interface = rng.choice(["cuda", "cuda", "cuda_mixed"])
    k_imag = rng.choice([0.0, 0.0, 0.0, round(0.1 * k, 3)])
    if kind == "operator":
        space = rng.choice(["DP0", "P1", "P1", "RWG"])
        n = _log_int(rng, 4, {"DP0": 50, "P1": 37, "RWG": 24}[space])
        if space == "RWG":
            name = rng.choice(["electric_field", "magnetic_field"])
            return _operator("maxwell", name, "RWG", n, k, k_imag, interface)
        equation = rng.choice(["helmholtz", "helmholtz", "laplace", "modified_helmholtz"])
        names = ["single_layer", "double_layer", "adjoint_double_layer"]
        if space == "P1":
            names.append("hypersingular")
        elif equation == "helmholtz":
            names.append("combined_field")
        return _operator(equation, rng.choice(names), space, n, 0.0 if equation == "laplace" else k,
                         k_imag if equation == "helmholtz" else 0.0, interface)
    if kind == "potential":
        equation = rng.choice(["helmholtz", "maxwell", "maxwell", "laplace", "modified_helmholtz"])
        far = equation in ("helmholtz", "maxwell") and rng.random() < 0.5
        name = rng.choice(["electric_field", "magnetic_field"] if equation == "maxwell"
                          else ["single_layer", "double_layer"])
        space = "RWG" if equation == "maxwell" else rng.choice(["DP0", "P1"])
        return _potential(equation, name, space, _log_int(rng, 4, 32), _log_int(rng, 64, 10000),
                          0.0 if equation == "laplace" else k,
                          k_imag if equation in ("helmholtz", "maxwell") and not far else 0.0, interface, far)
    if kind == "batch":
        least = rng.randint(3, 6)
        return {"kind": "batch", "count": rng.randint(8, 24), "n_least": least, "n_most": rng.randint(least + 2, 24),
                "precision": rng.choice(["fp64", "mixed"]),
                "kernel": rng.choice(["helmholtz_single_layer", "helmholtz_combined_field"])}
    if kind == "solve":
        return {"kind": "solve", "n": _log_int(rng, 8, 32), "k": k, "interface": interface}
    return {"kind": "gradient", "n": _log_int(rng, 5, 16), "k": round(rng.uniform(1.0, 4.0), 3),
            "directions": rng.randint(8, 64), "solver": rng.choice(["lu", "gmres"])}


# -------------------------------------------------------------------------------------------- the meshes


def _elements_of(n):
    return 8 * n * n


def _octahedral_mesh(n):
    """Unit directions (nv, 3) and outward triangles (ne, 3) of an octahedron with n parts per edge.  The
    elements of a face follow a space-filling (Morton) curve, neighbours in space being near in number, as
    refinement and mesh generators leave them."""
    r = np.arange(n)
    rows, cols = np.meshgrid(r, r, indexing="ij")
    up = (rows + cols < n).ravel()
    down = (rows + cols < n - 1).ravel()
    a, b = rows.ravel(), cols.ravel()
    tri = np.concatenate([
        np.stack([[a, b], [a + 1, b], [a, b + 1]])[:, :, up].transpose(2, 0, 1),
        np.stack([[a + 1, b], [a + 1, b + 1], [a, b + 1]])[:, :, down].transpose(2, 0, 1),
    ])  # (n^2, corner, (i, j)), the third index being n - i - j
    key = np.zeros(len(tri), dtype=np.int64)
    mid = 2 * tri.sum(axis=1) // 3
    for bit in range(12):
        key |= ((mid[:, 0] >> bit) & 1) << (2 * bit)
        key |= ((mid[:, 1] >> bit) & 1) << (2 * bit + 1)
    tri = tri[np.argsort(key, kind="stable")]
    corners = []
    for sx in (1, -1):
        for sy in (1, -1):
            for sz in (1, -1):
                p = np.stack([sx * tri[:, :, 0], sy * tri[:, :, 1], sz * (n - tri[:, :, 0] - tri[:, :, 1])], axis=2)
                corners.append(p if sx * sy * sz > 0 else p[:, ::-1])
    p = np.concatenate(corners).reshape(-1, 3)
    code = ((p[:, 0] + n) * (2 * n + 1) + p[:, 1] + n) * (2 * n + 1) + p[:, 2] + n
    uniq, first, inverse = np.unique(code, return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")  # vertices numbered by first use
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    v = p[first[order]].astype(np.float64)
    v = np.sin(0.5 * np.pi * v / n)  # nearly equal edges after the projection
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return v, rank[inverse.ravel()].reshape(-1, 3)


def _mesh(n, rng):
    """A smooth closed surface: an ellipsoid of about unit size with seeded bumps of a few per cent."""
    v, e = _octahedral_mesh(n)
    radius = np.ones(len(v))
    for _ in range(4):
        d = rng.standard_normal(3)
        radius += 0.02 * np.sin(v @ (2.0 * d / np.linalg.norm(d)) + rng.uniform(0, 2 * np.pi))
    axes = rng.uniform(0.95, 1.05, 3)
    return v * radius[:, None] * axes, e


def _rng(case, seed):
    return np.random.default_rng([int(seed), int(case.get("n", 0)), int(case.get("points", 0))])


def _points(case, rng):
    """Unit directions of a far field, else the points of a slice through the surface and around it."""
    m = case["points"]
    if case["far"]:
        d = rng.standard_normal((3, m))
        return d / np.linalg.norm(d, axis=0)
    p = np.zeros((3, m))
    p[0], p[1] = rng.uniform(-2.5, 2.5, (2, m))
    p[2] = rng.uniform(-0.3, 0.3)
    return p


def _coefficients(count, rng, is_complex=True):
    c = rng.standard_normal(count)
    return c + 1j * rng.standard_normal(count) if is_complex else c


def _batch_inputs(case, seed):
    """Mesh, wavenumber and 8 right-hand sides of each problem of a batch."""
    rng = np.random.default_rng([int(seed), case["count"]])
    out = []
    for i in range(case["count"]):
        # sizes spread over the range, the same ones for every seed
        t = i / max(case["count"] - 1, 1)
        n = int(round(case["n_least"] * (case["n_most"] / case["n_least"]) ** t))
        v, e = _mesh(n, rng)
        out.append((v, e, float(rng.uniform(1.0, 6.0)), _coefficients((len(e), 8), rng)))
    return out


# ------------------------------------------------------------------------------------- the timed calls

_SPACES = {"DP0": ("DP", 0), "P1": ("P", 1), "RWG": ("RWG", 0)}


def _factory_arguments(case):
    """The wavenumber arguments of an operator's factory."""
    if case["equation"] == "laplace":
        return ()
    if case["equation"] == "modified_helmholtz" or case["k_imag"] == 0.0:
        return (case["k"],)
    return (complex(case["k"], case["k_imag"]),)


def _boundary_operator(case, domain, dual):
    group = getattr(operators.boundary, case["equation"])
    extra = _factory_arguments(case)
    interface = case["interface"]
    if case["operator"] == "combined_field":
        dlp = group.double_layer(domain, domain, dual, *extra, device_interface=interface)
        slp = group.single_layer(domain, domain, dual, *extra, device_interface=interface)
        ident = operators.boundary.sparse.identity(domain, domain, dual, device_interface=interface)
        return dlp - 0.5 * ident - 1j * extra[0] * slp
    return getattr(group, case["operator"])(domain, domain, dual, *extra, device_interface=interface)


def _solve_case(case):
    return _operator("helmholtz", "combined_field", "DP0", case["n"], case["k"], interface=case["interface"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        problems = _batch_inputs(case, seed)
        grids = [Grid(v.T, e.T) for v, e, _, _ in problems]
        assembler = BatchAssembler(grids, [k for _, _, k, _ in problems], precision=case["precision"],
                                   kernel=case["kernel"])
        rhs = [torch.as_tensor(b, device="cuda") for _, _, _, b in problems]
        return {"kind": kind, "assembler": assembler, "rhs": rhs, "products": [torch.empty_like(b) for b in rhs]}
    rng = _rng(case, seed)
    v, e = _mesh(case["n"], rng)
    grid = Grid(v.T, e.T)
    if kind == "gradient":
        directions = shape_gradient.fibonacci_directions(case["directions"])
        objective = shape_gradient.FarFieldObjective(grid, directions=directions, solver=case["solver"])
        k = torch.tensor(case["k"], dtype=torch.float64, device="cuda", requires_grad=True)
        return {"kind": kind, "objective": objective, "k": k,
                "vertices": objective.vertices.clone().requires_grad_(True)}
    if kind == "solve":
        space = function_space(grid, "DP", 0)
        operator = _boundary_operator(_solve_case(case), space, space)
        operator.weak_form()
        k = case["k"]
        wave = device_callable(lambda x, n, domain: -torch.exp(1j * k * x[2]))
        return {"kind": kind, "operator": operator, "rhs": GridFunction(space, fun=wave)}
    space = function_space(grid, *_SPACES[case["space"]])
    if kind == "potential":
        group = getattr(operators.far_field if case["far"] else operators.potential, case["equation"])
        points = _points(case, rng)
        real = case["equation"] in ("laplace", "modified_helmholtz")
        coefficients = torch.as_tensor(_coefficients(space.global_dof_count, rng, not real), device="cuda")
        operator = getattr(group, case["operator"])(space, points, *_factory_arguments(case),
                                                    device_interface=case["interface"])
        return {"kind": kind, "operator": operator, "coefficients": coefficients}
    dual = function_space(grid, "SNC", 0) if case["space"] == "RWG" else space
    return {"kind": kind, "case": case, "domain": space, "dual": dual}


def run(state):
    kind = state["kind"]
    if kind == "operator":
        return _boundary_operator(state["case"], state["domain"], state["dual"]).weak_form().tensor
    if kind == "potential":
        return state["operator"].evaluate_device(state["coefficients"])
    if kind == "batch":
        state["assembler"].step(state["rhs"], state["products"])
        return {"matrices": state["assembler"].outputs, "products": state["products"]}
    if kind == "solve":
        solution, _ = linalg.gmres(state["operator"], state["rhs"], tol=1e-8)
        return solution.coefficients
    value = shape_gradient.far_field_objective(state["vertices"], state["k"], state["objective"])
    by_vertices, by_k = torch.autograd.grad(value, (state["vertices"], state["k"]))
    return {"value": value.detach(), "by_vertices": by_vertices, "by_k": by_k}


# ------------------------------------------------------------------------------------------------ work

# floating-point operations of one kernel value at a pair of points (an FMA counts two, a root, a
# quotient, a sine one)
_KERNEL_FLOPS = {"single_layer": 20, "hypersingular": 20, "double_layer": 30, "adjoint_double_layer": 30,
                 "combined_field": 35, "electric_field": 20, "magnetic_field": 28}
_REAL_FLOPS = {"single_layer": 13, "hypersingular": 13, "double_layer": 20, "adjoint_double_layer": 20}


def _dofs(space, n):
    ne = _elements_of(n)
    return {"DP0": ne, "P1": ne // 2 + 2, "RWG": 3 * ne // 2}[space]


def _matrix_work(equation, operator, space, n):
    """Every unordered pair of elements once, at 6 x 6 points, and the sums with the shape functions."""
    ne, dofs = _elements_of(n), _dofs(space, n)
    real = equation in ("laplace", "modified_helmholtz")
    per_point = (_REAL_FLOPS if real else _KERNEL_FLOPS)[operator] + (0 if space == "DP0" else 6 if real else 12)
    return {"bytes": dofs * dofs * (8 if real else 16) + 60 * ne, "flops": 36 * per_point * ne * (ne + 1) // 2}


def work(case):
    kind = case["kind"]
    if kind == "operator":
        return _matrix_work(case["equation"], case["operator"], case["space"], case["n"])
    if kind == "potential":
        ne, m = _elements_of(case["n"]), case["points"]
        maxwell = case["equation"] == "maxwell"
        per_pair = (24 if maxwell else 8) + (12 if case["far"] else 20)
        return {"bytes": 24 * m + 16 * m * (3 if maxwell else 1) + 60 * ne + 16 * _dofs(case["space"], case["n"]),
                "flops": per_pair * 6 * ne * m}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        name = "combined_field" if case["kernel"].endswith("combined_field") else "single_layer"
        for i in range(case["count"]):
            t = i / max(case["count"] - 1, 1)
            n = int(round(case["n_least"] * (case["n_most"] / case["n_least"]) ** t))
            w, ne = _matrix_work("helmholtz", name, "DP0", n), _elements_of(n)
            total["bytes"] += w["bytes"] + 256 * ne
            total["flops"] += w["flops"] + 64 * ne * ne
        return total
    ne = _elements_of(case["n"])
    if kind == "solve":
        # about 50 products with the matrix
        return {"bytes": 50 * 16 * ne * ne, "flops": 50 * 8 * ne * ne}
    w = _matrix_work("helmholtz", "combined_field", "DP0", case["n"])
    # the assembly, its derivative (twice the assembly's work), about 60 products in two solves
    return {"bytes": 61 * w["bytes"], "flops": 3 * w["flops"] + 60 * 8 * ne * ne}


def tolerance(case):
    """Double precision agrees to the rounding of its sums.  Mixed precision evaluates separated pairs in 32
    bits (about 1e-7 of the entries, which cancel in part), iterative solves stop at their residual."""
    if case["kind"] == "solve":
        return {"rel": 4e-7, "max": 1e-5}
    if case["kind"] == "gradient":
        return {"rel": 1e-9, "max": 1e-7}
    mixed = case.get("interface") == "cuda_mixed" or case.get("precision") == "mixed"
    return {"rel": 5e-7, "max": 1e-4} if mixed else {"rel": 1e-12, "max": 1e-10}


# ------------------------------------------------------------------------------------- 64-bit reference

_RULE_A, _RULE_B = 0.445948490915964886, 0.0915762135097707435
_RULE_WA, _RULE_WB = 0.223381589678011466, 0.109951743655321868
_CHUNK = 1 << 21


def _triangle_rule():
    """Barycentric points (6, 3) and weights (sum 1/2) of the degree-4 rule (Strang and Fix; Dunavant)."""
    pts, wts = [], []
    for a, w in ((_RULE_A, _RULE_WA), (_RULE_B, _RULE_WB)):
        for i in range(3):
            p = [a, a, a]
            p[i] = 1.0 - 2.0 * a
            pts.append(p)
            wts.append(0.5 * w)
    return torch.tensor(pts, dtype=torch.float64, device="cuda"), wts


def _touching_rule(adjacency):
    """Sauter-Schwab rule of order 4: barycentric points of both triangles (Q, 3) and weights (Q,)."""
    x, w = np.polynomial.legendre.leggauss(4)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    s, a, b, c = (g.ravel() for g in np.meshgrid(x, x, x, x, indexing="ij"))
    weight = np.prod(np.meshgrid(w, w, w, w, indexing="ij"), axis=0).ravel()
    ab, abc = a * b, a * b * c
    if adjacency == "same":
        weight = weight * s**3 * a**2 * b
        halves = [((s, s * (1 - a + ab)), (s * (1 - abc), s * (1 - a))),
                  ((s, s * (a - ab + abc)), (s * (1 - ab), s * (a - ab))),
                  ((s * (1 - abc), s * (a - abc)), (s, s * (a - ab)))]
        regions = [(t, u, weight) for t, u in halves] + [(u, t, weight) for t, u in halves]
    elif adjacency == "edge":
        weight = weight * s**3 * a**2
        regions = [((s, s * a * c), (s * (1 - ab), s * a * (1 - b)), weight),
                   ((s, s * a), (s * (1 - abc), s * ab * (1 - c)), weight * b),
                   ((s * (1 - ab), s * a * (1 - b)), (s, s * abc), weight * b),
                   ((s * (1 - abc), s * ab * (1 - c)), (s, s * a), weight * b),
                   ((s * (1 - abc), s * a * (1 - b * c)), (s, s * ab), weight * b)]
    else:
        weight = weight * s**3 * b
        one, two = (s, s * a), (s * b, s * b * c)
        regions = [(one, two, weight), (two, one, weight)]

    def barycentric(parts):
        first = np.concatenate([p[0] for p in parts])
        second = np.concatenate([p[1] for p in parts])  # on the triangle (0, 0), (1, 0), (1, 1)
        return torch.as_tensor(np.stack([1 - first, first - second, second], axis=1), device="cuda")

    return (barycentric([r[0] for r in regions]), barycentric([r[1] for r in regions]),
            torch.as_tensor(np.concatenate([r[2] for r in regions]), device="cuda"))


class _Surface(object):
    """Corners, normals and twice the areas of a mesh's elements."""

    def __init__(self, vertices, elements):
        self.vertices = vertices
        self.elements = elements
        self.corners = vertices[elements]  # (ne, 3, 3)
        j0 = self.corners[:, 1] - self.corners[:, 0]
        j1 = self.corners[:, 2] - self.corners[:, 0]
        cross = torch.linalg.cross(j0, j1)
        self.area2 = torch.linalg.vector_norm(cross, dim=1)
        self.normal = cross / self.area2[:, None]

    def points(self, barycentric):
        return torch.einsum("qc,ecd->eqd", barycentric, self.corners)

    def curls(self):
        """Surface curls (ne, 3, 3) of the hat functions: the opposite edge over twice the area."""
        c = self.corners
        edges = torch.stack([c[:, 2] - c[:, 1], c[:, 0] - c[:, 2], c[:, 1] - c[:, 0]], dim=1)
        return -edges / self.area2[:, None, None]

    def rwg(self):
        """(opposite corner (ne, 3, 3), edge length (ne, 3)) of the local edges 01, 20, 12."""
        c = self.corners
        lengths = torch.stack([torch.linalg.vector_norm(c[:, i] - c[:, j], dim=1) for i, j in ((0, 1), (2, 0), (1, 2))],
                              dim=1)
        return c[:, [2, 1, 0]], lengths


def _wavenumber(case):
    if case["equation"] == "laplace":
        return 0.0
    return 1j * case["k"] if case["equation"] == "modified_helmholtz" else complex(case["k"], case["k_imag"])


def _kernel(operator, k, x, y, nx, ny, keep=None):
    """Kernel of an operator at points x, y (broadcast); ``keep``: where it is needed (elsewhere finite)."""
    d = x - y
    r2 = (d * d).sum(-1)
    if keep is not None:
        r2 = torch.where(keep, r2, torch.ones_like(r2))
    r = torch.sqrt(r2)
    if isinstance(k, float) and k == 0.0:
        g, slope = 1.0 / (4.0 * math.pi * r), -1.0
    elif not isinstance(k, torch.Tensor) and complex(k).real == 0.0:
        g, slope = torch.exp(-k.imag * r) / (4.0 * math.pi * r), -k.imag * r - 1.0
    else:
        g, slope = torch.exp(1j * k * r) / (4.0 * math.pi * r), 1j * k * r - 1.0
    if operator in ("single_layer", "hypersingular", "electric_field"):
        return g
    radial = g * slope / r2
    if operator == "magnetic_field":
        return radial
    if operator == "adjoint_double_layer":
        return radial * (d * nx).sum(-1)
    double = -radial * (d * ny).sum(-1)
    return double if operator == "double_layer" else double - 1j * k * g


def _blocks(operator, k, m, surface, test, trial):
    """Local matrices from the moments m (..., i, j) = sum w w K phi_i phi_j of element pairs (without areas);
    ``test``, ``trial`` index the elements, broadcasting over the pairs."""
    areas = surface.area2[test] * surface.area2[trial]
    if operator == "hypersingular":
        curls = surface.curls()
        cc = (curls[test].unsqueeze(-2) * curls[trial].unsqueeze(-3)).sum(-1)
        nn = (surface.normal[test] * surface.normal[trial]).sum(-1)[..., None, None]
        return areas[..., None, None] * (cc * m.sum((-1, -2), keepdim=True) - k * k * nn * m)
    if operator in ("electric_field", "magnetic_field"):
        apex, length = surface.rwg()
        ct, cs, at, as_ = surface.corners[test], surface.corners[trial], apex[test], apex[trial]
        scale = length[test].unsqueeze(-1) * length[trial].unsqueeze(-2)
        total = 0.0
        for a in range(3):
            u = ct[..., a, :].unsqueeze(-2) - at  # (..., i, 3)
            for b in range(3):
                v = cs[..., b, :].unsqueeze(-2) - as_
                ui, vj = u.unsqueeze(-2), v.unsqueeze(-3)
                if operator == "electric_field":
                    f = (ui * vj).sum(-1)
                else:
                    cross = torch.linalg.cross(*torch.broadcast_tensors(ui, vj))
                    f = ((at.unsqueeze(-2) - as_.unsqueeze(-3)) * cross).sum(-1)
                total = total + m[..., a, b][..., None, None] * f
        if operator == "electric_field":
            total = -1j * k * total - 4.0 / (1j * k) * m.sum((-1, -2), keepdim=True)
        return scale * total
    return areas[..., None, None] * m


def _regular_blocks(operator, k, surface, rows, one, phi, weights, points):
    """Local matrices of the element pairs (rows, all), zero where the elements touch."""
    e = surface.elements
    touch = (e[rows][:, None, :, None] == e[None, :, None, :]).flatten(2).any(-1)
    m = 0.0
    for p in range(6):
        t = 0.0
        for q in range(6):
            kv = _kernel(operator, k, points[rows][:, p].unsqueeze(1), points[:, q].unsqueeze(0),
                         surface.normal[rows].unsqueeze(1), surface.normal.unsqueeze(0), ~touch)
            t = t + weights[q] * kv.unsqueeze(-1) * (phi[q] if not one else torch.ones(1, device="cuda"))
        f = phi[p].reshape(3, 1) if not one else torch.ones((1, 1), device="cuda")
        m = m + weights[p] * t.unsqueeze(-2) * f
    m = torch.where(touch[..., None, None], torch.zeros_like(m), m)
    everyone = torch.arange(len(e), device="cuda")
    return _blocks(operator, k, m, surface, rows[:, None], everyone[None, :])


def _touching_pairs(elements):
    """(rule, test, trial, corner orders (pairs, 3) of both) of the touching pairs.  The shared corners come
    first: ascending in the trial element for a shared edge; for one shared corner, it trades places with
    corner 0."""
    e = elements.cpu().numpy()
    ne = len(e)
    users = np.argsort(e.ravel(), kind="stable") // 3
    counts = np.bincount(e.ravel())
    starts = np.concatenate([[0], np.cumsum(counts)])
    most = counts.max()
    table = np.full((len(counts), most), -1)
    for j in range(most):
        has = counts > j
        table[has, j] = users[starts[:-1][has] + j]
    near = table[e].reshape(ne, -1)
    t = np.repeat(np.arange(ne), near.shape[1])
    s = near.ravel()
    pairs = np.unique(t[s >= 0] * ne + s[s >= 0])
    t, s = pairs // ne, pairs % ne
    same = e[t][:, :, None] == e[s][:, None, :]
    shared = same.any(2).sum(1)
    out = []
    pick = shared == 3
    plain = np.tile(np.arange(3), (pick.sum(), 1))
    out.append(("same", t[pick], s[pick], plain, plain))
    pick = shared == 2
    eq = same[pick]
    j = np.argsort(~eq.any(1), axis=1, kind="stable")[:, :2]  # shared corners of the trial element, ascending
    i = eq.argmax(1)[np.arange(len(j))[:, None], j]
    out.append(("edge", t[pick], s[pick], np.concatenate([i, 3 - i.sum(1, keepdims=True)], 1),
                np.concatenate([j, 3 - j.sum(1, keepdims=True)], 1)))
    pick = shared == 1
    swap = np.array([[0, 1, 2], [1, 0, 2], [2, 1, 0]])
    flat = same[pick].reshape(-1, 9).argmax(1)
    out.append(("vertex", t[pick], s[pick], swap[flat // 3], swap[flat % 3]))
    return out


def _touching_blocks(operator, k, surface, one):
    """(test, trial, local matrices) of the touching pairs, in chunks."""
    for rule, t, s, pt, ps in _touching_pairs(surface.elements):
        bt, bs, w = _touching_rule(rule)
        step = max(1, _CHUNK // len(w))
        for lo in range(0, len(t), step):
            ti, si, pti, psi = (torch.as_tensor(a[lo:lo + step], device="cuda") for a in (t, s, pt, ps))
            ct = torch.gather(surface.corners[ti], 1, pti[:, :, None].expand(-1, -1, 3))
            cs = torch.gather(surface.corners[si], 1, psi[:, :, None].expand(-1, -1, 3))
            x, y = torch.einsum("qc,pcd->pqd", bt, ct), torch.einsum("qc,pcd->pqd", bs, cs)
            kv = w * _kernel(operator, k, x, y, surface.normal[ti][:, None], surface.normal[si][:, None])
            if one:
                m = kv.sum(1)[:, None, None]
            else:
                m = torch.einsum("pq,qi,qj->pij", kv, bt.to(kv.dtype), bs.to(kv.dtype))
                m = torch.gather(m, 1, torch.argsort(pti, 1)[:, :, None].expand(-1, -1, 3))
                m = torch.gather(m, 2, torch.argsort(psi, 1)[:, None, :].expand(-1, 3, -1))
            yield ti, si, _blocks(operator, k, m, surface, ti, si)


def _dof_map(space, elements):
    """(ne, nshape) dof numbers and signs, and the dof count."""
    ne = len(elements)
    if space == "DP0":
        return torch.arange(ne, device="cuda")[:, None], torch.ones((ne, 1), device="cuda", dtype=torch.float64), ne
    if space == "P1":
        return elements, torch.ones((ne, 3), device="cuda", dtype=torch.float64), int(elements.max()) + 1
    e = elements.cpu().numpy()
    pairs = np.sort(np.stack([e[:, [0, 1]], e[:, [2, 0]], e[:, [1, 2]]], axis=1), axis=2).reshape(-1, 2)
    _, first, inverse = np.unique(pairs[:, 0] * ne + pairs[:, 1], return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")  # edges numbered by first visit
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    sign = -np.ones(3 * ne)
    sign[first] = 1.0  # positive on the element that comes first
    return (torch.as_tensor(rank[inverse.ravel()].reshape(ne, 3), device="cuda"),
            torch.as_tensor(sign.reshape(ne, 3), device="cuda"), len(first))


def _exact_matrix(operator, k, space, vertices, elements):
    surface = _Surface(torch.as_tensor(vertices, device="cuda"), torch.as_tensor(elements, device="cuda"))
    one = space == "DP0"
    dofs, signs, count = _dof_map(space, surface.elements)
    real = complex(k).real == 0.0
    out = torch.zeros((count, count), dtype=torch.float64 if real else torch.complex128, device="cuda")
    phi, weights = _triangle_rule()
    points = surface.points(phi)
    ne = len(elements)
    step = max(1, _CHUNK // (ne * (1 if one else 3)))
    for lo in range(0, ne, step):
        rows = torch.arange(lo, min(ne, lo + step), device="cuda")
        block = _regular_blocks(operator, k, surface, rows, one, phi, weights, points)
        block = block.real if real and block.is_complex() else block
        block = block * (signs[rows][:, None, :, None] * signs[None, :, None, :])
        if one:
            out[rows] += block[..., 0, 0]
            continue
        for i in range(3):
            row = torch.zeros((len(rows), count), dtype=out.dtype, device="cuda")
            for j in range(3):
                row.index_add_(1, dofs[:, j], block[..., i, j].to(out.dtype))
            out.index_add_(0, dofs[rows, i], row)
    for t, s, block in _touching_blocks(operator, k, surface, one):
        block = (block.real if real and block.is_complex() else block) * (signs[t][:, :, None] * signs[s][:, None, :])
        index = dofs[t][:, :, None] * count + dofs[s][:, None, :]
        out.view(-1).index_add_(0, index.reshape(-1), block.to(out.dtype).reshape(-1))
    return out


def _combined_matrix(k, vertices, elements):
    out = _exact_matrix("combined_field", k, "DP0", vertices, elements)
    surface = _Surface(torch.as_tensor(vertices, device="cuda"), torch.as_tensor(elements, device="cuda"))
    out.diagonal().sub_(0.25 * surface.area2)
    return out


def _exact_potential(case, seed):
    rng = _rng(case, seed)
    vertices, elements = _mesh(case["n"], rng)
    x = torch.as_tensor(_points(case, rng).T.copy(), device="cuda")
    surface = _Surface(torch.as_tensor(vertices, device="cuda"), torch.as_tensor(elements, device="cuda"))
    dofs, signs, count = _dof_map(case["space"], surface.elements)
    real = case["equation"] in ("laplace", "modified_helmholtz")
    c = torch.as_tensor(_coefficients(count, rng, not real), device="cuda")
    local = c[dofs] * signs
    k = _wavenumber(case)
    phi, weights = _triangle_rule()
    w = torch.tensor(weights, dtype=torch.float64, device="cuda")
    y = surface.points(phi)  # (ne, 6, 3)
    ny = surface.normal[:, None].expand_as(y).reshape(-1, 3)
    maxwell = case["equation"] == "maxwell"
    if maxwell:
        apex, length = surface.rwg()
        f = w[None, :, None] * (local * length)[:, None, :]  # (ne, 6, i)
        v = (f[..., None] * (y[:, :, None] - apex[:, None])).sum(2).reshape(-1, 3)
        div = 2.0 * f.sum(2).reshape(-1)
    elif case["space"] == "DP0":
        density = (w[None] * surface.area2[:, None] * local).reshape(-1)
    else:
        density = (w[None] * surface.area2[:, None] * (local @ phi.T.to(local.dtype))).reshape(-1)
    y = y.reshape(-1, 3)
    out = torch.zeros((3 if maxwell else 1, len(x)), dtype=torch.complex128, device="cuda")
    name = case["operator"]
    step = max(1, _CHUNK // len(y))
    for lo in range(0, len(x), step):
        p = x[lo:lo + step]
        if case["far"]:
            g = torch.exp(-1j * k.real * (p @ y.T)) / (4.0 * math.pi)
            if not maxwell:
                g = g * (-1j * k.real * (p @ ny.T)) if name == "double_layer" else g
                out[0, lo:lo + step] = g @ density
            else:
                field = 1j * k * (g @ v)
                if name == "electric_field":
                    field = field - p * (g @ div)[:, None]
                else:
                    field = torch.linalg.cross(p.to(field.dtype), field)
                out[:, lo:lo + step] = field.T
            continue
        if not maxwell:
            g = _kernel(name, k, p[:, None], y[None], None, ny[None])
            out[0, lo:lo + step] = g.to(torch.complex128) @ density.to(torch.complex128)
            continue
        radial = _kernel("magnetic_field", k, p[:, None], y[None], None, None)
        sums = torch.stack([radial @ (y[:, i, None] * v) for i in range(3)], dim=1)  # (m, i, d): sum y_i v_d
        if name == "magnetic_field":
            m = p[:, :, None] * (radial @ v)[:, None] - sums  # d_i v_d
            field = torch.stack([m[:, 1, 2] - m[:, 2, 1], m[:, 2, 0] - m[:, 0, 2], m[:, 0, 1] - m[:, 1, 0]], dim=1)
        else:
            g = _kernel("single_layer", k, p[:, None], y[None], None, None)
            d = p * (radial @ div)[:, None] - radial @ (y * div[:, None])
            field = 1j * k * (g @ v) - d / (1j * k)
        out[:, lo:lo + step] = field.T
    return out


def _exact_gradient(case, seed):
    """The objective, its adjoint, and autograd through the adjoint's contractions, a few rows at a time."""
    vertices, elements = _mesh(case["n"], _rng(case, seed))
    directions = torch.as_tensor(_spiral(case["directions"]), device="cuda")
    e = torch.as_tensor(elements, device="cuda")
    v = torch.as_tensor(vertices, device="cuda").requires_grad_(True)
    k = torch.tensor(case["k"], dtype=torch.float64, device="cuda", requires_grad=True)
    phi, weights = _triangle_rule()
    w = torch.tensor(weights, dtype=torch.float64, device="cuda")

    def ends():
        """Right-hand side and far-field matrix."""
        surface = _Surface(v, e)
        y = surface.points(phi)
        scale = w[None] * surface.area2[:, None]
        b = -(scale * torch.exp(1j * k * y[..., 2])).sum(1)
        g = torch.exp(-1j * k * torch.einsum("jd,eqd->jeq", directions, y)) / (4.0 * math.pi)
        f = (scale[None] * g).sum(2) * (-1j * k * (directions @ surface.normal.T) - 1j * k)
        return b, f

    with torch.no_grad():
        a = _combined_matrix(case["k"], vertices, elements)
        b, f = ends()
        density = torch.linalg.solve(a, b)
        u = f @ density
        adjoint = torch.linalg.solve(a.mH, f.mH @ u)
        value = (u.abs() ** 2).sum()
        del a
    b, f = ends()
    (2.0 * ((u.conj() * (f @ density)).sum() + (adjoint.conj() * b).sum()).real).backward()
    ne = len(e)
    step = max(1, (1 << 17) // ne)
    for lo in range(0, ne, step):
        surface = _Surface(v, e)
        rows = torch.arange(lo, min(ne, lo + step), device="cuda")
        block = _regular_blocks("combined_field", k, surface, rows, True, phi, weights, surface.points(phi))
        rest = (adjoint[rows].conj() * (-0.25 * surface.area2[rows]) * density[rows]).sum()
        (-2.0 * (adjoint[rows].conj() @ (block[..., 0, 0] @ density) + rest).real).backward()
    surface = _Surface(v, e)
    for t, s, block in _touching_blocks("combined_field", k, surface, True):
        (-2.0 * (adjoint[t].conj() * block[:, 0, 0] * density[s]).sum().real).backward(retain_graph=True)
    return {"value": value, "by_vertices": v.grad, "by_k": k.grad}


def _spiral(count):
    """Unit directions on a golden-angle spiral (count, 3)."""
    i = np.arange(count) + 0.5
    z = 1.0 - 2.0 * i / count
    angle = math.pi * (1.0 + math.sqrt(5.0)) * i
    rho = np.sqrt(1.0 - z * z)
    return np.stack([rho * np.cos(angle), rho * np.sin(angle), z], axis=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        return _exact_gradient(case, seed)
    with torch.no_grad():
        if kind == "potential":
            return _exact_potential(case, seed)
        if kind == "batch":
            problems = _batch_inputs(case, seed)
            combined = case["kernel"].endswith("combined_field")
            matrices = [_exact_matrix("combined_field" if combined else "single_layer", complex(k), "DP0", v, e)
                        for v, e, k, _ in problems]
            return {"matrices": matrices,
                    "products": [a @ torch.as_tensor(b, device="cuda") for a, (_, _, _, b) in zip(matrices, problems)]}
        vertices, elements = _mesh(case["n"], _rng(case, seed))
        if kind == "solve":
            matrix = _combined_matrix(complex(case["k"]), vertices, elements)
            surface = _Surface(torch.as_tensor(vertices, device="cuda"), torch.as_tensor(elements, device="cuda"))
            phi, weights = _triangle_rule()
            w = torch.tensor(weights, dtype=torch.float64, device="cuda")
            rhs = -(w * surface.area2[:, None] * torch.exp(1j * case["k"] * surface.points(phi)[..., 2])).sum(1)
            return torch.linalg.solve(matrix, rhs).cpu().numpy()
        if case["operator"] == "combined_field":
            return _combined_matrix(_wavenumber(case), vertices, elements)
        return _exact_matrix(case["operator"], _wavenumber(case), case["space"], vertices, elements)
