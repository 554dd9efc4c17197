"""Grids and spaces that have been used on the device can be copied and pickled: the copies' argument records point at
the copies' own tensors (device.py).  The device objects are filled with host tensors here; the GPU test goes
through whole calls."""

import copy
import gc
import pickle

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _grid_with_copies():
    """A grid whose cache holds a device grid, space and singular rule made of host tensors."""
    from bempp_cuda import device
    from bempp_cuda.shapes import ellipsoid

    grid = ellipsoid(0, 1.0, 1.0, 1.0)
    dgrid = device.DeviceGrid.__new__(device.DeviceGrid)
    dgrid.nvertices, dgrid.nelements, dgrid.radius = 6, 8, 1.0
    dgrid.geom, dgrid.elements = torch.zeros(25, 8, dtype=torch.float64), torch.zeros(8, 3, dtype=torch.int32)
    space = device.DeviceSpace.__new__(device.DeviceSpace)
    space.shapeset, space.nshape, space.nsupport, space.ndofs, space.dof_is_position = 0, 1, 8, 8, 1
    space.support, space.l2g = torch.arange(8, dtype=torch.int32), torch.arange(8, dtype=torch.int32).reshape(8, 1)
    space.mult, space.normal_mult = torch.ones(8, 1, dtype=torch.float64), torch.ones(8, dtype=torch.int32)
    rule = device.DeviceSingularRule.__new__(device.DeviceSingularRule)
    rule.npairs, rule.npoints_table, rule.nweights, rule._by_test = 4, 5, 6, None
    for name in ("test_points", "trial_points", "weights"):
        setattr(rule, name, torch.zeros(6, dtype=torch.float64))
    for name in ("test_elements", "trial_elements", "test_offsets", "trial_offsets", "weights_offsets", "npoints"):
        setattr(rule, name, torch.zeros(4, dtype=torch.int32))
    for obj in (dgrid, space, rule):
        obj._point_at_tensors()
    device._cache(grid).update({"grid": dgrid, "space": space, "rule": rule})
    return grid


@pytest.mark.parametrize("make", [copy.deepcopy, lambda g: pickle.loads(pickle.dumps(g))], ids=["copy", "pickle"])
def test_records_follow_their_tensors(make):
    from bempp_cuda import _lib, device

    grid = _grid_with_copies()
    cache, old = device._cache(make(grid)), device._cache(grid)
    dgrid, space, rule = cache["grid"], cache["space"], cache["rule"]
    assert dgrid.geom.data_ptr() != old["grid"].geom.data_ptr()
    assert dgrid.record().geom == dgrid.geom.data_ptr() and dgrid.record().elements == dgrid.elements.data_ptr()
    assert dgrid.record().nelements == 8
    record = space.record()
    for name in ("support", "l2g", "mult", "normal_mult"):
        assert getattr(record, name) == getattr(space, name).data_ptr()
    assert (record.nsupport, record.ndofs, record.dof_is_position) == (8, 8, 1)
    args = _lib.SingularArgs()
    rule.fill(args)
    assert args.npairs == 4 and args.npoints_table == 5 and args.nweights == 6
    for name in ("test_points", "trial_points", "weights", "test_elements", "trial_elements", "test_offsets",
                 "trial_offsets", "weights_offsets", "npoints"):
        assert getattr(args, name) == getattr(rule, name).data_ptr()


@pytest.mark.gpu
def test_copied_space_assembles():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bempp_cuda import operators
    from bempp_cuda.shapes import ellipsoid
    from bempp_cuda.space import function_space

    single = operators.boundary.helmholtz.single_layer
    space = function_space(ellipsoid(2, 1.0, 0.8, 1.2), "DP", 0)
    ref = single(space, space, space, 1.5).weak_form().A
    twin = copy.deepcopy(space)
    other = pickle.loads(pickle.dumps(space))
    del space
    gc.collect()
    torch.cuda.empty_cache()
    for s in (twin, other):
        np.testing.assert_allclose(single(s, s, s, 1.5).weak_form().A, ref, rtol=0, atol=1e-15 * abs(ref).max())
