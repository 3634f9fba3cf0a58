"""The reference-order element kernel moves its rows through shared memory a
warp's 32 elements at a time: element counts around its tiles, bit for bit
against the oracle (elastic), gradients and stresses included."""
import numpy as np
import pytest

from akantu_b200 import _abi
from akantu_b200.mesh import (bar_segment2, box_hexahedron8, box_tetrahedron4, plate_triangle3)
from tests.golden_cases import OracleAdapter

pytestmark = pytest.mark.gpu

MESHES = [lambda: bar_segment2(2), lambda: bar_segment2(34), lambda: bar_segment2(130),
          lambda: plate_triangle3(1, 1, 1.0, 1.0), lambda: plate_triangle3(16, 1, 4.0, 1.0),
          lambda: plate_triangle3(13, 5, 2.0, 1.0), lambda: box_tetrahedron4(1, 1, 1, 1., 1., 1.),
          lambda: box_tetrahedron4(3, 1, 2, 3., 1., 2.), lambda: box_tetrahedron4(4, 4, 3, 1., 1., 1.),
          lambda: box_hexahedron8(1, 1, 1, 1., 1., 1.), lambda: box_hexahedron8(31, 1, 1, 31., 1., 1.),
          lambda: box_hexahedron8(5, 5, 5, 1., 1., 1.)]


@pytest.mark.parametrize("k", range(len(MESHES)))
def test_bitwise_at_tile_edges(k):
    from akantu_b200.model import MaterialElastic, SolidMechanicsModel
    mesh = MESHES[k]()
    x = np.asarray(mesh.nodes)
    rng = np.random.default_rng(k)
    u0 = 1e-3 * rng.normal(size=x.shape)
    v0 = rng.normal(size=x.shape)
    mat = dict(kind=_abi.MATERIAL_ELASTIC, rho=2700.0, E=70e9, nu=0.3)
    cpu = OracleAdapter(mesh, mat)
    dev = SolidMechanicsModel(mesh, [MaterialElastic(rho=2700.0, E=70e9, nu=0.3)])
    dev.initFull()
    dt = 0.3 * dev.getStableTimeStep()
    dev.setTimeStep(dt)
    cpu.set_time_step(dt)
    for f, v in ((_abi.FIELD_DISPLACEMENT, u0), (_abi.FIELD_VELOCITY, v0)):
        dev.setField(f, v)
        cpu.set(f, v)
    dev.solveSteps(5)
    cpu.solve_steps(5)
    for f in (_abi.FIELD_DISPLACEMENT, _abi.FIELD_VELOCITY, _abi.FIELD_ACCELERATION,
              _abi.FIELD_INTERNAL_FORCE):
        assert np.array_equal(dev.getField(f), cpu.get(f)), f
    dev.close()


@pytest.mark.parametrize("k", range(len(MESHES)))
def test_the_step_leaves_its_gradients_and_stresses(k):
    """grad u and the stress as the step's element kernel writes them (read in
    place: a copy to the host computes them anew), bit for bit."""
    import torch
    from akantu_b200.model import MaterialElastic, SolidMechanicsModel
    mesh = MESHES[k]()
    x = np.asarray(mesh.nodes)
    rng = np.random.default_rng(100 + k)
    v0 = rng.normal(size=x.shape)
    cpu = OracleAdapter(mesh, dict(kind=_abi.MATERIAL_ELASTIC, rho=2700.0, E=70e9, nu=0.3))
    dev = SolidMechanicsModel(mesh, [MaterialElastic(rho=2700.0, E=70e9, nu=0.3)])
    dev.initFull()
    dt = 0.3 * dev.getStableTimeStep()
    dev.setTimeStep(dt)
    cpu.set_time_step(dt)
    dev.setField(_abi.FIELD_VELOCITY, v0)
    cpu.set(_abi.FIELD_VELOCITY, v0)
    views = {f: dev.deviceTensor(f) for f in (_abi.FIELD_GRAD_U, _abi.FIELD_STRESS)}
    for t in views.values():
        t.fill_(7.0)
    torch.cuda.synchronize()
    dev.solveSteps(3)
    dev.synchronize()
    cpu.solve_steps(3)
    for f, t in views.items():
        rows = t.transpose(1, 2).reshape(t.shape[0], -1).cpu().numpy()  # column-major again
        assert np.array_equal(rows, np.asarray(cpu.get(f)).reshape(rows.shape)), f
    dev.close()


@pytest.mark.parametrize("n", [(2, 1, 1), (8, 4, 1), (11, 3, 1), (6, 4, 2), (7, 7, 1)])
def test_few_hexahedra(n):
    """Up to 48 hexahedra the lanes move their own rows: either side of the change
    and of a warp, bit for bit, the step's gradients and stresses included."""
    import torch
    from akantu_b200.model import MaterialElastic, SolidMechanicsModel
    mesh = box_hexahedron8(*n, *[0.5 * k for k in n])
    mat = dict(kind=_abi.MATERIAL_ELASTIC, rho=2700.0, E=70e9, nu=0.3)
    rng = np.random.default_rng(sum(n))
    v0 = rng.normal(size=np.asarray(mesh.nodes).shape)
    cpu = OracleAdapter(mesh, mat)
    dev = SolidMechanicsModel(mesh, [MaterialElastic(rho=2700.0, E=70e9, nu=0.3)])
    dev.initFull()
    dt = 0.3 * dev.getStableTimeStep()
    dev.setTimeStep(dt)
    cpu.set_time_step(dt)
    dev.setField(_abi.FIELD_VELOCITY, v0)
    cpu.set(_abi.FIELD_VELOCITY, v0)
    views = {f: dev.deviceTensor(f) for f in (_abi.FIELD_GRAD_U, _abi.FIELD_STRESS)}
    dev.solveSteps(5)
    dev.synchronize()
    cpu.solve_steps(5)
    for f, t in views.items():
        rows = t.transpose(1, 2).reshape(t.shape[0], -1).cpu().numpy()
        assert np.array_equal(rows, np.asarray(cpu.get(f)).reshape(rows.shape)), f
    for f in (_abi.FIELD_DISPLACEMENT, _abi.FIELD_VELOCITY, _abi.FIELD_ACCELERATION,
              _abi.FIELD_INTERNAL_FORCE):
        assert np.array_equal(dev.getField(f), cpu.get(f)), f
    dev.close()
