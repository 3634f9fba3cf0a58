"""Batches whose instances differ in what the fused step's kernels are chosen
by: each instance's state has the bits of a model of that mesh alone with the
same patch_elements."""
import numpy as np
import pytest

from akantu_b200 import _abi, mesh as mesh_mod
from akantu_b200.batch import BatchModel
from akantu_b200.model import SolidMechanicsModel, material_from_dict

pytestmark = pytest.mark.gpu

STATE = (_abi.FIELD_DISPLACEMENT, _abi.FIELD_VELOCITY, _abi.FIELD_ACCELERATION)
SMALL = dict(kind=_abi.MATERIAL_ELASTIC, rho=2.0, E=100.0, nu=0.3)
FINITE = dict(kind=_abi.MATERIAL_ELASTIC, rho=2.0, E=90.0, nu=0.25, finite_deformation=True)
NEOHOOKEAN = dict(kind=_abi.MATERIAL_NEOHOOKEAN, rho=2.0, E=80.0, nu=0.2)


def compare(meshes, materials, opts, steps=40):
    rng = np.random.default_rng(5)
    u0 = [1e-3 * rng.normal(size=m.nodes.shape) for m in meshes]
    b = BatchModel(meshes, [material_from_dict(m) for m in materials], precision=_abi.MODE_FP64,
                   **opts)
    b.initFull()
    b.setField(_abi.FIELD_DISPLACEMENT, np.concatenate(u0))
    dts = 0.5 * np.asarray(b.getStableTimeSteps())
    b.setTimeSteps(dts)
    b.solveSteps(steps)
    got = {f: b.getField(f) for f in STATE}
    for k, mesh in enumerate(meshes):
        m = SolidMechanicsModel(mesh, [material_from_dict(materials[k])],
                                precision=_abi.MODE_FP64, **opts)
        m.initFull()
        m.setField(_abi.FIELD_DISPLACEMENT, u0[k])
        m.setTimeStep(dts[k])
        m.solveSteps(steps)
        for f in STATE:
            want = m.getField(f)
            assert np.isfinite(want).all()
            assert np.array_equal(got[f][b.instance_rows(k)], want), (k, f)
        m.close()
    b.close()


@pytest.mark.parametrize("patch_elements", [128, 300, 512])
def test_small_strain_plates_beside_other_laws(patch_elements):
    meshes = [mesh_mod.plate_triangle3(nx, ny, 0.1 * nx, 0.1 * ny)
              for nx, ny in ((30, 20), (7, 3), (41, 9), (25, 17))]
    laws = [SMALL, FINITE, dict(SMALL, plane_stress=True, E=70.0), NEOHOOKEAN]
    compare(meshes, laws, dict(patch_elements=patch_elements))
    compare(meshes[:3:2], laws[:3:2], dict(patch_elements=patch_elements))


@pytest.mark.parametrize("patch_elements", [768, 1536])
def test_small_strain_boxes_beside_other_laws(patch_elements):
    meshes = [mesh_mod.box_tetrahedron4(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
              for nx, ny, nz in ((9, 8, 7), (2, 3, 1), (6, 5, 11))]
    compare(meshes, [SMALL, FINITE, SMALL], dict(patch_elements=patch_elements))
    compare(meshes, [SMALL, NEOHOOKEAN, FINITE], dict(patch_elements=patch_elements))


def distorted_block(nx, ny, nz, seed):
    m = mesh_mod.box_hexahedron8(nx, ny, nz, 0.1 * nx, 0.1 * ny, 0.1 * nz)
    nodes = m.nodes + 0.015 * np.random.default_rng(seed).uniform(-1, 1, m.nodes.shape)
    return mesh_mod.Mesh(3, _abi.HEXAHEDRON_8, nodes, m.connectivity)


@pytest.mark.parametrize("patch_elements", [0, 100, 256])
def test_blocks_of_parallelepipeds_beside_others(patch_elements):
    """Undistorted, distorted and partly distorted blocks of hexahedra."""
    sheared = mesh_mod.box_hexahedron8(5, 7, 6, 0.5, 0.7, 0.6)
    sheared = mesh_mod.Mesh(3, _abi.HEXAHEDRON_8,
                            sheared.nodes @ np.array([[1, 0, 0], [0.3, 1, 0], [0.1, -0.2, 1]]),
                            sheared.connectivity)
    meshes = [mesh_mod.box_hexahedron8(7, 6, 9, 0.7, 0.6, 0.9), distorted_block(6, 5, 8, 1), sheared]
    compare(meshes, [NEOHOOKEAN, SMALL, FINITE], dict(patch_elements=patch_elements))
    compare(meshes, [SMALL, NEOHOOKEAN, NEOHOOKEAN], dict(patch_elements=patch_elements))
