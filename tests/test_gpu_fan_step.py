"""The fan step's branches at the sizes where they can go wrong, against the
CPU oracle: one element to a few patches, affine and distorted hexahedra in
one mesh or apart, several materials in a patch, external forces (the finish
with f_ext), a persistent grid of one CTA, and plans too large for an SM (the
chunk records). Tolerance: FP64 <= 1e-10 of the field's maximum
(test_gpu_patch_layout.py)."""
import numpy as np
import pytest

from akantu_b200 import _abi, configs
from akantu_b200.mesh import box_hexahedron8, box_tetrahedron4, plate_triangle3
from oracle.oracle import OracleModel, material_desc
from tests.golden_cases import OracleAdapter

pytestmark = pytest.mark.gpu

NEO = configs.neohookean_from_lame(1.0e6, 0.4e6, 1100.0)
ELASTIC = dict(kind=_abi.MATERIAL_ELASTIC, rho=2700.0, E=70e9, nu=0.33)
STIFF = dict(kind=_abi.MATERIAL_ELASTIC, rho=7800.0, E=210e9, nu=0.3)
FINITE = dict(kind=_abi.MATERIAL_ELASTIC, rho=2700.0, E=70e9, nu=0.33, finite_deformation=True)


def build(kind, n, jitter):
    mesh = {"hex": lambda: box_hexahedron8(*n, *[0.1 * k for k in n]),
            "tet": lambda: box_tetrahedron4(*n, *[0.1 * k for k in n]),
            "tri": lambda: plate_triangle3(n[0], n[1], 0.1 * n[0], 0.1 * n[1])}[kind]()
    if jitter:  # moves the nodes of the right half only: affine elements remain
        x = mesh.nodes
        rng = np.random.default_rng(1)
        move = x[:, 0] > 0.05 * n[0]
        x[move] += rng.uniform(-0.01, 0.01, x[move].shape)
    return mesh


CASES = [
    ("hex", (1, 1, 1), NEO, 0, {}), ("hex", (3, 2, 1), NEO, 1, {}), ("hex", (9, 8, 7), NEO, 0, {}),
    ("hex", (11, 7, 5), NEO, 1, {}), ("hex", (6, 5, 9), ELASTIC, 1, dict(patch_grid=1)),
    ("hex", (8, 8, 8), NEO, 0, dict(patch_elements=512, patch_nodes=800)),
    ("tet", (1, 1, 1), ELASTIC, 0, {}), ("tet", (7, 6, 5), [ELASTIC, STIFF], 1, {}),
    ("tet", (9, 9, 4), FINITE, 0, dict(patch_grid=1)), ("tet", (10, 9, 8), ELASTIC, 1,
                                                       dict(patch_elements=1, patch_nodes=8)),
    ("tri", (1, 1), ELASTIC, 0, {}), ("tri", (40, 31), [STIFF, ELASTIC], 1, {}),
    ("tri", (64, 3), FINITE, 1, dict(patch_elements=100, patch_nodes=90, patch_grid=1)),
    ("tri", (60, 60), ELASTIC, 0, dict(patch_elements=8000, patch_nodes=6000)),
]


@pytest.mark.parametrize("load", [False, True], ids=["free", "loaded"])
@pytest.mark.parametrize("kind,n,mats,jitter,patch", CASES)
def test_against_oracle(kind, n, mats, jitter, patch, load):
    from akantu_b200.model import SolidMechanicsModel, material_from_dict
    mesh = build(kind, n, jitter)
    mats = mats if isinstance(mats, list) else [mats]
    em = None if len(mats) == 1 else (np.arange(mesh.getNbElement()) % 3 == 0).astype(np.uint32)
    x = mesh.nodes
    rng = np.random.default_rng(2)
    blocked = np.zeros(x.shape, dtype=np.uint8)
    blocked[np.isclose(x[:, 0], 0.0)] = 1
    v0 = rng.normal(0.0, 0.05 if mats[0] is NEO else 1.0, x.shape)
    v0[blocked != 0] = 0.0
    fext = np.zeros(x.shape)
    if load:
        fext[np.isclose(x[:, 0], x[:, 0].max()), 0] = 1e-5 * mats[0]["E"] * 0.01
    cpu = OracleAdapter(mesh, mats)
    if em is not None:
        cpu.m = OracleModel(mesh, [material_desc(**m) for m in mats], em)
    dev = SolidMechanicsModel(mesh, [material_from_dict(m) for m in mats], element_material=em,
                              precision=_abi.MODE_FP64, **patch)
    dev.initFull()
    dt = 0.5 * dev.getStableTimeStep()
    dev.setBlockedDOFs(blocked)
    dev.setField(_abi.FIELD_VELOCITY, v0)
    dev.setField(_abi.FIELD_EXTERNAL_FORCE, fext)
    dev.setTimeStep(dt)
    cpu.set_blocked(blocked)
    cpu.set(_abi.FIELD_VELOCITY, v0)
    cpu.set(_abi.FIELD_EXTERNAL_FORCE, fext)
    cpu.set_time_step(dt)
    dev.solveSteps(40)
    cpu.solve_steps(40)
    for f in (_abi.FIELD_DISPLACEMENT, _abi.FIELD_VELOCITY):
        a, b = np.array(dev.getField(f)), cpu.get(f)
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max(), f
    v = np.array(dev.getVelocity())
    m = np.array(dev.getMass())
    assert dev.getEnergy("kinetic") == pytest.approx(0.5 * (m * v * v).sum(), rel=1e-12)
    dev.close()


def test_a_patch_above_an_sm_is_refused():
    """4913 nodes in one patch: neither the fan record's staging nor the chunk
    records' fits 227 KB."""
    from akantu_b200._lib import AkbError
    from akantu_b200.model import SolidMechanicsModel, material_from_dict
    m = SolidMechanicsModel(box_hexahedron8(16, 16, 16, 1.6, 1.6, 1.6), [material_from_dict(NEO)],
                            precision=_abi.MODE_FP64, patch_elements=4096, patch_nodes=6000)
    with pytest.raises(AkbError, match="shared memory"):
        m.initFull()


@pytest.mark.parametrize("kind,n,mats,patch", [
    ("tri", (33, 31), ELASTIC, {}), ("tri", (32, 32), ELASTIC, {}),
    ("tet", (127, 1, 1), ELASTIC, {}), ("tet", (8, 4, 4), ELASTIC, {}),
    ("tri", (60, 20), ELASTIC, dict(patch_elements=768)),
    ("tri", (60, 20), ELASTIC, dict(patch_elements=769)),
    ("tet", (9, 8, 6), ELASTIC, dict(patch_elements=767)),
    ("tet", (9, 8, 6), ELASTIC, dict(patch_elements=768)),
    ("hex", (8, 8, 8), NEO, dict(patch_elements=256)),
    ("hex", (8, 8, 8), NEO, dict(patch_elements=257)),
])
def test_both_sides_of_the_dispatch(kind, n, mats, patch):
    """Mesh and patch sizes next to where fan and chunk records change over."""
    test_against_oracle(kind, n, mats, 1, patch, True)


@pytest.mark.parametrize("kind,n,law,patch,name", [
    ("tri", (2047, 1), ELASTIC, {}, "patch_step"), ("tri", (64, 32), ELASTIC, {}, "fan_step"),
    ("tet", (31, 11, 2), ELASTIC, {}, "patch_step"), ("tet", (683, 1, 1), ELASTIC, {}, "fan_step"),
    ("tri", (149, 151), FINITE, {}, "patch_step"), ("tri", (150, 150), FINITE, {}, "fan_step"),
    ("tet", (19, 19, 20), FINITE, {}, "patch_step"), ("tet", (20, 20, 19), FINITE, {}, "fan_step"),
    ("tri", (200, 219), NEO, {}, "patch_step"), ("tri", (200, 220), NEO, {}, "fan_step"),
    ("tet", (21, 21, 21), NEO, {}, "patch_step"), ("tet", (21, 21, 22), NEO, {}, "fan_step"),
    ("tri", (60, 20), ELASTIC, dict(patch_elements=768), "fan_step"),
    ("tri", (60, 20), ELASTIC, dict(patch_elements=769), "patch_step"),
    ("tri", (8, 3), NEO, dict(patch_elements=256), "patch_step"),
    ("tri", (8, 3), NEO, dict(patch_elements=257), "fan_step"),
    ("tet", (9, 8, 6), ELASTIC, dict(patch_elements=767), "patch_step"),
    ("tet", (9, 8, 6), NEO, dict(patch_elements=768), "fan_step"),
    ("hex", (1, 1, 1), NEO, {}, "fan_step"),
    ("hex", (8, 8, 8), NEO, dict(patch_elements=256), "fan_step"),
    ("hex", (8, 8, 8), NEO, dict(patch_elements=257), "patch_step"),
    ("tet", (20, 20, 20), ELASTIC, dict(patch_elements=8191, patch_nodes=6000), "patch_step"),
])
def test_kernel_of_each_side(kind, n, law, patch, name):
    """akb_kernel_name says which kernel steps the model: fan records from 4096
    small-strain triangles or tetrahedra on, later for the longer laws, and for
    the patch sizes they are built for; chunk records below, beside them, in FP32
    and where a patch of fans does not fit an SM."""
    from akantu_b200._lib import lib
    from akantu_b200.model import SolidMechanicsModel, material_from_dict
    for mode, want in ((_abi.MODE_FP64, name), (_abi.MODE_FP32_BULK, "patch_step")):
        m = SolidMechanicsModel(build(kind, n, 0), [material_from_dict(law)], precision=mode,
                                **patch)
        m.initFull()
        assert lib().akb_kernel_name(m.handle, 0).decode() == want
        assert lib().akb_kernel_name(m.handle, 1).decode() == "patch_finish_list"
        m.close()


@pytest.mark.parametrize("kind,n,count,law,name", [
    ("tet", (4, 4, 5), 12, ELASTIC, "patch_step"), ("tet", (5, 4, 5), 12, ELASTIC, "fan_step"),
    ("tet", (6, 6, 6), 40, FINITE, "patch_step"), ("tet", (7, 7, 7), 25, FINITE, "fan_step"),
    ("tet", (6, 8, 7), 30, NEO, "patch_step"), ("tet", (11, 11, 11), 8, NEO, "fan_step"),
    ("tri", (15, 15), 200, NEO, "patch_step"), ("tri", (21, 21), 100, NEO, "fan_step"),
    ("tri", (8, 8), 40, ELASTIC, "fan_step"), ("hex", (2, 2, 2), 20, NEO, "fan_step"),
])
def test_kernel_of_batches(kind, n, count, law, name):
    """The same of batches, whose instances can be too small for fans."""
    from akantu_b200._lib import lib
    from akantu_b200.batch import BatchModel
    from akantu_b200.model import material_from_dict
    b = BatchModel([build(kind, n, 0)] * count, [material_from_dict(law)] * count,
                   precision=_abi.MODE_FP64)
    b.initFull()
    assert lib().akb_kernel_name(b.handle, 0).decode() == name
    b.close()


@pytest.mark.parametrize("load", [False, True], ids=["free", "loaded"])
@pytest.mark.parametrize("kind,n,mats,jitter,patch", [
    ("tet", (1, 1, 1), ELASTIC, 0, dict(patch_elements=1536)),
    ("tet", (7, 6, 5), [ELASTIC, STIFF], 1, dict(patch_elements=1536)),
    ("tet", (9, 9, 4), FINITE, 0, dict(patch_elements=768, patch_grid=1)),
    ("tet", (8, 7, 9), [FINITE, ELASTIC], 1, dict(patch_elements=1024)),
    ("tet", (6, 5, 7), NEO, 1, dict(patch_elements=768)),
    ("tri", (1, 1), ELASTIC, 0, dict(patch_elements=768)),
    ("tri", (40, 31), [STIFF, ELASTIC], 1, dict(patch_elements=768)),
    ("tri", (33, 20), [FINITE, STIFF], 1, dict(patch_elements=300, patch_grid=1)),
    ("tri", (40, 21), NEO, 0, dict(patch_elements=512)),
])
def test_fans_of_small_meshes(kind, n, mats, jitter, patch, load):
    """Meshes that step on fan records only where the caller gives the patch size."""
    test_against_oracle(kind, n, mats, jitter, patch, load)


def test_a_plan_that_just_misses_an_sm():
    """One patch whose fan layout takes 48 bytes less than an SM's 227 KB, which
    the kernel's static shared memory no longer leaves: chunk records."""
    from akantu_b200._lib import lib
    from akantu_b200.mesh import Mesh
    from akantu_b200.model import SolidMechanicsModel, material_from_dict
    box = box_tetrahedron4(8, 8, 8, 8.0, 8.0, 8.0)
    nodes, conn = [box.nodes], [box.connectivity.astype(np.int64)]
    for j in range(1, 15):  # tetrahedra of their own
        z = 100.0 + 3 * j
        conn.append(np.arange(4)[None] + sum(len(x) for x in nodes))
        nodes.append(np.array([[0, 0, z], [1, 0, z], [0, 1, z], [0, 0, z + 1]], dtype=float))
    mesh = Mesh(3, _abi.TETRAHEDRON_4, np.concatenate(nodes),
                np.concatenate(conn).astype(np.uint32))
    m = SolidMechanicsModel(mesh, [material_from_dict(ELASTIC)], precision=_abi.MODE_FP64,
                            patch_elements=8191, patch_nodes=6000)
    m.initFull()
    assert lib().akb_kernel_name(m.handle, 0).decode() == "patch_step"
    m.setTimeStep(0.5 * m.getStableTimeStep())
    m.solveSteps(2)
    assert np.isfinite(m.getDisplacement()).all()
    m.close()
