"""The per-step calls where they choose how to reach the device: Dirichlet
lists around the size that fits the launch (192 values), out-of-range node
ids, and energies queued into pinned, pageable, device and unaligned memory,
each against the blocking calls."""
import ctypes as C

import numpy as np
import pytest

from akantu_b200 import _abi, configs

pytestmark = pytest.mark.gpu


def model(mode):
    from akantu_b200.model import SolidMechanicsModel, material_from_dict
    w = configs.plate_tri3(40, 20, 2.0, 1.0)
    m = SolidMechanicsModel(w["mesh"], [material_from_dict(x) for x in w["materials"]], precision=mode)
    m.initFull()
    m.setField(_abi.FIELD_DISPLACEMENT, w["u0"])
    m.setTimeStep(0.5 * m.getStableTimeStep())
    return m


@pytest.mark.parametrize("mode", [_abi.MODE_FP64_REFERENCE, _abi.MODE_FP64])
@pytest.mark.parametrize("count", [1, 95, 96, 97, 191, 192, 193, 400])
def test_dirichlet_lists(mode, count):
    rng = np.random.default_rng(count)
    m = model(mode)
    nn = m.mesh.getNbNodes()
    nodes = rng.choice(nn, count, replace=False).astype(np.uint32)
    nodes[0] = nn + 7 if count > 1 else nodes[0]  # ignored
    both = rng.normal(scale=1e-6, size=(count, 2))
    u = np.array(m.getDisplacement())
    b = np.zeros(u.shape, dtype=bool)
    m.applyDirichlet(nodes, _abi.ALL_COMPONENTS, both)
    m.applyDirichlet(nodes, 1, 2 * both[:, 1])
    ok = nodes < nn
    u[nodes[ok]] = both[ok]
    u[nodes[ok], 1] = 2 * both[ok, 1]
    b[nodes[ok]] = True
    assert np.array_equal(m.getDisplacement(), u)
    assert np.array_equal(m.getBlockedDOFs(), b)
    m.solveSteps(3)
    assert np.array_equal(np.array(m.getDisplacement())[b], u[b])
    m.close()


@pytest.mark.parametrize("mode", [_abi.MODE_FP64_REFERENCE, _abi.MODE_FP64])
def test_energy_destinations(mode):
    import torch
    m = model(mode)
    raw = (C.c_char * 20)()
    pinned = torch.zeros(2, dtype=torch.float64).pin_memory()
    device = torch.zeros(2, dtype=torch.float64, device="cuda")
    pageable = np.zeros(2)
    unaligned = C.addressof(raw) + 4 - C.addressof(raw) % 8
    for _ in range(40):  # past the ring of queued results
        m.solveStep()
        for k, kind in enumerate(("kinetic", "potential")):
            m.getEnergyAsync(kind, pinned.data_ptr() + 8 * k)
            m.getEnergyAsync(kind, device.data_ptr() + 8 * k)
            m.getEnergyAsync(kind, pageable.ctypes.data + 8 * k)
        m.getEnergyAsync("kinetic", unaligned)
    m.synchronize()
    want = [m.getEnergy("kinetic"), m.getEnergy("potential")]
    assert pinned.tolist() == device.tolist() == pageable.tolist() == want
    assert np.frombuffer(C.string_at(unaligned, 8))[0] == want[0]
    m.close()
