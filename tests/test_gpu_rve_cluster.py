"""The RVE relaxation by a cluster of CTAs (FP32; 1, 2 or 4 CTAs by the number
of cells) and the sizes it leaves to one CTA, against the oracle and between
akb_rve_solve and akb_rve_solve_indexed."""
import numpy as np
import pytest

from akantu_b200 import _abi, fe2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [2, 4, 6, 8, 10, 12, 14, 16])
def test_fixed_updates_match_oracle(cells):
    """After 30 updates at a fixed count the FP32 fluctuation and stress follow
    the FP64 oracle: 2e-4 on the stress, the bound of the converged test."""
    import torch
    from akantu_b200.rve import SolidMechanicsModelRVE
    from tests.fe2_cases import oracle_rve
    rng = np.random.default_rng(cells)
    vm = (rng.random(cells ** 3) < 0.3).astype(np.uint8)
    mats = fe2.matrix_inclusion_materials()
    H = fe2.sample_gradients(3, seed=cells, amplitude=0.1)
    R = SolidMechanicsModelRVE(cells, vm, mats, precision=_abi.MODE_FP32_BULK, tolerance=-1.0,
                               max_iterations=30)
    w = R.zero_fluctuation(3)
    out = R.solve(H, w)
    O = oracle_rve(cells, vm, mats)
    for k in range(3):
        Po = O.solve(H[k], tolerance=-1.0, max_iterations=30, time_step_factor=0.6,
                     damping_factor=0.6)[0]
        err = np.abs(out["stress"][k].cpu().numpy() - Po).max() / np.abs(Po).max()
        assert err <= 2e-4, (k, err)
    # the internal force and stress of the state it left, and the listed solve
    P, f = R.stress(H, w)
    assert torch.equal(P, out["stress"])
    idx = torch.tensor([2, 0], dtype=torch.int32, device="cuda")
    cnt = torch.tensor([2], dtype=torch.int32, device="cuda")
    Hc = torch.as_tensor(H, device="cuda").transpose(1, 2).reshape(-1, 9).contiguous()
    Pi = torch.zeros_like(Hc)
    R.solve_indexed(idx, cnt, Hc, Pi)
    Pi = Pi.reshape(-1, 3, 3).transpose(1, 2)
    assert torch.equal(Pi[0], out["stress"][0]) and torch.equal(Pi[2], out["stress"][2])
    assert not bool(Pi[1].any())


def test_many_instances_leave_the_clusters():
    """From 6144 instances of 16^3 on, one CTA per RVE: the same FP32 updates
    bit for bit; the stress is a FP64 sum of 32768 terms in another order
    (2^-53 each, of terms at most 30 times the mean)."""
    import torch
    from akantu_b200.rve import SolidMechanicsModelRVE
    vm = (np.random.default_rng(0).random(16 ** 3) < 0.3).astype(np.uint8)
    H = fe2.sample_gradients(6144, seed=3, amplitude=0.1)
    R = SolidMechanicsModelRVE(16, vm, fe2.matrix_inclusion_materials(),
                               precision=_abi.MODE_FP32_BULK, tolerance=-1.0, max_iterations=5)
    w, w1 = R.zero_fluctuation(6144), R.zero_fluctuation(6143)
    many, fewer = R.solve(H, w)["stress"], R.solve(H[:6143], w1)["stress"]
    assert bool(torch.isfinite(many).all())
    assert torch.equal(w[:6143], w1)
    assert float((many[:6143] - fewer).abs().max()) <= 1.1e-10 * float(fewer.abs().max())


def test_a_list_takes_as_long_as_the_batch():
    """The listed RVEs are strided over by no more clusters than run at once: the
    same 1024 RVEs of 16^3 (40 updates each) take about as long listed as in a
    batch (the tail of 1024 over some 36 clusters: at most 1 / 28). With clusters
    beyond the resident ones the list waits for a second round: twice as long."""
    import torch
    from akantu_b200.rve import SolidMechanicsModelRVE
    vm = (np.random.default_rng(0).random(16 ** 3) < 0.3).astype(np.uint8)
    H = torch.as_tensor(fe2.sample_gradients(1024, seed=3, amplitude=0.1), device="cuda")
    R = SolidMechanicsModelRVE(16, vm, fe2.matrix_inclusion_materials(),
                               precision=_abi.MODE_FP32_BULK, tolerance=-1.0, max_iterations=40)
    Hc = H.transpose(1, 2).reshape(-1, 9).contiguous()
    P = torch.empty_like(Hc)
    idx = torch.arange(1024, dtype=torch.int32, device="cuda")
    cnt = torch.tensor([1024], dtype=torch.int32, device="cuda")

    def ms(call):
        best = float("inf")
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    listed, batch = ms(lambda: R.solve_indexed(idx, cnt, Hc, P)), ms(lambda: R.solve(H))
    assert listed <= 1.3 * batch, (listed, batch)


@pytest.mark.parametrize("kinds", ["neohookean", "elastic inclusion"])
def test_stress_does_not_tell_the_kernel(kinds):
    """An RVE of 16^3 has the same bits alone, in a list and in a batch large
    enough for one CTA per RVE: fluctuation, stress, residual and, of the relaxed
    state, the internal force."""
    import torch
    from akantu_b200.rve import SolidMechanicsModelRVE
    vm = (np.random.default_rng(1).random(16 ** 3) < 0.3).astype(np.uint8)
    mats = fe2.matrix_inclusion_materials()
    if kinds != "neohookean":
        mats[1]["kind"] = _abi.MATERIAL_ELASTIC
    nb, few = 6144, 40
    H = torch.as_tensor(fe2.sample_gradients(nb, seed=5, amplitude=0.1), device="cuda")
    R = SolidMechanicsModelRVE(16, vm, mats, precision=_abi.MODE_FP32_BULK, tolerance=-1.0,
                               max_iterations=12)
    w, w1 = R.zero_fluctuation(nb), R.zero_fluctuation(few)
    many, alone = R.solve(H, w), R.solve(H[:few], w1)
    assert torch.equal(w[:few], w1)
    for k in ("stress", "residual"):
        assert torch.equal(many[k][:few], alone[k]), k
    P, f = R.stress(H, w)
    P1, f1 = R.stress(H[:few], w1)
    assert torch.equal(P[:few], P1) and torch.equal(P, many["stress"])
    assert torch.equal(f[:few], f1)
    Hc = H[:few].transpose(1, 2).reshape(-1, 9).contiguous()
    Pi = torch.zeros_like(Hc)
    idx = torch.arange(few, dtype=torch.int32, device="cuda")
    R.solve_indexed(idx, torch.tensor([few], dtype=torch.int32, device="cuda"), Hc, Pi)
    assert torch.equal(Pi.reshape(-1, 3, 3).transpose(1, 2), alone["stress"])


@pytest.mark.parametrize("cells", [2, 4, 6, 8, 10, 12, 14, 16])
def test_internal_force_matches_oracle(cells):
    """The internal force of given states, the reads of the neighbour CTA's
    planes among them, against the FP64 oracle on the same (FP32) fluctuation.
    A node's force adds 8 voxels' corner forces, each the sum of three edge
    sums of 8 Gauss points: at most some 100 roundings of 6e-8 on terms of the
    size of the largest force, 2e-5 with a margin of three."""
    import torch
    from akantu_b200.rve import SolidMechanicsModelRVE
    from tests.fe2_cases import oracle_rve
    rng = np.random.default_rng(cells)
    vm = (rng.random(cells ** 3) < 0.3).astype(np.uint8)
    mats = fe2.matrix_inclusion_materials()
    H = fe2.sample_gradients(3, seed=cells, amplitude=0.1)
    w = (0.05 / cells * rng.uniform(-1, 1, (3, cells ** 3, 3))).astype(np.float32)
    R = SolidMechanicsModelRVE(cells, vm, mats, precision=_abi.MODE_FP32_BULK)
    P, f = R.stress(H, torch.as_tensor(w, device="cuda"))
    O = oracle_rve(cells, vm, mats)
    for k in range(3):
        Po, fo = O.stress(H[k], w[k].astype(np.float64))
        assert np.abs(f[k].cpu().numpy() - fo).max() <= 2e-5 * np.abs(fo).max(), k
        assert np.abs(P[k].cpu().numpy() - Po).max() <= 2e-5 * np.abs(Po).max(), k
