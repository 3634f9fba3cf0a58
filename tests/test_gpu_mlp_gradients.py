"""The gradient kernels of a training step (all layers' weight partials and
bias chains in one launch) where their tiling can go wrong, against the FP64
oracle with the same BF16 roundings, and the BF16 weight copies that the Adam
kernel writes against those a fresh upload of the same weights makes.
Tolerances: those of test_gpu_mlp.test_gradient_check_against_cpu."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 127, 128, 129, 511, 640, 2049])
@pytest.mark.parametrize("width,nh", [(256, 3), (128, 1)])
def test_gradients_at_tile_edges(nb, width, nh):
    from tests.test_gpu_mlp import setup
    net, X, T, x, t, O = setup(nb=max(nb, 2), seed=nb, width=width, nh=nh)
    X, T, x, t = X[:nb].contiguous(), T[:nb].contiguous(), x[:nb], t[:nb]
    loss, g = net.gradients_features(X, T)
    lo, go = O.gradients(x, t, emulate_bf16=True)
    assert loss == pytest.approx(lo, rel=2e-3)
    off = 0
    for k, n in net.layer_shapes():
        for size in (k * n, n):
            a, b = g[off:off + size], go[off:off + size]
            off += size
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-12


@pytest.mark.parametrize("width,nh", [(256, 3), (128, 2)])
def test_adam_leaves_the_weights_it_reports(width, nh):
    from tests.test_gpu_mlp import setup
    net, X, T, x, t, O = setup(nb=300, seed=5, width=width, nh=nh)
    for _ in range(3):
        net.train_step_features(X, T, 1e-2)
    y = net.forward_features(X).cpu().numpy()
    net.set_parameters(net.get_parameters())
    assert np.array_equal(net.forward_features(X).cpu().numpy(), y)


@pytest.mark.parametrize("width,nh", [(256, 3), (128, 1)])
def test_adam_leaves_the_transposed_weights_too(width, nh):
    """The transposed copies, which only the backward pass reads: the gradients
    after some steps are those of a fresh upload of the same weights."""
    from tests.test_gpu_mlp import setup
    net, X, T, x, t, O = setup(nb=300, seed=6, width=width, nh=nh)
    for _ in range(3):
        net.train_step_features(X, T, 1e-2)
    loss, g = net.gradients_features(X, T)
    net.set_parameters(net.get_parameters())
    loss2, g2 = net.gradients_features(X, T)
    assert loss == loss2 and np.array_equal(g, g2)


def test_a_batch_too_large_for_memory_leaves_the_network_usable():
    """The workspace of 2^34 samples (550 GB for the inputs alone) is refused
    before any launch; the next call of an ordinary size has a workspace again."""
    import ctypes as C
    from akantu_b200._lib import AkbError, check, lib
    from tests.test_gpu_mlp import setup
    net, X, T, x, t, O = setup(nb=300, seed=7, width=128, nh=1)
    loss, g = net.gradients_features(X, T)
    out = np.zeros(net.nb_parameters, np.float32)
    value = C.c_float()
    with pytest.raises(AkbError, match="memory"):
        check(lib().akb_mlp_gradients(net._h, 2 ** 34, X.data_ptr(), T.data_ptr(),
                                      out.ctypes.data_as(C.POINTER(C.c_float)), C.byref(value)))
    loss2, g2 = net.gradients_features(X, T)
    assert loss == loss2 and np.array_equal(g, g2)
