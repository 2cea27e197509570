"""The fused training step at its edges: waits on MMAs that expire with the MMAs in flight, device arrays
on any float boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
E_TIMEOUT = 6


def _pairs(rows, seed):
    r = np.random.default_rng(seed)
    return r.uniform(-1, 1, size=(rows, 96)).astype(np.float32), r.uniform(-0.5, 0.5, size=(rows, 3)).astype(np.float32)


@pytest.mark.parametrize("batch", [128, 8192, 16384])
def test_expired_mma_wait_is_reported_and_recovers(vsdmo, batch):
    """The operand loads land, the first MMAs are issued and no wait for them is granted any time: the kernel
    reports it, lets them land (at the default limit), frees its tensor memory and returns."""
    X, T = _pairs(1000, 3)
    m = vsdmo.ProposalModel(seed=7)
    p = m.get_params()
    try:
        vsdmo.debug_set_train_mma_wait_limit_ns(0)
        with pytest.raises(vsdmo.VSDMOError) as e:
            m.train(X, T, steps=3, batch=batch, lr=1e-3, seed=1)
        assert e.value.status == E_TIMEOUT
        with pytest.raises(vsdmo.VSDMOError) as e:
            m.gradients(X[:128], T[:128])
        assert e.value.status == E_TIMEOUT
    finally:
        vsdmo.debug_set_train_mma_wait_limit_ns(-1)
    assert np.array_equal(m.get_params(), p)
    fresh = vsdmo.ProposalModel(seed=7)
    for a, b in zip(m.gradients(X[:384], T[:384]), fresh.gradients(X[:384], T[:384])):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_device_arrays_on_any_float_boundary(vsdmo, offset):
    import torch
    X, T = _pairs(700, 4)
    params = []
    for o in (0, offset):
        f = torch.zeros(X.size + 4, device="cuda")
        t = torch.zeros(T.size + 4, device="cuda")
        f[o:o + X.size] = torch.from_numpy(X.ravel()).cuda()
        t[o:o + T.size] = torch.from_numpy(T.ravel()).cuda()
        torch.cuda.synchronize()
        m = vsdmo.ProposalModel(seed=3)
        hist = m.train(None, None, steps=3, batch=256, lr=1e-3, seed=2, n_rows=len(X),
                       device_ptrs=(f.data_ptr() + 4 * o, t.data_ptr() + 4 * o))
        params.append((hist, m.get_params()))
    assert np.array_equal(params[0][0], params[1][0]) and np.array_equal(params[0][1], params[1][1])
