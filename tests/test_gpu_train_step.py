"""The two-launch training step: gradients against the oracle at one tile, one tile per part, two tiles
per part and batches that keep the separate launches; the rows it draws (a 64-bit Mersenne twister
restated here) through the losses of steps that change nothing; an expired wait is reported, leaves
the parameters alone and the model usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
E_TIMEOUT = 6


@pytest.fixture(scope="module")
def mo():
    from oracle import mlp_oracle
    return mlp_oracle


def _model(vsdmo, mo, seed):
    m = vsdmo.ProposalModel(seed=seed)
    r = np.random.default_rng(seed)
    P = mo.unflatten(m.get_params())
    for k in ("b1", "b2", "b3"):
        P[k] = r.uniform(0.0, 0.1, size=P[k].shape)
    p = mo.flatten(P).astype(np.float32)
    m.set_params(p)
    return m, p


# tolerances as for the separate launches (test_gpu_learned.py): BF16 operands, FP32 sums
@pytest.mark.parametrize("rows", [128, 384, 8192, 16384, 8320])
def test_gradients_match_oracle(vsdmo, mo, rows):
    m, p = _model(vsdmo, mo, 5)
    r = np.random.default_rng(rows)
    X = r.uniform(-1, 1, size=(rows, 96)).astype(np.float32)
    T = r.uniform(-0.5, 0.5, size=(rows, 3)).astype(np.float32)
    loss, g = m.gradients(X, T)
    loss_r, g_r = mo.loss_and_grad(p, X, T)
    assert abs(loss - loss_r) <= 1e-4 * abs(loss_r) + 1e-7
    o = 0
    for name, shape in mo.SHAPES:
        n = int(np.prod(shape))
        rel = np.linalg.norm(g[o:o + n] - g_r[o:o + n]) / max(np.linalg.norm(g_r[o:o + n]), 1e-12)
        assert rel < 2e-2, (name, rel)
        o += n


def _mt64(seed):
    """Words of the 64-bit Mersenne twister (Nishimura and Matsumoto)."""
    M = (1 << 64) - 1
    mt = [seed & M]
    for i in range(1, 312):
        mt.append((6364136223846793005 * (mt[-1] ^ (mt[-1] >> 62)) + i) & M)
    while True:
        for i in range(312):
            x = (mt[i] & 0xFFFFFFFF80000000) | (mt[(i + 1) % 312] & 0x7FFFFFFF)
            mt[i] = mt[(i + 156) % 312] ^ (x >> 1) ^ (0xB5026F5AA96619E9 if x & 1 else 0)
        for x in list(mt):
            x ^= (x >> 29) & 0x5555555555555555
            x ^= (x << 17) & 0x71D67FFFEDA60000 & M
            x ^= (x << 37) & 0xFFF7EEE000000000 & M
            yield x ^ (x >> 43)


@pytest.mark.parametrize("n_rows,batch,steps", [(1000, 128, 30), (1, 128, 2), (77777, 8192, 3)])
def test_rows_are_the_generators(vsdmo, mo, n_rows, batch, steps):
    m, p = _model(vsdmo, mo, 6)
    r = np.random.default_rng(n_rows)
    X = r.uniform(-1, 1, size=(n_rows, 96)).astype(np.float32)
    T = (r.uniform(-1, 1, size=(n_rows, 3)) * 10.0 ** r.uniform(-1, 2, size=(n_rows, 1))).astype(np.float32)
    hist = m.train(X, T, steps=steps, batch=batch, lr=0.0, seed=n_rows)
    assert np.array_equal(m.get_params(), p)
    y = mo.forward(p, X)[0]
    rows_loss = ((y - T).astype(np.float64) ** 2).mean(1)
    g = _mt64(n_rows)
    for i in range(steps):
        idx = [(next(g) * n_rows) >> 64 for _ in range(batch)]
        want = rows_loss[idx].mean()
        assert abs(hist[i] - want) <= 1e-4 * want + 1e-7, i


def test_expired_wait_is_reported_and_recovers(vsdmo, mo):
    m, p = _model(vsdmo, mo, 7)
    r = np.random.default_rng(3)
    X = r.uniform(-1, 1, size=(512, 96)).astype(np.float32)
    T = r.uniform(-0.5, 0.5, size=(512, 3)).astype(np.float32)
    try:
        vsdmo.debug_set_wait_limit_ns(0)
        with pytest.raises(vsdmo.VSDMOError) as e:
            m.train(X, T, steps=2, batch=256, lr=1e-3, seed=1)
        assert e.value.status == E_TIMEOUT
    finally:
        vsdmo.debug_set_wait_limit_ns(-1)
    assert np.array_equal(m.get_params(), p)
    hist = m.train(X, T, steps=50, batch=256, lr=1e-3, seed=1)
    assert np.all(np.isfinite(hist)) and hist[-5:].mean() < hist[0]
