"""The bound behind the tet search's candidate filter, in float32 on the CPU.

For a ring key qLast > 0 the filter drops a candidate p when, for some tet,
g(p) = det(p) - sqrt(thr) (1.5 r L(p) - 0.5 r^3) + allowance < 0, with thr just below qLast, r^2
about L at the level's centre and the allowance 2^-18 of the magnitudes entering g. Exactness
needs that no candidate whose tet keys (det^2 / L^3 in float32, det >= 0) are all at least qLast
gets a negative g. The float32 restatement below uses plain products where the device uses fused
ones (more roundings, not fewer) and a square root off by up to 2^-22."""
import numpy as np
import pytest

F = np.float32
OFF = np.array([7, 5, 3, 1, -1, -3, -5, -7], F) / F(7)


def _coeffs(a, b, c):
    u, w, v = b - a, c - a, c - b
    n = np.cross(u, w)
    sq = lambda q: (q * q).sum(-1, dtype=F)
    A = np.concatenate([-n, (a * n).sum(-1, dtype=F)[:, None]], 1).astype(F)
    C = sq(a) + sq(b) + sq(c) + sq(u) + sq(w) + sq(v)
    B = np.concatenate([F(-2) * (a + b + c), C[:, None]], 1).astype(F)
    return A, B


def _key_parts(A, B, p):
    """det and L of every (candidate, tet) in float32."""
    det = A[:, 3] + p @ A[:, :3].T
    L = B[:, 3] + p @ B[:, :3].T + F(3) * (p * p).sum(1, dtype=F)[:, None]
    return det.astype(F), L.astype(F)


def _g(A, B, c, S, thr, rng):
    off = lambda: F(1) + F(rng.uniform(-1, 1) * 2.0 ** -22)
    sq = F(np.sqrt(thr)) * off() * F(1 - 2.0 ** -20) if thr > 0 else F(0)
    low = F(0) if thr > 0 else thr
    m = np.abs(c) + S
    det, L = (x[0] for x in _key_parts(A, B, c[None]))
    r = (np.sqrt(np.maximum(L, F(0))) * off()).astype(F)
    b = F(1.5) * (sq * r)
    a = (b * F(1 / 3)) * (r * r)
    mag = np.abs(A[:, 3]) + np.abs(A[:, :3]) @ m + b * (B[:, 3] + np.abs(B[:, :3]) @ m + F(3) * (m * m).sum(dtype=F)) + a - low
    g = (det - low) + (a - b * L) + F(2.0 ** -18) * mag
    out = g[:, None, None, None]
    for ax in range(3):
        P = S[ax] * (A[:, ax] - b * (B[:, ax] + F(6) * c[ax]))
        Q = (F(3) * b) * (S[ax] * S[ax])
        t = (OFF[None] * P[:, None] - (OFF * OFF)[None] * Q[:, None]).astype(F)
        shape = [len(A), 1, 1, 1]
        shape[1 + ax] = 8
        out = out + t.reshape(shape)
    return out.astype(F)


@pytest.mark.parametrize("kind", ["regular", "sliver", "flipped"])
def test_no_candidate_that_can_win_is_dropped(kind):
    rng = np.random.default_rng({"regular": 0, "sliver": 1, "flipped": 2}[kind])
    kept = won = 0
    for _ in range(400):
        k = int(rng.integers(4, 40))
        # outer triangles on a sphere around the vertex, wound outwards
        d = rng.normal(size=(k, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        e = np.cross(d, rng.normal(size=(k, 3)))
        e /= np.linalg.norm(e, axis=1, keepdims=True)
        f = np.cross(d, e)
        size = rng.uniform(0.2, 0.6, (k, 1)) * (10.0 ** rng.uniform(-4, 0, (k, 1)) if kind == "sliver" else 1.0)
        centre = d * rng.uniform(0.3, 0.9, (k, 1)) * (rng.choice([-0.2, 1.0], (k, 1), p=[0.1, 0.9]) if kind == "flipped" else 1.0)
        a, b, c = (centre + size * (np.cos(t) * e + np.sin(t) * f) for t in (0.0, 2.1, 4.2))
        A, B = _coeffs(*(np.asarray(x, F) for x in (a, b, c)))
        at = np.asarray(rng.uniform(-0.1, 0.1, 3), F)
        S = np.asarray(rng.uniform(0.5, 1.0, 3) * rng.choice([0.5, 0.14, 0.04, 0.012]), F)
        grid = np.stack(np.meshgrid(*(at[i] + OFF * S[i] for i in range(3)), indexing="ij"), -1).reshape(-1, 3).astype(F)
        det, L = _key_parts(A, B, grid)
        with np.errstate(all="ignore"):
            key = np.where(det < 0, det, (det * det) / ((L * L) * L))
        ring = np.where((det < 0).any(1), det.min(1), key.min(1))
        # the current key: the centre's, and one that only the best candidates beat
        det0, L0 = (x[0] for x in _key_parts(A, B, at[None]))
        here = det0.min() if (det0 < 0).any() else ((det0 * det0) / ((L0 * L0) * L0)).min()
        for q in (F(here), F(np.sort(ring)[-20])):
            thr = F(q - F(F(np.abs(q) * F(2.0 ** -14)) + F(1e-37)))
            g = _g(A, B, at, S, thr, rng).min(0).reshape(-1)
            wins = ring > q
            assert not (g[wins] < 0).any(), (kind, float(q))
            kept += int((~(g < 0)).sum())
            won += int(wins.sum())
    assert won > 1000 and kept < 3 * won + 40000   # the bound is not vacuous
