"""GPU tests of single pairs against extended precision: the chord form with its
hardware-seeded square root and reciprocal, one pair at a time, and the vector sums
of far panel pairs at the two edges of their class.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
C1, C2, CONS = LD(1.0 - 6.21196), LD(2.7 + 6.0), LD(-2.343256857908601e-9)


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _val(mp):
    """sal_grad_gfunc's scalar in extended precision, from 2 - 2g."""
    mp = mp.astype(LD)
    g, q = 1 - mp / 2, np.sqrt(mp)
    return (C1 / (q * mp + LD(1e-16)) + C2 * (2 * g + q) / (2 * (g * g - 1) + LD(1e-16))) * CONS


def test_single_pairs_over_all_chords():
    """Source (1, 0, 0), 6,000 targets from chord 1.05e-3 to 1.9995: nx and ny are
    exact or one rounding, so what is left is the value's.  The kernel's own
    2 - 2g (its operation order, in numpy) goes into the extended-precision value.
    So does its 1 - tz^2, which cancels at the pole.  Bar: 16 roundings of 2^-53
    (square root and reciprocal one ulp each, 14 operations), and the + 1e-16 that
    the chord form leaves out of p2, 1e-16 / (2 (1 - g^2)) = 2e-16 / (mp (4 - mp)) of
    a term that is 1.7 q of the pair at small q and all of it at most; twice that."""
    torch = _torch()
    import salgpu as S
    rng = np.random.default_rng(17)
    n = 6001
    q = np.concatenate([np.geomspace(1.05e-3, 1.0, 4000), np.linspace(1.0, 1.9995, 2000)])
    a, b = 2 * np.arcsin(q / 2), rng.uniform(0.0, 2 * np.pi, n - 1)
    t = np.stack([np.cos(a), np.sin(a) * np.cos(b), np.sin(a) * np.sin(b)], 1)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    p = np.concatenate([[[1.0, 0.0, 0.0]], t])
    w = np.zeros(n)
    w[0] = 1.0
    dev = [torch.tensor(np.ascontiguousarray(v), device="cuda") for v in (p[:, 0], p[:, 1], p[:, 2], w)]
    gx, gy = S.direct_sum(*dev, torch.arange(1, n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    x, y, z = t[:, 0], t[:, 1], t[:, 2]
    mp = 2.0 - 2.0 * x
    f = _val(mp) / np.sqrt((1.0 - z * z).astype(LD))
    bar = 16 * 2.0 ** -53 + 2 * np.minimum(1.0, 1.7 * np.sqrt(mp)) * 2e-16 / (mp * (4.0 - mp))
    for got, ref in ((gx, -y.astype(LD) * f), (gy, -z.astype(LD) * x.astype(LD) * f)):
        err = np.abs(got.cpu().numpy().astype(LD) - ref) / np.abs(ref)
        assert np.all(err <= bar), (float(err.max()), float(q[np.argmax(err / bar)]))


def test_far_panel_pairs_at_the_edges_of_their_class():
    """Points at the centres of level-7 panels around (1, 0, 0) and (-1, 0, 0), one a
    leaf, every interaction particle-particle: neighbours' chords lie about 0.01225
    (the near edge of the far class, mp = 1.5e-4: 0.01225), those of antipodal panels
    about sqrt(3.999).  Weights on every second point, values at the others.  Bar:
    2 - 2g carries two roundings of g and one of its own, 2^-52 each at most, so a
    value 1.5 times 3 x 2^-52 / 1.5e-4 (7e-12), and its sum of 144 one-signed or
    distant terms no more; 1e-11 of the largest."""
    _torch()
    import salgpu as S
    m = 12
    e = (np.arange(m) - m / 2 + 0.5) * (np.pi / 2 / 128)
    u, v = np.meshgrid(np.tan(e), np.tan(e), indexing="ij")
    p = np.stack([np.ones(m * m), u.ravel(), v.ravel()], 1)
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    p = np.concatenate([p, -p])
    n = len(p)
    xyz = [np.ascontiguousarray(p[:, k]) for k in range(3)]
    src = (np.add.outer(np.arange(m), np.arange(m)) % 2).ravel().astype(bool)
    src = np.concatenate([src, src])
    h = np.where(src, np.random.default_rng(3).uniform(0.5, 1.5, n), 0.0)
    t = S.tree_traverse(*xyz, n, 2)
    L = S.dual_tree_traversal(t, 0.0, 2)
    gx, gy = np.zeros(n), np.zeros(n)
    S.fast_sum(gx, gy, L, t, *xyz, np.ones(n), h, n, 2)
    T, Q, w = p[~src].astype(LD), p[src].astype(LD), h[src].astype(LD)
    g = T @ Q.T
    omz = 1 - T[:, 2:] ** 2
    f = _val(2 - 2 * g) * w / np.sqrt(omz)
    rx = ((T[:, :1] * Q[:, 1] - T[:, 1:2] * Q[:, 0]) * f).sum(1)
    ry = ((Q[:, 2] * omz - T[:, 2:] * (T[:, :2] @ Q[:, :2].T)) * f).sum(1)
    for got, ref in ((gx[~src], rx), (gy[~src], ry)):
        assert np.abs(got.astype(LD) - ref).max() <= 1e-11 * np.abs(ref).max()
