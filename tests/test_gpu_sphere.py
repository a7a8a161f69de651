"""GPU tests of the FP64 pair kernel on points off the unit sphere, whose self
pairs are no rounding noise: the particle-particle sums and the direct sum against
the oracle at the pair kernel's 1e-12, with near panel pairs alone and with far ones
(whose bounds widen with the distance from the sphere).  Each component by its own
largest value: a self pair's north component is up to 1e4 times the rest, and its east
component is zero.  Where a target beyond |z| = 1 makes the reference NaN, so is the
result.  Random radii: coordinates
in single precision (6e-8), just below and above the distance at which a self pair
counts as a plain one (2.5e-7), and far above it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _close(got, ref):
    for g, r in zip(got, ref):
        assert np.array_equal(np.isnan(g), np.isnan(r))
        assert np.nanmax(np.abs(g - r)) <= 1e-12 * np.nanmax(np.abs(r))


@pytest.mark.parametrize("off", [6e-8, 2e-7, 1e-6, 1e-4, 1e-2])
@pytest.mark.parametrize("caps", [False, True])
def test_points_off_the_sphere(off, caps):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import salgpu as S
    from oracle import oracle as O
    n = 540
    rng = np.random.default_rng(int(1e9 * off) + caps)
    if caps:   # within 0.2 of the face centres: neighbouring faces are far from one another
        p = np.concatenate([np.insert(rng.uniform(-0.2, 0.2, (n // 6, 2)), a, s, axis=1) for a in range(3) for s in (1.0, -1.0)])
    else:
        p = rng.standard_normal((n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    p *= 1.0 + off * rng.uniform(-1.0, 1.0, (n, 1))
    p[1::90] = p[0::90]   # coincident points
    xyz = [np.ascontiguousarray(p[:, k]) for k in range(3)]
    area, h = rng.uniform(0.9, 1.1, n), rng.standard_normal(n)
    ot = O.tree_traverse(*xyz, 200)
    L = O.dual_tree_traversal(ot, 0.0, 200)
    rx, ry = O.fast_sum(ot, L, *xyz, area, h, 8)
    gx, gy = np.zeros(n), np.zeros(n)
    S.fast_sum(gx, gy, L, S.tree_traverse(*xyz, n, 200), *xyz, area, h, n, 8)
    _close((gx, gy), (rx, ry))
    tg = np.arange(0, n, 3, dtype=np.int32)
    rx, ry = O.direct_sum(*xyz, area, h, tg)
    dx, dy = S.direct_sum(*[torch.tensor(v, device="cuda") for v in (*xyz, area * h, tg)])
    torch.cuda.synchronize()
    _close((dx.cpu().numpy(), dy.cpu().numpy()), (rx, ry))
