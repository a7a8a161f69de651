"""GPU tests of the FP64 pair kernel over the chords where its evaluation
changes: self pairs, near duplicates, the switch from the reference's operation
order to the chord form (chord 1e-3), close and distant neighbours, and
(near-)antipodes, where the reference's value is rounding noise.

Every interaction of such a point set is a particle-particle one (one leaf per
root face), so fast_sum is the direct sum of the reference kernel.  Bar:
rel-L2 <= 1e-12 against the oracle.  The chord form differs from the
reference's operations by their cancellation noise in g^2 - 1, at most
2.2e-16 / (2 q^2) of a term that is 3.3 q of the pair (4e-13 at q = 1e-3,
less beyond), plus 2e-13 for the second + 1e-16 there.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chord", [0.0, 1e-9, 1e-7, 1e-5, 9e-4, 1.001e-3, 1.2e-3, 3e-3, 1.2e-2, 0.1, 1.9])
@pytest.mark.parametrize("antipodal", [False, True])
def test_pair_kernel_over_chords_matches_oracle(chord, antipodal):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import salgpu as S
    from oracle import oracle as O
    rng = np.random.default_rng(int(1e9 * chord) + antipodal)
    p = rng.standard_normal((40, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    d = np.cross(p, rng.standard_normal((40, 3)))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    a = 2.0 * np.arcsin(0.5 * chord)
    q = np.cos(a) * p + np.sin(a) * d                  # at the chord from p
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    pts = np.concatenate([p, -q if antipodal else q])
    xs, ys, zs = (np.ascontiguousarray(pts[:, k]) for k in range(3))
    area, h = rng.uniform(0.9, 1.1, 80), rng.standard_normal(80)
    ot = O.tree_traverse(xs, ys, zs, 200)
    L = O.dual_tree_traversal(ot, 0.0, 200)
    ox, oy = O.fast_sum(ot, L, xs, ys, zs, area, h, 8)
    t = S.tree_traverse(xs, ys, zs, 80, 200)
    gx, gy = np.zeros(80), np.zeros(80)
    S.fast_sum(gx, gy, L, t, xs, ys, zs, area, h, 80, 8)
    assert rel_l2(gx, gy, ox, oy) <= 1e-12


@pytest.mark.parametrize("n,nt", [(1, 1), (4, 3), (255, 127), (256, 128), (257, 129), (1023, 33), (2048, 200),
                                  (2049, 2049), (9001, 1), (40000, 300)])
def test_direct_sum_at_tile_and_chunk_edges_matches_oracle(n, nt):
    """sal_direct_sum and its allocation-free form at the edges of the target
    blocks (128), source tiles (256) and source chunks (1,024 and more), on
    random points, whose close pairs reach chords of about 1e-2 / sqrt(n): the
    same 1e-12 bar as the pair kernel's."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import salgpu as S
    from oracle import oracle as O
    rng = np.random.default_rng(n + nt)
    p = rng.standard_normal((n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    xs, ys, zs = (np.ascontiguousarray(p[:, k]) for k in range(3))
    area, h = rng.uniform(0.9, 1.1, n), rng.standard_normal(n)
    tg = np.sort(rng.choice(n, nt, replace=False)).astype(np.int32)
    rx, ry = O.direct_sum(xs, ys, zs, area, h, tg)
    dev = [torch.tensor(v, device="cuda") for v in (xs, ys, zs, area * h, tg)]
    ox, oy = S.direct_sum(*dev)
    nx, ny = torch.full_like(ox, float("nan")), torch.full_like(ox, float("nan"))
    S.direct_sum_noalloc(*dev, nx, ny)
    torch.cuda.synchronize()
    for x, y in ((ox, oy), (nx, ny)):
        assert rel_l2(x.cpu().numpy(), y.cpu().numpy(), rx, ry) <= 1e-12
