"""GPU tests of the FP64 pair kernels on weights that are not finite: a pair of a
source with an infinite weight is a signed infinity, of one with a NaN weight NaN,
as in the reference's sum, and stays so in the chord form, in the vector sums of
far panel pairs and behind the single-tree lists' bitmasks.  Where sums over points
are finite their bar is the pair kernel's 1e-12.  (Sums over proxy weights of random
signs have no such bar: here the reference's own operations are 5.7e-12 off the
value in extended precision.  Their accuracy on fields is the parity tests'.)
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

BAD = {"inf": [np.inf], "-inf": [-np.inf], "nan": [np.nan], "inf, inf": [np.inf, np.inf], "inf, -inf": [np.inf, -np.inf]}


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _caps(per, seed):
    """`per` points within 0.2 of each of the six face centres: two neighbouring
    faces' points are far from one another, those of one face and of opposite
    faces near (close, or antipodal)."""
    rng = np.random.default_rng(seed)
    p = []
    for axis in range(3):
        for sign in (1.0, -1.0):
            c = rng.uniform(-0.2, 0.2, (per, 3))
            c[:, axis] = sign
            p.append(c / np.linalg.norm(c, axis=1, keepdims=True))
    p = np.concatenate(p)
    return [np.ascontiguousarray(p[:, k]) for k in range(3)], rng


def _same(gx, gy, rx, ry, bar=1e-12):
    for g, r in ((gx, rx), (gy, ry)):
        assert np.array_equal(np.isnan(g), np.isnan(r))
        assert np.array_equal(np.isposinf(g), np.isposinf(r)) and np.array_equal(np.isneginf(g), np.isneginf(r))
    ok = np.isfinite(rx) & np.isfinite(ry)
    if ok.any() and bar:
        assert rel_l2(gx[ok], gy[ok], rx[ok], ry[ok]) <= bar


def _fields(n, rng, bad):
    h = rng.standard_normal(n)
    at = rng.choice(n, len(BAD[bad]), replace=False)
    h[at] = BAD[bad]
    return h, at


@pytest.mark.parametrize("bad", list(BAD))
def test_direct_sum(bad):
    torch = _torch()
    import salgpu as S
    from oracle import oracle as O
    xyz, rng = _caps(60, 11)
    n = len(xyz[0])
    h, at = _fields(n, rng, bad)
    tg = np.setdiff1d(np.arange(n), at).astype(np.int32)
    with np.errstate(all="ignore"):
        rx, ry = O.direct_sum(*xyz, np.ones(n), h, tg)
    ox, oy = S.direct_sum(*[torch.tensor(v, device="cuda") for v in (*xyz, h, tg)])
    torch.cuda.synchronize()
    _same(ox.cpu().numpy(), oy.cpu().numpy(), rx, ry)


@pytest.mark.parametrize("per", [30, 90])
@pytest.mark.parametrize("bad", list(BAD))
def test_reference_form(bad, per):
    """One leaf a face and every interaction particle-particle, far stages among
    them; 90 targets leave a last chunk of 26 lanes, 30 are folded."""
    _torch()
    import salgpu as S
    from oracle import oracle as O
    xyz, rng = _caps(per, per)
    n = len(xyz[0])
    h, at = _fields(n, rng, bad)
    ot = O.tree_traverse(*xyz, 200)
    L = O.dual_tree_traversal(ot, 0.0, 200)
    rx, ry = O.fast_sum(ot, L, *xyz, np.ones(n), h, 4)
    gx, gy = np.zeros(n), np.zeros(n)
    S.fast_sum(gx, gy, L, S.tree_traverse(*xyz, n, 200), *xyz, np.ones(n), h, n, 4)
    keep = np.setdiff1d(np.arange(n), at)   # the self pair's value is rounding noise
    _same(gx[keep], gy[keep], rx[keep], ry[keep])


@pytest.mark.parametrize("bad", list(BAD))
def test_single_tree_lists(bad):
    """Particle-cluster sums of given proxy weights and particle-particle sums,
    with bitmasks."""
    _torch()
    import salgpu as S
    from oracle import oracle as O
    xyz, rng = _caps(200, 5)
    n, d, leaf = len(xyz[0]), 3, 12
    h, at = _fields(n, rng, bad)
    ot = O.tree_traverse(*xyz, leaf)
    pc, pp = O.single_tree_traversal(ot, 0.7, leaf, *xyz)
    pt = S.tree_traverse(*xyz, n, leaf)
    grid = S.mom6_grid(pt, pc, pp, *xyz, np.ones(n), d, ref_compat=False)
    rx, ry = O.pp_compute(ot, pp, *xyz, np.ones(n), h)
    gx, gy = np.zeros(n), np.zeros(n)
    grid.pp_compute_host(h, gx, gy)
    keep = np.setdiff1d(np.arange(n), at)
    _same(gx[keep], gy[keep], rx[keep], ry[keep])
    used = (pc[:, 1] - 1)[rng.choice(len(pc), len(BAD[bad]), replace=False)]
    w = rng.standard_normal((d + 1) ** 2 * pt.npanels)
    w[(d + 1) ** 2 * used + rng.integers(0, (d + 1) ** 2, len(used))] = BAD[bad]
    rx, ry = O.pc_compute(ot, pc, *xyz, d, w)
    gx, gy = np.zeros(n), np.zeros(n)
    grid.pc_compute_host(w, gx, gy)
    assert not np.isfinite(rx).all()
    _same(gx, gy, rx, ry, None)
