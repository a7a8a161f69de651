"""GPU tests of the evaluation and batched kernels at the sizes where their
tiles, row blocks, teams and compile-time degrees change.

Bars, rel-L2 over both components: the FP64 form against the oracle 1e-11 (the
pair kernel's 1e-12, and the BLI bases' own rounding: products of two sums of
up to 15 terms at the 1e-16 level, weighed by a Lebesgue constant below 10,
against sums of random signs that cancel by up to sqrt(n)); the batched form,
on evenly spaced points, against the FP64 accurate form of the same algorithm
5e-6, per field, as for every batched pass: coordinates of a leaf of radius R in
FP32 move a neighbour at the spacing s by 2^-24 R, which is 3 sqrt(3) 2^-24 R / s
of its term, 2.5e-6 at R = 8 s (points closer than the spacing have no such
bound).  Runs that differ only in timing are equal bit for bit.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _points(n, seed):
    rng = np.random.default_rng(seed)
    p = rng.standard_normal((n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    return [np.ascontiguousarray(p[:, k]) for k in range(3)], rng.uniform(0.9, 1.1, n) * 4 * np.pi / n, rng


def _lattice(n, seed):
    k = np.arange(n)
    z = 1.0 - (2.0 * k + 1.0) / n
    a = k * np.pi * (3.0 - np.sqrt(5.0))
    r = np.sqrt(1.0 - z * z)
    rng = np.random.default_rng(seed)
    return [r * np.cos(a), r * np.sin(a), z], rng.uniform(0.9, 1.1, n) * 4 * np.pi / n, rng


def _grid(S, n, leaf, degree, max_fields, seed, points=_points):
    xyz, area, rng = points(n, seed)
    t = S.tree_traverse(*xyz, n, leaf)
    L = S.dual_tree_traversal(t, 0.7, leaf)
    return S.Grid(t, *xyz, area, degree, S.MODE_DTT, L, max_fields=max_fields), xyz, area, rng


# leaves of up to `leaf` points of a uniform set hold about leaf / 2.5 on
# average: one target, a chunk less or more than full, several chunks, 256
@pytest.mark.parametrize("n,leaf,degree", [(400, 2, 1), (900, 11, 2), (1500, 31, 3), (1500, 33, 4), (2500, 64, 5),
                                           (3000, 100, 6), (3500, 129, 7), (4000, 148, 8), (5000, 199, 9),
                                           (6000, 256, 10), (2500, 40, 11), (2500, 40, 12), (3000, 65, 13),
                                           (3000, 97, 14)])
def test_fp64_form_over_leaf_sizes_and_degrees_matches_oracle(n, leaf, degree):
    torch = _torch()
    import salgpu as S
    from oracle import oracle as O
    grid, xyz, area, rng = _grid(S, n, leaf, degree, 1, 7 * n + degree)
    h = rng.standard_normal(n)
    ot = O.tree_traverse(*xyz, leaf)
    rx, ry = O.fast_sum(ot, O.dual_tree_traversal(ot, 0.7, leaf), *xyz, area, h, degree)
    ox, oy = grid.solve(torch.tensor(h[None], device="cuda"), form=S.FORM_REF)
    torch.cuda.synchronize()
    assert rel_l2(ox[0].cpu().numpy(), oy[0].cpu().numpy(), rx, ry) <= 1e-11


@pytest.mark.parametrize("n,leaf,degree,nf,block", [
    (600, 8, 8, 3, 64), (2000, 16, 8, 64, 64), (2000, 17, 8, 1, 64), (3000, 33, 8, 2, 64), (4001, 65, 8, 5, 64),
    (6007, 129, 8, 2, 64), (9001, 200, 8, 1, 64), (2500, 40, 1, 2, 64), (2500, 40, 2, 2, 64), (2500, 40, 3, 2, 64),
    (2500, 40, 4, 2, 64), (2500, 40, 5, 2, 64), (2500, 60, 6, 2, 64), (3000, 60, 7, 2, 64), (3000, 60, 9, 2, 64),
    (3000, 60, 10, 2, 64), (600, 8, 8, 3, 32), (2000, 17, 8, 32, 32), (4001, 65, 8, 9, 32), (6007, 129, 6, 1, 32)])
def test_batched_form_over_row_blocks_and_degrees_matches_accurate(n, leaf, degree, nf, block):
    """The leaf, proxy, upward and transfer kernels, FP16 and TF32, tree and
    direct passes."""
    torch = _torch()
    import salgpu as S
    grid, xyz, area, rng = _grid(S, n, leaf, degree, block, 3 * n + degree + block, _lattice)
    ssh = torch.tensor(rng.standard_normal((nf, n)), device="cuda")
    ax, ay = (v.cpu().numpy() for v in grid.solve(ssh, form=S.FORM_ACCURATE))
    for f16, tree in ((0, 1), (1, 1), (0, 0), (1, 0)) if block == 64 else ((0, 1),):
        if block == 64:
            grid.tune(f16=f16, tree_passes=tree, chain_ksteps=32 if f16 else 64)
        mx, my = (v.cpu().numpy() for v in grid.solve(ssh, form=S.FORM_MIXED))
        for f in range(nf):
            assert rel_l2(mx[f], my[f], ax[f], ay[f]) <= 5e-6, (f16, tree, f)


@pytest.mark.parametrize("form,n,leaf", [("REF", 800, 20), ("MIXED", 3000, 40)])
def test_solves_behind_one_another_equal_solves_alone(form, n, leaf):
    """Kernels that come up before their predecessors are through read nothing
    early: solves of changing inputs in the same buffer, one behind the other
    and on two streams, against the same solves with the device idle between."""
    torch = _torch()
    import salgpu as S
    grid, xyz, area, rng = _grid(S, n, leaf, 8, 64, n)
    f = getattr(S, "FORM_" + form)
    hs = [torch.tensor(rng.standard_normal((1, n)) * 10.0 ** k, device="cuda") for k in range(6)]
    alone = []
    for h in hs:
        r = grid.solve(h, form=f)
        torch.cuda.synchronize()
        alone.append([v.clone() for v in r])
    buf = torch.empty_like(hs[0])
    for streams in ([torch.cuda.current_stream()], [torch.cuda.Stream(), torch.cuda.Stream()]):
        torch.cuda.synchronize()
        got = []
        for k in range(18):
            if k:
                streams[k % len(streams)].wait_stream(streams[(k - 1) % len(streams)])
            with torch.cuda.stream(streams[k % len(streams)]):
                buf.copy_(hs[k % 6])
                got.append([v.clone() for v in grid.solve(buf, form=f)])
        torch.cuda.synchronize()
        for k, (x, y) in enumerate(got):
            assert torch.equal(x, alone[k % 6][0]) and torch.equal(y, alone[k % 6][1]), k
