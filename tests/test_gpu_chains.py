"""GPU test of solves enqueued directly behind one another: every kernel of a solve
comes up while the one before it ends, also across two solves, and must read nothing
of the solve before.  Expectations come from fresh grids, one solve each; the runs
take distinct inputs, filled beforehand, in shuffled order, into outputs of their
own, with nothing in between, on one stream and with solve graphs.  Equal bit for
bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,block,f16,tree", [("REF", 1, 0, 1), ("ACCURATE", 1, 0, 1), ("MIXED", 32, 0, 1),
                                                 ("MIXED", 64, 0, 1), ("MIXED", 64, 1, 1), ("MIXED", 64, 1, 0)])
@pytest.mark.parametrize("graphs", [False, True])
def test_back_to_back_solves_equal_fresh_grids(form, block, f16, tree, graphs):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if graphs and form != "MIXED":
        pytest.skip("graphs hold batched solves")
    import salgpu as S
    n, leaf = 2000, 30
    rng = np.random.default_rng(block + f16)
    p = rng.standard_normal((n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    xyz, area = [np.ascontiguousarray(p[:, k]) for k in range(3)], rng.uniform(0.9, 1.1, n)
    t = S.tree_traverse(*xyz, n, leaf)
    L = S.dual_tree_traversal(t, 0.7, leaf)

    def grid():
        g = S.Grid(t, *xyz, area, 6, S.MODE_DTT, L, max_fields=block)
        if block == 64:
            g.tune(f16=f16, tree_passes=tree, chain_ksteps=64)
        return g

    f = getattr(S, "FORM_" + form)
    hs = [torch.tensor(rng.standard_normal((2, n)) * 10.0 ** (k % 5 - 2), device="cuda") for k in range(7)]
    alone = []
    for h in hs:
        r = grid().solve(h, form=f)
        torch.cuda.synchronize()
        alone.append([v.clone() for v in r])
    g = grid()
    outs = [[torch.full_like(hs[0], float("nan")) for _ in range(2)] for _ in hs]
    g.set_graphs(graphs)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        for _ in range(3 if graphs else 0):   # each shape is captured on its second solve
            for k in range(len(hs)):
                g.solve(hs[k], form=f, out=outs[k])
        torch.cuda.synchronize()
        for _ in range(6):
            for o in outs:
                for v in o:
                    v.fill_(float("nan"))
            for k in rng.permutation(len(hs)):
                g.solve(hs[k], form=f, out=outs[k])
            torch.cuda.synchronize()
            for k in range(len(hs)):
                assert torch.equal(outs[k][0], alone[k][0]) and torch.equal(outs[k][1], alone[k][1]), k
