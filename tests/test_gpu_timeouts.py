"""GPU test of the batched leaf pass's time-out path: with sal_grid_inject_timeout
its loaders stop after one stage, so waits of every group run out at their limit of
2 s (no trap, no fault, no endless loop).  The host sees SAL_ETIMEOUT, the flag
clears, and the next solves equal the ones before bit for bit.  What was never
issued is not waited for: the CTAs' limits run side by side, so one solve takes
one limit (2 s) and, with as much again for anything else, less than 4 s.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# TF32; FP16 operands; the kernel-tile store while it records, replays all tiles
# (1) and every second one (2)
@pytest.mark.parametrize("f16,store,solves", [(0, 0, 1), (1, 0, 1), (1, 1, 0), (1, 1, 2), (1, 2, 2)])
def test_batched_leaf_pass_gives_up_and_recovers(f16, store, solves):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import salgpu as S
    from conftest import grid_and_ssh
    g, hh = grid_and_ssh("small_3000", nfields=3, seed=5)
    pt = S.tree_traverse(g.xs, g.ys, g.zs, g.n, 100)
    L = S.dual_tree_traversal(pt, 0.7, 100)
    ssh = torch.tensor(np.ascontiguousarray(hh), device="cuda")

    def grid():
        x = S.Grid(pt, g.xs, g.ys, g.zs, g.areas, 8, S.MODE_DTT, L, max_fields=64)
        x.tune(f16=f16, tile_store=store, chain_ksteps=64)
        return x

    ref = [v.clone() for v in grid().solve(ssh, form=S.FORM_MIXED)]
    x = grid()
    for _ in range(solves):
        x.solve(ssh, form=S.FORM_MIXED)
    torch.cuda.synchronize()
    x.inject_timeout(1)
    t0 = time.perf_counter()
    x.solve(ssh, form=S.FORM_MIXED)
    torch.cuda.synchronize()
    took = time.perf_counter() - t0
    with pytest.raises(S.SalError) as e:
        x.sync()
    assert e.value.code == S.SAL_ETIMEOUT
    x.sync()                       # the flag was cleared
    for _ in range(3):             # recorded again, replayed
        got = x.solve(ssh, form=S.FORM_MIXED)
        torch.cuda.synchronize()
        x.sync()
        assert all(torch.equal(a, b) for a, b in zip(got, ref))
    assert took < 4.0
