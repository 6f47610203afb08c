"""Selection where scores are below the smallest normal fp32 number: the kernels' approximate scores are then off by more
than their relative error bound says, and the choice has to be the exact expression's all the same."""
import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu

TINY = np.float32(2.0 ** -149)


@pytest.mark.parametrize("n,nc", [(512, 225), (512, 3), (1500, 225), (300, 362), (120, 4672)])    # each of the kernels
def test_selection_among_subnormal_scores(lib, oracle, n, nc):
    """Priors of a few units of 2^-149 over equal visit counts: quotients that lie half way between two such units, which
    a product with a rounded reciprocal puts on either side."""
    import torch
    from omoknuni_small_b200 import capi
    t = synth.make_selection_tree(n, nc, seed=n)
    rng = np.random.default_rng(nc)
    t["W"][:] = 0
    t["VL"][:] = 0
    t["N"][:] = rng.integers(1, 40, (n, 1))
    t["node_visits"][:] = 1
    t["P"][:, :nc] = (rng.integers(0, 60, (n, 1)) + rng.integers(0, 4, (n, nc))) * TINY
    dt = capi.DeviceTree(t)
    sel = dt.select(c_puct=1.0, vl_value=3, apply_vl=False)
    torch.cuda.synchronize()
    assert np.array_equal(sel.cpu().numpy(), oracle.puct_select(synth.copy_tree(t), c_puct=1.0, vl_value=3, apply_vl=False))


def test_descent_among_subnormal_scores(lib, oracle):
    import torch
    from omoknuni_small_b200 import capi
    t = synth.make_selection_tree(512, 225, seed=5)
    rng = np.random.default_rng(6)
    t["W"][:] = 0
    t["VL"][:] = 0
    t["N"][:] = rng.integers(1, 40, (512, 1))
    t["node_visits"][:] = 1
    t["P"][:, :225] = (rng.integers(0, 60, (512, 1)) + rng.integers(0, 4, (512, 225))) * TINY
    t["child_node"] = np.full(t["N"].shape, -1, np.int32)
    ref = synth.copy_tree(t)
    roots = np.arange(512, dtype=np.int32)
    dt = capi.DeviceTree(t)
    paths, plen = dt.traverse(torch.from_numpy(roots).cuda(), sims_per_tree=2, c_puct=1.0, vl_value=0, max_depth=4)
    rp, rl = oracle.traverse(ref, roots, 2, 1.0, 0, 4)
    assert np.array_equal(plen.cpu().numpy(), rl) and np.array_equal(paths.cpu().numpy(), rp)

