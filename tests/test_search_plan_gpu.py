"""The two kernels that plan a round's expansion at the edges of their ranges: one simulation, a full block of 1,024
(a thread each) and one game more (the general kernel); the table on, so that edges and positions coincide."""
import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,spt,R", [(1, 1, 40), (64, 16, 6), (65, 16, 6), (1, 64, 12)])
def test_expansion_plan_equals_the_oracle(lib, oracle, T, spt, R):
    from omoknuni_small_b200 import capi
    w = synth.make_weights(synth.net_tensor_shapes(15, 17, 64, 1, 225, 2, 1), seed=9, init="torch_default", bn="random")
    net = capi.Net(17, 15, 1, 64, 225, 2, 1, 256, T * spt).load(w)
    games = synth.make_gomoku_games(T, 15, seed=40 + T, max_moves=20)[0]
    s = capi.Search(net, n_trees=T, sims_per_move=spt * R, leaf_batch=T * spt, max_depth=64, dirichlet_epsilon=0.25,
                    transposition_table=True, seed=7)
    s.debug_hooks(value_quantum=256.0, record_rounds=R)
    _, visits, st = s.run(games)
    pol, val, noise = s.record()
    dev = s.tree()
    ref = oracle.search_move(games, pol[0, :T], noise, 0.25, pol[1:], val[1:], spt, T * (1 + R * spt), c_puct=1.5, vl_value=3,
                             max_depth=64, value_sign=1.0, value_quantum=256.0, tt_seed=7)
    n = ref["nodes"]
    assert dev["nodes"] == n and st["terminal_leaves"] == ref["terminal_leaves"] and capi.device_error_code() == 0
    for key in ("legal_bits", "child_node", "N", "VL", "node_visits"):
        assert np.array_equal(dev[key][:n], ref[key][:n]), key
    for key in ("P", "W"):
        assert np.array_equal(dev[key][:n].view(np.uint32), ref[key][:n].view(np.uint32)), key
    assert np.array_equal(visits, ref["N"][:T, :225])
