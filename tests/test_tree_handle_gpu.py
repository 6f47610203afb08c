"""The tree handle's calls on host arrays against the oracle, on both sides of the sizes at which ids, results and priors
are copied instead of read and written in page-locked memory, for rows of each selection kernel."""
import ctypes as C

import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu

FIELDS = {"N": (0, np.int32), "W": (1, np.float32), "P": (2, np.float32), "VL": (3, np.int32), "node_visits": (6, np.int32)}


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


class Handle:
    """An ob200_tree holding a selection tree's nodes and statistics."""

    def __init__(self, t):
        from omoknuni_small_b200 import capi
        self.lib, self.check = capi.lib(), capi.check
        self.h = C.c_void_p()
        self.nodes, self.pitch = t["N"].shape
        self.check(self.lib.ob200_tree_create(0, self.nodes, t["n_children"], C.byref(self.h)))
        first = C.c_int32()
        words = t["legal_bits"].shape[1]
        self.check(self.lib.ob200_tree_add_nodes(self.h, self.nodes, ptr(t["legal_bits"]), words, C.byref(first)))
        for key, (field, _) in FIELDS.items():
            self.check(self.lib.ob200_tree_write(self.h, field, 0, self.nodes, ptr(t[key])))

    def read(self, key):
        field, dtype = FIELDS[key]
        a = np.empty(self.nodes if key == "node_visits" else (self.nodes, self.pitch), dtype)
        self.check(self.lib.ob200_tree_read(self.h, field, 0, self.nodes, ptr(a)))
        return a

    def close(self):
        self.lib.ob200_tree_destroy(self.h)


@pytest.mark.parametrize("nc", [225, 362, 4672])
@pytest.mark.parametrize("n", [1, 7, 512, 513, 1100])
def test_one_iteration_of_a_host_loop(lib, oracle, nc, n):
    """select + virtual loss, its revert, backup, priors: indices, counters and priors equal, value sums (multiples of
    1/8, exact in any order) too.  The priors' total lies below and above 256 KB, with rows that are whole 128-byte lines
    (4,672) and rows that are not."""
    t = synth.make_selection_tree(1200, nc, seed=nc + n)
    t["W"] = np.round(t["W"] * 8) / np.float32(8)
    ref = synth.copy_tree(t)
    tree = Handle(t)
    rng = np.random.default_rng(n)
    ids = rng.permutation(1200)[:n].astype(np.int32)
    sel = np.empty(n, np.int32)
    tree.check(tree.lib.ob200_tree_select(tree.h, ptr(ids), n, 1.5, 3, 1, ptr(sel)))
    want = oracle.puct_select(ref, ids, c_puct=1.5, vl_value=3, apply_vl=True)
    assert np.array_equal(sel, want) and np.array_equal(tree.read("VL"), ref["VL"])
    tree.check(tree.lib.ob200_tree_virtual_loss(tree.h, ptr(ids), ptr(sel), n, -3))
    oracle.vl_revert(ref, want, 3, ids)
    assert np.array_equal(tree.read("VL"), ref["VL"])
    depth = 5
    paths = np.stack([rng.integers(0, 1200, (n, depth)), rng.integers(0, nc, (n, depth))], 2).astype(np.int32)
    length = rng.integers(0, depth + 1, n).astype(np.int32)
    values = (rng.integers(-8, 9, n) / 8).astype(np.float32)
    tree.check(tree.lib.ob200_tree_backup(tree.h, ptr(paths), ptr(length), ptr(values), n, depth, 3))
    oracle.backup(ref, paths, length, values, 3)
    policy = rng.uniform(-0.2, 1.2, (n, nc)).astype(np.float32)
    tree.check(tree.lib.ob200_tree_set_priors(tree.h, ptr(ids), n, ptr(policy), nc))
    oracle.set_priors(ref, ids, policy)
    for key in FIELDS:
        assert np.array_equal(tree.read(key), ref[key]), key
    tree.close()


@pytest.mark.parametrize("nc,policy_size", [(3, 3), (225, 225), (225, 100), (256, 256), (257, 257), (362, 362), (362, 100),
                                             (4672, 4672), (4672, 4673), (4672, 3)])
@pytest.mark.parametrize("actions", [False, True])
def test_set_priors(lib, oracle, nc, policy_size, actions):
    """The prior kernel on device arrays: rows of one block of 256 slots and of several, policies shorter than the rows
    (0.01 for what they do not reach), slot-to-action tables with actions out of range, ids out of range (skipped)."""
    import torch
    from omoknuni_small_b200 import capi
    t = synth.make_selection_tree(40, nc, seed=nc)
    ref = synth.copy_tree(t)
    rng = np.random.default_rng(policy_size)
    ids = rng.permutation(40)[:21].astype(np.int32)
    policy = rng.uniform(-0.2, 1.2, (23, policy_size)).astype(np.float32)
    policy[3, 0], policy[4, -1] = np.nan, np.inf
    table = rng.integers(-3, policy_size + 3, t["N"].shape).astype(np.int32) if actions else None
    oracle.set_priors(ref, ids, policy[:21], table)
    dt = capi.DeviceTree(t)
    all_ids = torch.from_numpy(np.concatenate([ids, np.array([-1, 40], np.int32)])).cuda()
    dt.set_priors(all_ids, torch.from_numpy(policy).cuda(), None if table is None else torch.from_numpy(table).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(dt.host("P"), ref["P"])


@pytest.mark.parametrize("n,depth", [(8192, 16), (8193, 16), (131073, 1)])    # 1 MB of paths, and just beyond
def test_backup_of_many_paths(lib, oracle, n, depth):
    t = synth.make_selection_tree(300, 225, seed=n)
    t["W"] = np.round(t["W"] * 8) / np.float32(8)
    ref = synth.copy_tree(t)
    tree = Handle(t)
    rng = np.random.default_rng(depth)
    paths = np.stack([rng.integers(0, 300, (n, depth)), rng.integers(0, 225, (n, depth))], 2).astype(np.int32)
    length = rng.integers(0, depth + 1, n).astype(np.int32)
    values = (rng.integers(-8, 9, n) / 8).astype(np.float32)
    tree.check(tree.lib.ob200_tree_backup(tree.h, ptr(paths), ptr(length), ptr(values), n, depth, 3))
    oracle.backup(ref, paths, length, values, 3)
    for key in FIELDS:
        assert np.array_equal(tree.read(key), ref[key]), key
    tree.close()
