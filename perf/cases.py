"""Performance cases: the work a program that uses this library has it do, through the entry points it calls.

  listed()          the named cases
  draw(rng)         one more case of the same ranges
  prepare(case, s)  inputs and handles such a program holds before the call
  run(state)        one pass through the public entry points, and what it returns
  work(case)        bytes and floating-point operations the pass cannot do without
  tolerance(case)   how far another correct implementation at the same precision may be off

Kinds of case
  eval_host    Gomoku positions in host memory -> policy and value in host memory (Net.infer_gomoku): what an engine's
               evaluator or batch collector calls.
  eval_device  the same on device arrays (Net.forward_gomoku_device): what a device-resident search calls per leaf batch.
  search       one move for a group of games (Search.run), trees and network on the device.
  go_device    Go positions on the device: encoder + 128-filter network (encode_go, Net.forward_device).
  planes_host  input planes in host memory -> network -> host memory (Net.infer_planes): games that make their own planes.
  chess_device 119 fp32 planes on the device -> board tensor -> 256-filter network with 4,672 logits.
  select       PUCT selection with virtual loss over many nodes, then its revert (DeviceTree), rows of 225 / 362 / 4,672.
  tree_host    one iteration of a host search loop on a device tree (ob200_tree_*): select, backup, priors of new nodes.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from omoknuni_small_b200 import capi, synth

DEVICE = "cuda:0"


# ---- the cases ------------------------------------------------------------------
def _eval(kind, batch, board=15, blocks=10, planes=19, heads=32, dtype="bf16", **kw):
    return dict(kw, kind=kind, batch=batch, board=board, blocks=blocks, planes=planes, heads=heads, dtype=dtype)


def listed():
    return [
        # a single position, as an engine without a batch collector or a player on the board asks for it; the network
        # with the reference's own 32-channel heads
        _eval("eval_host", 1, name="eval_host_1"),
        # a batch of the collector (its limit is 256; it rarely fills the last few)
        _eval("eval_host", 250, name="eval_host_250"),
        # the leaf batch of 64 concurrent games, fp16 storage, small heads: the benchmark's step
        _eval("eval_device", 1024, planes=17, heads=2, dtype="f16", name="eval_device_1024"),
        # a whole replay shard evaluated in one call
        _eval("eval_device", 4096, planes=17, heads=2, name="eval_device_4096"),
        # one interactive game, 800 simulations in batches of 16 leaves
        dict(name="search_1_game", kind="search", trees=1, sims=800, leaves=16, heads=32, dtype="bf16", table=False),
        # self-play: 64 games, 800 simulations each, leaf batch 1,024, transposition table
        dict(name="search_64_games", kind="search", trees=64, sims=800, leaves=16, heads=2, dtype="f16", table=True),
        # Go 19x19, 20 blocks of 128 filters: the large-batch evaluation, encoder included
        dict(name="go_device_2048", kind="go_device", batch=2048, board=19, blocks=20, heads=2),
        # Go planes made by the host, a partly filled batch
        dict(name="planes_host_go_93", kind="planes_host", batch=93, board=19, planes=17, filters=128, blocks=20),
        # chess, 20 blocks of 256 filters, convolutional policy head
        dict(name="chess_device_4096", kind="chess_device", batch=4096, blocks=20),
        # one selection over the nodes of a large set of Gomoku trees
        dict(name="select_65536x225", kind="select", nodes=65536, children=225),
        # the same over chess-wide rows
        dict(name="select_2048x4672", kind="select", nodes=2048, children=4672),
        # a host search loop that keeps its statistics on the device, 256 leaves per iteration
        dict(name="tree_host_256", kind="tree_host", nodes=4096, children=225, batch=256, depth=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval_host", "eval_host", "eval_device", "eval_device", "search", "search", "go_device", "planes_host",
                       "chess_device", "select", "select", "tree_host"])
    if kind in ("eval_host", "eval_device"):
        return _eval(kind, _log_int(rng, 1, 4096), board=rng.choice([9, 13, 15, 15, 15, 19]), blocks=rng.choice([5, 10, 10]),
                     planes=rng.choice([17, 19]), heads=rng.choice([2, 32]), dtype=rng.choice(["bf16", "f16"]))
    if kind == "search":
        trees = _log_int(rng, 1, 64)
        return dict(kind=kind, trees=trees, sims=_log_int(rng, 100, 800), leaves=rng.choice([8, 16, 24, 32] if trees <= 32 else [8, 16]),
                    heads=rng.choice([2, 32]), dtype=rng.choice(["bf16", "f16"]), table=rng.choice([False, True]))
    if kind == "go_device":
        return dict(kind=kind, batch=_log_int(rng, 1, 2048), board=rng.choice([9, 13, 19, 19]), blocks=rng.choice([10, 20]),
                    heads=rng.choice([2, 32]))
    if kind == "planes_host":
        board = rng.choice([8, 9, 15, 19, 19])
        return dict(kind=kind, batch=_log_int(rng, 1, 512), board=board, planes=rng.choice([10, 17, 20, 24]),
                    filters=rng.choice([64, 128, 256]), blocks=rng.choice([10, 20]))
    if kind == "chess_device":
        return dict(kind=kind, batch=_log_int(rng, 1, 4096), blocks=rng.choice([10, 20]))
    if kind == "select":
        children = rng.choice([225, 225, 362, 4672])
        return dict(kind=kind, nodes=_log_int(rng, 1, {225: 65536, 362: 40000, 4672: 4096}[children]), children=children)
    return dict(kind=kind, nodes=4096, children=rng.choice([225, 362]), batch=_log_int(rng, 1, 2048), depth=rng.randint(1, 12))


# ---- networks -------------------------------------------------------------------
def _net_shape(case):
    """Arguments of synth.net_tensor_shapes for the case's network."""
    kind = case["kind"]
    if kind in ("eval_host", "eval_device", "search"):
        board = case.get("board", 15)
        heads = case["heads"]
        return dict(board_size=board, input_channels=case.get("planes", 17), filters=64, blocks=case.get("blocks", 10),
                    policy_size=board * board, policy_head_ch=heads, value_head_ch=1 if heads == 2 else heads)
    if kind == "go_device":
        S, heads = case["board"], case["heads"]
        return dict(board_size=S, input_channels=10, filters=128, blocks=case["blocks"], policy_size=S * S + 1, policy_head_ch=heads,
                    value_head_ch=1 if heads == 2 else heads)
    if kind == "planes_host":
        S = case["board"]
        return dict(board_size=S, input_channels=case["planes"], filters=case["filters"], blocks=case["blocks"],
                    policy_size=S * S + 1, policy_head_ch=2, value_head_ch=1)
    return dict(board_size=8, input_channels=119, filters=256, blocks=case["blocks"], policy_size=4672, policy_head_ch=73,
                value_head_ch=1, policy_planes=True)


@functools.lru_cache(maxsize=2)
def _weights(shape_items):
    shape = dict(shape_items)
    # the benchmark's distributions: Kaiming-normal for the 64-filter network, the library default with random
    # BatchNorm statistics for the wider ones
    small = shape["filters"] == 64
    return synth.make_weights(synth.net_tensor_shapes(**shape), seed=42, init="kaiming_normal" if small else "torch_default",
                              bn="identity" if small else "random")


def _net(case, max_batch):
    s = _net_shape(case)
    planes = s.get("policy_planes", False)
    dtype = capi.DTYPE_F16 if case.get("dtype") == "f16" else capi.DTYPE_BF16
    net = capi.Net(s["input_channels"], s["board_size"], s["blocks"], s["filters"], s["policy_size"], s["policy_head_ch"],
                   s["value_head_ch"], 256, max_batch, 0, policy_kind=capi.POLICY_CONV_PLANES if planes else capi.POLICY_FC,
                   tower_dtype=dtype)
    return net.load(_weights(tuple(sorted(s.items()))))


def _net_flops(case):
    s = _net_shape(case)
    if s.pop("policy_planes", False):
        S2, F = s["board_size"] ** 2, s["filters"]
        return (synth.net_flops_per_eval(s["board_size"], s["input_channels"], F, s["blocks"], 0, 0, s["value_head_ch"])
                + 2 * S2 * F * s["policy_head_ch"])
    return synth.net_flops_per_eval(**s)


def _net_weight_bytes(case):
    """Tower weights in 16 bits, everything else in 32."""
    return sum(int(np.prod(shape)) * (2 if len(shape) == 4 and shape[-1] == 3 else 4)
               for _, shape in synth.net_tensor_shapes(**_net_shape(case)))


# ---- inputs ---------------------------------------------------------------------
def _histories(batch, board, seed):
    """Positions of 0 to 100 stones as an encoder takes them: the 16 most recent moves (distinct cells), how many there
    are, the side to move."""
    rng = np.random.default_rng(seed)
    hist = np.argsort(rng.random((batch, board * board), dtype=np.float32), axis=1)[:, :16].astype(np.int16)
    stones = rng.integers(0, min(100, board * board) + 1, batch)
    n_hist = np.minimum(stones, 16).astype(np.uint8)
    hist[np.arange(16)[None, :] >= n_hist[:, None]] = -1
    return np.ascontiguousarray(hist), n_hist, (1 + stones % 2).astype(np.uint8)


def _selection_tree(nodes, children, seed):
    """Edge statistics with the distributions of synth.make_selection_tree, drawn on the GPU."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    pitch, words = synth.tree_pitch(children), synth.tree_mask_words(children)
    words = (words + 3) // 4 * 4
    N = torch.poisson(torch.full((nodes, pitch), 8.0, device=DEVICE), generator=g)
    W = N * (torch.rand((nodes, pitch), device=DEVICE, generator=g) * 2 - 1)
    VL = torch.randint(0, 4, (nodes, pitch), device=DEVICE, generator=g, dtype=torch.int32)
    share = 0.3 + 0.7 * torch.rand((nodes, 1), device=DEVICE, generator=g)
    legal = torch.rand((nodes, children), device=DEVICE, generator=g) < share
    legal[:, 0] |= ~legal.any(1)
    P = torch.zeros((nodes, pitch), device=DEVICE)
    gamma = torch._standard_gamma(torch.full((nodes, children), 0.3, device=DEVICE), generator=g) * legal
    P[:, :children] = gamma / gamma.sum(1, keepdim=True).clamp_min(1e-30)
    visits = 1 + (N[:, :children] * legal).sum(1)
    bits = np.zeros((nodes, words * 32), np.uint8)
    bits[:, :children] = legal.cpu().numpy()
    return {"N": N.int().cpu().numpy(), "W": W.cpu().numpy(), "P": P.cpu().numpy(), "VL": VL.cpu().numpy(),
            "legal_bits": np.packbits(bits, axis=1, bitorder="little").view(np.uint32), "node_visits": visits.int().cpu().numpy(),
            "n_children": children}


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


class _TreeHandle:
    """An ob200_tree, destroyed with the last thing that refers to it."""

    def __init__(self, nodes, children):
        self.value = ctypes.c_void_p()
        capi.check(capi.lib().ob200_tree_create(0, nodes, children, ctypes.byref(self.value)))

    def __del__(self):
        capi.lib().ob200_tree_destroy(self.value)


class _DeviceArray:
    """A device array of a tree handle, for torch.as_tensor; keeps the handle alive."""

    def __init__(self, handle, address, shape, typestr):
        self.handle = handle
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": typestr, "version": 3}


class _HostTree:
    """A tree handle filled with statistics."""

    def __init__(self, nodes, children, seed):
        self.lib = capi.lib()
        self.handle = _TreeHandle(nodes, children)
        self.h = self.handle.value
        t = _selection_tree(nodes, children, seed)
        words = synth.tree_mask_words(children)
        first = ctypes.c_int32()
        capi.check(self.lib.ob200_tree_add_nodes(self.h, nodes, _ptr(np.ascontiguousarray(t["legal_bits"][:, :words])), words,
                                                 ctypes.byref(first)))
        for field, key in ((0, "N"), (1, "W"), (2, "P"), (6, "node_visits")):
            capi.check(self.lib.ob200_tree_write(self.h, field, 0, nodes, _ptr(t[key])))
        v = capi.TreeView()
        capi.check(self.lib.ob200_tree_view_of(self.h, ctypes.byref(v)))
        self.arrays = {key: torch.as_tensor(_DeviceArray(self.handle, getattr(v, key), (nodes, v.pitch), typestr), device=DEVICE)
                       for key, typestr in (("N", "<i4"), ("W", "<f4"), ("P", "<f4"), ("VL", "<i4"))}
        self.legal = np.unpackbits(t["legal_bits"].view(np.uint8), axis=1, bitorder="little")[:, :children]


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind in ("eval_host", "eval_device"):
        B = case["batch"]
        state["net"] = _net(case, B)
        arrays = _histories(B, case["board"], seed)
        A = case["board"] ** 2
        if kind == "eval_host":
            state["in"] = arrays
        else:
            state["in"] = tuple(torch.from_numpy(a).to(DEVICE) for a in arrays)
            state["out"] = (torch.empty((B, A), device=DEVICE), torch.empty(B, device=DEVICE))
    elif kind == "search":
        T = case["trees"]
        leaf_batch = T * case["leaves"]
        state["net"] = _net(case, leaf_batch)
        state["search"] = capi.Search(state["net"], n_trees=T, sims_per_move=case["sims"], leaf_batch=leaf_batch,
                                      transposition_table=case["table"], seed=seed % (1 << 62))
        state["moves"] = synth.make_gomoku_games(T, 15, seed=seed, max_moves=20)[0]   # openings of 0 to 20 stones
    elif kind == "go_device":
        B, S = case["batch"], case["board"]
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        state["net"] = _net(case, B)
        # 0 to 70 % of the points taken, colours even; legal: the empty points
        fill = 0.7 * torch.rand((B, 1), device=DEVICE, generator=g)
        stones = (torch.rand((B, S * S), device=DEVICE, generator=g) < fill).to(torch.int8)
        stones *= torch.randint(1, 3, (B, S * S), device=DEVICE, generator=g, dtype=torch.int8)
        bits = np.zeros((B, (S * S + 31) // 32 * 32), np.uint8)
        bits[:, :S * S] = (stones == 0).cpu().numpy()
        legal = torch.from_numpy(np.packbits(bits, axis=1, bitorder="little").view(np.int32)).to(DEVICE)
        state["in"] = (stones, torch.full((B,), -1, dtype=torch.int32, device=DEVICE),
                       torch.randint(1, 3, (B,), device=DEVICE, generator=g, dtype=torch.uint8), legal)
        state["out"] = (torch.empty((B, S * S + 1), device=DEVICE), torch.empty(B, device=DEVICE))
    elif kind == "planes_host":
        B, S, planes = case["batch"], case["board"], case["planes"]
        state["net"] = _net(case, B)
        state["in"] = (np.random.default_rng(seed).random((B, planes, S, S), dtype=np.float32) < 0.2).astype(np.float32)
    elif kind == "chess_device":
        B = case["batch"]
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        state["net"] = _net(case, B)
        planes = (torch.rand((B, 119, 8, 8), device=DEVICE, generator=g) < 0.1).float()
        planes[:, 112:] = torch.rand((B, 7, 1, 1), device=DEVICE, generator=g)         # scalar planes
        state["in"] = planes
        state["out"] = (torch.empty((B, 4672), device=DEVICE), torch.empty(B, device=DEVICE))
    elif kind == "select":
        state["tree"] = capi.DeviceTree(_selection_tree(case["nodes"], case["children"], seed), DEVICE)
        state["sel"] = torch.empty(case["nodes"], dtype=torch.int32, device=DEVICE)
    else:
        n, depth, nodes = case["batch"], case["depth"], case["nodes"]
        tree = _HostTree(nodes, case["children"], seed)
        rng = np.random.default_rng(seed)
        ids = rng.integers(0, nodes, (n, depth)).astype(np.int32)
        slots = np.argmax(tree.legal[ids] * rng.random((n, depth, case["children"]), dtype=np.float32), axis=2).astype(np.int32)
        policy = rng.random((n, case["children"]), dtype=np.float32)
        state.update(tree=tree, leaf=np.ascontiguousarray(ids[:, -1]), paths=np.ascontiguousarray(np.stack([ids, slots], axis=2)),
                     length=rng.integers(1, depth + 1, n).astype(np.int32), values=rng.uniform(-1, 1, n).astype(np.float32),
                     policy=policy / policy.sum(1, keepdims=True), new=rng.choice(nodes, n, replace=False).astype(np.int32),
                     sel=np.empty(n, np.int32))
    return state


# ---- one pass -------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "eval_host":
        return state["net"].infer_gomoku(*state["in"])
    if kind == "eval_device":
        state["net"].forward_gomoku_device(*state["in"], *state["out"])
        return state["out"]
    if kind == "search":
        pi, visits, _ = state["search"].run(state["moves"])
        return pi, visits
    if kind == "go_device":
        net = state["net"]
        bt = capi.encode_go(*state["in"], state["case"]["board"], net.input_tensor_channels())
        net.forward_device(bt, state["case"]["batch"], *state["out"])
        return state["out"]
    if kind == "planes_host":
        return state["net"].infer_planes(state["in"])
    if kind == "chess_device":
        net = state["net"]
        bt = capi.planes_to_board_tensor(state["in"], net.input_tensor_channels())
        net.forward_device(bt, state["case"]["batch"], *state["out"])
        return state["out"]
    if kind == "select":
        tree = state["tree"]
        tree.select(out=state["sel"])
        tree.vl_revert(state["sel"])
        return state["sel"], tree.t["VL"]
    tree, lib, n, depth = state["tree"], state["tree"].lib, len(state["leaf"]), state["case"]["depth"]
    capi.check(lib.ob200_tree_select(tree.h, _ptr(state["leaf"]), n, 1.5, 3, 1, _ptr(state["sel"])))
    capi.check(lib.ob200_tree_virtual_loss(tree.h, _ptr(state["leaf"]), _ptr(state["sel"]), n, -3))
    capi.check(lib.ob200_tree_backup(tree.h, _ptr(state["paths"]), _ptr(state["length"]), _ptr(state["values"]), n, depth, 3))
    capi.check(lib.ob200_tree_set_priors(tree.h, _ptr(state["new"]), n, _ptr(state["policy"]), state["case"]["children"]))
    return state["sel"], tree.arrays


# ---- what a pass needs, and how exact it is ----------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "select":
        return {"bytes": case["nodes"] * synth.selection_bytes_per_node(case["children"]), "flops": 0}
    if kind == "tree_host":
        row = case["children"] * 16 + synth.tree_mask_words(case["children"]) * 4 + 12
        return {"bytes": case["batch"] * (row + 16 + case["depth"] * 40 + case["children"] * 8), "flops": 0}
    flops, weights = _net_flops(case), _net_weight_bytes(case)
    if kind in ("eval_host", "eval_device"):
        B = case["batch"]
        return {"bytes": weights + B * (34 + 4 * case["board"] ** 2 + 4), "flops": B * flops}
    if kind == "search":
        # per simulation: one evaluation, one new row of statistics written, the rows of a descent of two levels read
        rounds = -(-case["sims"] // case["leaves"])
        sims = rounds * case["leaves"] * case["trees"]
        return {"bytes": weights * rounds + sims * (225 * 20 + 2 * 225 * 16 + 225 * 8), "flops": (sims + case["trees"]) * flops}
    B, s = case["batch"], _net_shape(case)
    inputs = {"go_device": s["board_size"] ** 2 + 53, "planes_host": case.get("planes", 0) * 4 * s["board_size"] ** 2,
              "chess_device": 119 * 64 * 4}[kind]
    return {"bytes": weights + B * (inputs + 4 * s["policy_size"] + 4), "flops": B * flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "select":
        return "exact"                                  # indices and counters
    if kind == "tree_host":
        # value sums are added in fp32 in no fixed order, so a near-tie may flip
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.01}
    if kind == "search":
        # visit counts of a search in which near-ties may fall either way (value sums are added in no fixed order)
        return {"rel": 0.02, "max": 0.5, "differ": 0.01}
    return {"rel": 2e-3 if case.get("dtype") == "f16" else 1e-2}     # 16-bit storage between the layers
