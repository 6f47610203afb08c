"""The heads' fully connected layers (tensor cores, fp32 precision) against an fp64 evaluation of the heads on the
very tower output the device produced: inner dimensions around the chunk sizes, output widths around the tile,
batches around the tile of boards and in each of the ways a layer is spread over CTAs."""
import ctypes

import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu

# Error bound per output, as a multiple of sum |x||w|: 16 accumulations of a chunk that may truncate (2^-23 each), 64
# fp32 additions of the 1x1 convolution and at most 40 of chunks, groups and bias (2^-24 each).
BOUND = 16 * 2.0 ** -23 + (64 + 40) * 2.0 ** -24


@pytest.fixture(scope="module")
def api(lib):
    from omoknuni_small_b200 import capi
    return capi


def tower_planes(api, net, S, B):
    nb = int(api.lib().ob200_board_tensor_bytes(S, B, 64))
    raw = np.empty(nb, np.uint8)
    api.check(api.lib().ob200_copy_to_host(raw.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(net.tower_output_ptr()), nb))
    return api.board_tensor_to_planes(raw.view(np.uint16), S, B, 64)[0].astype(np.float64)


def head64(w, name, x):
    g = {k: w[f"{name}_bn.{k}"].astype(np.float64) for k in ("weight", "bias", "running_mean", "running_var")}
    scale = g["weight"] / np.sqrt(g["running_var"] + 1e-5)
    y = np.einsum("bchw,oc->bohw", x, w[f"{name}_conv.weight"][:, :, 0, 0].astype(np.float64), optimize=True)
    y = (y - g["running_mean"][:, None, None]) * scale[:, None, None] + g["bias"][:, None, None]
    return np.maximum(y, 0).reshape(len(x), -1)


@pytest.mark.parametrize("S,pc,vc,H,A,B", [
    (5, 1, 1, 1, 25, 1),            # one chunk, narrower than a stage; one output
    (8, 2, 1, 130, 128, 127),       # 128 and 64 terms: a whole chunk, half a chunk; a tile of outputs exactly, and two more
    (8, 16, 17, 256, 129, 129),     # 1,024 and 1,088 terms: either side of the chunk-size rule
    (15, 2, 1, 256, 225, 300),
    (15, 32, 32, 256, 225, 2),      # single chunks
    (15, 32, 32, 255, 226, 700),    # groups of chunks
    (15, 32, 32, 256, 225, 2100),   # whole layers per CTA, or groups
    (15, 2, 1, 256, 513, 3), (15, 32, 32, 256, 1030, 2), (8, 2, 1, 64, 4672, 40), (15, 32, 32, 64, 1281, 130),   # long rows
])
def test_head_fc_against_fp64(api, S, pc, vc, H, A, B):
    shapes = synth.net_tensor_shapes(S, 17, 64, 1, A, pc, vc, value_hidden=H)
    w = synth.make_weights(shapes, seed=S + pc + B, init="torch_default", bn="random")
    net = api.Net(17, S, 1, 64, A, pc, vc, H, B).load(w)
    logits, v = net.infer_planes(synth.make_stone_planes(B, S, 17, seed=B, max_stones=S * S), api.OUT_LOGITS)
    x = tower_planes(api, net, S, B)
    hp, hv = head64(w, "policy", x), head64(w, "value", x)
    wp, w1, w2 = (w[k].astype(np.float64) for k in ("policy_fc.weight", "value_fc1.weight", "value_fc2.weight"))
    want = hp @ wp.T + w["policy_fc.bias"]
    scale = hp @ np.abs(wp).T + np.abs(w["policy_fc.bias"])
    assert (np.abs(logits - want) <= BOUND * scale).all(), (np.abs(logits - want) / scale).max()
    hidden = np.maximum(hv @ w1.T + w["value_fc1.bias"], 0)
    scale = (hv @ np.abs(w1).T + np.abs(w["value_fc1.bias"])) @ np.abs(w2[0]) + np.abs(w["value_fc2.bias"])
    # tanh is a contraction; its own fp32 error and the H additions of the last layer come on top
    assert (np.abs(v - np.tanh(hidden @ w2[0] + w["value_fc2.bias"])) <= (BOUND + H * 2.0 ** -24) * scale + 2.0 ** -21).all()
    # probabilities of the same logits; fp32: exponentials within 2 ulp of arguments rounded to 2^-24 of their size, A additions
    probs, _ = net.infer_planes(synth.make_stone_planes(B, S, 17, seed=B, max_stones=S * S))
    e = np.exp(logits.astype(np.float64) - logits.max(1, keepdims=True))
    spread = np.abs(logits - logits.max(1, keepdims=True)).max()
    assert (np.abs(probs - e / e.sum(1, keepdims=True)) <= e / e.sum(1, keepdims=True) * (A + 16 + 2 * spread) * 2.0 ** -23).all()
    # a position's result does not depend on the batch it comes in
    if B > 2:
        part = net.infer_planes(synth.make_stone_planes(B, S, 17, seed=B, max_stones=S * S)[1:2], api.OUT_LOGITS)
        assert np.array_equal(part[0][0], logits[1]) and part[1][0] == v[1]
    net.close()


@pytest.mark.parametrize("F,S,B,pc,vc,dtype", [
    (64, 19, 230, 2, 1, 0),         # 719 tiles of 128 positions: CTAs of one and of two
    (128, 19, 150, 2, 1, 1), (128, 19, 290, 33, 31, 0), (128, 15, 1, 1, 1, 0),
    (256, 19, 100, 2, 1, 0), (256, 8, 40, 40, 30, 1),       # 70 channels: two groups
])
def test_head_convolution_tiles(api, F, S, B, pc, vc, dtype):
    """The stand-alone 1x1 convolutions over towers of every width, several tiles a CTA."""
    w = synth.make_weights(synth.net_tensor_shapes(S, 17, F, 0, 130, pc, vc, value_hidden=64), seed=F + B, init="torch_default", bn="random")
    net = api.Net(17, S, 0, F, 130, pc, vc, 64, B, tower_dtype=dtype).load(w)
    logits, v = net.infer_planes(synth.make_stone_planes(B, S, 17, seed=B, max_stones=S * S), api.OUT_LOGITS)
    nb = int(api.lib().ob200_board_tensor_bytes(S, B, F))
    raw = np.empty(nb, np.uint8)
    api.check(api.lib().ob200_copy_to_host(raw.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(net.tower_output_ptr()), nb))
    x = api.board_tensor_to_planes(raw.view(np.uint16), S, B, F, dtype)[0].astype(np.float64)
    hp, hv = head64(w, "policy", x), head64(w, "value", x)
    wp, w1, w2 = (w[k].astype(np.float64) for k in ("policy_fc.weight", "value_fc1.weight", "value_fc2.weight"))
    bound = BOUND + F * 2.0 ** -24
    assert (np.abs(logits - hp @ wp.T - w["policy_fc.bias"]) <= bound * (hp @ np.abs(wp).T + np.abs(w["policy_fc.bias"]))).all()
    hidden = np.maximum(hv @ w1.T + w["value_fc1.bias"], 0)
    scale = (hv @ np.abs(w1).T + np.abs(w["value_fc1.bias"])) @ np.abs(w2[0]) + np.abs(w["value_fc2.bias"])
    assert (np.abs(v - np.tanh(hidden @ w2[0] + w["value_fc2.bias"])) <= (bound + 64 * 2.0 ** -24) * scale + 2.0 ** -21).all()
    assert api.device_error_code() == 0
    net.close()
