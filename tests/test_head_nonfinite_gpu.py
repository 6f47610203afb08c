"""Networks that overflow: bf16 storage does not saturate, so a tower can hold infinities, and weights can be infinite or
beyond bf16's largest number.  The heads compute with inputs and weights split into 16-bit terms; what comes out has to be
what one fp32 product per weight gives (inf * w is an infinity, inf * 0 and inf - inf are NaN, relu and tanh keep NaN)."""
import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu


def class_of(x):
    return np.where(np.isnan(x), 2, np.where(np.isposinf(x), 1, np.where(np.isneginf(x), -1, 0)))


def heads64(w, x):
    """The heads on the tower's planes x in fp64, where only an infinity makes one: (logits, sum |input||weight|), value."""
    relu = lambda v: np.where(v <= 0, 0.0, v)
    out = []
    for name in ("policy", "value"):
        g = {k: w[f"{name}_bn.{k}"].astype(np.float64) for k in ("weight", "bias", "running_mean", "running_var")}
        scale = g["weight"] / np.sqrt(g["running_var"] + 1e-5)
        k = w[f"{name}_conv.weight"][:, :, 0, 0].astype(np.float64) * scale[:, None]
        y = sum(x[:, None, c] * k[None, :, c, None, None] for c in range(x.shape[1]))
        out.append(relu(y + (g["bias"] - g["running_mean"] * scale)[None, :, None, None]).reshape(len(x), -1))
    fc = lambda h, m: np.stack([(h * row).sum(1) for row in m.astype(np.float64)], 1)
    logits = fc(out[0], w["policy_fc.weight"]) + w["policy_fc.bias"]
    hidden = relu(fc(out[1], w["value_fc1.weight"]) + w["value_fc1.bias"])
    value = np.tanh((hidden * w["value_fc2.weight"][0]).sum(1) + w["value_fc2.bias"])
    return logits, fc(out[0], np.abs(w["policy_fc.weight"])) + np.abs(w["policy_fc.bias"]), value


def identity_bn(w, name, c):
    w[name + ".weight"][c], w[name + ".bias"][c], w[name + ".running_mean"][c], w[name + ".running_var"][c] = 1.0, 0.0, 0.0, 1.0


def run(monkeypatch, S, pc, vc, n_inf, resident, change=None, dtype=0):
    """A network of a stem alone, five boards: where a board's planes 2 c and 2 c + 1 are both set, channel c < n_inf of
    the tower is the sum of two numbers of 2e38.  Board 0 has no such cell, board b has b of them, board 4 the last
    cell among them."""
    from omoknuni_small_b200 import capi
    monkeypatch.setenv("OB200_TOWER_RESIDENT", resident)
    A, B = S * S, 5
    w = synth.make_weights(synth.net_tensor_shapes(S, 17, 64, 0, A, pc, vc, value_hidden=32), seed=3, init="torch_default", bn="random")
    for c in range(n_inf):
        w["input_conv.weight"][c] = 0.0
        w["input_conv.weight"][c, 2 * c:2 * c + 2, 1, 1] = 2e38
        identity_bn(w, "input_bn", c)
    if change:
        change(w)
    rng = np.random.default_rng(S)
    planes = np.zeros((B, 17, S, S), np.float32)
    planes[:, 8:] = rng.random((B, 9, S, S)) < 0.3
    for b in range(1, B):
        cells = rng.choice(S * S - 1, b, replace=False)
        cells[3:] = S * S - 1
        for p in range(2 * n_inf):
            planes[b, p].flat[cells] = 1.0
    net = capi.Net(17, S, 0, 64, A, pc, vc, 32, B, tower_dtype=dtype).load(w)
    with np.errstate(all="ignore"):
        logits, value = net.infer_planes(planes, capi.OUT_LOGITS)
        nb = int(capi.lib().ob200_board_tensor_bytes(S, B, 64))
        raw = np.empty(nb, np.uint8)
        capi.check(capi.lib().ob200_copy_to_host(raw.ctypes.data, net.tower_output_ptr(), nb))
        x = capi.board_tensor_to_planes(raw.view(np.uint16), S, B, 64, dtype)[0].astype(np.float64)
        want, scale, want_v = heads64(w, x)
    assert (class_of(x) == 1).any() == (n_inf > 0) and np.isfinite(x[0]).all() and capi.device_error_code() == 0
    net.close()
    return logits, value, want, scale, want_v


@pytest.mark.parametrize("S,resident", [(5, "1"), (5, "0"), (15, "1"), (19, "0")])
@pytest.mark.parametrize("weights", [(0.1,), (-0.1,), (0.3, 0.7), (0.1, -0.1)])
def test_head_convolution_of_infinities(lib, monkeypatch, S, resident, weights):
    """One or two channels of infinities under a single head channel: inf * 0.1 is an infinity (0.1's lower terms in bf16
    have the other sign), inf * -0.1 is zero after relu, their sum is NaN.  Where the head channel is not finite, the
    logits are not; where it is, they are right."""
    def change(w):
        identity_bn(w, "policy_bn", 0)
        w["policy_conv.weight"][0, :len(weights), 0, 0] = weights
    logits, _, want, scale, _ = run(monkeypatch, S, 1, 1, len(weights), resident, change)
    finite = np.isfinite(want)
    assert finite[0].all() and finite.all() == (weights == (-0.1,))
    assert not np.isfinite(logits[~finite]).any()
    assert (np.abs(logits[finite] - want[finite]) <= 2e-5 * scale[finite]).all()


@pytest.mark.parametrize("S,resident", [(15, "1"), (19, "0")])
@pytest.mark.parametrize("weight,dtype", [(np.inf, 0), (-np.inf, 0), (np.nan, 0), (3.4e38, 0), (np.inf, 1), (-np.inf, 1), (np.nan, 1)])
def test_head_convolution_with_weights_out_of_range(lib, monkeypatch, S, resident, weight, dtype):
    """Infinite weights (inf * 0 = NaN on the cells without a stone), and the largest finite ones."""
    def change(w):
        w["input_conv.weight"][40] = 0.0
        w["input_conv.weight"][40, 8, 1, 1] = 0.25                      # channel 40: a quarter where plane 8 has a stone
        identity_bn(w, "input_bn", 40)
        w["policy_conv.weight"][1, 40] = weight
        identity_bn(w, "policy_bn", 1)
        w["policy_fc.weight"] *= 1e-2                                   # products with 8.5e37 and their sums stay finite
    logits, _, want, scale, _ = run(monkeypatch, S, 3, 2, 0, resident, change, dtype)
    finite = np.isfinite(want)
    assert finite.all() == bool(np.isfinite(weight)) and not np.isfinite(logits[~finite]).any()
    assert (np.abs(logits[finite] - want[finite]) <= 2e-5 * scale[finite]).all()


@pytest.mark.parametrize("S,resident", [(5, "1"), (8, "0"), (15, "1"), (19, "0")])
@pytest.mark.parametrize("n_inf", [1, 2])
def test_fully_connected_layers_of_infinities(lib, monkeypatch, S, resident, n_inf):
    """Every logit and value is the infinity, the NaN or the number that fp32 products give; K = 75 to 1,083 terms, which
    end inside a block of 32, the last cell infinite among others."""
    def change(w):
        w["policy_conv.weight"][:, :2] = np.abs(w["policy_conv.weight"][:, :2]) * np.sign(w["policy_bn.weight"])[:, None, None, None]
        w["policy_fc.weight"][0] = np.abs(w["policy_fc.weight"][0])
        w["policy_fc.weight"][1] = -np.abs(w["policy_fc.weight"][1])
        w["policy_fc.weight"][2] = 0.0
        w["policy_fc.weight"][3] = 2.0 ** -3                            # one term: the lower two of the split are zero
    logits, value, want, scale, want_v = run(monkeypatch, S, 3, 2, n_inf, resident, change)
    assert set(np.unique(class_of(want))) == {-1, 0, 1, 2}
    assert np.array_equal(class_of(logits), class_of(want)) and np.array_equal(class_of(value), class_of(want_v))
    finite = np.isfinite(want)
    assert (np.abs(logits[finite] - want[finite]) <= 2e-5 * scale[finite]).all()
    assert np.allclose(value[np.isfinite(want_v)], want_v[np.isfinite(want_v)], atol=1e-5)


@pytest.mark.parametrize("weight", [np.inf, np.nan, 3.4e38, -3.4e38])
def test_fully_connected_weights_out_of_range(lib, monkeypatch, weight):
    def change(w):
        w["policy_bn.weight"] *= 0.05                                   # inputs well below one
        w["policy_bn.bias"] *= 0.05
        w["policy_fc.weight"][7, 0] = weight
    logits, _, want, scale, _ = run(monkeypatch, 15, 3, 2, 0, "1", change)
    assert np.array_equal(class_of(logits), class_of(want))
    finite = np.isfinite(want)
    assert (np.abs(logits[finite] - want[finite]) <= 2e-5 * scale[finite]).all() and finite[:, 8:].all()
