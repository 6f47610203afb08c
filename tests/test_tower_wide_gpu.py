"""The streamed-weight tower kernel where its split of tiles over CTAs changes: 64 output channels a CTA, one tile a CTA,
CTAs of one and of two tiles in one launch, a last unit of one tile after several of two.  Integer inputs and weights
keep every sum exact, so outputs must equal a plain fp32 convolution's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def integer_layer(rng, B, S, cin, cout):
    """{0, 1} inputs, {-1, 0, 1} weights (4 % non-zero), integer bias and residual: sums are integers far below 2^24."""
    x = (rng.random((B, cin, S, S)) < 0.3).astype(np.float32)
    w = np.sign(rng.normal(size=(cout, cin, 3, 3))).astype(np.float32) * (rng.random((cout, cin, 3, 3)) < 0.04)
    return x, w.astype(np.float32), rng.integers(-3, 4, cout).astype(np.float32), rng.integers(-9, 10, (B, cout, S, S)).astype(np.float32)


@pytest.mark.parametrize("B,S,cin,cout,residual", [
    (1, 15, 64, 128, False),        # 2 tiles, 4 CTAs of 64 channels
    (37, 15, 128, 128, True),       # 74 tiles x 2: the last count that is split by 64 channels on 148 SMs
    (38, 15, 128, 128, True),       # 76 tiles: one tile a CTA, its channels shared by the two epilogue groups
    (18, 15, 256, 256, True), (19, 15, 256, 256, True),
    (37, 15, 64, 256, False),       # 74 tiles: two parts, one tile a CTA
    (74, 15, 128, 128, True),       # 148 tiles
    (75, 15, 128, 128, True),       # 150 tiles: CTAs of one and of two tiles
    (112, 15, 128, 128, False),     # 224
    (186, 15, 128, 128, True),      # 372 tiles: CTAs of two and of three
    (3, 1, 64, 128, False), (1, 30, 64, 128, True),    # the smallest and the largest board
])
def test_wide_tiles_exact(lib, B, S, cin, cout, residual):
    import torch
    import torch.nn.functional as F
    from omoknuni_small_b200 import capi
    rng = np.random.default_rng(B * 100 + S)
    x, w, bias, res = integer_layer(rng, B, S, cin, cout)
    want = F.conv2d(torch.from_numpy(x), torch.from_numpy(w), padding=1).numpy() + bias[None, :, None, None] + (res if residual else 0)
    dev = lambda a: torch.from_numpy(a.view(np.int16)).cuda()
    out = capi.conv3x3(dev(capi.planes_to_board_tensor_host(x, cin)), dev(capi.pack_conv3x3(w, None, cin)), torch.from_numpy(bias).cuda(),
                       dev(capi.planes_to_board_tensor_host(res, cout)) if residual else None, B, S, cin, cout, relu=False)
    torch.cuda.synchronize()
    assert capi.device_error_code() == 0
    got, pad_zero = capi.board_tensor_to_planes(out.cpu().numpy().view(np.uint16), S, B, cout)
    assert np.abs(want).max() <= 256 and np.array_equal(got, want) and pad_zero


@pytest.mark.parametrize("F,cin,B,dtype", [
    (128, 17, 1, 0), (128, 100, 2, 1), (128, 17, 3, 0),    # 1 and 2 input slices; half a unit, a unit, a unit and a half
    (256, 119, 1, 0), (256, 200, 5, 1),                     # 2 and 4 slices
    (256, 119, 74, 1), (256, 119, 75, 0),                   # the last batch of two-board units on 148 SMs, the first of four
    (128, 17, 148, 0), (128, 17, 149, 1),
    (256, 20, 151, 0), (256, 20, 301, 1),                   # CTAs of one and two units; of two and three, the last a quarter full
])
def test_board8_tower_exact(lib, F, cin, B, dtype):
    """Towers on 8x8 boards: stem and one block, rounded to 16 bits after every layer, in exact integer arithmetic."""
    import torch
    import torch.nn.functional as tf
    from omoknuni_small_b200 import capi, synth
    rng = np.random.default_rng(F + B)
    w = synth.make_weights(synth.net_tensor_shapes(8, cin, F, 1, 65, 2, 1), seed=1, init="torch_default", bn="identity")
    x, w["input_conv.weight"], w["input_bn.bias"], _ = integer_layer(rng, B, 8, cin, F)
    _, w["res_blocks.0.conv1.weight"], w["res_blocks.0.bn1.bias"], _ = integer_layer(rng, 1, 8, F, F)
    _, w["res_blocks.0.conv2.weight"], w["res_blocks.0.bn2.bias"], _ = integer_layer(rng, 1, 8, F, F)
    net = capi.Net(cin, 8, 1, F, 65, 2, 1, 256, B + 2, tower_dtype=dtype).load(w)
    stored = torch.float16 if dtype else torch.bfloat16

    def layer(h, conv, bn, res=0.0):
        h = tf.conv2d(h, torch.from_numpy(w[conv]), padding=1) + torch.from_numpy(w[bn])[None, :, None, None] + res
        assert float(h.abs().max()) < 2 ** 15
        return h.clamp(min=0).to(stored).float()

    h0 = layer(torch.from_numpy(x), "input_conv.weight", "input_bn.bias")
    want = layer(layer(h0, "res_blocks.0.conv1.weight", "res_blocks.0.bn1.bias"), "res_blocks.0.conv2.weight", "res_blocks.0.bn2.bias", h0).numpy()
    n16 = int(capi.lib().ob200_board_tensor_bytes(8, B, F)) // 2

    class Out:
        __cuda_array_interface__ = None

    for own_input in (False, True):          # a caller's input tensor, then the handle's own
        if own_input:
            net.infer_planes(x)
        else:
            bt = torch.from_numpy(capi.planes_to_board_tensor_host(x, net.input_tensor_channels(), dtype).view(np.int16)).cuda()
            net.tower_device(bt, B)
        torch.cuda.synchronize()
        Out.__cuda_array_interface__ = dict(data=(net.tower_output_ptr(), False), shape=(n16,), typestr="<i2", version=3)
        tower = torch.as_tensor(Out(), device="cuda").cpu().numpy().view(np.uint16)
        tower = tower.copy()
        tower[(capi.GUARD + B * 81) * F:] = 0          # beyond the batch's boards lie the handle's other boards
        got, pad_zero = capi.board_tensor_to_planes(tower, 8, B, F, dtype)
        assert np.array_equal(got, want) and pad_zero, (own_input, np.abs(got - want).max())
    assert capi.device_error_code() == 0 and np.abs(want).max() > 0
