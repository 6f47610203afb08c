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
