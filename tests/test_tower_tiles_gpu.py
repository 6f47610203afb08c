"""The board-resident tower where its tiles can go wrong: several boards to a tile (boards up to 10x10 in batches beyond
the SM count), odd and even board widths, incomplete last tiles, head channel counts around the extra layer's limits.
Outputs must equal the launch-per-layer path's bit for bit (same products, same order of additions)."""
import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,B,pc,vc,dtype", [
    (5, 1100, 1, 1, 0),       # seven boards to a tile
    (7, 700, 16, 16, 1),
    (9, 333, 17, 3, 0),       # two boards to a tile, the last tile half full
    (10, 297, 2, 1, 1),       # two boards whose rows fill a tile to the last pair
    (10, 298, 32, 32, 0),
    (12, 150, 5, 1, 0), (13, 149, 63, 1, 1), (14, 300, 2, 1, 0), (15, 149, 64, 1, 1),    # 65 channels: their own kernel
])
def test_resident_tiles_equal_layer_by_layer(lib, monkeypatch, S, B, pc, vc, dtype):
    from omoknuni_small_b200 import capi
    w = synth.make_weights(synth.net_tensor_shapes(S, 17, 64, 2, S * S, pc, vc), seed=S, init="torch_default", bn="random")
    x = synth.make_stone_planes(B, S, 17, seed=B, max_stones=S * S)
    outs = []
    for resident in ("1", "0"):
        monkeypatch.setenv("OB200_TOWER_RESIDENT", resident)
        monkeypatch.setenv("OB200_TOWER_FUSED", "0")
        net = capi.Net(17, S, 2, 64, S * S, pc, vc, 256, B, tower_dtype=dtype).load(w)
        outs.append(net.infer_planes(x, capi.OUT_LOGITS))
        assert net.tower_path() == (2 if resident == "1" else 0)
        net.close()
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    assert np.isfinite(outs[0][0]).all() and np.abs(outs[0][0]).max() > 0 and capi.device_error_code() == 0
