"""Results of the host-buffer calls where the way they travel changes: written by the last kernel (a call alone on its
handle, up to 256 KB, rows of up to 512 outputs) or copied (beyond, and while another call is in flight)."""
import threading

import numpy as np
import pytest

from omoknuni_small_b200 import synth

pytestmark = pytest.mark.gpu


def make(S, A, max_batch, filters=64, planes=17, seed=8):
    from omoknuni_small_b200 import capi
    w = synth.make_weights(synth.net_tensor_shapes(S, planes, filters, 1, A, 2, 1), seed=seed, init="torch_default", bn="random")
    return capi, capi.Net(planes, S, 1, filters, A, 2, 1, 256, max_batch).load(w)


def on_device(net, B, A, hist, nh, tm):
    import torch
    pol, val = torch.empty((B, A), device="cuda"), torch.empty(B, device="cuda")
    net.forward_gomoku_device(*(torch.from_numpy(a).cuda() for a in (hist, nh, tm)), pol, val)
    torch.cuda.synchronize()
    return pol.cpu().numpy(), val.cpu().numpy()


@pytest.mark.parametrize("S,A,B", [(15, 225, 1), (15, 225, 289), (15, 225, 290),      # 256 KB lie between 289 and 290 boards
                                   (15, 512, 127), (15, 512, 128), (15, 513, 3), (19, 362, 180), (19, 362, 181)])
def test_results_around_the_limits(lib, S, A, B):
    import torch
    capi, net = make(S, A, 300)
    games = [synth.make_gomoku_games(B, S, seed=70 + i)[1:] for i in range(5)]
    want = [on_device(net, B, A, *g) for g in games]
    for pinned in (False, True):
        t = [(torch.full((B, A), -1.0), torch.full((B,), -1.0)) for _ in games]
        if pinned:
            t = [(p.pin_memory(), v.pin_memory()) for p, v in t]
        outs = [(p.numpy(), v.numpy()) for p, v in t]
        net.infer_gomoku(*games[0], out=outs[0])                          # alone
        tickets = [net.submit_gomoku(*games[i], outs[i]) for i in (1, 2)]  # the second while the first is in flight
        net.wait(tickets[1])                                             # out of order
        third = net.submit_gomoku(*games[3], outs[3])
        net.wait(tickets[0])
        net.wait(third)
        net.infer_gomoku(*games[4], out=outs[4])
        for got, ref in zip(outs, want):
            assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    assert capi.device_error_code() == 0
    net.close()


@pytest.mark.parametrize("B", [40, 300])
def test_four_threads_on_one_handle(lib, B):
    """Batches that are written in place when they happen to be alone, and batches that never are; histories and planes."""
    capi, net = make(15, 225, 300)
    games = [synth.make_gomoku_games(B, 15, seed=90 + i)[1:] for i in range(4)]
    planes = [synth.make_stone_planes(B, 15, 17, seed=i, max_stones=100) for i in range(4)]
    want = [net.infer_gomoku(*games[k]) if k % 2 else net.infer_planes(planes[k]) for k in range(4)]
    bad = []

    def worker(k):
        for _ in range(25):
            got = net.infer_gomoku(*games[k]) if k % 2 else net.infer_planes(planes[k])
            if not (np.array_equal(got[0], want[k][0]) and np.array_equal(got[1], want[k][1])):
                bad.append(k)
    threads = [threading.Thread(target=worker, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and capi.device_error_code() == 0
    net.close()
