"""9..16 tokens of small weights, where a linear takes one launch or two by the kind of its rows: both types in turn on one
workspace, counts on either side of the rule's lines, rows that allow 16-byte loads and rows that do not, results on the device
and on the host, and the explicit choice of a family.  Bit for bit."""
import numpy as np
import pytest
import torch

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1024, 1500, 1025])
@pytest.mark.parametrize("M", [9, 10, 11, 12, 13, 16])
def test_both_types_on_one_workspace(gpu, oracle, M, K):
    _, dom, _ = gpu
    N = 300
    B, sw = make_weights(K, N, seed=K)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    assert ws.schedule()[0] == 3
    data = {d: make_activations(M, K, seed=M, dtype=d) for d in ("f16", "f32")}
    ref = {d: oracle.linear(a, B, sw) for d, a in data.items()}
    stream = torch.cuda.current_stream().cuda_stream
    for turn in range(3):
        if turn == 2:
            assert ws.set_schedule(3, 0) == 0            # asked for by name: one launch whatever the rows
        for d, a in data.items():
            half = d == "f16"
            out = np.zeros((M, N), np.uint16 if half else np.float32)
            assert (ws.run_f16 if half else ws.run_f32)(w, a, out) == 0
            assert np.array_equal(bits(out), bits(ref[d][1])), (turn, d)
            acc = np.zeros((M, N), np.int32)
            assert ws.run_acc_i32(w, a, acc) == 0 and np.array_equal(acc, ref[d][2]), (turn, d)
            da = torch.from_numpy(a.view(np.int16) if half else a).cuda()
            do = torch.zeros((M, N), dtype=da.dtype, device="cuda")
            before = ws.launch_count()
            assert (ws.enqueue_f16 if half else ws.enqueue_f32)(w, da, do, stream) == 0
            torch.cuda.synchronize()
            two = turn < 2 and (K % 8 != 0 and M > 10 if half else M > (12 if K % 8 == 0 else 8))
            assert ws.launch_count() - before == (2 if two else 1)
            assert ws.finish() == 0 and np.array_equal(bits(do.cpu().numpy().view(out.dtype)), bits(ref[d][1])), (turn, d)
    bad = data["f32"].copy()
    bad[M - 1, K - 1] = np.nan
    assert ws.run_f32(w, bad, np.zeros((M, N), np.float32)) != 0
    out = np.zeros((M, N), np.float32)
    assert ws.run_f32(w, data["f32"], out) == 0 and np.array_equal(bits(out), bits(ref["f32"][1]))
    ws.free()
    w.free()
