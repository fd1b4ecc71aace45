"""Results of blocking calls on host arrays around the rule that has the kernel store them over the bus: rows that do not start
on a sector, each kernel family, both types, ordinary and page-locked arrays, nothing outside the result touched."""
import numpy as np
import pytest
import torch

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "f32"])
@pytest.mark.parametrize("M, K, N", [(3, 512, 7001), (4, 640, 4911), (4, 256, 14330), (8, 512, 2900), (8, 512, 4911), (6, 256, 28672), (8, 128, 40000), (13, 512, 4910),
                                     (16, 512, 2900), (40, 512, 1023)])
def test_ragged_results(gpu, oracle, M, K, N, dtype):
    _, dom, _ = gpu
    B, sw = make_weights(K, N, seed=N)
    A = make_activations(M, K, seed=M, dtype=dtype)
    ref = bits(oracle.linear(A, B, sw)[1])
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    run = ws.run_f16 if dtype == "f16" else ws.run_f32
    for pinned in (False, True):
        a = torch.from_numpy(A.view(np.int16) if dtype == "f16" else A)
        flat = torch.full((M * N + 128,), 0x5555 if dtype == "f16" else -7, dtype=a.dtype)
        if pinned:
            a, flat = a.pin_memory(), flat.pin_memory()
        out = flat[64:-64].numpy().view(ref.dtype)
        for _ in range(2):
            out.fill(0)
            assert run(w, a.numpy().view(A.dtype), out.view(np.uint16 if dtype == "f16" else np.float32)) == 0
            assert np.array_equal(out.reshape(M, N), ref)
        assert torch.all(flat[:64] == flat[0]) and torch.all(flat[-64:] == flat[0])
    ws.free()
    w.free()
