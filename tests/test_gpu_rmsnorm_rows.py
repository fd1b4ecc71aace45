"""Residual add + RMSNorm where its register form changes shape: the fewest and the most chunks per thread, rows that are no
multiple of the lanes, tokens that do not fill a CTA, the longest rows of either layout, both layouts bit for bit against the
oracle's double-precision statement."""
import numpy as np
import pytest
import torch

import rknpu2_matmul_open_b200 as rk
from rknpu2_matmul_open_b200 import rmsnorm
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row_major", [True, False])
@pytest.mark.parametrize("shape", [(1, 8), (1, 32768), (3, 264), (7, 4104), (9, 8192), (33, 8200), (129, 2040), (65, 16384), (600, 4096), (2050, 4096), (1300, 6552)],
                         ids=lambda s: "x".join(map(str, s)))
def test_rows(gpu, oracle, shape, row_major):
    _, dom, _ = gpu
    M, D = shape
    rng = np.random.default_rng(M + D)
    x = rng.normal(0, 0.8, (M, D)).astype(np.float16).view(np.uint16)
    r = rng.normal(0, 1.5, (M, D)).astype(np.float16).view(np.uint16)
    if M > 2:
        x[1] = 0                                  # a row of zeros
        r[1] = 0
        x[2], r[2] = 0x7BFF, 0x0400               # the largest value next to the smallest normal one
    gamma = rng.normal(1, 0.2, D).astype(np.float16).view(np.uint16)
    gamma[: min(D, 4)] = (0, 0x0001, 0x7BFF, 0x8000)[: min(D, 4)]
    plan = rmsnorm.AddRmsNormPlan(dom, rmsnorm.default_config(M, D), gamma)
    lay = (lambda a: a.reshape(-1)) if row_major else rmsnorm.to_block8
    back = (lambda a: a.reshape(M, D)) if row_major else (lambda a: rmsnorm.from_block8(a, M, D))
    dx, dr = (torch.from_numpy(lay(a).astype(np.int16)).cuda() for a in (x, r))
    ds, dn = torch.full_like(dx, 77), torch.full_like(dx, 77)
    assert plan.enqueue(M, row_major, dx.data_ptr(), dr.data_ptr(), ds.data_ptr(), dn.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    want_s, want_n = oracle.add_rmsnorm_f16(x, r, gamma)
    assert np.array_equal(back(ds.cpu().numpy().view(np.uint16)), want_s)
    assert np.array_equal(back(dn.cpu().numpy().view(np.uint16)), want_n)
    plan.free()


@pytest.mark.parametrize("row_major", [True, False])
@pytest.mark.parametrize("M, K, D", [(1, 512, 1024), (8, 4096, 512), (50, 640, 2048), (300, 512, 1280)])
def test_input_written_by_the_launch_in_front(gpu, oracle, M, K, D, row_major):
    # a linear of every kind writes x on the same stream directly in front; both launches may start before the one in front
    # of them has ended, and x holds other rows every time
    _, dom, _ = gpu
    B, sw = make_weights(K, D, seed=D)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, D, K))
    gamma = np.random.default_rng(D).normal(1, 0.2, D).astype(np.float16).view(np.uint16)
    plan = rmsnorm.AddRmsNormPlan(dom, rmsnorm.default_config(M, D), gamma)
    shaped = (lambda a: a.reshape(M, D)) if row_major else (lambda a: rmsnorm.from_block8(a.reshape(-1), M, D))
    residual = np.random.default_rng(M).normal(0, 1.5, (M, D)).astype(np.float16).view(np.uint16)
    dr = torch.from_numpy(residual.astype(np.int16)).cuda()
    inputs = [make_activations(M, K, seed=s, dtype="f16") for s in range(3)]
    want = [oracle.add_rmsnorm_f16(shaped(oracle.linear(A, B, sw)[1]), shaped(residual), gamma) for A in inputs]
    dev = [torch.from_numpy(A.view(np.int16)).cuda() for A in inputs]
    x = torch.zeros((M, D), dtype=torch.int16, device="cuda")
    outs = [[torch.zeros_like(x), torch.zeros_like(x)] for _ in range(12)]
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for turn, (ds, dn) in enumerate(outs):
        assert ws.enqueue_f16(w, dev[turn % 3], x, stream) == 0
        assert plan.enqueue(M, row_major, x.data_ptr(), dr.data_ptr(), ds.data_ptr(), dn.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    for turn, (ds, dn) in enumerate(outs):
        assert np.array_equal(shaped(ds.cpu().numpy().view(np.uint16)), want[turn % 3][0]), turn
        assert np.array_equal(shaped(dn.cpu().numpy().view(np.uint16)), want[turn % 3][1]), turn
    for h in (plan, ws, w):
        h.free()
