"""Residual add + RMSNorm where its register form changes shape: the fewest and the most chunks per thread, rows that are no
multiple of the lanes, tokens that do not fill a CTA, the longest rows of either layout, both layouts bit for bit against the
oracle's double-precision statement."""
import numpy as np
import pytest
import torch

from rknpu2_matmul_open_b200 import rmsnorm

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
