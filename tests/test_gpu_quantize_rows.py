"""Activation rows to int8 codes at the edges of the row kernel: one and two tokens per CTA and an odd last one, every block
size on either side of its lines, rows shorter than one step of a CTA, rows that just fill a thread's registers and rows beyond them, a ragged last
unit, rows that do not allow 16-byte loads; one non-finite element among many rows; collected row maxima against scanned
ones.  Codes, scales and results bit for bit."""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200 import capi, w8a8

pytestmark = pytest.mark.gpu


def rows(M, K, seed):
    rng = np.random.default_rng(seed)
    a = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-6, 7, size=(M, 1)))).astype(np.float32)
    a[0] = 0
    a[M // 2, :min(K, 255)] = np.arange(min(K, 255)) - 127         # whole numbers and, at 127 / 127, exact ties below
    a[M // 2, 1:5] = [.5, -.5, 1.5, -1.5]
    a[M - 1, K - 1] = 300                                          # the maximum is the last element of the last row
    return a


@pytest.mark.parametrize("M, K", [(17, 36), (17, 8200), (18, 16392), (33, 533), (129, 4096), (592, 128), (593, 4096), (593, 4100), (601, 8200),
                                  (296, 1032), (297, 1032), (297, 8184), (297, 8192), (297, 8200), (591, 2056), (592, 2048), (592, 2056), (592, 4096), (592, 4104)])
def test_codes_and_scales(gpu, oracle, M, K):
    _, dom, _ = gpu
    rng = np.random.default_rng(K)
    N = 32
    B, sw = rng.integers(-8, 8, size=(K, N), dtype=np.int8), rng.uniform(1e-3, 3e-3, N).astype(np.float32)
    w = rk.Weights(dom, B, sw)
    ws = rk.Workspace(dom, rk.default_config(M, N, K))
    a = rows(M, K, seed=M + K)
    half = oracle.float_to_half(a)
    for A, run in ((a, ws.run_f32), (half, ws.run_f16)):
        out = np.zeros((M, N), A.dtype)
        assert run(w, A, out) == 0 and ws.run_acc_i32(w, A, np.zeros((M, N), np.int32)) == 0
        rc, s, q = ws.last_quant()
        _, want, inv = oracle.scales(A)
        assert rc == 0 and np.array_equal(bits(s), bits(want)) and np.array_equal(q, oracle.quantize(A, inv))
    for m, k in ((0, 0), (M - 1, K - 1)):
        bad = a.copy()
        bad[m, k] = np.nan if m else np.inf
        assert run(w, oracle.float_to_half(bad), out) == capi.RK_NPU_ERR_PARAM and ws.run_f32(w, bad, np.zeros((M, N), np.float32)) == capi.RK_NPU_ERR_PARAM
    assert run(w, half, out) == 0
    ws.free()
    w.free()


@pytest.mark.parametrize("M, K, F", [(17, 64, 96), (594, 64, 4352), (296, 64, 8256), (297, 64, 8256), (591, 64, 160), (23, 64, 4096), (24, 64, 4096)])
def test_collected_maxima_give_the_scanned_codes(gpu, M, K, F):
    _, dom, _ = gpu
    rng = np.random.default_rng(F)
    N = 64
    gu = rk.Weights(dom, rng.integers(-8, 8, size=(K, 2 * F), dtype=np.int8), rng.uniform(1e-2, 3e-2, 2 * F).astype(np.float32))
    dn = rk.Weights(dom, rng.integers(-8, 8, size=(F, N), dtype=np.int8), rng.uniform(1e-3, 3e-3, N).astype(np.float32))
    w1, w2 = rk.Workspace(dom, rk.default_config(M, 2 * F, K)), rk.Workspace(dom, rk.default_config(M, N, F))
    x = rows(M, K, seed=3)
    for _ in range(2):
        middle, out, again = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32), np.zeros((M, N), np.float32)
        assert rk.run_ffn_f32(w1, gu, w2, dn, x, middle, out) == 0
        assert w2.run_f32(dn, middle, again) == 0 and np.array_equal(bits(out), bits(again))
    for o in (w1, w2, gu, dn):
        o.free()


@pytest.mark.parametrize("dtype", [np.float32, np.uint16], ids=["f32", "f16"])
@pytest.mark.parametrize("M, K", [(17, 40), (593, 4096), (600, 16400)])
def test_typed_operator(gpu, oracle, M, K, dtype):
    _, dom, _ = gpu
    rng = np.random.default_rng(M)
    N = 32
    B, sw = rng.integers(-128, 128, size=(K, N), dtype=np.int8), rng.uniform(1e-3, 3e-3, N).astype(np.float32)
    half = dtype == np.uint16
    family, kinds = ("f16i8f16", (w8a8.F16_DYNAMIC, w8a8.F16_STATIC)) if half else ("f32i8f32", (w8a8.F32_DYNAMIC, w8a8.F32_STATIC))
    w = w8a8.MatmulWeights(dom, family, B, sw)
    a = rows(M, K, seed=5)
    A = oracle.float_to_half(a) if half else a
    scale = rng.uniform(.01, .5, M).astype(np.float32)            # rows beyond 127 steps are clamped
    out = np.zeros((M, N), dtype)
    dyn, sta = (w8a8.MatmulWorkspace(dom, w8a8.default_strategy(k, M, N, K)) for k in kinds)
    assert dyn.run_dynamic(w, A, out) == 0 and np.array_equal(bits(out), bits(oracle.w8_linear(A, B, sw)["out"]))
    assert sta.run_static(w, A, scale, out) == 0 and np.array_equal(bits(out), bits(oracle.w8_linear(A, B, sw, scale)["out"]))
    for o in (dyn, sta, w):
        o.free()
