"""Quantise launches on either side of the lines between their shapes (bytes of a row, tokens), and rows of the typed operators that need
the careful rounding among rows that do not: NaN and infinities, scales that underflow, the caller's scales.  Bit for bit."""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200 import w8a8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, K", [(20, 2048), (20, 2056), (21, 4096), (22, 4104), (591, 8192), (592, 8200), (593, 2048), (594, 4104), (592, 8192), (17, 16392)])
def test_codes_and_scales(gpu, oracle, M, K):
    _, dom, _ = gpu
    rng = np.random.default_rng(K)
    w = rk.Weights(dom, rng.integers(-8, 8, size=(K, 32), dtype=np.int8), rng.uniform(1e-3, 3e-3, 32).astype(np.float32))
    ws = rk.Workspace(dom, rk.default_config(M, 32, K))
    a = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-6, 7, size=(M, 1)))).astype(np.float32)
    a[M // 2] = np.resize(np.arange(-127, 128) / 2, K)             # exact ties
    a[M - 1, K - 1] = -300
    for A, run in ((a, ws.run_f32), (oracle.float_to_half(a), ws.run_f16)):
        assert run(w, A, np.zeros((M, 32), A.dtype)) == 0
        rc, s, q = ws.last_quant()
        _, want, inv = oracle.scales(A)
        assert rc == 0 and np.array_equal(bits(s), bits(want)) and np.array_equal(q, oracle.quantize(A, inv))
    ws.free()
    w.free()


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("M, K", [(18, 40), (40, 4104), (600, 1032), (24, 20480)])
def test_careful_rows(gpu, oracle, M, K, dtype):
    _, dom, _ = gpu
    rng = np.random.default_rng(M + K)
    half = dtype == "f16"
    B, sw = rng.integers(-128, 128, size=(K, 32), dtype=np.int8), rng.uniform(1e-3, 3e-3, 32).astype(np.float32)
    a = rng.standard_normal((M, K)).astype(np.float32)
    a[1, K - 1], a[2, 0], a[2, K // 2], a[3, 5] = np.nan, -np.nan, 1e30, np.inf
    a[4] = 0
    a[5] = 0
    a[5, K - 2] = 6e-8 if half else 1e-45                          # the smallest magnitudes: subnormal, or nothing left of it over 127
    a[6] *= 1e-38 if not half else 1e-6
    a[M - 1, :3] = [-np.inf, np.nan, 3]
    with np.errstate(over="ignore", under="ignore"):
        A = oracle.float_to_half(a) if half else a
    family, kinds = ("f16i8f16", (w8a8.F16_DYNAMIC, w8a8.F16_STATIC)) if half else ("f32i8f32", (w8a8.F32_DYNAMIC, w8a8.F32_STATIC))
    w = w8a8.MatmulWeights(dom, family, B, sw)
    dyn, sta = (w8a8.MatmulWorkspace(dom, w8a8.default_strategy(k, M, 32, K)) for k in kinds)
    scale = rng.uniform(1e-3, .5, M).astype(np.float32)            # products far beyond 127 steps
    out = np.zeros((M, 32), A.dtype)
    for rc, ref in ((lambda: dyn.run_dynamic(w, A, out), oracle.w8_linear(A, B, sw)["out"]), (lambda: sta.run_static(w, A, scale, out), oracle.w8_linear(A, B, sw, scale)["out"])):
        assert rc() == 0
        got, want = (x.view(np.float16) if half else x for x in (out, ref))
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(bits(out)[~np.isnan(want)], bits(ref)[~np.isnan(want)])
    for o in (dyn, sta, w):
        o.free()


@pytest.mark.parametrize("M, K", [(296, 8200), (297, 8200), (298, 4104), (591, 4100), (300, 8192), (297, 16384), (299, 16392), (297, 8196)])
def test_codes_and_scales_of_long_rows_in_more_than_a_round(gpu, oracle, M, K):
    test_codes_and_scales(gpu, oracle, M, K)
