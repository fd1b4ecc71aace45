"""The persistent tcgen05 kernel where its items, runs and fragments can go wrong: every width of an item (multiples of 32 up
to the widest of each kernel, the last one cut by the tokens there are), equal runs that begin and end inside a channel tile,
K in parts, an odd number of k-blocks, rows that do not allow a thread's four channels in one store, scales that leave the
fast SiLU, and sums that are zero.  Outputs are exact, so every comparison is bit for bit."""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from rknpu2_matmul_open_b200 import w8a8
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


def bits(x):
    return x.view(np.uint32) if x.dtype == np.float32 else x


# (tokens, K, N): one item of each width and a token more, runs over several channel tiles, long K with few tiles
WIDTHS = [(m, 384, 300) for m in (31, 33, 64, 95, 97, 128, 159, 161, 191, 193, 224, 225, 256, 257, 289)] + [
    (353, 640, 5000), (800, 256, 2304), (777, 5120, 1024), (176, 1152, 14336), (1200, 128, 4096)]


@pytest.mark.parametrize("shape", WIDTHS, ids=lambda s: "x".join(map(str, s)))
def test_linear(gpu, oracle, monkeypatch, shape):
    _, dom, _ = gpu
    M, K, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    B, sw = make_weights(K, N, seed=K + N)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    A = make_activations(M, K, seed=M, dtype="f16")
    rc, ref, ref_acc, _ = oracle.linear(A, B, sw)
    assert rc == 0
    acc = np.zeros((M, N), np.int32)
    assert ws.run_acc_i32(w, A, acc) == 0 and np.array_equal(acc, ref_acc)
    out = np.zeros((M, N), np.uint16)
    assert ws.run_f16(w, A, out) == 0 and np.array_equal(out, ref)
    ws.free()
    w.free()


@pytest.mark.parametrize("dtype", ["f16", "f32", "acc"])
@pytest.mark.parametrize("shape", [(70, 512, 4911), (193, 384, 2050), (300, 8192, 131)], ids=lambda s: "x".join(map(str, s)))
def test_rows_without_wide_stores(gpu, oracle, monkeypatch, shape, dtype):
    _, dom, _ = gpu
    M, K, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    B, sw = make_weights(K, N, seed=K + N)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    A = make_activations(M, K, seed=M, dtype="f32" if dtype == "f32" else "f16")
    rc, ref, ref_acc, _ = oracle.linear(A, B, sw)
    assert rc == 0
    if dtype == "acc":
        out = np.zeros((M, N), np.int32)
        assert ws.run_acc_i32(w, A, out) == 0 and np.array_equal(out, ref_acc)
    else:
        out = np.zeros((M, N), np.uint16 if dtype == "f16" else np.float32)
        assert (ws.run_f16 if dtype == "f16" else ws.run_f32)(w, A, out) == 0 and np.array_equal(bits(out), bits(ref))
    ws.free()
    w.free()


# gate scales below 2^-20 take the careful SiLU; a quarter of the channels has no codes, so that their sums are zero
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e-30])
@pytest.mark.parametrize("shape", [(40, 256, 96, 64), (161, 640, 2080, 128), (250, 384, 4000, 64), (300, 128, 224, 64)],
                         ids=lambda s: "x".join(map(str, s)))
def test_ffn(gpu, oracle, monkeypatch, shape, scale):
    _, dom, _ = gpu
    M, K, F, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    Bg, sg = make_weights(K, 2 * F, seed=K)
    Bd, sd = make_weights(F, N, seed=F)
    Bg[:, ::4] = 0
    sg = (sg * np.float32(scale)).astype(np.float32)
    A = make_activations(M, K, seed=M, dtype="f32")
    wg, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bd, sd)
    g, d = rk.Workspace(dom, rk.default_config(M, 2 * F, K)), rk.Workspace(dom, rk.default_config(M, N, F))
    ref = oracle.ffn(A, Bg, sg, Bd, sd, mode=1)
    middle, C = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32)
    assert rk.run_ffn_f32(g, wg, d, wd, A, middle, C) == 0
    assert np.array_equal(bits(middle), bits(ref["middle"])) and np.array_equal(bits(C), bits(ref["C"]))
    for x in (g, d, wg, wd):
        x.free()


@pytest.mark.parametrize("shape", [(33, 384, 900), (96, 4224, 260), (225, 640, 4100), (257, 256, 333), (777, 1152, 2000)],
                         ids=lambda s: "x".join(map(str, s)))
def test_int8_weights(gpu, oracle, shape):
    _, dom, _ = gpu
    M, K, N = shape
    rng = np.random.default_rng(K + N)
    B = rng.integers(-128, 128, size=(K, N), dtype=np.int8)
    s = rng.uniform(1e-3, 1e-2, size=N).astype(np.float32)
    A = make_activations(M, K, seed=M, dtype="f32")
    w, ws = w8a8.MatmulWeights(dom, "f32i8f32", B, s), w8a8.MatmulWorkspace(dom, w8a8.default_strategy(w8a8.F32_DYNAMIC, M, N, K))
    out = np.zeros((M, N), np.float32)
    assert ws.run_dynamic(w, A, out) == 0 and np.array_equal(bits(out), bits(oracle.w8_linear(A, B, s)["out"]))
    ws.free()
    w.free()
