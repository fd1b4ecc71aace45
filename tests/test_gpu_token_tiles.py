"""Token counts around the widths of items, as the plan cuts them (test_gpu_persist_items.py forces cuts): whole and cut last items,
one k-block and an odd number of them, several items per CTA pair, and an FFN whose two launches cut the tokens differently, its
workspace used as a linear and as a SwiGLU launch in turn.  Bit for bit."""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200 import w8a8
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, K, N", [(260, 128, 4096), (1157, 128, 1024), (777, 640, 4100), (130, 128, 6000), (195, 384, 6000), (777, 1152, 4096)])
def test_linear(gpu, oracle, M, K, N):
    _, dom, _ = gpu
    B, sw = make_weights(K, N, seed=M)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    A = make_activations(M, K, seed=K, dtype="f16")
    rc, ref, ref_acc, _ = oracle.linear(A, B, sw)
    acc, out = np.zeros((M, N), np.int32), np.zeros((M, N), np.uint16)
    for _ in range(2):
        assert rc == 0 and ws.run_acc_i32(w, A, acc) == 0 and np.array_equal(acc, ref_acc)
        assert ws.run_f16(w, A, out) == 0 and np.array_equal(bits(out), bits(ref))
    ws.free()
    w.free()


@pytest.mark.parametrize("M, K, F, N", [(273, 128, 2048, 96), (390, 256, 3008, 130), (130, 128, 3008, 64)])
def test_ffn(gpu, oracle, M, K, F, N):
    _, dom, _ = gpu
    Bg, sg = make_weights(K, 2 * F, seed=1)
    Bd, sd = make_weights(F, N, seed=2)
    A = make_activations(M, K, seed=3, dtype="f32")
    wg, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bd, sd)
    g, d = rk.Workspace(dom, rk.default_config(M, 2 * F, K)), rk.Workspace(dom, rk.default_config(M, N, F))
    ref = oracle.ffn(A, Bg, sg, Bd, sd, mode=1)
    out = np.zeros((M, 2 * F), np.float32)
    for _ in range(2):                            # the same workspace as a linear and as a SwiGLU launch in turn
        middle, C = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32)
        assert rk.run_ffn_f32(g, wg, d, wd, A, middle, C) == 0
        assert np.array_equal(bits(middle), bits(ref["middle"])) and np.array_equal(bits(C), bits(ref["C"]))
        assert g.run_f32(wg, A, out) == 0 and np.array_equal(bits(out), bits(oracle.linear(A, Bg, sg)[1]))
    for x in (g, d, wg, wd):
        x.free()


@pytest.mark.parametrize("M, K, N", [(260, 128, 8192), (390, 128, 6000), (208, 520, 14336)])
def test_int8_weights(gpu, oracle, M, K, N):
    _, dom, _ = gpu
    rng = np.random.default_rng(M)
    B, sw = rng.integers(-128, 128, size=(K, N), dtype=np.int8), rng.uniform(1e-3, 3e-3, N).astype(np.float32)
    A = make_activations(M, K, seed=K, dtype="f32")
    w = w8a8.MatmulWeights(dom, "f32i8f32", B, sw)
    ws = w8a8.MatmulWorkspace(dom, w8a8.default_strategy(w8a8.F32_DYNAMIC, M, N, K))
    out = np.zeros((M, N), np.float32)
    assert ws.run_dynamic(w, A, out) == 0 and np.array_equal(bits(out), bits(oracle.w8_linear(A, B, sw)["out"]))
    ws.free()
    w.free()
