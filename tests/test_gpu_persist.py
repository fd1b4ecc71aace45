"""The persistent tcgen05 kernel as the plan cuts a problem: a few tokens to many, cut channel tiles, K of one stage, of an odd
number of k-blocks and in parts (few channel tiles, long K), part counters and buffers used again.  Sums and outputs are exact, so
every comparison is bit for bit.  (test_gpu_persist_items.py forces the cuts.)"""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from rknpu2_matmul_open_b200 import w8a8
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


def bits(x):
    return x.view(np.uint32) if x.dtype == np.float32 else x


# (tokens, K, N): few channel tiles and many, long K and one k-block, cut channel tiles
SHAPES = [(17, 640, 3400), (64, 8192, 260), (65, 4224, 1100), (96, 384, 1281), (128, 11008, 512), (129, 128, 257), (200, 6000, 300),
          (256, 1100, 2049), (257, 2048, 130), (1030, 4096, 1024)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_linear(gpu, oracle, monkeypatch, shape):
    _, dom, _ = gpu
    M, K, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    B, sw = make_weights(K, N, seed=K + N)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    assert ws.schedule()[0] == 2
    for dtype in ("f16", "f32"):
        A = make_activations(M, K, seed=M, dtype=dtype)
        rc, ref, ref_acc, _ = oracle.linear(A, B, sw)
        assert rc == 0
        acc = np.zeros((M, N), np.int32)
        assert ws.run_acc_i32(w, A, acc) == 0 and np.array_equal(acc, ref_acc)
        for _ in range(2):                        # the part counters must come back clean
            out = np.zeros((M, N), np.uint16 if dtype == "f16" else np.float32)
            assert (ws.run_f16 if dtype == "f16" else ws.run_f32)(w, A, out) == 0
            assert np.array_equal(bits(out), bits(ref))
    ws.free()
    w.free()


@pytest.mark.parametrize("shape", [(50, 8192, 256), (190, 4096, 384), (250, 1152, 1024), (450, 640, 512), (1000, 2176, 256)], ids=lambda s: "x".join(map(str, s)))
def test_new_activations_in_the_same_buffers(gpu, oracle, monkeypatch, shape):
    # the leader's MMAs read both CTAs' activations: a launch that ran ahead of the peer's copy would multiply the rows of
    # the launch before (other rows every time, the same buffers)
    _, dom, _ = gpu
    M, K, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    B, sw = make_weights(K, N, seed=K + N)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    rows = [make_activations(M, K, seed=s, dtype="f16") for s in range(4)]
    refs = [oracle.linear(A, B, sw)[1] for A in rows]
    out = np.zeros((M, N), np.uint16)
    for turn in range(24):
        out.fill(0x7C00)
        assert ws.run_f16(w, rows[turn % 4], out) == 0
        assert np.array_equal(out, refs[turn % 4]), turn
    ws.free()
    w.free()


@pytest.mark.parametrize("shape", [(33, 512, 128, 300), (64, 8192, 192, 130), (128, 4096, 320, 512), (130, 1024, 2496, 257), (520, 640, 1280, 2048)],
                         ids=lambda s: "x".join(map(str, s)))
def test_ffn(gpu, oracle, monkeypatch, shape):
    _, dom, _ = gpu
    M, K, F, N = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    Bg, sg = make_weights(K, 2 * F, seed=K)
    Bd, sd = make_weights(F, N, seed=F)
    A = make_activations(M, K, seed=M, dtype="f32")
    wg, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bd, sd)
    g, d = rk.Workspace(dom, rk.default_config(M, 2 * F, K)), rk.Workspace(dom, rk.default_config(M, N, F))
    ref = oracle.ffn(A, Bg, sg, Bd, sd, mode=1)
    for _ in range(2):
        middle, C = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32)
        assert rk.run_ffn_f32(g, wg, d, wd, A, middle, C) == 0
        assert np.array_equal(bits(middle), bits(ref["middle"])) and np.array_equal(bits(C), bits(ref["C"]))
    for x in (g, d, wg, wd):
        x.free()


@pytest.mark.parametrize("shape", [(1, 300, 64), (64, 4096, 520), (65, 1000, 1300), (128, 8192, 260), (300, 640, 2050)],
                         ids=lambda s: "x".join(map(str, s)))
def test_int8_weights(gpu, oracle, shape):
    _, dom, _ = gpu
    M, K, N = shape
    rng = np.random.default_rng(K + N)
    B = rng.integers(-128, 128, size=(K, N), dtype=np.int8)
    s = rng.uniform(1e-3, 1e-2, size=N).astype(np.float32)
    A = make_activations(M, K, seed=M, dtype="f16")
    w, ws = w8a8.MatmulWeights(dom, "f16i8f16", B, s), w8a8.MatmulWorkspace(dom, w8a8.default_strategy(w8a8.F16_DYNAMIC, M, N, K))
    ref = oracle.w8_linear(A, B, s)["out"]
    for _ in range(2):
        out = np.zeros((M, N), np.uint16)
        assert ws.run_dynamic(w, A, out) == 0 and np.array_equal(out, ref)
    ws.free()
    w.free()
