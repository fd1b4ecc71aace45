"""The persistent tcgen05 kernel where its items, runs and fragments can go wrong, with cuts of the test's own
(persist_cuts.py) where a width or a run is meant, with the plan's elsewhere: every width of an item in every kernel, several items
a CTA pair, equal runs that begin and end inside a channel tile, K in parts, an odd number of k-blocks, rows that do not allow
a thread's four channels in one store, scales that leave the fast SiLU, and sums that are zero.  Outputs are exact, so every
comparison is bit for bit."""
import numpy as np
import pytest

import rknpu2_matmul_open_b200 as rk
from persist_cuts import GRIDS, LONG, LONG_FFN, PARTS, RUNS, WHOLE, WHOLE_FFN
from rknpu2_matmul_open_b200 import w8a8
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu


def bits(x):
    return x.view(np.uint32) if x.dtype == np.float32 else x


CUTS = [(WHOLE, WHOLE_FFN, GRIDS + RUNS), (LONG, LONG_FFN, PARTS)]


@pytest.mark.parametrize("cuts", CUTS, ids=["whole", "parts"])
def test_linear_in_every_cut(gpu, oracle, monkeypatch, cuts):
    _, dom, _ = gpu
    (M, K, N), _, names = cuts
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    B, sw = make_weights(K, N, seed=K + N)
    w = rk.Weights(dom, B, sw)
    A = make_activations(M, K, seed=M, dtype="f16")
    rc, ref, ref_acc, _ = oracle.linear(A, B, sw)
    assert rc == 0
    for name in names:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", name)
        ws = rk.Workspace(dom, rk.default_config(M, N, K))
        for _ in range(2):                        # the part counters must come back clean
            acc, out = np.zeros((M, N), np.int32), np.zeros((M, N), np.uint16)
            assert ws.run_acc_i32(w, A, acc) == 0 and np.array_equal(acc, ref_acc), name
            assert ws.run_f16(w, A, out) == 0 and np.array_equal(out, ref), name
        ws.free()
    w.free()


@pytest.mark.parametrize("cuts", CUTS, ids=["whole", "parts"])
def test_ffn_in_every_cut(gpu, oracle, monkeypatch, cuts):
    _, dom, _ = gpu
    _, (M, K, columns), names = cuts
    F, N = columns // 2, 64
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    Bg, sg = make_weights(K, 2 * F, seed=K)
    Bd, sd = make_weights(F, N, seed=F)
    A = make_activations(M, K, seed=M, dtype="f32")
    wg, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bd, sd)
    ref = oracle.ffn(A, Bg, sg, Bd, sd, mode=1)
    for name in names:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", name)
        g, d = rk.Workspace(dom, rk.default_config(M, 2 * F, K)), rk.Workspace(dom, rk.default_config(M, N, F))
        for _ in range(2):
            middle, C = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32)
            assert rk.run_ffn_f32(g, wg, d, wd, A, middle, C) == 0
            assert np.array_equal(bits(middle), bits(ref["middle"])) and np.array_equal(bits(C), bits(ref["C"])), name
        g.free()
        d.free()
    wg.free()
    wd.free()


@pytest.mark.parametrize("cuts", CUTS, ids=["whole", "parts"])
def test_int8_weights_in_every_cut(gpu, oracle, monkeypatch, cuts):
    _, dom, _ = gpu
    (M, K, N), _, names = cuts
    rng = np.random.default_rng(K + N)
    B = rng.integers(-128, 128, size=(K, N), dtype=np.int8)
    s = rng.uniform(1e-3, 1e-2, size=N).astype(np.float32)
    A = make_activations(M, K, seed=M, dtype="f32")
    w = w8a8.MatmulWeights(dom, "f32i8f32", B, s)
    ref = oracle.w8_linear(A, B, s)["out"]
    for name in names:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", name)
        ws = w8a8.MatmulWorkspace(dom, w8a8.default_strategy(w8a8.F32_DYNAMIC, M, N, K))
        for _ in range(2):
            out = np.zeros((M, N), np.float32)
            assert ws.run_dynamic(w, A, out) == 0 and np.array_equal(bits(out), bits(ref)), name
        ws.free()
    w.free()


# (tokens, K, N) as the plan cuts them: a token before, at and behind a width, runs over several channel tiles, long K with few tiles
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


# odd rows and rows of two modulo four elements: the plan's cuts, and each kernel's with items cut by the tokens there are
@pytest.mark.parametrize("dtype", ["f16", "f32", "acc"])
@pytest.mark.parametrize("shape", [(70, 512, 4911, None), (193, 384, 2050, None), (300, 8192, 131, None), (117, 384, 1031, "64,1,0,1"), (117, 384, 1030, "64,1,0,1"),
                                   (341, 384, 1031, "160,1,0,1"), (341, 384, 1030, "160,1,0,1"), (485, 256, 1031, "256,1,0,1"), (485, 256, 1030, "256,1,0,1"),
                                   (165, 4200, 701, "160,1,0,3"), (165, 4200, 702, "160,1,0,3")], ids=lambda s: "x".join(map(str, s)))
def test_rows_without_wide_stores(gpu, oracle, monkeypatch, shape, dtype):
    _, dom, _ = gpu
    M, K, N, cut = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    if cut:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", cut)
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
@pytest.mark.parametrize("shape", [(40, 256, 96, 64, None), (161, 640, 2080, 128, None), (250, 384, 4000, 64, None), (300, 128, 224, 64, None),
                                   (341, 384, 2080, 64, "160,1,0,1"), (485, 384, 4000, 64, "256,1,0,1")], ids=lambda s: "x".join(map(str, s)))
def test_ffn(gpu, oracle, monkeypatch, shape, scale):
    _, dom, _ = gpu
    M, K, F, N, cut = shape
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "2")
    if cut:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", cut)
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
