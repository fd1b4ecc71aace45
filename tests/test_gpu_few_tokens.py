"""Up to sixteen tokens, where the kernel family is chosen call by call: sizes on either side of the rule's lines, both types in turn
on one workspace, rows without 16-byte loads, a projection behind another, and a named family or split, which stay.  Bit for bit."""
import numpy as np
import pytest
import torch

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu

# (M, K, N, launches of a call with fp32 rows, with binary16 rows)
LINEAR = [(1, 8192, 512, 1, 1), (1, 1024, 9500, 1, 1), (3, 3200, 4640, 1, 1), (4, 2044, 4400, 1, 2), (5, 1500, 2048, 1, 1), (5, 3070, 3100, 2, 2),
          (6, 4096, 1040, 2, 1), (8, 4096, 1024, 1, 1), (8, 2048, 1056, 1, 1), (8, 2048, 3200, 1, 1), (7, 1500, 2048, 1, 1), (8, 3104, 3104, 2, 1),
          (9, 1024, 512, 1, 1), (9, 1024, 520, 2, 2), (16, 1030, 2050, 2, 2)]


@pytest.mark.parametrize("M,K,N,fp32,binary16", LINEAR)
def test_linear(gpu, oracle, M, K, N, fp32, binary16):
    _, dom, _ = gpu
    B, sw = make_weights(K, N, seed=K)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    family = ws.schedule()[0]
    stream = torch.cuda.current_stream().cuda_stream
    data = [(d, a := make_activations(M, K, seed=M, dtype=d), oracle.linear(a, B, sw)[1]) for d in ("f32", "f16")]
    for named in (None, 0, 2):                             # by the rule, a family by name, a split
        if named is not None:
            assert ws.set_schedule(family if named == 0 else 0, named) == 0
        for d, a, ref in data:
            half = d == "f16"
            da = torch.from_numpy(a.view(np.int16) if half else a).cuda()
            do = torch.zeros((M, N), dtype=da.dtype, device="cuda")
            before = ws.launch_count()
            assert (ws.enqueue_f16 if half else ws.enqueue_f32)(w, da, do, stream) == 0
            torch.cuda.synchronize()
            assert ws.launch_count() - before == (1 if named is not None else binary16 if half else fp32), (named, d)
            assert ws.finish() == 0 and np.array_equal(bits(do.cpu().numpy().view(ref.dtype)), bits(ref)), (named, d)
            out = np.zeros((M, N), np.uint16 if half else np.float32)
            assert (ws.run_f16 if half else ws.run_f32)(w, a, out) == 0 and np.array_equal(bits(out), bits(ref)), (named, d)
    ws.free()
    w.free()


# (K, F, N)
FFN = [(512, 9024, 192), (256, 4800, 300), (1502, 512, 256), (1024, 5152, 320), (640, 1024, 2304)]


@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("K,F,N", FFN)
def test_ffn(gpu, oracle, M, K, F, N):
    _, dom, _ = gpu
    (Bg, sg), (Bd, sd) = make_weights(K, 2 * F, seed=1), make_weights(F, N, seed=2)
    wg, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bd, sd)
    stream = torch.cuda.current_stream().cuda_stream
    x = torch.from_numpy(make_activations(M, K, seed=M, dtype="f32")).cuda()
    outs = []
    for named in (False, True):
        g, d = (rk.Workspace(dom, rk.default_config(M, n, k)) for n, k in ((2 * F, K), (N, F)))
        if named:
            assert g.set_schedule(g.schedule()[0], 0) == 0 and d.set_schedule(d.schedule()[0], 0) == 0
        for _ in range(2):
            mid, out = torch.zeros((M, F), device="cuda"), torch.zeros((M, N), device="cuda")
            assert rk.enqueue_ffn_f32(g, wg, d, wd, x, mid, out, stream) == 0
            torch.cuda.synchronize()
            assert g.finish() == 0 and d.finish() == 0
            outs.append((mid.cpu().numpy(), out.cpu().numpy()))
        g.free()
        d.free()
    for mid, out in outs[1:]:
        assert np.array_equal(bits(mid), bits(outs[0][0])) and np.array_equal(bits(out), bits(outs[0][1]))
    ref = oracle.linear(outs[0][0], Bd, sd)[1]
    assert np.array_equal(bits(outs[0][1]), bits(ref))
    wg.free()
    wd.free()


@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("M", [1, 9, 17, 31])
def test_ring_parts_of_padded_tiles(gpu, oracle, monkeypatch, M, split):
    # whole warps of a CTA have only tokens or channels that do not exist: launches back to back, nothing written beside the result
    _, dom, _ = gpu
    monkeypatch.setenv("RK_NPU_B200_VARIANT", "1")
    K, N, F = 1100, 130, 96
    (B, sw), (Bg, sg) = make_weights(K, N, seed=3), make_weights(K, 2 * F, seed=4)
    w, wg = rk.Weights(dom, B, sw), rk.Weights(dom, Bg, sg)
    ws, gu = rk.Workspace(dom, rk.default_config(M, N, K)), rk.Workspace(dom, rk.default_config(M, 2 * F, K))
    assert ws.set_schedule(1, split) == 0 and gu.set_schedule(1, split) == 0
    a = make_activations(M, K, seed=M, dtype="f32")
    x = torch.from_numpy(a).cuda()
    ref, (_, _, acc, scales) = oracle.linear(a, B, sw)[1], oracle.linear(a, Bg, sg)
    middle, maxima = oracle.swiglu(acc, scales, sg)
    stream = torch.cuda.current_stream().cuda_stream
    outs, mids = ([torch.full((M + 1, n), -7.0, device="cuda") for _ in range(20)] for n in (N, F))
    tops = torch.zeros((20, M + 1), dtype=torch.int32, device="cuda")
    for out, mid, top in zip(outs, mids, tops):
        assert ws.enqueue_f32(w, x, out, stream) == 0 and gu.enqueue_swiglu_collect_f32(wg, x, mid, top, stream) == 0
    torch.cuda.synchronize()
    assert ws.finish() == 0 and gu.finish() == 0
    for out, mid, top in zip(outs, mids, tops):
        out, mid, top = (t.cpu().numpy() for t in (out, mid, top))
        assert np.array_equal(bits(out[:M]), bits(ref)) and np.all(out[M] == -7.0)
        assert np.array_equal(bits(mid[:M]), bits(middle)) and np.all(mid[M] == -7.0)
        assert np.array_equal(bits(top[:M]), maxima) and top[M] == 0
    for o in (ws, gu, w, wg):
        o.free()


# sizes on the rule's lines by the rounds of the three kernels
LINES = [(7, 4100, 1000, 1, 2), (5, 4100, 1000, 1, 1), (2, 5120, 5632, 1, 2), (4, 4096, 6464, 2, 1), (8, 5120, 9216, 2, 1), (3, 3584, 7680, 2, 1), (6, 5120, 5184, 2, 2), (5, 2048, 4800, 1, 2),
         (2, 4102, 7200, 2, 1), (8, 4096, 11776, 2, 1), (8, 4096, 12288, 2, 2), (1, 8320, 4768, 1, 1)]


@pytest.mark.parametrize("M,K,N,fp32,binary16", LINES)
def test_linear_where_the_ring_is_thin(gpu, oracle, M, K, N, fp32, binary16):
    _, dom, _ = gpu
    B, sw = make_weights(K, N, seed=K)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    stream = torch.cuda.current_stream().cuda_stream
    for d, launches in (("f32", fp32), ("f16", binary16)):
        a = make_activations(M, K, seed=M, dtype=d)
        ref, half = oracle.linear(a, B, sw)[1], d == "f16"
        da = torch.from_numpy(a.view(np.int16) if half else a).cuda()
        do = torch.zeros((M, N), dtype=da.dtype, device="cuda")
        before = ws.launch_count()
        assert (ws.enqueue_f16 if half else ws.enqueue_f32)(w, da, do, stream) == 0
        torch.cuda.synchronize()
        assert ws.launch_count() - before == launches, d
        assert ws.finish() == 0 and np.array_equal(bits(do.cpu().numpy().view(ref.dtype)), bits(ref)), d
    ws.free()
    w.free()
