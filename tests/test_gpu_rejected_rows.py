"""A row with NaN or Inf rejects its call and no other: good and bad calls back to back on one workspace, without a wait between
them, for the kernels that run behind a quantise launch.  Good outputs bit for bit, outputs of bad calls untouched."""
import numpy as np
import pytest
import torch

import rknpu2_matmul_open_b200 as rk
from conftest import bits
from rknpu2_matmul_open_b200 import capi
from rknpu2_matmul_open_b200.synthetic import make_activations, make_weights

pytestmark = pytest.mark.gpu

# kernel family, cut of the persistent kernel (items of one width, K in parts, runs of several items), tokens, K, N
CASES = [(1, None, 12, 1032, 260), (1, None, 40, 2048, 200), (4, None, 24, 1024, 300), (2, "32,1,0,1", 40, 640, 700), (2, "64,1,0,3", 129, 2048, 512),
         (2, "32,5,2,1", 700, 384, 1300), (2, None, 600, 4104, 256)]


@pytest.mark.parametrize("family, cut, M, K, N", CASES)
def test_good_and_bad_calls_in_turn(gpu, oracle, monkeypatch, family, cut, M, K, N):
    _, dom, _ = gpu
    monkeypatch.setenv("RK_NPU_B200_VARIANT", str(family))
    if cut:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", cut)
    B, sw = make_weights(K, N, seed=K)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    good = make_activations(M, K, seed=M, dtype="f32")
    _, ref, _, _ = oracle.linear(good, B, sw)
    one, every = good.copy(), good.copy()
    one[M - 1, K - 1] = np.nan
    every[:, 3] = np.inf
    a = {"good": torch.from_numpy(good).cuda(), "one": torch.from_numpy(one).cuda(), "every": torch.from_numpy(every).cuda()}
    turns = ["good", "one", "good", "good", "every", "one", "good", "every"]
    outs = [torch.full((M, N), -7.0, device="cuda") for _ in turns]
    stream = torch.cuda.current_stream().cuda_stream
    for kind, out in zip(turns, outs):
        assert ws.enqueue_f32(w, a[kind], out, stream) == 0
    torch.cuda.synchronize()
    for i, (kind, out) in enumerate(zip(turns, outs)):
        got = out.cpu().numpy()
        assert np.array_equal(bits(got), bits(ref)) if kind == "good" else np.all(got == -7.0), (i, kind)
    assert ws.finish() == capi.RK_NPU_ERR_PARAM
    host = np.full((M, N), -7.0, np.float32)
    assert ws.run_f32(w, every, host) == capi.RK_NPU_ERR_PARAM
    assert ws.run_f32(w, good, host) == 0 and np.array_equal(bits(host), bits(ref))
    assert ws.enqueue_f32(w, a["good"], outs[1], stream) == 0
    torch.cuda.synchronize()
    assert ws.finish() == 0 and np.array_equal(bits(outs[1].cpu().numpy()), bits(ref))
    ws.free()
    w.free()


# kernel family, tokens, channels (41 tiles of 256 at twelve tokens)
@pytest.mark.parametrize("family, M, N", [(1, 12, 260), (2, 40, 700), (3, 8, 260), (4, 24, 300), (5, 4, 260), (0, 8, 260), (0, 12, 10300)])
def test_a_verdict_is_reported_once(gpu, oracle, monkeypatch, family, M, N):
    _, dom, _ = gpu
    if family:
        monkeypatch.setenv("RK_NPU_B200_VARIANT", str(family))
    K = 1032
    B, sw = make_weights(K, N, seed=K)
    w, ws = rk.Weights(dom, B, sw), rk.Workspace(dom, rk.default_config(M, N, K))
    good = make_activations(M, K, seed=M, dtype="f32")
    bad = good.copy()
    bad[M - 1, 0] = np.nan
    ref = oracle.linear(good, B, sw)[1]
    stream = torch.cuda.current_stream().cuda_stream
    dev, out, host = {"good": torch.from_numpy(good).cuda(), "bad": torch.from_numpy(bad).cuda()}, torch.zeros((M, N), device="cuda"), np.zeros((M, N), np.float32)

    def queue(kind):
        assert ws.enqueue_f32(w, dev[kind], out, stream) == 0
        torch.cuda.synchronize()

    assert ws.finish() == 0
    queue("bad")
    assert ws.finish() == capi.RK_NPU_ERR_PARAM and ws.finish() == 0
    assert ws.run_f32(w, good, host) == 0 and np.array_equal(bits(host), bits(ref)) and ws.finish() == 0
    assert ws.run_f32(w, bad, host) == capi.RK_NPU_ERR_PARAM and ws.finish() == 0
    timings = capi.W4A8Timings()                                   # (the verdict of a timed call passes through the device's block)
    assert ws.run_f32(w, bad, host, timings) == capi.RK_NPU_ERR_PARAM and ws.finish() == 0
    queue("bad")
    assert ws.run_f32(w, good, host) == 0 and ws.finish() == capi.RK_NPU_ERR_PARAM      # the queued call's
    queue("bad")
    queue("good")
    assert ws.finish() == 0 and np.array_equal(bits(out.cpu().numpy()), bits(ref))
    ws.free()
    w.free()


# kernel family, cut of the persistent kernel, tokens (families 3 and 5 have tickets of their own)
@pytest.mark.parametrize("family, cut, M", [(1, None, 12), (1, None, 40), (2, "32,1,0,1", 40), (2, "64,1,0,3", 129), (2, "32,5,2,1", 200), (4, None, 24), (3, None, 8), (5, None, 4)])
def test_ffn_calls_good_and_bad_in_turn(gpu, oracle, monkeypatch, family, cut, M):
    # one pair of workspaces: NaN in the input, a middle that is not finite, in between good calls with small and large maxima
    _, dom, _ = gpu
    monkeypatch.setenv("RK_NPU_B200_VARIANT", str(family))
    if cut:
        monkeypatch.setenv("RK_NPU_B200_PERSIST_CUT", cut)
    K, F, N = 1024, 1152, 260
    (Bg, sg), (Bd, sd) = make_weights(K, 2 * F, seed=1), make_weights(F, N, seed=2)
    huge = np.where(np.arange(2 * F) % 64 == 5, np.float32(1e30), sg).astype(np.float32)
    wg, wh, wd = rk.Weights(dom, Bg, sg), rk.Weights(dom, Bg, huge), rk.Weights(dom, Bd, sd)
    gu, dn = (rk.Workspace(dom, rk.default_config(M, n, k)) for n, k in ((2 * F, K), (N, F)))
    good = make_activations(M, K, seed=M, dtype="f32")
    nan = good.copy()
    nan[M - 1, K - 1] = np.nan
    rows = {"good": good, "large": 30 * good, "nan": nan, "overflow": good}
    ref = {kind: oracle.ffn(rows[kind], Bg, sg, Bd, sd, mode=1) for kind in ("good", "large")}
    dev = {kind: torch.from_numpy(np.ascontiguousarray(a)).cuda() for kind, a in rows.items()}
    turns = ["large", "nan", "good", "overflow", "good", "nan", "overflow", "large", "good"]
    mids, outs = ([torch.full((M, n), -7.0, device="cuda") for _ in turns] for n in (F, N))
    stream = torch.cuda.current_stream().cuda_stream
    for kind, mid, out in zip(turns, mids, outs):
        assert rk.enqueue_ffn_f32(gu, wh if kind == "overflow" else wg, dn, wd, dev[kind], mid, out, stream) == 0
    torch.cuda.synchronize()
    assert gu.finish() == 0 and dn.finish() == 0
    for i, (kind, mid, out) in enumerate(zip(turns, mids, outs)):
        mid, out = mid.cpu().numpy(), out.cpu().numpy()
        if kind in ref:
            assert np.array_equal(bits(mid), bits(ref[kind]["middle"])) and np.array_equal(bits(out), bits(ref[kind]["C"])), (i, kind)
        else:
            assert np.all(mid == -7.0) if kind == "nan" else not np.isfinite(mid).all() and np.all(out == -7.0), (i, kind)
    middle, result = np.zeros((M, F), np.float32), np.zeros((M, N), np.float32)
    for kind, w in (("overflow", wh), ("good", wg), ("nan", wg), ("large", wg), ("good", wg)):
        rc = rk.run_ffn_f32(gu, w, dn, wd, rows[kind], middle, result)
        assert rc == (0 if kind in ref else capi.RK_NPU_ERR_PARAM), kind
        if kind in ref:
            assert np.array_equal(bits(middle), bits(ref[kind]["middle"])) and np.array_equal(bits(result), bits(ref[kind]["C"])), kind
    for o in (gu, dn, wg, wh, wd):
        o.free()
