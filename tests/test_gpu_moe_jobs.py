"""The streamed expert projections at the edges of their jobs, items and stages: jobs of one, eight, nine and sixteen rows
and one row more, a last item with two of its four blocks, a last stage with one 128-k record, K that is no multiple of
128, more stages than the ring holds; int8 and int4 records; more jobs than SMs.  Bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import bits
from rknpu2_matmul_open_b200 import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form, H, I, E", [("w8", 64, 32, 2), ("w8", 96, 160, 3), ("w8", 544, 512, 160), ("w8", 2656, 64, 2), ("w8", 8128, 512, 2),
                                           ("quant", 64, 64, 2), ("quant", 576, 512, 160), ("quant", 2112, 64, 2), ("quant", 8128, 448, 2)])
def test_jobs_items_and_stages(gpu, oracle, form, H, I, E):
    _, dom, _ = gpu
    rng = np.random.default_rng(H + I)
    lo, hi = (-128, 128) if form == "w8" else (-8, 8) if H < 4096 else (-4, 4)      # (a K tile has to certify)
    grow = 1 if form == "w8" else 16
    ex = dict(gate_up=rng.integers(lo, hi, size=(E, H, 2 * I), dtype=np.int8),
              gate_up_scales=rng.uniform(2e-4, 6e-4, size=(E, 2 * I)).astype(np.float32) * np.float32(grow),
              down=rng.integers(lo, hi, size=(E, I, H), dtype=np.int8),
              down_scales=rng.uniform(1e-3, 3e-3, size=(E, H)).astype(np.float32))
    w = moe.MoeWeights(dom, shared_expert=0, form=form, **ex)
    ws = moe.MoeWorkspace(dom, moe.default_config(H, I, E, 0, 2, 40), form=form)
    for rows in (1, 8, 9, 16, 17, 33):
        codes = rng.integers(-127, 128, size=(rows, H), dtype=np.int8)
        scales = rng.uniform(0.01, 0.05, size=rows).astype(np.float32)
        ids = np.stack([np.full(rows, E - 1), np.arange(rows) % E], axis=1).astype(np.int32)     # one expert takes every row
        routes = rng.uniform(0.05, 0.95, size=(rows, 2)).astype(np.float32)
        out = np.empty((rows, H), np.float32)
        rc, ref = oracle.moe_run(ex, 0, 2, codes, scales, ids, routes, mode=1)
        for _ in range(3):                   # the launches of the first runs of a size are kept and used again
            out.fill(-1)
            assert rc == 0 and ws.run_quantized(w, codes, scales, ids, routes, out) == 0
            assert np.array_equal(bits(out), bits(ref)), rows
        x = rng.standard_normal((rows, H)).astype(np.float32)
        rc, q, s = oracle.moe_quantize_rows(x)
        assert rc == 0
        rc, ref = oracle.moe_run(ex, 0, 2, q, s, ids, routes, mode=1)
        for _ in range(3):
            out.fill(-1)
            assert rc == 0 and ws.run_f32(w, x, ids, routes, out) == 0
            assert np.array_equal(bits(out), bits(ref)), rows
    ws.free()
    w.free()


def test_fewer_rows_than_the_workspace_holds(gpu, oracle):
    # a workspace for 256 rows: batches whose rows still fit the page-locked piece although a power of two of them would not
    # (85 rows of 1536 floats do, 86 do not), and those on either side
    _, dom, _ = gpu
    H, I, E = 1536, 32, 4
    rng = np.random.default_rng(7)
    ex = dict(gate_up=rng.integers(-128, 128, size=(E, H, 2 * I), dtype=np.int8),
              gate_up_scales=rng.uniform(2e-4, 6e-4, size=(E, 2 * I)).astype(np.float32),
              down=rng.integers(-128, 128, size=(E, I, H), dtype=np.int8),
              down_scales=rng.uniform(1e-3, 3e-3, size=(E, H)).astype(np.float32))
    w = moe.MoeWeights(dom, shared_expert=0, form="w8", **ex)
    ws = moe.MoeWorkspace(dom, moe.default_config(H, I, E, 0, 2, 256), form="w8")
    for rows in (64, 65, 70, 85, 86, 128, 129, 256, 70):
        x = rng.standard_normal((rows, H)).astype(np.float32)
        ids = np.stack([np.arange(rows) % E, (np.arange(rows) + 1) % E], axis=1).astype(np.int32)
        routes = rng.uniform(0.05, 0.95, size=(rows, 2)).astype(np.float32)
        rc, q, s = oracle.moe_quantize_rows(x)
        assert rc == 0
        rc, ref = oracle.moe_run(ex, 0, 2, q, s, ids, routes, mode=1)
        assert rc == 0
        for _ in range(3):
            out = np.full((rows, H), -1, np.float32)
            assert ws.run_f32(w, x, ids, routes, out) == 0
            assert np.array_equal(bits(out), bits(ref)), rows
            out.fill(-1)
            assert ws.run_quantized(w, q, s, ids, routes, out) == 0
            assert np.array_equal(bits(out), bits(ref)), rows
    ws.free()
    w.free()


@pytest.mark.parametrize("f32", [True, False])
def test_large_results_do_not_wait_for_other_streams(gpu, oracle, f32):
    # results beyond 512 KB are copied from the device; what the caller has running on the default stream is not waited for
    import torch
    _, dom, _ = gpu
    H, I, E, rows = 1024, 32, 4, 200
    rng = np.random.default_rng(3)
    ex = dict(gate_up=rng.integers(-128, 128, size=(E, H, 2 * I), dtype=np.int8),
              gate_up_scales=rng.uniform(2e-4, 6e-4, size=(E, 2 * I)).astype(np.float32),
              down=rng.integers(-128, 128, size=(E, I, H), dtype=np.int8),
              down_scales=rng.uniform(1e-3, 3e-3, size=(E, H)).astype(np.float32))
    w = moe.MoeWeights(dom, shared_expert=0, form="w8", **ex)
    ws = moe.MoeWorkspace(dom, moe.default_config(H, I, E, 0, 2, rows), form="w8")
    x = rng.standard_normal((rows, H)).astype(np.float32)
    ids = np.stack([np.arange(rows) % E, (np.arange(rows) + 1) % E], axis=1).astype(np.int32)
    routes = rng.uniform(0.05, 0.95, size=(rows, 2)).astype(np.float32)
    rc, q, s = oracle.moe_quantize_rows(x)
    assert rc == 0
    rc, ref = oracle.moe_run(ex, 0, 2, q, s, ids, routes, mode=1)
    out = np.zeros((rows, H), np.float32)
    run = (lambda: ws.run_f32(w, x, ids, routes, out)) if f32 else (lambda: ws.run_quantized(w, q, s, ids, routes, out))
    for _ in range(3):                       # (the launches are kept from the second run on)
        assert rc == 0 and run() == 0 and np.array_equal(bits(out), bits(ref))
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(600_000_000)           # a third of a second on the default stream
    busy.record()
    out.fill(0)
    assert run() == 0
    assert not busy.query(), "the call waited for the default stream"
    assert np.array_equal(bits(out), bits(ref))
    torch.cuda.synchronize()
    ws.free()
    w.free()
