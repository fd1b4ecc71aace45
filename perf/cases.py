"""The work that users have this library do, as cases that can be timed and compared.

Each case is one pass through the Python mirror of the C interface: quantised linears (one call, or the seven of a
decoder layer), the fused FFN, the typed W8A8 operators, routed experts and the residual add + RMSNorm in front of an
FFN, with the value distributions of the repository's benchmark: weights N(0, 0.02) quantised per output channel,
activations N(0, 1) with 0.5 % of the channels scaled by 20.  What a program sets up once (context, packed weights,
workspaces, plans, output tensors) is made in prepare(); run() makes the calls that recur.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rknpu2_matmul_open_b200 as rk
from rknpu2_matmul_open_b200 import capi, moe, rmsnorm, w8a8

_MOE_FORMS = ("w8", "quant", "w4")            # int8 experts; int4 experts; int4 experts with an int8 shared one
_W8_KINDS = {"f16_dynamic": w8a8.F16_DYNAMIC, "f32_dynamic": w8a8.F32_DYNAMIC, "f16_static": w8a8.F16_STATIC,
             "i8": w8a8.I8I8I32}


def listed():
    return [
        # The smallest complete call: one linear on ordinary host arrays, blocking, a handful of tokens (a host program
        # that offloads single operators, as callers of the original interface do).
        {"name": "linear_host_16", "kind": "linear", "M": 16, "K": 2048, "N": 2048, "dtype": "f16", "where": "host"},
        # Generating one token: the seven projections of a 7B decoder layer on the engine's stream, q|k|v and gate|up as
        # one launch each.
        {"name": "decode_layer_1", "kind": "layer", "M": 1, "hidden": 4096, "inter": 11008, "grouped": True},
        # The same layer for a batch of eight sequences, one call per projection.
        {"name": "decode_layer_8", "kind": "layer", "M": 8, "hidden": 4096, "inter": 11008, "grouped": False},
        # The fused FFN of an 8B layer for one token.
        {"name": "ffn_decode_1", "kind": "ffn", "M": 1, "K": 4096, "F": 14336, "N": 4096, "where": "device"},
        # The FFN of a 70B layer's quarter shard for a serving batch whose size is no multiple of anything.
        {"name": "ffn_batch_50", "kind": "ffn", "M": 50, "K": 8192, "F": 7168, "N": 8192, "where": "device"},
        # A down projection for a short prompt (the one size the original publishes a time for).
        {"name": "linear_prompt_128", "kind": "linear", "M": 128, "K": 11008, "N": 4096, "dtype": "f16", "where": "device"},
        # Prefill of 2048 tokens through one projection of an 8B layer.
        {"name": "linear_prefill_2048", "kind": "linear", "M": 2048, "K": 4096, "N": 14336, "dtype": "f16", "where": "device"},
        # Prefill of 4096 tokens through the whole FFN: the largest case.
        {"name": "ffn_prefill_4096", "kind": "ffn", "M": 4096, "K": 4096, "F": 14336, "N": 4096, "where": "device"},
        # The typed int8-weight operator on a prompt of ragged length, scales taken per token.
        {"name": "w8_prompt_777", "kind": "w8", "M": 777, "K": 4096, "N": 11008, "op": "f16_dynamic"},
        # Routed experts for a batch of 64 tokens (host arrays in and out, as this operator is defined).
        {"name": "experts_64", "kind": "moe", "M": 64, "hidden": 1536, "inter": 512, "experts": 128, "shared": 1, "top_k": 8,
         "form": "w8", "input": "f32"},
        # Routed int4 experts for one token.
        {"name": "experts_int4_1", "kind": "moe", "M": 1, "hidden": 1536, "inter": 512, "experts": 128, "shared": 1, "top_k": 8,
         "form": "quant", "input": "f32"},
        # Residual add + RMSNorm of a prefill's tokens on device tensors.
        {"name": "add_rmsnorm_4096", "kind": "rmsnorm", "M": 4096, "D": 4096, "layout": "rows", "where": "device"},
    ]


def _spread(rng, low, high):
    """Integers of [low, high], even over their logarithm."""
    return int(min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _size(rng, low, high):
    """A layer width: most are multiples of 128 or 64, some of 16, a few of nothing."""
    step = rng.choice((128, 128, 64, 64, 16, 1))
    return max(step, _spread(rng, low, high) // step * step)


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "layer", "layer", "ffn", "ffn", "ffn", "w8", "w8", "moe", "moe", "rmsnorm"))
    if kind == "linear":
        where = rng.choice(("device", "device", "device", "host", "pinned"))
        M = _spread(rng, 1, 3000 if where == "device" else 128)
        return {"kind": kind, "M": M, "K": _size(rng, 1024, 11008), "N": _size(rng, 1024, 14336),
                "dtype": rng.choice(("f16", "f16", "f32")), "where": where}
    if kind == "layer":
        M = _spread(rng, 1, 32)
        return {"kind": kind, "M": M, "hidden": _spread(rng, 1536, 5120) // 128 * 128, "inter": _spread(rng, 4096, 13824) // 64 * 64,
                "grouped": M <= 4 and rng.random() < 0.5}
    if kind == "ffn":
        where = rng.choice(("device", "device", "device", "host"))
        M = _spread(rng, 1, 3000 if where == "device" else 128)
        return {"kind": kind, "M": M, "K": _size(rng, 1024, 8192), "F": _spread(rng, 2048, 14336) // 64 * 64,
                "N": _size(rng, 1024, 4096), "where": where}
    if kind == "w8":
        return {"kind": kind, "M": _spread(rng, 1, 2048), "K": _size(rng, 1024, 8192), "N": _size(rng, 1024, 11008),
                "op": rng.choice(("f16_dynamic", "f16_dynamic", "f32_dynamic", "f16_static", "i8"))}
    if kind == "moe":
        form = rng.choice(_MOE_FORMS)
        return {"kind": kind, "M": _spread(rng, 1, 256), "hidden": _spread(rng, 1024, 2400) // 64 * 64,
                "inter": rng.choice((256, 320, 384, 512)), "experts": rng.choice((8, 16, 32, 64, 96)),
                "shared": 1 if form == "w4" else rng.choice((0, 1)), "top_k": rng.choice((2, 4, 6, 8)), "form": form,
                "input": rng.choice(("f32", "codes"))}
    where = rng.choice(("device", "device", "device", "host"))
    return {"kind": kind, "M": _spread(rng, 1, 8192 if where == "device" else 256), "D": _spread(rng, 1024, 8192) // 8 * 8,
            "layout": "block8" if where == "host" else rng.choice(("rows", "rows", "block8")), "where": where}


# ---- what a program has in hand before the call --------------------------------------------------------------------

_shared = {}


def _domain():
    """One context and domain for the process, as a program opens them."""
    if not _shared:
        _shared["context"] = rk.Context("cuda:%d" % torch.cuda.current_device())
        _shared["domain"] = _shared["context"].domain(0)
    return _shared["domain"]


class _State:
    """Inputs, outputs and handles of one case; the handles are given back with it."""

    def __init__(self, case, seed):
        self.case = case
        self.dom = _domain()
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.stream = torch.cuda.current_stream().cuda_stream
        self.handles = []
        self.out = None

    def keep(self, handle):
        self.handles.append(handle)
        return handle

    def __del__(self):
        for h in reversed(self.handles):
            h.free()
        self.handles = []

    # tensors
    def codes(self, K, N, most):
        """Codes [K, N] in [-most, most] and scales [N] of normal weights quantised per output channel, on the host."""
        w = torch.randn((K, N), generator=self.gen, device="cuda").mul_(0.02)
        scale = w.abs().amax(0).clamp_(min=1e-6).div_(most)
        codes = w.div_(scale).round_().clamp_(-most, most).to(torch.int8)
        return codes.cpu().numpy(), scale.cpu().numpy()

    def activations(self, M, K):
        x = torch.randn((M, K), generator=self.gen, device="cuda")
        x[:, torch.randperm(K, generator=self.gen, device="cuda")[: max(1, round(0.005 * K))]] *= 20
        return x.half()

    def placed(self, tensor, where):
        """The tensor as the caller holds it: on the GPU, in ordinary host memory or in page-locked host memory."""
        if where == "device":
            return tensor
        host = tensor.cpu()
        return (host.pin_memory() if where == "pinned" else host).numpy()

    def empty(self, shape, dtype, where):
        return self.placed(torch.zeros(shape, dtype=dtype, device="cuda"), where)

    # handles
    def weights(self, K, N):
        return self.keep(rk.Weights(self.dom, *self.codes(K, N, 7)))

    def workspace(self, M, N, K):
        return self.keep(rk.Workspace(self.dom, rk.default_config(M, N, K)))


def _prepare_linear(s, M, K, N, dtype, where):
    x = s.activations(M, K)
    kind = torch.float16 if dtype == "f16" else torch.float32
    s.w, s.ws = s.weights(K, N), s.workspace(M, N, K)
    s.a, s.out = s.placed(x.to(kind), where), s.empty((M, N), kind, where)


def _prepare_layer(s, M, hidden, inter):
    shapes = [(hidden, hidden)] * 4 + [(hidden, inter)] * 2 + [(inter, hidden)]      # q, k, v, o, gate, up, down
    inputs = [s.activations(M, hidden), s.activations(M, hidden), s.activations(M, hidden), s.activations(M, inter)]
    s.w = [s.weights(K, N) for K, N in shapes]
    s.ws = [s.workspace(M, N, K) for K, N in shapes]
    s.a = [inputs[i] for i in (0, 0, 0, 1, 2, 2, 3)]
    s.out = [torch.zeros((M, N), dtype=torch.float16, device="cuda") for _, N in shapes]


def _prepare_ffn(s, M, K, F, N, where):
    s.w = [s.weights(K, 2 * F), s.weights(F, N)]
    s.ws = [s.workspace(M, 2 * F, K), s.workspace(M, N, F)]
    s.a = s.placed(s.activations(M, K).float(), where)
    s.out = [s.empty((M, F), torch.float32, where), s.empty((M, N), torch.float32, where)]


def _prepare_w8(s, M, K, N, op):
    B, scale = s.codes(K, N, 127)
    family = {"f16_dynamic": "f16i8f16", "f16_static": "f16i8f16", "f32_dynamic": "f32i8f32", "i8": "i8i8i32"}[op]
    s.w = s.keep(w8a8.MatmulWeights(s.dom, family, B, None if op == "i8" else scale))
    s.ws = s.keep(w8a8.MatmulWorkspace(s.dom, w8a8.default_strategy(_W8_KINDS[op], M, N, K)))
    x = s.activations(M, K).float()
    row = x.abs().amax(1).div_(127)
    s.scale = row.cpu().numpy()
    if op == "i8":
        s.a, kind = (x / row[:, None]).round_().clamp_(-127, 127).to(torch.int8), torch.int32
    else:
        kind = torch.float32 if op == "f32_dynamic" else torch.float16
        s.a = x.to(kind)
    s.out = torch.zeros((M, N), dtype=kind, device="cuda")


def _prepare_moe(s, M, hidden, inter, experts, shared, top_k, form, input):
    E = experts + shared
    parts = {"gate_up": [], "gate_up_scales": [], "down": [], "down_scales": []}
    for e in range(E):
        most = 127 if form == "w8" or (form == "w4" and e >= experts) else 7
        for name, K, N in (("gate_up", hidden, 2 * inter), ("down", inter, hidden)):
            codes, scale = s.codes(K, N, most)
            parts[name].append(codes)
            parts[name + "_scales"].append(scale)
    s.w = s.keep(moe.MoeWeights(s.dom, shared_expert=shared, form=form, **{k: np.stack(v) for k, v in parts.items()}))
    s.ws = s.keep(moe.MoeWorkspace(s.dom, moe.default_config(hidden, inter, experts, shared, top_k, M), form))
    x = s.activations(M, hidden).float()
    s.scale = np.ascontiguousarray((x.abs().amax(1) / 127).cpu().numpy())
    s.a = x.cpu().numpy()
    if input == "codes":
        s.a = np.clip(np.rint(s.a / s.scale[:, None]), -127, 127).astype(np.int8)
    best = torch.randn((M, experts), generator=s.gen, device="cuda").softmax(1).topk(top_k, dim=1)
    s.ids = best.indices.to(torch.int32).cpu().numpy()
    s.routes = (best.values / best.values.sum(1, keepdim=True)).cpu().numpy()
    s.out = np.zeros((M, hidden), np.float32)


def _prepare_rmsnorm(s, M, D, where):
    gamma = (1 + 0.2 * torch.randn(D, generator=s.gen, device="cuda")).half().cpu().numpy().view(np.uint16)
    s.plan = s.keep(rmsnorm.AddRmsNormPlan(s.dom, rmsnorm.default_config(M, D), gamma))
    x = torch.randn((M, D), generator=s.gen, device="cuda").mul_(0.8).half()
    residual = torch.randn((M, D), generator=s.gen, device="cuda").mul_(1.5).half()
    if where == "device":
        s.a = [x, residual]
        s.out = [torch.zeros_like(x), torch.zeros_like(x)]
    else:
        s.buffers = [s.keep(rmsnorm.Buffer(s.dom, 2 * M * D)) for _ in range(4)]
        for buffer, t in zip(s.buffers, (x, residual)):
            buffer.array()[:] = t.reshape(-1).cpu().numpy().view(np.uint16)
        s.out = [buffer.array() for buffer in s.buffers[2:]]


def prepare(case, seed):
    s = _State(case, seed)
    c = {k: v for k, v in case.items() if k not in ("name", "kind", "grouped", "layout")}
    {"linear": _prepare_linear, "layer": _prepare_layer, "ffn": _prepare_ffn, "w8": _prepare_w8, "moe": _prepare_moe,
     "rmsnorm": _prepare_rmsnorm}[case["kind"]](s, **c)
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------

def _accept(rc):
    if rc != capi.RK_NPU_OK:
        raise rk.W4A8Error(rc, "call")


def _run_linear(s, case):
    if case["where"] == "device":
        _accept((s.ws.enqueue_f16 if case["dtype"] == "f16" else s.ws.enqueue_f32)(s.w, s.a, s.out, s.stream))
    else:
        _accept((s.ws.run_f16 if case["dtype"] == "f16" else s.ws.run_f32)(s.w, s.a, s.out))


def _run_layer(s, case):
    if case["grouped"]:
        for i, j in ((0, 3), (3, 4), (4, 6), (6, 7)):
            _accept(rk.enqueue_batch_f16(s.ws[i:j], s.w[i:j], s.a[i:j], s.out[i:j], s.stream))
    else:
        for ws, w, a, out in zip(s.ws, s.w, s.a, s.out):
            _accept(ws.enqueue_f16(w, a, out, s.stream))


def _run_ffn(s, case):
    if case["where"] == "device":
        _accept(rk.enqueue_ffn_f32(s.ws[0], s.w[0], s.ws[1], s.w[1], s.a, s.out[0], s.out[1], s.stream))
    else:
        _accept(rk.run_ffn_f32(s.ws[0], s.w[0], s.ws[1], s.w[1], s.a, s.out[0], s.out[1]))


def _run_w8(s, case):
    if case["op"] == "i8":
        _accept(s.ws.run_i8(s.w, s.a, s.out))
    elif case["op"] == "f16_static":
        _accept(s.ws.run_static(s.w, s.a, s.scale, s.out))
    else:
        _accept(s.ws.run_dynamic(s.w, s.a, s.out))


def _run_moe(s, case):
    if case["input"] == "codes":
        _accept(s.ws.run_quantized(s.w, s.a, s.scale, s.ids, s.routes, s.out))
    else:
        _accept(s.ws.run_f32(s.w, s.a, s.ids, s.routes, s.out))


def _run_rmsnorm(s, case):
    if case["where"] == "device":
        _accept(s.plan.enqueue(case["M"], case["layout"] == "rows", s.a[0].data_ptr(), s.a[1].data_ptr(), s.out[0].data_ptr(),
                               s.out[1].data_ptr(), s.stream))
    else:
        _accept(s.plan.run(*s.buffers))


_RUN = {"linear": _run_linear, "layer": _run_layer, "ffn": _run_ffn, "w8": _run_w8, "moe": _run_moe, "rmsnorm": _run_rmsnorm}


def run(state):
    _RUN[state.case["kind"]](state, state.case)
    return state.out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def _linear_work(M, K, N, weight_bits, in_bytes, out_bytes):
    return K * N * weight_bits // 8 + 4 * N + in_bytes * M * K + out_bytes * M * N, 2 * M * K * N


def work(case):
    M = case["M"]
    if case["kind"] == "linear":
        size = 2 if case["dtype"] == "f16" else 4
        parts = [_linear_work(M, case["K"], case["N"], 4, size, size)]
    elif case["kind"] == "layer":
        h, i = case["hidden"], case["inter"]
        parts = [_linear_work(M, K, N, 4, 2, 2) for K, N in [(h, h)] * 4 + [(h, i)] * 2 + [(i, h)]]
    elif case["kind"] == "ffn":
        parts = [_linear_work(M, case["K"], 2 * case["F"], 4, 4, 2), _linear_work(M, case["F"], case["N"], 4, 0, 4)]
    elif case["kind"] == "w8":
        in_bytes, out_bytes = {"f16_dynamic": (2, 2), "f16_static": (2, 2), "f32_dynamic": (4, 4), "i8": (1, 4)}[case["op"]]
        parts = [_linear_work(M, case["K"], case["N"], 8, in_bytes, out_bytes)]
    elif case["kind"] == "moe":
        # the experts that a batch of uniformly routed tokens meets; the shared one always
        met = case["experts"] * (1 - (1 - case["top_k"] / case["experts"]) ** M)
        codes = 3 * case["hidden"] * case["inter"]
        bits = 8 if case["form"] == "w8" else 4
        shared_bits = 4 if case["form"] == "quant" else 8
        parts = [(int(codes * (met * bits + case["shared"] * shared_bits) / 8) + M * case["hidden"] * (8 if case["input"] == "f32" else 5),
                  2 * M * (case["top_k"] + case["shared"]) * codes)]
    else:
        parts = [(8 * M * case["D"], 5 * M * case["D"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """Integer sums are exact and the expression around them is fixed by the interface, so every result but one is.  The
    RMSNorm's sum of squares may be added in another order: a last bit of a binary16 result then and now."""
    return {"rel": 1e-4, "max": 2e-3} if case["kind"] == "rmsnorm" else "exact"
