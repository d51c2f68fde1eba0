"""Workloads of the tensor-parallel reduction path, for timing and for comparing two builds of it.

A case is one call pattern of a decode or prefill loop: the FP8 row-parallel projection from device or
host buffers, the MXFP4 routed-expert step, the vocabulary head, and the projection of a whole
tensor-parallel group.  Everything runs eagerly through ``weightstream_b200.tp`` on the current stream,
as a host engine calls it.
"""
import numpy as np
import torch

from weightstream_b200 import synth, tp

N_OUT, K_FULL = 7168, 8192              # attention output projection
VOCAB, K_HEAD = 129280, 7168
EXPERTS, K_EXPERT, TOP_K = 384, 2048, 6
N_NATIVE, K_NATIVE = 5120, 2304         # the reference model's own shared-expert / expert down shape
WORK_MAX = 2000 * N_OUT * K_FULL        # rows x outputs x K of the largest listed case
LAYER_BYTES = 58 << 20                  # small shards: one call for each of as many layers as this holds


def _fp8(name, m, n, k, scale="f32", act="bf16", layers=1):
    return {"name": name, "kind": "fp8", "m": m, "n": n, "k": k, "scale": scale, "act": act, "layers": layers}


def listed():
    return [
        # One decoded token: the attention output projection of one layer (58.7 MB of weights).
        _fp8("oproj_row", 1, N_OUT, K_FULL),
        # The same token on one rank of eight: its K slice is 7.3 MB a layer, so launches and latency
        # count.  Eight consecutive layers, because a decode step never meets the same weights twice.
        _fp8("oproj_shard_row", 1, N_OUT, K_FULL // 8, layers=8),
        # The drop-in form for an engine that keeps its activations on the host: slice in, vector out.
        {"name": "oproj_host_row", "kind": "host", "m": 1, "n": N_OUT, "k": K_FULL},
        # A serving batch of a ragged number of sequences, one token each.
        _fp8("oproj_batch", 40, N_OUT, K_FULL),
        # A prompt's prefill, not a multiple of any tile.
        _fp8("oproj_prefill", 2000, N_OUT, K_FULL),
        # The reference's own parameter set: 32x32 power-of-two scales and fp32 activations, a small batch.
        _fp8("native_batch", 19, N_NATIVE, K_NATIVE, scale="ue8m0", act="f32", layers=5),
        # One decoded token through its six routed experts of 384, all on this rank.
        {"name": "moe_row", "kind": "moe", "m": 1, "n": N_OUT, "k": K_EXPERT, "local": EXPERTS, "act": "bf16"},
        # A full serving batch: about 244 of the 384 experts are hit, some by several tokens.
        {"name": "moe_batch", "kind": "moe", "m": 64, "n": N_OUT, "k": K_EXPERT, "local": EXPERTS, "act": "bf16"},
        # The reference's own expert shape on one rank of four, fp32 hidden states, a ragged batch.
        {"name": "moe_native_batch", "kind": "moe", "m": 21, "n": N_NATIVE, "k": K_NATIVE, "local": EXPERTS // 4, "act": "f32"},
        # Greedy decoding: only the token index is wanted (927 MB of weights).
        {"name": "head_argmax_row", "kind": "head", "m": 1, "n": VOCAB, "k": K_HEAD, "logits": False},
        # Sampling in a serving batch: the logits themselves and the argmax.
        {"name": "head_logits_batch", "kind": "head", "m": 12, "n": VOCAB, "k": K_HEAD, "logits": True},
        # All eight ranks of a group in one process: K slices, exchange, rank-ordered sums on every rank.
        {"name": "group_oproj", "kind": "group", "m": 3, "n": N_OUT, "k": K_FULL, "world": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _multiple(rng, lo, hi, step):
    return max(lo, _log_int(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(["fp8", "fp8", "fp8", "host", "moe", "moe", "head", "group"])
    if kind == "fp8":
        scale = rng.choice(["f32", "f32", "ue8m0"])
        m = _log_int(rng, 1, 2000)
        n = _multiple(rng, 1024, 8192, 16)
        k = _multiple(rng, 512, 8192, 128 if scale == "f32" else 32)
        m = max(1, min(m, WORK_MAX // (n * k)))
        layers = max(1, min(8, LAYER_BYTES // (n * k))) if m <= 32 else 1
        c = _fp8("", m, n, k, scale, rng.choice(["bf16", "f32"]), layers)
    elif kind == "host":
        c = {"kind": kind, "m": _log_int(rng, 1, 64), "n": _multiple(rng, 1024, 8192, 16), "k": _multiple(rng, 512, 8192, 128)}
    elif kind == "moe":
        shape = rng.choice([(N_OUT, K_EXPERT), (N_NATIVE, K_NATIVE), None])
        n, k = shape or (_multiple(rng, 2048, 7168, 16), _multiple(rng, 512, 2560, 256))
        c = {"kind": kind, "m": _log_int(rng, 1, 85), "n": n, "k": k, "local": EXPERTS // rng.choice([1, 2, 4, 8]),
             "act": rng.choice(["bf16", "f32"])}
    elif kind == "head":
        c = {"kind": kind, "m": _log_int(rng, 1, 64), "n": _multiple(rng, 16160, VOCAB, 16), "k": _multiple(rng, 2048, K_HEAD, 128),
             "logits": rng.random() < 0.5}
    else:
        world = rng.choice([2, 4, 8])
        c = {"kind": kind, "m": _log_int(rng, 1, 64), "n": _multiple(rng, 2048, N_OUT, 16),
             "k": world * _multiple(rng, 512, K_FULL // world, 128), "world": world}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------ inputs
def _ue8m0_weight(n, k, seed, dev):
    """W ~ N(0, 0.02) as E4M3 with one power-of-two scale byte per 32x32 block."""
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    v = torch.randn((n, k), generator=g, device=dev) * 0.02
    pad = (-n) % 32
    amax = torch.nn.functional.pad(v.abs(), (0, 0, 0, pad)).reshape(-1, 32, k // 32, 32).amax(dim=(1, 3)).clamp_min(1e-4)
    e = torch.ceil(torch.log2(amax / 448.0)).to(torch.int32)
    s = torch.ldexp(torch.ones_like(amax), e).repeat_interleave(32, 0)[:n].repeat_interleave(32, 1)
    q = (v / s).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.view(torch.uint8), (e + 127).to(torch.uint8)


def _weight(n, k, scale, seed, dev):
    if scale == "ue8m0":
        return _ue8m0_weight(n, k, seed, dev)
    return synth.torch_fp8_weight(n, k, seed=seed, device=dev)


def _activations(shape, act, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    x = torch.randn(shape, generator=g, device=dev)
    return x.to(torch.bfloat16) if act == "bf16" else x


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind, m, n, k = case["kind"], case["m"], case["n"], case["k"]
    s = {"kind": kind}
    if kind == "fp8":
        s["ep"] = tp.Endpoint(max_m=m, max_n=n)
        s["block"] = (32, 32) if case["scale"] == "ue8m0" else (128, 128)
        s["layers"] = []
        for i in range(case["layers"]):
            w, sc = _weight(n, k, case["scale"], 1000 * seed + 2 * i, dev)
            s["layers"].append((_activations((m, k), case["act"], 1000 * seed + 2 * i + 1, dev), w, sc))
    elif kind == "host":
        s["ep"] = tp.Endpoint(max_m=m, max_n=n)
        s["w"], s["sc"] = _weight(n, k, "f32", 1000 * seed, dev)
        x = _activations((m, k), "bf16", 1000 * seed + 1, dev)
        s["x"] = x.view(torch.int16).cpu().numpy().view(np.uint16)
    elif kind == "moe":
        s["ep"] = tp.Endpoint(max_m=m, max_n=n)
        s["w2"], s["s2"] = synth.torch_fp4_experts(case["local"], n, k, seed=1000 * seed, device=dev)
        ids, rw = synth.routes(np.random.default_rng(seed), m, EXPERTS, TOP_K)
        s["ids"], s["rw"] = torch.from_numpy(ids).to(dev), torch.from_numpy(rw).to(dev)
        s["h"] = _activations((m * TOP_K, k), case["act"], 1000 * seed + 1, dev)
    elif kind == "head":
        s["ep"] = tp.Endpoint(max_m=m, max_n=16, max_vocab=n)
        s["w"], s["sc"] = _weight(n, k, "f32", 1000 * seed, dev)
        s["x"] = _activations((m, k), "bf16", 1000 * seed + 1, dev)
        s["logits"], s["vocab"] = case["logits"], n
    else:
        world = case["world"]
        s["grp"] = tp.LocalGroup(world, max_m=m, max_n=n)
        w, sc = _weight(n, k, "f32", 1000 * seed, dev)
        x = _activations((m, k), "bf16", 1000 * seed + 1, dev)
        cuts = [tp.Sharding(world, r).slice_of(k) for r in range(world)]
        s["xs"] = [x[:, a:a + ln].contiguous() for a, ln in cuts]
        s["ws"] = [tp.shard_weight(w, (n, k), tp.WShard.Cols(a, ln)) for a, ln in cuts]
        s["scs"], s["k0s"] = [sc] * world, [a for a, _ in cuts]
    return s


def run(state):
    kind = state["kind"]
    if kind == "fp8":
        ep, block = state["ep"], state["block"]
        return [ep.fp8_rowpar_gemm_allreduce(x, w, sc, block=block) for x, w, sc in state["layers"]]
    if kind == "host":
        return state["ep"].fp8_rowpar_gemm_allreduce_host(state["x"], state["w"], state["sc"])
    if kind == "moe":
        return state["ep"].moe_down_combine_allreduce(state["h"], state["ids"], state["rw"], state["w2"], state["s2"], 0)
    if kind == "head":
        logits, arg = state["ep"].lm_head_allgather_argmax(state["x"], state["w"], state["sc"], vocab_row0=0, vocab=state["vocab"],
                                                           want_logits=state["logits"])
        return [arg] if logits is None else [arg, logits]
    return state["grp"].fp8_rowpar_gemm_allreduce(state["xs"], state["ws"], state["scs"], k0s=state["k0s"])


# ------------------------------------------------------------------------------------------ yardsticks
def work(case):
    kind, m, n, k = case["kind"], case["m"], case["n"], case["k"]
    if kind == "moe":
        # distinct local experts that m tokens hit, in expectation: routes are uniform over the experts
        hit = case["local"] * (1.0 - (1.0 - TOP_K / EXPERTS) ** m)
        routes = m * TOP_K * case["local"] / EXPERTS
        es = 2 if case["act"] == "bf16" else 4
        return {"bytes": hit * (n * k / 2 + n * k / 32) + routes * k * es + 4.0 * m * n, "flops": 2.0 * routes * n * k}
    if kind == "fp8":
        calls, es = case["layers"], 2 if case["act"] == "bf16" else 4
        scales = (n / 32) * (k / 32) if case["scale"] == "ue8m0" else 4.0 * -(-n // 128) * (k / 128)
    else:
        calls, es, scales = 1, 2, 4.0 * -(-n // 128) * (k / 128)
    outs = 4.0 * m * n
    if kind == "head":
        outs = 4.0 * m + (outs if case["logits"] else 0.0)
    elif kind == "group":
        outs *= case["world"]
    return {"bytes": calls * (n * k + scales + m * k * es + outs), "flops": calls * 2.0 * m * n * k}


def tolerance(case):
    # exact products of quantised operands, fp32 sums in an order of the implementation's choosing
    return {"rel": 1e-5}
