"""The work that a user of this package has it do, as a list of cases with their inputs, cost and tolerance.

Three kinds of work, each through the public entry points:

* ``linear``    one ``QuantLinear.forward``: the call that every linear of a loaded checkpoint makes, from one row of
                activations (a decode step) to a long prompt (prefill);
* ``pack``      one ``QuantLinear.pack`` on the GPU: what quantising a model does once per layer;
* ``generate``  a whole decoder: a prompt through ``GPTQDecoder.prefill`` and then decode steps from the captured graph.
                The tokens are given (as when a text is scored), so that a near-tie between two logits cannot send two
                correct implementations down different texts.
"""
import math

import torch

from autogptq.tvm_b200 import QuantLinear, synth
from autogptq.tvm_b200.decoder import DecoderConfig, GPTQDecoder


def _linear(name, bits, K, N, M, group=128, act=False, bias=False):
    return dict(name=name, kind="linear", bits=bits, K=K, N=N, M=M, group=group, act=act, bias=bias)


def listed():
    return [
        # One token, the smallest linear of a Llama-7B layer (o_proj): latency, launches and host work.
        _linear("decode_b4_4096x4096_m1", 4, 4096, 4096, 1),
        # One token, up_proj of the same layer in a 3-bit act-order checkpoint: the benchmark's headline layer.
        _linear("decode_b3_act_4096x11008_m1", 3, 4096, 11008, 1, act=True),
        # One token, down_proj of a checkpoint quantised for accuracy (groups of 32 rows, act-order).
        _linear("decode_b4_g32_act_11008x4096_m1", 4, 11008, 4096, 1, group=32, act=True),
        # One token, first FFN linear of an OPT-66B layer, with bias: the largest single weight matrix, 127 MB.
        _linear("decode_b3_act_9216x36864_m1", 3, 9216, 36864, 1, act=True, bias=True),
        # A decode step of eight sequences through a fused q|k|v projection.
        _linear("decode_b4_4096x12288_m8", 4, 4096, 12288, 8),
        # A decode step of three sequences in an 8-bit checkpoint.
        _linear("decode_b8_4096x11008_m3", 8, 4096, 11008, 3),
        # A decode step of sixteen sequences, out_proj of an OPT-66B layer (3-bit, act-order, bias).
        _linear("batch_b3_act_9216x9216_m16", 3, 9216, 9216, 16, act=True, bias=True),
        # A short prompt of odd length through down_proj, groups of 64 rows.
        _linear("prefill_b4_g64_11008x4096_m77", 4, 11008, 4096, 77, group=64),
        # A long prompt through a fused q|k|v projection.
        _linear("prefill_b4_4096x12288_m2048", 4, 4096, 12288, 2048),
        # A medium prompt in an 8-bit checkpoint.
        _linear("prefill_b8_4096x4096_m512", 8, 4096, 4096, 512),
        # Quantising a model: up_proj of a Llama-7B layer is packed, rows assigned to groups in act-order.
        dict(name="pack_b4_act_4096x11008", kind="pack", bits=4, K=4096, N=11008, group=128, act=True),
        # The Llama-7B architecture, 4-bit: a 512-token prompt, then 64 tokens one by one.
        dict(name="generate_llama7b_b4_p512_d64", kind="generate", arch="llama", layers=32, hidden=4096, heads=32,
             inter=11008, vocab=32000, bits=4, act=False, batch=1, prompt=512, steps=64),
    ]


def _between(rng, lo, hi, step):
    """A multiple of ``step`` in [lo, hi], uniform over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def _draw_bits(rng):
    return rng.choice([4, 4, 4, 4, 3, 3, 8, 2])


def _draw_size(rng, hi):
    # most models have widths that are multiples of 128; the packed format asks for 32
    return _between(rng, 1024, hi, 128 if rng.random() < 0.75 else 32)


def draw(rng):
    kind = rng.random()
    if kind < 0.08:
        group = rng.choice([32, 64, 128, 128, -1])
        return dict(kind="pack", bits=_draw_bits(rng), K=_draw_size(rng, 11008), N=_draw_size(rng, 11008), group=group,
                    act=group != -1 and rng.random() < 0.5)
    if kind < 0.20:
        llama = rng.random() < 0.5
        heads = rng.choice([8, 16, 32])
        hidden = heads * (128 if llama else rng.choice([64, 128]))
        return dict(kind="generate", arch="llama" if llama else "opt", layers=rng.randint(2, 16), hidden=hidden, heads=heads,
                    inter=_between(rng, 2 * hidden, 4 * hidden, 128), vocab=32 * rng.randint(250, 1571),
                    bits=rng.choice([3, 4, 4]), act=rng.random() < 0.3, batch=rng.choice([1, 1, 2, 4, 8, 16]),
                    prompt=_between(rng, 8, 256, 1), steps=rng.randint(8, 48))
    # single linears: half of them decode batches of up to 8 rows, half prefill
    M = rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]) if rng.random() < 0.5 else _between(rng, 9, 2048, 1)
    group = rng.choice([32, 64, 128, 128, 128, -1])
    return dict(kind="linear", bits=_draw_bits(rng), K=_draw_size(rng, 11008), N=_draw_size(rng, 12288), M=M, group=group,
                act=group != -1 and rng.random() < 0.4, bias=rng.random() < 0.3)


DEVICE = "cuda"


def _prepare_linear(c, seed):
    """A loaded layer (weights on the device, run-time layout built, as after ``from_quantized``) and its input."""
    layer = synth.make_layer(c["bits"], c["K"], c["N"], c["group"], c["act"], bias=c["bias"], seed=seed, device=DEVICE)
    mod = QuantLinear(c["bits"], c["group"], c["K"], c["N"], c["bias"])
    mod.qweight, mod.qzeros, mod.scales, mod.g_idx = layer.qweight, layer.qzeros, layer.scales, layer.g_idx
    if c["bias"]:
        mod.bias = layer.bias
    mod = mod.to(DEVICE)
    mod.post_init()
    return dict(kind="linear", mod=mod, x=synth.make_x(c["M"], c["K"], seed=seed, device=DEVICE).reshape(1, c["M"], c["K"]))


def _prepare_pack(c, seed):
    """What the quantiser hands over: the already rounded fp16 weight, and scales and zero-points per group."""
    bits, K, N = c["bits"], c["K"], c["N"]
    gs = c["group"] if c["group"] != -1 else K
    G = -(-K // gs)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    rows = torch.randperm(K, generator=gen, device=DEVICE) if c["act"] else torch.arange(K, device=DEVICE)
    g_idx = (rows // gs).to(torch.int32)
    maxq = 2 ** bits - 1
    scales = torch.rand((N, G), generator=gen, device=DEVICE) * 0.02 + 1e-3
    zeros = torch.randint(1, maxq + 1, (N, G), generator=gen, device=DEVICE).float()
    q = torch.randint(0, maxq + 1, (N, K), generator=gen, device=DEVICE).float()
    g = g_idx.long()
    linear = torch.nn.Linear(K, N, bias=False, device="meta", dtype=torch.float16)
    linear.weight = torch.nn.Parameter((scales[:, g] * (q - zeros[:, g])).half(), requires_grad=False)
    return dict(kind="pack", mod=QuantLinear(bits, c["group"], K, N, False), linear=linear, scales=scales, zeros=zeros,
                g_idx=g_idx)


def _prepare_generate(c, seed):
    """A loaded model with its decode step captured, a prompt and the tokens that follow it."""
    cfg = DecoderConfig(arch=c["arch"], layers=c["layers"], hidden=c["hidden"], heads=c["heads"], inter=c["inter"],
                        vocab=c["vocab"], bits=c["bits"], group_size=128, desc_act=c["act"],
                        max_seq=c["prompt"] + c["steps"] + 8)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    text = torch.randint(0, c["vocab"], (c["batch"], c["prompt"] + c["steps"]), generator=gen, device=DEVICE)
    model = GPTQDecoder(cfg, batch=c["batch"], device=DEVICE)
    prompt = text[:, :c["prompt"]].contiguous()
    model.prefill(prompt)
    model.capture()
    # the captured step writes its logits into this tensor every time it is replayed
    return dict(kind="generate", model=model, prompt=prompt, tokens=text[:, c["prompt"]:].t().contiguous(),
                step_logits=model.last_logits)


def prepare(case, seed):
    return {"linear": _prepare_linear, "pack": _prepare_pack, "generate": _prepare_generate}[case["kind"]](case, seed)


def _run_generate(s):
    model, tokens, step_logits = s["model"], s["tokens"], s["step_logits"]
    model.prefill(s["prompt"])
    first = model.last_logits
    out = torch.empty((tokens.shape[0],) + tuple(step_logits.shape), dtype=step_logits.dtype, device=step_logits.device)
    for i in range(tokens.shape[0]):
        model.tokens.copy_(tokens[i])
        model.decode(1)
        out[i].copy_(step_logits)
    return first, out


def run(state):
    if state["kind"] == "linear":
        with torch.inference_mode():
            return state["mod"](state["x"])
    if state["kind"] == "pack":
        mod = state["mod"]
        mod.pack(state["linear"], state["scales"], state["zeros"], state["g_idx"])
        return mod.qweight, mod.qzeros, mod.scales, mod.g_idx
    return _run_generate(state)


def _packed_bytes(bits, K, N, group):
    G = -(-K // (group if group != -1 else K))
    return K * N * bits / 8 + G * N * bits / 8 + G * N * 2


def _generate_work(c):
    H, I, B, L = c["hidden"], c["inter"], c["batch"], c["layers"]
    up = (2 if c["arch"] == "llama" else 1) * I
    shapes = [(H, 3 * H), (H, H), (H, up), (I, H)]
    weights = L * sum(_packed_bytes(c["bits"], K, N, 128) for K, N in shapes)
    params = L * sum(K * N for K, N in shapes)
    head = c["vocab"] * H
    P, S = c["prompt"], c["steps"]
    cache_row = L * 2 * H * 2 * B           # keys and values of one position of every sequence
    # every step reads the weights, the vocabulary projection and the cache so far, and writes one row of it
    nbytes = (S + 1) * (weights + head * 2) + cache_row * (P + sum(P + i + 2 for i in range(S)))
    flops = 2.0 * B * (params * (P + S) + head * (S + 1)) + 4.0 * B * L * H * (P * (P + 1) / 2 + sum(P + i + 1 for i in range(S)))
    return {"bytes": nbytes, "flops": flops}


def work(case):
    c = case
    if c["kind"] == "generate":
        return _generate_work(c)
    K, N = c["K"], c["N"]
    packed = _packed_bytes(c["bits"], K, N, c["group"])
    index = 4 * K if c["act"] else 0
    if c["kind"] == "pack":
        G = -(-K // (c["group"] if c["group"] != -1 else K))
        return {"bytes": 2 * K * N + 8 * N * G + packed + index, "flops": 3.0 * K * N}
    M = c["M"]
    return {"bytes": packed + index + 2 * M * (K + N) + (2 * N if c["bias"] else 0), "flops": 2.0 * M * K * N}


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"                       # the words of a checkpoint
    if case["kind"] == "generate":
        return {"rel": 1e-2, "max": 0.1}     # fp16 activations through every layer of the model
    return {"rel": 1e-3, "max": 1e-2}        # fp32 sums of fp16 products, fp16 weights and results
