"""The decoder layers of a step in one launch (``b200gptq_step_plan_*``) against the kernels launched one by one."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import decoder, ops, synth
    DEV = torch.device("cuda:0")


def _model(arch, bits, act, layers, hidden, heads, inter, prompt, group=128, batch=1, max_seq=None):
    cfg = decoder.DecoderConfig(arch=arch, layers=layers, hidden=hidden, heads=heads, inter=inter, vocab=1000, bits=bits,
                                group_size=group, desc_act=act, max_seq=max_seq or prompt + 8)
    text = torch.randint(0, cfg.vocab, (batch, prompt + 4), generator=torch.Generator().manual_seed(prompt)).to(DEV)
    return decoder.GPTQDecoder(cfg, batch=batch, device=DEV), text


def _steps(m, text, prompt, one_launch, steps=4):
    m.one_launch = one_launch
    m.prefill(text[:, :prompt].contiguous())
    logits = []
    for i in range(steps):
        m.tokens.copy_(text[:, prompt + i])
        m._decode_step()
        logits.append(m.last_logits.double().clone())
    ops.check_status(DEV)
    return torch.stack(logits), [(L.k_cache.clone(), L.v_cache.clone()) for L in m.layers]


def _close(got, want, layers):
    """Both round to fp16 at the same places, some eight per layer, and sum in fp32 in another order: a rounding may go the other way, by
    2^-11 of the value, each on its own."""
    assert float((got - want).norm() / want.norm()) <= (8 * layers) ** 0.5 * 2.0 ** -11


@pytest.mark.parametrize("shape", [
    ("llama", 4, False, 2, 256, 2, 512, 12),             # units for two of the eight warps
    ("llama", 4, False, 3, 1024, 8, 2816, 40),           # half a slot; 22 units, the second slot cut
    ("llama", 4, True, 2, 4096, 32, 11008, 2),           # gather of x; pairs of strips, three per CTA
    ("llama", 4, False, 2, 6144, 48, 6272, 9),           # as many slots as are read at once; an odd number of units
    ("llama", 3, True, 2, 2048, 16, 5504, 400),          # three CTAs per head; three slots
    ("llama", 3, False, 2, 512, 8, 1024, 193),           # zero-points that start inside a 16-byte piece; two CTAs per head, 64 dims
    ("llama", 2, True, 2, 1024, 8, 1152, 30),
    ("opt", 3, True, 2, 1024, 16, 4096, 1),
    ("opt", 4, False, 2, 1024, 8, 2048, 700, 256),       # two units per group; four CTAs per head
    ("opt", 4, True, 2, 768, 12, 3072, 65, 384),         # three units per group
    ("opt", 2, False, 1, 512, 4, 640, 5),
    ("llama", 4, False, 6, 2048, 16, 1024, 12),          # half the warps have no units of the second FFN linear and are ahead of the others
    ("opt", 3, True, 6, 1024, 8, 256, 40),
    ("llama", 4, False, 1, 256, 2, 512, 2100),           # sixteen CTAs per head; a second block for some warps
    ("llama", 4, False, 1, 1024, 8, 1152, 641),          # six, two batches of parts
    ("opt", 3, False, 1, 512, 8, 1024, 1030),            # five of 64 dims, the last with a few positions; several blocks
    ("llama", 2, False, 1, 4096, 32, 1024, 1500),        # four that go through several blocks
])
def test_one_launch_computes_what_the_kernels_compute(shape):
    prompt, layers = shape[7], shape[3]
    m, text = _model(*shape)
    want, caches = _steps(m, text, prompt, False)
    got, own = _steps(m, text, prompt, True)
    assert m._plan is not None and m._plan[1] is not None, "a shape that the kernel takes"
    _close(got, want, layers)
    for (k0, v0), (k1, v1) in zip(caches, own):
        _close(k1.double(), k0.double(), layers)
        _close(v1.double(), v0.double(), layers)
        assert torch.equal(k0[:, :, prompt + 4:], k1[:, :, prompt + 4:])
    again, _ = _steps(m, text, prompt, True)
    assert torch.equal(again, got), "the same bits every time"
    # captured, and several steps in a row on the caller's stream
    m.prefill(text[:, :prompt].contiguous())
    m.capture()
    for i in range(4):
        m.tokens.copy_(text[:, prompt + i])
        m.graph.replay()
        assert torch.equal(m.last_logits.double(), got[i])


def test_what_the_kernel_does_not_take_goes_kernel_by_kernel():
    for args, kw in ((("llama", 4, False, 1, 256, 2, 512, 12), dict(batch=2)), (("llama", 8, False, 1, 256, 2, 512, 12), {}),
                     (("opt", 3, False, 1, 320, 5, 512, 12), dict(group=64))):
        m, text = _model(*args, **kw)
        m.prefill(text[:, :12].contiguous())
        m._decode_step()
        assert m._step_plan() is None
    # a hook sees every call of its layer; without it the plan is back
    m, text = _model("llama", 4, False, 2, 256, 2, 512, 12)
    want, _ = _steps(m, text, 12, True)
    calls = []
    hook = m.layers[1].o.register_forward_hook(lambda *a: calls.append(1))
    _steps(m, text, 12, True)
    assert len(calls) == 5                               # the prompt and four steps
    hook.remove()
    got, _ = _steps(m, text, 12, True)
    assert torch.equal(got, want)


def test_replaced_tensors_are_followed():
    m, text = _model("llama", 4, True, 2, 512, 4, 1024, 20)
    first, _ = _steps(m, text, 20, True)
    kept = m._plan[1]
    m.layers[0].down.scales = m.layers[0].down.scales * 2
    m.layers[1].norm1_w = m.layers[1].norm1_w * 0.5
    want, _ = _steps(m, text, 20, False)
    got, _ = _steps(m, text, 20, True)
    assert m._plan[1] is not kept and not torch.equal(got, first)
    _close(got, want, 2)
    m.layers[1].up.qzeros.zero_()                        # in place: read as it is
    want, _ = _steps(m, text, 20, False)
    got, _ = _steps(m, text, 20, True)
    _close(got, want, 2)


@pytest.mark.parametrize("name,change,error", [
    ("scales", lambda t: t.float(), TypeError), ("qzeros", lambda t: t.cpu(), RuntimeError), ("scales", lambda t: t.cpu(), RuntimeError)])
def test_tensors_that_the_layers_refuse_are_refused(name, change, error):
    m, text = _model("llama", 4, False, 2, 256, 2, 512, 12)
    _steps(m, text, 12, True)
    o = m.layers[1].o
    setattr(o, name, change(getattr(o, name)))
    assert m._step_plan() is None
    for m.one_launch in (False, True):
        with pytest.raises(error):
            m._decode_step()


def test_a_forward_of_one_layer_or_a_hook_of_all_is_called():
    m, text = _model("llama", 4, False, 2, 256, 2, 512, 12)
    want, _ = _steps(m, text, 12, True)
    o, calls = m.layers[1].o, []
    o.forward = lambda x: (calls.append(1), type(o).forward(o, x))[1]
    _close(_steps(m, text, 12, True)[0], want, 2)
    assert len(calls) == 5                               # the prompt and four steps
    del o.forward
    hook = torch.nn.modules.module.register_module_forward_hook(lambda mod, *a: calls.append(1) if mod is o else None)
    try:
        _steps(m, text, 12, True)
    finally:
        hook.remove()
    assert len(calls) == 10 and m._step_plan() is not None


def test_a_copy_makes_a_plan_of_its_own():
    m, text = _model("llama", 4, False, 2, 512, 4, 1024, 20)
    want, _ = _steps(m, text, 20, True)
    c = copy.deepcopy(m)
    assert c._plan[1] is None
    assert torch.equal(_steps(c, text, 20, True)[0], want) and c._plan[1] is not m._plan[1]


def test_a_position_outside_the_caches_writes_none():
    m, text = _model("llama", 4, False, 2, 256, 2, 512, 12)
    _steps(m, text, 12, True)
    before = [(L.k_cache.clone(), L.v_cache.clone()) for L in m.layers]
    for pos in (m.cfg.max_seq, -1):
        m.pos.fill_(pos)
        x = torch.ones(1, 256, dtype=torch.float16, device=DEV)
        assert m._step_plan().run(x)
        for L, (k, v) in zip(m.layers, before):
            assert torch.equal(L.k_cache, k) and torch.equal(L.v_cache, v)
        assert bool(torch.isfinite(x).all())
    ops.check_status(DEV)


def test_a_smaller_model_leaves_the_larger_one_running():
    """The limit of dynamic shared memory belongs to the kernel, not to a plan: a plan that needs less, made later, must not lower it."""
    large, text = _model("llama", 4, False, 1, 1024, 8, 2816, 12)
    want, _ = _steps(large, text, 12, True)
    small, other = _model("llama", 4, False, 1, 256, 2, 512, 12)
    _steps(small, other, 12, True)
    assert small._plan[1] is not None and large._plan[1] is not None
    assert torch.equal(_steps(large, text, 12, True)[0], want)


@pytest.mark.parametrize("arch,bits", [("llama", 4), ("opt", 3)])
def test_a_second_ffn_linear_with_rows_of_its_own_order_goes_kernel_by_kernel(arch, bits):
    m, text = _model(arch, bits, False, 2, 512, 4, 1024, 12)
    L = m.layers[1]
    L.down = decoder._to_module(synth.make_layer(bits, 1024, 512, 128, True, bias=arch == "opt", seed=5, device=DEV), DEV)
    assert L.down._x_perm is not None
    want, _ = _steps(m, text, 12, False)
    got, _ = _steps(m, text, 12, True)
    assert torch.equal(got, want) and m._step_plan() is None


def test_the_folded_activation_that_was_asked_for_is_used():
    m, text = _model("llama", 4, False, 2, 256, 2, 512, 12)
    want, _ = _steps(m, text, 12, False)
    m.fold_activation = True
    down, calls = m.layers[1].down, []
    down.forward_act = lambda *a: (calls.append(1), type(down).forward_act(down, *a))[1]
    assert torch.equal(_steps(m, text, 12, True)[0], want), "bit-identical to the separate kernel"
    assert len(calls) == 4


@pytest.mark.parametrize("bits,group", [(8, 128), (4, 64)])
def test_tensors_of_a_shape_that_the_kernel_does_not_take_are_not_looked_at(bits, group):
    """(that costs the host of a step without a graph as much as three launches per layer)"""
    m, text = _model("llama", bits, False, 2, 256, 2, 512, 12, group)
    m.prefill(text[:, :12].contiguous())
    calls = []
    for L in m.layers:
        L.qkv._ready = lambda: (calls.append(1), True)[1]
    assert m._step_plan() is None and not calls


def test_maps_of_a_plan_whose_memory_is_used_again():
    """Every replaced tensor makes a plan, in memory that a plan of other tensor maps has left: the copies must not see those."""
    m, text = _model("llama", 4, False, 2, 512, 4, 1024, 20)
    _steps(m, text, 20, True)
    at, pieces = [], []
    for i in range(6):
        L = m.layers[i % 2]
        pieces.append(torch.empty(4096 * (i + 1), dtype=torch.uint8, device=DEV))     # (other addresses for what is replaced)
        L.up.qweight = L.up.qweight.roll(32 * (i + 1), dims=1)
        L.down.scales, L.o.qzeros = L.down.scales.flip(1).contiguous(), L.o.qzeros.roll(4, dims=1)
        want, _ = _steps(m, text, 20, False)
        got, _ = _steps(m, text, 20, True)
        _close(got, want, 2)
        at.append(m._plan[1]._memory.data_ptr())
    assert len(set(at)) < len(at), "no plan's memory was used again"


def test_the_captured_plan_has_memory_of_the_stream_that_replays_it():
    """Not of the warm-up's: freed with the model, that could be handed out on another stream while a replay still writes it."""
    m, text = _model("llama", 4, False, 2, 512, 4, 1024, 20)
    m.prefill(text[:, :20].contiguous())
    m.capture()
    at = m._graph_plan[1]._memory.data_ptr()
    streams = [s["stream"] for s in torch.cuda.memory_snapshot() if s["address"] <= at < s["address"] + s["total_size"]]
    assert streams == [torch.cuda.current_stream().cuda_stream]


def test_a_model_that_is_faster_kernel_by_kernel_goes_that_way_unless_told():
    m, text = _model("llama", 4, False, 1, 4864, 38, 512, 12)
    assert m._step_plan() is None
    m.one_launch = True
    assert m._step_plan() is not None
    m, text = _model("llama", 4, False, 1, 256, 2, 512, 12)
    assert m._step_plan() is not None


def test_two_models_on_two_streams():
    """Each launch holds the whole GPU, and is there as a whole or not at all: steps of two models that nothing orders wait for one another
    and give what they give alone."""
    models = [_model("llama", 4, False, 2, 512, 4, 1024, 20), _model("opt", 3, False, 3, 512, 8, 1024, 20)]
    streams, want, got = [torch.cuda.Stream(DEV) for _ in models], [], []
    for m, text in models:
        want.append(_steps(m, text, 20, True, 1)[0][0])
        m.prefill(text[:, :20].contiguous())
        m.capture()
        m.tokens.copy_(text[:, 20])
    torch.cuda.synchronize()
    for _ in range(20):
        for (m, text), s in zip(models, streams):
            with torch.cuda.stream(s):
                m.tokens.copy_(text[:, 20])
                m.pos.fill_(20)
                m.graph.replay()
                got.append(m.last_logits.double())
    torch.cuda.synchronize()
    ops.check_status(DEV)
    for i, logits in enumerate(got):
        assert torch.equal(logits, want[i % 2])


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("big", [0, 512, 16384])
def test_no_further_from_64_bits_than_the_kernels(bits, big):
    """The second FFN linear of a step alone: the input is zero, the output projection's scales are zero, so that x becomes down(relu(bias of the
    first)).  `big`: the largest value of every unit of 128 rows, which meets weights of zero, so that what x in fixed point takes from the
    small ones' precision is seen: no more than the kernel by itself, which has fp16 products here, loses in fp32 sums (2 and 3 bits: far less)."""
    H, inter = 1024, 4096
    m, text = _model("opt", bits, False, 1, H, 8, inter, 4)
    m.one_launch = True
    L = m.layers[0]
    gen = torch.Generator().manual_seed(bits + big)
    act = torch.rand(inter, generator=gen) + 0.5
    q = torch.randint(0, 2 ** bits, (inter, H), generator=gen)
    zeros = torch.randint(1, 2 ** bits, (inter // 128, H), generator=gen)
    if big:
        at = torch.arange(inter // 128) * 128 + torch.randint(0, 128, (inter // 128,), generator=gen)
        act[at] = float(big)
        q[at] = zeros
    act = act.half()
    L.up.bias = act.to(DEV)
    L.o.scales.zero_(), L.o.bias.zero_(), L.down.bias.zero_()
    L.down.qweight = ops.pack_fields(q.to(torch.int32).to(DEV), bits)
    L.down.qzeros = ops.pack_fields((zeros - 1).to(torch.int32).t().contiguous().to(DEV), bits).t().contiguous()
    L.down.post_init()
    W = (q - zeros.repeat_interleave(128, 0)).double() * L.down.scales.cpu().double().repeat_interleave(128, 0)
    exact = act.double() @ W
    m.pos.fill_(0)
    x = torch.zeros(1, H, dtype=torch.float16, device=DEV)
    assert m._step_plan().run(x)
    one = (x.cpu().double()[0] - exact).norm() / exact.norm()
    kernel = (L.down(act.to(DEV)[None]).cpu().double()[0] - exact).norm() / exact.norm()
    ops.check_status(DEV)
    # (both hold the result's rounding to fp16, 2.0e-4 of it, over 1024 columns: the same within a few per cent where that is all)
    assert float(one) <= 1.1 * float(kernel), (float(one), float(kernel))
