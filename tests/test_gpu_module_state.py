"""A QuantLinear whose tensors are replaced between calls: the prepared launches (plans, the native call object) hold
addresses, and every route -- one row, sixteen, the GEMM -- has to follow the module.  The yardstick is a fresh module with
the same tensors, to the bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import QuantLinear, _lib, ops, synth
    DEV = torch.device("cuda:0")

K, N, GS, BITS = 512, 256, 128, 4
ROWS = (1, 8, 16, 32)


def _module(layer):
    m = QuantLinear(BITS, GS, K, N, True)
    m.qweight, m.qzeros, m.scales, m.g_idx, m.bias = layer.qweight, layer.qzeros, layer.scales, layer.g_idx, layer.bias
    return m


def _fresh(mod):
    m = QuantLinear(BITS, GS, K, N, True)
    for name in ("qweight", "qzeros", "scales", "g_idx", "bias"):
        t = getattr(mod, name)
        setattr(m, name, None if t is None else t.clone())
    return m


@pytest.mark.parametrize("how", ["new tensor", "data"])
@pytest.mark.parametrize("name", ["scales", "qzeros", "bias", "qweight", "g_idx"])
@pytest.mark.parametrize("act", [False, True])
def test_replaced_tensors_are_the_ones_used(name, how, act):
    a = synth.make_layer(BITS, K, N, GS, act, bias=True, seed=1, device=DEV)
    b = synth.make_layer(BITS, K, N, GS, act, bias=True, seed=2, device=DEV)
    mod = _module(a)
    xs = [synth.make_x(M, K, seed=M, device=DEV) for M in ROWS]
    first = [mod(x) for x in xs]                    # the Python route, which prepares
    assert all(torch.equal(y, mod(x)) for x, y in zip(xs, first))
    new = getattr(b, name) if act or name != "g_idx" else torch.flip(a.g_idx, (0,)).contiguous()
    if how == "data":
        getattr(mod, name).data = new
    else:
        setattr(mod, name, new)
    for _ in range(3):                              # prepared anew, then prepared
        want = [_fresh(mod)(x) for x in xs]
        for M, x, w, old in zip(ROWS, xs, want, first):
            y = mod(x)
            assert torch.equal(y, w), f"{M} rows"
            assert not torch.equal(y, old)
    if name == "bias" and how == "new tensor":
        mod.bias = None
        for x in xs:
            assert torch.equal(mod(x), _fresh(mod)(x))


@pytest.mark.parametrize("name", ["scales", "qzeros", "bias"])
def test_replaced_tensors_with_a_folded_activation(name):
    a = synth.make_layer(BITS, K, N, GS, False, bias=True, seed=1, device=DEV)
    b = synth.make_layer(BITS, K, N, GS, False, bias=True, seed=2, device=DEV)
    mod, x = _module(a), synth.make_x(2, K, seed=5, device=DEV)
    mod.forward_act(x, _lib.ACT_RELU)
    setattr(mod, name, getattr(b, name))
    assert torch.equal(mod.forward_act(x, _lib.ACT_RELU), _fresh(mod).forward_act(x, _lib.ACT_RELU))


def _outcome(f):
    try:
        return f()
    except Exception as e:      # noqa: BLE001  (its type is what is compared)
        return type(e)


@pytest.mark.parametrize("M", [1, 32])
def test_wrapped_tensors_take_the_python_route(M):
    """Tensors without memory of their own (vmap, grad, jvp) raise in Python, as they do before the native call object exists."""
    mod, x = _module(synth.make_layer(BITS, K, N, GS, False, bias=True, seed=1, device=DEV)), synth.make_x(M, K, seed=3, device=DEV)
    want = mod(x)
    transforms = [lambda: torch.func.vmap(mod)(torch.stack([x, x])),
                  lambda: torch.func.grad(lambda t: mod(t).float().sum())(x),
                  lambda: torch.func.jvp(mod, (x,), (x,))[0]]
    for f in transforms:
        mod(x)
        assert mod._native is not None
        got = _outcome(f)
        mod._native = None
        plain = _outcome(f)
        assert got is plain if isinstance(plain, type) else torch.equal(got, plain)
    assert torch.equal(mod(x), want)
