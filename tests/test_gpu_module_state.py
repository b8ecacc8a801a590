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


def _counting(f):
    calls = []

    def g(*a):
        calls.append(1)
        return f(*a)
    return g, calls


def _fresh(mod):
    m = QuantLinear(BITS, GS, K, N, True)
    for name in ("qweight", "qzeros", "scales", "g_idx", "bias"):
        t = getattr(mod, name)
        setattr(m, name, None if t is None else t.clone())
    return m


@pytest.mark.parametrize("how", ["new tensor", "data", "in place"])
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
    elif how == "in place":
        getattr(mod, name).copy_(new)               # as load_state_dict does
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


def test_other_threads_go_on_while_a_launch_waits():
    """The device's queue is full behind a kernel of most of a second; the launches that wait for it hold no GIL."""
    import threading
    import time
    mod, x = _module(synth.make_layer(BITS, K, N, GS, False, bias=True, seed=1, device=DEV)), synth.make_x(1, K, seed=3, device=DEV)
    want = mod(x)
    mod(x)
    torch.cuda.synchronize()
    outs = []

    def work():
        torch.cuda._sleep(1_500_000_000)
        outs.extend([mod(x) for _ in range(4000)][-1:])

    t = threading.Thread(target=work)
    t.start()
    longest, last = 0.0, time.perf_counter()
    while t.is_alive():
        time.sleep(0.005)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    t.join()
    torch.cuda.synchronize()
    assert torch.equal(outs[0], want)
    assert longest < 0.25, f"this thread stood still for {longest:.2f} s"


def test_threads_and_streams_share_a_module():
    """Four threads, each on a stream of its own, in the rows' three routes, while the scratch of each stream grows."""
    import threading
    mod = _module(synth.make_layer(BITS, K, N, GS, True, bias=True, seed=1, device=DEV))
    xs = [synth.make_x(M, K, seed=M, device=DEV) for M in (1, 16, 32, 1500)]
    want = [mod(x) for x in xs]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                for x, w in list(zip(xs, want))[i:] + list(zip(xs, want))[:i]:
                    y = mod(x)
                    if not torch.equal(y, w):
                        wrong.append((i, x.shape[0]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
    ops.check_status(DEV)


@pytest.mark.parametrize("act", [False, True])
def test_copies_of_a_used_module(act):
    import copy
    import io
    mod = _module(synth.make_layer(BITS, K, N, GS, act, bias=True, seed=1, device=DEV))
    xs = [synth.make_x(M, K, seed=M, device=DEV) for M in ROWS]
    want = [mod(x) for x in xs]
    f = io.BytesIO()
    torch.save(mod, f)
    f.seek(0)
    for c in (copy.deepcopy(mod), torch.load(f, weights_only=False)):
        for _ in range(2):
            assert all(torch.equal(c(x), w) for x, w in zip(xs, want))


@pytest.mark.parametrize("M", [1, 32])
@pytest.mark.parametrize("name", ["scales", "qzeros"])
def test_new_constants_are_waited_for_once(monkeypatch, M, name):
    """The kernels read scales and zero-points before the kernel in front of them has ended; the call after they were written
    puts an ordinary operation in between, later ones and the first after post_init() do not."""
    mod, x = _module(synth.make_layer(BITS, K, N, GS, False, bias=True, seed=1, device=DEV)), synth.make_x(M, K, seed=3, device=DEV)
    settle, calls = _counting(ops.settle)
    monkeypatch.setattr(ops, "settle", settle)
    mod(x), mod(x)
    assert not calls
    getattr(mod, name).add_(1 if name == "qzeros" else 0.5)
    mod(x), mod(x), mod(x)
    assert len(calls) == 1
    setattr(mod, name, getattr(mod, name) * 2)
    mod(x), mod(x)
    assert len(calls) == 2 and torch.equal(mod(x), _fresh(mod)(x))
