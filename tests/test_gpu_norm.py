"""b200gptq_add_norm against 64 bits: rows that fill part of a warp, whole warps, 1024 threads and two passes of them, and rows
whose mean is several hundred times their spread (LayerNorm of more than 16 rows sums the variance around the mean)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from autogptq.tvm_b200 import ops
    DEV = torch.device("cuda:0")


@pytest.mark.parametrize("H", [8, 64, 264, 1032, 4096, 8184, 8192, 8200, 9216, 12288])
@pytest.mark.parametrize("rms,rows,offset", [(True, 5, 60.0), (False, 5, 0.0), (False, 16, 0.0), (False, 17, 0.0), (False, 17, 60.0)])
@pytest.mark.parametrize("add", [False, True])
def test_add_norm(H, rms, rows, offset, add):
    eps = 1e-5
    g = torch.Generator().manual_seed(H)
    draw = lambda *s: torch.randn(*s, generator=g)
    x, d = (offset + 0.1 * draw(rows, H)).half(), (0.1 * draw(rows, H)).half()
    x[1, 0], x[2, H // 2] = 500., -300.         # one value far from all others, also where the sums begin
    w, b = (1 + 0.1 * draw(H)).half(), (0.1 * draw(H)).half()
    xd, out = x.to(DEV), torch.empty(rows, H, dtype=torch.float16, device=DEV)
    ops.add_norm(xd, d.to(DEV) if add else None, w.to(DEV), None if rms else b.to(DEV), out, eps, rms)
    s = x + d if add else x
    assert torch.equal(xd.cpu(), s)
    v = s.double()
    if rms:
        ref = v * torch.rsqrt(v.pow(2).mean(1, keepdim=True) + eps) * w.double()
    else:
        ref = torch.nn.functional.layer_norm(v, (H,), w.double(), b.double(), eps)
    # Two fp16 roundings (RMSNorm's value and the result), and fp32 sums of H values of the mean's size: an error of
    # sqrt(H) 2^-24 of the mean, divided by the spread, in a value below 6 spreads.
    bound = 2.0 ** -10 * ref.abs() + 2.0 ** -24 * H ** 0.5 * (offset + 1) / 0.1 + 1e-5
    assert bool(((out.cpu().double() - ref).abs() <= bound).all())
