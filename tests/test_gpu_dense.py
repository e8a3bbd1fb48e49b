"""Element-wise kernels of the decoder's decode step against the tensor operations they stand for."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def call(fn, *args):
    from alignedkv_b200 import _lib
    _lib.check(fn, getattr(_lib.load(), fn)(*args, torch.cuda.current_stream().cuda_stream))


def rand(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)) * scale).half()


def close(a, b, steps):
    """Equal up to `steps` fp16 steps of the larger value (rounding once from fp32 sums added in another order)."""
    return bool(((a.float() - b.float()).abs() <= steps * 2.0 ** -10 * b.float().abs() + 2.0 ** -20).all())


@pytest.mark.parametrize("B,H,Hkv,D,pos", [(1, 1, 1, 16, 0), (3, 4, 4, 64, 7), (16, 32, 32, 128, 1024), (5, 32, 8, 128, 131071),
                                           (2, 7, 1, 96, 300), (2, 3, 3, 256, 5000)])
def test_rope_split(B, H, Hkv, D, pos):
    from alignedkv_b200.llama import _rope, _rope_tables
    qkv = rand(B, 1, H + 2 * Hkv, D, seed=D)
    p = torch.tensor([pos], device="cuda")
    q, k, v = (torch.empty(B, 1, n, D, dtype=torch.half, device="cuda") for n in (H, Hkv, Hkv))
    call("akv_rope_split", qkv.data_ptr(), p.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), B, H, Hkv, D, 10000.0)
    cos, sin = (t.double() for t in _rope_tables(p, D, 10000.0))
    x = qkv[:, :, :H + Hkv].double()
    want = x * cos + torch.cat([x[..., D // 2:], x[..., :D // 2]], -1) * sin
    # fp32 products and sum of two terms, then fp16: half an fp16 step, and fp32 steps of the terms where they cancel
    got = torch.cat([q, k], 2).double()
    assert bool(((got - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -22 * 8 + 2.0 ** -25).all())
    assert torch.equal(v, qkv[:, :, H + Hkv:])
    # (and the tensor operations themselves, up to the same rounding)
    assert float((torch.cat([q, k], 2).float() - _rope(qkv[:, :, :H + Hkv], _rope_tables(p, D, 10000.0)).float()).abs().max()) <= 2.0 ** -8


@pytest.mark.parametrize("rows,width", [(1, 8), (3, 1032), (16, 11008), (7, 14336)])
def test_silu_mul(rows, width):
    x = rand(rows, 2 * width, seed=width, scale=3.0)
    x[0, 0], x[0, 1] = -60000.0, 60000.0
    out = torch.empty(rows, width, dtype=torch.half, device="cuda")
    call("akv_silu_mul", x.data_ptr(), out.data_ptr(), rows, width)
    gate, up = x.chunk(2, dim=-1)
    want = F.silu(gate) * up
    fin = want.isfinite()
    assert torch.equal(fin, out.isfinite()) and close(out[fin], want[fin], 2)


@pytest.mark.parametrize("rows,width", [(1, 8), (3, 1032), (16, 11008), (7, 14336)])
def test_silu_mul_is_the_tensor_operations(rows, width):
    x = rand(rows, 2 * width, seed=width, scale=3.0)
    x[0, 0], x[0, 1] = -60000.0, 60000.0
    out = torch.empty(rows, width, dtype=torch.half, device="cuda")
    call("akv_silu_mul", x.data_ptr(), out.data_ptr(), rows, width)
    gate, up = x.chunk(2, dim=-1)
    want = F.silu(gate) * up
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    fin = want.isfinite()
    assert close(out[fin].float(), (gate.double() * torch.sigmoid(gate.double())).half().double().mul(up.double())[fin].float(), 2)


def test_silu_of_every_value():
    """Every fp16 gate, NaN and infinities among them, against the tensor operations bit for bit and against 64 bits."""
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.half)
    for up in (1.0, 0.3333, -1000.0, 65504.0, torch.inf, torch.nan, 1e-7):
        x = torch.stack([gate, torch.full_like(gate, up)])
        out = torch.empty_like(gate)
        call("akv_silu_mul", x.data_ptr(), out.data_ptr(), 1, gate.numel())
        want = F.silu(x[0]).mul_(x[1])
        assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[~want.isnan()], want[~want.isnan()])
        if up == 1.0:
            d = gate.double()
            fin = d.isfinite()
            exact = (d / (1 + torch.exp(-d)))[fin]
            # (one rounding of an fp32 quotient that is off by a few fp32 steps; gates whose exponential overflows give -0)
            assert bool(((out[fin].double() - exact).abs() <= (2.0 ** -11 + 2.0 ** -20) * exact.abs() + 2.0 ** -25).all())


def test_silu_of_many_rows():
    x = rand(70000, 16, seed=3)
    out = torch.empty(70000, 8, dtype=torch.half, device="cuda")
    call("akv_silu_mul", x.data_ptr(), out.data_ptr(), 70000, 8)
    assert torch.equal(out, F.silu(x[:, :8]) * x[:, 8:])


@pytest.mark.parametrize("rows,width", [(1, 8), (2, 520), (16, 4096), (3, 8192), (2, 16384), (64, 4104)])
def test_rms_norm(rows, width):
    x, w = rand(rows, width, seed=width, scale=2.0), rand(width, seed=1)
    out = torch.empty_like(x)
    call("akv_rms_norm", x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, width, 1e-5)
    d = x.double()
    want = d / (d.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()
    assert bool(((out.double() - want).abs() <= (2.0 ** -11 + 2.0 ** -20) * want.abs() + 2.0 ** -25).all())


def test_refused():
    from alignedkv_b200 import _lib
    lib, x = _lib.load(), rand(64)
    st = torch.cuda.current_stream().cuda_stream
    assert lib.akv_rms_norm(x.data_ptr(), x.data_ptr(), x.data_ptr(), 1, 12, 1e-5, st) == -2
    assert lib.akv_silu_mul(x.data_ptr(), x.data_ptr(), 1, 12, st) == -2
    assert lib.akv_silu_mul(x.data_ptr() + 2, x.data_ptr(), 1, 8, st) == -3
    assert lib.akv_rope_split(x.data_ptr(), x.data_ptr(), x.data_ptr(), x.data_ptr(), x.data_ptr(), 1, 1, 1, 8, 1e4, st) == -2
