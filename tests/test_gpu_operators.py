"""The cache classes' `decoding_compute` as one library call against the tensor operations it stands for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(B, H, D, P, seed, extra=0):
    from alignedkv_b200.extension.k_cache_file import K_Cache_Class
    from alignedkv_b200.extension.v_cache_file import V_Cache_Class
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randn(B, P, H, D, device="cuda", generator=g)
    k[..., [3, 34]] *= 20
    v = torch.randn(B, P, H, D, device="cuda", generator=g)
    L = -(-(P + 1) // 64) * 64 + extra
    kc, vc = K_Cache_Class(B, L, H, D, 0), V_Cache_Class(B, L, H, D, 0)
    kc.save(k.half(), 0, P)
    vc.save(v.half(), 0, P)
    return kc, vc, torch.randn(B, 1, H, D, device="cuda", generator=g).half()


def both(monkeypatch, call):
    """(result of one library call, result of the tensor operations)"""
    from alignedkv_b200.extension import k_cache_file, v_cache_file
    seen = []
    for m in (k_cache_file, v_cache_file):
        ok = m.one_call
        monkeypatch.setattr(m, "one_call", lambda *a, ok=ok: seen.append(ok(*a)) or seen[-1])
    one = call()
    assert seen == [True], "the call took the tensor operations"
    for m in (k_cache_file, v_cache_file):
        monkeypatch.setattr(m, "one_call", lambda *a: False)
    many = call()
    monkeypatch.undo()
    return one, many


def same(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("reference", [False, True])
@pytest.mark.parametrize("B,H,D,P", [(1, 1, 64, 1), (2, 3, 128, 63), (1, 8, 128, 64), (3, 5, 128, 65), (2, 4, 192, 191),
                                     (1, 2, 256, 130), (2, 32, 128, 2085), (1, 2, 320, 70)])
def test_scores(monkeypatch, B, H, D, P, reference):
    kc, _, q = make(B, H, D, P, P)
    one, many = both(monkeypatch, lambda: kc.decoding_compute(q, P - 1, 1, reference))
    n = P // 64 * 64
    assert one.shape == many.shape and same(one[..., :n], many[..., :n]) and same(one[..., P:], many[..., P:])
    # residual tokens: a dot product rounded to fp16, then a division rounded to fp16, each off by at most one fp16 step when
    # the fp32 sum is added in another order or divided through the reciprocal
    a, b = one[..., n:P].float(), many[..., n:P].float()
    assert bool(((a - b).abs() <= 2 * 2.0 ** -10 * b.abs() + 2.0 ** -14).all())


@pytest.mark.parametrize("reference", [False, True])
@pytest.mark.parametrize("B,H,D,P,kind", [(1, 1, 64, 64, "softmax"), (2, 3, 128, 65, "softmax"), (2, 4, 192, 127, "softmax"),
                                          (2, 2, 256, 200, "softmax"), (2, 32, 128, 2085, "softmax"), (1, 3, 128, 640, "flat"),
                                          (2, 3, 128, 300, "negative"), (2, 3, 128, 321, "nan"), (1, 2, 128, 8192, "ties")])
def test_output(monkeypatch, B, H, D, P, kind, reference):
    _, vc, _ = make(B, H, D, P, P, extra=64 if P % 128 else 0)
    g = torch.Generator(device="cuda").manual_seed(P)
    W = -(-(P + 1) // 64) * 64
    s = torch.randn(B, H, 1, W, device="cuda", generator=g) * (0.02 if kind == "flat" else 1.0)
    s[..., P:] = -torch.inf
    p = torch.softmax(s, -1).half()
    if kind == "negative":                     # any fp16 value is a legal "probability" of the operator
        p = torch.randn(B, H, 1, W, device="cuda", generator=g).half().neg().abs().neg()
        p[..., ::3] = -0.0
    elif kind == "nan":
        p[0, 0, 0, 40], p[0, 0, 0, 104], p[1, 2, 0, 7] = torch.nan, torch.nan, torch.inf
    elif kind == "ties":
        p = torch.full_like(p, 1 / 4096)
    one, many = both(monkeypatch, lambda: vc.decoding_compute(p, P - 1, 1, reference))
    assert one.shape == many.shape
    if P % 64 == 0:
        assert bool(((one == many) | (one.isnan() & many.isnan())).all())
        return
    # the residual part is rounded to fp16 before it is added: its last bit may differ, then the sum's
    nan = many.isnan()
    assert bool((one.isnan() == nan).all())
    a, b = one[~nan].float(), many[~nan].float()
    rest = torch.matmul(p[..., P // 64 * 64:P].float(), vc.restv.transpose(1, 2)[:, :, :P % 64].float())[~nan].abs()
    fin = b.isfinite()
    assert bool((a == b)[~fin].all())
    assert bool(((a - b).abs() <= 2.0 ** -10 * (b.abs() + rest) + 2.0 ** -14)[fin].all())


def test_routes():
    """What has to be seen by autograd, is not contiguous or has another top_max_k keeps the tensor operations."""
    from alignedkv_b200.extension._planes import one_call
    kc, _, q = make(2, 3, 128, 70, 1)
    planes = (kc.k_cache_first_8, kc.k_cache_mid_4, kc.k_cache_last_4)
    shapes = ((2, 64, 3, 128), (2, 1, 3, 128))
    assert one_call(q, kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    assert not one_call(q.clone().requires_grad_(), kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    with torch.no_grad():
        assert one_call(q.clone().requires_grad_(), kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    assert not one_call(q.float(), kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    assert not one_call(q.transpose(2, 3).contiguous().transpose(2, 3), kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    assert not one_call(torch.nn.Parameter(q, requires_grad=False), kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    flat = torch.empty(q.numel() + 1, dtype=torch.half, device="cuda")[1:].view(q.shape)
    assert not one_call(flat, kc.restk, kc.k_cache_exp_column_max, planes, *shapes)
    qg = q.clone().requires_grad_()
    s = kc.decoding_compute(qg, 69, 1)
    s[..., 64:70].float().sum().backward()
    assert qg.grad is not None and bool((qg.grad != 0).any())


def counting(f, seen):
    def wrapped(*a, **kw):
        seen.append(f.__name__)
        return f(*a, **kw)
    return wrapped


@pytest.mark.parametrize("where", ["instance", "class", "subclass"])
def test_replaced_probe_is_called(monkeypatch, where):
    """A `test_compute` put in the class's place, wherever it was put, is the one that runs."""
    from alignedkv_b200.extension.v_cache_file import V_Cache_Class
    _, vc, _ = make(2, 3, 128, 130, 7)
    p = torch.softmax(torch.randn(2, 3, 1, 192, device="cuda"), -1).half()
    want = vc.decoding_compute(p, 129, 1)
    seen, own = [], V_Cache_Class.test_compute
    replaced = lambda self, *a: seen.append("test_compute") or own(self, *a)  # noqa: E731
    if where == "instance":
        vc.test_compute = lambda *a: replaced(vc, *a)
    elif where == "class":
        monkeypatch.setattr(V_Cache_Class, "test_compute", replaced)
    else:
        vc.__class__ = type("Sub", (V_Cache_Class,), {"test_compute": replaced})
    got = vc.decoding_compute(p, 129, 1)
    assert seen == ["test_compute"]
    assert bool(((got.float() - want.float()).abs() <= 2.0 ** -9 * want.float().abs() + 2.0 ** -14).all())


@pytest.mark.parametrize("where", ["object", "class", "module"])
def test_wrapped_operators_are_called(monkeypatch, where):
    """Operators of `cuda_module` that a program wraps (to log, count or replace them) are called as before."""
    from helpers import CudaModuleSpy
    from alignedkv_b200.extension import k_cache_file, v_cache_file
    cm = k_cache_file.cuda_module
    kc, vc, q = make(2, 3, 128, 130, 7)
    p = torch.softmax(torch.randn(2, 3, 1, 192, device="cuda"), -1).half()
    names = ["k_cache_compute", "v_cache_test_compute", "v_cache_compute"]
    seen = []
    if where == "module":
        spy = CudaModuleSpy(cm)
        for m in (k_cache_file, v_cache_file):
            monkeypatch.setattr(m, "cuda_module", spy)
    else:
        at = cm if where == "object" else type(cm)
        for n in names:
            f = counting(getattr(at, n), seen)
            if where == "object":
                monkeypatch.setitem(vars(cm), n, f)      # (undone without a trace: setattr would leave the bound method on the object)
            else:
                monkeypatch.setattr(at, n, f)
    kc.decoding_compute(q, 129, 1)
    vc.decoding_compute(p, 129, 1)
    assert (list(spy.calls) if where == "module" else seen) == names


def test_modes_see_the_operations():
    """Dispatch and function modes, autocast and functorch transforms keep the tensor operations; a default device does not."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    from alignedkv_b200.extension._planes import observed
    kc, vc, q = make(2, 3, 128, 130, 7)
    p = torch.softmax(torch.randn(2, 3, 1, 192, device="cuda"), -1).half()
    seen = []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))

    for mode in (Dispatch, Function):
        seen.clear()
        with mode():
            kc.decoding_compute(q, 129, 1)
            vc.decoding_compute(p, 129, 1)
        assert sum("matmul" in n or "bmm" in n for n in seen) >= 2 and any("max" in n for n in seen), seen
    # autocast computes the residual tokens' products in its own type
    with torch.autocast("cuda", torch.bfloat16):
        s = kc.decoding_compute(q, 129, 1)
    rest = torch.matmul(q.transpose(1, 2).bfloat16(), kc.restk[:, :2].permute(0, 2, 3, 1).bfloat16()) / 128 ** 0.5
    assert torch.equal(s[..., 128:130], rest.half())
    assert not observed()
    with torch.device("cuda"):
        assert not observed()
    torch.func.vmap(lambda x: seen.append(observed()) or x)(q)
    assert seen[-1] is True
