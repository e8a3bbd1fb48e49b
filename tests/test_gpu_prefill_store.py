"""Prompt ingestion adds the K nibbles onto what the planes hold, whoever wrote it; stores them where a caller of the library says
that the planes are zero."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def planes(layer):
    return [t.clone() for t in (layer.k_first_8, layer.k_mid_4, layer.k_last_4, layer.v_first_8, layer.v_mid_4, layer.v_last_4,
                                layer.k_exp_max, layer.v_exp_max, layer.restk, layer.restv)]


def call_ex(layer, k, v, flags):
    """akv_prefill_ex on the layer's buffers"""
    B, S, H, D = k.shape
    n = layer.lib.akv_prefill_scratch_bytes(B, H, D, S)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    return layer.lib.akv_prefill_ex(*(t.data_ptr() for t in (
        layer.k_first_8, layer.k_mid_4, layer.k_last_4, layer.v_first_8, layer.v_mid_4, layer.v_last_4, layer.k_exp_max,
        layer.v_exp_max, layer.restk, layer.restv, k, v, ws)), n, B, H, D, layer.L, S, flags, torch.cuda.current_stream().cuda_stream)


def inputs(B, H, D, S):
    g = torch.Generator(device="cuda").manual_seed(S)
    return [torch.randn(B, n, H, D, device="cuda", generator=g).half() for n in (S, S, 1)]


@pytest.mark.parametrize("B,H,D,S", [(1, 1, 128, 64), (2, 3, 128, 130), (3, 8, 128, 63), (2, 2, 64, 200), (1, 4, 128, 1027)])
def test_store_and_add(B, H, D, S):
    from alignedkv_b200.decode import DecodeLayer
    g = torch.Generator(device="cuda").manual_seed(S)
    k, v, q = (torch.randn(B, n, H, D, device="cuda", generator=g).half() for n in (S, S, 1))
    make = lambda: DecodeLayer(B, -(-(S + 70) // 64) * 64, H, D, "cuda:0")  # noqa: E731
    stored, added, dirty = make(), make(), make()
    assert stored._nibbles_known()
    added.k_mid_4.add_(0)                                  # a tensor operation: the layer can no longer know
    assert not added._nibbles_known()
    dirty.k_mid_4.fill_(1)
    for layer in (stored, added, dirty):
        layer.prefill(k, v)
    for a, b in zip(planes(stored), planes(added)):
        assert torch.equal(a, b)
    n = S // 64
    assert torch.equal(dirty.k_mid_4[:, :, :n], stored.k_mid_4[:, :, :n] + 1)       # (bytewise, modulo 256)
    assert torch.equal(dirty.k_last_4, stored.k_last_4)
    # rewound to nothing and filled again, also over a block that a step flushed
    empty = make()
    snap = empty.snapshot()
    empty.prefill(k, v)
    for _ in range(64 - S % 64):
        empty.decode(q, k[:, :1].contiguous(), v[:, :1].contiguous())
    empty.restore(snap)
    assert int(empty.k_mid_4.count_nonzero()) == 0 and int(empty.k_last_4.count_nonzero()) == 0
    empty.prefill(k, v)
    for a, b in zip(planes(empty)[:3], planes(stored)[:3]):
        assert torch.equal(a[:, :, :n], b[:, :, :n])


@pytest.mark.parametrize("B,H,D,S", [(1, 1, 128, 64), (2, 3, 128, 130), (3, 8, 128, 63), (2, 2, 64, 200), (1, 4, 128, 1027)])
def test_store_on_request(B, H, D, S):
    """AKV_PREFILL_STORE on planes that are zero leaves what adding leaves."""
    from alignedkv_b200.decode import DecodeLayer
    k, v, _ = inputs(B, H, D, S)
    stored, added = (DecodeLayer(B, -(-(S + 70) // 64) * 64, H, D, "cuda:0") for _ in range(2))
    assert call_ex(stored, k, v, 1) == 0
    added.prefill(k, v)
    for a, b in zip(planes(stored), planes(added)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("writer", ["operator", "data", "dlpack", "tensor"])
def test_adds_onto_what_others_wrote(D, writer):
    """Writers that a tensor's version counter does not see: the library's own K block writer, `.data`, DLPack."""
    from alignedkv_b200.decode import DecodeLayer
    from alignedkv_b200.extension.KV_cache_cpp_extention import cuda_module
    B, H, S = 2, 3, 130
    k, v, _ = inputs(B, H, D, S)
    clean, layer = (DecodeLayer(B, 192, H, D, "cuda:0") for _ in range(2))
    clean.prefill(k, v)
    if writer == "operator":
        cuda_module.k_cache_save(layer.k_first_8, layer.k_mid_4, layer.k_last_4, k.flip(1).contiguous().view(torch.uint8), B, H, 2, 3,
                                 D, 64, 0, S)
    elif writer == "data":
        layer.k_mid_4.data.fill_(7)
        layer.k_last_4.data.fill_(9)
    elif writer == "dlpack":
        torch.from_dlpack(layer.k_mid_4).fill_(7)
    else:
        layer.k_last_4.fill_(200)
    was = layer.k_mid_4.clone(), layer.k_last_4.clone()
    assert any(int(t.count_nonzero()) for t in was)
    layer.prefill(k, v)
    assert torch.equal(layer.k_mid_4[:, :, :2], was[0][:, :, :2] + clean.k_mid_4[:, :, :2])       # (modulo 256)
    assert torch.equal(layer.k_last_4[:, :, :2], was[1][:, :, :2] + clean.k_last_4[:, :, :2])


def test_inference_tensors_add():
    from alignedkv_b200.decode import DecodeLayer
    with torch.inference_mode():
        layer = DecodeLayer(1, 128, 1, 128, "cuda:0")
        assert not layer._nibbles_known()
        layer.prefill(torch.randn(1, 100, 1, 128, device="cuda").half(), torch.randn(1, 100, 1, 128, device="cuda").half())


def test_inference_tensors_add_the_same():
    from alignedkv_b200.decode import DecodeLayer
    k, v, _ = inputs(1, 1, 128, 100)
    clean = DecodeLayer(1, 128, 1, 128, "cuda:0")
    clean.prefill(k, v)
    with torch.inference_mode():
        layer = DecodeLayer(1, 128, 1, 128, "cuda:0")
        layer.k_mid_4.fill_(3)
        layer.prefill(k, v)
    assert torch.equal(layer.k_mid_4[:, :, :1], clean.k_mid_4[:, :, :1] + 3)


def test_unknown_flags_are_refused():
    from alignedkv_b200.decode import DecodeLayer
    k, v, _ = inputs(1, 1, 128, 64)
    layer = DecodeLayer(1, 128, 1, 128, "cuda:0")
    for flags in (2, 3, -1):
        assert call_ex(layer, k, v, flags) == -2 and int(layer.k_first_8.count_nonzero()) == 0
