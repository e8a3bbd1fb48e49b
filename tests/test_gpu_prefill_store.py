"""Prompt ingestion stores the K nibbles while nobody but the layer has written its planes, and adds them otherwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def planes(layer):
    return [t.clone() for t in (layer.k_first_8, layer.k_mid_4, layer.k_last_4, layer.v_first_8, layer.v_mid_4, layer.v_last_4,
                                layer.k_exp_max, layer.v_exp_max, layer.restk, layer.restv)]


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


def test_inference_tensors_add():
    from alignedkv_b200.decode import DecodeLayer
    with torch.inference_mode():
        layer = DecodeLayer(1, 128, 1, 128, "cuda:0")
        assert not layer._nibbles_known()
        layer.prefill(torch.randn(1, 100, 1, 128, device="cuda").half(), torch.randn(1, 100, 1, 128, device="cuda").half())
