"""Calls of different sizes of one kernel from two host threads, each on its own stream: the kernels' shared-memory limit is an
attribute that all threads see, so no call may lower it under another one's launch."""
import threading

import pytest
import torch

from test_gpu_ext import check, stream

pytestmark = pytest.mark.gpu


def _prompt(lib, D):
    """A prompt of one block and a bit: head sizes beyond 192 need more than the default 48 KB."""
    B, H, S, L = 1, 1, 80, 128
    k, v = (torch.randn(B, S, H, D, device="cuda").half() for _ in range(2))
    planes = [torch.zeros(B * H * L * D // n, dtype=torch.uint8, device="cuda") for n in (1, 2, 2, 1, 2, 2)]
    exps = [torch.zeros(B * H * D, dtype=torch.uint8, device="cuda") for _ in range(2)]
    rest = [torch.zeros(B, 64, H, D, dtype=torch.half, device="cuda") for _ in range(2)]
    ws = torch.empty(lib.akv_prefill_scratch_bytes(B, H, D, S), dtype=torch.uint8, device="cuda")
    keep = (k, v, planes, exps, rest, ws)
    args = [x.data_ptr() for x in (*planes, *exps, *rest, k, v, ws)]
    return keep, lambda: check(lib, lib.akv_prefill(*args, ws.numel(), B, H, D, L, S, stream()))


def _k_save(lib, D):
    """One block of keys: head sizes beyond 384 need more than the default 48 KB."""
    k = torch.randn(1, 64, 1, D, device="cuda").half()
    planes = [torch.zeros(64 * D // n, dtype=torch.uint8, device="cuda") for n in (1, 2, 2)]
    args = [x.data_ptr() for x in (*planes, k)]
    return (k, planes), lambda: check(lib, lib.akv_k_cache_save(*args, 1, 1, 1, 1, D, 64, 0, 64, stream()))


@pytest.mark.parametrize("make,sizes", [(_prompt, (256, 224)), (_k_save, (768, 400))])
def test_two_sizes_on_two_threads(akv_lib, make, sizes):
    failed = []

    def work(D):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                keep, call = make(akv_lib, D)
                for _ in range(20000):
                    call()
                torch.cuda.current_stream().synchronize()
                del keep
        except Exception as e:  # noqa: BLE001
            failed.append(f"{D}: {e}")

    threads = [threading.Thread(target=work, args=(D,)) for D in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
