"""Pieces shared by the K and V plane stores: constants, exponent extraction, residual-token buffering."""
from __future__ import annotations

import torch
from torch.autograd import forward_ad

# One K channel row of a block holds 256 bits of high bytes = 64 tokens (extension/k_cache_file.py:5-6).
bits_in_a_channel = 256
column_block = bits_in_a_channel // 4


def cdiv(a: int, b: int) -> int:
    return -(-a // b)


def exponent_field(x: torch.Tensor) -> torch.Tensor:
    """5-bit biased exponent of every fp16 element, as uint8 (the reference's
    `(x.view(int16) >> 10).to(uint8) & 0x1F`, e.g. extension/k_cache_file.py:77-78,98-99,136)."""
    return (x.view(torch.int16) >> 10).to(torch.uint8) & 0x1F


def observed() -> bool:
    """Whether something is in force that sees, records or changes single tensor operations, so that they have to run as such:
    a dispatch or function mode (one that only names the default device aside), a functorch transform, forward-mode
    derivatives, tracing, autocast.  A private query that this torch does not have counts as a yes."""
    try:
        if torch._C._len_torch_dispatch_stack() or forward_ad._current_level >= 0 or torch.jit.is_tracing() or \
                torch.is_autocast_enabled("cuda") or torch._C._functorch.peek_interpreter_stack() is not None:
            return True
        n = torch._C._len_torch_function_stack()
        return n > 0 and any(type(torch._C._get_function_stack_at(i)).__module__ != "torch.utils._device" for i in range(n))
    except (AttributeError, TypeError):
        return True


def one_call(x: torch.Tensor, rest: torch.Tensor | None, exp_max: torch.Tensor, planes, rest_shape, exp_shape) -> bool:
    """Whether `decoding_compute` may run as one library call (`cuda_module.k_scores` / `v_output`) instead of tensor
    operations: plain contiguous 16-byte aligned CUDA tensors of the cache's own shapes on one device, nothing that autograd, a
    tensor subclass or what `observed` asks for would have to see.  Everything else takes the tensor operations, and fails there
    where it failed before."""
    if type(x) is not torch.Tensor or not x.is_cuda or x.dtype != torch.half or not x.is_contiguous() or type(rest) is not torch.Tensor:
        return False
    if rest.dtype != torch.half or rest.shape != rest_shape or not rest.is_contiguous() or rest.device != x.device:
        return False
    if exp_max.dtype != torch.uint8 or exp_max.shape != exp_shape or not exp_max.is_contiguous() or exp_max.device != x.device:
        return False
    if torch.is_grad_enabled() and (x.requires_grad or rest.requires_grad):
        return False
    if observed():
        return False
    at = x.data_ptr() | rest.data_ptr() | exp_max.data_ptr()
    for p in planes:
        if p.device != x.device:
            return False
        at |= p.data_ptr()
    return at % 16 == 0


class ResidualBuffer:
    """The fp16 staging area for tokens that do not yet fill a 64-token block.

    The reference keeps them in `restk` / `restv` of shape [bsz, 64, heads, head_dim] with a fill count and the
    position of the first buffered token (extension/k_cache_file.py:92-96,100-118; extension/v_cache_file.py:92-96,
    101-116).  Only whole blocks ever reach the plane writers.
    """

    def __init__(self, bsz: int, heads: int, head_dim: int, device):
        self.shape = (bsz, column_block, heads, head_dim)
        self.device = device
        self.data: torch.Tensor | None = None
        self.fill = 0
        self.start = 0

    def fresh(self) -> torch.Tensor:
        self.data = torch.zeros(self.shape, dtype=torch.half, device=self.device)
        return self.data

    def load_tail(self, new: torch.Tensor, seqlen: int) -> None:
        """After a prefill: keep the seqlen % 64 trailing tokens."""
        tail = seqlen % column_block
        self.fresh()
        self.data[:, :tail, :, :] = new[:, seqlen - tail:, :]
        self.fill = tail
        self.start = seqlen - tail

    def push(self, new: torch.Tensor, seqlen: int) -> bool:
        """Append decode tokens; True when the buffer now holds a whole block."""
        self.data[:, self.fill:self.fill + seqlen, :, :] = new
        self.fill += seqlen
        return self.fill == column_block

    def advance(self) -> None:
        """The buffered block has been written to the planes."""
        self.fill = 0
        self.start += column_block
        self.fresh()
