"""Front-end of the tcgen05 flash-attention kernel (packed QKV layout, head dim 128)."""
from __future__ import annotations

import torch

from .. import _native
from .gemm import status_buffer, status_ptr

import os

LAUNCHES = 0
# 0: the launcher takes the kernel that suits the size
VERSION = int(os.environ.get("FLUIDMOE_FLASH_VERSION", "0"))
BWD_VERSION = int(os.environ.get("FLUIDMOE_FLASH_BWD_VERSION", "2"))


_t_flash_fwd = _native.tensor_call(globals(), "t_flash_fwd")
_t_flash_bwd = _native.tensor_call(globals(), "t_flash_bwd")


def supported(qkv: torch.Tensor, head_dim: int) -> bool:
    return (qkv.is_cuda and qkv.dtype == torch.bfloat16 and head_dim == 128 and qkv.is_contiguous()
            and _native.available() and hasattr(_native.lib(), "flash_attn_fwd"))


def can_push(qkv: torch.Tensor, rows_per_rank: int, version: int = 0) -> bool:
    """Whether the forward kernel can do the HP -> SP exchange in its epilogue for this input."""
    return (version or VERSION) in (0, 2) and qkv.shape[1] == 1 and rows_per_rank > 0 and rows_per_rank % 128 == 0


def flash_attn_fwd_packed(qkv: torch.Tensor, q_per_group: int, head_dim: int, scale: float, version: int = 0,
                          push=None):
    """qkv: [s, b, G, (qpg + 2) * d] -> (out [s, b, G*qpg, d], lse [b, G*qpg, s]).

    ``push`` (``dict(dst_table, flags_table, me, P, rows_per_rank, row_blocks)``): every output row is
    also stored into the sequence owner's buffer and the owner's arrival counter is raised, which
    replaces the separate HP -> SP push (fluid/attention/forward.py:435-476)."""
    global LAUNCHES
    if push is None and qkv.is_cuda:
        res = _t_flash_fwd(qkv, q_per_group, head_dim, scale, version or VERSION, status_ptr(qkv))
        if res is not None:
            LAUNCHES += 1
            return res
    s, b, G, gs = qkv.shape
    hq = G * q_per_group
    out = torch.empty(s, b, hq, head_dim, dtype=qkv.dtype, device=qkv.device)
    lse = torch.empty(b, hq, s, dtype=torch.float32, device=qkv.device)
    LAUNCHES += 1
    if push is None:
        _native.lib().flash_attn_fwd(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), s, b, G, q_per_group,
                                     head_dim, float(scale), 0, status_buffer(qkv.device).data_ptr(),
                                     version or VERSION, _native.stream_ptr())
    else:
        _native.lib().flash_attn_fwd_push(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), s, b, G, q_per_group,
                                          head_dim, float(scale), 0, status_buffer(qkv.device).data_ptr(),
                                          version or VERSION, push["dst_table"], push["flags_table"],
                                          push["me"], push["P"], push["rows_per_rank"], push["row_blocks"],
                                          _native.stream_ptr())
    return out, lse


def _head_split(s: int, b: int, groups: int, q_per_group: int, sms: int = 148) -> int:
    """CTAs that share the query heads of a K/V block and KV head in the backward kernel.

    A CTA walks the query tiles behind its block for each of its heads, so the CTA of the first block is the longest.
    Heads are split until it takes no more than one and a half times an SM's share of all steps; a further split only
    adds the fp32 sums of dK and dV and a conversion.  One against two and four CTAs, 8 KV heads of 4: 4096
    positions (longest 128 steps, share 114) 345, 378, 415 us; 3072 (96, 65) 253, 247, 265; 2048 (64, 29) 171, 134, 155;
    1024 (32, 8) 93, 73, 69.  1 of 8, 4096 (256, 29): 548, 289, 165, eight CTAs 110."""
    tiles = (s + 127) // 128
    share = tiles * (tiles + 1) // 2 * groups * b * q_per_group / sms
    split = 1
    while q_per_group % (split * 2) == 0 and tiles * q_per_group / split > 1.5 * share:
        split *= 2
    return split


def flash_attn_bwd_packed(dout: torch.Tensor, qkv: torch.Tensor, out: torch.Tensor, lse: torch.Tensor,
                          q_per_group: int, head_dim: int, scale: float, version: int = 0,
                          head_split=None, wait=None) -> torch.Tensor:
    """Gradient of the packed projection buffer, ``[s, b, G, (qpg + 2) * d]`` (dq heads, dk, dv per
    KV group), from the saved output and log-sum-exp.  ``wait`` (``dict(flags, n, expected, wait_ns)``,
    addresses as ints): per-source arrival counters of ``dout`` that the first kernel waits for."""
    global LAUNCHES
    s, b, G, gs = qkv.shape
    hq = G * q_per_group
    dout = dout.contiguous()
    ver = version or BWD_VERSION
    hsplit = 1
    if ver == 2 and head_split is not False:
        hsplit = head_split or _head_split(s, b, G, q_per_group)
    if ver == 2 and wait is None and qkv.is_cuda:
        res = _t_flash_bwd(dout, qkv, out, lse, q_per_group, head_dim, scale, hsplit, status_ptr(qkv))
        if res is not None:
            LAUNCHES += 3 + (1 if hsplit > 1 else 0)
            return res
    delta = torch.empty(b, hq, s, dtype=torch.float32, device=qkv.device)
    # the default kernel sums dQ in whole tiles of 128 rows, in a layout of its own
    rows = (s + 127) // 128 * 128 if ver == 2 else s
    dq_accum = torch.empty(rows, b, hq, head_dim, dtype=torch.float32, device=qkv.device)
    dqkv = torch.empty_like(qkv)
    dkv = torch.empty(s, b, G, 2, head_dim, dtype=torch.float32, device=qkv.device) if hsplit > 1 else None
    LAUNCHES += 3 + (1 if hsplit > 1 else 0)
    args = (qkv.data_ptr(), out.data_ptr(), dout.data_ptr(), lse.data_ptr(), delta.data_ptr(),
            dq_accum.data_ptr(), dqkv.data_ptr(), s, b, G, q_per_group, head_dim, float(scale),
            0, status_buffer(qkv.device).data_ptr(), ver, dkv.data_ptr() if dkv is not None else 0, hsplit)
    if wait is None:
        _native.lib().flash_attn_bwd(*args, _native.stream_ptr())
    else:
        # `dout` is still being filled by peers: the first kernel waits for their arrival counters
        _native.lib().flash_attn_bwd_gated(*args, wait["flags"], wait["n"], wait["expected"], wait["wait_ns"],
                                           _native.stream_ptr())
    return dqkv
