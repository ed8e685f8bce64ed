"""Expert-grouped products over routes sorted by expert (the prefill side of ``gather_vqmm``).

Stands in for the reference's sorted-route kernels: ``gather_vqmm_tiled_down`` /
``gather_vqmm_mma*_blocks`` (``src/ramp/kernels/gather_vqmm.py:597-928``) and the native
``nax_e8p_fp16_sorted_matmul_steel[_m32n64]`` (``src/ramp/kernels/nax.py:330-366,3601-3632``).

16-bit E8P codes with fp16 / bf16 activations whose shapes fit go to ``keepvq_grouped_projection``
(int8 tensor cores: the tcgen05 kernel from 5 routes per expert on, 8 where a row has several scale
groups, the mma.sync ones below); 8-bit codes go to ``keepvq_grouped_projection_bytes`` (tcgen05) where
``byte_codes_served`` says so; everything else (fp32 activations, odd shapes, custom 16-bit tables with
even nibbles) to the general routed kernel.
"""

from __future__ import annotations

import ctypes
import threading
from functools import lru_cache

import torch

from . import _lib
from .kernels import routed_matvec

_UNSUPPORTED = -5  # KEEPVQ_ERR_UNSUPPORTED
_all_odd: dict = {}     # table data_ptr, device -> (the tensor, its version, every nibble odd): read back once per table, never per call
_all_odd_lock = threading.Lock()  # of the entries' insertion and eviction
_MAX_CACHED = 8


def _table_all_odd(table: torch.Tensor) -> bool:
    """Whether every nibble of the table is odd (what the int8 kernels need).  The cache holds the
    tensor itself, so its address cannot be handed to another table while the entry lives, and an
    in-place change of the table (a new version) is looked at again.  Another thread may drop the
    entry at any time: the answer comes from what was looked up or worked out here."""
    key = (table.data_ptr(), table.get_device())
    hit = _all_odd.get(key)
    if hit is None or hit[0] is not table or hit[1] != table._version:
        version = table._version
        nibbles = (table.cpu().to(torch.int64) & 0xFFFFFFFF)[:, None] >> (4 * torch.arange(8))[None] & 1
        hit = (table, version, bool(nibbles.all()))
        with _all_odd_lock:
            if len(_all_odd) >= _MAX_CACHED and key not in _all_odd:
                _all_odd.pop(next(iter(_all_odd)))
            _all_odd[key] = hit
    return hit[2]


@lru_cache(maxsize=256)
def _scratch_bytes(routes: int, in_dim: int) -> int:
    nbytes = int(_lib.load().keepvq_grouped_projection_workspace_bytes(routes, in_dim))
    if nbytes < 0:
        _lib.check(nbytes, "keepvq_grouped_projection_workspace_bytes")
    return nbytes


@lru_cache(maxsize=256)
def byte_codes_served(routes: int, slots: int, out_dim: int, in_dim: int, groups: int) -> bool:
    """Whether 8-bit calls of these sizes go to the grouped kernel (the rule and its figures: csrc/grouped.cu)."""
    return bool(_lib.load().keepvq_grouped_projection_bytes_served(routes, slots, out_dim, in_dim, groups))


def tensor_core_projection(rows, codes, scales, table, rhs, *, x_div: int = 1, code_bits: int = 16, residual=None, hot_of_slot=None):
    """``keepvq_grouped_projection`` (``_bytes`` for 8-bit codes): route ``r`` against activation row ``r // x_div`` of ``rows``
    (fp16 / bf16), optionally with a nested residual ``(res_codes, res_scales, res_table)``.
    Returns None when the library says these shapes are not for the tensor-core kernels."""
    routes = rhs.numel()
    if rows.shape[0] * x_div != routes:
        return None
    slots, out_dim = codes.shape[0], codes.shape[1]
    return project(rows, routes, rows.shape[1], codes, slots, out_dim, scales, scales.shape[2], table, rhs, (routes, out_dim),
                   x_div=x_div, code_bits=code_bits, residual=residual, hot_of_slot=hot_of_slot)


def project(rows, routes, in_dim, codes, slots, out_dim, scales, groups, table, rhs, out_shape, *, x_div=1, code_bits=16, residual=None, hot_of_slot=None):
    """The same with the sizes given beside the tensors (one matrix's codes and scales, say, without an
    experts' dimension; ``rhs`` may hold more than ``routes``), and the shape of the answer."""
    if codes.dtype != (torch.uint8 if code_bits == 8 else torch.uint16) or in_dim % 256 or rows.dtype not in (torch.float16, torch.bfloat16):
        return None
    if code_bits == 8 and not byte_codes_served(routes, slots, out_dim, in_dim, groups):
        return None  # (asked first: a call prepared to be refused cost 20 us)
    lib = _lib.load()
    device = rows.device
    stream = torch.cuda.current_stream(device).cuda_stream
    nbytes = _scratch_bytes(routes, in_dim)
    # Scratch of this call alone, from the caching allocator: calls of other threads, of other streams
    # and of other captured graphs have their own, and a graph's stays the graph's.
    ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
    out = torch.empty(out_shape, dtype=rows.dtype, device=device)  # (16-bit rows: qmv_output_dtype is theirs)
    rows = rows.contiguous()
    if rhs.dtype != torch.int32 or not rhs.is_contiguous():
        rhs = rhs.to(torch.int32).contiguous()
    if rows.data_ptr() % 16:  # a view that starts inside an allocation: the kernels read 16 bytes at a time
        rows = rows.clone()
    dtype, res = _lib.dtype_tag(rows.dtype), (0, 0, 0, 0, 0, 0)
    if residual is not None:
        res_codes, res_scales, res_table = residual
        if res_scales.dtype != scales.dtype:
            return None
        res = (res_codes.data_ptr(), res_scales.data_ptr(), res_codes.shape[0], res_scales.shape[2], res_table.data_ptr(), hot_of_slot.data_ptr())
    args = _lib.pack_grouped_args(
        rows.data_ptr(), dtype, routes, rhs.data_ptr(), codes.data_ptr(), scales.data_ptr(), _lib.dtype_tag(scales.dtype), slots, out_dim, in_dim, groups,
        table.data_ptr(), int(code_bits == 16 and _table_all_odd(table)), out.data_ptr(), dtype, ws.data_ptr(), nbytes, int(x_div), *res)
    with _lib.on_device(device):
        status = (lib.keepvq_grouped_projection_bytes if code_bits == 8 else lib.keepvq_grouped_projection)(args, ctypes.c_void_p(stream))
    if status == _UNSUPPORTED:
        return None
    _lib.check(status, "keepvq_grouped_projection")
    return out


def grouped_matmul_sorted(x, codes, scales, table, sorted_rhs, sorted_lhs, *, code_bits: int, tile_descriptors=None):
    """``out[r] = W[sorted_rhs[r]] @ x[sorted_lhs[r]]`` (``x[r]`` when ``sorted_lhs`` is None),
    ``[routes, out]`` in the given order.  ``tile_descriptors`` is accepted for callers that
    pre-build it; the CUDA kernels derive their own grouping from ``sorted_rhs``."""
    del tile_descriptors
    if x.dtype in (torch.float16, torch.bfloat16) and scales.dtype in (torch.float32, torch.float16, torch.bfloat16):
        rows = x if sorted_lhs is None else x[sorted_lhs.long()]  # the gather the reference does before its kernels
        out = tensor_core_projection(rows, codes, scales, table, sorted_rhs, code_bits=code_bits)
        if out is not None:
            return out
    return routed_matvec(x, codes, scales, table, sorted_rhs, lhs=sorted_lhs, x_div=1, code_bits=code_bits)
