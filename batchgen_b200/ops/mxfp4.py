"""MXFP4 (e2m1 values, one e8m0 scale per 32) expert weights: GEMMs and conversion.

On CUDA the GEMMs run ``gemm_mxfp4_block.cu``: the weights and their scales are operands of the block-scaled tensor-core product, and a
bf16 row is two e4m3 parts that sum up to it (``Parts``).  With the fused SiLU epilogue, for long segments and for shapes that its loads do not
take they run ``gemm_mxfp4.cu``, which expands the weights to bf16 on their way to TMEM.  On CPU the same contract is met by dequantising and multiplying in fp32.

Reference parity: quantiser / layout batchgen/quantization/mxfp4.py:30 and
batchgen/models/moonshotai/kimi_linear/k3/mxfp4_layout.py:37-38,179-182; grouped GEMMs
batchgen_kernels/src/moe/mxfp4/marlin_grouped_gemm.cu and batchgen/moe/fused_moe_mxfp4_resident.py:946-1125.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Optional, Union

import torch

from . import _ext, ref

EPI_STORE, EPI_SILU_MUL = 0, 1


def quantize(w: torch.Tensor):
    """[..., N, K] float -> (packed uint8 [..., N, K/2], scales uint8 [..., N, K/32])."""
    lead = w.shape[:-2]
    N, K = w.shape[-2:]
    q, s = ref.mxfp4_quant(w.reshape(-1, K))
    return q.view(*lead, N, K // 2), s.view(*lead, N, K // 32)


def dequantize(wq: torch.Tensor, ws: torch.Tensor, dtype=torch.bfloat16) -> torch.Tensor:
    """Expand packed weights to ``dtype`` (exact: every MXFP4 value is representable in bf16)."""
    lead = wq.shape[:-1]
    K = wq.shape[-1] * 2
    if not wq.is_cuda:
        return ref.mxfp4_dequant(wq.reshape(-1, K // 2), ws.reshape(-1, K // 32)).view(*lead, K).to(dtype)
    wq = wq.contiguous()
    ws = ws.contiguous()
    out = torch.empty(*lead, K, dtype=torch.bfloat16, device=wq.device)
    rc = _ext.lib().bg_mxfp4_dequant(_ext.ptr(wq), _ext.ptr(ws), _ext.ptr(out), ctypes.c_longlong(out.numel()),
                                     _ext.stream())
    _ext.check(rc, "bg_mxfp4_dequant")
    return out.to(dtype)


def _launch(epi, x, wq2d, ws2d, out, offsets, groups, M, N, K, counts=None):
    rc = _ext.lib().bg_mxfp4_gemm(
        ctypes.c_int(epi), _ext.ptr(x), _ext.ptr(wq2d), _ext.ptr(ws2d), _ext.ptr(out), ctypes.c_int(out.stride(0)),
        _ext.ptr(offsets), _ext.ptr(counts), ctypes.c_int(groups), ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K),
        ctypes.c_int(_ext.num_sms(x.device)), _ext.ptr(_ext.status_word(x.device)), _ext.stream())
    _ext.check(rc, "bg_mxfp4_gemm")


@dataclass
class Parts:
    """bf16 rows [rows, K] as the block-scaled product takes them: ``p`` uint8 [rows / 8 rounded up, 2, 8, K] (e4m3, eight rows' first parts and
    then their second parts), ``s`` uint8 [K / 128 rounded up, rows, 4] (e8m0 of the first part, one per 32 elements; the second part's is five
    less)."""
    p: torch.Tensor
    s: torch.Tensor

    @property
    def shape(self):
        return self.s.shape[1], self.p.shape[3]

    @property
    def is_cuda(self) -> bool:
        return self.p.is_cuda


def _new_parts(rows: int, K: int, device) -> Parts:
    return Parts(torch.empty(-(-rows // 8), 2, 8, K, dtype=torch.uint8, device=device), torch.empty(-(-K // 128), rows, 4, dtype=torch.uint8, device=device))


def split(x: torch.Tensor, pos: Optional[torch.Tensor] = None, rows: Optional[int] = None) -> Parts:
    """Rows of x [T, K] as parts; with ``pos`` (int32 [T, k]) token t goes to every row pos[t, j] >= 0 of ``rows``, the others stay undefined."""
    T, K = x.shape
    rows = T if rows is None else rows
    out = _new_parts(rows, K, x.device)
    rc = _ext.lib().bg_mx_split(_ext.ptr(x), ctypes.c_longlong(x.stride(0)), _ext.ptr(pos), ctypes.c_int(pos.shape[1] if pos is not None else 0),
                                ctypes.c_int(T), _ext.ptr(out.p), _ext.ptr(out.s), ctypes.c_int(rows), ctypes.c_int(K),
                                _ext.stream())
    _ext.check(rc, "bg_mx_split")
    return out


def gated_parts(gate_up: torch.Tensor, kind: int, limit: float, offsets: Optional[torch.Tensor], row_src: Optional[torch.Tensor]) -> Parts:
    """The gated activation of ``moe.activation`` (kind 0, 1, 2 of its kernel) with its rows as parts."""
    R, I = gate_up.shape[0], gate_up.shape[1] // 2
    out = _new_parts(R, I, gate_up.device)
    rc = _ext.lib().bg_gated_parts(ctypes.c_int(kind), _ext.ptr(gate_up), ctypes.c_longlong(gate_up.stride(0)), _ext.ptr(out.p), _ext.ptr(out.s),
                                   ctypes.c_int(R), ctypes.c_int(I), ctypes.c_float(limit),
                                   _ext.ptr(offsets[-1:] if offsets is not None else None), _ext.ptr(row_src),
                                   ctypes.c_int(_ext.num_sms(gate_up.device)), _ext.stream())
    _ext.check(rc, "bg_gated_parts")
    return out


BLOCK_MAX_ROWS = 80
BLOCK_NARROW_ROWS = 30                # rows of a segment up to which a tile has 32 tokens (gemm_mxfp4_block.cu)


def block_scaled(wq: torch.Tensor, ws: torch.Tensor, rows: float, split: bool = False) -> bool:
    """The block-scaled product takes weights wq [.., N, K / 2], ws [.., N, K / 32] for segments of ``rows`` expected rows: up to 80 of them (128 experts of
    6,144 x 2,880, against weights expanded to bf16: 5 rows 287 / 553 us, 28 rows 369 / 559, 47 rows 449 / 573, 94 rows 643 / 605), K to 12,288, addresses and
    rows as its loads need them.  K below 1,024 from one and a half rounds of tiles on: a tile of few steps is over before its start is paid
    (layers, 16 rows: 16 experts of 512 x 768 55.4 / 53.3, of 2,048 x 768 67.6 / 72.6, 128 of 512 x 768 105.6 / 113.6).  Where the parts take a launch of their own (``split``), K beyond 2,048, and
    beyond 4,096 with tiles of 96 tokens (dense, 24 tokens, 1,024 x 1,024 15.3 / 12.5, 4,096 x 1,024 15.3 / 14.4, 2,048 x 2,048 17.4 / 18.5, 2,880 x 3,072 19.4 / 22.6;
    31 tokens, 2,880 x 3,072 23.6 / 22.5, 4,096 x 4,096 29.5 / 26.7, x 6,144 31.7 / 34.9).  With tiles of 96 tokens K to 10,112, past which shared memory has two
    stages (40 tokens, 4,096 x 9,216 39.9 / 49.2, x 12,288 64.5 / 63.5, 80 tokens 68.6 / 65.5)."""
    K, wide = 2 * wq.shape[-1], rows > BLOCK_NARROW_ROWS
    if rows > BLOCK_MAX_ROWS or (wide and K > 10112):
        return False
    if split and K <= (4096 if wide else 2048):
        return False
    if K < 1024 and 2 * (wq.numel() // (wq.shape[-1] * wq.shape[-2])) * -(-wq.shape[-2] // 128) < 3 * _ext.num_sms(wq.device):
        return False
    return bool(_ext.lib().bg_mxfp4_block_takes(_ext.ptr(wq), _ext.ptr(ws), ctypes.c_longlong(wq.shape[-2]), ctypes.c_int(K)))


def _block_gemm(x: Union[torch.Tensor, Parts], wq2d, ws2d, out, offsets, groups, M, N, K, counts, rows) -> None:
    if isinstance(x, torch.Tensor):
        x = x.contiguous()
        x = split(x if x.data_ptr() % 16 == 0 else x.clone())
    rc = _ext.lib().bg_mxfp4_block_gemm(
        _ext.ptr(x.p), _ext.ptr(x.s), _ext.ptr(wq2d), _ext.ptr(ws2d), _ext.ptr(out), ctypes.c_int(out.stride(0)),
        _ext.ptr(offsets), _ext.ptr(counts), ctypes.c_int(groups), ctypes.c_int(M), ctypes.c_int(N), ctypes.c_int(K), ctypes.c_float(rows),
        ctypes.c_int(_ext.num_sms(out.device)), _ext.ptr(_ext.status_word(out.device)), _ext.stream())
    _ext.check(rc, "bg_mxfp4_block_gemm")


def mxfp4_gemm(x: torch.Tensor, wq: torch.Tensor, ws: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """[T, K] bf16 x MXFP4 [N, K] -> [T, N] bf16."""
    N, K = wq.shape[0], wq.shape[1] * 2
    if not x.is_cuda:
        return (x.float() @ dequantize(wq, ws, torch.float32).t()).to(x.dtype)
    T = x.shape[0]
    if out is None:
        out = torch.empty(T, N, dtype=torch.bfloat16, device=x.device)
    if T:
        if block_scaled(wq, ws, T, split=True):
            _block_gemm(x, wq, ws, out, None, 1, T, N, K, None, T)
        else:
            _launch(EPI_STORE, x.contiguous(), wq, ws, out, None, 1, T, N, K)
    return out


def grouped_mxfp4_gemm(x: Union[torch.Tensor, Parts], wq: torch.Tensor, ws: torch.Tensor, offsets: torch.Tensor,
                       silu_mul: bool = False, out: Optional[torch.Tensor] = None,
                       counts: Optional[torch.Tensor] = None, rows_hint: Optional[float] = None) -> torch.Tensor:
    """Ragged grouped GEMM over rows grouped by expert (segment e = offsets[e]:offsets[e+1]; ``counts``: rows present in
    every segment, the others stay undefined).  wq [E, N, K/2], ws [E, N, K/32].  ``silu_mul``: the rows of each expert
    are stored gate/up interleaved in blocks of 32 and the output is silu(gate) * up with N/2 columns.  ``x``: bf16 rows, or their
    ``Parts`` (without ``silu_mul``); ``rows_hint``: rows that are expected to be present in all."""
    E, N, Kh = wq.shape
    K = Kh * 2
    R = x.shape[0]
    if not x.is_cuda:
        from .gemm import interleave_gate_up_rows
        y = torch.zeros(R, N, dtype=torch.float32)
        off = offsets.tolist()
        w = dequantize(wq, ws, torch.float32)
        for e in range(E):
            a, b = off[e], off[e + 1]
            if b > a:
                y[a:b] = x[a:b].float() @ w[e].t()
        if silu_mul:
            inv = torch.argsort(interleave_gate_up_rows(N))
            y = ref.silu_mul(y[:, inv])
        return y.to(x.dtype)
    n_out = N // 2 if silu_mul else N
    if out is None:
        out = torch.empty(R, n_out, dtype=torch.bfloat16, device=wq.device)
    if R:
        assert offsets.dtype == torch.int32 and offsets.is_cuda
        wq2d, ws2d = wq.view(E * N, Kh), ws.view(E * N, K // 32)
        rows = (R if rows_hint is None else rows_hint) / max(E, 1)
        if isinstance(x, Parts) or not silu_mul and block_scaled(wq, ws, rows, split=True):
            assert not silu_mul
            _block_gemm(x, wq2d, ws2d, out, offsets, E, R, N, K, counts, rows)
        else:
            _launch(EPI_SILU_MUL if silu_mul else EPI_STORE, x.contiguous(), wq2d, ws2d, out, offsets, E, R, N, K, counts)
    return out
