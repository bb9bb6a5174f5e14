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


_P, _I = ctypes.c_void_p, ctypes.c_int
# argument types are set once, so that plain integers pass: three of these calls a layer are host time of a decode step of few rows
_ARGS = {
    "bg_mx_split": (_P, ctypes.c_longlong, _P, _I, _I, _P, _P, _I, _I, _P),
    "bg_gated_parts": (_I, _P, ctypes.c_longlong, _P, _P, _I, _I, ctypes.c_float, _P, _P, _I, _P),
    "bg_mxfp4_block_gemm": (_P, _P, _P, _P, _P, _I, _P, _P, _I, _I, _I, _I, ctypes.c_float, _I, _P, _P),
}


def _call(name: str, *args) -> None:
    fn = getattr(_ext.lib(), name)
    if fn.argtypes is None:
        fn.argtypes = _ARGS[name]
    _ext.check(fn(*args, _ext.stream()), name)


def _at(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


class Parts:
    """bf16 rows [rows, K] as the block-scaled product takes them: ``p`` uint8 [rows / 8 rounded up, 2, 8, K] (e4m3, eight rows' first parts and
    then their second parts), ``s`` uint8 [K / 128 rounded up, rows, 4] (e8m0 of the first part, one per 32 elements; the second part's is five
    less), in one allocation."""
    __slots__ = ("shape", "data")

    def __init__(self, rows: int, K: int, device):
        self.shape = (rows, K)
        self.data = torch.empty(self._scales_at() + -(-K // 128) * rows * 4, dtype=torch.uint8, device=device)

    def _scales_at(self) -> int:
        rows, K = self.shape
        return -(-rows // 8) * 16 * K

    @property
    def p(self) -> torch.Tensor:
        return self.data[:self._scales_at()].view(-1, 2, 8, self.shape[1])

    @property
    def s(self) -> torch.Tensor:
        return self.data[self._scales_at():].view(-1, self.shape[0], 4)

    @property
    def is_cuda(self) -> bool:
        return self.data.is_cuda

    def pointers(self):
        at = self.data.data_ptr()
        return at, at + self._scales_at()


def split(x: torch.Tensor, pos: Optional[torch.Tensor] = None, rows: Optional[int] = None) -> Parts:
    """Rows of x [T, K] as parts; with ``pos`` (int32 [T, k]) token t goes to every row pos[t, j] >= 0 of ``rows``, the others stay undefined."""
    T, K = x.shape
    rows = T if rows is None else rows
    out = Parts(rows, K, x.device)
    _call("bg_mx_split", x.data_ptr(), x.stride(0), _at(pos), pos.shape[1] if pos is not None else 0, T, *out.pointers(), rows, K)
    return out


def gated_parts(gate_up: torch.Tensor, kind: int, limit: float, offsets: Optional[torch.Tensor], row_src: Optional[torch.Tensor]) -> Parts:
    """The gated activation of ``moe.activation`` (kind 0, 1, 2 of its kernel) with its rows as parts."""
    R, I = gate_up.shape[0], gate_up.shape[1] // 2
    out = Parts(R, I, gate_up.device)
    _call("bg_gated_parts", kind, gate_up.data_ptr(), gate_up.stride(0), *out.pointers(), R, I, limit,
          offsets.data_ptr() + 4 * (offsets.numel() - 1) if offsets is not None else None, _at(row_src), _ext.num_sms(gate_up.device))
    return out


BLOCK_MAX_ROWS = 80
BLOCK_NARROW_ROWS = 30                # rows of a segment up to which a tile has 32 tokens (gemm_mxfp4_block.cu)


def block_scaled(wq: torch.Tensor, ws: torch.Tensor, rows: float, split: bool = False) -> bool:
    """The block-scaled product takes weights wq [.., N, K / 2], ws [.., N, K / 32] for segments of ``rows`` expected rows: up to 80 of them (128 experts of
    6,144 x 2,880, against weights expanded to bf16: 5 rows 287 / 553 us, 28 rows 369 / 559, 47 rows 449 / 573, 94 rows 643 / 605), K to 12,288, addresses and
    rows as its loads need them.  K below 1,024 from one and a half rounds of tiles on: a tile of few steps is over before its start is paid
    (layers, 16 rows: 16 experts of 512 x 768 55.4 / 53.3, of 2,048 x 768 67.6 / 72.6, 128 of 512 x 768 105.6 / 113.6).  Where the parts take a launch of their own
    (``split``), K beyond 2,048, and beyond 4,096 with tiles of 96 tokens (dense, 24 tokens, 1,024 x 1,024 15.3 / 12.5, 4,096 x 1,024 15.3 / 14.4, 2,048 x 2,048 17.4 / 18.5, 2,880 x 3,072 19.4 / 22.6;
    31 tokens, 2,880 x 3,072 23.6 / 22.5, 4,096 x 4,096 29.5 / 26.7, x 6,144 31.7 / 34.9).  With tiles of 96 tokens K to 10,112, past which shared memory has two
    stages (40 tokens, 4,096 x 9,216 39.9 / 49.2, x 12,288 64.5 / 63.5, 80 tokens 68.6 / 65.5)."""
    N, Kh = wq.shape[-2:]
    K, wide = 2 * Kh, rows > BLOCK_NARROW_ROWS
    if rows > BLOCK_MAX_ROWS or (wide and K > 10112):
        return False
    if split and K <= (4096 if wide else 2048):
        return False
    if K < 1024 and 2 * (wq.numel() // (N * Kh)) * -(-N // 128) < 3 * _ext.num_sms(wq.device):
        return False
    # as bg_mxfp4_block_takes has it
    return 128 <= K <= 12288 and K % 64 == 0 and N * (K // 32) % 16 == 0 and wq.data_ptr() % 32 == 0 and ws.data_ptr() % 16 == 0


def _block_gemm(x: Union[torch.Tensor, Parts], wq, ws, out, offsets, groups, M, N, K, counts, rows) -> None:
    if isinstance(x, torch.Tensor):
        x = x.contiguous()
        x = split(x if x.data_ptr() % 16 == 0 else x.clone())
    _call("bg_mxfp4_block_gemm", *x.pointers(), wq.data_ptr(), ws.data_ptr(), out.data_ptr(), out.stride(0), _at(offsets), _at(counts), groups, M, N, K, rows,
          _ext.num_sms(out.device), _ext.status_word(out.device).data_ptr())


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
        if not (wq.is_contiguous() and ws.is_contiguous()):          # the kernels take addresses
            wq, ws = wq.view(E * N, Kh), ws.view(E * N, K // 32)
        rows = (R if rows_hint is None else rows_hint) / max(E, 1)
        if isinstance(x, Parts) or not silu_mul and block_scaled(wq, ws, rows, split=True):
            assert not silu_mul
            _block_gemm(x, wq, ws, out, offsets, E, R, N, K, counts, rows)
        else:
            _launch(EPI_SILU_MUL if silu_mul else EPI_STORE, x.contiguous(), wq, ws, out, offsets, E, R, N, K, counts)
    return out
