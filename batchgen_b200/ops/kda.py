"""Kimi Delta Attention (KDA): gated delta-rule linear attention with a width-4 causal depthwise convolution
on q, k, v, L2-normalised q / k, a per-channel decay gate and a sigmoid-gated RMSNorm on the output.

``kda_forward`` serves prefill (packed sequences, optional continuation from a stored state) and decode (one
token per sequence) alike.  On CUDA it launches ``csrc/kda.cu``: token by token, or for longer pieces in chunks of 64 tokens; on CPU (and as the oracle of the tests) it
runs the recurrence in fp32.  State lives in two pools indexed by a sequence's state slot:

    conv_state [slots, 3 * H * D, 3] fp32   the last three raw inputs of each q / k / v channel, oldest first
    rec_state  [slots, H, D, D]      fp32   S[key, value]

Reference parity: batchgen/models/moonshotai/kimi_linear/serving_modules.py:579-722 (projections and the
fused decode contract), :1074 (prefill), :1202 (decode); attention/kda_fused_decode.cu:147.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import List, Optional, Sequence

import torch
import torch.nn.functional as F

from . import _ext


@dataclass
class KDAParams:
    conv_w: torch.Tensor            # [3 * H * D, 4] fp32 (tap 3 multiplies the current token)
    conv_b: Optional[torch.Tensor]  # [3 * H * D] fp32 or None
    A_log: torch.Tensor             # [H] fp32
    dt_bias: torch.Tensor           # [H * D] fp32
    norm_w: torch.Tensor            # [D] fp32


def causal_conv1d_ref(x: torch.Tensor, w: torch.Tensor, b: Optional[torch.Tensor], window: torch.Tensor):
    """x [n, C] one sequence, w [C, 4], window [C, 3] (previous raw inputs, oldest first) ->
    (silu(conv) [n, C], new window [C, 3]).  fp32."""
    full = torch.cat([window.t().float(), x.float()], 0)               # [n + 3, C]
    n = x.shape[0]
    y = sum(full[i:i + n] * w[:, i].float() for i in range(4))
    if b is not None:
        y = y + b.float()
    return F.silu(y), full[-3:].t().contiguous()


def kda_gate(f: torch.Tensor, A_log: torch.Tensor, dt_bias: torch.Tensor, H: int, D: int) -> torch.Tensor:
    """Log decay per token, head and key channel: -exp(A_log[h]) * softplus(f + dt_bias)  (<= 0)."""
    return -A_log.float().exp().view(1, H, 1) * F.softplus(f.float().view(-1, H, D) + dt_bias.float().view(1, H, D))


def kda_recurrent_ref(q, k, v, g, beta, S, scale: float):
    """One sequence, fp32.  q, k, v, g [n, H, D]; beta [n, H] (after sigmoid); S [H, D, D] updated in place.
    Returns o [n, H, D]."""
    n = q.shape[0]
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * scale
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    out = torch.empty_like(v)
    for t in range(n):
        S.mul_(g[t].exp().unsqueeze(-1))
        u = beta[t].unsqueeze(-1) * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S.add_(k[t].unsqueeze(-1) * u.unsqueeze(-2))
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out


def kda_chunk_ref(q, k, v, g, beta, S, scale: float, chunk: int = 64):
    """The same recurrence in chunk form (the shape a tensor-core prefill kernel takes): inside a chunk the
    writes u_i = beta_i (v_i - S_(i-1)'^T k_i) solve a unit lower-triangular system, after which outputs and the
    state at the chunk end are plain matrix products.  With G the running sum of the log decay inside the chunk,

        M[i, j]  = sum_c k_i[c] k_j[c] exp(G_i[c] - G_j[c])          (j < i)
        (I + diag(beta) M) U = diag(beta) (V - (K * exp(G)) S_0)
        O        = (Q * exp(G)) S_0 + tril(Q-to-K decayed products) U
        S_end    = exp(G_last) * S_0 + sum_j (k_j * exp(G_last - G_j)) u_j^T

    q, k, v, g [n, H, D]; beta [n, H] (after sigmoid); S [H, D, D] updated in place; returns o [n, H, D].  fp32."""
    n, H, D = q.shape
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * scale
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    out = torch.empty_like(v)
    for a in range(0, n, chunk):
        b = min(n, a + chunk)
        C = b - a
        qc, kc, vc, bc = (t[a:b].transpose(0, 1) for t in (q, k, v, beta.unsqueeze(-1)))     # [H, C, D] / [H, C, 1]
        G = g[a:b].transpose(0, 1).cumsum(1)                                               # [H, C, D]
        # decayed pair products; the exponent is <= 0 wherever it is used (j <= i)
        diff = (G.unsqueeze(2) - G.unsqueeze(1)).clamp_max(0.0).exp()                       # [H, i, j, D]
        kk = torch.einsum("hid,hjd,hijd->hij", kc, kc, diff)
        qk = torch.einsum("hid,hjd,hijd->hij", qc, kc, diff)
        eye = torch.eye(C, dtype=q.dtype, device=q.device)
        A = eye + bc * torch.tril(kk, -1)
        rhs = bc * (vc - torch.einsum("hcd,hdv->hcv", kc * G.exp(), S))
        U = torch.linalg.solve_triangular(A, rhs, upper=False)
        out[a:b] = (torch.einsum("hcd,hdv->hcv", qc * G.exp(), S) + torch.tril(qk) @ U).transpose(0, 1)
        last = G[:, -1:, :]                                                                 # [H, 1, D]
        S.mul_(last.squeeze(1).exp().unsqueeze(-1))
        S.add_(torch.einsum("hcd,hcv->hdv", kc * (last - G).exp(), U))
    return out


CHUNK = 64
CHUNK_MIN_TOKENS = 48                 # shorter pieces never go through the chunk form
_CHUNK_FLOATS = (9 * CHUNK // 2 + 2 * CHUNK + 1) * 128   # scratch of a (chunk, head): nine bf16 and two fp32 [64, 128] results, decays
_CHUNK_SCRATCH = 1 << 30              # bytes of scratch a round of chunks may take


def chunk_form_pays(lens: Sequence[int], heads: int, sms: int) -> bool:
    """Whether pieces of ``lens`` tokens go through chunks.  Token by token a CTA serves a (piece, head): 1.6 to 2.0 us a token of the longest piece with a
    CTA on an SM, 2.42 with two, and 2.42 a token of every further round of two CTAs an SM.  For chunks the line counts 90 us to start, 0.52 us a (chunk,
    head) and 0.25 us a (piece, head) for its state, on 148 SMs, which is what they cost with their chain on CUDA cores.  They are faster now, and win
    nearly everywhere: us, chunks / tokens, 32 heads 1 x 64 73 / 137, 4 x 48 83 / 107, 16 x 128 423 / 628, 4 x 512 413 / 1,030, 8 x 300 521 / 737, 8 x 1,024
    1,519 / 2,460, 64 x 64 861 / 1,100, 64 x 128 1,574 / 2,166, 64 x 512 5,994 / 8,547, 1 x 4,096 929 / 8,100; 8 heads 16 x 128 138 / 266, 64 x 512 1,521 / 2,457; 64 heads 4 x
    48 142 / 129, 8 x 300 974 / 1,446.  So the line sends to the tokens what chunks would serve up to 1.5 times as fast (of these points 32 heads 4 x 48, 8 x 300, 16 x
    128, 64 x 64, 64 x 128 and 64 x 512): it lies where both took the same time with the older chain."""
    if not lens:
        return False
    pairs, longest, total = heads * len(lens), max(lens), sum(lens)
    if pairs <= sms:
        tokens = (1.6 + 0.4 * pairs / sms) * longest
    elif pairs <= 2 * sms:
        tokens = 2.42 * longest
    else:
        tokens = 2.42 * max(longest, heads * total / (2 * sms) + 0.3 * total / len(lens))
    return 90 + (0.52 * heads * sum(-(-n // CHUNK) for n in lens) + 0.25 * pairs) * 148 / sms < 30 + tokens


def chunk_scratch_bytes(tokens: int, heads: int, dim: int) -> int:
    """Most scratch that ``kda_forward`` takes for a step of ``tokens`` tokens: a record per (chunk, head) of a round of chunks."""
    if dim != 128:
        return 0
    chunks = -(-tokens // CHUNK) + tokens // CHUNK_MIN_TOKENS        # every piece may end in a part of a chunk
    most = max(1, _CHUNK_SCRATCH // (4 * _CHUNK_FLOATS * heads))      # of a round
    return min(chunks, most) * heads * _CHUNK_FLOATS * 4


def chunk_plan(cu: Sequence[int], min_tokens: int, most_items: int):
    """Rounds of chunks of the pieces of at least ``min_tokens``: a list of (items, seqs) with items (sequence, first token, tokens,
    tokens of the piece before it) and seqs (sequence, first item, items, 1 at the start of a piece), at most ``most_items`` items a
    round, a sequence's chunks in order.  Longer pieces first: their chains take longest."""
    order = sorted((i for i in range(len(cu) - 1) if cu[i + 1] - cu[i] >= max(min_tokens, 1)), key=lambda i: cu[i] - cu[i + 1])
    rounds, items, seqs = [], [], []
    for i in order:
        a, b = int(cu[i]), int(cu[i + 1])
        t = a
        while t < b:
            if len(items) == most_items:
                rounds.append((items, seqs))
                items, seqs = [], []
            n = min(most_items - len(items), -(-(b - t) // CHUNK))
            seqs.append((i, len(items), n, int(t == a)))
            for _ in range(n):
                items.append((i, t, min(CHUNK, b - t), t - a))
                t = min(t + CHUNK, b)
    if items:
        rounds.append((items, seqs))
    return rounds


@dataclass
class StepPlan:
    """What ``kda_forward`` needs of a prompt step's lengths on the device: the same for every layer of the step."""
    cu: torch.Tensor                       # [nseq + 1] int32
    rounds: list                           # of chunks: (items, sequence pieces) in ``tables``
    tables: Optional[torch.Tensor]         # [.., 4] int32, round after round: items, then pieces
    short: int                             # tokens of the longest piece that goes token by token


def step_plan(cu_seqlens: Sequence[int], heads: int, dim: int, device) -> StepPlan:
    cu = [int(c) for c in cu_seqlens]
    lens = [b - a for a, b in zip(cu, cu[1:])]
    rounds, tables, short = [], None, (1 << 31) - 1
    if dim == 128 and chunk_form_pays([n for n in lens if n >= CHUNK_MIN_TOKENS], heads, _ext.num_sms(device)):
        made = chunk_plan(cu, CHUNK_MIN_TOKENS, max(1, _CHUNK_SCRATCH // (4 * _CHUNK_FLOATS * heads)))
        rounds = [(len(it), len(sq)) for it, sq in made]
        tables = torch.tensor([r for it, sq in made for r in it + sq], dtype=torch.int32, device=device)
        short = CHUNK_MIN_TOKENS - 1 if any(0 < n < CHUNK_MIN_TOKENS for n in lens) else 0
    return StepPlan(torch.tensor(cu, dtype=torch.int32, device=device), rounds, tables, short)


def _forward_ref(qkv, f, beta, z, p: KDAParams, conv_state, rec_state, slots, cu, has_initial, H, D, scale, eps):
    T = qkv.shape[0]
    HD = H * D
    out = torch.zeros(T, HD, dtype=torch.float32, device=qkv.device)
    for i, slot in enumerate(slots):
        if slot < 0:
            continue
        a, b = cu[i], cu[i + 1]
        if b <= a:
            continue
        if has_initial is not None and not has_initial[i]:
            conv_state[slot].zero_()
            rec_state[slot].zero_()
        y, win = causal_conv1d_ref(qkv[a:b, : 3 * HD], p.conv_w, p.conv_b, conv_state[slot])
        conv_state[slot].copy_(win)
        qh, kh, vh = (y[:, s * HD:(s + 1) * HD].view(-1, H, D) for s in range(3))
        g = kda_gate(f[a:b], p.A_log, p.dt_bias, H, D)
        S = rec_state[slot].float()
        step = kda_chunk_ref if (b - a) > 128 else kda_recurrent_ref           # long prompts: chunk form
        o = step(qh, kh, vh, g, torch.sigmoid(beta[a:b].float()), S, scale)
        rec_state[slot].copy_(S)
        o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + eps) * p.norm_w.float()
        out[a:b] = (o * torch.sigmoid(z[a:b].float().view(-1, H, D))).reshape(-1, HD)
    return out.to(qkv.dtype)


def kda_forward(qkv: torch.Tensor, f: torch.Tensor, beta: torch.Tensor, z: torch.Tensor, p: KDAParams,
                conv_state: torch.Tensor, rec_state: torch.Tensor, slots, cu_seqlens: Optional[Sequence[int]],
                has_initial: Optional[Sequence[int]], H: int, D: int, scale: float, eps: float,
                plan: Optional[StepPlan] = None) -> torch.Tensor:
    """qkv [T, >= 3HD] (raw q | k | v, may be a column view), f / z [T, HD], beta [T, >= H] (views allowed; unit
    column stride).  ``slots``: int32 tensor (or list) [nseq], < 0 skips; ``cu_seqlens`` None = one token per
    sequence; ``has_initial`` None = continue from the stored state; ``plan``: ``step_plan`` of these lengths and heads, made here
    when None (CUDA: a blocking copy of its tables).  Returns [T, HD] in qkv's dtype and
    updates both pools."""
    nseq = len(slots)
    if not qkv.is_cuda or qkv.dtype != torch.bfloat16:
        sl = slots.tolist() if isinstance(slots, torch.Tensor) else list(slots)
        cu = list(range(nseq + 1)) if cu_seqlens is None else list(cu_seqlens)
        return _forward_ref(qkv, f, beta, z, p, conv_state, rec_state, sl, cu, has_initial, H, D, scale, eps)
    dev = qkv.device
    for t in (qkv, f, beta, z):
        assert t.stride(1) == 1
    if not isinstance(slots, torch.Tensor):
        slots = torch.tensor(list(slots), dtype=torch.int32, device=dev)
    hi_t = None if has_initial is None else (
        has_initial if isinstance(has_initial, torch.Tensor) else torch.tensor([int(x) for x in has_initial], dtype=torch.int32, device=dev))
    out = torch.empty(qkv.shape[0], H * D, dtype=torch.bfloat16, device=dev)
    if isinstance(cu_seqlens, torch.Tensor):
        plan = StepPlan(cu_seqlens, [], None, (1 << 31) - 1)
    elif cu_seqlens is not None and plan is None:
        plan = step_plan(cu_seqlens, H, D, dev)
    rounds, short = (plan.rounds, plan.short) if plan is not None and cu_seqlens is not None else ([], (1 << 31) - 1)
    if z.stride(0) % 4 or z.data_ptr() % 8 or rec_state.data_ptr() % 16:      # the chunk form reads four gates, and four numbers of a state, at a time
        rounds, short = [], (1 << 31) - 1
    cu_t = plan.cu if cu_seqlens is not None else None
    assert cu_t is None or cu_t.shape[0] == nseq + 1
    tables, scratch = (plan.tables, torch.empty(max(n for n, _ in rounds) * H * _CHUNK_FLOATS, dtype=torch.float32, device=dev)) if rounds else (None, None)
    at = 0
    for n, (items, pieces) in enumerate(rounds or [(0, 0)]):
        last = n == max(len(rounds), 1) - 1
        rc = _ext.lib().bg_kda_forward(
            _ext.ptr(qkv), ctypes.c_int(qkv.stride(0)), _ext.ptr(f), ctypes.c_int(f.stride(0)), _ext.ptr(beta),
            ctypes.c_int(beta.stride(0)), _ext.ptr(z), ctypes.c_int(z.stride(0)), _ext.ptr(p.conv_w), _ext.ptr(p.conv_b),
            _ext.ptr(p.A_log), _ext.ptr(p.dt_bias), _ext.ptr(p.norm_w), _ext.ptr(conv_state), _ext.ptr(rec_state),
            _ext.ptr(cu_t), _ext.ptr(slots), _ext.ptr(hi_t), _ext.ptr(out), ctypes.c_int(nseq), ctypes.c_int(H),
            ctypes.c_int(D), ctypes.c_float(scale), ctypes.c_float(eps), _ext.ptr(tables[at:] if items else None), ctypes.c_int(items),
            _ext.ptr(tables[at + items:] if items else None), ctypes.c_int(pieces), ctypes.c_int(short if last else 0),
            _ext.ptr(scratch if items else None), _ext.ptr(_ext.status_word(dev)), _ext.stream())
        _ext.check(rc, "bg_kda_forward", kernels=(3 if items else 0) + int(last and short > 0))
        at += items + pieces
    return out
