"""Performance cases: steps of the served model families at their real widths and a few layers deep.

A case is one step of a model, as the engine runs it: a prompt micro-batch through ``model.forward`` or a decode step
through the captured graph of ``DecodeGraphRunner`` (grouped-query models decode through ``model.forward``).  Weights
come through the checkpoint ``loader`` of ``build_model``; they are made from the seed, already on the grid of the format
they are served in (block FP8, MXFP4, bf16), so that loading loses nothing.  Embeddings carry a component along the router rows of each token's experts: like a trained
router, this one has a clear opinion about every token, and rounding noise does not change which experts run.

``exact`` computes the same step in 64 bits from the same weights with torch alone.
"""
import hashlib
import math

import torch
import torch.nn.functional as F

from batchgen_b200.config import get_model_config
from batchgen_b200.models import build_model
from batchgen_b200.models.transformer import AttnMeta
from batchgen_b200.runtime.graphs import DecodeGraphRunner
from batchgen_b200.runtime.kv_cache import PagedKVCache
from batchgen_b200.runtime.sequence import Sequence

PAGE = 64
DEVICE = "cuda:0"

# Layers and vocabulary are cut so that three models fit the card; every width is the preset's own.
MODELS = {
    # MLA, block-FP8 projections and experts (256, groups), one dense and one mixture layer
    "deepseek": ("deepseek-v3-671b", dict(num_layers=2, first_k_dense=1)),
    # grouped-query attention of 64-wide heads with sinks, one layer with a window and one without, MXFP4 experts (128; their
    # 2,880 columns are padded to the 3,072 that the 4-bit kernels tile)
    "gpt-oss": ("gpt-oss-120b", dict(num_layers=2, moe_intermediate_size=3072)),
    # grouped-query attention of 128-wide heads, block-FP8 everywhere
    "minimax": ("minimax-m2.5", dict(num_layers=2)),
    # three linear-attention (KDA) layers and one MLA layer, one dense and three mixture layers in bf16
    "kimi-linear": ("kimi-linear-48b", dict(num_layers=4, kda_layers=(0, 1, 2))),
}
VOCAB = 16384


def _config(case):
    preset, cut = MODELS[case["model"]]
    return get_model_config(preset, vocab_size=VOCAB, **cut)


def listed():
    return [
        # a few interactive rows: launches and latency count
        dict(name="deepseek-decode-4", model="deepseek", step="decode", rows=4, longest=1000, cached=0),
        # the batch decode step of the flagship
        dict(name="deepseek-decode-256", model="deepseek", step="decode", rows=256, longest=4096, cached=0),
        # short prompts: one small micro-batch
        dict(name="deepseek-prefill-short", model="deepseek", step="prefill", rows=3, longest=301, cached=0),
        # a full prompt micro-batch of ragged prompts
        dict(name="deepseek-prefill-4x2k", model="deepseek", step="prefill", rows=4, longest=2048, cached=0),
        # a later piece of a long prompt, or a turn on a reused prefix: attention over cached rows
        dict(name="deepseek-prefill-piece", model="deepseek", step="prefill", rows=1, longest=1536, cached=5000),
        # one interactive row
        dict(name="gpt-oss-decode-1", model="gpt-oss", step="decode", rows=1, longest=900, cached=0),
        # a batch decode step
        dict(name="gpt-oss-decode-160", model="gpt-oss", step="decode", rows=160, longest=4096, cached=0),
        # ragged prompts
        dict(name="gpt-oss-prefill-3x2k", model="gpt-oss", step="prefill", rows=3, longest=2047, cached=0),
        # ragged prompts behind a shared, cached system prompt
        dict(name="minimax-prefill-2x1k", model="minimax", step="prefill", rows=2, longest=1100, cached=333),
        # a batch decode step: recurrent states, one layer of cached latents
        dict(name="kimi-linear-decode-128", model="kimi-linear", step="decode", rows=128, longest=2048, cached=0),
        # one long prompt: little parallelism in the recurrence
        dict(name="kimi-linear-prefill-1x4k", model="kimi-linear", step="prefill", rows=1, longest=4096, cached=0),
        # many ragged prompts
        dict(name="kimi-linear-prefill-8x1k", model="kimi-linear", step="prefill", rows=8, longest=1024, cached=0),
    ]


def draw(rng):
    model = rng.choice(sorted(MODELS))
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if rng.random() < 0.4:
        rows = log(1, 256)
        return dict(model=model, step="decode", rows=rows, longest=log(64, 4096), cached=0)
    tokens = log(200, 6000 if model in ("deepseek", "kimi-linear") else 4096)
    rows = min(log(1, 16), max(1, tokens // 64))
    longest = min(max(64, tokens // rows), 4096)
    # a recurrent model continues from its state, not from cached rows: its pieces start at the front here
    cached = 0 if model == "kimi-linear" or rng.random() < 0.6 else log(64, 4096)
    return dict(model=model, step="prefill", rows=rows, longest=longest, cached=cached)


def _lengths(case):
    """Tokens of every sequence: the longest first, the others between a quarter of it and all of it."""
    n, top = case["rows"], case["longest"]
    return [top] + [max(1, int(top * (0.25 + 0.75 * ((i * 0.6180339887) % 1.0)))) for i in range(1, n)]


def _contexts(case):
    """Tokens cached before the step, per sequence."""
    lens = _lengths(case)
    if case["step"] == "decode":
        return [n - 1 for n in lens]
    return [max(0, case["cached"] - 37 * i) for i in range(len(lens))]


def _new(case):
    return [1] * case["rows"] if case["step"] == "decode" else _lengths(case)


# ------------------------------------------------------------------ weights
def _generator(seed, name):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int.from_bytes(hashlib.sha256(("%d:%s" % (seed, name)).encode()).digest()[:7], "little"))
    return g


class Weights:
    """The checkpoint: tensors by name, fp32, on the card."""

    def __init__(self, cfg, seed):
        self.cfg, self.seed = cfg, seed
        self.gates = {}

    def _fp8(self, name, shape, std):
        """Values of the block-FP8 grid: every 128 x 128 block has a power of two as its scale."""
        x = torch.randn(shape, device=DEVICE, generator=_generator(self.seed, name)).mul_(112).clamp_(-448, 448)
        x = x.to(torch.float8_e4m3fn).float()
        x[::128, ::128] = 448.0
        return x.mul_(2.0 ** round(math.log2(std / 112)))

    def _fp4(self, name, shape, std):
        """Values of the MXFP4 grid: every group of 32 has the largest value in it."""
        x = torch.randn(shape, device=DEVICE, generator=_generator(self.seed, name)).mul_(2)
        edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=DEVICE)
        grid = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], device=DEVICE)
        x = grid[torch.bucketize(x.abs(), edges)].mul_(x.sign())
        x[:, ::32] = 6.0
        x[1::2, ::32] = -6.0
        return x.mul_(2.0 ** round(math.log2(std / 2)))

    def gate(self, layer):
        """Router rows [experts, width]."""
        if layer not in self.gates:
            cfg = self.cfg
            shape = (cfg.n_routed_experts, cfg.hidden_size)
            g = _generator(self.seed, "gate%d" % layer)
            self.gates[layer] = (torch.randn(shape, device=DEVICE, generator=g) * 0.3 / cfg.hidden_size ** 0.5).bfloat16().float()
        return self.gates[layer]

    def _experts_of_tokens(self, layer):
        """[vocabulary, k]: the experts that a token leans to, two from a group where routing is limited to groups."""
        cfg = self.cfg
        g = _generator(self.seed, "experts%d" % layer)
        V, E, k, G = cfg.vocab_size, cfg.n_routed_experts, cfg.num_experts_per_tok, max(1, cfg.n_group)
        if G == 1:
            return torch.rand(V, E, device=DEVICE, generator=g).topk(k, -1)[1]
        per = k // cfg.topk_group
        groups = torch.rand(V, G, device=DEVICE, generator=g).topk(cfg.topk_group, -1)[1]
        inside = torch.rand(V, cfg.topk_group, E // G, device=DEVICE, generator=g).topk(per, -1)[1]
        return (groups.unsqueeze(-1) * (E // G) + inside).reshape(V, k)

    def _embed(self, shape):
        cfg = self.cfg
        g = _generator(self.seed, "embed")
        e = torch.randn(shape, device=DEVICE, generator=g)
        for l in range(cfg.num_layers):
            if cfg.is_moe_layer(l):
                rows = F.normalize(self.gate(l), dim=-1)
                idx = self._experts_of_tokens(l)
                alpha = torch.empty(idx.shape, device=DEVICE).uniform_(8, 12, generator=g)
                for j in range(idx.shape[1]):
                    e += alpha[:, j:j + 1] * rows[idx[:, j]]
        return e

    def __call__(self, name, shape):
        cfg, last = self.cfg, name.split(".")[-2] if name.endswith(".weight") else name.split(".")[-1]
        g = _generator(self.seed, name)
        randn = lambda: torch.randn(shape, device=DEVICE, generator=g)  # noqa: E731
        rand = lambda: torch.rand(shape, device=DEVICE, generator=g)  # noqa: E731
        if last == "embed_tokens":
            return self._embed(shape).bfloat16().float()
        if last == "gate":
            return self.gate(int(name.split(".")[2]))
        if last == "e_score_correction_bias":
            return randn() * 0.01
        if last == "A_log":
            return (1 + 15 * rand()).log()
        if last == "dt_bias":
            return torch.expm1(torch.exp(math.log(1e-3) + rand() * math.log(100.0))).log()
        if last.endswith("conv1d"):
            return randn() * 0.4
        if last == "sinks":
            return randn()
        if len(shape) == 1:
            return (1 + 0.1 * randn()).bfloat16().float()
        std = (0.4 if last in ("o_proj", "down_proj") else 1.0) / shape[1] ** 0.5
        if cfg.quant == "fp8_block" and last not in ("lm_head", "kv_b_proj"):
            return self._fp8(name, shape, std)
        if cfg.quant == "mxfp4" and ".experts." in name:
            return self._fp4(name, shape, std)
        return (randn() * std).bfloat16().float()


# ------------------------------------------------------------------ inputs
def _inputs(case, cfg, seed):
    """Token ids, and the pages of every sequence in a shuffled pool."""
    new, ctx = _new(case), _contexts(case)
    g = torch.Generator().manual_seed(seed)
    ids = torch.randint(2, cfg.vocab_size, (sum(new),), generator=g)
    need = [-(-(c + n) // PAGE) for c, n in zip(ctx, new)]
    order = torch.randperm(sum(need), generator=g).tolist()
    pages = []
    for n in need:
        pages.append(order[:n])
        order = order[n:]
    return ids, pages


def _cache(case, cfg, seed, num_pages):
    """Paged rows [layers, pages, PAGE, row] as earlier steps leave them, and the recurrent states of decode rows."""
    layers = sum(1 for l in range(cfg.num_layers) if not cfg.layer_is_kda(l))
    shape = (layers, num_pages, PAGE, cfg.kv_cache_dim)
    if not any(_contexts(case)):
        return torch.zeros(shape, device=DEVICE, dtype=torch.bfloat16)
    return torch.randn(shape, device=DEVICE, generator=_generator(seed, "rows"), dtype=torch.bfloat16)


def _states(case, cfg, seed):
    """Recurrent states and convolution windows of the KDA layers, one slot a sequence."""
    n, H, D, B = len(cfg.kda_layers), cfg.kda_num_heads, cfg.kda_head_dim, case["rows"]
    rec = torch.randn(n, B, H, D, D, device=DEVICE, generator=_generator(seed, "rec")) * 0.1
    conv = torch.randn(n, B, 3 * H * D, 3, device=DEVICE, generator=_generator(seed, "conv")).bfloat16().float()
    return rec, conv


def prepare(case, seed):
    cfg = _config(case)
    model = build_model(cfg, device=DEVICE, dtype="bf16", loader=Weights(cfg, seed))
    ids, pages = _inputs(case, cfg, seed)
    new, ctx = _new(case), _contexts(case)
    B = len(new)
    total = sum(len(p) for p in pages)
    kv = PagedKVCache(cfg, total, PAGE, DEVICE, torch.bfloat16, state_slots=B if cfg.has_kda else 0)
    kv.kv.copy_(_cache(case, cfg, seed, total))
    state = dict(model=model, kv=kv, step=case["step"])
    if case["step"] == "decode" and cfg.is_mla:
        if cfg.has_kda:
            rec, conv = _states(case, cfg, seed)
            kv.state.rec.copy_(rec)
            kv.state.conv.copy_(conv)
        rows = []
        for i, p in enumerate(pages):
            s = Sequence(i, [])
            s.gpu_pages, s.state_slot = p, i if cfg.has_kda else -1
            rows.append(s)
        runner = DecodeGraphRunner(model, kv, max_batch=B, max_pages_per_seq=max(len(p) for p in pages), num_buckets=1)
        runner.capture_all()
        slots = [p[c // PAGE] * PAGE + c % PAGE for p, c in zip(pages, ctx)]
        state.update(runner=runner, rows=rows, ids=ids.tolist(), pos=ctx, slots=slots, lens=[c + 1 for c in ctx])
        return state
    table = torch.zeros(B, max(len(p) for p in pages), dtype=torch.int32)
    pos, slots, cu = [], [], [0]
    for i, p in enumerate(pages):
        table[i, :len(p)] = torch.tensor(p)
        t = torch.arange(ctx[i], ctx[i] + new[i])
        pos.append(t)
        slots.append(torch.tensor(p)[t // PAGE] * PAGE + t % PAGE)
        cu.append(cu[-1] + new[i])
    state.update(ids=ids.int().to(DEVICE), pos=torch.cat(pos).int().to(DEVICE), slots=torch.cat(slots).to(DEVICE),
                 table=table.to(DEVICE), cu=cu, ctx=ctx, last=torch.tensor([c - 1 for c in cu[1:]], device=DEVICE))
    if case["step"] == "decode":
        state.update(lens=torch.tensor([c + 1 for c in ctx], dtype=torch.int32, device=DEVICE))
    elif cfg.has_kda:
        state.update(state_slots=torch.arange(B, dtype=torch.int32, device=DEVICE),
                     fresh=torch.zeros(B, dtype=torch.int32, device=DEVICE))
    return state


def run(state):
    model, kv = state["model"], state["kv"]
    if "runner" in state:
        logits, _ = state["runner"].decode(None, state["rows"], state["ids"], state["pos"], state["slots"], state["lens"])
    elif state["step"] == "decode":
        meta = AttnMeta(mode="decode", positions=state["pos"], slot_mapping=state["slots"], block_table=state["table"],
                        seqlens=state["lens"])
        logits = model.forward(state["ids"], meta, kv)
    else:
        meta = AttnMeta(mode="prefill", positions=state["pos"], slot_mapping=state["slots"], block_table=state["table"],
                        cu_seqlens=state["cu"], ctx_lens=state["ctx"], logit_rows=state["last"],
                        state_slots=state.get("state_slots"), state_has_initial=state.get("fresh"))
        logits = model.forward(state["ids"], meta, kv)
    out = dict(logits=logits, rows=kv.kv)
    if kv.state is not None:
        out.update(rec=kv.state.rec, conv=kv.state.conv)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    cfg = _config(case)
    new, ctx = _new(case), _contexts(case)
    T, B, H = sum(new), len(new), cfg.hidden_size
    pairs = sum(n * c + n * (n + 1) / 2 for n, c in zip(new, ctx))
    bits = {"fp8_block": 1.0, "none": 2.0, "mxfp4": 2.0}[cfg.quant]
    expert_bits = {"fp8_block": 1.0, "none": 2.0, "mxfp4": 0.5 + 1 / 32}[cfg.quant]
    by = fl = 0.0
    for l in range(cfg.num_layers):
        if cfg.layer_is_kda(l):
            n, D = cfg.kda_num_heads, cfg.kda_head_dim
            p = H * (5 * n * D + n + cfg.kda_rank) + cfg.kda_rank * n * D
            state = B * n * (D * D + 9 * D) * 4
            by += p * bits + state * (2 if case["step"] == "decode" else 1)
            fl += 2 * T * p + T * n * D * D * 8
        elif cfg.is_mla:
            n, qk, r = cfg.num_heads, cfg.qk_head_dim, cfg.kv_lora_rank
            kvb = n * (cfg.qk_nope_head_dim + cfg.v_head_dim) * r
            p = H * (cfg.q_lora_rank + r + cfg.qk_rope_head_dim) + cfg.q_lora_rank * n * qk + n * cfg.v_head_dim * H
            by += p * bits + kvb * 2 + (sum(ctx) + T) * cfg.kv_cache_dim * 2
            fl += 2 * T * (p + kvb)
            # decode stays in latent space; prompts pay for per-head keys and values
            fl += 2 * n * pairs * ((2 * r + cfg.qk_rope_head_dim) if case["step"] == "decode" else (qk + cfg.v_head_dim))
        else:
            n, D = cfg.num_heads, cfg.head_dim
            w = cfg.sliding_window if l % 2 == 0 else 0
            seen = pairs
            held = sum(ctx)
            if w:
                seen = sum(sum(min(w, c + i + 1) for i in range(k)) for k, c in zip(new, ctx))
                held = sum(min(w, c) for c in ctx)
            p = H * D * (n + 2 * cfg.num_kv_heads) + n * D * H
            by += p * bits + (held + T) * cfg.kv_cache_dim * 2
            fl += 2 * T * p + 4 * n * D * seen
        if cfg.is_moe_layer(l):
            E, k, I = cfg.n_routed_experts, cfg.num_experts_per_tok, cfg.moe_intermediate_size
            hit = E * (1 - (1 - k / E) ** T)
            shared = 3 * H * I * cfg.n_shared_experts
            by += hit * 3 * H * I * expert_bits + shared * bits + E * H * 2
            fl += 2 * T * (3 * H * I * k + shared + E * H)
        else:
            by += 3 * H * cfg.intermediate_size * bits
            fl += 6 * T * H * cfg.intermediate_size
    by += T * H * 2 + VOCAB * H * 2 + B * VOCAB * 4
    fl += 2 * B * H * VOCAB
    return dict(bytes=by, flops=fl)


def tolerance(case):
    """About four times the distance from ``exact`` in bf16; with FP8 activations that would be more than 0.1, and rounding
    that falls the other way in a few places stays within this."""
    fp8 = _config(case).quant == "fp8_block"
    return dict(rel=0.03 if fp8 else 0.02, max=0.6 if fp8 else 0.3)


# ------------------------------------------------------------------ the same step in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _turns(cfg, dim, pos):
    inv = 1.0 / (cfg.rope_theta ** (torch.arange(0, dim, 2, dtype=torch.float64, device=DEVICE) / dim))
    if cfg.rope_scaling_factor > 1.0:      # YaRN
        at = lambda turns: dim * math.log(cfg.rope_original_max_pos / (turns * 2 * math.pi)) / (2 * math.log(cfg.rope_theta))  # noqa: E731
        low, high = max(math.floor(at(cfg.rope_beta_fast)), 0), min(math.ceil(at(cfg.rope_beta_slow)), dim - 1)
        keep = 1 - ((torch.arange(dim // 2, dtype=torch.float64, device=DEVICE) - low) / (high - low)).clamp(0, 1)
        inv = inv / cfg.rope_scaling_factor * (1 - keep) + inv * keep
    a = pos.double().unsqueeze(-1) * inv
    return a.cos(), a.sin()


def _rotate(x, turns, interleaved):
    """x [T, heads, dim]."""
    cos, sin = (t.unsqueeze(1) for t in turns)
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, start, scale, window=0, sinks=None):
    """One sequence: q [n, h, d]; k [L, g, d], v [L, g, e]; query i stands at position start + i."""
    n, h, L, g = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    at = torch.arange(n, device=DEVICE).unsqueeze(1) + start
    key = torch.arange(L, device=DEVICE).unsqueeze(0)
    hidden = key > at
    if window:
        hidden = hidden | (key <= at - window)
    out = torch.empty(n, h, v.shape[-1], dtype=torch.float64, device=DEVICE)
    step = max(1, int(4e8 // (n * L)))
    for a in range(0, h, step):
        heads = torch.arange(a, min(h, a + step), device=DEVICE)
        of = heads // (h // g)
        s = torch.einsum("nhd,lhd->hnl", q[:, heads], k[:, of]) * scale
        s.masked_fill_(hidden, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sinks is not None:
            top = torch.maximum(top, sinks.double()[heads].view(-1, 1, 1))
        s = (s - top).exp_()
        z = s.sum(-1, keepdim=True)
        if sinks is not None:
            z = z + (sinks.double()[heads].view(-1, 1, 1) - top).exp()
        out[:, heads] = torch.einsum("hnl,lhe->nhe", s / z, v[:, of])
    return out


def exact(case, seed):
    cfg = _config(case)
    W = Weights(cfg, seed)
    ids, pages = _inputs(case, cfg, seed)
    ids = ids.to(DEVICE)
    new, ctx = _new(case), _contexts(case)
    decode = case["step"] == "decode"
    rows = _cache(case, cfg, seed, sum(len(p) for p in pages)).double()
    rec = conv = None
    if cfg.has_kda:
        rec, conv = (t.double() for t in _states(case, cfg, seed))
        if not decode:
            rec.zero_()
            conv.zero_()
    H, eps = cfg.hidden_size, cfg.rms_eps
    cu = [0]
    for n in new:
        cu.append(cu[-1] + n)
    pos = torch.cat([torch.arange(c, c + n, device=DEVICE) for c, n in zip(ctx, new)])
    where = [torch.tensor(p, device=DEVICE) for p in pages]
    flat = [p[torch.arange(c + n, device=DEVICE) // PAGE] * PAGE + torch.arange(c + n, device=DEVICE) % PAGE
            for p, c, n in zip(where, ctx, new)]
    lin = lambda x, name, *shape: x @ W(name + ".weight", shape).double().t()  # noqa: E731

    def mlp(x, name, width):
        return lin(F.silu(lin(x, name + ".gate_proj", width, H)) * lin(x, name + ".up_proj", width, H), name + ".down_proj", H, width)

    def mla(x, p, at):
        n, r, rd, nope, vd = cfg.num_heads, cfg.kv_lora_rank, cfg.qk_rope_head_dim, cfg.qk_nope_head_dim, cfg.v_head_dim
        q_a = lin(x, p + "q_a_proj", cfg.q_lora_rank, H)
        kv = lin(x, p + "kv_a_proj_with_mqa", r + rd, H)
        turns = _turns(cfg, rd, pos)
        store = rows[at].view(-1, r + rd)
        c = _norm(kv[:, :r], W(p + "kv_a_layernorm.weight", (r,)), eps)
        k_pe = _rotate(kv[:, None, r:], turns, cfg.rope_interleaved)[:, 0]
        q = lin(_norm(q_a, W(p + "q_a_layernorm.weight", (cfg.q_lora_rank,)), eps), p + "q_b_proj", n * cfg.qk_head_dim, cfg.q_lora_rank)
        q = q.view(-1, n, nope + rd)
        q = torch.cat([q[..., :nope], _rotate(q[..., nope:], turns, cfg.rope_interleaved)], -1)
        w = W(p + "kv_b_proj.weight", (n * (nope + vd), r)).double().view(n, nope + vd, r)
        o = torch.empty(x.shape[0], n, vd, dtype=torch.float64, device=DEVICE)
        for i in range(len(new)):
            a, b = cu[i], cu[i + 1]
            store[flat[i][ctx[i]:]] = torch.cat([c[a:b], k_pe[a:b]], -1)
            past = store[flat[i]]
            if decode:                     # in latent space
                qa = torch.einsum("nhd,hdr->nhr", q[a:b, :, :nope], w[:, :nope])
                lat = _attend(torch.cat([qa, q[a:b, :, nope:]], -1), past[:, None], past[:, None, :r], ctx[i], cfg.softmax_scale)
                o[a:b] = torch.einsum("nhr,hvr->nhv", lat, w[:, nope:])
            else:
                for h0 in range(0, n, 32):
                    h1 = min(n, h0 + 32)
                    up = torch.einsum("lr,hdr->lhd", past[:, :r], w[h0:h1])
                    k = torch.cat([up[..., :nope], past[:, None, r:].expand(-1, h1 - h0, -1)], -1)
                    o[a:b, h0:h1] = _attend(q[a:b, h0:h1], k, up[..., nope:], ctx[i], cfg.softmax_scale)
        return lin(o.flatten(1), p + "o_proj", H, n * vd)

    def gqa(x, p, at, layer):
        n, g, D = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
        turns = _turns(cfg, D, pos)
        q = _rotate(lin(x, p + "q_proj", n * D, H).view(-1, n, D), turns, cfg.rope_interleaved)
        k = _rotate(lin(x, p + "k_proj", g * D, H).view(-1, g, D), turns, cfg.rope_interleaved)
        v = lin(x, p + "v_proj", g * D, H)
        sinks = W(p + "sinks", (n,)) if cfg.attention_sinks else None
        window = cfg.sliding_window if layer % 2 == 0 else 0
        store = rows[at].view(-1, 2 * g * D)
        o = torch.empty(x.shape[0], n, D, dtype=torch.float64, device=DEVICE)
        for i in range(len(new)):
            a, b = cu[i], cu[i + 1]
            store[flat[i][ctx[i]:]] = torch.cat([k[a:b].flatten(1), v[a:b]], -1)
            past = store[flat[i]]
            o[a:b] = _attend(q[a:b], past[:, :g * D].view(-1, g, D), past[:, g * D:].view(-1, g, D), ctx[i],
                             cfg.softmax_scale, window, sinks)
        return lin(o.flatten(1), p + "o_proj", H, n * D)

    def kda(x, p, at):
        n, D = cfg.kda_num_heads, cfg.kda_head_dim
        raw = torch.cat([lin(x, p + m + "_proj", n * D, H) for m in "qkv"], -1)
        taps = torch.cat([W(p + m + "_conv1d.weight", (n * D, 4)) for m in "qkv"], 0).double()
        z = lin(x, p + "g_proj", n * D, H).view(-1, n, D)
        f = lin(lin(x, p + "f_a_proj", cfg.kda_rank, H), p + "f_b_proj", n * D, cfg.kda_rank)
        beta = lin(x, p + "b_proj", n, H).sigmoid()
        rate = F.softplus(f + W(p + "dt_bias", (n * D,)).double()).view(-1, n, D)
        decay = (-W(p + "A_log", (n,)).double().exp().view(1, n, 1) * rate).exp()
        o = torch.empty(x.shape[0], n, D, dtype=torch.float64, device=DEVICE)
        y = torch.empty_like(raw)
        for i in range(len(new)):
            a, b = cu[i], cu[i + 1]
            full = torch.cat([conv[at, i].t(), raw[a:b]], 0)
            y[a:b] = F.silu(sum(full[j:j + b - a] * taps[:, j] for j in range(4)))
            conv[at, i] = full[-3:].t()
        q, k, v = (t.view(-1, n, D) for t in y.chunk(3, -1))
        q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5
        k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        first = torch.tensor(cu[:-1], device=DEVICE)
        S = rec[at]
        for t in range(max(new)):          # all sequences that still have a token, side by side
            live = torch.tensor([i for i in range(len(new)) if new[i] > t], device=DEVICE)
            r = first[live] + t
            s = S[live] * decay[r].unsqueeze(-1)
            u = beta[r].unsqueeze(-1) * (v[r] - torch.einsum("bhkv,bhk->bhv", s, k[r]))
            s += k[r].unsqueeze(-1) * u.unsqueeze(-2)
            S[live] = s
            o[r] = torch.einsum("bhkv,bhk->bhv", s, q[r])
        o = _norm(o, W(p + "o_norm.weight", (D,)), eps) * z.sigmoid()
        return lin(o.flatten(1), p + "o_proj", H, n * D)

    def moe(x, p, layer):
        E, k, I = cfg.n_routed_experts, cfg.num_experts_per_tok, cfg.moe_intermediate_size
        logits = x @ W.gate(layer).double().t()
        if cfg.scoring_func == "softmax":
            val, idx = logits.topk(k, -1)
            w = val.softmax(-1)
        else:
            score = logits.sigmoid()
            choice = score + W(p + "gate.e_score_correction_bias", (E,)).double()
            if cfg.n_group > 1:
                by_group = choice.view(-1, cfg.n_group, E // cfg.n_group)
                keep = by_group.topk(2, -1)[0].sum(-1).topk(cfg.topk_group, -1)[1]
                allowed = torch.zeros_like(by_group[..., 0]).scatter_(1, keep, 1.0).bool()
                choice = by_group.masked_fill(~allowed.unsqueeze(-1), -math.inf).view(-1, E)
            idx = choice.topk(k, -1)[1]
            w = score.gather(1, idx)
            w = w / w.sum(-1, keepdim=True)
        w = w * cfg.routed_scaling_factor
        y = torch.zeros_like(x)
        for e in range(E):
            t, j = (idx == e).nonzero(as_tuple=True)
            if not t.numel():
                continue
            name = p + "experts.%d" % e
            if cfg.activation == "swiglu_clamped":
                gate = lin(x[t], name + ".gate_proj", I, H).clamp(max=7.0)
                up = lin(x[t], name + ".up_proj", I, H).clamp(-7.0, 7.0)
                part = lin((up + 1) * gate * (1.702 * gate).sigmoid(), name + ".down_proj", H, I)
            else:
                part = mlp(x[t], name, I)
            y.index_add_(0, t, part * w[t, j].unsqueeze(-1))
        if cfg.n_shared_experts:
            y += mlp(x, p + "shared_experts", I * cfg.n_shared_experts)
        return y

    h = W("model.embed_tokens.weight", (VOCAB, H)).double()[ids]
    paged = 0
    for l in range(cfg.num_layers):
        p = "model.layers.%d." % l
        x = _norm(h, W(p + "input_layernorm.weight", (H,)), eps)
        if cfg.layer_is_kda(l):
            h = h + kda(x, p + "self_attn.", cfg.kda_layers.index(l))
        else:
            h = h + (mla(x, p + "self_attn.", paged) if cfg.is_mla else gqa(x, p + "self_attn.", paged, l))
            paged += 1
        x = _norm(h, W(p + "post_attention_layernorm.weight", (H,)), eps)
        h = h + (moe(x, p + "mlp.", l) if cfg.is_moe_layer(l) else mlp(x, p + "mlp", cfg.intermediate_size))
    h = _norm(h[torch.tensor([c - 1 for c in cu[1:]], device=DEVICE)], W("model.norm.weight", (H,)), eps)
    out = dict(logits=lin(h, "lm_head", VOCAB, H), rows=rows)
    if cfg.has_kda:
        out.update(rec=rec, conv=conv)
    return out
