"""Per-head batched GEMM (MLA absorb / out-absorb) and the grouped GEMM's real-row counts, against fp32
references of the same ops."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-9)).item()


@pytest.mark.parametrize("T,H", [(1, 16), (200, 16), (384, 128), (130, 8)])
def test_q_absorb_and_out_absorb(T, H):
    from batchgen_b200.ops import _ext, attention
    g = torch.Generator().manual_seed(T + H)
    nope, rope, lora, v = 128, 64, 512, 128
    q = torch.randn(T, H, nope + rope, generator=g).to(torch.bfloat16).cuda()
    w_uk_t = (torch.randn(H, lora, nope, generator=g) * 0.05).to(torch.bfloat16).cuda()
    w_uv = (torch.randn(H, v, lora, generator=g) * 0.05).to(torch.bfloat16).cuda()
    q_abs = attention.mla_q_absorb(q, w_uk_t, nope)
    _ext.check_status()
    want = torch.einsum("thk,hnk->thn", q[..., :nope].float(), w_uk_t.float())
    assert q_abs.shape == (T, H, lora) and _rel(q_abs, want) < 5e-3
    o_lat = torch.randn(T, H, lora, generator=g).to(torch.bfloat16).cuda()
    out = attention.mla_out_absorb(o_lat, w_uv)
    _ext.check_status()
    want = torch.einsum("thk,hnk->thn", o_lat.float(), w_uv.float()).reshape(T, H * v)
    assert out.shape == (T, H * v) and _rel(out, want) < 5e-3


def test_grouped_gemm_with_real_counts():
    from batchgen_b200.ops import _ext, gemm, ref
    FP8 = torch.float8_e4m3fn
    g = torch.Generator().manual_seed(3)
    E, N, K = 4, 256, 256
    rows = [5, 0, 130, 128]
    starts, cur = [], 0
    for r in rows:
        starts.append(cur)
        cur += (r + 127) // 128 * 128
    offsets = torch.tensor(starts + [cur], dtype=torch.int32)
    x = torch.randn(cur, K, generator=g)
    xq, xs = ref.act_quant(x)
    wq = (torch.randn(E, N, K, generator=g) * 0.1).to(FP8)
    ws = torch.rand(E, N // 128, K // 128, generator=g) + 0.5
    counts = torch.tensor(rows, dtype=torch.int32).cuda()
    sentinel = 768.0
    out = torch.full((cur, N), sentinel, dtype=torch.bfloat16, device="cuda")
    xs_dev = xs.cuda().t().contiguous().t()
    gemm.grouped_fp8_gemm(xq.cuda(), xs_dev, wq.cuda(), ws.cuda(), offsets.cuda(), out=out, counts=counts)
    _ext.check_status()
    want = ref.grouped_fp8_gemm(xq, xs, wq, ws, offsets)
    out = out.cpu().float()
    for e in range(E):
        a, n = starts[e], rows[e]
        if n:
            assert _rel(out[a:a + n], want[a:a + n]) < 1e-2
        pad_end = offsets[e + 1].item()
        assert (out[a + n:pad_end] == sentinel).all(), "padding rows must not be stored"


@pytest.mark.parametrize("H", [4, 16])
def test_expanded_mla_prefill_attention(H):
    """Varlen causal attention over up-projected keys / values, with cached context on one sequence."""
    from batchgen_b200.ops import _ext, attention
    g = torch.Generator().manual_seed(H)
    lens, ctx = [300, 70, 129], [0, 200, 64]                 # new tokens and cached context per sequence
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    k_starts, tk = [], 0
    for n, c in zip(lens, ctx):
        k_starts.append(tk)
        tk += n + c
    Tq = cu[-1]
    q = (torch.randn(Tq, H, 192, generator=g) * 0.5).to(torch.bfloat16)
    kv = (torch.randn(tk, H, 256, generator=g) * 0.5).to(torch.bfloat16)
    lat = (torch.randn(tk, 576, generator=g) * 0.5).to(torch.bfloat16)
    kpe = lat[:, 512:]                                        # strided view, as the model passes it
    work = attention.mha_prefill_work(cu, ctx, k_starts)
    scale = 192 ** -0.5
    got = attention.mha_prefill(q.cuda(), kv.cuda(), lat.cuda()[:, 512:], work, scale).cpu().float()
    _ext.check_status()
    want = attention.mha_prefill(q.float(), kv.float(), kpe.float(), work, scale)
    assert _rel(got, want) < 1.5e-2


@pytest.mark.parametrize("lens,ctx", [([1, 128, 129, 64], [0, 0, 63, 1]), ([256, 257, 65], [64, 500, 0]), ([600], [191])])
def test_expanded_mla_prefill_halves(lens, ctx):
    """Tiles whose second half is missing, a single query or whole; queries whose keys end at, before and behind a key tile."""
    from batchgen_b200.ops import _ext, attention
    H, g = 3, torch.Generator().manual_seed(len(lens))
    cu, k_starts, tk = [0], [], 0
    for n, c in zip(lens, ctx):
        cu.append(cu[-1] + n)
        k_starts.append(tk)
        tk += n + c
    q, kv, kpe = (torch.randn(*shape, generator=g).to(torch.bfloat16) for shape in ((cu[-1], H, 192), (tk, H, 256), (tk, 64)))
    work = attention.mha_prefill_work(cu, ctx, k_starts)
    got = attention.mha_prefill(q.cuda(), kv.cuda(), kpe.cuda(), work, 0.1).cpu().double()
    _ext.check_status()
    for i, (n, c) in enumerate(zip(lens, ctx)):
        a, k0 = cu[i], k_starts[i]
        k = torch.cat([kv[k0:k0 + n + c, :, :128], kpe[k0:k0 + n + c, None].expand(-1, H, -1)], -1).double()
        s = torch.einsum("nhd,lhd->nhl", q[a:a + n].double(), k) * 0.1
        s.masked_fill_((torch.arange(n + c) > torch.arange(n).view(-1, 1) + c).unsqueeze(1), -float("inf"))
        p, v = s.softmax(-1), kv[k0:k0 + n + c, :, 128:].double()
        # probabilities and output rounded to 8 bits, exponents of fp32 sums of 192 products
        bound = torch.einsum("nhl,lhd->nhd", p, v.abs()) * 2.0 ** -7 + 1e-6
        assert ((got[a:a + n] - torch.einsum("nhl,lhd->nhd", p, v)).abs() <= bound).all(), i


def _uneven(n_q, ctx, H, seed):
    """Queries behind ``ctx`` cached keys of which one group of 32 (one warp's rows) scores every tile of 64 keys 2^12 above the tile before, all others flat."""
    g = torch.Generator().manual_seed(seed)
    tk = n_q + ctx
    q, kv, kpe = torch.zeros(n_q, H, 192), torch.zeros(tk, H, 256), torch.zeros(tk, 64)
    steep = torch.arange(n_q) // 32 % 4 == seed % 4
    q[steep, :, 0] = 1.0
    kv[:, :, 0] = (12.0 * (torch.arange(tk) // 64)).view(-1, 1)
    kv[:, :, 128:] = torch.randn(tk, H, 128, generator=g) + 1
    return tuple(v.to(torch.bfloat16) for v in (q, kv, kpe))


def _attention64(q, kv, ctx, scale):
    """Softmax attention of one sequence in 64 bits, and the same of the values' magnitudes."""
    k, v = kv[..., :128].double(), kv[..., 128:].double()
    s = torch.einsum("nhd,lhd->nhl", q[..., :128].double(), k) * scale
    s.masked_fill_((torch.arange(kv.shape[0]) > torch.arange(q.shape[0]).view(-1, 1) + ctx).unsqueeze(1), -float("inf"))
    p = s.softmax(-1)
    return torch.einsum("nhl,lhd->nhd", p, v), torch.einsum("nhl,lhd->nhd", p, v.abs())


@pytest.mark.parametrize("n_q,ctx,seed", [(128, 1000, 0), (65, 640, 1), (100, 1900, 3), (256, 900, 2), (200, 576, 0), (700, 0, 1)])
def test_expanded_mla_prefill_uneven_warps(n_q, ctx, seed):
    """A warp that rescales at every tile beside three that never do: each tile's probabilities are multiplied when all four have stored theirs."""
    from batchgen_b200.ops import _ext, attention
    H, scale = 32, math.log(2.0)                        # scores in powers of two
    q, kv, kpe = _uneven(n_q, ctx, H, seed)
    work = attention.mha_prefill_work([0, n_q], [ctx], [0])
    args = (q.cuda(), kv.cuda(), kpe.cuda(), work, scale)
    got = attention.mha_prefill(*args)
    again = [attention.mha_prefill(*args) for _ in range(4)]
    _ext.check_status()
    assert all(torch.equal(got, a) for a in again)
    want, mag = _attention64(q, kv, ctx, scale)
    # probabilities and output rounded to 8 bits; scores are exact, exponents up to 2^9 are fp32 sums
    assert ((got.cpu().double() - want).abs() <= mag * 2.0 ** -7 + 1e-6).all()


@pytest.mark.parametrize("n_q,ctx,seed", [(1, 64, 0), (40, 200, 0), (128, 1025, 2), (129, 511, 3), (256, 0, 1), (512, 700, 0)])
def test_expanded_mla_prefill_last_tiles(n_q, ctx, seed):
    """Values that are zero but in the last two key tiles: a warp that ends first still waits for both."""
    from batchgen_b200.ops import _ext, attention
    H, scale = 48, math.log(2.0)
    q, kv, kpe = _uneven(n_q, ctx, H, seed)
    last = (n_q + ctx - 1) // 64
    kv[:max(0, (last - 1) * 64), :, 128:] = 0
    work = attention.mha_prefill_work([0, n_q], [ctx], [0])
    args = (q.cuda(), kv.cuda(), kpe.cuda(), work, scale)
    got = attention.mha_prefill(*args)
    again = [attention.mha_prefill(*args) for _ in range(4)]
    _ext.check_status()
    assert all(torch.equal(got, a) for a in again)
    want, mag = _attention64(q, kv, ctx, scale)
    assert ((got.cpu().double() - want).abs() <= mag * 2.0 ** -7 + 1e-6).all()          # as above


@pytest.mark.parametrize("lens,ctx", [([1], [0]), ([128], [70]), ([129], [0]), ([255, 300, 64], [1, 64, 500]), ([1200], [63])])
def test_expanded_mla_prefill_halves_as_ctas(lens, ctx):
    """Few tiles take a CTA for each half of a tile: the bits of the same heads among so many that a CTA has both."""
    from batchgen_b200.ops import _ext, attention
    g = torch.Generator().manual_seed(sum(lens))
    cu, k_starts, tk = [0], [], 0
    for n, c in zip(lens, ctx):
        cu.append(cu[-1] + n)
        k_starts.append(tk)
        tk += n + c
    q, kv, kpe = (torch.randn(*shape, generator=g).to(torch.bfloat16).cuda() for shape in ((cu[-1], 2, 192), (tk, 2, 256), (tk, 64)))
    work = attention.mha_prefill_work(cu, ctx, k_starts)
    sms = _ext.num_sms(q.device)
    assert 2 * work.shape[0] * 2 <= sms
    many = sms // 2 + 1                                  # pairs of heads, all the same: one CTA an item and head
    few = attention.mha_prefill(q, kv, kpe, work, 0.1)
    all_ = attention.mha_prefill(q.repeat(1, many, 1), kv.repeat(1, many, 1), kpe, work, 0.1).view(cu[-1], many, 2, 128)
    _ext.check_status()
    assert (all_ == few.unsqueeze(1)).all()


@pytest.mark.parametrize("scale", [0.0, -0.07, 0.07])
@pytest.mark.parametrize("n_q,ctx", [(70, 0), (300, 40)])
def test_expanded_mla_prefill_any_scale(n_q, ctx, scale):
    """Keys behind a query stay out whatever the scale's sign; a scale of zero is the mean of the values."""
    from batchgen_b200.ops import _ext, attention
    H, g = 2, torch.Generator().manual_seed(n_q)
    q, kv = (torch.randn(n, H, d, generator=g).to(torch.bfloat16) for n, d in ((n_q, 192), (n_q + ctx, 256)))
    q[..., 128:] = 0
    work = attention.mha_prefill_work([0, n_q], [ctx], [0])
    got = attention.mha_prefill(q.cuda(), kv.cuda(), torch.zeros(n_q + ctx, 64, dtype=torch.bfloat16, device="cuda"), work, scale).cpu().double()
    _ext.check_status()
    want, mag = _attention64(q, kv, ctx, scale)
    # probabilities and output rounded to 8 bits, exponents of fp32 sums of 128 products
    assert ((got - want).abs() <= mag * 2.0 ** -7 + 1e-6).all()


def test_model_prefill_uses_expanded_attention_and_matches_cpu():
    from batchgen_b200.config import get_model_config
    from batchgen_b200.models import build_model
    from batchgen_b200.models.transformer import AttnMeta
    from batchgen_b200.runtime.kv_cache import PagedKVCache, build_block_table, slots_for_range
    cfg = get_model_config("tiny-deepseek-v3", hidden_size=1024, q_lora_rank=512, kv_lora_rank=512,
                           qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128, num_heads=16,
                           intermediate_size=2048, moe_intermediate_size=512, n_routed_experts=16,
                           num_experts_per_tok=4, n_group=4, topk_group=2, vocab_size=4096, quant="fp8_block")
    lens = [330, 200]
    ids = torch.randint(2, cfg.vocab_size, (sum(lens),), generator=torch.Generator().manual_seed(5), dtype=torch.int32)

    def run(device, dtype_name, dtype):
        model = build_model(cfg, device, dtype_name, seed=0)
        kv = PagedKVCache(cfg, 16, 64, device, dtype)
        pages = [kv.alloc.alloc((n + 63) // 64) for n in lens]
        pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens]).to(device)
        slots = torch.tensor(sum((slots_for_range(p, 0, n, 64) for p, n in zip(pages, lens)), []), device=device)
        meta = AttnMeta(mode="prefill", positions=pos, slot_mapping=slots, block_table=build_block_table(pages, device),
                        cu_seqlens=[0, lens[0], sum(lens)], ctx_lens=[0, 0])
        return model, model.forward(ids.to(device), meta, kv).float().cpu()

    _, cpu = run("cpu", "fp32", torch.float32)
    model, gpu = run("cuda", "bf16", torch.bfloat16)
    assert model.w.layers[0].w_kvb is not None
    rel = ((gpu - cpu).norm() / cpu.norm()).item()
    assert rel < 0.08, rel


@pytest.mark.parametrize("T,N,K,silu", [(300, 512, 256, False), (128, 256, 128, False), (515, 768, 1024, True), (1, 2112, 7168, False)])
def test_wide_tile_fp8_gemm_matches_reference(T, N, K, silu):
    """128 x 256-tile kernel: same contract as the 128 x 128 one."""
    from batchgen_b200.ops import _ext, gemm, ref
    FP8 = torch.float8_e4m3fn
    g = torch.Generator().manual_seed(T + N)
    x = torch.randn(T, K, generator=g)
    xq, xs = ref.act_quant(x)
    wq = (torch.randn(N, K, generator=g) * 0.1).to(FP8)
    ws = torch.rand((N + 127) // 128, K // 128, generator=g) + 0.5
    want = ref.fp8_gemm(xq, xs, wq, ws)
    wq_dev = wq.cuda()
    if silu:
        perm = gemm.interleave_gate_up_rows(N)
        wq_dev = wq.view(torch.uint8)[perm].contiguous().view(FP8).cuda()
        want = ref.silu_mul(want)
    xs_dev = xs.cuda().t().contiguous().t()
    got = gemm.fp8_gemm(xq.cuda(), xs_dev, wq_dev, ws.cuda(), silu_mul=silu, wide=True).cpu().float()
    narrow = gemm.fp8_gemm(xq.cuda(), xs_dev, wq_dev, ws.cuda(), silu_mul=silu, wide=False).cpu().float()
    _ext.check_status()
    assert _rel(got, want) < 1e-2
    # the narrow kernel may split K over CTAs at these sizes (a different but fixed summation order)
    assert _rel(narrow, want) < 1e-2 and _rel(got, narrow) < 2e-3


@pytest.mark.parametrize("T,N,wide", [(130, 9472, False), (130, 9600, True), (300, 6400, True), (600, 3840, True)])
def test_tile_width_of_a_second_round(T, N, wide):
    """Either side of one round of 128 x 128 tiles (148 SMs): the bytes of the kernel that the rule names."""
    from batchgen_b200.ops import _ext, gemm, ref
    if _ext.num_sms(torch.device("cuda")) != 148:
        pytest.skip("rounds of 148 SMs")
    xq, xs = ref.act_quant(torch.randn(T, 128))
    wq, ws = (torch.randn(N, 128) * 0.1).to(torch.float8_e4m3fn), torch.rand((N + 127) // 128, 1) + 0.5
    a = [v.cuda() for v in (xq, xs, wq, ws)]
    got = gemm.fp8_gemm(*a)
    assert torch.equal(got, gemm.fp8_gemm(*a, wide=wide))
    assert _rel(got.float().cpu(), ref.fp8_gemm(xq, xs, wq, ws)) < 1e-2


@pytest.mark.parametrize("T,N,pad,off", [(40, 300, 0, 0), (130, 300, 3, 1), (40, 264, 8, 4), (257, 129, 0, 0), (1, 301, 0, 3), (40, 256, 0, 0)])
@pytest.mark.parametrize("K", [256, 4096])
def test_narrow_tile_rows_of_any_alignment(T, N, pad, off, K):
    """Rows whose stride or start is no multiple of 16 bytes: the values, and nothing beside them, of every epilogue of the 128 x 128 kernel; split K too."""
    from batchgen_b200.ops import _ext, gemm, ref
    g = torch.Generator().manual_seed(T + N)
    ld = N + pad

    def into(rows, cols, dtype):
        buf = torch.full((rows * ld + off + 8,), 768.0, dtype=dtype, device="cuda")
        return buf, buf[off:off + rows * ld].view(rows, ld)[:, :cols]

    def check(buf, view, want, rel):
        _ext.check_status()
        assert ((view.cpu().double() - want).abs() <= rel).all()
        view.fill_(768.0)
        assert (buf == 768).all()

    x, w = torch.randn(T, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) * 0.1).bfloat16()
    want, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t() * K * 2.0 ** -24
    buf, out = into(T, N, torch.bfloat16)
    gemm._launch(gemm.KIND_BF16, gemm.EPI_STORE, x.cuda(), None, 0, w.cuda(), None, out, None, 1, T, N, K)
    check(buf, out, want, want.abs() * 2.0 ** -8 + mag)
    if ld % 4 == 0:
        buf, out = into(T, N, torch.float32)
        gemm.bf16_gemm(x.cuda(), w.cuda(), out=out, fp32_out=True)
        check(buf, out, want, mag + want.abs() * 2.0 ** -23)
    xq, xs = ref.act_quant(torch.randn(T, K, generator=g))
    wq, ws = (torch.randn(N, K, generator=g) * 0.1).to(torch.float8_e4m3fn), torch.rand((N + 127) // 128, K // 128, generator=g) + 0.5
    buf, out = into(T, N, torch.bfloat16)
    gemm.fp8_gemm(xq.cuda(), xs.cuda(), wq.cuda(), ws.cuda(), out=out, wide=False)
    want = ref.fp8_gemm(xq, xs, wq, ws).double()
    _ext.check_status()
    assert _rel(out.cpu(), want) < 1e-2
    if N % 256 == 0:
        out.fill_(768.0)
        half = out[:, :N // 2]
        perm = gemm.interleave_gate_up_rows(N)
        gemm.fp8_gemm(xq.cuda(), xs.cuda(), wq.view(torch.uint8)[perm].contiguous().view(torch.float8_e4m3fn).cuda(), ws.cuda(), out=half, silu_mul=True, wide=False)
        assert _rel(half.cpu(), ref.silu_mul(want.float())) < 1e-2 and (out[:, N // 2:] == 768).all()


def test_tile_width_rule(monkeypatch):
    """Either side of each border of the rule itself: one round of narrow tiles for dense products, two for grouped ones, row strides, operands, hooks."""
    from batchgen_b200.ops import _ext, gemm
    monkeypatch.setattr(_ext, "num_sms", lambda device=None: 148)
    monkeypatch.setattr(gemm, "_WIDE", "auto")
    D = torch.empty(2, 16, dtype=torch.bfloat16, device="cuda")
    odd = torch.empty(2, 12, dtype=torch.bfloat16, device="cuda")
    use = lambda M, N, dense=True, D=D, kind=gemm.KIND_FP8, wide=None: gemm._use_wide(kind, D, M, N, wide, dense)  # noqa: E731
    assert not use(128, 148 * 128) and use(128, 149 * 128) and use(129, 75 * 128) and not use(129, 74 * 128)
    assert not use(128, 295 * 128, dense=False) and use(128, 296 * 128, dense=False)
    assert not use(128, 200 * 128, D=odd) and use(128, 296 * 128, D=odd)
    assert not use(128, 400 * 128, kind=gemm.KIND_BF16) and not use(128, 400 * 128, wide=False) and use(1, 128, wide=True)
    gemm.hooks_pending()
    assert not use(128, 400 * 128) and use(128, 400 * 128)


@pytest.mark.parametrize("T,N,pad,silu", [(129, 320, 0, False), (131, 320, 8, False), (126, 256, 24, False), (3, 264, 8, False), (131, 256, 0, True), (129, 512, 8, True)])
def test_wide_tile_stores(T, N, pad, silu):
    """Row groups cut by the last row, column slices cut by N, rows that start inside a sector: the same values, nothing beside them."""
    from batchgen_b200.ops import gemm, ref
    g = torch.Generator().manual_seed(T + N)
    xq, xs = ref.act_quant(torch.randn(T, 256, generator=g))
    wq = (torch.randn(N, 256, generator=g) * 0.1).to(torch.float8_e4m3fn)
    ws = torch.rand((N + 127) // 128, 2, generator=g) + 0.5
    want = ref.fp8_gemm(xq, xs, wq, ws)
    if silu:
        want = ref.silu_mul(want)
        wq = wq.view(torch.uint8)[gemm.interleave_gate_up_rows(N)].contiguous().view(torch.float8_e4m3fn)
    n = want.shape[1]
    buf = torch.full((T + 4, n + pad), 768.0, dtype=torch.bfloat16, device="cuda")
    gemm.fp8_gemm(xq.cuda(), xs.cuda().t().contiguous().t(), wq.cuda(), ws.cuda(), out=buf[:T, pad:], silu_mul=silu, wide=True)
    assert _rel(buf[:T, pad:].float().cpu(), want) < 1e-2              # as above: bf16 results of the same sums
    assert (buf[T:] == 768).all() and (buf[:, :pad] == 768).all()


def test_wide_tile_grouped_gemm_with_counts():
    from batchgen_b200.ops import _ext, gemm, ref
    FP8 = torch.float8_e4m3fn
    g = torch.Generator().manual_seed(11)
    E, N, K = 3, 512, 256
    rows = [130, 0, 7]
    starts, cur = [], 0
    for r in rows:
        starts.append(cur)
        cur += (r + 127) // 128 * 128
    offsets = torch.tensor(starts + [cur], dtype=torch.int32)
    xq, xs = ref.act_quant(torch.randn(cur, K, generator=g))
    wq = (torch.randn(E, N, K, generator=g) * 0.1).to(FP8)
    ws = torch.rand(E, N // 128, K // 128, generator=g) + 0.5
    out = torch.full((cur, N), 768.0, dtype=torch.bfloat16, device="cuda")
    gemm.grouped_fp8_gemm(xq.cuda(), xs.cuda().t().contiguous().t(), wq.cuda(), ws.cuda(), offsets.cuda(), out=out,
                          counts=torch.tensor(rows, dtype=torch.int32).cuda(), wide=True)
    _ext.check_status()
    want = ref.grouped_fp8_gemm(xq, xs, wq, ws, offsets)
    out = out.cpu().float()
    for e in range(E):
        a, n = starts[e], rows[e]
        if n:
            assert _rel(out[a:a + n], want[a:a + n]) < 1e-2
        assert (out[a + n:offsets[e + 1].item()] == 768.0).all()


def test_router_logits_fp32_epilogue():
    from batchgen_b200.ops import _ext, moe
    g = torch.Generator().manual_seed(9)
    x = torch.randn(300, 1024, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(256, 1024, generator=g) * 0.05).cuda()
    got = moe.router_logits(x, w)
    _ext.check_status()
    assert got.dtype == torch.float32 and got.shape == (300, 256)
    want = x.float() @ w.to(torch.bfloat16).float().t()
    assert _rel(got, want) < 1e-4
    # batch invariance: a row's logits do not depend on which other rows are in the batch
    assert torch.equal(moe.router_logits(x[:7].contiguous(), w), got[:7])
