"""Paged GQA decode kernel (sinks, sliding window, split KV) against the fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,D", [(64, 8, 64), (48, 8, 128), (8, 8, 64)])
@pytest.mark.parametrize("window,use_sinks,splits", [(0, False, 1), (128, True, 1), (0, True, 3), (100, False, 2)])
def test_gqa_decode(Hq, Hkv, D, window, use_sinks, splits):
    from batchgen_b200.ops import _ext, attention, ref
    g = torch.Generator().manual_seed(Hq + D + window)
    page, lens = 64, [1, 63, 64, 65, 300, 517]
    B = len(lens)
    npg = [(n + page - 1) // page for n in lens]
    cache = (torch.randn(sum(npg) + 2, page, 2 * Hkv * D, generator=g) * 0.7).to(torch.bfloat16)
    bt = torch.zeros(B, max(npg), dtype=torch.int32)
    nxt = 1
    for b, n in enumerate(npg):
        bt[b, :n] = torch.arange(nxt, nxt + n)
        nxt += n
    q = torch.randn(B, Hq, D, generator=g).to(torch.bfloat16)
    sinks = torch.randn(Hq, generator=g) if use_sinks else None
    sl = torch.tensor(lens, dtype=torch.int32)
    scale = D ** -0.5
    got = attention.gqa_decode(q.cuda(), cache.cuda(), bt.cuda(), sl.cuda(), Hkv, scale, window=window,
                               sinks=sinks.cuda() if use_sinks else None, num_splits=splits).cpu().float()
    _ext.check_status()
    want = attention.gqa_decode(q.float(), cache.float(), bt, sl, Hkv, scale, window=window, sinks=sinks)
    err = ((got - want).norm() / want.norm()).item()
    assert err < 1.5e-2, err


@pytest.mark.parametrize("Hq,Hkv,D,page,interleaved,bias", [(16, 2, 64, 64, False, False), (6, 6, 128, 16, True, True),
                                                             (24, 2, 128, 128, False, True), (5, 1, 64, 32, True, False)])
@pytest.mark.parametrize("window,use_sinks", [(0, False), (0, True), (100, True), (1, False), (64, False)])
def test_gqa_prompt(Hq, Hkv, D, page, interleaved, bias, window, use_sinks):
    """Projections to attention output: lengths at the edges of tiles and pages, cached context, rows without a slot, stale rows of
    the last page that are not finite.  Operands are the bf16 numbers the kernels see, so what is left is the fp32
    sums and the rounding of the output (8 significant bits: up to 2^-8 of a value)."""
    from batchgen_b200.ops import _ext, attention, ref, talking
    g = torch.Generator().manual_seed(Hq * D + page + window)
    lens, ctx = [1, 63, 64, 65, 127, 128, 129, 300, 2], [0, 0, 64, 1, 0, 33, 500, 7, 1000]
    n, T = len(lens), sum(lens)
    need = [-(-(a + b) // page) for a, b in zip(lens, ctx)]
    order = torch.randperm(sum(need), generator=g).tolist()
    cache = torch.full((sum(need), page, 2 * Hkv * D), float("nan"), dtype=torch.bfloat16)
    bt = torch.zeros(n, max(need) + 1, dtype=torch.int32)
    pos, slots, old = [], [], []
    for i in range(n):
        bt[i, :need[i]] = torch.tensor([order.pop() for _ in range(need[i])], dtype=torch.int32)
        p = torch.arange(ctx[i] + lens[i])
        where = bt[i].long()[p // page] * page + p % page
        past = torch.randn(ctx[i], 2 * Hkv * D, generator=g).bfloat16()
        cache.view(-1, 2 * Hkv * D)[where[:ctx[i]]] = past
        old.append(past)
        pos.append(p[ctx[i]:])
        slots.append(where[ctx[i]:])
    pos, slots = torch.cat(pos).int(), torch.cat(slots)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, generator=g).bfloat16()
    b = torch.randn(qkv.shape[1], generator=g).bfloat16() if bias else None
    inv = ref.rope_inv_freq(D, 10000.0)
    ang = torch.arange(2048, dtype=torch.float32).unsqueeze(1) * inv
    cos, sin = ang.cos(), ang.sin()
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    # what the heads kernel makes of the projections
    x = qkv.double() + (b.double() if bias else 0)
    turn = lambda t: ref.apply_rope(t.float(), cos[pos.long()], sin[pos.long()], interleaved)  # noqa: E731
    want_q = turn(x[:, :Hq * D].view(T, Hq, D))
    want_kv = torch.cat([turn(x[:, Hq * D:(Hq + Hkv) * D].view(T, Hkv, D)).reshape(T, -1), x[:, (Hq + Hkv) * D:].float()], 1)
    dev, dc = qkv.cuda(), cache.cuda()
    skip = slots.clone()
    skip[0] = -1                                              # the only row of the first sequence: its key is written by hand below
    attention.gqa_heads(dev, b.cuda() if bias else None, pos.cuda(), cos.cuda(), sin.cuda(), skip.cuda(), dc, Hq, Hkv, D, interleaved)
    got_q, flat = dev[:, :Hq * D].cpu().view(T, Hq, D), dc.view(-1, 2 * Hkv * D)
    assert not torch.isfinite(flat[slots[0].item()].float()).any()
    flat[slots[0].item()] = want_kv[0].bfloat16().cuda()
    got_kv = flat[slots.cuda()].cpu()
    assert (got_q.float() - want_q).abs().max() <= want_q.abs().max() * 2 ** -8
    assert (got_kv.float() - want_kv).abs().max() <= want_kv.abs().max() * 2 ** -8
    work = torch.tensor(talking.prefill_work(cu, ctx, 0, 1, window), dtype=torch.int32).cuda()
    out = torch.full((T, Hq * D), 7.0, dtype=torch.bfloat16, device="cuda")
    sinks = torch.randn(Hq, generator=g) if use_sinks else None
    attention.gqa_prefill(dev[:, :Hq * D].unflatten(1, (Hq, D)), dc, bt.cuda(), work, Hkv, D ** -0.5, out, window=window,
                          sinks=sinks.cuda() if use_sinks else None)
    torch.cuda.synchronize()
    _ext.check_status()
    for i in range(n):
        a, e = cu[i], cu[i + 1]
        rows = torch.cat([old[i], got_kv[a:e]]).double()
        k, v = (t.view(-1, Hkv, D).repeat_interleave(Hq // Hkv, 1) for t in rows.split(Hkv * D, 1))
        s = torch.einsum("nhd,lhd->hnl", got_q[a:e].double(), k) * D ** -0.5
        at, key = pos[a:e].long().unsqueeze(1), torch.arange(rows.shape[0]).unsqueeze(0)
        s = s.masked_fill((key > at) | ((key <= at - window) if window else torch.zeros_like(key > at)), float("-inf"))
        if use_sinks:
            s = torch.cat([s, sinks.double().view(Hq, 1, 1).expand(Hq, s.shape[1], 1)], -1)
        o = torch.einsum("hnl,lhd->nhd", s.softmax(-1)[..., :rows.shape[0]], v).reshape(e - a, -1)
        err = (out[a:e].cpu().double() - o).abs()
        # a value rounded to 8 significant bits: 2^-8 of it; fp32 sums of up to 1,000 terms (1,000 * 2^-24 = 6e-5): 7e-5
        assert (err <= o.abs() * 2 ** -8 + 7e-5 * v.abs().max()).all(), (i, err.max())


@pytest.mark.parametrize("Hq,Hkv,D,page", [(16, 1, 64, 64), (12, 4, 128, 16), (24, 2, 128, 128), (7, 7, 64, 32)])
@pytest.mark.parametrize("window,use_sinks,splits", [(0, False, 1), (0, True, 0), (33, True, 2), (1, False, 3), (700, False, 5)])
def test_gqa_decode_fine(Hq, Hkv, D, page, window, use_sinks, splits):
    """Rows of every length class, one without keys, queries in columns of a wider tensor, stale rows that are not finite."""
    from batchgen_b200.ops import _ext, attention
    g = torch.Generator().manual_seed(Hq + page + splits)
    lens = [1, 15, 16, 17, 0, 64, 65, 700, 1023]
    B = len(lens)
    need = [-(-n // page) for n in lens]
    order = torch.randperm(sum(need), generator=g).tolist()
    cache = torch.full((sum(need), page, 2 * Hkv * D), float("nan"), dtype=torch.bfloat16)
    bt = torch.zeros(B, max(need), dtype=torch.int32)
    rows = []
    for i, n in enumerate(lens):
        bt[i, :need[i]] = torch.tensor([order.pop() for _ in range(need[i])], dtype=torch.int32)
        p = torch.arange(n)
        rows.append(torch.randn(n, 2 * Hkv * D, generator=g).bfloat16())
        cache.view(-1, 2 * Hkv * D)[bt[i].long()[p // page] * page + p % page] = rows[-1]
    wide = torch.randn(B, (Hq + 2) * D, generator=g).bfloat16()
    sinks = torch.randn(Hq, generator=g) if use_sinks else None
    got = attention.gqa_decode(wide.cuda()[:, :Hq * D].unflatten(1, (Hq, D)), cache.cuda(), bt.cuda(), torch.tensor(lens, dtype=torch.int32).cuda(),
                               Hkv, D ** -0.5, window=window, sinks=sinks.cuda() if use_sinks else None, num_splits=splits).cpu().double()
    _ext.check_status()
    for i, n in enumerate(lens):
        if n == 0:
            assert (got[i] == 0).all()
            continue
        r = rows[i][max(0, n - window) if window else 0:].double()
        k, v = (t.view(-1, Hkv, D).repeat_interleave(Hq // Hkv, 1) for t in r.split(Hkv * D, 1))
        s = torch.einsum("hd,lhd->hl", wide[i, :Hq * D].view(Hq, D).double(), k) * D ** -0.5
        if use_sinks:
            s = torch.cat([s, sinks.double().view(Hq, 1)], -1)
        o = torch.einsum("hl,lhd->hd", s.softmax(-1)[:, :r.shape[0]], v)
        # a value rounded to 8 significant bits: 2^-8 of it; fp32 sums of up to 1,023 terms (1,023 * 2^-24 = 6e-5): 7e-5
        assert ((got[i] - o).abs() <= o.abs() * 2 ** -8 + 7e-5 * v.abs().max()).all(), i


@pytest.mark.parametrize("new,ctx", [(1, 899), (1, 3000), (700, 0), (300, 900)])
@pytest.mark.parametrize("Hq,Hkv,D", [(16, 2, 64), (12, 2, 128), (24, 2, 64)])
def test_gqa_probabilities_stay_whole(Hq, Hkv, D, new, ctx):
    """Probabilities reach the product with V with all 24 bits (three bf16 parts).  Seen through the outputs' rounding to 8 bits: an output that differs
    from the rounded 64-bit value had that value within its error of a border.  fp32 sums leave errors of some 1e-6 of an output, so some
    2 * 1e-6 / 2^-7.5 = 4e-4 of the outputs differ; with two rounded parts (2^-17 of a probability) it were 2e-3."""
    from batchgen_b200.ops import _ext, attention, talking
    g = torch.Generator().manual_seed(new + ctx + D)
    window, n, page = (128 if new > 1 else 0), new + ctx, 64
    wrong = total = 0
    for _ in range(2 if new > 1 else 40):
        pages = torch.randperm(-(-n // page), generator=g)
        pos = torch.arange(n)
        rows = torch.randn(n, 2 * Hkv * D, generator=g).bfloat16()
        cache = torch.zeros(len(pages), page, 2 * Hkv * D).bfloat16()
        cache.view(-1, 2 * Hkv * D)[pages[pos // page] * page + pos % page] = rows
        q = (torch.randn(new, Hq, D, generator=g) * 0.5).bfloat16().cuda()
        c, bt = cache.cuda(), pages.int().view(1, -1).cuda()
        if new > 1:
            out = torch.empty(new, Hq * D, dtype=torch.bfloat16, device="cuda")
            work = torch.tensor(talking.prefill_work([0, new], [ctx], 0, 1, window), dtype=torch.int32).cuda()
            attention.gqa_prefill(q, c, bt, work, Hkv, D ** -0.5, out, window=window)
            out = out.view(new, Hq, D)
        else:
            out = attention.gqa_decode(q, c, bt, torch.tensor([n], dtype=torch.int32).cuda(), Hkv, D ** -0.5)
        k, v = (t.view(n, Hkv, D).double().cuda() for t in rows.split(Hkv * D, 1))
        at, key = (ctx + torch.arange(new, device="cuda"))[:, None], torch.arange(n, device="cuda")[None]
        hidden = (key > at) | ((key <= at - window) if window else torch.zeros_like(key > at))
        for h in range(Hq):
            s = (q[:, h].double() @ k[:, h // (Hq // Hkv)].t() * D ** -0.5).masked_fill(hidden, float("-inf"))
            want = s.softmax(-1) @ v[:, h // (Hq // Hkv)]
            wrong += (out[:, h] != want.float().bfloat16()).sum().item()
            total += want.numel()
    _ext.check_status()
    assert wrong <= 8e-4 * total, wrong / total


@pytest.mark.parametrize("first", [1, 8, 3])
@pytest.mark.parametrize("splits", [1, 2])
def test_gqa_decode_takes_queries_at_any_address(first, splits):
    """Queries that are a contiguous view at any element of a buffer: the same bits as their copy."""
    from batchgen_b200.ops import _ext, attention
    g = torch.Generator(device="cuda").manual_seed(first)
    B, Hq, Hkv, D = 3, 16, 2, 64
    cache = torch.randn(8, 64, 2 * Hkv * D, generator=g, device="cuda").bfloat16()
    bt = torch.arange(6, dtype=torch.int32, device="cuda").view(3, 2) + 1
    lens = torch.tensor([1, 70, 128], dtype=torch.int32, device="cuda")
    buf = torch.randn(first + B * Hq * D, generator=g, device="cuda").bfloat16()
    q = buf[first:].view(B, Hq, D)
    assert q.is_contiguous() and (q.data_ptr() % 16 == 0) == (first == 8)
    got = attention.gqa_decode(q, cache, bt, lens, Hkv, D ** -0.5, num_splits=splits)
    want = attention.gqa_decode(torch.stack(list(q)), cache, bt, lens, Hkv, D ** -0.5, num_splits=splits)
    _ext.check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("new,ctx,at,splits", [(1, 199, 5, 1), (1, 199, 198, 3), (200, 100, 40, 0), (200, 0, 130, 0), (129, 64, 192, 0)])
@pytest.mark.parametrize("Hq,Hkv,D", [(16, 2, 64), (12, 2, 128), (24, 2, 64)])
def test_gqa_infinite_values_stay_infinite(Hq, Hkv, D, new, ctx, at, splits):
    """An infinite value under probabilities above zero gives infinity in its column, as in fp32, whatever bits a probability has: the
    key at ``at`` has the largest score, so where its tile is the first its probability is exactly one before the division."""
    from batchgen_b200.ops import _ext, attention, talking
    g = torch.Generator().manual_seed(new + at)
    n, page = new + ctx, 64
    rows = torch.randn(n, 2, Hkv, D, generator=g).bfloat16()
    rows[:, 0, :, 0] = 0
    rows[at, 0, :, :] = 0
    rows[at, 0, :, 0] = 8
    rows[at, 1, 0, 3], rows[at, 1, 1, 7] = float("inf"), -float("inf")
    rows[0, 1, 0, 5] = float("inf")                                  # seen by all, a probability of any bits
    q = (torch.randn(new, Hq, D, generator=g) * 0.2).bfloat16()
    q[..., 0] = 4
    cache = torch.zeros(-(-n // page) * page, 2 * Hkv * D).bfloat16()
    cache[:n] = rows.view(n, -1)
    c, bt = cache.view(-1, page, 2 * Hkv * D).cuda(), torch.arange(-(-n // page)).int().view(1, -1).cuda()
    if new > 1:
        out = torch.empty(new, Hq * D, dtype=torch.bfloat16, device="cuda")
        work = torch.tensor(talking.prefill_work([0, new], [ctx], 0, 1, 0), dtype=torch.int32).cuda()
        attention.gqa_prefill(q.cuda(), c, bt, work, Hkv, D ** -0.5, out)
    else:
        out = attention.gqa_decode(q.cuda(), c, bt, torch.tensor([n], dtype=torch.int32).cuda(), Hkv, D ** -0.5, num_splits=splits)
    _ext.check_status()
    out = out.view(new, Hq, D).float().cpu()
    seen = torch.arange(new) + ctx >= at                              # rows before it: its tile's products may hold 0 * inf
    G = Hq // Hkv
    assert (out[seen, :G, 3] == float("inf")).all() and (out[seen, G:, 7] == -float("inf")).all()
    assert (out[:, :G, 5] == float("inf")).all()
    finite = torch.ones(Hq, D, dtype=torch.bool)
    finite[:G, 3] = finite[:G, 5] = finite[G:, 7] = False
    assert torch.isfinite(out[:, finite]).all()
