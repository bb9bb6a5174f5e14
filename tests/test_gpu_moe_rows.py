"""Grouped rows of unquantised and 4-bit experts: the activation kernel, and the expert stack around it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plain(z, kind, limit):
    g, u = z.double().chunk(2, -1)
    if kind == "silu":
        return g * torch.sigmoid(g) * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return (u + 1) * g * torch.sigmoid(1.702 * g) if kind == "swiglu_clamped" else g * torch.sigmoid(g) * u


@pytest.mark.parametrize("kind,limit", [("silu", 0.0), ("swiglu_clamped", 7.0), ("silu_limit", 2.5)])
@pytest.mark.parametrize("rows,F,pad", [(1, 8, 0), (3, 72, 16), (300, 3072, 0), (4000, 264, 8)])
def test_activation_rows(kind, limit, rows, F, pad):
    from batchgen_b200.ops import moe
    g = torch.Generator().manual_seed(rows + F)
    z = (torch.randn(rows, 2 * F + pad, generator=g) * 4).bfloat16()
    z[0, :4] = torch.tensor([float("nan"), float("inf"), -float("inf"), 100.0])
    z[0, F:F + 4] = torch.tensor([1.0, 2.0, 3.0, float("nan")])
    present = max(1, rows - 5)
    src = torch.arange(rows, dtype=torch.int32)
    src[1::7] = -1
    offsets = torch.tensor([0, present], dtype=torch.int32)
    d = z.cuda()[:, :2 * F]
    want = _plain(z[:, :2 * F], kind, limit)
    for off, s in ((None, None), (offsets.cuda(), src.cuda())):
        got = moe.activation(d, kind, limit, off, s).double().cpu()
        keep = torch.ones(rows, dtype=torch.bool) if off is None else (src >= 0) & (torch.arange(rows) < present)
        a, b = got[keep], want[keep]
        fine = torch.isfinite(b)
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a[~fine & ~torch.isnan(b)], b[~fine & ~torch.isnan(b)])
        # one rounding to 8 significant bits, and fp32 arithmetic: a few 2^-24
        assert ((a - b).abs()[fine] <= b.abs()[fine] * (2 ** -8 + 1e-5) + 1e-30).all()


@pytest.mark.parametrize("kind,limit", [("silu", 0.0), ("swiglu_clamped", 7.0), ("silu_limit", 2.5)])
def test_activation_keeps_fp32(kind, limit):
    """The activation is computed in fp32 and rounded once, for gates down to where the exponential overflows: an output differs from the rounded 64-bit
    value only where that value lies as near to the border between two bf16 numbers as fp32 arithmetic is exact."""
    from batchgen_b200.ops import moe
    g = torch.Generator().manual_seed(2)
    F = 1 << 14
    z = torch.cat([torch.rand(16, F, generator=g) * 95 - 87.5, torch.randn(16, F, generator=g)], 1).bfloat16()
    z[:, 0] = -87.5
    got, want = moe.activation(z.cuda(), kind, limit).double().cpu(), _plain(z, kind, limit)
    near = want.float().bfloat16().double()
    # expf 2 units of 2^-24, the sum, the quotient and two products half a unit each, of which 1.702 g moves the exponent: |1.702 g| 2^-24
    slack = 2.0 ** -24 * (4 + (1.702 * z[:, :F].double().abs() if kind == "swiglu_clamped" else 0))
    # an ulp of bf16 is 2^-7 to 2^-8 of the value: the border lies half of it away
    step = torch.exp2(want.abs().clamp_min(1e-300).log2().floor() - 7)
    border = ((want / step).abs() % 1 - 0.5).abs() * step
    assert ((got == near) | ((border <= want.abs() * slack) & ((got - near).abs() <= step * 1.01)) | (want.abs() < 1e-35)).all()


@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("quant", ["none", "mxfp4"])
@pytest.mark.parametrize("kind", ["silu", "swiglu_clamped"])
def test_expert_stack(T, quant, kind):
    """Pairs of a few tokens over experts of which some stay empty, padding tokens, a row added at the sum."""
    from batchgen_b200.ops import _ext, moe, mxfp4
    E, K, H, I = 9, 3, 192, 128
    g = torch.Generator().manual_seed(T)
    w13, w2 = torch.randn(E, 2 * I, H, generator=g) * 0.1, torch.randn(E, H, I, generator=g) * 0.1
    x, extra = torch.randn(T, H, generator=g).bfloat16(), torch.randn(T, H, generator=g).bfloat16()
    idx = torch.stack([torch.randperm(E - 2, generator=g)[:K] for _ in range(T)]).int()
    w = torch.rand(T, K, generator=g)
    if quant == "none":
        ew = moe.ExpertWeights(w13.bfloat16().cuda(), w2.bfloat16().cuda(), activation=kind)
        f13, f2 = w13.bfloat16().double(), w2.bfloat16().double()
    else:
        q13, s13 = mxfp4.quantize(w13)
        q2, s2 = mxfp4.quantize(w2)
        f13, f2 = mxfp4.dequantize(q13, s13, torch.float32).double(), mxfp4.dequantize(q2, s2, torch.float32).double()
        ew = moe.ExpertWeights(q13.cuda(), q2.cuda(), s13.cuda(), s2.cuda(), quant="mxfp4", activation=kind).to_device_layout()
    valid = T - T // 3
    got = moe.experts_forward(x.cuda(), torch.where(torch.arange(T).unsqueeze(1) < valid, idx, -1).int().cuda(), w.cuda(), ew, 0, E,
                              extra=extra.cuda(), num_valid=torch.tensor([valid], dtype=torch.int32).cuda())
    torch.cuda.synchronize()
    _ext.check_status()
    want = extra.double()
    for t in range(valid):
        for k in range(K):
            e = int(idx[t, k])
            z = _plain((x[t].double() @ f13[e].t()).bfloat16(), kind, 7.0).bfloat16().double()
            want[t] += w[t, k].double() * (z @ f2[e].t()).bfloat16().double()
    err = (got.double().cpu() - want).norm() / want.norm()
    # four roundings to bf16 on the way (pre-activation, activation, expert row, sum), each some 2^-9 of its value
    assert err < 4 * 2 ** -9, err


@pytest.mark.parametrize("quant", ["none", "mxfp4"])
def test_expert_stack_takes_tokens_at_any_address(quant):
    """Tokens that are a contiguous view at any element of a buffer: the same bits as their copy."""
    from batchgen_b200.ops import _ext, moe, mxfp4
    E, K, H, I, T = 4, 2, 192, 128, 7
    g = torch.Generator().manual_seed(5)
    w13, w2 = torch.randn(E, 2 * I, H, generator=g) * 0.1, torch.randn(E, H, I, generator=g) * 0.1
    if quant == "none":
        ew = moe.ExpertWeights(w13.bfloat16().cuda(), w2.bfloat16().cuda())
    else:
        (q13, s13), (q2, s2) = mxfp4.quantize(w13), mxfp4.quantize(w2)
        ew = moe.ExpertWeights(q13.cuda(), q2.cuda(), s13.cuda(), s2.cuda(), quant="mxfp4").to_device_layout()
    x = torch.randn(3 + T * H, generator=g).bfloat16().cuda()[3:].view(T, H)
    assert x.is_contiguous() and x.data_ptr() % 16
    idx = torch.randint(0, E, (T, K), generator=g).int().cuda()
    w = torch.rand(T, K, generator=g).cuda()
    got, want = (moe.experts_forward(h, idx, w, ew, 0, E) for h in (x, torch.stack(list(x))))
    _ext.check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("counts,align", [([1, 0, 17, 130], 8), ([256, 257, 5, 600], 8), ([15, 16, 31, 33], 16), ([3, 0, 0, 0], 8)])
@pytest.mark.parametrize("N,K", [(128, 64), (200, 192), (384, 1024)])
def test_grouped_bf16_token_tiles(counts, align, N, K):
    """Segments at the edges of the token tiles (16 and 256 rows), rows past a segment's count not finite, weight rows that end inside
    a tile."""
    from batchgen_b200.ops import _ext, gemm
    g = torch.Generator().manual_seed(N + sum(counts))
    offs = [0]
    for c in counts:
        offs.append(offs[-1] + (c + align - 1) // align * align + align)
    x = torch.full((offs[-1], K), float("nan")).bfloat16()
    for e, c in enumerate(counts):
        x[offs[e]:offs[e] + c] = torch.randn(c, K, generator=g).bfloat16()
    w = torch.randn(len(counts), N, K, generator=g).bfloat16()
    off, cnt = torch.tensor(offs, dtype=torch.int32).cuda(), torch.tensor(counts, dtype=torch.int32).cuda()
    swapped = torch.empty(offs[-1], N, dtype=torch.bfloat16, device="cuda")
    gemm._bf16_swap(x.cuda(), w.cuda(), swapped, off, cnt, len(counts), N)
    for got in (swapped.cpu().double(), gemm.grouped_bf16_gemm(x.cuda(), w.cuda(), off, cnt).cpu().double()):
        _ext.check_status()
        for e, c in enumerate(counts):
            xe, we = x[offs[e]:offs[e] + c].double(), w[e].double()
            want = xe @ we.t()
            # one rounding to 8 significant bits; fp32 sums of K exact products: K * 2^-24 of their magnitudes
            assert ((got[offs[e]:offs[e] + c] - want).abs() <= want.abs() * 2 ** -8 + (xe.abs() @ we.abs().t()) * K * 2 ** -24).all(), e


@pytest.mark.parametrize("T,N,K", [(1030, 3144, 128), (257, 14208, 64), (4096, 1000, 192)])
def test_dense_bf16_token_tiles(T, N, K):
    """Enough tiles of 256 tokens for the SMs, rows and outputs that end inside a tile, output rows inside a wider tensor."""
    from batchgen_b200.ops import _ext, gemm
    g = torch.Generator().manual_seed(T)
    x, w = torch.randn(T, K, generator=g).bfloat16(), torch.randn(N, K, generator=g).bfloat16()
    wide = torch.full((T, N + 24), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.bf16_gemm(x.cuda(), w.cuda(), out=wide[:, 8:8 + N])
    _ext.check_status()
    got, want = wide.cpu().double(), x.double() @ w.double().t()
    assert (got[:, :8] == 7).all() and (got[:, 8 + N:] == 7).all()
    assert ((got[:, 8:8 + N] - want).abs() <= want.abs() * 2 ** -8 + (x.double().abs() @ w.double().abs().t()) * K * 2 ** -24).all()


@pytest.mark.parametrize("T,N,K,pad", [(1, 8, 64, 0), (33, 264, 192, 24), (256, 512, 1024, 3), (257, 300, 64, 0), (700, 1000, 128, 8)])
def test_dense_bf16_pairs(T, N, K, pad):
    """Products on pairs of CTAs: tokens and outputs that end inside a CTA's half, rows that are not 16-byte aligned; the one-CTA form's bits."""
    import ctypes
    from batchgen_b200.ops import _ext
    g = torch.Generator().manual_seed(T)
    x, w = torch.randn(T, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    outs = []
    for fn, mid in (("bg_gemm_bf16_pair", (None, None, 1)), ("bg_gemm_bf16_swap", ())):
        out = torch.full((T, N + pad), 7.0, dtype=torch.bfloat16, device="cuda")
        mid = tuple(ctypes.c_void_p(0) if m is None else ctypes.c_int(m) for m in mid)
        rc = getattr(_ext.lib(), fn)(_ext.ptr(x), _ext.ptr(w), _ext.ptr(out), ctypes.c_int(N + pad), *mid, ctypes.c_int(T), ctypes.c_int(N),
                                     ctypes.c_int(K), ctypes.c_int(_ext.num_sms(x.device)), _ext.ptr(_ext.status_word(x.device)), _ext.stream())
        assert rc == 0
        _ext.check_status()
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and (outs[0][:, N:] == 7).all()
    got, want = outs[0][:, :N].cpu().double(), (x.cpu().double() @ w.cpu().double().t())
    assert ((got - want).abs() <= want.abs() * 2 ** -8 + (x.cpu().double().abs() @ w.cpu().double().abs().t()) * K * 2 ** -24).all()


@pytest.mark.parametrize("T,K,local", [(1, 128, (0, 16)), (37, 640, (3, 9)), (700, 7168, (0, 16)), (1536, 2176, (12, 16))])
def test_quantised_rows_of_tokens(T, K, local):
    """A token's bytes and scales in the row of each of its local experts: those of the whole batch, by either walk."""
    from batchgen_b200.ops import fused, moe, ref

    torch.manual_seed(T)
    x = (torch.randn(T, K + 8, device="cuda") * 3).to(torch.bfloat16)[:, 8:]
    idx = torch.rand(T, 16, device="cuda").topk(5, -1)[1].to(torch.int32)
    src, pos, offs = moe.permute(idx, *local)
    assert ((pos >= 0) == ((idx >= local[0]) & (idx < local[1]))).all()
    wq, ws = ref.act_quant(x.contiguous())
    for kw in ({}, {"pos": pos}):
        q, s = moe.gather_quant(x, src, offs, zero_padding=False, **kw)
        rows = pos[pos >= 0].long()
        token = torch.arange(T, device="cuda").unsqueeze(1).expand_as(pos)[pos >= 0]
        fq, fs = fused.act_quant(x)
        assert (q[rows].view(torch.uint8) == fq[token].view(torch.uint8)).all() and (s[rows] == fs[token]).all()
        assert torch.allclose(s[rows], ws[token], rtol=1e-6, atol=0)          # the reference divides where the kernel multiplies: an ulp or two
        assert (q[rows].view(torch.uint8) != wq[token].view(torch.uint8)).float().mean() < 2e-3     # as for whole batches: a byte at a rounding line


@pytest.mark.parametrize("rope,D,pad", [(16, 24, 0), (64, 192, 8), (48, 128, 2), (24, 40, 0), (64, 64, 1)])
def test_rotated_queries(rope, D, pad):
    """Pieces of sixteen bytes where rows and dims allow them, pairs one by one elsewhere: the same rounding."""
    from batchgen_b200.ops import fused, ref

    torch.manual_seed(rope)
    T, H = 19, 5
    pos = torch.randint(0, 200, (T,), device="cuda", dtype=torch.int32)
    ang = torch.rand(200, rope // 2, device="cuda") * 6
    cos, sin = ang.cos(), ang.sin()
    for inter in (True, False):
        q = torch.randn(T, H * D + pad, device="cuda").to(torch.bfloat16)[:, pad:].unflatten(1, (H, D))
        want = q.double().clone()
        want[..., -rope:] = ref.apply_rope(q[..., -rope:].double(), cos[pos.long()].double(), sin[pos.long()].double(), inter).double()
        bound = want.abs() * 2.0 ** -8 + q.double().abs().amax() * 2.0 ** -22         # one bf16 rounding of two fp32 products and a sum
        assert ((fused.rope_q_(q.clone() if pad == 0 else q, pos, cos, sin, rope, inter).double() - want).abs() <= bound).all()


@pytest.mark.parametrize("K", [128, 384, 2048, 7168])
@pytest.mark.parametrize("padding", [False, True])
def test_quantised_activation_of_few_and_many_rows(K, padding):
    """SiLU * up quantised by warps that walk the rows and, from 18,944 blocks on, by a CTA a row: the same bytes."""
    from batchgen_b200.ops import fused

    T = -(-148 * 128 // (K // 128))                          # the first number of rows that takes the second form
    g = torch.Generator(device="cuda").manual_seed(K)
    x = (torch.randn(T, 2 * K + 8, device="cuda", generator=g) * 3).to(torch.bfloat16)[:, 8:]
    src = torch.arange(T, device="cuda", dtype=torch.int32)
    kw = {}
    if padding:
        src[::7] = -1
        kw = dict(valid_rows=torch.tensor([T - 3], dtype=torch.int32, device="cuda"), row_src=src)
    kept = (src >= 0) & (torch.arange(T, device="cuda") < (T - 3 if padding else T))
    q, s = fused.act_quant(x, silu_mul=True, **kw)
    few = [fused.act_quant(x[a:b], silu_mul=True) for a, b in ((0, T // 2), (T // 2, T))]
    assert (q.view(torch.uint8)[kept] == torch.cat([f[0].view(torch.uint8) for f in few])[kept]).all() and (s[kept] == torch.cat([f[1] for f in few])[kept]).all()
    y = x.double()
    want = (torch.nn.functional.silu(y[:, :K]) * y[:, K:])[kept]
    step = s[kept].double().repeat_interleave(128, 1)
    # a value rounded to 8 bits, then to 4, in units of the scale down to 2^-9 of it
    assert ((q[kept].double() * step - want).abs() <= want.abs() * (2.0 ** -4 + 2.0 ** -8) + step * 2.0 ** -10).all()


@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("T,H,D,rope", [(400, 16, 192, 64), (1025, 1, 64, 64), (1024, 8, 64, 64), (30, 9, 64, 64), (30, 40, 24, 16), (30, 16, 128, 48), (30, 5, 128, 128)])
def test_rotated_queries_do_not_depend_on_alignment(interleaved, T, H, D, rope):
    """Rows in 16-byte pieces and rows that start between them: the same bytes, those of a x cos - round(b x sin) and a x sin + round(b x cos)."""
    from batchgen_b200.ops import fused

    g = torch.Generator(device="cuda").manual_seed(0)
    pos = torch.randint(0, 4096, (T,), device="cuda", dtype=torch.int32, generator=g)
    ang = torch.rand(4096, rope // 2, device="cuda", generator=g) * 6
    cos, sin = ang.cos(), ang.sin()
    q = torch.randn(T, H, D, device="cuda", generator=g).to(torch.bfloat16)
    got = []
    for shift in (0, 1):
        rows = torch.zeros(T, H * D + 8, device="cuda", dtype=torch.bfloat16)[:, shift:shift + H * D].unflatten(1, (H, D)).copy_(q)
        got.append(fused.rope_q_(rows, pos, cos, sin, rope, interleaved).clone())
    assert torch.equal(got[0], got[1])
    x = q[..., D - rope:].double()
    a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :rope // 2], x[..., rope // 2:])
    c, s = (v[pos.long()].double().unsqueeze(1) for v in (cos, sin))
    u, v = a * c - (b * s).float().double(), a * s + (b * c).float().double()
    want = torch.stack([u, v], -1).flatten(-2) if interleaved else torch.cat([u, v], -1)
    assert torch.equal(got[0][..., D - rope:], want.float().to(torch.bfloat16)) and torch.equal(got[0][..., :D - rope], q[..., :D - rope])


@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("counts,align", [([1, 0, 17, 130], 8), ([256, 257, 5, 600], 8), ([15, 16, 31, 33], 16), ([3, 0, 0, 0], 8)])
@pytest.mark.parametrize("N,K", [(128, 64), (200, 192), (384, 1024)])
def test_grouped_bf16_forms(pairs, counts, align, N, K, monkeypatch):
    """Segments on pairs of CTAs and on one, whichever the rule would take."""
    from batchgen_b200.ops import gemm
    monkeypatch.setattr(gemm, "use_pairs_grouped", lambda *a: pairs)
    test_grouped_bf16_token_tiles(counts, align, N, K)


@pytest.mark.parametrize("pad,off", [(0, 0), (4, 0), (0, 4), (3, 1)])
@pytest.mark.parametrize("counts", [None, [130, 0, 300, 7]])
def test_bf16_rows_that_are_not_in_16_byte_pieces(counts, pad, off, monkeypatch):
    """Such rows stay on one CTA even where pairs pay; the same bits, nothing beside them."""
    from batchgen_b200.ops import _ext, gemm
    g = torch.Generator().manual_seed(1)
    N, K, E = 520, 704, 1 if counts is None else len(counts)
    offs = [0]
    for c in counts or [437]:
        offs.append(offs[-1] + c)
    M = offs[-1]
    monkeypatch.setattr(gemm, "use_pairs", lambda *a: True)
    monkeypatch.setattr(gemm, "use_pairs_grouped", lambda *a: True)
    names = []
    lib = _ext.lib()
    monkeypatch.setattr(_ext, "lib", lambda: type("L", (), {"__getattr__": lambda self, n: (names.append(n), getattr(lib, n))[1]})())
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(E, N, K, generator=g).bfloat16().cuda()
    tables = [None, None] if counts is None else [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (offs, counts)]
    whole = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    gemm._bf16_swap(x, w.view(E * N, K), whole, *tables, E, N)
    buf = torch.full((M * (N + pad) + off,), 7.0, dtype=torch.bfloat16, device="cuda")
    out = buf[off:].view(M, N + pad)[:, :N]
    gemm._bf16_swap(x, w.view(E * N, K), out, *tables, E, N)
    _ext.check_status()
    assert names == ["bg_gemm_bf16_pair", "bg_gemm_bf16_swap_grouped" if pad % 8 or off % 8 else "bg_gemm_bf16_pair"] and torch.equal(out, whole)
    out.fill_(7.0)
    assert (buf == 7).all()
    xe = x.double().cpu()
    want = torch.cat([xe[offs[e]:offs[e + 1]] @ w[e].double().cpu().t() for e in range(E)])
    mag = torch.cat([xe[offs[e]:offs[e + 1]].abs() @ w[e].double().cpu().abs().t() for e in range(E)])
    assert ((whole.cpu().double() - want).abs() <= want.abs() * 2 ** -8 + mag * K * 2 ** -24).all()
