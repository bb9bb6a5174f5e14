"""MXFP4-weight tcgen05 GEMM against fp32 references of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-9)).item()


def test_dequant_kernel_exact():
    from batchgen_b200.ops import mxfp4, ref
    w = torch.randn(96, 256) * 3
    q, s = mxfp4.quantize(w)
    d = mxfp4.dequantize(q.cuda(), s.cuda(), torch.float32).cpu()
    assert torch.equal(d, ref.mxfp4_dequant(q, s))


@pytest.mark.parametrize("T,N,K", [(128, 128, 64), (200, 384, 512), (1, 7168, 3584), (515, 200, 1024)])
def test_dense_gemm(T, N, K):
    from batchgen_b200.ops import _ext, mxfp4
    g = torch.Generator().manual_seed(T + N)
    w = torch.randn(N, K, generator=g) * 0.05
    q, s = mxfp4.quantize(w)
    x = (torch.randn(T, K, generator=g)).to(torch.bfloat16)
    y = mxfp4.mxfp4_gemm(x.cuda(), q.cuda(), s.cuda())
    _ext.check_status()
    want = x.float() @ mxfp4.dequantize(q, s, torch.float32).t()
    assert _rel(y.cpu(), want) < 6e-3


@pytest.mark.parametrize("silu", [False, True])
def test_grouped_gemm(silu):
    from batchgen_b200.ops import _ext, mxfp4
    from batchgen_b200.ops.gemm import interleave_gate_up_rows
    g = torch.Generator().manual_seed(5)
    E, N, K = 5, 256, 384
    rows = [128, 0, 37, 256, 1]
    starts, cur = [0], 0
    for r in rows:
        cur += (r + 127) // 128 * 128
        starts.append(cur)
    offsets = torch.tensor([starts[i] for i in range(E)] + [starts[-1]], dtype=torch.int32)
    # segment e holds rows[e] real rows followed by padding up to the next 128-aligned start
    ends = [starts[e] + rows[e] for e in range(E)]
    x = torch.zeros(starts[-1], K)
    for e in range(E):
        x[starts[e]:ends[e]] = torch.randn(rows[e], K, generator=g)
    x = x.to(torch.bfloat16)
    w = torch.randn(E, N, K, generator=g) * 0.05
    q, s = mxfp4.quantize(w)
    wd = mxfp4.dequantize(q, s, torch.float32)
    qd, sd = q.cuda(), s.cuda()
    if silu:
        perm = interleave_gate_up_rows(N)
        qd, sd = qd[:, perm.cuda()].contiguous(), sd[:, perm.cuda()].contiguous()
    y = mxfp4.grouped_mxfp4_gemm(x.cuda(), qd, sd, offsets.cuda(), silu_mul=silu).cpu()
    _ext.check_status()
    for e in range(E):
        if rows[e] == 0:
            continue
        ref_e = x[starts[e]:ends[e]].float() @ wd[e].t()
        if silu:
            ref_e = torch.nn.functional.silu(ref_e[:, : N // 2]) * ref_e[:, N // 2:]
        assert _rel(y[starts[e]:ends[e]], ref_e) < 8e-3, e


@pytest.mark.parametrize("silu", [False, True])
def test_int4_grouped_gemm(silu):
    from batchgen_b200.ops import _ext, int4
    from batchgen_b200.ops.gemm import interleave_gate_up_rows
    g = torch.Generator().manual_seed(8)
    E, N, K = 3, 256, 256
    rows = [130, 0, 5]
    starts, cur = [], 0
    for r in rows:
        starts.append(cur)
        cur += (r + 127) // 128 * 128
    offsets = torch.tensor(starts + [cur], dtype=torch.int32)
    x = torch.randn(cur, K, generator=g).to(torch.bfloat16)
    q, s = int4.quantize(torch.randn(E, N, K, generator=g) * 0.05)
    wd = int4.dequantize(q, s)
    qd, sd = q.cuda(), s.cuda()
    if silu:
        perm = interleave_gate_up_rows(N).cuda()
        qd, sd = qd[:, perm].contiguous(), sd[:, perm].contiguous()
    y = int4.grouped_int4_gemm(x.cuda(), qd, sd, offsets.cuda(), silu_mul=silu).cpu()
    _ext.check_status()
    for e in range(E):
        a, n = starts[e], rows[e]
        if not n:
            continue
        want = x[a:a + n].float() @ wd[e].t()
        if silu:
            want = torch.nn.functional.silu(want[:, : N // 2]) * want[:, N // 2:]
        assert _rel(y[a:a + n], want) < 8e-3, e
    assert _rel(int4.int4_gemm(x[:40].cuda(), q[0].cuda(), s[0].cuda()).cpu(), x[:40].float() @ wd[0].t()) < 8e-3


@pytest.mark.parametrize("counts", [[1, 0, 17, 130], [192, 193, 5, 400], [16, 15, 33, 64]])
@pytest.mark.parametrize("fmt", ["mxfp4", "int4"])
@pytest.mark.parametrize("N,K,silu", [(256, 64, True), (384, 192, False), (200, 320, False)])
def test_w4_token_tiles_and_scales(counts, fmt, N, K, silu):
    """Segments at the edges of the token tiles (16 and 192 rows), rows past a segment's count not finite, weight rows that end inside a
    tile, scales from 2^-127 to above 2 (the largest ones beside ordinary ones)."""
    from batchgen_b200.ops import _ext, int4, mxfp4
    from batchgen_b200.ops.gemm import interleave_gate_up_rows
    g = torch.Generator().manual_seed(N + sum(counts))
    E = len(counts)
    offs = [0]
    for c in counts:
        offs.append(offs[-1] + (c + 7) // 8 * 8 + 8)
    x = torch.full((offs[-1], K), float("nan")).bfloat16()
    for e, c in enumerate(counts):
        x[offs[e]:offs[e] + c] = torch.randn(c, K, generator=g).bfloat16()
    wq = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.uint8)
    if fmt == "mxfp4":
        ws = torch.randint(120, 129, (E, N, K // 32), generator=g, dtype=torch.uint8)
        ws[0, ::5] = 0
        ws[1, 3::64] = 131
        ws[2, 1::7, 0] = 150
        w = mxfp4.dequantize(wq, ws, torch.float32).double()
    else:
        ws = (torch.rand(E, N, K // 32, generator=g) * 0.1).bfloat16()
        w = int4.dequantize(wq, ws).bfloat16().double()
    off, cnt = torch.tensor(offs, dtype=torch.int32).cuda(), torch.tensor(counts, dtype=torch.int32).cuda()
    run = mxfp4.grouped_mxfp4_gemm if fmt == "mxfp4" else int4.grouped_int4_gemm
    got = run(x.cuda(), wq.cuda(), ws.cuda(), off, silu_mul=silu, counts=cnt).cpu().double()
    _ext.check_status()
    for e, c in enumerate(counts):
        xe = x[offs[e]:offs[e] + c].double()
        want, mag = xe @ w[e].t(), xe.abs() @ w[e].abs().t()
        if silu:
            back = torch.argsort(interleave_gate_up_rows(N))
            want, mag = want[:, back], mag[:, back]
            a, u = want.chunk(2, -1)
            am, um = mag.chunk(2, -1)
            want = torch.nn.functional.silu(a) * u
            mag = am * (u.abs() + 1) * 1.1 + um * a.abs()
        # one rounding to 8 significant bits; fp32 sums of up to 320 exact products: 320 * 2^-24 of their magnitudes; products of
        # subnormal weights may be flushed (below 1e-36)
        assert ((got[offs[e]:offs[e] + c] - want).abs() <= want.abs() * 2 ** -8 + mag * 2e-5 + 1e-36).all(), e


@pytest.mark.parametrize("counts", [[1, 0, 210, 40], [193, 7, 0, 385]])
@pytest.mark.parametrize("fmt", ["mxfp4", "int4"])
@pytest.mark.parametrize("K", [320, 384, 448, 512, 2880])
@pytest.mark.parametrize("N,silu", [(640, False), (512, True)])
def test_w4_many_tiles_a_cta(counts, fmt, K, N, silu, monkeypatch):
    """Two CTAs walk all tiles, a dozen and more each: operand slots, rings and accumulators across tile borders, with K steps that are and
    are not a multiple of the expansion groups."""
    from batchgen_b200.ops import _ext, int4, mxfp4
    from batchgen_b200.ops.gemm import interleave_gate_up_rows
    g = torch.Generator().manual_seed(K + N + sum(counts))
    E = len(counts)
    offs = [0]
    for c in counts:
        offs.append(offs[-1] + (c + 7) // 8 * 8)
    x = torch.randn(offs[-1], K, generator=g).bfloat16()
    wq = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.uint8)
    if fmt == "mxfp4":
        ws = torch.randint(120, 124, (E, N, K // 32), generator=g, dtype=torch.uint8)
        w = mxfp4.dequantize(wq, ws, torch.float32).double()
    else:
        ws = (torch.rand(E, N, K // 32, generator=g) * 0.1).bfloat16()
        w = int4.dequantize(wq, ws).bfloat16().double()
    off, cnt = torch.tensor(offs, dtype=torch.int32).cuda(), torch.tensor(counts, dtype=torch.int32).cuda()
    monkeypatch.setattr(_ext, "num_sms", lambda device=None: 2)
    run = mxfp4.grouped_mxfp4_gemm if fmt == "mxfp4" else int4.grouped_int4_gemm
    got = run(x.cuda(), wq.cuda(), ws.cuda(), off, silu_mul=silu, counts=cnt).cpu().double()
    _ext.check_status()
    for e, c in enumerate(counts):
        xe = x[offs[e]:offs[e] + c].double()
        want, mag = xe @ w[e].t(), xe.abs() @ w[e].abs().t()
        if silu:
            back = torch.argsort(interleave_gate_up_rows(N))
            want, mag = want[:, back], mag[:, back]
            a, u = want.chunk(2, -1)
            am, um = mag.chunk(2, -1)
            want = torch.nn.functional.silu(a) * u
            mag = am * (u.abs() + 1) * 1.1 + um * a.abs()
        # one rounding to 8 significant bits; fp32 sums of K exact products: K * 2^-24 of their magnitudes
        assert ((got[offs[e]:offs[e] + c] - want).abs() <= want.abs() * 2 ** -8 + mag * K * 2 ** -24 + 1e-36).all(), e


SPARSE = {0: 3, 15: 1, 16: 200, 40: 17, 47: 385, 69: 5}           # rows of the segments that have any, of 70


@pytest.mark.parametrize("only", [sorted(SPARSE), [69], [16], [0], []])
@pytest.mark.parametrize("kernel", ["mxfp4", "swap"])
def test_segments_that_are_passed_over(only, kernel, monkeypatch):
    """70 segments of which few have rows, first and last and in blocks of 16 of their own: every row of theirs, and nothing else, is written."""
    from batchgen_b200.ops import _ext, gemm, mxfp4
    g = torch.Generator().manual_seed(len(only))
    E, N, K = 70, 256, 192
    counts = [SPARSE.get(e, 0) if e in only else 0 for e in range(E)]
    offs = [0]
    for c in counts:
        offs.append(offs[-1] + (c + 7) // 8 * 8)
    rows = max(offs[-1], 8)
    x = torch.randn(rows, K, generator=g).bfloat16()
    off, cnt = torch.tensor(offs, dtype=torch.int32).cuda(), torch.tensor(counts, dtype=torch.int32).cuda()
    out = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device="cuda")
    monkeypatch.setattr(_ext, "num_sms", lambda device=None: 3)
    if kernel == "mxfp4":
        wq = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.uint8)
        ws = torch.randint(120, 124, (E, N, K // 32), generator=g, dtype=torch.uint8)
        w = mxfp4.dequantize(wq, ws, torch.float32).double()
        mxfp4.grouped_mxfp4_gemm(x.cuda(), wq.cuda(), ws.cuda(), off, out=out, counts=cnt)
    else:
        wb = torch.randn(E, N, K, generator=g).bfloat16()
        w = wb.double()
        gemm._bf16_swap(x.cuda(), wb.cuda(), out, off, cnt, E, N)
    _ext.check_status()
    got, seen = out.cpu().double(), torch.zeros(rows, dtype=torch.bool)
    for e, c in enumerate(counts):
        xe = x[offs[e]:offs[e] + c].double()
        # one rounding to 8 significant bits; fp32 sums of K exact products: K * 2^-24 of their magnitudes
        assert ((got[offs[e]:offs[e] + c] - xe @ w[e].t()).abs() <= (xe @ w[e].t()).abs() * 2 ** -8 + xe.abs() @ w[e].abs().t() * K * 2 ** -24).all(), e
        seen[offs[e]:offs[e] + c] = True
    assert (got[~seen] == 7).all()


def _block_case(counts, lead, N, K, seed):
    """Segments that start anywhere (``lead`` rows before each), rows of 20 binades, weights and scales of every size."""
    g = torch.Generator().manual_seed(seed)
    offs = [lead]
    for c in counts:
        offs.append(offs[-1] + c + lead)
    x = torch.randn(offs[-1], K, generator=g) * torch.exp2(torch.randint(-10, 11, (offs[-1], K), generator=g).float())
    wq = torch.randint(0, 256, (len(counts), N, K // 2), generator=g, dtype=torch.uint8)
    ws = torch.randint(110, 135, (len(counts), N, K // 32), generator=g, dtype=torch.uint8)
    return x.bfloat16(), wq, ws, torch.tensor(offs, dtype=torch.int32), torch.tensor(counts, dtype=torch.int32)


@pytest.mark.parametrize("counts,lead", [([1, 0, 17, 40], 0), ([32, 33, 5, 3], 3), ([96, 97, 1, 8], 8), ([7, 31, 9, 64], 5)])
@pytest.mark.parametrize("N,K,rows", [(256, 128, 10), (136, 192, 100), (200, 2880, 10), (640, 448, 40)])
def test_block_scaled_products(counts, lead, N, K, rows, monkeypatch):
    """Tiles of 32 and of 96 tokens whose segments start and end inside an eight of rows, weight rows that end inside a tile, the last half step of K,
    output rows that are not 16-byte aligned; a few CTAs walk all tiles."""
    from batchgen_b200.ops import _ext, mxfp4
    x, wq, ws, off, cnt = _block_case(counts, lead, N, K, N + K + lead)
    E = len(counts)
    monkeypatch.setattr(_ext, "num_sms", lambda device=None: 3)
    out = torch.full((x.shape[0] * (N + 8) + 1,), 7.0, dtype=torch.bfloat16, device="cuda")[1:].view(-1, N + 8)
    mxfp4._block_gemm(x.cuda(), wq.cuda().view(E * N, -1), ws.cuda().view(E * N, -1), out, off.cuda(), E, x.shape[0], N, K, cnt.cuda(), rows)
    _ext.check_status()
    w, got, seen = mxfp4.dequantize(wq, ws, torch.float32).double(), out.cpu().double(), torch.zeros(x.shape[0], dtype=torch.bool)
    for e, c in enumerate(counts):
        a = int(off[e])
        xe = x[a:a + c].double()
        want, mag = xe @ w[e].t(), xe.abs() @ w[e].abs().t()
        # what the parts leave out: 2^-22 of the largest of 32 elements, for each of them
        tops = xe.abs().view(c, K // 32, 32).amax(-1, keepdim=True).expand(c, K // 32, 32).reshape(c, K)
        lost = 2.0 ** -22 * (tops @ w[e].abs().t())
        assert ((got[a:a + c, :N] - want).abs() <= want.abs() * 2 ** -8 + mag * K * 2 ** -24 + lost).all(), e
        seen[a:a + c] = True
    assert (got[~seen] == 7).all() and (got[:, N:] == 7).all()


@pytest.mark.parametrize("what", [float("inf"), float("-inf"), float("nan")])
def test_block_scaled_products_not_finite(what):
    """An infinity or NaN in a row: what the product of bf16 operands gives, and nothing in other rows."""
    from batchgen_b200.ops import _ext, mxfp4
    x, wq, ws, off, cnt = _block_case([5, 20], 0, 256, 192, 3)
    x[2, 7] = what
    x[9, [3, 190]] = torch.tensor([what, -what]).bfloat16()
    x[12, 100] = what
    x[12, 64] = 3e38
    args = (x.cuda(), wq.cuda().view(512, -1), ws.cuda().view(512, -1))
    new, old = (torch.empty(25, 256, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    mxfp4._block_gemm(*args, new, off.cuda(), 2, 25, 256, 192, cnt.cuda(), 10)
    mxfp4._launch(mxfp4.EPI_STORE, *args, old, off.cuda(), 2, 25, 256, 192, cnt.cuda())
    _ext.check_status()
    odd = ~torch.isfinite(old)
    assert odd[2].all() and odd[9].all() and odd[12].all() and not odd[[0, 1, 3, 8, 10, 24]].any()
    assert torch.equal(new[odd].nan_to_num(nan=1.0, posinf=2.0, neginf=3.0), old[odd].nan_to_num(nan=1.0, posinf=2.0, neginf=3.0))
    assert torch.isfinite(new[~odd]).all()


@pytest.mark.parametrize("kind", ["swiglu_clamped", "silu", "silu_limit"])
def test_gated_parts(kind):
    """The activation's rows as parts are the rows: every element but the ones far below their block's largest."""
    from batchgen_b200.ops import _ext, moe, mxfp4
    g = torch.Generator().manual_seed(1)
    z = (torch.randn(37, 2 * 2880, generator=g) * 3).bfloat16().cuda()
    src = torch.arange(37, dtype=torch.int32).cuda()
    src[5] = -1
    off = torch.tensor([0, 30], dtype=torch.int32).cuda()
    want = moe.activation(z, kind, 2.0, off, src).cpu().double()
    p = mxfp4.gated_parts(z, *moe._activation_kind(kind, 2.0), off, src)
    _ext.check_status()
    parts = p.p.view(torch.float8_e4m3fn).cpu().double().transpose(1, 2).reshape(-1, 2, 2880)
    scale = torch.exp2(p.s.cpu().double().permute(1, 0, 2).reshape(37, -1)[:, :90] - 127).repeat_interleave(32, 1)
    rows = [r for r in range(30) if r != 5]
    got = scale[rows] * (parts[rows, 0] + parts[rows, 1] / 32)
    top = want[rows].abs().view(-1, 90, 32).amax(-1).repeat_interleave(32, 1)
    assert ((got - want[rows]).abs() <= top * 2.0 ** -22).all() and (got == want[rows])[want[rows].abs() > top * 2.0 ** -13].all()


@pytest.mark.parametrize("rows", [10, 31])
def test_block_scaled_products_longest_rows(rows, monkeypatch):
    """K of 12,288, the largest that the loads take: four stages beside tiles of 32 tokens, two beside tiles of 96."""
    test_block_scaled_products([3, 40, 0, 97], 5, 136, 12288, rows, monkeypatch)


def test_block_scaled_products_where_they_pay(monkeypatch):
    """Which product runs on either side of the borders: short K, a launch for the parts alone, few stages, many rows; all of them the same numbers."""
    from batchgen_b200.ops import _ext, mxfp4
    calls = []
    block, expand = mxfp4._block_gemm, mxfp4._launch
    monkeypatch.setattr(mxfp4, "_block_gemm", lambda *a: (calls.append("block"), block(*a)))
    monkeypatch.setattr(mxfp4, "_launch", lambda *a, **k: (calls.append("expand"), expand(*a, **k)))
    g = torch.Generator().manual_seed(4)

    def product(T, N, K, E=0):
        calls.clear()
        x = torch.randn(T, K, generator=g).bfloat16()
        wq, ws = torch.randint(0, 256, (max(E, 1), N, K // 2), generator=g, dtype=torch.uint8), torch.randint(118, 124, (max(E, 1), N, K // 32), generator=g, dtype=torch.uint8)
        w = mxfp4.dequantize(wq, ws, torch.float32).double()
        if E:
            off = torch.arange(0, T + 1, T // E, dtype=torch.int32)
            rows = mxfp4.split(x.cuda()) if mxfp4.block_scaled(wq.cuda(), ws.cuda(), T / E) else x.cuda()
            got = mxfp4.grouped_mxfp4_gemm(rows, wq.cuda(), ws.cuda(), off.cuda())
            want = torch.cat([x[off[e]:off[e + 1]].double() @ w[e].t() for e in range(E)])
            mag = torch.cat([x[off[e]:off[e + 1]].double().abs() @ w[e].abs().t() for e in range(E)])
        else:
            got = mxfp4.mxfp4_gemm(x.cuda(), wq[0].cuda(), ws[0].cuda())
            want, mag = x.double() @ w[0].t(), x.double().abs() @ w[0].abs().t()
        _ext.check_status()
        assert ((got.cpu().double() - want).abs() <= want.abs() * 2 ** -8 + mag * (K * 2 ** -24 + 2.0 ** -12)).all()
        return calls[0]

    assert product(24, 256, 2048) == "expand" and product(24, 256, 2112) == "block"
    assert product(31, 256, 4096) == "expand" and product(31, 256, 4160) == "block" and product(30, 256, 4096) == "block"
    assert product(80, 256, 4160) == "block" and product(81, 256, 4160) == "expand"
    assert product(31, 256, 10112) == "block" and product(31, 256, 10176) == "expand" and product(30, 256, 10176) == "block"
    assert product(32, 256, 960, E=4) == "expand" and product(32, 256, 1024, E=4) == "block"
    if _ext.num_sms(torch.device("cuda")) == 148:
        assert product(8, 28 * 128, 192, E=8) == "block" and product(8, 27 * 128, 192, E=8) == "expand"


@pytest.mark.parametrize("above", [8, 14, 16, 20])
def test_parts_beside_an_outlier(above):
    """A first element of every 32 that dwarfs the others: elements down to 2^-14 of it are whole, smaller ones within 2^-22 of it, and no output whose weight
    for it is zero sees more than that."""
    from batchgen_b200.ops import _ext, mxfp4
    g = torch.Generator().manual_seed(above)
    T, N, K = 40, 256, 1024
    x = torch.randn(T, K, generator=g)
    x[:, ::32] = 2.0 ** above * (1 + torch.rand(T, K // 32, generator=g))
    x = x.bfloat16()
    p = mxfp4.split(x.cuda())
    parts = p.p.view(torch.float8_e4m3fn).cpu().double().transpose(1, 2).reshape(-1, 2, K)
    scale = torch.exp2(p.s.cpu().double().permute(1, 0, 2).reshape(T, -1)[:, :K // 32] - 127).repeat_interleave(32, 1)
    got, top = scale * (parts[:T, 0] + parts[:T, 1] / 32), x[:, ::32].double().repeat_interleave(32, 1)
    assert (got == x.double())[x.double().abs() >= top * 2.0 ** -14].all() and ((got - x.double()).abs() <= top * 2.0 ** -22).all()
    wq, ws = torch.randint(0, 256, (N, K // 2), generator=g, dtype=torch.uint8), torch.randint(118, 124, (N, K // 32), generator=g, dtype=torch.uint8)
    wq.view(N, K // 32, 16)[:, :, 0] &= 0xF0
    out = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    mxfp4._block_gemm(p, wq.cuda(), ws.cuda(), out, None, 1, T, N, K, None, T)
    _ext.check_status()
    w, x64 = mxfp4.dequantize(wq, ws, torch.float32).double(), x.double()
    want, mag = x64 @ w.t(), x64.abs() @ w.abs().t()
    small = torch.where(x64.abs() < top * 2.0 ** -14, top * 2.0 ** -22, 0.0)
    # one rounding to 8 bits, fp32 sums of K products, and what the parts leave out of the small elements
    assert ((out.cpu().double() - want).abs() <= want.abs() * 2 ** -8 + mag * K * 2 ** -24 + small @ w.abs().t()).all()
