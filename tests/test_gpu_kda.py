"""KDA kernel (conv + gated delta rule + gated norm, prefill and decode) against the fp32 reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


def _inputs(T, H, D, seed=0):
    from batchgen_b200.ops import kda
    g = torch.Generator().manual_seed(seed)
    HD = H * D
    wide = torch.randn(T, 4 * HD + 24, generator=g).to(torch.bfloat16)     # q | k | v | z | beta (+ padding) in one buffer
    f = torch.randn(T, HD, generator=g).to(torch.bfloat16)
    p = kda.KDAParams(conv_w=torch.randn(3 * HD, 4, generator=g) * 0.5, conv_b=torch.randn(3 * HD, generator=g) * 0.1,
                      A_log=torch.randn(H, generator=g) * 0.3, dt_bias=torch.randn(HD, generator=g) * 0.3,
                      norm_w=1.0 + 0.1 * torch.randn(D, generator=g))
    return wide, f, p


def _views(wide, H, D):
    HD = H * D
    return wide[:, : 3 * HD], wide[:, 4 * HD: 4 * HD + H], wide[:, 3 * HD: 4 * HD]


@pytest.mark.parametrize("D,H", [(128, 3), (64, 4)])
def test_kda_prefill_continuation_and_decode(D, H):
    from batchgen_b200.ops import kda
    lens = [37, 1, 130]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T = cu[-1]
    wide, f, p = _inputs(T, H, D)
    slots = [2, 0, 3]
    nslots = 5
    conv_c, rec_c = torch.zeros(nslots, 3 * H * D, 3), torch.zeros(nslots, H, D, D)
    g = torch.Generator().manual_seed(5)
    rec_c[3] = torch.randn(H, D, D, generator=g) * 0.1        # sequence 2 continues from a stored state
    conv_c[3] = torch.randn(3 * H * D, 3, generator=g)
    conv_g, rec_g = conv_c.cuda(), rec_c.cuda()
    qkv, beta, z = _views(wide.float(), H, D)
    want = kda.kda_forward(qkv, f.float(), beta, z, p, conv_c, rec_c, slots, cu, [0, 0, 1], H, D, D ** -0.5, 1e-6)
    pg = kda.KDAParams(*(None if t is None else t.cuda() for t in (p.conv_w, p.conv_b, p.A_log, p.dt_bias, p.norm_w)))
    wg = wide.cuda()
    qkv_g, beta_g, z_g = _views(wg, H, D)
    got = kda.kda_forward(qkv_g, f.cuda(), beta_g, z_g, pg, conv_g, rec_g, slots, cu, [0, 0, 1], H, D, D ** -0.5, 1e-6)
    torch.cuda.synchronize()
    for i in range(3):
        assert _rel(got[cu[i]:cu[i + 1]].cpu(), want[cu[i]:cu[i + 1]]) < 2e-2, i
    assert _rel(rec_g.cpu(), rec_c) < 1e-3 and _rel(conv_g.cpu(), conv_c) < 1e-6
    assert rec_g[1].abs().max() == 0 and rec_g[4].abs().max() == 0
    # one decode step for the three sequences plus a padding row (slot -1)
    wide2, f2, _ = _inputs(4, H, D, seed=9)
    qkv2, beta2, z2 = _views(wide2.float(), H, D)
    want2 = kda.kda_forward(qkv2, f2.float(), beta2, z2, p, conv_c, rec_c, slots + [-1], None, None, H, D, D ** -0.5, 1e-6)
    w2g = wide2.cuda()
    q2g, b2g, z2g = _views(w2g, H, D)
    got2 = kda.kda_forward(q2g, f2.cuda(), b2g, z2g, pg, conv_g, rec_g,
                           torch.tensor(slots + [-1], dtype=torch.int32, device="cuda"), None, None, H, D, D ** -0.5, 1e-6)
    torch.cuda.synchronize()
    assert _rel(got2[:3].cpu(), want2[:3]) < 2e-2
    assert _rel(rec_g.cpu(), rec_c) < 1e-3


def test_model_with_kda_layers_on_gpu_matches_cpu():
    from batchgen_b200.config import EngineConfig, get_model_config
    from batchgen_b200.models import build_model
    from batchgen_b200.runtime.engine import Engine
    from batchgen_b200.runtime.sequence import SamplingParams
    from batchgen_b200.ops.policy import set_library_fallback
    cfg = get_model_config("tiny-kimi-linear")
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(2, cfg.vocab_size, (n,), generator=g).tolist() for n in (40, 9)]
    logits = {}
    set_library_fallback(True)        # the MLA layer of this preset has a test-sized latent (64): library path
    for dev, dt in (("cpu", torch.float32), ("cuda", torch.bfloat16)):
        model = build_model(cfg, device=dev, dtype=dt, seed=4)
        eng = Engine(model, EngineConfig(page_size=64, max_decode_batch=4, enable_cuda_graph=False, device=dev),
                     num_gpu_pages=16)
        seen = []
        orig = model.forward

        def spy(ids, meta, cache, _o=orig, _s=seen):
            out = _o(ids, meta, cache)
            _s.append(out.float().cpu())
            return out
        model.forward = spy
        eng.generate(prompts, SamplingParams(max_new_tokens=3, temperature=0.0, ignore_eos=True))
        logits[dev] = seen
    set_library_fallback(False)
    # prefill logits and the first decode step (same tokens fed as long as greedy picks agree; compare what is comparable)
    assert _rel(logits["cuda"][0], logits["cpu"][0]) < 0.06


def _recurrence64(qkv, f, beta, z, p, conv, rec, slots, cu, has, H, D, scale, eps):
    """The recurrence token by token in 64 bits; conv and rec [slots, ..] are updated."""
    HD = H * D
    out = torch.zeros(qkv.shape[0], HD, dtype=torch.float64)
    d = lambda t: t.double().cpu()  # noqa: E731
    w, b, A, dt, nw = d(p.conv_w), d(p.conv_b), d(p.A_log), d(p.dt_bias), d(p.norm_w)
    for i, s in enumerate(slots):
        a, e = cu[i], cu[i + 1]
        if s < 0 or e <= a:
            continue
        if not has[i]:
            conv[s].zero_()
            rec[s].zero_()
        full = torch.cat([conv[s].t(), d(qkv[a:e])], 0)
        y = torch.nn.functional.silu(sum(full[j:j + e - a] * w[:, j] for j in range(4)) + b)
        conv[s] = full[-3:].t()
        q, k, v = (t.view(-1, H, D) for t in y.chunk(3, -1))
        q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * scale
        k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        g = (-A.exp().view(1, H, 1) * torch.nn.functional.softplus(d(f[a:e]) + dt).view(-1, H, D)).exp()
        bt, S = d(beta[a:e]).sigmoid(), rec[s].clone()
        o = torch.empty(e - a, H, D, dtype=torch.float64)
        for t in range(e - a):
            S *= g[t].unsqueeze(-1)
            S += k[t].unsqueeze(-1) * (bt[t].unsqueeze(-1) * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))).unsqueeze(-2)
            o[t] = torch.einsum("hkv,hk->hv", S, q[t])
        rec[s] = S
        o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + eps) * nw
        out[a:e] = (o * d(z[a:e]).view(-1, H, D).sigmoid()).reshape(-1, HD)
    return out


@pytest.mark.parametrize("decay", ["slow", "mixed", "fast"])
@pytest.mark.parametrize("scratch", [1 << 30, 7 << 20])
def test_chunk_form_against_64_bits(decay, scratch, monkeypatch):
    """Pieces at the edges of chunks and blocks, fresh and continued, one without a slot, several rounds; the chunk form is as near to
    64 bits as the token-by-token form."""
    from batchgen_b200.ops import kda
    H, D = 3, 128
    HD = H * D
    g = torch.Generator().manual_seed(5)
    lens = [1, 47, 48, 63, 64, 65, 3, 127, 128, 129, 300, 50, 80]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T, B = cu[-1], len(lens)
    slots = [i if i != 11 else -1 for i in range(B)]
    has = [i % 2 for i in range(B)]
    qkv, z = torch.randn(T, 3 * HD, generator=g).bfloat16(), torch.randn(T, HD, generator=g).bfloat16()
    f, beta = torch.randn(T, HD, generator=g).bfloat16(), (torch.randn(T, H, generator=g) * 2).bfloat16()
    A = {"slow": torch.full((H,), -4.0), "mixed": torch.tensor([-3.0, 0.0, 2.7]), "fast": torch.full((H,), 4.5)}[decay]
    p = kda.KDAParams(*(t.cuda() for t in (torch.randn(3 * HD, 4, generator=g) * 0.5, torch.randn(3 * HD, generator=g) * 0.1, A,
                                           torch.randn(HD, generator=g) - 1, 1 + 0.1 * torch.randn(D, generator=g))))
    conv0, rec0 = torch.randn(B, 3 * HD, 3, generator=g).bfloat16().float(), torch.randn(B, H, D, D, generator=g) * 0.3
    conv64, rec64 = conv0.double(), rec0.double()
    want = _recurrence64(qkv, f, beta, z, p, conv64, rec64, slots, cu, has, H, D, D ** -0.5, 1e-6)
    monkeypatch.setattr(kda, "_CHUNK_SCRATCH", scratch)
    monkeypatch.setattr(kda, "chunk_form_pays", lambda lens, heads, sms: bool(lens))
    err = {}
    for form, least in (("chunks", kda.CHUNK_MIN_TOKENS), ("tokens", 1 << 30)):
        monkeypatch.setattr(kda, "CHUNK_MIN_TOKENS", least)
        conv, rec = conv0.cuda(), rec0.cuda()
        out = kda.kda_forward(qkv.cuda(), f.cuda(), beta.cuda(), z.cuda(), p, conv, rec, slots, cu, has, H, D, D ** -0.5, 1e-6)
        torch.cuda.synchronize()
        live = torch.ones(T, dtype=torch.bool)
        live[cu[11]:cu[12]] = False
        assert torch.equal(conv.cpu().double(), conv64)
        assert torch.equal(rec[11].cpu(), rec0[11])
        d = (out.cpu().double() - want)[live]
        err[form] = ((rec.cpu().double() - rec64).norm() / rec64.norm()).item(), (d.norm() / want[live].norm()).item()
        # a value rounded to 8 significant bits; the recurrence in fp32
        assert (d.abs() <= want[live].abs() * 2 ** -8 + 2e-4).all(), (form, d.abs().max())
    assert err["chunks"][0] <= 1.5 * err["tokens"][0] + 1e-7 and err["chunks"][1] <= 1.02 * err["tokens"][1], err


def _prompt(H, lens, seed, f=None):
    """One set of pieces, fresh and continued in turn, heads of 128: inputs, parameters, states."""
    from batchgen_b200.ops import kda
    HD = H * 128
    g = torch.Generator().manual_seed(seed)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    T, B = cu[-1], len(lens)
    qkv, z = torch.randn(T, 3 * HD, generator=g).bfloat16(), torch.randn(T, HD, generator=g).bfloat16()
    if f is None:
        f = torch.randn(T, HD, generator=g).bfloat16()
    beta = (torch.randn(T, H, generator=g) * 2).bfloat16()
    p = [torch.randn(3 * HD, 4, generator=g) * 0.5, torch.randn(3 * HD, generator=g) * 0.1, torch.full((H,), 4.5),
         torch.zeros(HD), 1 + 0.1 * torch.randn(128, generator=g)]
    conv, rec = torch.randn(B, 3 * HD, 3, generator=g).bfloat16().float(), torch.randn(B, H, 128, 128, generator=g) * 0.3
    return cu, list(range(B)), [i % 2 for i in range(B)], qkv, z, f, beta, kda.KDAParams(*(t.cuda() for t in p)), conv, rec


def _both_forms(monkeypatch, cu, slots, has, qkv, z, f, beta, p, conv0, rec0, H):
    from batchgen_b200.ops import kda
    monkeypatch.setattr(kda, "chunk_form_pays", lambda lens, heads, sms: bool(lens))
    out = {}
    for form, least in (("chunks", 48), ("tokens", 1 << 30)):
        monkeypatch.setattr(kda, "CHUNK_MIN_TOKENS", least)
        conv, rec = conv0.cuda(), rec0.cuda()
        o = kda.kda_forward(qkv.cuda(), f.cuda(), beta.cuda(), z.cuda(), p, conv, rec, slots, cu, has, H, 128, 128 ** -0.5, 1e-6)
        out[form] = o.cpu().double(), conv.cpu().double(), rec.cpu().double()
    return out


def test_chunk_form_with_strong_and_weak_decays_in_turn(monkeypatch):
    """Channels where a token forgets everything (2^-400) beside ones that forget almost nothing (2^-0.001): the weak decays behind a strong
    one count with their own precision, as token by token."""
    H, lens = 3, [64, 129, 300]
    g = torch.Generator().manual_seed(11)
    shape = (sum(lens), H * 128)
    f = torch.where(torch.rand(shape, generator=g) < 0.4, torch.rand(shape, generator=g) * 3 + 2, -8 - 6 * torch.rand(shape, generator=g)).bfloat16()
    cu, slots, has, qkv, z, f, beta, p, conv0, rec0 = _prompt(H, lens, 12, f)
    conv64, rec64 = conv0.double(), rec0.double()
    want = _recurrence64(qkv, f, beta, z, p, conv64, rec64, slots, cu, has, H, 128, 128 ** -0.5, 1e-6)
    err = {}
    for form, (o, conv, rec) in _both_forms(monkeypatch, cu, slots, has, qkv, z, f, beta, p, conv0, rec0, H).items():
        assert torch.equal(conv, conv64)
        err[form] = ((rec - rec64).norm() / rec64.norm()).item(), ((o - want).norm() / want.norm()).item()
    print(err)
    assert err["chunks"][0] <= 1.5 * err["tokens"][0] + 1e-7 and err["chunks"][1] <= 1.02 * err["tokens"][1], err


@pytest.mark.parametrize("where", ["f", "q", "k", "v", "beta"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [0, 9, 15, 16, 40, 63, 64, 100])
def test_chunk_form_keeps_what_is_not_finite_to_later_tokens(where, value, at, monkeypatch):
    """A value that is not finite at one token: the tokens before it are what they are without it, and a NaN is passed on wherever it is token
    by token.  (An infinite decay input forgets everything and harms nothing.)"""
    H, lens = 2, [130]
    cu, slots, has, qkv, z, f, beta, p, conv0, rec0 = _prompt(H, lens, 13)
    p.A_log.fill_(-1.0)
    clean = _both_forms(monkeypatch, cu, slots, has, qkv, z, f, beta, p, conv0, rec0, H)["chunks"][0]
    {"f": f, "q": qkv[:, :256], "k": qkv[:, 256:512], "v": qkv[:, 512:], "beta": beta}[where][at, 1] = value
    form = _both_forms(monkeypatch, cu, slots, has, qkv, z, f, beta, p, conv0, rec0, H)
    (o, _, rec), (ot, _, rect) = form["chunks"], form["tokens"]
    assert torch.equal(o[:at], clean[:at])
    assert (torch.isnan(o) | ~torch.isnan(ot)).all() and (torch.isnan(rec) | ~torch.isnan(rect)).all()
    if where == "f" and value == float("inf"):
        assert torch.isfinite(o).all() and torch.isfinite(rec).all()


def test_one_plan_serves_the_layers_of_a_step(monkeypatch):
    """Three KDA layers of a prompt step: its lengths go to the device once; another step makes its own plan."""
    from batchgen_b200.config import get_model_config
    from batchgen_b200.models import build_model
    from batchgen_b200.models.transformer import AttnMeta
    from batchgen_b200.ops import kda
    from batchgen_b200.ops.policy import set_library_fallback
    from batchgen_b200.runtime.kv_cache import PagedKVCache
    cfg = get_model_config("tiny-kimi-linear", kda_head_dim=128, kda_num_heads=4)
    made = []
    inner = kda.step_plan
    monkeypatch.setattr(kda, "step_plan", lambda cu, *a: made.append(list(cu)) or inner(cu, *a))
    set_library_fallback(True)
    try:
        model = build_model(cfg, device="cuda", dtype=torch.bfloat16, seed=4)
        kv = PagedKVCache(cfg, 16, 64, "cuda", torch.bfloat16, state_slots=2)
        meta, got = None, []
        for lens in ([200, 70], [200, 70], [20, 90]):
            T = sum(lens)
            pos = torch.cat([torch.arange(n) for n in lens]).int().cuda()
            table = torch.arange(8, dtype=torch.int32).view(2, 4).cuda()
            slots = torch.cat([table[i].cpu().long()[torch.arange(n) // 64] * 64 + torch.arange(n) % 64 for i, n in enumerate(lens)]).cuda()
            new = dict(positions=pos, slot_mapping=slots, block_table=table, cu_seqlens=[0, lens[0], T], ctx_lens=[0, 0])
            if meta is None:
                meta = AttnMeta(mode="prefill", state_slots=torch.tensor([0, 1], dtype=torch.int32).cuda(),
                                state_has_initial=torch.zeros(2, dtype=torch.int32).cuda(), **new)
            for k, v in new.items():                     # the same AttnMeta, reused
                setattr(meta, k, v)
            ids = (torch.arange(T, dtype=torch.int32) % 50 + 2).cuda()
            got.append(model.forward(ids, meta, kv).float().cpu())
            alone = AttnMeta(mode="prefill", state_slots=meta.state_slots, state_has_initial=meta.state_has_initial, **new)
            assert torch.equal(got[-1], model.forward(ids, alone, kv).float().cpu())
        torch.cuda.synchronize()
    finally:
        set_library_fallback(False)
    a, b = [0, 200, 270], [0, 20, 110]
    assert made == [a, a, a, b, b], made                 # first step, its twin; twin of the second; third and its twin
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("lens,shift", [([64, 65], 0), ([130, 48, 200], 1), ([192], 4)])
def test_chunk_form_of_unaligned_rows(lens, shift, monkeypatch):
    """Inputs as columns of a wider projection: rows that are and are not in 16-byte pieces give the same numbers; the state's columns of both CTAs of a head."""
    from batchgen_b200.ops import kda
    H = 2
    cu, slots, has, qkv, z, f, beta, p, conv0, rec0 = _prompt(H, lens, 21)
    monkeypatch.setattr(kda, "chunk_form_pays", lambda lens, heads, sms: bool(lens))
    got = []
    for wide in (False, True):
        conv, rec = conv0.cuda(), rec0.cuda()
        q, ff = qkv.cuda(), f.cuda()
        if wide:
            q = torch.zeros(q.shape[0], q.shape[1] + 5 + shift, dtype=q.dtype, device="cuda")[:, shift:shift + q.shape[1]].copy_(q)
            ff = torch.zeros(ff.shape[0], ff.shape[1] + 3, dtype=q.dtype, device="cuda")[:, 1:1 + ff.shape[1]].copy_(ff)
        o = kda.kda_forward(q, ff, beta.cuda(), z.cuda(), p, conv, rec, slots, cu, has, H, 128, 128 ** -0.5, 1e-6)
        got.append((o, conv, rec))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    conv64, rec64 = conv0.double(), rec0.double()
    want = _recurrence64(qkv, f, beta, z, p, conv64, rec64, slots, cu, has, H, 128, 128 ** -0.5, 1e-6)
    o, _, rec = got[0]
    # a value rounded to 8 significant bits; the recurrence in fp32
    assert ((o.cpu().double() - want).abs() <= want.abs() * 2 ** -8 + 2e-4).all()
    for half in (rec[..., :64], rec64.cuda()[..., :64]), (rec[..., 64:], rec64.cuda()[..., 64:]):
        assert (half[0].double() - half[1]).norm() <= 5e-7 * half[1].norm()


def _one_write(H, bias_v, dt_bias, A_log, f_token, form, monkeypatch, last=None):
    """A piece of 64 tokens of which the last alone has a key, the first unit vector with weight one, or (``f_token`` zero) a decay, on a state of zeros or
    ones: afterwards row 0 of the state is SiLU(bias_v), or row i the decay of channel i.  ``last``: values of the last token itself, to which bias_v is added."""
    from batchgen_b200.ops import kda
    T, HD = 64, H * 128
    monkeypatch.setattr(kda, "chunk_form_pays", lambda lens, heads, sms: bool(lens) and form == "chunks")
    qkv = torch.zeros(T, 3 * HD, dtype=torch.bfloat16, device="cuda")
    if f_token != 0:
        qkv[-1, HD:2 * HD:128] = 32.0
    if last is not None:
        qkv[-1, 2 * HD:] = last.flatten().cuda()
    w = torch.zeros(3 * HD, 4, device="cuda")
    w[:, 3] = 1.0
    bias = torch.zeros(3 * HD, device="cuda")
    bias[2 * HD:] = bias_v.flatten().cuda()
    f = torch.full((T, HD), -1e5, dtype=torch.bfloat16, device="cuda")           # no decay
    f[-1] = f_token
    p = kda.KDAParams(conv_w=w, conv_b=bias, A_log=A_log.cuda(), dt_bias=dt_bias.flatten().cuda(), norm_w=torch.ones(128, device="cuda"))
    rec = torch.ones(1, H, 128, 128, device="cuda") if f_token == 0 else torch.zeros(1, H, 128, 128, device="cuda")
    kda.kda_forward(qkv, f, torch.full((T, H), 100.0, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, HD, dtype=torch.bfloat16, device="cuda"), p,
                    torch.zeros(1, 3 * HD, 3, device="cuda"), rec, [0], [0, T], [1], H, 128, 1.0, 1e-6)
    return rec[0].cpu()


def _arguments(n, seed):
    """Floats around the borders of the formulas, and of every size."""
    g = torch.Generator().manual_seed(seed)
    edge = torch.tensor([0.0, 40.0, 20.0, 1.0, 0.6931472, 16.0, 88.0, 87.33, 86.0, 5.0, 2.0 ** -126, 2.0 ** -100, 2.0 ** -24, 2.0 ** -12, 1e-3, 64.0])
    near = torch.cat([edge, torch.nextafter(edge, edge + 1), torch.nextafter(edge, edge - 1), edge * (1 + 2.0 ** -20)])
    size = torch.exp2(torch.rand(n, generator=g) * 40 - 33)                      # up to 2^7
    x = torch.cat([near, -near, size * (1 - 2 * torch.randint(0, 2, (n,), generator=g))])[:n]
    x[0] = 64.0                                                                  # SiLU is the number itself
    return x


def test_silu_of_the_chunk_form(monkeypatch):
    """The chunk form's quotient against the token form's division: the same float or its neighbour; both against 64 bits."""
    H = 96
    x = _arguments(H * 128, 1).view(H, 128)
    x[:, 0] = 64.0
    none, A = torch.zeros(H, 128), torch.zeros(H)
    got = {form: _one_write(H, x, none, A, -1e5, form, monkeypatch)[:, 0] for form in ("chunks", "tokens")}
    x64 = x.double()
    want = x64 / (1 + (-x64).exp())
    whole = want.abs() >= 2.0 ** -100             # all three parts of the state's number are normal floats
    for y in got.values():
        assert (y[:, 0] == 64).all()                                             # the key is exactly one
        # e^-x off by 2 + 1.173 |x| units (CUDA's bound), the sum and the quotient by one each
        rel = ((2 + 1.173 * x64.abs()) * (-x64).exp() / (1 + (-x64).exp()) + 2) * 2.0 ** -23
        assert ((y.double() - want).abs()[whole] <= (rel * want.abs())[whole]).all()
        assert ((y.double() - want).abs()[~whole] <= 2.0 ** -100).all()
    a, b = got["chunks"][whole], got["tokens"][whole]
    assert ((a == b) | (torch.nextafter(a, b) == b)).all()
    assert whole.sum() > 0.9 * whole.numel()


def test_silu_of_the_chunk_form_not_finite(monkeypatch):
    """Infinities and NaN leave the formula as they leave the token form's division, and no other column is touched."""
    x = torch.ones(1, 128)
    x[0, 3], x[0, 70], x[0, 71], x[0, 90], x[0, 127] = float("inf"), float("nan"), -float("inf"), -300.0, 3e38
    none = torch.zeros(1, 128)
    a, b = (_one_write(1, none, none, torch.zeros(1), -1e5, form, monkeypatch, last=x)[0, 0] for form in ("chunks", "tokens"))
    assert a[3] == b[3] == float("inf") and a[[70, 71]].isnan().all() and b[[70, 71]].isnan().all() and a[90] == b[90] == 0 and a[127] == b[127]
    fine = torch.ones(128, dtype=torch.bool)
    fine[[3, 70, 71, 90, 127]] = False
    assert (a[fine] == a[0]).all() and abs(float(a[0]) - 0.7310586) < 1e-6


def test_softplus_of_the_chunk_form(monkeypatch):
    """Decays of one token over 2^-110 to 2^12 of softplus: the series within the bounds of its exponential, and no further from 64 bits than log1p(e^x)."""
    lo, hi = -110, 12
    H = hi - lo
    g = torch.Generator().manual_seed(2)
    top = torch.exp2(torch.arange(lo, hi).double()).view(H, 1)
    sp = top * (1 + torch.rand(H, 128, generator=g).double())                    # softplus wanted
    x = torch.where(sp > 30, sp, torch.expm1(sp.clamp(max=30)).log()).float()
    x64, a64 = x.double(), (4 - torch.arange(lo, hi).double()).view(H, 1) * math.log(2.0)                        # exponents of some 16 to 32
    A = a64.float().flatten()
    sp = x64.clamp_min(0) + torch.log1p((-x64.abs()).exp())
    err = {}
    for form in ("chunks", "tokens"):
        S = _one_write(H, torch.zeros(H, 128), x, A, 0.0, form, monkeypatch)[:, :, 5].double()
        e = (-S.log() / A.double().exp().view(H, 1) / sp - 1).abs()
        part = torch.log1p((-x64.abs()).exp()) / sp                               # the exponential's share of the sum
        # __expf off by 2 + 1.173 |x| units (CUDA's bound) in both places, eight roundings, ex2 off by two units of a state, which stands for 16 of the exponent
        units = (2 + 1.173 * x64.abs()) * part + 2 + 1.173 * a64.abs() + 8 + 1
        if form == "chunks":
            assert (e <= units * 2.0 ** -23).all()
        err[form] = e.square().mean().sqrt()
    assert err["chunks"] <= 1.05 * err["tokens"]
