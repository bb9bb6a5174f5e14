"""Later pieces of prompts: which form of MLA prefill attention a step with cached context takes, and that both agree."""
import pytest
import torch


def test_expanded_parts_group_sequences_within_a_block():
    from batchgen_b200.models.transformer import expanded_parts
    cu, ctx = [0, 1500, 1500, 2500, 4000], [5000, 700, 0, 3000]
    assert expanded_parts(cu, ctx, 16384) == [[0, 2, 3]]
    assert expanded_parts(cu, ctx, 8000) == [[0, 2], [3]]
    assert expanded_parts(cu, ctx, 6499) is None                      # the first sequence alone is longer than a block
    assert expanded_parts([0, 64], [8000], 16384) is None             # too few queries for their keys
    assert expanded_parts([0, 0], [8000], 16384) is None


@pytest.mark.parametrize("ctx", [[0, 0], [200, 0]])
def test_slots_follow_the_pages_of_a_reused_step(ctx):
    """A second step of the same lengths through one AttnMeta: the rows that are read are those of its pages then."""
    from types import SimpleNamespace
    from batchgen_b200.models.transformer import AttnMeta, Transformer
    cu, page = [0, 300, 700], 64
    need = [-(-(ctx[i] + cu[i + 1] - cu[i]) // page) for i in range(2)]
    me = SimpleNamespace(expanded_block_rows=16384)
    for name in ("_expanded_blocks", "_expanded_plan"):
        if hasattr(Transformer, name):
            setattr(me, name, getattr(Transformer, name).__get__(me))
    meta = AttnMeta(mode="prefill", positions=torch.zeros(cu[-1], dtype=torch.int32), slot_mapping=torch.zeros(cu[-1], dtype=torch.int64),
                    block_table=torch.zeros(2, max(need), dtype=torch.int32), cu_seqlens=cu, ctx_lens=ctx)
    for seed in range(3):
        order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)).int()
        for i in range(2):
            meta.block_table[i, :need[i]] = order[sum(need[:i]):sum(need[:i + 1])]
        rows = [torch.arange(ctx[i] + cu[i + 1] - cu[i]) for i in range(2)]
        want = [meta.block_table[i].long()[r // page] * page + r % page for i, r in enumerate(rows)]
        meta.slot_mapping.copy_(torch.cat([w[ctx[i]:] for i, w in enumerate(want)]))
        (slots, work), = me._expanded_blocks(meta, cu[-1], 8, page)
        assert torch.equal(slots, torch.cat(want)), seed


@pytest.mark.gpu
@pytest.mark.parametrize("block_rows", [16384, 1300])
def test_pieces_with_cached_context_take_the_expanded_form(block_rows):
    """A later piece of prompts: attention over up-projected keys and values, in one block or several, against the absorbed form and the
    same model in fp32 on the CPU."""
    from batchgen_b200.config import get_model_config
    from batchgen_b200.models import build_model
    from batchgen_b200.models.transformer import AttnMeta, Transformer
    from batchgen_b200.ops import _ext
    from batchgen_b200.runtime.kv_cache import PagedKVCache
    cfg = get_model_config("tiny-deepseek-v3", hidden_size=1024, q_lora_rank=512, kv_lora_rank=512, qk_nope_head_dim=128,
                           qk_rope_head_dim=64, v_head_dim=128, num_heads=8, intermediate_size=512, num_layers=1, first_k_dense=1,
                           vocab_size=512, quant="none")
    g = torch.Generator().manual_seed(3)
    new, ctx, page = [400, 1, 330], [777, 64, 901], 64
    need = [-(-(a + b) // page) for a, b in zip(new, ctx)]
    order = torch.randperm(sum(need), generator=g).tolist()
    bt = torch.zeros(len(new), max(need), dtype=torch.int32)
    pos, slots, cu = [], [], [0]
    past = torch.randn(sum(need), page, 576, generator=g).bfloat16()
    for i in range(len(new)):
        bt[i, :need[i]] = torch.tensor([order.pop() for _ in range(need[i])])
        t = torch.arange(ctx[i], ctx[i] + new[i])
        pos.append(t)
        slots.append(bt[i].long()[t // page] * page + t % page)
        cu.append(cu[-1] + new[i])
    ids = torch.randint(2, 512, (cu[-1],), generator=g).int()
    pos, slots = torch.cat(pos).int(), torch.cat(slots)

    def run(dev, dtype, rows):
        model = build_model(cfg, device=dev, dtype=dtype, seed=1)
        model.expanded_block_rows = rows
        kv = PagedKVCache(cfg, sum(need), page, dev, torch.float32 if dev == "cpu" else torch.bfloat16)
        kv.kv[0].copy_(past)
        meta = AttnMeta(mode="prefill", positions=pos.to(dev), slot_mapping=slots.to(dev), block_table=bt.to(dev), cu_seqlens=cu, ctx_lens=ctx)
        used = []
        if dev != "cpu":
            inner = Transformer._expanded_blocks
            model._expanded_blocks = lambda *a: used.append(inner(model, *a)) or used[-1]
        out = model.forward(ids.to(dev), meta, kv).double().cpu()
        return out, used

    want, _ = run("cpu", "fp32", 0)
    absorbed, used0 = run("cuda:0", "bf16", 0)
    expanded, used = run("cuda:0", "bf16", block_rows)
    _ext.check_status()
    assert used0 == [None] and len(used[0]) == (1 if block_rows > 2000 else 2)
    e0, e1 = ((o - want).norm() / want.norm() for o in (absorbed, expanded))
    # both round some ten intermediate tensors to bf16 (2^-9 of a value each)
    assert e1 < 2e-2 and e1 < 1.3 * e0 + 1e-3, (e0, e1)
