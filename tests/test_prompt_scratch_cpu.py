"""The memory plan knows what a layer of a prompt takes beside its activations."""
import pytest
import torch

from batchgen_b200.config import EngineConfig, get_model_config
from batchgen_b200.ops import kda
from batchgen_b200.runtime import planner


@pytest.mark.parametrize("lens,heads,budget", [([16384], 32, 1 << 30), ([48] * 300, 8, 1 << 30), ([300, 1000, 65], 4, 1 << 26), ([64], 300, 1 << 20)])
def test_kda_scratch_is_bounded_by_the_plan(lens, heads, budget, monkeypatch):
    monkeypatch.setattr(kda, "_CHUNK_SCRATCH", budget)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    rounds = kda.chunk_plan(cu, kda.CHUNK_MIN_TOKENS, max(1, budget // (4 * kda._CHUNK_FLOATS * heads)))
    taken = max(len(items) for items, _ in rounds) * heads * kda._CHUNK_FLOATS * 4
    assert taken <= kda.chunk_scratch_bytes(cu[-1], heads, 128) <= max(budget, heads * kda._CHUNK_FLOATS * 4)
    assert kda.chunk_scratch_bytes(cu[-1], heads, 64) == 0          # 64-wide heads go token by token


@pytest.mark.parametrize("name,least", [("kimi-linear-48b", 1 << 29), ("deepseek-v3", 1 << 30), ("gpt-oss-120b", 0)])
def test_plan_holds_the_scratch_of_a_prompt(name, least, monkeypatch):
    cfg = get_model_config(name)
    ecfg = EngineConfig(max_prefill_tokens=16384)
    scratch = planner.prompt_scratch_bytes(cfg, ecfg)
    assert scratch >= least and (least > 0 or scratch == 0)
    plan = planner.plan_deployment(cfg, ecfg, planner.MACHINES["b200"])
    monkeypatch.setattr(planner, "prompt_scratch_bytes", lambda *a: 0)
    assert plan.workspace_bytes - planner.plan_deployment(cfg, ecfg, planner.MACHINES["b200"]).workspace_bytes == scratch
    # the pool on the live machine leaves it too
    pages = {}
    for s in (0, 1 << 30):
        monkeypatch.setattr(planner, "prompt_scratch_bytes", lambda *a, s=s: s)
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: (100 << 30, 180 << 30))
        pages[s] = planner.size_kv_pool(cfg, ecfg, "cuda:0", torch.bfloat16)[0]
    per_page = cfg.kv_bytes_per_token(2) * ecfg.page_size
    assert abs((pages[0] - pages[1 << 30]) * per_page - (1 << 30)) <= per_page
