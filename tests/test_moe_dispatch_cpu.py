"""Which bf16 kernel a product takes: grouped ones by the rows that are expected on this rank, not by the capacity of the buffer; dense ones
by their tiles, unless a few tokens stream the weights."""
from types import SimpleNamespace

import pytest
import torch

from batchgen_b200.ops import gemm, moe
from batchgen_b200.parallel import comm


@pytest.mark.parametrize("capacity,hint,swapped", [(200, None, True), (100, None, False), (200, 127.0, False), (1000, 128.0, True), (1000, 13.0, False)])
def test_grouped_kernel_by_expected_rows(capacity, hint, swapped, monkeypatch):
    taken = []
    monkeypatch.setattr(gemm, "_bf16_swap", lambda *a, **k: taken.append(True))
    monkeypatch.setattr(gemm, "_launch", lambda *a, **k: taken.append(False))
    E = 4
    x, w = torch.empty(E * capacity, 64).bfloat16(), torch.empty(E, 32, 64).bfloat16()
    gemm.grouped_bf16_gemm(x, w, None, None, rows_hint=None if hint is None else hint * E)
    assert taken == [swapped]


@pytest.mark.parametrize("replicated", [True, False])
def test_expert_parallel_rank_expects_its_share(replicated, monkeypatch):
    """8 ranks of 4 experts each: an eighth of the step's pairs."""
    T, K, H, E, W = 64, 3, 16, 32, 8
    seen = []

    def grouped(xq, xs, offsets, ew, x_dense=None, rows_hint=None, **kw):
        seen.append(rows_hint)
        return torch.zeros(x_dense.shape[0], H)

    monkeypatch.setattr(moe, "grouped_experts", grouped)
    me = SimpleNamespace(world=W, rank=2, tp_reduce=lambda x: x, all_gather_rows=lambda x: x, reduce_scatter_rows=lambda x: x)
    idx = torch.stack([torch.randperm(E)[:K] for _ in range(T)]).int()
    ew = moe.ExpertWeights(torch.zeros(E // W, 2 * 8, H), torch.zeros(E // W, H, 8))
    comm.NcclComm.moe(me, torch.randn(T, H), idx, torch.rand(T, K), ew, E, replicated=replicated)
    moe.experts_forward(torch.randn(T, H), idx, torch.rand(T, K), moe.ExpertWeights(torch.zeros(E, 16, H), torch.zeros(E, H, 8)), 0, E)
    assert seen == [T * K / W, T * K]


@pytest.mark.parametrize("T,N,K,swapped", [(4096, 16576, 2304, True), (1024, 4096, 2880, True), (300, 2304, 4096, False), (1, 14208, 2304, True),
                                           (1, 14080, 2304, False), (28, 16576, 2304, True), (29, 16576, 2304, False), (128, 16576, 2304, False),
                                           (129, 16576, 2304, True), (9, 16384, 7168, True), (10, 16384, 7168, False), (128, 32768, 512, True),
                                           (64, 16384, 1472, True), (64, 16384, 1536, False), (512, 16384, 96, False)])
def test_dense_kernel_by_tiles_and_tokens(T, N, K, swapped):
    assert gemm.swap_dense(T, N, K, 148) == swapped


@pytest.mark.parametrize("T,N,K,pairs", [(4096, 16576, 2304, True), (4096, 16576, 512, True), (4096, 16576, 448, False), (2500, 2304, 4096, False), (4650, 2880, 4096, False),
                                         (37 * 256, 1024, 704, True), (36 * 256, 1024, 704, False)])
def test_dense_pairs_by_tiles_and_k(T, N, K, pairs):
    assert gemm.use_pairs(T, N, 148, K) == pairs


@pytest.mark.parametrize("rows,groups,N,K,pairs", [(128, 256, 2048, 2304, True), (128, 256, 2304, 512, True), (128, 256, 2304, 448, False), (200, 8, 2048, 2304, True),
                                                   (200, 8, 2048, 2240, False), (300, 64, 304, 1536, False), (256, 37, 512, 1024, True), (256, 36, 512, 1024, False),
                                                   (257, 19, 512, 1024, True)])
def test_grouped_pairs_by_tiles_and_k(rows, groups, N, K, pairs):
    assert gemm.use_pairs_grouped(rows, groups, N, K, 148) == pairs
