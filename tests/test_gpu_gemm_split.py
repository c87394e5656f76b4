"""GEMMs whose output is a few tiles: clusters of two or four CTA pairs share a tile's contraction and exchange partial tiles through
distributed shared memory. Ragged rows, contractions that do not divide by the split, every operand order and epilogue."""

import math

import pytest
import torch

from cosmos_predict25_b200.ops import functional as F_ops
from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUND = 1.5 * 2.0 ** -9        # one bf16 rounding of the result in the 2-norm


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _clusters():
    """Pairs, and clusters of two, four and three pairs, that this GPU holds at once."""
    return native.load().gemm_clusters(torch.cuda.current_device())


def _check():
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 0


# tiles x k-blocks: below the split's limit, both splits, uneven shares (9, 13, 33 blocks), more tiles than half the pairs (no split)
@pytest.mark.parametrize("M,N,K", [(256, 256, 448), (256, 256, 576), (264, 512, 832), (520, 2048, 2048), (512, 2048, 8192), (1000, 1024, 2112),
                                   (2056, 1024, 1536), (2304, 1024, 2048), (7040, 2048, 1024)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False), (True, True)])
def test_operand_orders(M, N, K, trans_a, trans_b):
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) / math.sqrt(K)).bfloat16()
    want = a.double() @ b.double().t()
    args = (a.t().contiguous() if trans_a else a, b.t().contiguous() if trans_b else b, None, 0, trans_a, trans_b)
    got = native.load().gemm_bf16(*args)
    again = native.load().gemm_bf16(*args)
    _check()
    assert _rel(got, want) < ROUND and torch.equal(got, again)


@pytest.mark.parametrize("M,N,K", [(264, 512, 832), (512, 1024, 4096), (2048, 512, 640)])
def test_epilogues(M, N, K):
    torch.manual_seed(1)
    ops = native.load()
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) / math.sqrt(K)).bfloat16()
    bias = torch.randn(N, device=DEV).bfloat16()
    L = 8
    gate = torch.randn(M // L, 3 * N, device=DEV)[:, N:2 * N]
    resid = torch.randn(M, N, device=DEV).bfloat16()
    prod = a.double() @ b.double().t()
    pre_want = prod + bias.double()
    y, pre = ops.gemm_bf16_gelu_pre(a, b, bias)
    out, p = ops.gemm_bf16_gate_residual_pre(a, b, resid, gate, L)
    only = ops.gemm_bf16_gate_residual(a, b, resid, gate, L)
    _check()
    assert _rel(pre, pre_want) < ROUND and _rel(y, torch.nn.functional.gelu(pre_want)) < ROUND
    sum_want = resid.double() + gate.double().repeat_interleave(L, 0) * prod
    assert _rel(p, prod) < ROUND and _rel(out, sum_want) < ROUND and torch.equal(out, only)


# 18 and 20 tiles: no room for clusters of four pairs in one wave, so three pairs share a tile; shares of 13 to 15 and 43 k-blocks, ragged rows
@pytest.mark.parametrize("M,N,K", [(768, 1536, 8256), (1000, 1280, 2624), (904, 1280, 2752)])
def test_three_pairs(M, N, K):
    torch.manual_seed(2)
    ops = native.load()
    _, c2, c4, c3 = _clusters()
    assert ops.gemm_pairs_per_tile(-(-M // 256) * (N // 256), K // 64, 74, c2, c4, c3) == 3
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) / math.sqrt(K)).bfloat16()
    L = 8
    gate = torch.randn(M // L, 3 * N, device=DEV)[:, N:2 * N]
    resid = torch.randn(M, N, device=DEV).bfloat16()
    prod = a.double() @ b.double().t()
    got, again = ops.gemm_bf16(a, b, None, 0, False, False), ops.gemm_bf16(a, b, None, 0, False, False)
    out, p = ops.gemm_bf16_gate_residual_pre(a, b, resid, gate, L)
    _check()
    assert _rel(got, prod) < ROUND and torch.equal(got, again) and torch.equal(p, got)
    assert _rel(out, resid.double() + gate.double().repeat_interleave(L, 0) * prod) < ROUND


# The gated residual of several tiles per pair: the rows of the next tile are fetched while this one is finished; gates that change
# inside a warp's rows, a last row tile that is mostly empty
@pytest.mark.parametrize("M,N,K,L", [(7040, 2048, 128, 3520), (19208, 1024, 192, 8), (20000, 1024, 64, 40)])
def test_gated_tiles_in_a_row(M, N, K, L):
    torch.manual_seed(3)
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) / math.sqrt(K)).bfloat16()
    gate = torch.randn(M // L, 3 * N, device=DEV)[:, 2 * N:]
    resid = torch.randn(M, N, device=DEV).bfloat16()
    got = native.load().gemm_bf16_gate_residual(a, b, resid, gate, L)
    _check()
    assert _rel(got, resid.double() + gate.double().repeat_interleave(L, 0) * (a.double() @ b.double().t())) < ROUND


# Tiles whose k-blocks are shared out over all pairs: one tile for all of them, several pairs a tile with none left over for the tail, a tail
# whose pairs reach into two and three tiles, more tiles than half of the pairs; ragged rows, a last k-block of 8. `shared`: what the rule says
# for every GPU that holds 70 pairs and more; None: it depends on the clusters that the GPU holds.
@pytest.mark.parametrize("M,N,K,shared", [(256, 256, 65536, True), (300, 512, 32768, True), (1000, 1024, 65536, None), (2500, 1024, 65536, None),
                                          (1280, 2304, 32768, True), (520, 768, 32776, True), (256, 256, 16384, False), (2304, 1024, 16384, None)])
@pytest.mark.parametrize("bias,act", [(False, 0), (True, 0), (True, 1)])
def test_long_contractions_are_shared_over_all_pairs(M, N, K, shared, bias, act):
    ops = native.load()
    pairs, c2, c4, c3 = _clusters()
    taken = ops.gemm_stream_plan(-(-M // 256) * (N // 256), -(-K // 64), pairs, c2, c4, c3)[0]
    if shared is not None:
        assert taken == shared
    assert ops.gemm_launches(M, N, K) == (2 if taken else 1)
    torch.manual_seed(5)
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) / K ** 0.5).bfloat16()
    store = torch.randn(N + 1, device=DEV).bfloat16()
    b = store[1:] if bias else None                     # two bytes off a 16-byte boundary
    y = ops.gemm_bf16(x, w, b, act, False, False)
    again = ops.gemm_bf16(x, w, b, act, False, False)
    torch.cuda.synchronize()
    assert ops.kernel_error(torch.cuda.current_device(), True) == 0
    assert torch.equal(y, again)
    want = x.double() @ w.double().t()
    if bias:
        want = want + b.double()
    pre = want
    if act:
        want = torch.nn.functional.gelu(want)
    # one rounding to bf16; fp32 sums of 65,536 products of unit variance over sqrt(K) stay at 1e-6 of it
    assert ((y.double() - want).norm() / want.norm()).item() < 1.5 * 2.0 ** -9
    if act:
        y2, got_pre = ops.gemm_bf16_gelu_pre(x, w, b)
        assert torch.equal(y2, y) and ((got_pre.double() - pre).norm() / pre.norm()).item() < 1.5 * 2.0 ** -9


def test_shared_contraction_counts_both_kernels():
    """The sums of all pairs are added by a kernel of its own, which the launch count includes; ordinary products are one launch."""
    for M, N, K, act in ((512, 512, 65536, "none"), (512, 512, 65536, "gelu"), (512, 512, 1024, "none"), (512, 512, 8192, "gelu")):
        x = torch.randn(M, K, device=DEV).bfloat16().requires_grad_(act == "gelu")
        w = torch.randn(N, K, device=DEV).bfloat16()
        before = native.launches()
        F_ops.linear(x, w, None, act)
        assert native.launches() - before == (2 if K == 65536 else 1)
    _check()
