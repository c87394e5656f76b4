"""GEMMs over several weights of one input in one launch (the context's keys and values, a block's q, k and v): partial N tiles inside a
group, ragged rows, and groups whose tiles are few enough that clusters of CTA pairs share their contraction."""

import math
from dataclasses import replace

import pytest
import torch

from cosmos_predict25_b200.models import dit
from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUND = 1.5 * 2.0 ** -9        # one bf16 rounding of the result in the 2-norm


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _split(tiles, k_blocks):
    """CTA pairs per tile for the clusters that this GPU holds."""
    _, c2, c4, c3 = native.load().gemm_clusters(torch.cuda.current_device())
    return native.load().gemm_pairs_per_tile(tiles, k_blocks, 74, c2, c4, c3)


# (batch, tokens, context width, model width, CTA pairs per tile): below one launch; unsplit with whole and partial N tiles; every split;
# ragged rows; more tiles than half the pairs.
@pytest.mark.parametrize("B,S,C,D,split", [(2, 40, 512, 256, 1), (1, 256, 512, 256, 1), (2, 512, 512, 1024, 1), (2, 512, 1024, 2048, 1),
                                           (1, 256, 1024, 1024, 4), (1, 512, 1024, 2048, 2), (1, 264, 1024, 512, 4), (1, 264, 2048, 384, 1),
                                           (1, 520, 640, 640, 1), (3, 88, 2112, 256, 4)])
def test_keys_and_values_of_all_blocks(B, S, C, D, split):
    torch.manual_seed(0)
    ops = native.load()
    tiles = -(-B * S // 256) * -(-D // 256) * 2
    if D % 256 == 0 and B * S >= 256:
        assert _split(tiles, C // 64) == split
    ctx = torch.randn(B, S, C, device=DEV).bfloat16()
    widths = (D, 128, D)                                       # blocks of another width between
    ws = []
    for d in widths:
        ws += [(torch.randn(d, C, device=DEV) / math.sqrt(C)).bfloat16() for _ in range(2)] + [(1 + 0.2 * torch.randn(128, device=DEV)).bfloat16()]
    got, again = ops.dit_context_kv(ctx, ws, 1e-6), ops.dit_context_kv(ctx, ws, 1e-6)
    torch.cuda.synchronize()
    assert ops.kernel_error(0, True) == 0
    for i, d in enumerate(widths):
        wk, wv, wn = (w.double() for w in ws[3 * i: 3 * i + 3])
        k = (ctx.double() @ wk.t()).view(B, S, d // 128, 128)
        k = k * torch.rsqrt(k.pow(2).mean(-1, keepdim=True) + 1e-6) * wn
        v = (ctx.double() @ wv.t()).view(B, S, d // 128, 128)
        assert _rel(got[2 * i + 1], v) < ROUND
        assert _rel(got[2 * i], k) < math.sqrt(2) * ROUND      # the product is rounded, and the normalised keys are
        assert torch.equal(got[2 * i], again[2 * i]) and torch.equal(got[2 * i + 1], again[2 * i + 1])


# 256 to 528 tokens: 12 to 36 tiles of q, k and v over 16 k-blocks, split up to as many tiles as clusters of two pairs fit; 80 prompt rows to 1,024. The other widths, the widest
# with the row kernels for more than 4096 channels: few tokens, split and unsplit.
@pytest.mark.parametrize("preset,shape,tokens,split", [("mini", (1, 1, 32, 32), 40, 4), ("mini", (2, 1, 32, 32), 128, 2), ("mini", (1, 1, 24, 44), 256, 2),
                                                       ("mini", (1, 2, 26, 40), 512, 1), ("2b", (1, 1, 32, 32), 512, 2), ("2b", (1, 1, 8, 12), 24, None),
                                                       ("2b", (2, 3, 32, 36), 40, 1), ("14b", (1, 1, 8, 8), 32, None), ("14b", (1, 3, 24, 32), 256, 1)])
def test_query_key_value_of_few_tiles(preset, shape, tokens, split):
    """The native block loop against the module path, whose q, k and v are launches of their own: the same sums in another order, so a few
    bf16 roundings (2^-9 each) through the blocks."""
    torch.manual_seed(0)
    make = {"mini": dit.dit_mini, "2b": dit.dit_2b, "14b": dit.dit_14b}[preset]
    with torch.device(DEV):
        net = dit.CosmosDiT(replace(make(), num_blocks=2 if preset != "14b" else 1, crossattn_proj_in_channels=512, crossattn_emb_channels=512))
    net.init_weights()
    for n, p in net.named_parameters():
        if "adaln_modulation" in n:
            torch.nn.init.normal_(p, 0.0, 0.05)
    net = net.to(torch.bfloat16).eval().requires_grad_(False)
    B, T, H, W = shape
    rows, D = B * T * H * W // 4, net.cfg.model_channels
    if split is not None:                                       # below 256 rows q, k and v are launches of their own
        assert _split(-(-rows // 256) * (D // 256) * 3, D // 64) == split
    x, text = torch.randn(B, 16, T, H, W, device=DEV).bfloat16(), torch.randn(B, tokens, 512, device=DEV).bfloat16()
    t, fps = torch.rand(B, T, device=DEV) * 1000, torch.full((B,), 16.0, device=DEV)
    served = []
    real = dit.native_block_weights

    def run():
        dit.native_block_weights = lambda *a: served.append(real(*a)) or served[-1]
        try:
            with torch.no_grad():
                cache = net.build_context_cache(text)
                return net(x, t, None, fps=fps, context_cache=cache), cache.cross_kv
        finally:
            dit.native_block_weights = real

    got, kv = run()
    hooks = [m.register_forward_hook(lambda *a: None) for m in (net.blocks[-1].mlp.layer1, net.blocks[0].cross_attn.k_proj)]
    want, kv_want = run()
    for h in hooks:
        h.remove()
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 0 and served[0] is not None and served[1] is None
    assert _rel(got, want.double()) < 4 * 2.0 ** -9
    for a, b in zip([t for p in kv for t in p], [t for p in kv_want for t in p]):
        assert _rel(a, b.double()) < 4 * 2.0 ** -9


# Blocks of one width: every key and value in one launch (several from 40 blocks on), tiles by weight, the keys normalised in the epilogue.
# Ragged rows, contraction that is no whole k-block count of the ring, a width of many N tiles, more blocks than a launch takes.
@pytest.mark.parametrize("B,S,C,D,blocks", [(2, 512, 1024, 2048, 5), (1, 264, 1024, 1024, 10), (3, 88, 576, 512, 20), (1, 77 * 8, 1024, 5120, 2),
                                            (1, 512, 512, 256, 41)])
@pytest.mark.parametrize("norm_dtype", [torch.bfloat16, torch.float32])
def test_all_blocks_in_one_launch(B, S, C, D, blocks, norm_dtype):
    torch.manual_seed(1)
    ops = native.load()
    assert ops.dit_context_launches(B * S, C, [D] * blocks) == -(-blocks // 40)
    assert ops.dit_context_launches(B * S, C, [D, D + 256]) == 4 and ops.dit_context_launches(248, C, [D] * blocks) == 3 * blocks
    ctx = torch.randn(B, S, C, device=DEV).bfloat16()
    ws = []
    for _ in range(blocks):
        ws += [(torch.randn(D, C, device=DEV) / math.sqrt(C)).bfloat16() for _ in range(2)] + [(1 + 0.2 * torch.randn(128, device=DEV)).to(norm_dtype)]
    got, again = ops.dit_context_kv(ctx, ws, 1e-6), ops.dit_context_kv(ctx, ws, 1e-6)
    torch.cuda.synchronize()
    assert ops.kernel_error(0, True) == 0 and len(got) == 2 * blocks
    for i in range(blocks):
        wk, wv, wn = (w.double() for w in ws[3 * i: 3 * i + 3])
        k = (ctx.double() @ wk.t()).view(B, S, D // 128, 128)
        k = k * torch.rsqrt(k.pow(2).mean(-1, keepdim=True) + 1e-6) * wn
        v = (ctx.double() @ wv.t()).view(B, S, D // 128, 128)
        assert _rel(got[2 * i], k) < ROUND and _rel(got[2 * i + 1], v) < ROUND       # one rounding each
        assert torch.equal(got[2 * i], again[2 * i]) and torch.equal(got[2 * i + 1], again[2 * i + 1])
