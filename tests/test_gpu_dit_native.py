"""The sampling-time block loop as one native operator against the same blocks run module by module, and every form of a block that it
does not know goes through the modules."""

import pytest
import torch

from cosmos_predict25_b200.models import dit
from cosmos_predict25_b200.ops import functional as F_ops
from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _net(**kw):
    torch.manual_seed(0)
    cfg = dit.dit_mini(num_blocks=2, crossattn_proj_in_channels=256, crossattn_emb_channels=256, **kw)
    with torch.device(DEV):
        net = dit.CosmosDiT(cfg)
    net.init_weights()
    for n, p in net.named_parameters():
        if "adaln_modulation" in n:
            torch.nn.init.normal_(p, 0.0, 0.05)
        if "norm.weight" in n:
            torch.nn.init.normal_(p, 1.0, 0.1)
    return net.to(torch.bfloat16).eval().requires_grad_(False)


def _inputs(B, T, H, W, tokens=40):
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(B, 16, T, H, W, generator=g, device=DEV).bfloat16()
    t = torch.rand(B, T, generator=g, device=DEV) * 1000
    text = torch.randn(B, tokens, 256, generator=g, device=DEV).bfloat16()
    return x, t, text


def _same(a, b, what):
    """Both paths run the same kernels; q, k and v as one launch have more tiles, which may change how a contraction is split over CTA
    pairs. Then fp32 sums differ in their order, some bf16 roundings with them (2^-9 of a value each), and through two blocks' residual
    streams no more than a few such roundings accumulate in the 2-norm."""
    err = ((a.double() - b.double()).norm() / b.double().norm()).item()
    assert err < 4 * 2.0 ** -9, (what, err)


@pytest.fixture
def calls(monkeypatch):
    seen = []
    real = dit.native_block_weights
    monkeypatch.setattr(dit, "native_block_weights", lambda *a: seen.append(real(*a)) or seen[-1])
    return seen


def _run(net, x, t, text):
    with torch.no_grad():
        cache = net.build_context_cache(text)
        out = net(x, t, None, fps=torch.full((x.shape[0],), 16.0, device=DEV), context_cache=cache)
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 0
    return out, [t for kv in cache.cross_kv for t in kv]


@pytest.mark.parametrize("shape", [(1, 1, 8, 8), (2, 1, 16, 16), (1, 3, 12, 16), (2, 5, 24, 24)])
@pytest.mark.parametrize("variant", ["plain", "fp32 norms", "narrow mlp"])
def test_native_blocks_equal_the_modules(shape, variant, calls):
    net = _net(**({"mlp_ratio": 1.5} if variant == "narrow mlp" else {}))
    if variant == "fp32 norms":
        for m in net.modules():
            if type(m) is dit.RMSNorm and m.weight.numel() == 128:
                m.weight.data = m.weight.data.float()
    args = _inputs(*shape)
    before = native.launches()
    got, kv = _run(net, *args)
    counted = native.launches() - before
    assert calls[-1] is not None, "the native loop did not serve a plain network"
    hook = net.blocks[1].mlp.layer1.register_forward_hook(lambda *a: None)      # a hook wants to be called: module by module
    k_hook = net.blocks[0].cross_attn.k_proj.register_forward_hook(lambda *a: None)
    before = native.launches()
    want, kv_want = _run(net, *args)
    assert calls[-1] is None and native.launches() - before >= counted
    hook.remove(), k_hook.remove()
    _same(got, want, "output")
    for a, b in zip(kv, kv_want):
        _same(a, b, "keys / values")


def test_other_forms_go_through_the_modules(calls):
    net = _net()
    args = _inputs(1, 1, 16, 16)
    want, _ = _run(net, *args)

    def expect_modules():
        out, _ = _run(net, *args)
        assert calls[-1] is None
        return out

    net.blocks[0].forward = net.blocks[0].forward               # an instance's own forward
    _same(expect_modules(), want, "own forward")
    del net.blocks[0].forward
    net.blocks[1].self_attn.q_norm.eps = 1e-5                    # norms of different epsilon
    expect_modules()
    net.blocks[1].self_attn.q_norm.eps = 1e-6
    layer = net.blocks[0].mlp.layer2
    net.blocks[0].mlp.layer2 = torch.nn.Linear(layer.in_features, layer.out_features, bias=False, device=DEV, dtype=torch.bfloat16)
    net.blocks[0].mlp.layer2.weight = layer.weight               # another type of projection
    assert (expect_modules() - want).norm() / want.norm() < 2e-2
    net.blocks[0].mlp.layer2 = layer
    F_ops.settings.attention = "cudnn"
    try:
        expect_modules()
    finally:
        F_ops.settings.attention = "native"
    x, t, text = args
    with torch.no_grad():
        cache = net.build_context_cache(text)
        short = dit.ContextCache(cache.context, [(k[:, :24], v[:, :24]) for k, v in cache.cross_kv])      # B = 1: still contiguous
        net(x, t, None, fps=torch.full((1,), 16.0, device=DEV), context_cache=short)
        assert calls[-1] is not None
        strided = dit.ContextCache(cache.context, [(k.transpose(1, 2).contiguous().transpose(1, 2), v) for k, v in cache.cross_kv])
        out = net(x, t, None, fps=torch.full((1,), 16.0, device=DEV), context_cache=strided)
    assert calls[-1] is None
    _same(out, want, "strided keys")
