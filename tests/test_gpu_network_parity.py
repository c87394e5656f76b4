"""Whole-network evidence on a GPU: the bf16 DiT on this package's kernels against the same weights run in fp32 on the CPU
oracle path (outputs and every parameter gradient), and a seeded three-step training run that must repeat its losses.

The reference checks its context-parallel network the same way: outputs and all gradients of the whole model against a
single-device run (cosmos_predict2/_src/predict2/context_parallel_test.py:191-266), and pins three training losses
(cosmos_predict2/_src/predict2/tests/training_loss_test.py:34-85)."""

import copy

import pytest
import torch

from cosmos_predict25_b200.models.dit import CosmosDiT, dit_mini
from cosmos_predict25_b200.models.rectified_flow import Video2WorldModelRectifiedFlow, Video2WorldRFConfig
from cosmos_predict25_b200.ops import native
from cosmos_predict25_b200.trainer.optim import OptimizerConfig
from cosmos_predict25_b200.trainer.trainer import Trainer, TrainerConfig

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


def test_bf16_network_matches_its_fp32_cpu_oracle():
    torch.manual_seed(0)
    cfg = dit_mini(model_channels=512, num_heads=4, crossattn_proj_in_channels=512, crossattn_emb_channels=512, checkpoint_mode="none")
    ref_net = CosmosDiT(cfg)
    ref_net.init_weights()
    with torch.no_grad():   # zero-initialised output projections would hide most of the network: give them signal
        for name, p in ref_net.named_parameters():
            if p.abs().max() == 0:
                p.normal_(0, 0.02)
            p.copy_(p.bfloat16().float())
    net = copy.deepcopy(ref_net).to("cuda", torch.bfloat16)
    x = torch.randn(1, 16, 4, 32, 32)
    t = torch.tensor([[400.0]])
    ctx = torch.randn(1, 64, 512)
    mask = torch.zeros(1, 1, 4, 32, 32)
    mask[:, :, :1] = 1
    pm = torch.zeros(1, 1, 32, 32)
    dy = torch.randn(1, 16, 4, 32, 32)
    want = ref_net(x, t, ctx, condition_video_input_mask_B_C_T_H_W=mask, padding_mask=pm, fps=torch.tensor([16.0]))
    want.backward(dy)
    native.reset_launches()
    got = net(x.cuda().bfloat16(), t.cuda(), ctx.cuda().bfloat16(), condition_video_input_mask_B_C_T_H_W=mask.cuda().bfloat16(),
              padding_mask=pm.cuda(), fps=torch.tensor([16.0], device="cuda"))
    got.float().backward(dy.cuda())
    torch.cuda.synchronize()
    assert native.launches() > 20, "the network did not run on the extension's kernels"
    assert native.load().kernel_error(0, True) == 0
    assert _rel(got, want) < 3e-2, f"output relative error {_rel(got, want):.4f}"
    worst = ("", 0.0)
    ref_params = dict(ref_net.named_parameters())
    for name, p in net.named_parameters():
        r = ref_params[name]
        if r.grad is None:
            assert p.grad is None or p.grad.abs().max() == 0, name
            continue
        assert p.grad is not None, name
        e = _rel(p.grad, r.grad)
        if e > worst[1]:
            worst = (name, e)
    assert worst[1] < 8e-2, f"gradient of {worst[0]} differs by {worst[1]:.4f} (relative L2)"


def _three_losses(seed):
    torch.manual_seed(seed)
    dev = torch.device("cuda", 0)
    cfg = Video2WorldRFConfig(net=dit_mini(crossattn_proj_in_channels=1024, checkpoint_mode="save_attention"), state_t=4)
    model = Video2WorldModelRectifiedFlow(cfg, device=dev).train()
    trainer = Trainer(TrainerConfig(output_dir="/tmp/cosmos_b200_golden", logging_iter=0, seed=seed), model, OptimizerConfig(lr=1e-4))
    g = torch.Generator().manual_seed(seed + 1)
    batch = {"latents": torch.randn(1, 16, 4, 32, 32, generator=g), "t5_text_embeddings": torch.randn(1, 64, 1024, generator=g).bfloat16(),
             "fps": torch.tensor([16.0]), "padding_mask": torch.zeros(1, 1, 32, 32), "num_conditional_frames": 1}
    torch.manual_seed(seed + 2)   # noise and time sampling of the three steps
    return [trainer.train_step(dict(batch)) for _ in range(3)]


def test_seeded_training_losses_repeat():
    """Same seed, same three losses. Every kernel on this path is deterministic except the dQ accumulation of the long-sequence
    attention backward, which this sequence length (1,024 tokens) does not select; so the losses must agree to the last bit."""
    a = _three_losses(11)
    b = _three_losses(11)
    assert all(x == x for x in a), a
    assert a == b, (a, b)
    c = _three_losses(12)
    assert a != c


def _block_step(mode, selective_by_operator=False):
    """Output, input gradients and weight gradients of one checkpointed block; launches counted on the way."""
    from cosmos_predict25_b200.models import checkpointing
    from cosmos_predict25_b200.models.dit import Block
    from cosmos_predict25_b200.ops import native

    torch.manual_seed(3)
    block = Block(dit_mini(model_channels=512, num_heads=4, crossattn_emb_channels=256)).to("cuda", torch.bfloat16).train()
    block.init_weights()
    for m in block.adaln_mlps():
        torch.nn.init.normal_(m[-1].weight, std=0.02)
    if selective_by_operator:
        block.keeps_attention_itself = lambda x: False
    x = torch.randn(1, 2, 96, 512, device="cuda").bfloat16().requires_grad_(True)
    emb = torch.randn(1, 2, 512, device="cuda").requires_grad_(True)
    ctx = torch.randn(1, 40, 256, device="cuda").bfloat16().requires_grad_(True)
    before = native.launches()
    y = checkpointing.run_block(block, mode, x, emb, ctx, None, None)
    return block, y, (x, emb, ctx), before


def test_kept_attention_results_give_the_gradients_of_the_other_modes():
    from cosmos_predict25_b200.ops import native

    got = []
    for mode, by_operator in (("none", False), ("save_attention", False), ("save_attention", True)):
        block, y, inputs, before = _block_step(mode, by_operator)
        y.float().pow(2).sum().backward()
        got.append(([y.detach()] + [t.grad for t in inputs] + [p.grad for p in block.parameters()], native.launches() - before))
    for other, _ in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0][0], other))
    assert got[1][1] == got[2][1]           # both count the attention kernels once


def test_kept_attention_results_are_used_once_and_unchanged():
    block, y, _, _ = _block_step("save_attention")
    y.sum().backward(retain_graph=True)
    with pytest.raises(RuntimeError, match="only once"):
        y.sum().backward()
    # a second region inside the first one's backward, and a region that is dropped, leave nothing behind
    from cosmos_predict25_b200.ops.functional import AttentionResults
    assert getattr(AttentionResults._active, "scope", None) is None
    q = torch.randn(1, 64, 1, 128, device="cuda").bfloat16()
    results = AttentionResults()
    with results.keep():
        o, _ = AttentionResults.forward(q, q, q, 0.1)
    o.add_(1)
    with results.reuse(), pytest.raises(RuntimeError, match="in place"):
        AttentionResults.forward(q, q, q, 0.1)
