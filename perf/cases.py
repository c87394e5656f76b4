"""Workloads that stand for what a program built on this package spends its GPU time on.

Every case is one call that such a program repeats: a denoising step of the sampler, the preparation of a prompt, a training step
(forward, backward, gradients reduced to fp32 shards), and the video tokenizer's encode and decode. Sizes come from the resolution
tables (``data/utils.py``), the network presets (``models/dit.py: NET_PRESETS``) and the benchmark's clip (720p, 24 latent frames).

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges, ``prepare`` builds what the program holds before the
call, ``run`` makes the call, ``work`` counts what the call cannot do without and ``tolerance`` says how far two correct bf16
implementations lie apart.
"""

from __future__ import annotations

import math
from dataclasses import replace

import torch

from cosmos_predict25_b200.models.conditioner import DataType
from cosmos_predict25_b200.models.dit import DiTConfig, dit_14b, dit_2b, dit_mini
from cosmos_predict25_b200.models.rectified_flow import Video2WorldModelRectifiedFlow, Video2WorldRFConfig
from cosmos_predict25_b200.models.vae_wan import Wan2pt1VAEInterface

TEXT_TOKENS = 512        # prompts are padded to this length unless the caller trims them
TEXT_WIDTH = 100352      # concatenated hidden states of the text encoder
LATENT_CHANNELS = 16

_NETS = {"2B": dit_2b, "14B": dit_14b, "mini": dit_mini}


# ------------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # One 256 x 256 image with its positive and negative prompt as the two rows of the network's batch: the smallest calls. The
        # network's weights are read for a few hundred tokens, so launches and latency count.
        dict(name="denoise_image_256", kind="denoise", batch=1, frames=1, height=32, width=32, cond=0),
        # One 720p image (text to image).
        dict(name="denoise_image_720", kind="denoise", batch=1, frames=1, height=88, width=160, cond=0),
        # A 93-frame clip at the 256 resolution (320 x 192), continued from two latent frames: drafts and previews.
        dict(name="denoise_clip_256", kind="denoise", batch=1, frames=24, height=24, width=40, cond=2),
        # A 480p clip (832 x 480) continued from one image, 15 latent frames: the ordinary sampling step.
        dict(name="denoise_video_480p", kind="denoise", batch=1, frames=15, height=60, width=104, cond=1),
        # What a new prompt costs before the first step: text projection and the cross-attention keys / values of all blocks
        # (positive and negative prompt).
        dict(name="prompt_pair", kind="prompt", batch=2, tokens=512),
        # A training step of the small preset on a short low-resolution clip (unit runs, ablations): many small kernels.
        dict(name="train_mini_256", kind="train", net="mini", blocks=2, batch=1, frames=5, height=32, width=32, cond=1),
        # The 2B network's width at 480 (768 x 432), 93 frames, two blocks: post-training resolution.
        dict(name="train_2B_480", kind="train", net="2B", blocks=2, batch=1, frames=24, height=54, width=96, cond=1),
        # The benchmark's clip, 720p x 93 frames = 84,480 tokens, at the 2B network's width, one block: the largest sequence.
        dict(name="train_2B_720", kind="train", net="2B", blocks=1, batch=1, frames=24, height=88, width=160, cond=2),
        # Decoding one generated image at the 480p square size (640 x 640).
        dict(name="decode_image_480p", kind="decode", frames=1, height=80, width=80),
        # Decoding a 720p clip, 29 frames.
        dict(name="decode_video_720", kind="decode", frames=8, height=88, width=160),
        # Encoding the conditioning image of image-to-video at 720p.
        dict(name="encode_image_720", kind="encode", frames=1, height=704, width=1280),
        # Encoding a 29-frame training clip at the 480 resolution (768 x 432).
        dict(name="encode_clip_480", kind="encode", frames=29, height=432, width=768),
    ]


def _even(rng, lo, hi):
    """An even number, spread over the logarithm of its range (latent sizes are multiples of the 2 x 2 patch)."""
    return 2 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)) - 0.25 / hi))))


def draw(rng):
    """One more case: image to 93-frame clips, thumbnails to 720p, ragged frame sizes, other batch sizes and network widths."""
    largest = {}
    for c in listed():
        largest[c["kind"]] = max(largest.get(c["kind"], 0.0), _cost(c))
    while True:
        kind = rng.choice(("denoise", "denoise", "denoise", "prompt", "train", "train", "decode", "decode", "encode", "encode"))
        if kind == "prompt":
            c = dict(kind=kind, batch=rng.choice((1, 2, 3, 4, 6, 8)), tokens=rng.choice((TEXT_TOKENS, _log_int(rng, 64, TEXT_TOKENS))))
            if c["batch"] * c["tokens"] != 2 * TEXT_TOKENS:
                return c
            continue
        if kind == "denoise":
            frames = _log_int(rng, 1, 24)
            c = dict(kind=kind, batch=rng.choice((1, 1, 1, 2)), frames=frames, height=_even(rng, 20, 96), width=_even(rng, 20, 160),
                     cond=0 if frames == 1 else rng.choice((0, 1, 2)))
        elif kind == "train":
            frames = _log_int(rng, 1, 24)
            net = rng.choice(("mini", "2B", "2B", "14B"))
            c = dict(kind=kind, net=net, blocks=1 if net == "14B" else rng.choice((1, 2)), batch=rng.choice((1, 1, 2)), frames=frames,
                     height=_even(rng, 24, 96), width=_even(rng, 24, 160), cond=0 if frames == 1 else rng.choice((0, 1, 2)))
        elif kind == "decode":
            c = dict(kind=kind, frames=_log_int(rng, 1, 12), height=_even(rng, 24, 96), width=_even(rng, 24, 160))
        else:
            c = dict(kind=kind, frames=1 + 4 * (_log_int(rng, 1, 10) - 1), height=8 * _even(rng, 24, 96), width=8 * _even(rng, 24, 160))
        if _cost(c) <= largest[kind]:
            return c


# --------------------------------------------------------------------------------------------------------- what a program holds
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _model(net: DiTConfig, seed):
    """A Video2World model with weights of its own for every seed, built on the device. ``init_weights`` zeroes the last matrix of
    every modulation MLP; a trained network's are not zero, so they are filled."""
    torch.manual_seed(seed)
    cfg = Video2WorldRFConfig(net=net, precision="bfloat16")
    with torch.device("cuda"):
        model = Video2WorldModelRectifiedFlow(cfg, device=torch.device("cuda", torch.cuda.current_device()))
    with torch.no_grad():
        for name, p in model.net.named_parameters():
            if "adaln_modulation" in name and name.endswith(".2.weight"):
                p.normal_(0.0, 0.02)
    return model


def _batch(case, g):
    B, T, H, W = case["batch"], case["frames"], case["height"], case["width"]
    return {
        "latents": torch.randn(B, LATENT_CHANNELS, T, H, W, generator=g, device="cuda"),
        "t5_text_embeddings": torch.randn(B, TEXT_TOKENS, TEXT_WIDTH, generator=g, device="cuda", dtype=torch.bfloat16),
        "neg_t5_text_embeddings": torch.randn(B, TEXT_TOKENS, TEXT_WIDTH, generator=g, device="cuda", dtype=torch.bfloat16),
        "fps": torch.full((B,), 16.0, device="cuda"),
        "padding_mask": torch.zeros(B, 1, H, W, device="cuda"),
        "num_conditional_frames": case["cond"],
    }


class _TrainingState(dict):
    """A training program's state. The engine's gradient hooks tie it to its parameters in a cycle that the garbage collector does not
    see, so a process that builds many engines takes each one apart to get its memory back."""

    def __del__(self):
        engine = self["model"].engine
        for u in engine.units:
            vars(u).clear()
        vars(engine).clear()


def prepare(case, seed):
    kind, g = case["kind"], _generator(seed)
    if kind in ("denoise", "prompt"):
        model = _model(dit_2b(), seed)
        model.net.to(torch.bfloat16)
        model.eval()
        if kind == "prompt":
            emb = torch.randn(case["batch"], case["tokens"], TEXT_WIDTH, generator=g, device="cuda", dtype=torch.bfloat16)
            return {"case": case, "model": model, "text": emb}
        batch = _batch(case, g)
        with torch.no_grad():
            positive, negative = model.conditioner.get_condition_with_negative_prompt(batch)
            both = replace(positive, crossattn_emb=torch.cat([positive.crossattn_emb, negative.crossattn_emb]), fps=positive.fps.repeat(2),
                           padding_mask=positive.padding_mask.repeat(2, 1, 1, 1), data_type=DataType.VIDEO)
            both = both.set_video_condition(batch["latents"].repeat(2, 1, 1, 1, 1).to(torch.bfloat16), 0, 0, num_conditional_frames=case["cond"])
            cache = model.net.build_context_cache(both.crossattn_emb.to(torch.bfloat16))
        shape = batch["latents"].shape
        noise = torch.randn(shape, generator=g, device="cuda").repeat(2, 1, 1, 1, 1)
        x = torch.randn(shape, generator=g, device="cuda").repeat(2, 1, 1, 1, 1)
        t = (torch.rand(case["batch"], 1, generator=g, device="cuda") * 1000.0).repeat(2, 1)
        return {"case": case, "model": model, "condition": both, "cache": cache, "noise": noise, "x": x, "t": t}
    if kind == "train":
        model = _model(replace(_net_of(case), checkpoint_mode="save_attention"), seed).train()
        model.on_train_start()
        batch = _batch(case, g)
        del batch["neg_t5_text_embeddings"]
        return _TrainingState(case=case, model=model, batch=batch, seed=seed)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        tok = Wan2pt1VAEInterface(device="cuda", dtype=torch.bfloat16)
    T, H, W = case["frames"], case["height"], case["width"]
    if kind == "decode":
        return {"case": case, "tok": tok, "latent": torch.randn(1, LATENT_CHANNELS, T, H, W, generator=g, device="cuda")}
    # a smooth picture plus grain, in [-1, 1]: what a camera clip looks like to the encoder
    coarse = torch.randn(1, 3, T, H // 16, W // 16, generator=g, device="cuda")
    pixels = torch.nn.functional.interpolate(coarse, size=(T, H, W), mode="nearest")
    pixels = (0.4 * pixels + 0.1 * torch.randn(1, 3, T, H, W, generator=g, device="cuda")).clamp_(-1, 1)
    return {"case": case, "tok": tok, "pixels": pixels.to(torch.bfloat16)}


# ------------------------------------------------------------------------------------------------------------------ the call
def run(state):
    kind = state["case"]["kind"]
    if kind == "denoise":
        with torch.no_grad():
            return state["model"].denoise(state["noise"], state["x"], state["t"], state["condition"], context_cache=state["cache"])
    if kind == "prompt":
        with torch.no_grad():
            cache = state["model"].net.build_context_cache(state["text"])
        return {"context": cache.context, "kv": cache.cross_kv}
    if kind == "decode":
        return state["tok"].decode(state["latent"])
    if kind == "encode":
        return state["tok"].encode(state["pixels"])
    model = state["model"]
    torch.manual_seed(state["seed"])        # noise, noise level and dropout of the step: the same ones in every pass
    model.engine.zero_grad()
    _, loss = model.training_step(dict(state["batch"]), 0)
    loss.backward()
    model.engine.finish_backward()
    return {"loss": loss.detach(), "grads": [u.grad_shard for u in model.engine.units]}


# ------------------------------------------------------------------------------------------- what the call cannot do without
def _net_of(case):
    if case["kind"] in ("denoise", "prompt"):
        return dit_2b()
    return replace(_NETS[case["net"]](), num_blocks=case["blocks"])


def _dit_counts(net: DiTConfig, rows, seq, samples, frames):
    """FLOPs of the token GEMMs, of the few-row modulation MLPs, of self- and of cross-attention, for one forward pass."""
    D, L, C = net.model_channels, net.num_blocks, net.crossattn_emb_channels
    gemm = 2.0 * rows * (14 * D * D * L + 72 * D + 64 * D)
    few = 2.0 * samples * frames * (D * D + 3 * D * D + L * 3 * net.adaln_lora_dim * 4 * D)
    attn = 4.0 * samples * seq * seq * D * L
    cross = 4.0 * rows * TEXT_TOKENS * D * L
    text = 2.0 * samples * TEXT_TOKENS * (TEXT_WIDTH * C + 2 * L * C * D)
    return gemm, few, attn, cross, text


def _dit_params(net: DiTConfig):
    D, L, C, R = net.model_channels, net.num_blocks, net.crossattn_emb_channels, net.adaln_lora_dim
    body = L * (14 * D * D + 3 * R * 4 * D) + 72 * D + 64 * D + 4 * D * D + 3 * R * D
    return body, L * 2 * C * D, TEXT_WIDTH * C


def _resblock(cin, cout, vox):
    return 2.0 * vox * 27 * (cin * cout + cout * cout) + (2.0 * vox * cin * cout if cin != cout else 0.0)


def _mid_attention(c, t, hw):
    return t * (2.0 * hw * c * 4 * c + 4.0 * hw * hw * c)


def _decoder_flops(T, h, w):
    hw, t1, t2 = h * w, max(1, 2 * T - 1), max(1, 4 * T - 3)
    f = 2.0 * T * hw * 27 * 16 * 384 + 2 * _resblock(384, 384, T * hw) + _mid_attention(384, T, hw)
    f += 3 * _resblock(384, 384, T * hw)
    f += 2.0 * (T - 1) * hw * 3 * 384 * 768 + 2.0 * t1 * 4 * hw * 4 * 384 * 192            # nearest 2x + 3 x 3 = four 2 x 2 taps
    f += _resblock(192, 384, t1 * 4 * hw) + 2 * _resblock(384, 384, t1 * 4 * hw)
    f += 2.0 * (t1 - 1) * 4 * hw * 3 * 384 * 768 + 2.0 * t2 * 16 * hw * 4 * 384 * 192
    f += 3 * _resblock(192, 192, t2 * 16 * hw) + 2.0 * t2 * 64 * hw * 4 * 192 * 96
    f += 3 * _resblock(96, 96, t2 * 64 * hw) + 2.0 * t2 * 64 * hw * 27 * 96 * 3
    return f


def _encoder_flops(T, H, W):
    hw = H * W / 64
    t2, t1, t0 = T, 1 + (T - 1) // 2, 1 + (T - 1) // 4
    f = 2.0 * t2 * 64 * hw * 27 * 3 * 96 + 2 * _resblock(96, 96, t2 * 64 * hw) + 2.0 * t2 * 16 * hw * 9 * 96 * 96
    f += _resblock(96, 192, t2 * 16 * hw) + _resblock(192, 192, t2 * 16 * hw) + 2.0 * t2 * 4 * hw * 9 * 192 * 192
    f += 2.0 * (t1 - 1) * 4 * hw * 3 * 192 * 192
    f += _resblock(192, 384, t1 * 4 * hw) + _resblock(384, 384, t1 * 4 * hw) + 2.0 * t1 * hw * 9 * 384 * 384
    f += 2.0 * (t0 - 1) * hw * 3 * 384 * 384 + 4 * _resblock(384, 384, t0 * hw) + _mid_attention(384, t0, hw)
    f += 2.0 * t0 * hw * 27 * 384 * 32
    return f


def work(case):
    kind = case["kind"]
    if kind in ("decode", "encode"):
        T, H, W = case["frames"], case["height"], case["width"]
        if kind == "decode":
            return {"bytes": 4.0 * 16 * T * H * W + 2.0 * 3 * (4 * T - 3) * 64 * H * W + 2 * 73e6, "flops": _decoder_flops(T, H, W)}
        return {"bytes": 2.0 * 3 * T * H * W + 2.0 * 16 * (1 + (T - 1) // 4) * H * W / 64 + 2 * 54e6, "flops": _encoder_flops(T, H, W)}
    net = _net_of(case)
    D, L = net.model_channels, net.num_blocks
    body, kv, proj = _dit_params(net)
    if kind == "prompt":
        rows = case["batch"] * case["tokens"]
        out = 2.0 * rows * (net.crossattn_emb_channels + 2 * L * D)
        return {"bytes": 2.0 * (kv + proj) + 2.0 * rows * TEXT_WIDTH + out,
                "flops": 2.0 * rows * (TEXT_WIDTH * net.crossattn_emb_channels + 2 * L * net.crossattn_emb_channels * D)}
    B, T, seq = case["batch"], case["frames"], case["frames"] * case["height"] * case["width"] // 4
    latent = 4.0 * B * LATENT_CHANNELS * T * case["height"] * case["width"]
    if kind == "denoise":
        gemm, few, attn, cross, _ = _dit_counts(net, 2 * B * seq, seq, 2 * B, T)
        return {"bytes": 2.0 * body + 2.0 * 2 * B * TEXT_TOKENS * 2 * L * D + 5 * latent, "flops": gemm + few + attn + cross}
    gemm, few, attn, cross, text = _dit_counts(net, B * seq, seq, B, T)
    # backward: two GEMMs for each forward one (the projected text needs no input gradient), five attention GEMMs for two
    flops = 3 * (gemm + few) + 3.5 * (attn + cross) + 2 * text
    return {"bytes": (2.0 + 2.0 + 4.0) * (body + kv + proj) + 2.0 * B * TEXT_TOKENS * TEXT_WIDTH + 2 * latent, "flops": flops}


def _cost(case):
    """Rough seconds of a pass on one GPU, to keep drawn cases below the largest listed one of their kind."""
    w = work(case)
    return w["flops"] / 1e15 + w["bytes"] / 5e12


def tolerance(case):
    """Measured on B200 against the same case with cuDNN attention, cuBLAS GEMMs and cuDNN convolutions (the ``settings`` switches of
    ``ops/functional.py``), which round at other places and sum in another order. 2-norm of the difference over the result's: 0.3 %
    for the gradients, 0.45 % for the prompt's keys and values, 0.5 % for encode, 2 to 2.6 % for decode, and 1 % for a denoising
    step, where 84 bf16 additions to the residual stream lie between input and output. Stated: four times that, 3 % at most."""
    return {"rel": {"train": 0.012, "prompt": 0.018, "encode": 0.02, "decode": 0.03, "denoise": 0.03}[case["kind"]]}
