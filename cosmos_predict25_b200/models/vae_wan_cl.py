"""Channels-last decoder of the Wan2.1 VAE on the implicit-GEMM convolution kernel (``ops/csrc/conv3d_cl.cu``).

``DecoderCL`` takes the weights of a ``vae_wan.Decoder3d`` and runs the same streaming decode - one latent frame per step,
every causal convolution carrying the last two input frames of the previous step, the temporal up-sampler skipped on the first
step (cosmos_predict2/_src/predict2/tokenizers/wan2pt1.py:40-58, 84-137, 184-215, 358-462, 543-562) - with activations kept as
``[T, H, W, C]`` bf16 tensors throughout:

  * every convolution is one launch of ``conv_cl`` (TMA boxes shifted by the tap are the im2col; out-of-range boxes are the zero
    padding; bias and the residual add of a block are its epilogue);
  * "nearest 2x up-sampling + 3 x 3 convolution" is computed as four 2 x 2 phase convolutions on the low-resolution frame with
    pre-summed weights: output pixel (2y + a, 2x + b) only ever sees a 2 x 2 neighbourhood of the input, so 4 taps replace 9 and
    the up-sampled frame is never materialised; the phases interleave through the kernel's output mapping;
  * the temporal up-sampler's channel-to-frame interleave is an output mapping too (two launches, one per output-channel half);
  * RMS-norm + SiLU in front of a convolution is part of the epilogue of the convolution before it while one tile holds all channels
    (96 and 192), else one element-wise kernel.

The single-head frame attention of the middle block runs on ``fa_wide`` (head dimension 384) with its 1 x 1 projections on this
package's GEMM. Weights are repacked once (``[C_out, taps, C_in padded to 64]`` bf16, fp32 bias) when the object is built.
"""

from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import torch
import torch.nn.functional as F

from ..ops import functional as F_ops
from ..ops import native
from . import vae_parallel

CACHE_T = 2
STEP_BYTES = 3 << 29       # full-resolution activation of one streaming step (a step holds a handful of them, the stream two frames per layer)


def _n_tile(cout: int) -> int:
    if cout <= 256:
        return (cout + 15) // 16 * 16
    for t in (192, 256, 128):
        if cout % t == 0:
            return t
    return 256


class ConvCL:
    """One convolution with repacked weights. ``taps``: (dt, dh, dw) offsets added to an output coordinate to get the input
    coordinate; ``weight_taps``: [C_out, n_taps, C_in] fp32/bf16 in the same order."""

    def __init__(self, weight_taps: torch.Tensor, bias: Optional[torch.Tensor], taps: Sequence[Tuple[int, int, int]], device,
                 t_stride: int = 1, hw_stride: int = 1):
        cout, ntaps, cin = weight_taps.shape
        assert ntaps == len(taps) and cin % 16 == 0, (weight_taps.shape, len(taps))
        self.cout, self.cin, self.n_tile = cout, cin, _n_tile(cout)
        rows = (cout + self.n_tile - 1) // self.n_tile * self.n_tile
        cpad = (cin + 63) // 64 * 64
        w = torch.zeros(rows, ntaps, cpad, dtype=torch.bfloat16, device=device)
        w[:cout, :, :cin] = weight_taps.to(device=device, dtype=torch.bfloat16)
        self.w = w.view(rows, ntaps * cpad).contiguous()
        self.bias = bias.detach().to(device=device, dtype=torch.float32).contiguous() if bias is not None else None
        self.taps = [int(v) for t in taps for v in t]
        self.spatial = any(t[1] != 0 for t in taps)            # reads neighbouring rows: needs halo rows under row sharding
        self.taps_halo = [int(v) for t in taps for v in (t[0], t[1] + 1, t[2])]
        self.t_stride, self.hw_stride = t_stride, hw_stride

    def __call__(self, x: torch.Tensor, t_out: int, out: Optional[torch.Tensor] = None, out_map: Optional[List[int]] = None,
                 resid: Optional[torch.Tensor] = None, h_out: Optional[int] = None, w_out: Optional[int] = None) -> torch.Tensor:
        """x [T_in, H, W, C_in]. Default output: a new [t_out, H, W, C_out] tensor with the identity mapping. Under row-sharded
        decoding (``vae_parallel.row_sharded``) a convolution that reads neighbouring rows first receives one boundary row from
        each neighbouring rank (zeros at the frame border) and reads its input shifted by that row."""
        _, H, W, _ = x.shape
        x, taps = self._halo(x)
        return self._launch(x, taps, t_out, h_out or H, w_out or W, out, out_map, resid)

    def _halo(self, x):
        if self.spatial and vae_parallel.active() is not None:
            return vae_parallel.exchange_rows(x, 1, 1), self.taps_halo
        return x, self.taps

    def _launch(self, x, taps, t_out, h_out, w_out, out, out_map, resid, cache=None, pad=0, norm=None, normed=None, raw=True):
        if out is None and raw:
            out = torch.empty(t_out, h_out, w_out, self.cout, dtype=torch.bfloat16, device=x.device)
        if norm is not None and normed is None:
            normed = torch.empty(t_out, h_out, w_out, self.cout, dtype=torch.bfloat16, device=x.device)
        dst = out if raw else normed
        if out_map is None:
            out_map = [1, 0, 1, 0, 1, 0, dst.shape[1], dst.shape[2], dst.shape[3], 0]
        native.load().conv_cl(x, self.w, self.n_tile, self.cout, taps, t_out, h_out, w_out, out_map, dst, resid, self.bias, cache, pad,
                              self.t_stride, self.hw_stride, normed, None if norm is None else norm[0], norm is None or norm[1], raw)
        native.count_launch()
        return out if norm is None else (out, normed)

    def _finish(self, y: torch.Tensor, norm, raw: bool):
        """What a launch with ``norm`` returns, from its raw output: the norm as a kernel of its own."""
        if norm is None:
            return y
        n = native.load().rmsnorm_silu_cl(y, norm[0], norm[1])
        native.count_launch()
        return (y if raw else None), n

    def fuses_norm(self, x: torch.Tensor) -> bool:
        """The epilogue normalises when one N tile holds all channels (up to 256)."""
        return x.is_cuda and self.cout <= self.n_tile and self.cout % 8 == 0

    def strided(self, x: torch.Tensor, norm=None) -> torch.Tensor:
        """The spatially strided convolution of every frame of ``x``; pixels past the bottom / right edge are zeros. ``norm`` as in
        ``causal``."""
        T, H, W, _ = x.shape
        if not x.is_cuda:                                      # plain definition: stride 1, every second pixel
            return self._finish(self(x, T)[:, ::self.hw_stride, ::self.hw_stride].contiguous(), norm, True)
        fused = norm if self.fuses_norm(x) else None
        y = self._launch(x, self.taps, T, H // self.hw_stride, W // self.hw_stride, None, None, None, norm=fused)
        return y if fused is not None else self._finish(y, norm, True)

    def causal(self, x: torch.Tensor, state: "_Stream", pad_frames: int = CACHE_T, resid: Optional[torch.Tensor] = None, norm=None,
               raw: bool = True):
        """The causal convolution of the chunk ``x`` with the ``pad_frames`` input frames before it, which the stream carries (zeros
        before the first chunk); leaves this chunk's last frames in the stream. ``norm`` = (gamma, silu) of the RMS-norm that follows:
        the result is then (output, normalised output), the first None with ``raw`` False."""
        T, H, W, _ = x.shape
        t_out = T // self.t_stride
        if not x.is_cuda:
            full = _with_cache(self, x, state, pad_frames)
            return self._finish(self(full, T, resid=resid)[:t_out * self.t_stride:self.t_stride].contiguous(), norm, raw)
        x, taps = self._halo(x)
        prev = state.store.get(id(self))
        fused = norm if self.fuses_norm(x) else None
        y = self._launch(x, taps, t_out, H, W, None, None, resid, prev, pad_frames, fused, None, raw or fused is None)
        state.store[id(self)] = _last_frames(prev, x, pad_frames)
        return y if fused is not None else self._finish(y, norm, raw)


def _last_frames(prev: Optional[torch.Tensor], x: torch.Tensor, n: int) -> torch.Tensor:
    """The last ``n`` frames of [prev | x], or fewer when the stream has not seen as many. Copied out of a longer chunk: the stream has one
    such tensor per causal convolution, and a view would keep every chunk of the step alive until the next one."""
    if x.shape[0] > n:
        return x[-n:].clone()
    return x if x.shape[0] == n or prev is None else torch.cat([prev[x.shape[0] - n:], x], 0)


def _causal3_taps(kt: int, kh: int, kw: int):
    """Taps of a causal convolution whose input tensor starts with the (kt - 1) frames of temporal padding / stream cache."""
    return [(it, ih - kh // 2, iw - kw // 2) for it in range(kt) for ih in range(kh) for iw in range(kw)]


def _conv3d(mod, device) -> ConvCL:
    w = mod.weight.detach().float()                      # [Cout, Cin, kt, kh, kw]
    cout, cin, kt, kh, kw = w.shape
    wt = w.permute(0, 2, 3, 4, 1).reshape(cout, kt * kh * kw, cin)
    return ConvCL(wt, mod.bias, _causal3_taps(kt, kh, kw), device)


def _upsample_conv2d_phases(conv2d, device) -> List[Tuple[ConvCL, int, int]]:
    """The four phase convolutions of nearest-2x + ``conv2d`` (3 x 3, padding 1). Phase (a, b) produces output pixels
    (2y + a, 2x + b) from input pixels (y + u - 1 + a, x + v - 1 + b), u, v in {0, 1}; rows of the 3 x 3 kernel that read the
    same input row are summed (a = 0: {0}, {1, 2}; a = 1: {0, 1}, {2})."""
    w = conv2d.weight.detach().float()                   # [Cout, Cin, 3, 3]
    groups = {0: ([0], [1, 2]), 1: ([0, 1], [2])}
    phases = []
    for a in (0, 1):
        for b in (0, 1):
            taps, mats = [], []
            for u in (0, 1):
                for v in (0, 1):
                    m = sum(w[:, :, i, j] for i in groups[a][u] for j in groups[b][v])   # [Cout, Cin]
                    mats.append(m)
                    taps.append((0, u - 1 + a, v - 1 + b))
            phases.append((ConvCL(torch.stack(mats, 1), conv2d.bias, taps, device), a, b))
    return phases


class _Layer:
    """``run(x, state, xn, norm)``: ``xn`` is the layer's normalised input when the layer in front has produced it; ``norm`` = (gamma, silu)
    of the RMS-norm with which the layer behind begins. Returns the output and, when a convolution's epilogue has made it, the
    normalised output."""

    def run(self, x, state, xn=None, norm=None):
        raise NotImplementedError

    def __call__(self, x, state):
        return self.run(x, state)[0]


def _wants(layer):
    """(gamma, silu) of the RMS-norm with which a layer begins, or None."""
    if isinstance(layer, _ResBlockCL):
        return layer.g1, True
    if isinstance(layer, _AttnCL):
        return layer.gamma, False
    return None


def _run_layers(layers, y, yn, state, last):
    """The layers in order, each told which norm the layer behind it begins with (``last``: behind the last one), so that a convolution
    can produce the normalised tensor beside or instead of the raw one. Returns the last layer's normalised output."""
    for i, layer in enumerate(layers):
        norm = _wants(layers[i + 1]) if i + 1 < len(layers) else last
        y, yn = layer.run(y, state, yn, norm)
    if yn is None:
        yn = native.load().rmsnorm_silu_cl(y, *last)
        native.count_launch()
    return yn


class _Stream:
    """Last two input frames of every causal convolution (keyed by the ConvCL object)."""

    def __init__(self):
        self.store = {}


def _with_cache(conv: ConvCL, x: torch.Tensor, state: _Stream, pad_frames: int = CACHE_T) -> torch.Tensor:
    """[cache | x] along time and the cache update: the convolution's input tensor with its causal padding in front (tensors that the
    kernel does not serve; it reads the cache where it lies)."""
    prev = state.store.get(id(conv))
    if prev is None:
        prev = x.new_zeros(pad_frames, *x.shape[1:])
    full = torch.cat([prev, x], 0)
    state.store[id(conv)] = full[-pad_frames:].clone()
    return full


class _ResBlockCL(_Layer):
    def __init__(self, block, device):
        res = block.residual
        self.g1 = res[0].gamma.detach().float().reshape(-1).to(device).contiguous()
        self.c1 = _conv3d(res[2], device)
        self.g2 = res[3].gamma.detach().float().reshape(-1).to(device).contiguous()
        self.c2 = _conv3d(res[6], device)
        self.short = _conv3d(block.shortcut, device) if not isinstance(block.shortcut, torch.nn.Identity) else None

    def run(self, x, state, xn=None, norm=None):
        h = self.short(x, x.shape[0]) if self.short is not None else x
        if xn is None:
            xn = native.load().rmsnorm_silu_cl(x, self.g1, True)
            native.count_launch()
        _, y = self.c1.causal(xn, state, norm=(self.g2, True), raw=False)
        out = self.c2.causal(y, state, resid=h, norm=norm)
        return out if norm is not None else (out, None)


class _AttnCL(_Layer):
    def __init__(self, block, device):
        C = block.dim
        self.C = C
        self.gamma = block.norm.gamma.detach().float().reshape(-1).to(device).contiguous()
        self.w_qkv = block.to_qkv.weight.detach().reshape(3 * C, C).to(device=device, dtype=torch.bfloat16).contiguous()
        self.b_qkv = block.to_qkv.bias.detach().to(device=device, dtype=torch.bfloat16).contiguous()
        self.w_proj = block.proj.weight.detach().reshape(C, C).to(device=device, dtype=torch.bfloat16).contiguous()
        self.b_proj = block.proj.bias.detach().to(device=device, dtype=torch.bfloat16).contiguous()

    def run(self, x, state, xn=None, norm=None):
        T, H, W, C = x.shape
        y = xn
        if y is None:
            y = native.load().rmsnorm_silu_cl(x, self.gamma, False)
            native.count_launch()
        qkv = F_ops.linear(y.view(T * H * W, C), self.w_qkv, self.b_qkv).view(T, H * W, 3, C)
        q, k, v = (qkv[:, :, i] for i in range(3))                        # [T, HW, C], a single head of dimension C
        if vae_parallel.active() is not None:                             # local rows attend to the whole frame
            k, v = vae_parallel.gather_tokens(k.contiguous(), 1), vae_parallel.gather_tokens(v.contiguous(), 1)
        if x.is_cuda and C == 384:
            o = native.load().fa_wide(q, k, v, C ** -0.5)
            native.count_launch()
        else:                                                             # the kernel is built for the width of the released VAE
            o = F.scaled_dot_product_attention(q.unsqueeze(1), k.unsqueeze(1), v.unsqueeze(1)).squeeze(1)
        o = F_ops.linear(o.reshape(T * H * W, C), self.w_proj, self.b_proj)
        return o.view(T, H, W, C) + x, None


class _UpsampleCL(_Layer):
    def __init__(self, mod, device):
        self.mode = mod.mode
        self.dim = mod.dim
        self.phases = _upsample_conv2d_phases(mod.resample[1], device)
        self.time = None
        if mod.mode == "upsample3d":
            w = mod.time_conv.weight.detach().float()        # [2C, C, 3, 1, 1]
            C = mod.dim
            b = mod.time_conv.bias
            self.time = []
            for s in (0, 1):                                 # output-channel half s becomes frame 2t + s
                wt = w[s * C:(s + 1) * C, :, :, 0, 0].permute(0, 2, 1).contiguous()   # [C, 3, C]
                self.time.append(ConvCL(wt, b[s * C:(s + 1) * C] if b is not None else None, _causal3_taps(3, 1, 1), device))
        self._key = object()

    def run(self, x, state, xn=None, norm=None):
        T, H, W, C = x.shape
        if self.time is not None:
            prev = state.store.get(id(self._key))
            if prev is None:
                state.store[id(self._key)] = "first"          # first step: no temporal up-sampling
            else:
                cache = prev if isinstance(prev, torch.Tensor) else None      # nothing before the second step: zeros
                out = torch.empty(2 * T, H, W, C, dtype=x.dtype, device=x.device)
                for s, conv in enumerate(self.time):
                    conv._launch(x, conv.taps, T, H, W, out, [2, s, 1, 0, 1, 0, H, W, C, 0], None, cache, CACHE_T)
                state.store[id(self._key)] = _last_frames(cache, x, CACHE_T)
                x = out
                T = 2 * T
        cout = self.phases[0][0].cout
        out = torch.empty(T, 2 * H, 2 * W, cout, dtype=x.dtype, device=x.device)
        fused = norm is not None and self.phases[0][0].fuses_norm(x)
        normed = torch.empty_like(out) if fused else None
        for conv, a, b in self.phases:
            out_map = [1, 0, 2, a, 2, b, 2 * H, 2 * W, cout, 0]
            if fused:
                xh, taps = conv._halo(x)
                conv._launch(xh, taps, T, H, W, out, out_map, None, norm=norm, normed=normed)
            else:
                conv(x, T, out=out, out_map=out_map, h_out=H, w_out=W)
        return out, normed


class DecoderCL:
    """Streaming channels-last decoder built from a ``Decoder3d`` (weights are repacked at construction)."""

    def __init__(self, decoder, device):
        self.device = torch.device(device)
        dev = self.device
        self.z_pad = 64   # the 16 latent channels travel zero-padded to one 64-channel block
        w = decoder.conv1.weight.detach().float()            # [C0, z, 3, 3, 3]
        c0, z = w.shape[:2]
        wt = torch.zeros(c0, 27, self.z_pad)
        wt[:, :, :z] = w.permute(0, 2, 3, 4, 1).reshape(c0, 27, z)
        self.z_dim = z
        self.conv1 = ConvCL(wt, decoder.conv1.bias, _causal3_taps(3, 3, 3), dev)
        self.layers = []
        from . import vae_wan
        for layer in list(decoder.middle) + list(decoder.upsamples):
            if isinstance(layer, vae_wan.ResidualBlock):
                self.layers.append(_ResBlockCL(layer, dev))
            elif isinstance(layer, vae_wan.AttentionBlock):
                self.layers.append(_AttnCL(layer, dev))
            elif isinstance(layer, vae_wan.Resample):
                self.layers.append(_UpsampleCL(layer, dev))
            else:
                raise TypeError(type(layer))
        self.head_gamma = decoder.head[0].gamma.detach().float().reshape(-1).to(dev).contiguous()
        self.head = _conv3d(decoder.head[2], dev)
        self.state: Optional[_Stream] = None

    def reset(self):
        self.state = _Stream()

    def steps(self, frames: int, h: int, w: int) -> List[Tuple[int, int]]:
        """Ranges of latent frames to decode in one step each. A stream starts with a step of one frame (it skips the temporal
        up-sampling); after that as many frames as keep a full-resolution activation within ``STEP_BYTES``, because one latent frame
        is too few tiles for the low-resolution layers (384 channels at 88 x 160: 1.5 waves, 980 TFLOP/s; two frames 1,320)."""
        per_frame = 4 * 64 * h * w * self.head.cin * 2
        n = max(1, STEP_BYTES // per_frame)
        cuts = [0] + list(range(1 if self.state is None or not self.state.store else n, frames, n)) + [frames]
        return list(zip(cuts[:-1], cuts[1:]))

    @torch.no_grad()
    def step(self, x: torch.Tensor) -> torch.Tensor:
        """x [B=1, z, T, h, w] (already through the 1 x 1 ``conv2``) -> pixels [1, 3, T', 8h, 8w] for this chunk."""
        assert x.shape[0] == 1, "the channels-last decoder runs one video at a time"
        if self.state is None:
            self.reset()
        st = self.state
        T, h, w = x.shape[2:]
        xin = torch.zeros(T, h, w, self.z_pad, dtype=torch.bfloat16, device=self.device)
        xin[..., : self.z_dim] = x[0].permute(1, 2, 3, 0)
        first = _wants(self.layers[0])
        y, yn = self.conv1.causal(xin, st, norm=first) if first is not None else (self.conv1.causal(xin, st), None)
        y = self.head.causal(_run_layers(self.layers, y, yn, st, (self.head_gamma, True)), st)
        return y.permute(3, 0, 1, 2).unsqueeze(0)


def supported(decoder, z: torch.Tensor) -> bool:
    """The kernel path serves bf16 CUDA decodes of one video (whole frames or, under ``vae_parallel.row_sharded``, row bands)."""
    return (z.is_cuda and z.dtype == torch.bfloat16 and z.shape[0] == 1 and native.available()
            and hasattr(native.load(), "conv_cl") and not native.forward_mode())


# ------------------------------------------------------------------------------------------------------------------ encoder
class _DownsampleCL(_Layer):
    """``ZeroPad2d((0, 1, 0, 1)) + Conv2d(3 x 3, stride 2)`` and, for the 3-D mode, the causal ``(3, 1, 1)`` convolution with
    temporal stride 2 (wan2pt1.py:84-137): strided launches of the convolution kernel. Pixels past the bottom / right edge read its
    out-of-range fill, which is the zero padding; the time convolution's input is [last frame of the previous chunk | chunk]."""

    def __init__(self, mod, device):
        conv = mod.resample[1]
        w = conv.weight.detach().float()                     # [Cout, C, 3, 3]
        cout, C = w.shape[:2]
        self.space = ConvCL(w.permute(0, 2, 3, 1).reshape(cout, 9, C), conv.bias, [(0, i, j) for i in range(3) for j in range(3)], device,
                            hw_stride=2)
        self.time = None
        if mod.mode == "downsample3d":
            wt = mod.time_conv.weight.detach().float()[:, :, :, 0, 0].permute(0, 2, 1)          # [C, 3, C]
            self.time = ConvCL(wt, mod.time_conv.bias, _causal3_taps(3, 1, 1), device, t_stride=2)

    def run(self, x, state, xn=None, norm=None):
        first = self.time is not None and id(self.time) not in state.store
        if self.time is None or first:                                   # first chunk: no temporal down-sampling
            y = self.space.strided(x, norm)
            if first:
                state.store[id(self.time)] = (y if norm is None else y[0])[-1:]
            return (y, None) if norm is None else y
        y = self.time.causal(self.space.strided(x), state, pad_frames=1, norm=norm)
        return (y, None) if norm is None else y


class EncoderCL:
    """Streaming channels-last encoder built from an ``Encoder3d``: the same chunked semantics (a chunk of one frame first, then
    chunks of ``temporal_window`` frames; every causal convolution carries the last two input frames; the temporal down-samplers
    pass the first chunk through), every convolution on the kernel (wan2pt1.py:270-357, 500-533)."""

    def __init__(self, encoder, device):
        self.device = torch.device(device)
        dev = self.device
        from . import vae_wan
        w = encoder.conv1.weight.detach().float().cpu()      # [C0, 3, 3, 3, 3]
        c0, cin = w.shape[:2]
        self.in_pad = 16                                     # RGB travels zero-padded to 16 channels
        wt = torch.zeros(c0, 27, self.in_pad)
        wt[:, :, :cin] = w.permute(0, 2, 3, 4, 1).reshape(c0, 27, cin)
        self.cin = cin
        self.conv1 = ConvCL(wt, encoder.conv1.bias, _causal3_taps(3, 3, 3), dev)
        self.layers = []
        for layer in list(encoder.downsamples) + list(encoder.middle):
            if isinstance(layer, vae_wan.ResidualBlock):
                self.layers.append(_ResBlockCL(layer, dev))
            elif isinstance(layer, vae_wan.AttentionBlock):
                self.layers.append(_AttnCL(layer, dev))
            elif isinstance(layer, vae_wan.Resample):
                self.layers.append(_DownsampleCL(layer, dev))
            else:
                raise TypeError(type(layer))
        self.head_gamma = encoder.head[0].gamma.detach().float().reshape(-1).to(dev).contiguous()
        self.head = _conv3d(encoder.head[2], dev)
        self.state: Optional[_Stream] = None

    def reset(self):
        self.state = _Stream()

    def windows_per_step(self, H: int, W: int, window: int) -> int:
        """How many temporal windows one step takes: as many as keep a full-resolution activation within ``STEP_BYTES``. The result does
        not depend on it when a window passes both temporal down-samplers without a remainder."""
        if window % 4:
            return 1
        return max(1, STEP_BYTES // (window * H * W * self.conv1.cout * 2))

    @torch.no_grad()
    def step(self, x: torch.Tensor) -> torch.Tensor:
        """x [1, 3, T, H, W] (one chunk) -> [1, 2 z, T', H / 8, W / 8] (input of the 1 x 1 ``conv1`` of the VAE)."""
        assert x.shape[0] == 1, "the channels-last encoder runs one video at a time"
        if self.state is None:
            self.reset()
        st = self.state
        T, H, W = x.shape[2:]
        xin = torch.zeros(T, H, W, self.in_pad, dtype=torch.bfloat16, device=self.device)
        xin[..., : self.cin] = x[0].permute(1, 2, 3, 0)
        first = _wants(self.layers[0])
        y, yn = self.conv1.causal(xin, st, norm=first) if first is not None else (self.conv1.causal(xin, st), None)
        y = self.head.causal(_run_layers(self.layers, y, yn, st, (self.head_gamma, True)), st)
        return y.permute(3, 0, 1, 2).unsqueeze(0)


def _restated(encoder) -> bool:
    """Whether ``EncoderCL`` computes what the modules of this encoder would: the published layers, unhooked, without active dropout, and
    channel counts that the kernels take."""
    from . import vae_wan
    known = (vae_wan.Encoder3d, vae_wan.ResidualBlock, vae_wan.AttentionBlock, vae_wan.Resample, vae_wan.CausalConv3d, vae_wan.RMS_norm,
             torch.nn.Sequential, torch.nn.Conv2d, torch.nn.SiLU, torch.nn.Dropout, torch.nn.Identity, torch.nn.ZeroPad2d)
    for m in encoder.modules():
        if type(m) not in known or m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__:
            return False
        if isinstance(m, torch.nn.Dropout) and m.training and m.p > 0:
            return False
        if isinstance(m, vae_wan.RMS_norm) and (isinstance(m.bias, torch.Tensor) or m.gamma.numel() > 1024):
            return False
        if isinstance(m, (torch.nn.Conv2d, torch.nn.Conv3d)) and m is not encoder.conv1 and m.in_channels % 16:
            return False
    return True


def _only_the_result_is_wanted(x: torch.Tensor, module) -> bool:
    """No gradient, no functional transform, no tracing and no mode or global hook that would want to see the single operators."""
    glob = torch.nn.modules.module
    return (not (torch.is_grad_enabled() and (x.requires_grad or any(p.requires_grad for p in module.parameters())))
            and torch._C._len_torch_dispatch_stack() == 0 and torch._C._len_torch_function_stack() == 0
            and torch._C._functorch.peek_interpreter_stack() is None and not torch.compiler.is_compiling() and not torch.jit.is_tracing()
            and not glob._global_forward_hooks and not glob._global_forward_pre_hooks)


def encoder_supported(x: torch.Tensor, encoder) -> bool:
    """The kernel encoder serves bf16 CUDA videos, one at a time, whole frames (row-sharded encoding stays on the torch path),
    whose frames halve three times without a remainder (the kernel serves ragged tiles; 29 frames of 768 x 432, which are not whole
    16 x 8 pixel tiles at the last level: 218 ms on torch convolutions, 44 ms here). Frames that are whole tiles always go there; for
    the others the torch modules stay where their result can be differentiated, hooked or is made by other layers."""
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.shape[0] == 1 and x.shape[-2] % 8 == 0 and x.shape[-1] % 8 == 0
            and vae_parallel.active() is None and native.available() and hasattr(native.load(), "conv_cl")
            and not native.forward_mode()):
        return False
    return (x.shape[-2] % 64 == 0 and x.shape[-1] % 128 == 0) or (_restated(encoder) and _only_the_result_is_wanted(x, encoder))
