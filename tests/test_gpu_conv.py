"""The channels-last implicit-GEMM convolution kernel against ``F.conv3d`` / ``F.conv2d`` in fp32, and the channels-last VAE
decoder built on it against the torch decoder it restates."""

import pytest
import torch
import torch.nn.functional as F

from cosmos_predict25_b200.ops import functional as F_ops
from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(a, b, atol, rtol, name=""):
    a, b = a.float(), b.float()
    assert a.shape == b.shape, (a.shape, b.shape)
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    bad = (err > tol).float().mean().item()
    assert bad < 1e-4 and (err / tol).max().item() < 8, f"{name}: {bad * 100:.3f}% out of tolerance, max err {err.max().item():.4g}"


def _no_kernel_error():
    torch.cuda.synchronize()
    code = native.load().kernel_error(torch.cuda.current_device(), True)
    assert code == 0, f"a kernel reported bounded-wait error code {code}"


# (T, H, W, Cin, Cout): whole tiles; ragged frame (H, W not multiples of 8 / 16); 96 channels (a half-filled channel block);
# more output channels than one N tile; an N tile of 16 with 3 real channels (the decoder head)
@pytest.mark.parametrize("T,H,W,Cin,Cout", [(2, 16, 32, 64, 64), (3, 11, 20, 128, 192), (2, 24, 48, 96, 96), (1, 8, 16, 192, 384),
                                            (2, 9, 17, 96, 3), (2, 8, 16, 64, 768)])
def test_causal_conv3d_matches_torch(T, H, W, Cin, Cout):
    from cosmos_predict25_b200.models import vae_wan, vae_wan_cl
    torch.manual_seed(0)
    conv = vae_wan.CausalConv3d(Cin, Cout, 3, padding=1).to(DEV)
    conv.weight.data = conv.weight.data.bfloat16().float()
    x = torch.randn(1, Cin, T, H, W, device=DEV).bfloat16()
    cache = torch.randn(1, Cin, 2, H, W, device=DEV).bfloat16()
    want = conv(x.float(), cache.float())                                        # [1, Cout, T, H, W]
    cl = vae_wan_cl._conv3d(conv, DEV)
    xin = torch.cat([cache, x], 2)[0].permute(1, 2, 3, 0).contiguous()           # [T + 2, H, W, Cin]
    resid = torch.randn(T, H, W, Cout, device=DEV).bfloat16() if Cout % 8 == 0 else None
    got = cl(xin, T, resid=resid)
    _no_kernel_error()
    ref = want[0].permute(1, 2, 3, 0)
    if resid is not None:
        ref = ref + resid.float()
    _close(got, ref, 2e-2 * (27 * Cin) ** 0.5 / 8, 2e-2, "conv3d")


# voxel lines along the width or the height (whichever leaves fewer tiles), frames around the 8 x 16 and 16 x 16 tiles, one and two tiles per
# CTA, channel blocks of 16, 64 and 64 + 32; squares of taps in any order, and lists that are no squares (a box for each tap)
_LISTS = {"3x3": [(0, i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)], "2x2": [(0, i, j) for j in (0, 1) for i in (-1, 0)],
          "3x3x2": [(t, i, j) for j in (-1, 0, 1) for t in (1, 0) for i in (-1, 0, 1)], "rows": [(0, i, 0) for i in (-1, 0, 1)],
          "columns": [(0, 0, j) for j in (1, 0, -1)], "3x2": [(0, i, j) for i in (-1, 0, 1) for j in (0, 1)], "one": [(0, 1, -2)]}


@pytest.mark.parametrize("H,W", [(8, 16), (16, 8), (7, 33), (40, 9), (17, 17), (33, 31)])
@pytest.mark.parametrize("taps", sorted(_LISTS))
@pytest.mark.parametrize("Cin,Cout", [(16, 24), (96, 96), (64, 192), (96, 256)])
def test_taps_read_one_box(H, W, taps, Cin, Cout):
    from cosmos_predict25_b200.models import vae_wan_cl
    torch.manual_seed(15)
    lst = _LISTS[taps]
    w = (torch.randn(Cout, len(lst), Cin, device=DEV) / (len(lst) * Cin) ** 0.5).bfloat16()
    cl = vae_wan_cl.ConvCL(w, torch.randn(Cout, device=DEV), lst, DEV)
    x = torch.randn(3, H, W, Cin, device=DEV).bfloat16()
    got = cl(x, 2)
    _no_kernel_error()
    pad = F.pad(x.double(), (0, 0, 2, 2, 1, 1, 0, 0))
    want = cl.bias.double().expand(2, H, W, Cout).clone()
    for n, (dt, dh, dw) in enumerate(lst):
        want += pad[dt:dt + 2, 1 + dh:1 + dh + H, 2 + dw:2 + dw + W] @ w[:, n].double().t()
    # one rounding to bf16; the fp32 sums of at most 1,728 products stay far below it
    assert ((got.double() - want).norm() / want.norm()).item() < 1.5 * 2.0 ** -9
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


# a box for each column of taps: squares of a layer of 16 output channels, columns of three and two rows; one and two tiles per CTA
_COLUMNS = {"3x3": _LISTS["3x3"], "3x3x2": _LISTS["3x3x2"], "3x2": _LISTS["3x2"], "2x1": [(t, i, 1) for t in (0, 1) for i in (0, -1)]}


@pytest.mark.parametrize("H,W", [(17, 33), (40, 9), (32, 48)])
@pytest.mark.parametrize("taps", sorted(_COLUMNS))
def test_columns_of_taps_read_one_box(H, W, taps):
    from cosmos_predict25_b200.models import vae_wan_cl
    torch.manual_seed(17)
    lst = _COLUMNS[taps]
    w = (torch.randn(16, len(lst), 96, device=DEV) / (len(lst) * 96) ** 0.5).bfloat16()
    cl = vae_wan_cl.ConvCL(w, torch.randn(16, device=DEV), lst, DEV)
    assert native.load().conv_panels(cl.taps, 1, 96, cl.n_tile)[:2] == [2 if taps == "2x1" else 3, 1]
    x = torch.randn(3, H, W, 96, device=DEV).bfloat16()
    got = cl(x, 2)
    _no_kernel_error()
    pad = F.pad(x.double(), (0, 0, 2, 2, 1, 1, 0, 0))
    want = cl.bias.double().expand(2, H, W, 16).clone()
    for n, (dt, dh, dw) in enumerate(lst):
        want += pad[dt:dt + 2, 1 + dh:1 + dh + H, 2 + dw:2 + dw + W] @ w[:, n].double().t()
    # one rounding to bf16; the fp32 sums of at most 1,728 products stay far below it
    assert ((got.double() - want).norm() / want.norm()).item() < 1.5 * 2.0 ** -9
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


def test_upsample_phase_convolutions_match_nearest_then_conv():
    from cosmos_predict25_b200.models import vae_wan, vae_wan_cl
    torch.manual_seed(1)
    mod = vae_wan.Resample(128, "upsample2d").to(DEV)
    conv = mod.resample[1]
    conv.weight.data = conv.weight.data.bfloat16().float()
    T, H, W = 2, 12, 20
    x = torch.randn(T, H, W, 128, device=DEV).bfloat16()
    up = vae_wan_cl._UpsampleCL(mod, DEV)
    got = up(x, vae_wan_cl._Stream())
    _no_kernel_error()
    want = conv(F.interpolate(x.float().permute(0, 3, 1, 2), scale_factor=2.0, mode="nearest-exact")).permute(0, 2, 3, 1)
    _close(got, want, 6e-2, 3e-2, "upsample + conv2d")


# chunk lengths x kernel shape: one image (all but one frame of taps is padding), a one-frame first chunk (its cache is shorter than
# the padding), one-frame chunks, longer ones; an odd number of voxel tiles; 3, 2 and 1 taps per box; an N tile of 16
@pytest.mark.parametrize("chunks", [(1,), (1, 1, 1), (1, 4, 2), (3,), (2, 3)])
@pytest.mark.parametrize("ksize,H,W,Cin,Cout", [((3, 3, 3), 9, 17, 96, 96), ((3, 1, 1), 24, 16, 32, 64), ((3, 3, 3), 8, 16, 64, 3),
                                                ((3, 2, 2), 13, 40, 160, 384)])
def test_streamed_causal_convolution_reads_cached_frames(chunks, ksize, H, W, Cin, Cout):
    from cosmos_predict25_b200.models import vae_wan_cl
    torch.manual_seed(5)
    kt, kh, kw = ksize
    w = (torch.randn(Cout, Cin, kt, kh, kw, device=DEV) / (Cin * kt * kh * kw) ** 0.5).bfloat16().float()
    b = torch.randn(Cout, device=DEV)
    x = torch.randn(1, Cin, sum(chunks), H, W, device=DEV).bfloat16()
    want = F.conv3d(F.pad(x.float(), (kw // 2, (kw - 1) // 2, kh // 2, (kh - 1) // 2, kt - 1, 0)), w, b)[0].permute(1, 2, 3, 0)
    cl = vae_wan_cl.ConvCL(w.permute(0, 2, 3, 4, 1).reshape(Cout, -1, Cin), b, vae_wan_cl._causal3_taps(kt, kh, kw), DEV)
    st, got, lo = vae_wan_cl._Stream(), [], 0
    for n in chunks:
        got.append(cl.causal(x[0, :, lo:lo + n].permute(1, 2, 3, 0).contiguous(), st))
        lo += n
    _no_kernel_error()
    # unit-variance products summed in fp32, stored in bf16: half an ulp relative, plus the order of the sums
    _close(torch.cat(got, 0), want, 4e-3, 1e-2, "streamed conv")


@pytest.mark.parametrize("H,W,C", [(16, 32, 96), (22, 50, 32), (54, 96, 192), (2, 4, 384)])
def test_strided_convolutions_match_torch_resample(H, W, C):
    """The encoder's down-sampling (spatial stride 2 with bottom / right padding, causal temporal stride 2) chunk by chunk."""
    from cosmos_predict25_b200.models import vae_wan, vae_wan_cl
    torch.manual_seed(6)
    mod = vae_wan.Resample(C, "downsample3d").to(DEV)
    for p in mod.parameters():
        p.data = p.data.bfloat16().float()
    cl, st, st_t = vae_wan_cl._DownsampleCL(mod, DEV), vae_wan_cl._Stream(), vae_wan.StreamState()
    for T in (1, 4, 8, 2):
        x = torch.randn(1, C, T, H, W, device=DEV).bfloat16()
        with torch.no_grad():
            want = mod(x.float(), st_t)[0].permute(1, 2, 3, 0)
        got = cl(x[0].permute(1, 2, 3, 0).contiguous(), st)
        _no_kernel_error()
        _close(got, want, 3e-2, 2e-2, f"down-sampling, chunk of {T}")


# one and several 32-channel chunks per column half, uneven halves; N tiles that are no whole chunks; with and without residual and raw
# output; the interleaved output of an up-sampling phase
@pytest.mark.parametrize("Cout", [8, 48, 96, 192, 256])
@pytest.mark.parametrize("silu,raw,resid", [(True, False, False), (False, True, True), (True, True, False)])
def test_norm_in_the_epilogue(Cout, silu, raw, resid):
    from cosmos_predict25_b200.models import vae_wan_cl
    torch.manual_seed(9)
    T, H, W, Cin = 2, 11, 20, 64
    w = (torch.randn(Cout, Cin, 3, 3, 3, device=DEV) / (27 * Cin) ** 0.5).bfloat16().float()
    b, g = torch.randn(Cout, device=DEV), 1 + 0.2 * torch.randn(Cout, device=DEV)
    cl = vae_wan_cl.ConvCL(w.permute(0, 2, 3, 4, 1).reshape(Cout, -1, Cin), b, vae_wan_cl._causal3_taps(3, 3, 3), DEV)
    x = torch.randn(1, Cin, T, H, W, device=DEV).bfloat16()
    r = torch.randn(T, H, W, Cout, device=DEV).bfloat16() if resid else None
    y, n = cl.causal(x[0].permute(1, 2, 3, 0).contiguous(), vae_wan_cl._Stream(), resid=r, norm=(g, silu), raw=raw)
    _no_kernel_error()
    want = F.conv3d(F.pad(x.float(), (1, 1, 1, 1, 2, 0)), w, b)[0].permute(1, 2, 3, 0) + (r.float() if resid else 0)
    wn = F.normalize(want, dim=-1) * Cout ** 0.5 * g
    assert cl.fuses_norm(x) and (y is not None) == raw
    if raw:
        _close(y, want, 4e-3, 1e-2, "conv")
    _close(n, F.silu(wn) if silu else wn, 4e-3, 1e-2, "norm of the conv")


def _band(monkeypatch, whole, lo, hi):
    """Makes the layers believe that they hold rows [lo, hi) of a frame: the boundary rows come out of ``whole()``, the whole tensor."""
    from cosmos_predict25_b200.models import vae_parallel

    def exchange_rows(x, dim, n, top=True, bottom=True):
        f = F.pad(whole(), (0, 0, 0, 0, n, n))
        return f[:, lo:hi + 2 * n].contiguous()

    monkeypatch.setattr(vae_parallel, "_active", (None, 0, 2))
    monkeypatch.setattr(vae_parallel, "exchange_rows", exchange_rows)


@pytest.mark.parametrize("lo,hi", [(0, 7), (7, 20), (20, 24)])
def test_row_bands_equal_the_whole_frame(lo, hi, monkeypatch):
    """A band of rows with its neighbours' boundary rows (row-sharded decoding), chunk by chunk: the cached frames keep theirs. The ranks'
    exchange is replaced by reading the whole tensor."""
    from cosmos_predict25_b200.models import vae_wan, vae_wan_cl
    torch.manual_seed(14)
    C, H, W = 64, 24, 20
    w = torch.randn(96, C, 3, 3, 3, device=DEV) / (27 * C) ** 0.5
    cl = vae_wan_cl.ConvCL(w.permute(0, 2, 3, 4, 1).reshape(96, -1, C), torch.randn(96, device=DEV), vae_wan_cl._causal3_taps(3, 3, 3), DEV)
    up = vae_wan_cl._UpsampleCL(vae_wan.Resample(C, "upsample2d").to(DEV), DEV)
    norms = (1 + 0.1 * torch.randn(96, device=DEV), True), (torch.ones(C // 2, device=DEV), True)
    chunks = [torch.randn(T, H, W, C, device=DEV).bfloat16() for T in (1, 1, 4, 2)]
    st = vae_wan_cl._Stream()
    want = [(cl.causal(x, st, norm=norms[0]), up.run(x, st, None, norms[1])) for x in chunks]
    st, now = vae_wan_cl._Stream(), []
    _band(monkeypatch, lambda: now[-1], lo, hi)
    for x, (conv, ups) in zip(chunks, want):
        now.append(x)
        band = x[:, lo:hi].contiguous()
        for got, full in zip(cl.causal(band, st, norm=norms[0]), conv):
            assert torch.equal(got, full[:, lo:hi])
        for got, full in zip(up.run(band, st, None, norms[1]), ups):
            assert torch.equal(got, full[:, 2 * lo:2 * hi])
    _no_kernel_error()


def test_operands_that_the_kernels_cannot_read_are_refused():
    """Outputs off a 16-byte boundary (they are moved as 16-byte pieces) and a softmax scale that is not positive."""
    from cosmos_predict25_b200.models import vae_wan_cl
    cl = vae_wan_cl.ConvCL(torch.randn(64, 1, 64), None, [(0, 0, 0)], DEV)
    x, g = torch.randn(1, 8, 16, 64, device=DEV).bfloat16(), torch.ones(64, device=DEV)
    whole, odd = (torch.zeros(1 + x.numel(), device=DEV).bfloat16()[o:o + x.numel()].view_as(x) for o in (0, 1))
    for y, resid, norm in ((odd, None, None), (whole, odd, None), (whole, None, odd)):
        with pytest.raises(RuntimeError, match="16-byte"):
            cl._launch(x, cl.taps, 1, 8, 16, y, None, resid, norm=None if norm is None else (g, True), normed=norm)
    cl3 = vae_wan_cl.ConvCL(torch.randn(3, 1, 64), None, [(0, 0, 0)], DEV)          # channels that are stored one by one may lie anywhere
    y = torch.zeros(1 + 128 * 3, device=DEV).bfloat16()[1:].view(1, 8, 16, 3)
    assert torch.equal(cl3._launch(x, cl3.taps, 1, 8, 16, y, None, None), cl3(x, 1))
    q = torch.randn(1, 64, 384, device=DEV).bfloat16()
    for scale in (0.0, -0.1, float("nan")):
        with pytest.raises(RuntimeError, match="positive"):
            native.load().fa_wide(q, q, q, scale)
    _no_kernel_error()


def test_norm_behind_upsampling_phases():
    from cosmos_predict25_b200.models import vae_wan, vae_wan_cl
    torch.manual_seed(10)
    mod = vae_wan.Resample(128, "upsample2d").to(DEV)
    up, g = vae_wan_cl._UpsampleCL(mod, DEV), 1 + 0.2 * torch.randn(64, device=DEV)
    x = torch.randn(2, 12, 20, 128, device=DEV).bfloat16()
    y, n = up.run(x, vae_wan_cl._Stream(), None, (g, True))
    _no_kernel_error()
    assert torch.equal(y, up(x, vae_wan_cl._Stream()))
    _close(n, F.silu(F.normalize(y.float(), dim=-1) * 8 * g), 1e-2, 2e-2, "norm")       # the epilogue normalises before y is rounded


def test_wide_attention_waits_end():
    """Many launches beside a second stream's traffic, which delays single warps: no bounded wait may run out and every result is the
    same. (A softmax warp that was late once waited for a phase that only itself could bring about.)"""
    torch.manual_seed(13)
    qkv = torch.randn(4, 2000, 3, 384, device=DEV).bfloat16()
    want = native.load().fa_wide(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], 384 ** -0.5)
    side, noise = torch.cuda.Stream(), torch.randn(64 << 20, device=DEV)
    outs = []
    for i in range(200):
        with torch.cuda.stream(side):
            noise.mul_(1.0)
        outs.append(native.load().fa_wide(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], 384 ** -0.5))
        if len(outs) == 20:
            assert all(torch.equal(o, want) for o in outs)
            outs.clear()
    _no_kernel_error()


# queries and keys: below one tile, whole tiles, one row over, an odd and an even number of key tiles; large scores move the reference maximum
@pytest.mark.parametrize("B,Sq,Skv,gain", [(1, 5, 7, 1.0), (2, 128, 64, 1.0), (1, 129, 65, 4.0), (3, 300, 1000, 8.0), (1, 1024, 1024, 1.0)])
def test_wide_attention_matches_fp32(B, Sq, Skv, gain):
    torch.manual_seed(8)
    qkv = torch.randn(B, max(Sq, Skv), 3, 384, device=DEV).bfloat16()
    q, k, v = qkv[:, :Sq, 0] * gain, qkv[:, :Skv, 1] * torch.linspace(0.2, 2, Skv, device=DEV)[:, None].bfloat16(), qkv[:, :Skv, 2]
    got = native.load().fa_wide(q, k, v, 384 ** -0.5)
    _no_kernel_error()
    want = F.scaled_dot_product_attention(*(t.float().unsqueeze(1) for t in (q, k, v))).squeeze(1)
    # probabilities and the result are rounded to bf16: 2^-9 of a weighted mean of unit-variance values each, plus the order of the sums
    _close(got, want, 1e-2, 1e-2, "attention of width 384")


@pytest.mark.parametrize("C", [8, 16, 24, 32, 48, 56, 96, 160, 192, 384, 392, 512, 520, 768, 776, 1024])
def test_rmsnorm_silu_widths(C):
    torch.manual_seed(7)
    x = torch.randn(3, 5, 7, C, device=DEV).bfloat16()
    x[0, 0, 0] = 0
    g = (1 + 0.1 * torch.randn(C + 1, device=DEV)).float()[1:]             # four bytes off a 16-byte boundary
    for silu in (True, False):
        want = F.normalize(x.float(), dim=-1) * C ** 0.5 * g
        _close(native.load().rmsnorm_silu_cl(x, g, silu), F.silu(want) if silu else want, 4e-3, 8e-3, f"rmsnorm {C}")


@pytest.mark.parametrize("C,n", [(384, 444 * 16 * 2 + 5), (192, 444 * 32 + 1), (96, 444 * 64 * 3 - 1), (32, 444 * 128 + 77), (1024, 444 * 8 * 2 + 3), (16, 444 * 128 + 5),
                                 (512, 444 * 8 + 3), (768, 444 * 8 * 2 + 1)])
def test_rmsnorm_silu_of_more_voxels_than_one_pass(C, n):
    """Lanes go on from voxel to voxel: every voxel's result is the one it has in a call of its own few."""
    torch.manual_seed(16)
    x, g = torch.randn(n, C, device=DEV).bfloat16(), 1 + 0.1 * torch.randn(C, device=DEV)
    got = native.load().rmsnorm_silu_cl(x, g, True)
    for lo in (0, 444 * 256 // max(C // 8, 1) // 8 * 8, n // 2, max(n - 40, 0)):
        assert torch.equal(got[lo:lo + 40], native.load().rmsnorm_silu_cl(x[lo:lo + 40].contiguous(), g, True))


def test_rmsnorm_silu_channels_last():
    torch.manual_seed(2)
    x = torch.randn(5, 7, 9, 96, device=DEV).bfloat16()
    g = (1 + 0.1 * torch.randn(96, device=DEV)).float()
    got = native.load().rmsnorm_silu_cl(x, g, True)
    want = F.silu(F.normalize(x.float(), dim=-1) * 96 ** 0.5 * g)
    _close(got, want, 2e-2, 2e-2, "rmsnorm+silu")


def test_channels_last_decoder_matches_torch_decoder():
    """Whole streaming decode (3 latent frames -> 9 pixel frames) on the kernel path against the torch modules in fp32."""
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    torch.manual_seed(3)
    vae = WanVAE_(dim=32, z_dim=16).eval().requires_grad_(False).to(DEV)
    for p in vae.parameters():
        p.data = p.data.bfloat16().float()
    z = torch.randn(1, 16, 3, 16, 32, device=DEV)
    F_ops.settings.conv = "cudnn"
    try:
        want = vae.decode(z, (0.0, 1.0))
    finally:
        F_ops.settings.conv = "native"
    vae16 = vae.to(torch.bfloat16)
    got = vae16.decode(z.bfloat16(), (0.0, 1.0))
    _no_kernel_error()
    assert got.shape == want.shape == (1, 3, 9, 128, 256)
    assert getattr(vae16, "_dec_cl", None) is not None, "the kernel decoder did not serve the bf16 decode"
    err = (got.float() - want).abs()
    scale = want.abs().mean().item()
    assert err.mean().item() < 0.03 * scale + 1e-3 and err.max().item() < 0.5 * want.abs().max().item() + 0.05, \
        f"mean err {err.mean().item():.4g} (signal {scale:.4g}), max err {err.max().item():.4g}"


def test_channels_last_encoder_matches_torch_encoder():
    """Whole streaming encode (1 + 4 + 4 pixel frames -> 3 latent frames) on the kernel path against the torch modules in fp32."""
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    torch.manual_seed(4)
    vae = WanVAE_(dim=32, z_dim=16).eval().requires_grad_(False).to(DEV)
    for p in vae.parameters():
        p.data = p.data.bfloat16().float()
    x = torch.randn(1, 3, 9, 128, 256, device=DEV).clamp(-1, 1)
    F_ops.settings.conv = "cudnn"
    try:
        want = vae.encode(x, (0.0, 1.0))
    finally:
        F_ops.settings.conv = "native"
    vae16 = vae.to(torch.bfloat16)
    before = native.launches()
    got = vae16.encode(x.bfloat16(), (0.0, 1.0))
    _no_kernel_error()
    assert got.shape == want.shape == (1, 16, 3, 16, 32)
    assert getattr(vae16, "_enc_cl", None) is not None and native.launches() - before > 30, "the kernel encoder did not serve the bf16 encode"
    err = (got.float() - want).abs()
    scale = want.abs().mean().item()
    assert err.mean().item() < 0.03 * scale + 1e-3 and err.max().item() < 0.5 * want.abs().max().item() + 0.05, \
        f"mean err {err.mean().item():.4g} (signal {scale:.4g}), max err {err.max().item():.4g}"


@pytest.mark.parametrize("step_bytes", [1, 2 << 20, 3 << 29])
def test_frames_per_step_do_not_change_the_result(step_bytes, monkeypatch):
    """One latent frame / encoder window per step, a few, and all of them; one call and a stream that goes on over several calls."""
    from cosmos_predict25_b200.models import vae_wan_cl
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    torch.manual_seed(11)
    vae = WanVAE_(dim=32, z_dim=16).eval().requires_grad_(False).to(DEV).bfloat16()
    z = torch.randn(1, 16, 6, 9, 20, device=DEV).bfloat16()
    x = torch.randn(1, 3, 21, 72, 104, device=DEV).clamp(-1, 1).bfloat16()      # 1 frame and 5 windows
    one = (0.0, 1.0)
    want = vae.decode(z, one), vae.encode(x, one)
    monkeypatch.setattr(vae_wan_cl, "STEP_BYTES", step_bytes)
    got = vae.decode(z, one), vae.encode(x, one)
    parts = [vae.decode(z[:, :, :1], one, clear_decoder_cache=False), vae.decode(z[:, :, 1:4], one, clear_decoder_cache=False),
             vae.decode(z[:, :, 4:], one, clear_decoder_cache=False)]
    vae.clear_cache()
    vae._dec_cl.reset()
    _no_kernel_error()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and torch.equal(torch.cat(parts, 2), want[0])


@pytest.mark.parametrize("step_bytes", [1, 2 << 20, 3 << 29])
@pytest.mark.parametrize("frames", [4, 7, 8, 27])
def test_clip_lengths_with_a_remainder_are_refused(frames, step_bytes, monkeypatch):
    """A clip is one frame and groups of four; what is left over is refused by the kernel encoder as by the torch one, however many
    windows a step takes."""
    from cosmos_predict25_b200.models import vae_wan_cl
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    vae = WanVAE_(dim=32, z_dim=16).eval().requires_grad_(False).to(DEV).bfloat16()
    x = torch.zeros(1, 3, frames, 72, 104, device=DEV).bfloat16()
    monkeypatch.setattr(vae_wan_cl, "STEP_BYTES", step_bytes)
    for conv in ("native", "cudnn"):
        monkeypatch.setattr(F_ops.settings, "conv", conv)
        with pytest.raises(RuntimeError):
            vae.encode(x, (0.0, 1.0))
    monkeypatch.setattr(F_ops.settings, "conv", "native")
    assert vae.encode(x[:, :, :1].expand(-1, -1, 9, -1, -1), (0.0, 1.0)).shape == (1, 16, 3, 9, 13)
    _no_kernel_error()


def test_ragged_frames_stay_on_torch_where_more_than_the_result_is_wanted():
    """Frames that the kernel encoder came to serve last: gradients of pixels and weights, hooks and channel counts that the kernel does not
    take still go through the torch modules."""
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    torch.manual_seed(15)
    vae = WanVAE_(dim=16, z_dim=16, num_res_blocks=1).eval().requires_grad_(False).to(DEV).bfloat16()
    x = torch.randn(1, 3, 5, 24, 40, device=DEV).clamp(-1, 1).bfloat16()
    plain = vae.encode(x, (0.0, 1.0))
    assert vae._enc_cl is not None
    scale = plain.float().norm().item()
    xg = x.clone().requires_grad_(True)
    out = vae.encode(xg, (0.0, 1.0))
    out.float().sum().backward()
    assert xg.grad is not None and xg.grad.abs().sum().item() > 0
    vae.requires_grad_(True)
    vae.encode(x, (0.0, 1.0)).float().sum().backward()
    assert vae.encoder.conv1.weight.grad is not None
    vae.requires_grad_(False)
    seen = []
    hook = vae.encoder.middle[1].register_forward_hook(lambda m, a, o: seen.append(o.shape))
    hooked = vae.encode(x, (0.0, 1.0))
    hook.remove()
    assert len(seen) == 2                                    # the first frame and one window
    for y in (out.detach(), hooked):
        assert (y.float() - plain.float()).norm().item() < 0.05 * scale
    odd = WanVAE_(dim=24, z_dim=16, num_res_blocks=1).eval().requires_grad_(False).to(DEV).bfloat16()
    assert odd.encode(x, (0.0, 1.0)).shape == plain.shape and getattr(odd, "_enc_cl", None) is None
    small = vae.encode(x[..., :8, :8], (0.0, 1.0))           # one latent pixel
    F_ops.settings.conv = "cudnn"
    try:
        want = vae.encode(x[..., :8, :8], (0.0, 1.0))
    finally:
        F_ops.settings.conv = "native"
    assert small.shape == want.shape == (1, 16, 2, 1, 1) and (small.float() - want.float()).norm().item() < 0.05 * want.float().norm().item()
    _no_kernel_error()


@pytest.mark.parametrize("H,W,T", [(72, 104, 9), (24, 40, 5), (432, 136, 1)])
def test_ragged_frames_are_encoded_by_the_kernel(H, W, T):
    """Frames that halve three times but are no whole tiles, against the torch encoder in fp32 (bounds of the whole-tile test above)."""
    from cosmos_predict25_b200.models.vae_wan import WanVAE_
    torch.manual_seed(12)
    vae = WanVAE_(dim=32, z_dim=16).eval().requires_grad_(False).to(DEV)
    for p in vae.parameters():
        p.data = p.data.bfloat16().float()
    x = torch.randn(1, 3, T, H, W, device=DEV).clamp(-1, 1)
    F_ops.settings.conv = "cudnn"
    try:
        want = vae.encode(x, (0.0, 1.0))
    finally:
        F_ops.settings.conv = "native"
    vae16 = vae.to(torch.bfloat16)
    got = vae16.encode(x.bfloat16(), (0.0, 1.0))
    _no_kernel_error()
    assert getattr(vae16, "_enc_cl", None) is not None and got.shape == want.shape
    err, scale = (got.float() - want).abs(), want.abs().mean().item()
    assert err.mean().item() < 0.03 * scale + 1e-3 and err.max().item() < 0.5 * want.abs().max().item() + 0.05
