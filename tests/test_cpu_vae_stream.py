"""How the VAE cuts a clip into streaming steps, with the channels-last encoder replaced by a recorder (host logic only)."""

import pytest
import torch

from cosmos_predict25_b200.models import vae_wan, vae_wan_cl


class _Recorder:
    """Stands for ``EncoderCL``: the chunks it is given, the real rule for windows per step."""

    def __init__(self, base_channels):
        self.state, self.chunks = None, []
        self.conv1 = type("C", (), {"cout": base_channels})
        self.windows_per_step = lambda *a: vae_wan_cl.EncoderCL.windows_per_step(self, *a)

    def reset(self):
        self.state = object()

    def step(self, x):
        self.chunks.append(x.shape[2])
        return torch.zeros(1, 32, max(1, x.shape[2] // 4), x.shape[3] // 8, x.shape[4] // 8)


@pytest.mark.parametrize("frames", [1, 4, 5, 7, 8, 9, 25, 27, 29])
@pytest.mark.parametrize("windows", [1, 2, 6, 100])
@pytest.mark.parametrize("window", [4, 8, 6])
def test_only_whole_windows_share_a_step(frames, windows, window, monkeypatch):
    vae = vae_wan.WanVAE_(dim=8, z_dim=16, num_res_blocks=1, temporal_window=window).eval()
    rec = _Recorder(8)
    monkeypatch.setattr(vae, "_kernel_encoder", lambda x: rec)
    H, W = 16, 24
    monkeypatch.setattr(vae_wan_cl, "STEP_BYTES", windows * window * H * W * 8 * 2)
    with torch.no_grad():
        vae.encode(torch.zeros(1, 3, frames, H, W), (0.0, 1.0))
    whole, rest = divmod(frames - 1, window)
    per_step = windows if window % 4 == 0 else 1
    want = [1] + [min(per_step, whole - i) * window for i in range(0, whole, per_step)] + ([rest] if rest else [])
    assert rec.chunks == want


@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("chunks", [(1, 8, 8), (1, 1, 1, 3), (4,), (2, 1), (1, 2)])
def test_stream_keeps_the_last_frames_only(n, chunks):
    """What a causal convolution carries to the next chunk: at most its ``n`` last input frames, in storage of that size."""
    frames = torch.randn(sum(chunks), 3, 5, 4)
    prev, lo = None, 0
    for T in chunks:
        x = frames[lo:lo + T].clone()
        lo += T
        prev = vae_wan_cl._last_frames(prev, x, n)
        assert torch.equal(prev, frames[max(0, lo - n):lo]) and prev.is_contiguous()
        assert prev.untyped_storage().nbytes() <= n * frames[0].numel() * 4


def test_what_the_kernel_encoder_restates():
    """Channel counts, hooks, other layers and active dropout keep the torch modules."""
    enc = lambda **kw: vae_wan.Encoder3d(dim=kw.pop("dim", 16), z_dim=8, num_res_blocks=1, **kw).eval()
    ok = vae_wan_cl._restated
    assert ok(enc()) and ok(enc(dim=96)) and ok(enc(attn_scales=(0.5,))) and ok(enc(dropout=0.1)) and ok(enc(dropout=0.0).train())
    assert not ok(enc(dim=24)) and not ok(enc(dim=8)) and not ok(enc(dim=272)) and not ok(enc(dropout=0.1).train())
    e = enc()
    hook = e.middle[1].register_forward_hook(lambda *a: None)
    assert not ok(e)
    hook.remove()
    assert ok(e)
    e.head[2].forward = e.head[2].forward
    assert not ok(e)
    e = enc()
    e.middle[0].residual[2] = torch.nn.utils.parametrizations.weight_norm(e.middle[0].residual[2])
    assert not ok(e)
    x, want = torch.zeros(1), vae_wan_cl._only_the_result_is_wanted
    e = enc()
    assert not want(x, e)
    with torch.no_grad():
        assert want(x, e)
    e.requires_grad_(False)
    assert want(x, e) and not want(x.clone().requires_grad_(True), e)
