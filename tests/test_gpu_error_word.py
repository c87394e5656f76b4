"""After a kernel has reported an error, the kernels behind it return at once and leave their outputs as they are."""

import pytest
import torch

from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _set_error(flags, lonely):
    """A peer barrier whose flag nobody sets: it gives up after a millisecond and reports 101."""
    native.load().peer_barrier([flags.data_ptr(), lonely.data_ptr()], 0, 1, 0, 1000)


def _conv():
    from cosmos_predict25_b200.models import vae_wan_cl
    cl = vae_wan_cl.ConvCL(torch.randn(96, 27, 64), torch.randn(96), vae_wan_cl._causal3_taps(3, 3, 3), DEV)
    x, g = torch.randn(6, 40, 48, 64, device=DEV).bfloat16(), torch.ones(96, device=DEV)
    out = torch.empty(4, 40, 48, 96, dtype=torch.bfloat16, device=DEV)
    run = lambda: cl._launch(x, cl.taps, 4, 40, 48, out, None, None, norm=(g, True))[0]
    return run, out.numel()


def _wide():
    qkv = torch.randn(2, 1500, 3, 384, device=DEV).bfloat16()
    return lambda: native.load().fa_wide(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], 384 ** -0.5), 2 * 1500 * 384


def _attention():
    q, k, v = (torch.randn(1, 2000, 4, 128, device=DEV).bfloat16() for _ in range(3))
    return lambda: native.load().fa_fwd(q, k, v, 128 ** -0.5)[0], 2000 * 4 * 128


@pytest.mark.parametrize("case", [_conv, _wide, _attention])
def test_kernels_behind_an_error_return_at_once(case):
    run, n = case()
    native.load().kernel_error(0, True)
    want = run().clone()
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 0
    flags = [torch.zeros(64, dtype=torch.int32, device=DEV) for _ in range(2)]
    torch.cuda.empty_cache()
    marked = torch.full((n,), 7.0, dtype=torch.bfloat16, device=DEV)
    if case is _conv:
        run().fill_(7.0)
    else:
        del marked                                   # the output allocated next lies where the marks are
    _set_error(*flags)
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    begin.record()
    out = run()
    end.record()
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 101
    assert (out == 7.0).all(), "the kernel ran on after an earlier error"
    assert begin.elapsed_time(end) < 100            # far below the two seconds of one bounded wait
    again = run()
    torch.cuda.synchronize()
    assert native.load().kernel_error(0, True) == 0 and torch.equal(again, want)
