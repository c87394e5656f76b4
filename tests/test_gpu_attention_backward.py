"""The single-pass attention backward's dQ buffer: blocked by tiles of 128 queries, the last of them partly empty, for several batch items
and heads. Compared with the two-kernel backward, which has no such buffer, and with double precision."""

import math

import pytest
import torch

from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
# P, dS and the result are rounded to bf16 once each: 2^-9 at most, 0.58 of it in the 2-norm, three of them; twice that for inputs of few rows
TOL = 2 * math.sqrt(3) * 0.58 * 2.0 ** -9


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("B,Sq,Skv,H", [(2, 200, 300, 2), (3, 129, 257, 1), (1, 127, 128, 1), (2, 1, 128, 3), (2, 260, 2100, 2)])
def test_dq_of_ragged_tiles(B, Sq, Skv, H):
    torch.manual_seed(4)
    ops = native.load()
    q, do = (torch.randn(B, Sq, H, 128, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Skv, H, 128, device=DEV).bfloat16() for _ in range(2))
    scale = 1.0 / math.sqrt(128)
    o, lse = ops.fa_fwd(q, k, v, scale)
    got, want = ops.fa_bwd_variant(do, q, k, v, o, lse, scale, 3), ops.fa_bwd_variant(do, q, k, v, o, lse, scale, 1)
    torch.cuda.synchronize()
    assert ops.kernel_error(0, True) == 0
    qd, kd, vd = (t.double().transpose(1, 2).requires_grad_(True) for t in (q, k, v))
    (torch.softmax(qd @ kd.transpose(2, 3) * scale, -1) @ vd).backward(do.double().transpose(1, 2))
    for g, w, exact in zip(got, want, (qd.grad, kd.grad, vd.grad)):
        exact = exact.transpose(1, 2)
        assert _rel(g, exact) < max(TOL, 1.1 * _rel(w, exact))


# few queries against long keys keep the 128 x 64 kernel, short keys the two-kernel backward; the edges of both lines
@pytest.mark.parametrize("Sq,Skv,kernel", [(1, 2048, 2), (200, 2100, 2), (256, 2048, 2), (257, 2048, 3), (300, 2047, 1), (100, 512, 1)])
def test_kernel_by_lengths(Sq, Skv, kernel):
    torch.manual_seed(6)
    ops = native.load()
    assert ops.fa_bwd_kernel(Sq, Skv) == kernel
    q, do = (torch.randn(2, Sq, 2, 128, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(2, Skv, 2, 128, device=DEV).bfloat16() for _ in range(2))
    o, lse = ops.fa_fwd(q, k, v, 0.1)
    got = ops.fa_bwd(do, q, k, v, o, lse, 0.1)
    torch.cuda.synchronize()
    assert ops.kernel_error(0, True) == 0
    qd, kd, vd = (t.double().transpose(1, 2).requires_grad_(True) for t in (q, k, v))
    (torch.softmax(qd @ kd.transpose(2, 3) * 0.1, -1) @ vd).backward(do.double().transpose(1, 2))
    for g, exact in zip(got, (qd.grad, kd.grad, vd.grad)):
        assert _rel(g, exact.transpose(1, 2)) < TOL
