"""Edges of the row-wise kernels: modulation vectors that are slices of a wider buffer, channel counts around the widths a warp
holds, head counts that do not divide a warp's rows, row counts around the tiles of the few-row GEMM."""

import math

import pytest
import torch

from cosmos_predict25_b200.ops import functional as F_ops
from cosmos_predict25_b200.ops import native, ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _max_rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("D,L,T", [(8, 3, 2), (1024, 5, 3), (1032, 4, 1), (2048, 1, 7), (2056, 3, 2), (1024, 1777, 3),
                                   (1800, 3553, 1)])
@pytest.mark.parametrize("offset", [0, 2])
def test_modulation_slices_are_read_in_place(D, L, T, offset):
    """shift / scale / gate as thirds of one buffer; ``offset`` moves them off the 16-byte boundary (they are copied then)."""
    torch.manual_seed(0)
    x = torch.randn(1, T, L, D, device=DEV).bfloat16()
    y = torch.randn(1, T, L, D, device=DEV).bfloat16()
    buf = torch.randn(1, T, 3 * D + 4, device=DEV)
    sh, sc, g = (buf[..., offset + i * D: offset + (i + 1) * D] for i in range(3))
    mean_sq = 2.0 ** -9      # one bf16 rounding of the result (2^-9 relative), measured in the 2-norm
    assert _max_rel(F_ops.ln_modulate(x, sh, sc), ref.ln_modulate(x.double(), sh.double(), sc.double())) < 1.5 * mean_sq
    assert _max_rel(F_ops.gate_residual(x, g, y), x.double() + g.double().unsqueeze(2) * y.double()) < 1.5 * mean_sq
    dout = torch.randn_like(y)
    dy, dg = native.load().gate_residual_bwd(dout.view(-1, D), g.reshape(T, D), y.view(-1, D), L)
    assert _max_rel(dy.view_as(y), dout.double() * g.double().unsqueeze(2)) < 1.5 * mean_sq
    assert _max_rel(dg.view(1, T, D), (dout.double() * y.double()).sum(2)) < 1e-5


# a CTA or a warp per row (few rows, short frames, narrow rows) and batches of rows per CTA: partial warps and partial last pieces of a row, frames that end
# inside a batch, the row counts where the kernel changes, every instantiation
@pytest.mark.parametrize("D,L,T", [(8, 700, 3), (520, 4, 520), (1024, 2047, 1), (2048, 2048, 1), (2040, 41, 53), (2048, 3, 700), (2056, 1023, 1),
                                   (2056, 26, 41), (4104, 513, 2), (5120, 1041, 1), (5128, 130, 8), (8192, 7, 150), (8192, 5, 3),
                                   (256, 3, 691), (504, 1, 2051), (264, 2, 1024), (248, 769, 4), (8, 4097, 1), (256, 4096, 3)])
def test_layernorm_row_counts_and_widths(D, L, T):
    torch.manual_seed(6)
    x = (torch.randn(T * L, D, device=DEV) * 2 + 3 * torch.randn(T * L, 1, device=DEV)).bfloat16()
    mod = torch.randn(T, 2 * D, device=DEV)
    y, mean, rstd = native.load().ln_modulate_fwd(x, mod[:, :D], mod[:, D:], L, 1e-6)
    xd = x.double()
    want_mean, want_rstd = xd.mean(1), torch.rsqrt(xd.var(1, unbiased=False) + 1e-6)
    frame = torch.arange(T * L, device=DEV) // L
    want = (xd - want_mean[:, None]) * want_rstd[:, None] * (1 + mod[:, D:].double()[frame]) + mod[:, :D].double()[frame]
    assert _max_rel(y, want) < 1.5 * 2.0 ** -9
    # fp32 sums of at most 8192 terms in parts of 64 and a tree: a handful of roundings of 2^-24
    assert _max_rel(mean, want_mean) < 1e-6 and _max_rel(rstd, want_rstd) < 1e-6


def test_gated_gemm_epilogue_reads_strided_gates():
    torch.manual_seed(1)
    B, T, L, D, K = 1, 3, 88, 256, 128
    h = torch.randn(B, T * L, K, device=DEV).bfloat16()
    w = (torch.randn(D, K, device=DEV) / math.sqrt(K)).bfloat16()
    x = torch.randn(B, T, L, D, device=DEV).bfloat16()
    gate = torch.randn(B, T, 3 * D, device=DEV)[..., D:2 * D]
    with torch.no_grad():
        got = F_ops.linear_gate_residual(h, w, x, gate)
    want = x.double() + gate.double().unsqueeze(2) * (h.double() @ w.double().t()).view(B, T, L, D)
    assert _max_rel(got, want) < 1.5 * 2.0 ** -9


def test_row_operators_take_modulation_rows_of_any_shape():
    """[frames, D] as [B, T, D], as one flat row and as a strided slice are the same rows; rows that are too few are refused."""
    torch.manual_seed(4)
    ops = native.load()
    B, T, L, D, K = 2, 3, 8, 256, 64
    x, y = (torch.randn(B * T * L, D, device=DEV).bfloat16() for _ in range(2))
    h, w = torch.randn(B * T * L, K, device=DEV).bfloat16(), torch.randn(D, K, device=DEV).bfloat16()
    rows = torch.randn(B * T, D, device=DEV)
    mean, rstd = ops.ln_modulate_fwd(x, rows, rows, L, 1e-6)[1:]
    calls = {
        "gated GEMM": lambda g: ops.gemm_bf16_gate_residual(h, w, x, g, L),
        "gate": lambda g: ops.gate_residual_bwd(y, g, x, L)[0],
        "LN": lambda g: ops.ln_modulate_fwd(x, rows, g, L, 1e-6)[0],
        "LN backward": lambda g: ops.ln_modulate_bwd(y, x, mean, rstd, g, L)[0],
    }
    wide = torch.cat([rows, rows, rows], 1)
    for name, call in calls.items():
        want = call(rows)
        for form in (rows.view(B, T, D), rows.view(-1), wide[:, D:2 * D]):
            if form.dim() != 1 or name != "gated GEMM":          # the epilogue wants D in the last dimension
                assert torch.equal(call(form), want), (name, form.shape)
        with pytest.raises(RuntimeError):
            call(rows[:-1])
    flat = rows[0]                                                # one frame: a plain [D] vector
    assert torch.equal(ops.gemm_bf16_gate_residual(h, w, x, flat, B * T * L), ops.gemm_bf16_gate_residual(h, w, x, flat[None], B * T * L))


@pytest.mark.parametrize("HD,H,S,B", [(128, 5, 7, 2), (128, 16, 33, 1), (64, 3, 130, 2), (128, 40, 3, 1), (64, 1, 1, 1), (64, 8, 37, 1), (128, 12, 50, 2),
                                          (128, 24, 5, 1)])
@pytest.mark.parametrize("wdtype", [torch.bfloat16, torch.float32])
def test_rmsnorm_rope_head_counts(HD, H, S, B, wdtype):
    torch.manual_seed(2)
    x = torch.randn(B, S, H, HD, device=DEV).bfloat16().requires_grad_(True)
    w = (1 + 0.2 * torch.randn(HD, device=DEV)).to(wdtype).requires_grad_(True)
    half = torch.randn(S, HD // 2, device=DEV)
    rope = F_ops.RopeTable(torch.cat([half, half], 1))
    dy = torch.randn(B, S, H, HD, device=DEV).bfloat16()
    for table in (rope, None):
        x.grad = w.grad = None
        y = F_ops.rmsnorm_rope(x, w, table, 1e-6)
        y.backward(dy)
        xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
        n = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
        if table is not None:
            c, s = half.double().cos()[None, :, None], half.double().sin()[None, :, None]
            a, b = n[..., :HD // 2], n[..., HD // 2:]
            n = torch.cat([a * c - b * s, b * c + a * s], -1)
        n.backward(dy.double())
        assert _max_rel(y, n) < 1.5 * 2.0 ** -9
        assert _max_rel(x.grad, xr.grad) < 1.5 * 2.0 ** -9
        assert _max_rel(w.grad, wr.grad) < (2.0 ** -8 if wdtype == torch.bfloat16 else 1e-5)


# rows around the tiles of 4, 16, 32 and 48; columns off the 256-column tile; a reduction that is no multiple of the 64-deep stage
@pytest.mark.parametrize("R", [1, 4, 5, 16, 17, 32, 33, 48, 49, 100])
@pytest.mark.parametrize("K,N,Z", [(72, 264, 2), (2048, 256, 3), (256, 520, 1), (8, 8, 2)])
def test_few_row_gemm_tiles(R, K, N, Z):
    torch.manual_seed(3)
    store = torch.randn(Z * N * K + 1, device=DEV).bfloat16() / math.sqrt(K)
    for off in (0, 1):                          # off a 16-byte boundary: the weight is staged element by element
        ws = [store[off + z * N * K: off + (z + 1) * N * K].view(N, K) for z in range(Z)]
        a = torch.randn(Z, R, K, device=DEV)
        add = torch.randn(R, N // 2, device=DEV)
        got = F_ops.skinny_linears(a, ws, silu=True, add=add)
        want = torch.nn.functional.silu(a.double()) @ torch.stack(ws).double().transpose(1, 2)
        want[..., :N // 2] += add.double()
        assert _max_rel(got, want) < 1e-6       # fp32 products and sums: 2^-24 per term of a random walk, SiLU by the fast exponential
        dout = torch.randn(Z, R, N, device=DEV)
        da = F_ops._skinny_call(native.load(), Z, R, K, N, dout, R * N, N, 1, F_ops._ptr_table(ws), None, 0, 1, K, True, None, 0, Z, R, K, N,
                                False, False, False)
        assert _max_rel(da, dout.double() @ torch.stack(ws).double()) < 1e-6


# up to four rows: every number of warps to a weight row (K to 2048) and one element more than that kernel takes; columns around a warp's eight
# and a CTA's steps; weights off the 16-byte boundary; an added term for some of the columns
@pytest.mark.parametrize("R", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("K,N,Z", [(8, 1, 1), (256, 1543, 3), (264, 70, 2), (1032, 33, 2), (2048, 257, 84), (2056, 64, 1)])
def test_few_row_gemm_of_up_to_four_rows(R, K, N, Z):
    torch.manual_seed(7)
    assert native.load().skinny_rows(1, K, 1, True, False, False, Z, R, N, K) == (R <= 4 and K <= 2048)
    store = torch.randn(Z * N * K + 1, device=DEV).bfloat16() / math.sqrt(K)
    for off in (0, 1):
        ws = [store[off + z * N * K: off + (z + 1) * N * K].view(N, K) for z in range(Z)]
        add = torch.randn(R, max(N // 2, 1), device=DEV)
        for a in (torch.randn(Z, R, K, device=DEV), torch.randn(R, K, device=DEV)):
            for silu in (False, True):
                got = F_ops.skinny_linears(a, ws, silu=silu, add=add)
                x = torch.nn.functional.silu(a.double()) if silu else a.double()
                want = x @ torch.stack(ws).double().transpose(1, 2)
                want[..., :add.shape[1]] += add.double()
                if R > 4 or K > 2048:                  # the other kernels
                    assert _max_rel(got, want) < 1e-6
                    continue
                # Sums of terms of either sign: the bound is relative to the sum of their magnitudes. Roundings on the way of a term: 8 in
                # a lane, 5 over the warp, 7 over the warps, 1 for the added term, 2^-24 each. SiLU: the fast exponential is off by at
                # most 2 + 1.173 |a| = 7 units of 2^-23, the sum 1 + e by 2^-24, the fast division by 2 units of 2^-23: 19 x 2^-24.
                terms = x.abs() @ torch.stack(ws).double().abs().transpose(1, 2)
                terms[..., :add.shape[1]] += add.double().abs()
                assert a.abs().max() < 5.1 and ((got.double() - want).abs() <= (22 + 19 * silu) * 2.0 ** -24 * terms).all()


def test_few_row_gemm_takes_as_many_rows_as_its_widest_tile():
    """More rows than the 48-row tiles of the wide kernel can address go to the 64-row tile."""
    R, K, N = 48 * 65535 + 5, 8, 8
    torch.manual_seed(5)
    a, w = torch.randn(R, K, device=DEV), torch.randn(N, K, device=DEV).bfloat16()
    got = F_ops.skinny_linears(a, [w])
    want = a.double() @ w.double().t()
    assert _max_rel(got[0], want) < 1e-6
