"""Branches of the network kernels that are chosen by size: split reductions
of the GEMM and the column sum, and the 16-byte forms of the transpose, the
causal im2col pair and the ReLU, against float64 or exact references."""
import numpy as np
import pytest
import torch

from openems_b200 import _native as N

pytestmark = pytest.mark.gpu


def p(t):
    return t.data_ptr()


def rnd(*shape, seed=0, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


# K-blocks: 31 (no split), 32, one part shorter than the others, a K tail;
# edges of M and N inside a tile
@pytest.mark.parametrize("M,n,K", [(128, 64, 1984), (128, 64, 2048), (100, 40, 2056), (128, 640, 8200), (8, 256, 16384),
                                   (130, 200, 4104)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_gemm_split_k(M, n, K, beta):
    a, b = rnd(M, K, dtype=torch.bfloat16), rnd(n, K, seed=1, dtype=torch.bfloat16)
    c, bias = rnd(M, n + 3, seed=2), rnd(n, seed=3)
    want = a.double() @ b.double().T + beta * c[:, :n].double() + bias.double()
    N.check(N.lib().oems_tc_gemm_bf16(p(a), K, p(b), K, p(c), n + 3, M, n, K, beta, p(bias), None))
    N.check(N.lib().oems_tc_check(None))
    # an MMA adds 16 products at a time to an f32 sum that may be truncated:
    # K / 16 roundings of at most 2^-23 of a running sum below 5 K^1/2 (sums
    # of K products of variance 1), and the final additions
    assert (c[:, :n].double() - want).abs().max().item() <= (K / 16 + 4) * 2.0 ** -23 * 5 * K ** 0.5


@pytest.mark.parametrize("R,C,ldx,ldy", [(64, 64, 64, 64), (72, 200, 208, 72), (8, 8, 8, 16), (33, 40, 40, 40),
                                         (256, 1000, 1000, 256)])
def test_transpose(R, C, ldx, ldy):
    x = rnd(R, ldx, dtype=torch.bfloat16)
    y = torch.zeros(C, ldy, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().oems_pk_transpose_bf16(p(x), ldx, p(y), ldy, R, C, None))
    assert torch.equal(y[:, :R], x[:, :C].T) and not y[:, R:].any()


@pytest.mark.parametrize("B,T", [(3, 37), (5, 9001)])  # the latter past the line of the 4-channel gather
@pytest.mark.parametrize("C,pad", [(8, 0), (16, 8), (12, 4), (4, 3)])
def test_causal_columns(C, pad, B, T):
    from oracle.tailnet_ref import col2im_causal, im2col_causal, round_bf16
    ks, dil = 5, 4
    ldc = ks * C + pad
    x = rnd(B, T, C)
    cols = torch.zeros(B * T, ldc, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().oems_pk_im2col_causal(p(x), p(cols), B, T, C, ks, dil, ldc, None))
    want = round_bf16(im2col_causal(x.cpu().numpy().astype(np.float64), ks, dil))
    assert np.array_equal(cols[:, :ks * C].double().cpu().numpy(), want)
    d = rnd(B * T, ldc, seed=1)
    dx = torch.empty(B, T, C, device="cuda")
    N.check(N.lib().oems_pk_col2im_causal(p(d), ldc, p(dx), B, T, C, ks, dil, None))
    ref = col2im_causal(np.ascontiguousarray(d[:, :ks * C].double().cpu().numpy()), B, T, C, ks, dil)
    assert np.allclose(dx.cpu().numpy(), ref, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("rows,w", [(4095, 33), (4096, 33), (5000, 128), (70001, 8), (12265, 128), (12266, 128), (4096, 640),
                                    (24576, 3), (13001, 35)])
def test_column_sums_and_relu(rows, w):
    x = rnd(rows, w)
    db = torch.empty(w, device="cuda")
    N.check(N.lib().oems_pk_colsum(p(x), rows, w, p(db), None))
    assert torch.allclose(db.double(), x.double().sum(0), rtol=0, atol=rows ** 0.5 * 16 * 2.0 ** -24 * rows ** 0.5)
    y, yb = x.clone(), torch.empty(rows, w, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().oems_pk_relu(p(y), p(yb), rows, w, w, None))
    assert torch.equal(y, x.clamp(min=0)) and torch.equal(yb, y.to(torch.bfloat16))
