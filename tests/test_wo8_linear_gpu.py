"""The weight-only int8 linear of the text encoders (gpu_wo8_linear) against the reference's three-call flow: rotate the f32
rows (gpu_rotate_rows_f32, bit-identical to the reference's kernel), dequantize the weight (gpu_dequant_i8, likewise), fp32
product. The product here runs on the bf16 tensor cores with the activation split in two bf16 terms, so it is not
bit-identical to an fp32 GEMM (which has no canonical summation order either); the tolerance is stated against the exact
(fp64) product of the same rotated rows and dequantized weights: 1e-5 of the largest output magnitude, and no worse than
three times the error of an fp32 GEMM of the same operands."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
PLAIN, RMS, SWIGLU = 0, 1, 3


@pytest.mark.parametrize("M,N,K,pro", [(77, 1024, 1024, PLAIN), (300, 2560, 2560, RMS), (512, 1536, 4096, SWIGLU), (1, 768, 256, PLAIN)])
def test_against_the_fp32_flow(pkg, dev, M, N, K, pro):
    g = torch.Generator().manual_seed(M + N + K)
    L = pkg.linear
    width = 2 * K if pro == SWIGLU else K
    x = (torch.randn(M, width, generator=g) * 1.5).to(dev)
    x[:, 3] *= 30.0                                                # an outlier channel, as text-encoder states have
    norm_w = (torch.randn(K, generator=g) * 0.1 + 1.0).to(dev) if pro == RMS else None
    w = torch.randn(N, K, generator=g) * 0.03
    Wq, ws = L.convrot_requant(w.to(dev), 0)                       # int8 ConvRot weight + per-channel scale
    kw = dict(K=K, up_offset=K if pro == SWIGLU else 0, norm_w=norm_w, eps=1e-6)
    xr = L.rotate_rows_f32(x, pro, **kw)
    wf = L.dequant_i8(Wq, ws)
    exact = xr.double() @ wf.double().t()
    fp32 = (xr @ wf.t()).double()                                  # what the reference's flow computes (cuBLAS fp32)
    got = L.wo8_linear(x, Wq, ws, pro, **kw)
    scale = exact.abs().max().item()
    err, err32 = (got.double() - exact).abs().max().item(), (fp32 - exact).abs().max().item()
    assert err <= 1e-5 * scale, (err, scale)
    assert err <= max(3 * err32, 2e-6 * scale), (err, err32)
    # beta = 1 accumulates into the residual stream, as the attention-out and MLP-down linears do
    base = torch.randn(M, N, generator=g).to(dev)
    acc = base.clone()
    L.wo8_linear(x, Wq, ws, pro, out=acc, beta=1.0, **kw)
    assert (acc.double() - (base.double() + exact)).abs().max().item() <= 1e-5 * max(scale, base.abs().max().item())
    assert L.kernel_status() == 0


# The forms of the kernel under it: tiles of more than 128 columns have one accumulator pair (512 x 19456: 192 columns, 204 tiles for
# at most 74 clusters), narrower ones two; a cluster's second and third tile toggles their phases; ragged rows and columns, columns
# whose rows of output TMA cannot address (N % 4). `limit` keeps the GEMM to a few clusters, so that each has several tiles.
@pytest.mark.parametrize("M,N,K,limit", [(512, 19456, 256, 0), (512, 19456, 256, 5), (700, 2560, 512, 3), (300, 1030, 768, 2), (513, 770, 256, 1),
                                         (257, 1023, 1024, 3)])
def test_several_tiles_a_cluster_and_ragged_ones(pkg, dev, M, N, K, limit):
    g = torch.Generator().manual_seed(M + N + K)
    L = pkg.linear
    x = (torch.randn(M, K, generator=g) * 1.5).to(dev)
    Wq, ws = L.convrot_requant((torch.randn(N, K, generator=g) * 0.03).to(dev), 0)
    xr, wf = L.rotate_rows_f32(x, PLAIN), L.dequant_i8(Wq, ws)
    exact = xr.double() @ wf.double().t()
    scale = exact.abs().max().item()
    # Per output: hi + lo (each rounded to 8 bits) leaves at most 2^-18 of every term; adding K terms in f32 at most K 2^-24 of their
    # absolute sum. (Not "three times an fp32 product's error": a short sum in fp32 loses less than the 2^-18.)
    bound = (2.0 ** -18 + K * 2.0 ** -24) * (xr.double().abs() @ wf.double().abs().t())
    base = torch.randn(M, N, generator=g).to(dev)
    out = torch.full((M + 1, N), 7.0, device=dev)                  # a row more, which nothing writes
    acc = base.clone()
    was = L.set_gemm_cluster_limit(limit)
    try:
        L.wo8_linear(x, Wq, ws, PLAIN, out=out[:M])
        L.wo8_linear(x, Wq, ws, PLAIN, out=acc, beta=1.0)
    finally:
        L.set_gemm_cluster_limit(was)
    err = (out[:M].double() - exact).abs()
    assert err.max().item() <= 1e-5 * scale and bool((err <= bound).all()), (err.max().item(), scale, (err / bound).max().item())
    assert bool((out[M] == 7.0).all())
    assert (acc.double() - (base.double() + exact)).abs().max().item() <= 1e-5 * max(scale, base.abs().max().item())
    assert L.kernel_status() == 0


def test_argument_checks(pkg, dev):
    L = pkg.linear
    x = torch.zeros(4, 300, device=dev)
    Wq = torch.zeros(8, 300, dtype=torch.int8, device=dev)
    ws = torch.ones(8, device=dev)
    with pytest.raises(pkg.GpuKernelError, match="-1"):
        L.wo8_linear(x, Wq, ws)                                     # K % 256 != 0
    x = torch.zeros(4, 256, device=dev)
    Wq = torch.zeros(8, 256, dtype=torch.int8, device=dev)
    with pytest.raises(pkg.GpuKernelError, match="-207"):
        L.wo8_linear(x, Wq, ws, beta=0.5)
    with pytest.raises(pkg.GpuKernelError, match="-3"):
        L.wo8_linear(x, Wq, ws, 11)                                 # a prologue gpu_rotate_rows_f32 does not take
