"""The weight-only int8 linear of the text encoders (gpu_wo8_linear) against the reference's three-call flow: rotate the f32
rows (gpu_rotate_rows_f32, bit-identical to the reference's kernel), dequantize the weight (gpu_dequant_i8, likewise), fp32
product. The product here runs on the int8 tensor cores with the activation as fixed-point numbers in three 8-bit digits, so it is not
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


# Token tiles of 32 to 160, one and several, the last one ragged; columns around the 256 of a tile; tiles whose K boxes one, two or many
# clusters share (K = 256 is two boxes, 9728 seventy-six), and whole ones where the scratch has no room for that (N = 8).
@pytest.mark.parametrize("M,N,K", [(1, 8, 256), (20, 520, 9728), (32, 256, 1024), (33, 1000, 2560), (160, 257, 512), (161, 2560, 9728), (330, 255, 4096),
                                   (513, 5120, 768), (1024, 3584, 1280)])
def test_digits_keep_a_row_to_22_bits_of_its_maximum(pkg, dev, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    L = pkg.linear
    x = torch.randn(M, K, generator=g)
    x *= torch.exp2(torch.randint(-40, 40, (M, 1), generator=g).float())      # every row has a power of two of its own
    x[:, 5] *= 40.0
    x = x.to(dev)
    Wq, ws = L.convrot_requant((torch.randn(N, K, generator=g) * 0.03).to(dev), 0)
    xr, wf = L.rotate_rows_f32(x, PLAIN).double(), L.dequant_i8(Wq, ws).double()
    exact = xr @ wf.t()
    # a value is off by at most 2^-22 of the row's maximum (half a step of 2^-21 of the power of two below it); the three exact sums are
    # rounded once each when they become f32, then together, with the row's, the column's factor and, shared between clusters, once
    # more per cluster
    bound = xr.abs().amax(1, keepdim=True) * 2.0 ** -22 * wf.abs().sum(1) + exact.abs() * 2.0 ** -20 + xr.abs() @ wf.abs().t() * 2.0 ** -22
    out = torch.full((M + 1, N), 7.0, device=dev)
    L.wo8_linear(x, Wq, ws, PLAIN, out=out[:M])
    assert bool(((out[:M].double() - exact).abs() <= bound).all()) and bool((out[M] == 7.0).all())
    again = torch.empty(M, N, device=dev)
    L.wo8_linear(x, Wq, ws, PLAIN, out=again)
    assert torch.equal(again, out[:M])                             # whoever adds the shares up adds them in the same order
    base = torch.randn(M, N, generator=g).to(dev)
    acc = base.clone()
    L.wo8_linear(x, Wq, ws, PLAIN, out=acc, beta=1.0)
    assert torch.equal(acc, out[:M] + base)
    assert L.kernel_status() == 0


def test_rows_without_a_maximum(pkg, dev):
    """Rows holding an infinity or a NaN give NaN, zero rows zero, rows near either end of f32's range their values."""
    g = torch.Generator().manual_seed(3)
    L = pkg.linear
    N, K = 300, 512
    x = torch.randn(9, K, generator=g)
    x[1, 7], x[2, 300], x[3, 0] = float("inf"), float("nan"), -float("inf")
    x[4] = 0.0
    x[5] *= 2.0 ** 118
    x[6] *= 2.0 ** -95
    x[7] *= 2.0 ** -112
    x = x.to(dev)
    Wq, ws = L.convrot_requant((torch.randn(N, K, generator=g) * 0.03).to(dev), 0)
    out = L.wo8_linear(x, Wq, ws, PLAIN)
    exact = L.rotate_rows_f32(x, PLAIN).double() @ L.dequant_i8(Wq, ws).double().t()
    assert bool(out[1:4].isnan().all()) and bool((out[4] == 0).all())
    for m in (0, 5, 6, 7, 8):
        assert (out[m].double() - exact[m]).abs().max().item() <= 2e-6 * exact[m].abs().max().item(), m


def _keeps_what_a_group_holds(got, xr, wf, what):
    """Per output: a value is off by at most 2^-20 of the maximum of its rotation group (of 256); the sums of the groups are rounded to f32
    a few times each and added, one rounding per group. Where the products of 16 significant bits of each value would be closer, not
    further off than those either."""
    M, K = xr.shape
    err = (got.double() - xr @ wf.t()).abs()
    terms = xr.abs() @ wf.abs().t()
    groups = xr.abs().view(M, K // 256, 256).amax(2) @ wf.abs().view(-1, K // 256, 256).sum(2).t()
    bound = 2.0 ** -20 * groups + (K // 256 + 8) * 2.0 ** -24 * terms
    ok = err <= torch.minimum(bound, 2.0 ** -18 * terms)
    assert bool(ok.all()), (what, int((~ok).sum()), (err / terms).max().item() * 2.0 ** 18, (err / bound).max().item())


# Rows whose groups lie far apart (a massive activation beside ordinary ones), and weight rows that do not read the large group: what the small
# groups hold must not be lost beside it. Gaps around the line between one power of two per row and one per group (2 to 4 binary orders of
# magnitude), ordinary, and absurd ones; every row spread, every seventh, one row of a thousand; token tiles of every width, K boxes shared between
# clusters in the middle of a group, several tiles a cluster; rows of infinity, NaN and zeros and groups of zeros beside them.
@pytest.mark.parametrize("M,N,K,gap,every,limit,pro", [(1, 8, 512, 12, 1, 0, PLAIN), (20, 520, 9728, 8, 1, 0, PLAIN), (33, 1000, 2560, 20, 1, 0, PLAIN),
                                                       (64, 300, 512, 2, 1, 0, PLAIN), (64, 300, 512, 3, 1, 0, PLAIN), (64, 300, 512, 4, 1, 0, PLAIN),
                                                       (160, 257, 768, 16, 1, 0, PLAIN), (330, 255, 4096, 40, 7, 0, PLAIN), (1024, 3584, 1280, 10, 1024, 0, PLAIN),
                                                       (513, 5120, 768, 11, 5, 3, PLAIN), (96, 700, 2048, 140, 2, 0, PLAIN), (128, 512, 1536, 9, 3, 5, RMS),
                                                       (257, 1030, 2816, 13, 4, 0, SWIGLU)])
def test_small_groups_beside_large_ones(pkg, dev, M, N, K, gap, every, limit, pro):
    g = torch.Generator().manual_seed(M + N + K + gap)
    L = pkg.linear
    x = torch.randn(M, 2 * K if pro == SWIGLU else K, generator=g)
    far = torch.arange(M) % every == every // 2
    x[far, :256] *= 2.0 ** min(gap, 100)
    x[far, 256:K] *= 2.0 ** min(100 - gap, 0)
    odd = {}
    if M > 16:
        odd = {1: float("nan"), 4: float("inf"), 8: 0.0}
        for m, v in odd.items():
            x[m] = v if v == 0.0 else x[m].index_fill(0, torch.tensor([300]), v)
        x[far & (torch.arange(M) % 3 == 0), 256:512] = 0.0
    x = x.to(dev)
    kw = dict(K=K, up_offset=K if pro == SWIGLU else 0, norm_w=(torch.randn(K, generator=g) * 0.1 + 1.0).to(dev) if pro == RMS else None, eps=1e-6)
    Wq, ws = L.convrot_requant((torch.randn(N, K, generator=g) * 0.03).to(dev), 0)
    Wq[N // 2:, :256] = 0
    xr, wf = L.rotate_rows_f32(x, pro, **kw).double(), L.dequant_i8(Wq, ws).double()
    out = torch.full((M + 1, N), 7.0, device=dev)
    base = torch.randn(M, N, generator=g).to(dev)
    acc, again = base.clone(), torch.empty(M, N, device=dev)
    was = L.set_gemm_cluster_limit(limit)
    try:
        L.wo8_linear(x, Wq, ws, pro, out=out[:M], **kw)
        L.wo8_linear(x, Wq, ws, pro, out=again, **kw)
        L.wo8_linear(x, Wq, ws, pro, out=acc, beta=1.0, **kw)
    finally:
        L.set_gemm_cluster_limit(was)
    rows = [m for m in range(M) if m not in odd]
    _keeps_what_a_group_holds(out[rows], xr[rows], wf, f"{int(far.sum())} spread rows")
    for m, v in odd.items():
        assert bool((out[m] == 0).all() if v == 0.0 else out[m].isnan().all()), m
    assert bool((out[M] == 7.0).all()) and torch.equal(again[rows], out[rows]) and torch.equal(acc[rows], out[rows] + base[rows])
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


@pytest.mark.parametrize("pro,K", [(RMS, 512), (RMS, 2560), (SWIGLU, 512), (SWIGLU, 9728)])
def test_rows_without_a_maximum_behind_a_prologue(pkg, dev, pro, K):
    """The digits' second pass behind RMS and SWIGLU: a row with an infinity or a NaN becomes NaN, its ordinary neighbours in the same CTA keep their bits."""
    g = torch.Generator().manual_seed(K + pro)
    L = pkg.linear
    N, M = 264, 37
    x = torch.randn(M, 2 * K if pro == SWIGLU else K, generator=g)
    kw = dict(K=K, up_offset=K) if pro == SWIGLU else dict(norm_w=(torch.randn(K, generator=g) * 0.1 + 1.0).to(dev), eps=1e-6)
    odd = x.clone()
    odd[1, 7], odd[2, 300], odd[M - 1, K - 1] = float("inf"), float("nan"), float("inf")
    odd[5] = 0.0
    Wq, ws = L.convrot_requant((torch.randn(N, K, generator=g) * 0.03).to(dev), 0)
    plain, out = L.wo8_linear(x.to(dev), Wq, ws, pro, **kw), L.wo8_linear(odd.to(dev), Wq, ws, pro, **kw)
    keep = [m for m in range(M) if m not in (1, 2, 5, M - 1)]
    assert torch.equal(plain[keep], out[keep])
    assert bool(out[[1, 2, M - 1]].isnan().all()) and bool((out[5] == 0).all())
    assert L.kernel_status() == 0
