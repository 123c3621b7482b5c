"""Kernels that start before their predecessor ends (programmatic dependent launch) against the same calls launched the ordinary
way, bit for bit: whole blocks whose buffers are written again and again, eagerly and as graphs, chains of small linears between
two buffers, two streams with events between them, ordinary kernels in between. A GEMM cluster limit of at least the device's
pairs selects ordinary launches and restricts nothing."""
from __future__ import annotations

import pytest
import torch

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu
RMS, SWIGLU, SILU, LN_MOD = 1, 3, 5, 9


class _Ordinary:
    def __init__(self, L):
        self.L = L

    def __enter__(self):
        self.was = self.L.set_gemm_cluster_limit(1 << 20)

    def __exit__(self, *_):
        self.L.set_gemm_cluster_limit(self.was)


def _unet(L, dev, g):
    """GroupNorm, LayerNorm and GEGLU quantizers with their GEMMs, the residual stream updated in place three times."""
    P, C = 144, 320
    M, h = 2 * P, torch.float16
    rn = lambda *s: torch.randn(*s, generator=g).to(dev)
    lin = lambda n, k: (*L.sd_quant_rows((rn(n, k) * 0.05).half(), 64), (rn(n) * 0.1).half())
    x, one = torch.empty(2, P, C, dtype=h, device=dev), torch.ones(C, dtype=h, device=dev)
    w, b = rn(C) * 0.1 + 1, rn(C) * 0.1
    w_in, w_qkv, w_up, w_down, w_out = lin(C, C), lin(3 * C, C), lin(8 * C, C), lin(C, 4 * C), lin(C, C)
    t, qkv, up, y = (torch.empty(M, n, dtype=h, device=dev) for n in (C, 3 * C, 8 * C, C))

    def run():
        def linear(a, wt, **kw):
            return L.int8_gemm(a[0], wt[0], a[1], wt[1], wt[2], **kw)
        linear(L.sd_group_norm_quant_rows(x, w, b, 32, 1e-6, 64), w_in, out=t)
        linear(L.sd_ln_quant_rows(t, w, b, 1e-5, 64), w_qkv, out=qkv)
        linear(L.sd_quant_rows(qkv[:, :C], 64), w_out, rscale=one, resid=t, out=t)
        linear(L.sd_ln_quant_rows(t, w, b, 1e-5, 64), w_up, out=up)
        linear(L.sd_geglu_quant_rows(up, 64), w_down, rscale=one, resid=t, out=t)
        linear(L.sd_quant_rows(t, 64), w_out, rscale=one, resid=x.view(M, C), out=y)
    return [x], run, [t, qkv, up, y]


def _text(L, dev, g):
    """The MLP of a text encoder layer: the two terms and the widened weight share caller scratch between the two linears."""
    M, H, F = 77, 512, 1280
    rn = lambda *s: torch.randn(*s, generator=g).to(dev)
    x, stream, gu, norm = rn(M, H), rn(M, H), torch.empty(M, 2 * F, device=dev), rn(H) * 0.1 + 1
    (w1, s1), (w2, s2) = L.convrot_requant(rn(2 * F, H) * 0.05, 0), L.convrot_requant(rn(H, F) * 0.05, 0)
    scratch = tuple(torch.empty(4 * F * max(M, H), dtype=torch.uint8, device=dev) for _ in range(2))

    def run():
        stream.copy_(x)
        L.wo8_linear(stream, w1, s1, RMS, norm_w=norm, eps=1e-6, out=gu, scratch=scratch)
        L.wo8_linear(gu, w2, s2, SWIGLU, K=F, up_offset=F, out=stream, beta=1.0, scratch=scratch)
    return [x], run, [gu, stream]


def _w6(L, dev, g, M):
    """A W6A8 block from packed weights: the few-rows kernel with its clusters, one quantizer buffer for four linears."""
    H, F = 512, 1536
    rn = lambda *s: torch.randn(*s, generator=g).to(dev)
    lin = lambda n, k: (*L.w6_requant((rn(n, k) * 0.05).bfloat16(), 1), (rn(n) * 0.1).bfloat16())
    bf = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device=dev)
    x, one = bf(M, H), torch.ones(H, dtype=torch.bfloat16, device=dev)
    w_qkv, w_out, w_up, w_down = lin(3 * H, H), lin(H, H), lin(F, H), lin(H, F)
    qkv, x1, up, x2 = bf(M, 3 * H), bf(M, H), bf(M, F), bf(M, H)
    codes, scales = torch.empty(M * F, dtype=torch.int8, device=dev), torch.empty(M, device=dev)

    def run():
        def linear(src, k, w, pro=0, **kw):
            L.quant_rows(src, pro, 1, K=k, eps=1e-6, q=codes[:M * k].view(M, k), scales=scales)
            return L.w6a8_gemm(codes[:M * k].view(M, k), w[0], w[1], scales, w[2], w[3], **kw)
        linear(x, H, w_qkv, RMS, out=qkv)
        linear(qkv, H, w_out, rscale=one, resid=x, out=x1)
        linear(x1, H, w_up, RMS, act=1, out=up)
        linear(up, F, w_down, rscale=one, resid=x1, out=x2)
    return [x], run, [qkv, x1, up, x2]


def _dit(L, dev, g, M):
    """adaLN from one row (the weight-streaming kernel), the rotating epilogue, the in-place residual."""
    H, F = 512, 2048
    rn = lambda *s: torch.randn(*s, generator=g).to(dev)
    lin = lambda n, k: (*L.convrot_requant(rn(n, k) * 0.05, 0), (rn(n) * 0.1).bfloat16())
    bf = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device=dev)
    x, cond = bf(M, H), bf(1, H)
    w_ada, w_out, w_up, w_down = lin(3 * H, H), lin(H, H), lin(F, H), lin(H, F)
    mod, r, h = bf(1, 3 * H), bf(M, H), bf(M, F)
    parts, a, xs, af = torch.empty(F // 64, M, device=dev), torch.empty(M, H, dtype=torch.int8, device=dev), torch.empty(M, device=dev), \
        torch.empty(M, F, dtype=torch.int8, device=dev)

    def run():
        q1, s1 = L.quant_rows(cond, SILU, 1)
        L.int8_gemm(q1, w_ada[0], s1, w_ada[1], w_ada[2], out=mod)
        shift, scale, gate = mod.view(3, H).unbind(0)
        L.quant_rows(x, LN_MOD, 1, eps=1e-6, mod_scale=scale, mod_shift=shift, q=a, scales=xs)
        L.int8_gemm(a, w_out[0], xs, w_out[1], w_out[2], rscale=gate, resid=x, out=r)
        L.quant_rows(r, LN_MOD, 1, eps=1e-6, mod_scale=scale, mod_shift=shift, q=a, scales=xs)
        L.int8_gemm_act_rot(a, w_up[0], xs, w_up[1], w_up[2], act=1, out=h, amax_part=parts)
        L.quant_rows_rotated(h, parts, q=af, scales=xs)
        L.int8_gemm(af, w_down[0], xs, w_down[1], w_down[2], rscale=gate, resid=r, out=r)
    return [x, cond], run, [mod, h, r]


BLOCKS = {"unet": _unet, "text": _text, "w6_m17": lambda *a: _w6(*a, 17), "w6_m300": lambda *a: _w6(*a, 300), "dit_m5": lambda *a: _dit(*a, 5),
          "dit_m700": lambda *a: _dit(*a, 700)}


@pytest.mark.parametrize("block", list(BLOCKS))
def test_blocks_equal_their_ordinary_launches(pkg, dev, block):
    L = pkg.linear
    g = torch.Generator().manual_seed(len(block))
    inputs, run, outputs = BLOCKS[block](L, dev, g)
    values = [[torch.randn(t.shape, generator=g).to(t.dtype).to(dev) for t in inputs] for _ in range(2)]

    def load(i):
        for t, v in zip(inputs, values[i]):
            t.copy_(v)

    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = []
        with _Ordinary(L):
            for i in range(2):
                load(i)
                run()
                want.append([t.clone() for t in outputs])
        got = []
        for i in (0, 1, 1, 0, 1, 0):                 # no wait in between: a pass overwrites what the one before it reads
            load(i)
            run()
            got.append((i, [t.clone() for t in outputs]))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            run()
        for i in (1, 0, 0, 1):
            load(i)
            graph.replay()
            graph.replay()
            got.append((i, [t.clone() for t in outputs]))
    side.synchronize()
    for n, (i, outs) in enumerate(got):
        for k, (a, b) in enumerate(zip(outs, want[i])):
            assert_bits_equal(a, b, f"{block}, pass {n}, output {k}")
    assert L.kernel_status() == 0


@pytest.mark.parametrize("M", [1, 5, 77, 333, 1024])
@pytest.mark.parametrize("between", ["nothing", "torch", "streams"])
def test_chains_between_two_buffers(pkg, dev, M, between):
    """Twelve linears from one buffer into the other and back, one pair of quantizer buffers: every kernel reads what the one before
    it wrote and writes what the one two before it read. With an ordinary kernel, or a change of stream, between them."""
    L = pkg.linear
    g = torch.Generator().manual_seed(M)
    K = 768
    w, ws = L.convrot_requant((torch.randn(K, K, generator=g) * 0.06).to(dev), 0)
    x0 = torch.randn(M, K, generator=g).bfloat16().to(dev)
    bufs = [torch.empty(M, K, dtype=torch.bfloat16, device=dev) for _ in range(2)]
    q, s = torch.empty(M, K, dtype=torch.int8, device=dev), torch.empty(M, device=dev)
    streams = [torch.cuda.Stream(dev) for _ in range(2 if between == "streams" else 1)]
    for st in streams:
        st.wait_stream(torch.cuda.current_stream())

    def chain():
        last = None
        for n in range(12):
            st = streams[n % len(streams)]
            with torch.cuda.stream(st):
                if last is not None and len(streams) > 1:
                    st.wait_event(last)
                if n == 0:
                    bufs[0].copy_(x0)
                L.quant_rows(bufs[n % 2], 0, 1, q=q, scales=s)
                L.int8_gemm(q, w, s, ws, None, out=bufs[1 - n % 2])
                if between == "torch":
                    bufs[1 - n % 2].mul_(1.25)
                if len(streams) > 1:
                    last = st.record_event()
        torch.cuda.synchronize()
        return bufs[0].clone()

    with _Ordinary(L):
        want = chain()
    for n in range(3):
        assert_bits_equal(chain(), want, f"chain {n}")
    assert bool(want.float().abs().max() > 0) and L.kernel_status() == 0
