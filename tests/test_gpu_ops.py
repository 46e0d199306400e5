"""Bandwidth-bound kernels and attention against fp32 PyTorch references of the same ops."""
import ctypes as C
import math

import pytest
import torch

from sneppx_alg_b200 import ops
from sneppx_alg_b200.ops import _lib, functional as F_
from sneppx_alg_b200.ops._lib import c_int, c_ll, ptr, stream
from sneppx_alg_b200.optim.fused import adamw_flat_, adamw_reference, grad_norm_

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("per_head", [False, True])
def test_block_sparse_attention_tile_mask(causal, per_head):
    """Tile-level mask in the forward kernel: random masks (some query tiles with no visible tile at all, some steps
    masked for one of the two query tiles of a CTA only), shared or per head, ragged sequence ends."""
    from sneppx_alg_b200.ops.functional import block_sparse_attention, block_sparse_attention_reference
    torch.manual_seed(3)
    B, Sq, Skv, Hq, Hk, D = 2, 1000, 1000, 8, 2, 128
    q = torch.randn(B, Sq, Hq, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, Skv, Hk, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, Skv, Hk, D, device="cuda", dtype=torch.bfloat16)
    nq, nk = (Sq + 127) // 128, (Skv + 127) // 128
    bm = torch.rand(B if per_head else 1, Hq if per_head else 1, nq, nk, device="cuda") < 0.45
    bm[..., 3, :] = False          # a query tile that sees nothing
    bm[..., 0, 0] = True
    out = block_sparse_attention(q, k, v, bm if per_head else bm[0, 0], causal=causal)
    ops.check_status()
    ref = block_sparse_attention_reference(q.float(), k.float(), v.float(), bm, causal=causal)
    assert torch.isfinite(out.float()).all()
    assert _rel(out, ref) < 2e-2
    # an all-true mask is plain attention
    full = torch.ones(nq, nk, dtype=torch.bool, device="cuda")
    assert _rel(block_sparse_attention(q, k, v, full, causal=causal), ops.attention(q, k, v, causal=causal)) < 1e-3


def _rel(a, b):
    return (a.float() - b.float()).abs().max().item() / (b.float().abs().max().item() + 1e-6)


@pytest.mark.parametrize("T,d", [(64, 256), (333, 4096), (17, 1032)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(T, d, with_res):
    torch.manual_seed(0)
    x = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True) if with_res else None
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    y, h = F_.rmsnorm(x, w, 1e-5, r)
    gy, gh = torch.randn_like(y), torch.randn_like(y)
    (y * gy).sum().backward() if not with_res else ((y * gy).sum() + (h * gh).sum()).backward()
    xr = x.detach().float().requires_grad_(True)
    rr = r.detach().float().requires_grad_(True) if with_res else None
    wr = w.detach().float().requires_grad_(True)
    hr = xr + rr if with_res else xr
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    ((yr * gy.float()).sum() + ((hr * gh.float()).sum() if with_res else 0)).backward()
    assert _rel(y, yr) < 2e-2
    assert _rel(x.grad, xr.grad) < 3e-2
    assert _rel(w.grad, wr.grad) < 3e-2
    if with_res:
        assert _rel(r.grad, rr.grad) < 3e-2


def test_rope_fwd_bwd():
    torch.manual_seed(0)
    B, S, H, Hk, D = 2, 96, 4, 2, 128
    qkv = torch.randn(B, S, (H + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16)
    cos, sin = F_.rope_tables(S, D, 5e5, "cuda")
    ref = F_.rope_reference(qkv[..., : (H + Hk) * D].reshape(B, S, H + Hk, D), cos, sin).reshape(B, S, -1)
    x = qkv.clone().requires_grad_(True)
    out = F_.rope_qk_(x * 1.0, cos, sin, H + Hk, D)
    assert _rel(out[..., : (H + Hk) * D], ref) < 1e-2
    assert torch.equal(out[..., (H + Hk) * D:], qkv[..., (H + Hk) * D:])
    g = torch.randn_like(out)
    out.backward(g)
    # rotation is orthogonal: the backward of g is the inverse rotation
    gref = F_.rope_reference(g[..., : (H + Hk) * D].reshape(B, S, H + Hk, D), cos, -sin).reshape(B, S, -1)
    assert _rel(x.grad[..., : (H + Hk) * D], gref) < 1e-2


@pytest.mark.parametrize("act", ["silu", "gelu", "relu"])
def test_glu(act):
    torch.manual_seed(0)
    gu = torch.randn(100, 2 * 264, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    h = F_.glu(gu, act)
    g = torch.randn_like(h)
    h.backward(g)
    gr = gu.detach().float().requires_grad_(True)
    hr = F_.glu_reference(gr, act)
    hr.backward(g.float())
    assert _rel(h, hr) < 1e-2 and _rel(gu.grad, gr.grad) < 2e-2


@pytest.mark.parametrize("V", [1000, 32000])
def test_cross_entropy(V):
    torch.manual_seed(0)
    T = 77
    logits = (3 * torch.randn(T, V, device="cuda")).to(torch.bfloat16)
    tgt = torch.randint(0, V, (T,), device="cuda")
    tgt[5] = -100
    lr = logits.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lr, tgt, ignore_index=-100)
    ref.backward()
    lg = logits.clone().requires_grad_(True)
    loss = F_.cross_entropy(lg * 1.0, tgt)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * max(1, abs(ref.item()))
    assert (lg.grad.float() - lr.grad).abs().max().item() < 2e-4


def test_linear_cross_entropy():
    torch.manual_seed(0)
    T, d, V = 300, 256, 1024
    h = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (0.05 * torch.randn(V, d, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    tgt = torch.randint(0, V, (T,), device="cuda")
    loss = F_.linear_cross_entropy(h, w, tgt, chunk=128)
    loss.backward()
    hr, wr = h.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(hr @ wr.t(), tgt)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 5e-3
    assert _rel(h.grad, hr.grad) < 3e-2 and _rel(w.grad, wr.grad) < 3e-2


def test_adamw_flat_and_norm():
    torch.manual_seed(0)
    n = 100003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda").to(torch.bfloat16)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    pr, mr, vr = p.clone(), m.clone(), v.clone()
    p16 = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    out, flag = grad_norm_([g], max_norm=1.0)
    nrm = g.float().norm().item()
    assert abs(out[1].item() - nrm) < 1e-3 * nrm and flag.item() == 0
    coef = 1.0 / (nrm + 1e-6)
    for step in (1, 2):
        adamw_flat_(p, m, v, g, p16, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 1.0, out[2:3])
        adamw_reference(pr, mr, vr, g, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, coef)
    assert (p - pr).abs().max().item() < 1e-5
    assert torch.equal(p16, p.to(torch.bfloat16))


@pytest.mark.parametrize("B,S,H,Hk,D,causal,window", [
    (1, 128, 2, 2, 128, True, 0), (2, 384, 4, 2, 128, True, 0), (1, 200, 2, 1, 128, True, 0),
    (1, 256, 2, 2, 128, False, 0), (1, 512, 2, 2, 128, True, 128), (1, 256, 2, 2, 64, True, 0)])
def test_attention_forward(B, S, H, Hk, D, causal, window):
    torch.manual_seed(0)
    q = torch.randn(B, S, H, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, S, Hk, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, S, Hk, D, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        o = F_.attention(q, k, v, causal=causal, window=window)
    ops.check_status()
    ref = F_.attention_reference(q.float(), k.float(), v.float(), causal, window)
    assert _rel(o, ref) < 2e-2


@pytest.mark.parametrize("B,S,H,Hk,causal,window", [(1, 128, 2, 2, True, 0), (2, 320, 4, 2, True, 0),
                                                    (1, 256, 2, 1, False, 0), (1, 384, 2, 2, True, 128)])
def test_attention_backward(B, S, H, Hk, causal, window):
    torch.manual_seed(0)
    D = 128
    qkv = torch.randn(B, S, (H + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    q = qkv[..., : H * D].view(B, S, H, D)
    k = qkv[..., H * D: (H + Hk) * D].view(B, S, Hk, D)
    v = qkv[..., (H + Hk) * D:].view(B, S, Hk, D)
    o = F_.attention(q, k, v, causal=causal, window=window)
    g = torch.randn_like(o)
    o.backward(g)
    ops.check_status()
    r = qkv.detach().float().requires_grad_(True)
    qr = r[..., : H * D].view(B, S, H, D)
    kr = r[..., H * D: (H + Hk) * D].view(B, S, Hk, D)
    vr = r[..., (H + Hk) * D:].view(B, S, Hk, D)
    F_.attention_reference(qr, kr, vr, causal, window).backward(g.float())
    assert _rel(o, F_.attention_reference(qr, kr, vr, causal, window)) < 2e-2
    for name, sl in (("dq", slice(0, H * D)), ("dk", slice(H * D, (H + Hk) * D)), ("dv", slice((H + Hk) * D, None))):
        assert _rel(qkv.grad[..., sl], r.grad[..., sl]) < 3e-2, name


def test_differential_attention():
    torch.manual_seed(0)
    B, S, H, D = 1, 256, 2, 128
    q = torch.randn(B, S, 2 * H, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, S, 2 * H, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, S, H, D, device="cuda", dtype=torch.bfloat16)
    lam = torch.tensor([0.3, 0.6], device="cuda")
    with torch.no_grad():
        o = F_.differential_attention(q, k, v, lam)
    a = F_.attention_reference(q.float(), k.float(), v.float(), True).view(B, S, H, 2, D)
    ref = a[..., 0, :] - lam.view(1, 1, -1, 1) * a[..., 1, :]
    assert _rel(o, ref) < 3e-2


@pytest.mark.parametrize("B,S,H,Hk,window,pos", [(2, 77, 4, 2, 0, False), (1, 256, 8, 8, 0, True), (3, 130, 7, 1, 40, True), (1, 1, 4, 4, 0, False)])
def test_rope_attention_is_rope_then_attention(B, S, H, Hk, window, pos):
    """One node for rotation and attention against the two of them: the same kernels on the same operands, so outputs agree exactly and
    gradients up to the order of the dQ additions and one more bf16 rounding (dQ and dK are rounded, then turned back: 2^-8 of a value)."""
    torch.manual_seed(S)
    D = 128
    x = torch.randn(B, S, (H + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16)
    cos, sin = F_.rope_tables(512, D, 5e5, "cuda")
    positions = torch.randint(0, 512, (B, S), device="cuda") if pos else None
    a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    o = F_.rope_attention(a, cos, sin, H, Hk, D, positions, window)
    q, k, v = F_._split_heads(F_.rope_qk_(b, cos, sin, H + Hk, D, positions), H, Hk, D)
    ref = F_.attention(q, k, v, causal=True, window=window)
    assert o.shape == (B, S, H, D) and torch.equal(o, ref) and torch.equal(a, x)
    g = torch.randn_like(o)
    o.backward(g)
    ref.backward(g)
    assert _rel(a.grad, b.grad) < 2.0 ** -7


@pytest.mark.parametrize("heads,rot,D,interleaved,strided", [(6, 4, 128, False, False), (5, 5, 16, False, True), (3, 2, 24, False, False), (4, 2, 64, True, False)])
def test_rope_to_new_buffer(heads, rot, D, interleaved, strided):
    """Rotation into a new buffer and back: 16-byte kernel, a column slice of a wider tensor, and the sizes and layout that go through a copy.
    Products and sums are 32-bit, so one bf16 rounding each way is left."""
    torch.manual_seed(D)
    B, S = 2, 33
    wide = torch.randn(B, S, heads * D + 64, device="cuda", dtype=torch.bfloat16)
    x = wide[..., :heads * D] if strided else wide[..., :heads * D].contiguous()
    cos, sin = F_.rope_tables(S, D, 1e4, "cuda")
    before = wide.clone()
    y = F_.rope_qk_(x, cos, sin, rot, D, None, interleaved)
    ref = F_.rope_reference(x[..., :rot * D].reshape(B, S, rot, D).float(), cos, sin, None, interleaved).reshape(B, S, -1)
    assert torch.equal(wide, before) and torch.equal(y[..., rot * D:], x[..., rot * D:])
    assert bool(((y[..., :rot * D].float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all())


@pytest.mark.parametrize("T,d", [(1, 8), (3, 1024), (700, 1032), (2, 2048), (300, 2056), (5, 8192), (3, 8200), (2, 16384), (300, 8200), (700, 16384)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_row_sizes(T, d, with_res):
    """Edges of the register forms (one and two vectors a thread, two passes beyond), fewer and more rows than backward CTAs, and weight
    gradients from one to many partial rows. Inputs are bf16, everything else 32-bit: one rounding of each output, 2^-8 of its value plus
    2^-8 of the residual sum that is rounded first; the weight gradient sums T products."""
    torch.manual_seed(d)
    x, r, g, gh = (torch.randn(T, d, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16)
    ins = [t.clone().requires_grad_(True) for t in ((x, w, r) if with_res else (x, w))]
    y, h = F_.rmsnorm(ins[0], ins[1], 1e-5, ins[2] if with_res else None)
    (((y * g).sum() + (h * gh).sum()) if with_res else (y * g).sum()).backward()
    ref = [t.double().requires_grad_(True) for t in ((x, w, r) if with_res else (x, w))]
    hr = (ref[0] + ref[2]) if with_res else ref[0]
    hb = hr + (hr.detach().bfloat16().double() - hr.detach())          # the sum as it is stored
    yr = hb * torch.rsqrt(hb.pow(2).mean(-1, keepdim=True) + 1e-5) * ref[1]
    (((yr * g.double()).sum() + (hb * gh.double()).sum()) if with_res else (yr * g.double()).sum()).backward()
    close = lambda a, b, extra=0.0: bool(((a.double() - b).abs() <= b.abs() * 2.0 ** -8 + extra).all())  # noqa: E731
    assert close(y, yr.detach(), 1e-5)
    top = ref[0].grad.abs().max().item()
    assert close(ins[0].grad, ref[0].grad, 1e-4 * top)
    assert close(ins[1].grad, ref[1].grad, 1e-4 * ref[1].grad.abs().max().item())


def _copy_us(nbytes):
    """Time of a plain copy that reads and writes ``nbytes`` in all, buffers larger than L2."""
    a = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    b = torch.empty_like(a)
    return _median_us(lambda: b.copy_(a)) * nbytes / (2 * a.numel())


def _median_us(fn, n=11):
    for _ in range(3):
        fn()
    ts = []
    for _ in range(n):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(400000)          # the launches are queued before the first starts
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b) * 1e3)
    return sorted(ts)[n // 2]


@pytest.mark.parametrize("T,d", [(16, 4096), (128, 4096), (300, 16384), (600, 16384), (1000, 768)])
def test_norms_in_a_row_gain_by_starting_early(T, d):
    """Norms that are set up while their predecessors run are not slower for it: sixteen in a row take no longer than with an ordinarily launched kernel
    between each two, which they would wait for. With every norm signalling at once 16 of [300, 16384] took 212 us, 160 so."""
    x, w = torch.randn(T, d, device="cuda").bfloat16(), torch.ones(d, device="cuda").bfloat16()
    y, one = torch.empty_like(x), torch.zeros(1, device="cuda")

    def norms(spaced):
        for _ in range(8):
            for a, b in ((x, y), (y, x)):
                _lib.call("sx_rmsnorm_fwd", _lib.ptr(a), _lib.ptr(None), _lib.ptr(w), _lib.ptr(b), _lib.ptr(None), _lib.ptr(None), _lib.c_ll(T), _lib.c_int(d),
                          _lib.c_float(1e-5), stream())
                if spaced:
                    one.zero_()

    us = []
    for spaced in (False, True):
        norms(spaced)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            norms(spaced)
        us.append(_median_us(graph.replay))
    assert us[0] <= us[1] * 1.05, us


@pytest.mark.parametrize("T,heads,rot,D", [(1, 1, 1, 16), (131, 1, 1, 16), (300, 3, 2, 48), (64, 15, 15, 128), (147, 16, 10, 128), (148, 16, 10, 128),
                                           (5, 96, 80, 256), (200, 97, 90, 256)])
def test_rope_launch_shapes(T, heads, rot, D):
    """Tokens that share a CTA, with a last CTA that is not full; one CTA a token; a token over several CTAs. In place and into a new buffer,
    against 64 bits: products and sums are 32-bit, one bf16 rounding."""
    torch.manual_seed(T)
    x = torch.randn(1, T, heads * D, device="cuda", dtype=torch.bfloat16)
    cos, sin = F_.rope_tables(T, D, 1e4, "cuda")
    ref = F_.rope_reference(x[..., :rot * D].reshape(1, T, rot, D).double(), cos.double(), sin.double()).reshape(1, T, -1)
    y = F_.rope_qk_(x, cos, sin, rot, D)
    assert bool(((y[..., :rot * D].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all()) and torch.equal(y[..., rot * D:], x[..., rot * D:])
    z = x.clone()
    _lib.call("sx_rope", ptr(z), ptr(cos), ptr(sin), ptr(None), c_ll(T), c_int(T), c_int(rot), c_int(D), c_ll(heads * D), c_int(0), c_int(0), stream())
    assert torch.equal(z, y)


def test_rope_of_small_tokens_keeps_up_with_a_copy():
    """One head of 16 a token: 8 MB in and out. 74 us when a CTA held one token, 10 us now (both with the launch, from a cold cache)."""
    T, D = 131072, 16
    x = torch.randn(T, D, device="cuda", dtype=torch.bfloat16)
    cos, sin = F_.rope_tables(8192, D, 1e4, "cuda")
    us = _median_us(lambda: _lib.call("sx_rope", ptr(x), ptr(cos), ptr(sin), ptr(None), c_ll(T), c_int(8192), c_int(1), c_int(D), c_ll(D), c_int(0),
                                      c_int(0), stream()))
    assert us < 10 * _copy_us(2 * x.numel() * 2) + 15, us


@pytest.mark.parametrize("d", [8200, 12288, 16384])
def test_rmsnorm_backward_of_long_rows_keeps_up_with_a_copy(d):
    """Rows of more than 8192 read dy and the input and write dx: 2.4 to 2.7 times a copy's time, 5.6 to 6.9 when the kernel spilled registers."""
    T = 8192
    dy, x, dx = (torch.randn(T, d, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    w, dw, rstd = torch.randn(d, device="cuda").bfloat16(), torch.empty(d, device="cuda", dtype=torch.bfloat16), torch.ones(T, device="cuda")
    part = torch.empty(_lib.lib().sx_rmsnorm_bwd_parts(c_int(d)) * d, device="cuda")
    us = _median_us(lambda: _lib.call("sx_rmsnorm_bwd", ptr(dy), ptr(x), ptr(w), ptr(rstd), ptr(None), ptr(dx), ptr(part), ptr(dw), ptr(None), c_int(0),
                                      c_ll(T), c_int(d), stream()))
    assert us < 4 * _copy_us(3 * T * d * 2), us


@pytest.mark.parametrize("d,rows", [(8, 592), (2048, 592), (2056, 296), (16384, 296)])
def test_rmsnorm_backward_scratch(d, rows):
    """The scratch is what the widths use: with it, rows behind the scratch stay as they are."""
    assert _lib.lib().sx_rmsnorm_bwd_parts(c_int(d)) == rows
    T = 1000
    dy, x, dx = (torch.randn(T, d, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    w, dw, rstd = torch.randn(d, device="cuda").bfloat16(), torch.empty(d, device="cuda", dtype=torch.bfloat16), torch.ones(T, device="cuda")
    part = torch.full((rows + 8, d), 7.0, device="cuda")
    _lib.call("sx_rmsnorm_bwd", ptr(dy), ptr(x), ptr(w), ptr(rstd), ptr(None), ptr(dx), ptr(part), ptr(dw), ptr(None), c_int(0), c_ll(T), c_int(d), stream())
    assert bool((part[rows:] == 7.0).all()) and not bool((part[:rows] == 7.0).all(1).any())


def _attn_bwd_args(B, S, H, Hk, o=None):
    """Arguments of a causal sx_attn_bwd call, with everything that it fills poisoned; and the tensors that they point to."""
    D, bf = 128, torch.bfloat16
    q, do = (torch.randn(B, S, H, D, device="cuda").to(bf) for _ in range(2))
    k, v = (torch.randn(B, S, Hk, D, device="cuda").to(bf) for _ in range(2))
    o_fwd, lse = F_.attention_with_lse(q, k, v, causal=True)
    if o is not None:
        o.copy_(o_fwd)
    t = dict(q=q, k=k, v=v, do=do, o=o_fwd if o is None else o, lse=lse, acc=torch.full((B, H, (S + 63) // 64 * 64, D), float("nan"), device="cuda"),
             delta=torch.full((B, H, S), float("nan"), device="cuda"), dq=torch.empty_like(q), dk=torch.empty_like(k), dv=torch.empty_like(v))
    a = F_._attn_args(q, k, v, t["o"], lse, True, 0, D ** -0.5, 1)
    a.dO, a.dQ, a.dK, a.dV = (t[n].data_ptr() for n in ("do", "dq", "dk", "dv"))
    a.dq_accum, a.delta = t["acc"].data_ptr(), t["delta"].data_ptr()
    a.do_row_stride = H * D
    a.dq_row_stride, a.dk_row_stride, a.dv_row_stride = H * D, Hk * D, Hk * D
    a.dq_batch_stride, a.dk_batch_stride, a.dv_batch_stride = S * H * D, S * Hk * D, S * Hk * D
    return a, t


@pytest.mark.parametrize("B,S,H,Hk", [(1, 1, 4, 1), (1, 1, 32, 32), (3, 2, 8, 8), (1, 63, 8, 2), (2, 65, 4, 4), (1, 300, 7, 1)])
def test_attention_backward_prologue(B, S, H, Hk):
    """The accumulator of dQ is zeroed, whole tiles also where they hold few queries, and delta is the sum of dO O. delta: 128 products in
    32 bits, 2^-17 of the sum of magnitudes."""
    a, t = _attn_bwd_args(B, S, H, Hk)
    _lib.call("sx_attn_bwd", C.byref(a), stream())
    ops.check_status()
    prod = (t["do"].double() * t["o"].double()).permute(0, 2, 1, 3)
    assert bool(((t["delta"].double() - prod.sum(-1)).abs() <= prod.abs().sum(-1) * 2.0 ** -17).all())
    assert bool(t["acc"].isfinite().all()) and bool(t["dq"].isfinite().all())


@pytest.mark.parametrize("shift,pad", [(2, 0), (0, 2), (6, 10), (8, 4)])
def test_attention_backward_takes_an_output_on_four_bytes(shift, pad):
    """Rows of O that start on 4 but not on 16 bytes give what aligned ones give, bit for bit (one key tile: no order of additions)."""
    B, S, H, D = 2, 100, 4, 128
    torch.manual_seed(shift + pad)
    flat = torch.randn(B * S * (H * D + pad) + 64, device="cuda").bfloat16()
    a, t = _attn_bwd_args(B, S, H, 2, flat[shift:].as_strided((B, S, H, D), (S * (H * D + pad), H * D + pad, D, 1)))
    assert a.o_row_stride == H * D + pad
    _lib.call("sx_attn_bwd", C.byref(a), stream())
    want = F_.attention_backward(t["q"], t["k"], t["v"], t["o"].contiguous(), t["lse"], t["do"])
    ops.check_status()
    assert all(torch.equal(t[n], w) for n, w in zip(("dq", "dk", "dv"), want))


def test_attention_backward_of_one_query_zeroes_with_many_ctas():
    """Sixteen times the heads of one query take little longer than one head: 64 heads hold 2 MB of accumulator tiles, 24 us more than one head when
    one CTA zeroed them, 4 us now."""
    us = []
    for H in (4, 64):
        a, t = _attn_bwd_args(1, 1, H, H)
        us.append(_median_us(lambda: _lib.call("sx_attn_bwd", C.byref(a), stream())))
    assert us[1] < us[0] + 14, us


@pytest.mark.parametrize("Sq,Skv,causal,window", [(1, 200, True, 0), (33, 33, True, 0), (64, 300, False, 0), (65, 65, True, 0), (128 + 1, 129, True, 0), (128 + 64, 400, True, 0),
                                                  (128 + 65, 193, False, 0), (256 + 40, 296, True, 50)])
def test_attention_backward_reads_no_column_behind_the_last_query(Sq, Skv, causal, window):
    """A last tile of at most 64 queries leaves half of the probabilities' and their gradients' columns as they were. What lay there before, values of
    another call or NaN of one whose inputs were NaN, does not show: the bits of a call after one of finite values."""
    torch.manual_seed(Sq)
    H, Hk = 6, 2
    q, do = (torch.randn(1, Sq, H, 128, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(1, Skv, Hk, 128, device="cuda").bfloat16() for _ in range(2))
    o, lse = F_.attention_with_lse(q, k, v, causal=causal, window=window)
    bad = [torch.full((1, 1024, 37 * 4, 128), float("nan"), device="cuda").bfloat16() for _ in range(2)]
    got = []
    for poison in (False, True, True):
        if poison:      # every SM's shared memory and TMEM
            F_.attention_backward(bad[0], bad[0], bad[0], bad[0], torch.zeros(1, 37 * 4, 1024, device="cuda"), bad[1], causal=False)
        got.append(F_.attention_backward(q, k, v, o, lse, do, causal=causal, window=window))
    ops.check_status()
    for g in got[1:]:
        assert torch.equal(g[1], got[0][1]) and torch.equal(g[2], got[0][2])          # dK and dV keep their bits, dQ is summed in any order
        assert (g[0].float() - got[0][0].float()).norm() <= 2.0 ** -8 * got[0][0].float().norm()


def _attention64(q, k, v, do, causal, window):
    """Output and gradients in 64 bits, and the probabilities' sum over the keys."""
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    (B, Sq, H, D), Skv, rep = q.shape, k.shape[1], q.shape[2] // k.shape[2]
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(rep, 2)) / math.sqrt(D)
    i = torch.arange(Sq, device="cuda").view(-1, 1) + Skv - Sq
    j = torch.arange(Skv, device="cuda").view(1, -1)
    hidden = (j > i if causal else torch.zeros_like(j > i)) | ((j <= i - window) if window else torch.zeros_like(j > i))
    p = s.masked_fill(hidden, -math.inf).softmax(-1)
    o = torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(rep, 2))
    pk = torch.einsum("bhqk,bkhd->bqhd", p, k.repeat_interleave(rep, 2)).detach()
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), do.double())), pk


@pytest.mark.parametrize("H,Hk", [(2, 2), (7, 1)])
@pytest.mark.parametrize("Sq,Skv,causal,window", [
    (1, 1, True, 0), (63, 63, True, 0), (64, 64, True, 0), (65, 65, True, 0), (77, 77, True, 0), (129, 129, True, 0), (130, 130, False, 0), (257, 257, True, 0),
    (1, 300, True, 0), (65, 129, True, 0), (77, 200, True, 0), (130, 1000, True, 0), (100, 260, False, 0), (260, 100, False, 0),
    (64, 1024, True, 100), (192, 1000, True, 70), (700, 700, True, 64), (321, 321, True, 1)])
def test_attention_backward_tiles(H, Hk, Sq, Skv, causal, window):
    """One, two, three and more query tiles of a key tile, odd and even numbers of them over the heads of a group, key tiles that no query sees,
    partial tiles of both, queries that follow cached keys. Every row of every result by itself: P, dS, O and the results are rounded to bf16
    (2^-9 each, at random), so a row is within 2^-7 of its norm, and, where it cancels, of the root mean square of the rows. The rounding of O
    moves delta, by 2^-9 sum |dO O| at most, which goes into a row of dQ with the factor scale |P K|; into dK with P and over the queries, at random,
    below the terms before."""
    B = 1 if Skv == 1 else 2
    torch.manual_seed(Sq + Skv)
    q, do = (torch.randn(B, Sq, H, 128, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Skv, Hk, 128, device="cuda").bfloat16() for _ in range(2))
    if Sq == 1 and B == 2:
        q, do, k, v = q[:1], do[:1], k[:1], v[:1]
    ins = [t.clone().requires_grad_() for t in (q, k, v)]
    o = F_.attention(*ins, causal=causal, window=window)
    got = (o.detach(), *torch.autograd.grad(o, ins, do))
    ops.check_status()
    want, pk = _attention64(q, k, v, do, causal, window)
    delta = 2.0 ** -9 * (do.double() * want[0]).abs().sum(-1) * pk.norm(dim=-1) / math.sqrt(128)
    for name, a, e in zip(("o", "dq", "dk", "dv"), got, want):
        err, norm = (a.double() - e).norm(dim=-1), e.norm(dim=-1)
        bound = 2.0 ** -7 * norm + 2.0 ** -7 * norm.square().mean().sqrt() + 1e-4 + (delta if name == "dq" else 0.0)
        assert bool((err <= bound).all()), (name, (err / bound).max().item())


@pytest.mark.parametrize("D", [64, 128])
def test_attention_forward_of_a_batch_is_that_of_its_sequences(D):
    """Keys and values of more than 64 MB take the blocks one sequence after another, a sequence by itself starts heads and tiles heaviest first: the
    same bits, last partial tile and log-sum-exp included."""
    B, Sq, Skv, H = 5, 300, 4096, 16
    torch.manual_seed(D)
    q = torch.randn(B, Sq, H, D, device="cuda").bfloat16()
    k, v = (torch.randn(B, Skv, H, D, device="cuda").bfloat16() for _ in range(2))
    o, lse = F_.attention_with_lse(q, k, v, causal=True)
    for b in range(B):
        ob, lb = F_.attention_with_lse(q[b:b + 1], k[b:b + 1], v[b:b + 1], causal=True)
        assert torch.equal(ob[0], o[b]) and torch.equal(lb[0], lse[b])
    ops.check_status()


@pytest.mark.parametrize("causal", [True, False])
def test_attention_forward_of_many_short_sequences(causal):
    """More sequences than the second axis of a grid holds: the bits that a few of them give alone."""
    torch.manual_seed(3)
    B, S = 65536 + 70, 3
    q = torch.randn(B, S, 2, 64, device="cuda").bfloat16()
    k, v = (torch.randn(B, S, 1, 64, device="cuda").bfloat16() for _ in range(2))
    with torch.no_grad():
        o = F_.attention(q, k, v, causal=causal)
        for r in (slice(0, 40), slice(65520, 65560), slice(B - 40, B)):
            assert torch.equal(o[r], F_.attention(q[r], k[r], v[r], causal=causal))
    ops.check_status()


def test_attention_forward_of_many_queries():
    """More pairs of query tiles than the second axis of a grid holds, on three keys: the bits that the first and the last queries give alone."""
    torch.manual_seed(4)
    S = 65536 * 256 + 300
    q = torch.randn(1, S, 1, 64, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(1, 3, 1, 64, device="cuda").bfloat16() for _ in range(2))
    with torch.no_grad():
        o = F_.attention(q, k, v, causal=False)
        for r in (slice(0, 600), slice(1 << 23, (1 << 23) + 600), slice(S - 600, S)):
            assert torch.equal(o[:, r], F_.attention(q[:, r].contiguous(), k, v, causal=False))
    ops.check_status()


@pytest.mark.parametrize("key", [0, 70, 127, 128, 300])
def test_attention_forward_passes_nan_scores_on(key):
    """A key of NaN makes every query that sees it NaN and leaves the others as they are; queries that see no key are zero."""
    S, H = 333, 4
    torch.manual_seed(key)
    q, k, v = (torch.randn(1, S, H, 128, device="cuda").bfloat16() for _ in range(3))
    want = F_.attention_with_lse(q, k, v, causal=True)[0]
    k[:, key] = float("nan")
    o = F_.attention_with_lse(q, k, v, causal=True)[0]
    assert bool(o[:, key:].isnan().all()) and torch.equal(o[:, :key], want[:, :key])
    none = F_.attention_with_lse(q, k[:, :100], v[:, :100], causal=True)[0]      # the first 233 queries come before every key
    assert bool((none[:, :S - 100] == 0).all())
    ops.check_status()


@pytest.mark.parametrize("B,S,H,Hk,pad", [(1, 1, 1, 1, 0), (2, 31, 4, 2, 4), (3, 32, 3, 1, 12), (2, 33, 28, 4, 4), (2, 65, 2, 2, 0), (3, 129, 6, 3, 8)])
def test_attention_backward_converts_its_accumulator(B, S, H, Hk, pad):
    """dQ is the accumulator (pieces of 32 queries, groups of 4 columns, queries, columns), scaled and rounded once: equal bits; nothing is written
    between the rows of a dQ whose row stride is a multiple of 4 elements."""
    torch.manual_seed(S)
    a, t = _attn_bwd_args(B, S, H, Hk)
    P = (S + 63) // 64 * 2
    acc = torch.empty(B, H, P, 32, 32, 4, device="cuda")
    dq = torch.full((B, S, H * 128 + pad), 7.0, dtype=torch.bfloat16, device="cuda")
    a.dq_accum, a.dQ, a.dq_row_stride, a.dq_batch_stride = acc.data_ptr(), dq.data_ptr(), dq.stride(1), dq.stride(0)
    _lib.call("sx_attn_bwd", C.byref(a), stream())
    ops.check_status()
    want = (acc * torch.tensor(a.scale, dtype=torch.float32, device="cuda")).bfloat16()
    want = want.permute(0, 2, 4, 1, 3, 5).reshape(B, P * 32, H * 128)[:, :S]
    assert torch.equal(dq[..., :H * 128].view(torch.int16), want.view(torch.int16))
    assert bool((dq[..., H * 128:] == 7.0).all())


@pytest.mark.parametrize("S,H,Hk", [(1, 2, 1), (64, 3, 3), (65, 4, 2), (127, 2, 2), (128, 5, 1), (150, 4, 4), (193, 2, 1), (256, 3, 1), (513, 2, 2)])
def test_attention_backward_stays_inside_its_accumulator(S, H, Hk):
    """The last query tile may reach behind the accumulator, which holds multiples of 64 queries: nothing is added there, and the results are those
    of 64 bits. Three roundings to bf16 lie between (P or dS, an operand's and the result's, 2^-9 each): 2^-7 of the norm."""
    torch.manual_seed(S)
    a, t = _attn_bwd_args(1, S, H, Hk)
    n = H * ((S + 63) // 64 * 64) * 128
    acc = torch.full((n + 64 * 128,), 7.0, device="cuda")
    a.dq_accum = acc.data_ptr()
    _lib.call("sx_attn_bwd", C.byref(a), stream())
    ops.check_status()
    assert bool((acc[n:] == 7.0).all())
    want, _ = _attention64(t["q"], t["k"], t["v"], t["do"], True, 0)
    for name, e in zip(("dq", "dk", "dv"), want[1:]):
        if e.norm() > 1e-6:         # one key: no gradient of the scores
            assert (t[name].double() - e).norm() <= 2.0 ** -7 * e.norm(), name
