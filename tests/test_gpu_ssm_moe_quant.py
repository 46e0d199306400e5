"""conv1d, chunked SSD scan, router / MoE and quantisation kernels against fp32 PyTorch references."""
import pytest
import torch

from sneppx_alg_b200 import ops
from sneppx_alg_b200.ops import _lib, moe, quant, ssm

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return (a.float() - b.float()).abs().max().item() / (b.float().abs().max().item() + 1e-6)


@pytest.mark.parametrize("with_prev,act", [(False, True), (True, True), (False, False)])
def test_conv1d(with_prev, act):
    torch.manual_seed(0)
    B, L, C, K = 2, 200, 320, 4
    x = torch.randn(B, L, C, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (0.5 * torch.randn(C, K, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(C, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    prev = torch.randn(B, K - 1, C, device="cuda", dtype=torch.bfloat16) if with_prev else None
    y = ssm.causal_conv1d(x, w, b, act, prev)
    g = torch.randn_like(y)
    y.backward(g)
    xr, wr, br = [t.detach().float().requires_grad_(True) for t in (x, w, b)]
    yr = ssm.conv1d_reference(xr, wr, br, act, prev.float() if with_prev else None)
    yr.backward(g.float())
    assert _rel(y, yr) < 2e-2
    assert _rel(x.grad, xr.grad) < 3e-2 and _rel(w.grad, wr.grad) < 3e-2 and _rel(b.grad, br.grad) < 3e-2


@pytest.mark.parametrize("L,chunk,G", [(256, 64, 1), (512, 256, 2), (200, 64, 1)])
def test_ssd_chunked_vs_recurrence(L, chunk, G):
    torch.manual_seed(0)
    B, H, P, N = 2, 4, 64, 64
    x = torch.randn(B, L, H, P, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dt = (torch.rand(B, L, H, device="cuda") * 0.1 + 1e-3).requires_grad_(True)
    A = (-torch.rand(H, device="cuda") * 4 - 0.5).requires_grad_(True)
    Bm = torch.randn(B, L, G, N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    Cm = torch.randn(B, L, G, N, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    D = torch.randn(H, device="cuda", requires_grad=True)
    y = ssm.ssd_scan(x, dt, A, Bm, Cm, D, chunk=chunk)
    g = torch.randn_like(y)
    y.backward(g)
    ops.check_status()
    ref_in = [t.detach().float().requires_grad_(True) for t in (x, dt, A, Bm, Cm, D)]
    yr = ssm.ssd_reference(*ref_in)
    yr.backward(g.float())
    assert _rel(y, yr) < 3e-2
    for got, ref, name in zip((x, dt, A, Bm, Cm, D), ref_in, "x dt A B C D".split()):
        assert _rel(got.grad, ref.grad) < 6e-2, name


def test_conv1d_strided_input_and_gate_mul():
    """conv1d reads a column slice of a wider tensor in place; the output gate y * silu(z) does the same for z."""
    torch.manual_seed(2)
    B, L, C, W = 2, 300, 192, 512
    wide = torch.randn(B, L, W, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(C, 4, device="cuda") * 0.3).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(C, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    y = ssm.causal_conv1d(wide[..., 64:64 + C], w, b, act=True)
    out = ssm.gate_mul(y, wide[..., 320:320 + C])
    g = torch.randn_like(out)
    out.backward(g)
    wr, ww, bb = [t.detach().float().requires_grad_(True) for t in (wide, w, b)]
    yr = ssm.conv1d_reference(wr[..., 64:64 + C], ww, bb, True, None)
    outr = yr * torch.nn.functional.silu(wr[..., 320:320 + C])
    outr.backward(g.float())
    assert _rel(out, outr) < 2e-2
    assert _rel(wide.grad, wr.grad) < 3e-2 and _rel(w.grad, ww.grad) < 3e-2 and _rel(b.grad, bb.grad) < 3e-2


def test_ssd_scan_states_and_long_chunks():
    """Initial and final state, their gradients, chunk 128 with 128 state columns (the Mamba-2 2.7B tiling)."""
    torch.manual_seed(1)
    B, L, H, P, N, G = 1, 384, 8, 64, 128, 1
    mk = lambda *s, dt=torch.bfloat16: torch.randn(*s, device="cuda", dtype=dt)
    x = mk(B, L, H, P).requires_grad_(True)
    dt = (torch.rand(B, L, H, device="cuda") * 0.1 + 1e-3).requires_grad_(True)
    A = (-torch.rand(H, device="cuda") * 4 - 0.5).requires_grad_(True)
    Bm, Cm = mk(B, L, G, N).requires_grad_(True), mk(B, L, G, N).requires_grad_(True)
    D = mk(H, dt=torch.float32).requires_grad_(True)
    h0 = mk(B, H, P, N, dt=torch.float32).requires_grad_(True)
    ins = [x, dt, A, Bm, Cm, D, h0]
    y, hf = ssm.ssd_scan(x, dt, A, Bm, Cm, D, chunk=128, init_state=h0, return_state=True)
    g, gf = torch.randn_like(y), torch.randn_like(hf)
    grads = torch.autograd.grad((y.float() * g.float()).sum() + (hf * gf).sum(), ins)
    ops.check_status()
    ref = [t.detach().float().requires_grad_(True) for t in ins]
    yr, hr = ssm.ssd_reference(*ref[:6], init_state=ref[6], return_state=True)
    gr = torch.autograd.grad((yr * g.float()).sum() + (hr * gf).sum(), ref)
    assert _rel(y, yr) < 3e-2 and _rel(hf, hr) < 3e-2
    for got, want, name in zip(grads, gr, "x dt A B C D h0".split()):
        assert _rel(got, want) < 6e-2, name


def test_ssd_fused_chunk_kernel_matches_staged_path(monkeypatch):
    """tcgen05 output-stage kernel (chunk 128, state 128, headdim 64) against the staged path and the fp32 recurrence;
    x, B and C are column slices of one wider token-major tensor, as in the Mamba-2 block; two B/C groups."""
    torch.manual_seed(4)
    B, L, H, P, N, G = 2, 512, 8, 64, 128, 2
    wide = torch.randn(B, L, H * P + 2 * G * N + 64, device="cuda", dtype=torch.bfloat16)
    x = wide[..., :H * P].reshape(B, L, H, P)
    Bm = wide[..., H * P:H * P + G * N].reshape(B, L, G, N)
    Cm = wide[..., H * P + G * N:H * P + 2 * G * N].reshape(B, L, G, N)
    dt = torch.rand(B, L, H, device="cuda") * 0.1 + 1e-3
    A = -torch.rand(H, device="cuda") * 4 - 0.5
    D = torch.randn(H, device="cuda")
    h0 = torch.randn(B, H, P, N, device="cuda")
    with torch.no_grad():
        y1, f1 = ssm.ssd_scan(x, dt, A, Bm, Cm, D, chunk=128, init_state=h0, return_state=True)
        ops.check_status()
        monkeypatch.setenv("SX_SSD_FUSED", "0")
        y0, f0 = ssm.ssd_scan(x, dt, A, Bm, Cm, D, chunk=128, init_state=h0, return_state=True)
        yr = ssm.ssd_reference(x.float(), dt, A, Bm.float(), Cm.float(), D, init_state=h0)
    assert _rel(y1, yr) < 2e-2 and _rel(y0, yr) < 2e-2
    assert _rel(y1, y0) < 1e-2 and torch.equal(f1, f0)


@pytest.mark.parametrize("H,G", [(1, 1), (2, 1), (3, 1), (5, 1), (24, 1), (9, 3), (16, 8)])
def test_ssd_chunk_kernel_deals_heads_out(H, G):
    """One chunk deals its heads out over many CTAs, odd numbers and a last short share among them; two hundred copies of it take one CTA a group:
    the same bits. Against 64 bits: M is rounded to bf16 before its product and the sum to bf16 after it, 2^-9 of their magnitudes each."""
    from sneppx_alg_b200.ops import _lib
    from sneppx_alg_b200.ops._lib import c_int, c_ll, ptr, stream
    torch.manual_seed(H + G)
    Q, P, N, n = 128, 64, 128, 200
    rows = torch.randn(Q, H * P + 2 * G * N, device="cuda").bfloat16()
    state = torch.randn(H, P, N, device="cuda").bfloat16()
    dt = torch.rand(H, Q, device="cuda") * 0.1
    cs = torch.cumsum(-dt * (1 + 15 * torch.rand(H, 1, device="cuda")), -1)
    D = torch.randn(H, device="cuda")
    ys = []
    for bc in (1, n):
        u = rows.repeat(bc, 1)
        W, B_, C_ = u.shape[1], u[:, H * P:], u[:, H * P + G * N:]
        hp, cs_, dt_ = (t.repeat(bc, *[1] * (t.dim() - 1)) for t in (state, cs, dt))
        y = torch.full((bc * Q, H * P), float("nan"), device="cuda").bfloat16()
        _lib.call("sx_ssd_chunk_fwd", ptr(C_), c_ll(W), ptr(B_), c_ll(W), ptr(u), c_ll(W), ptr(hp), ptr(cs_), ptr(dt_), ptr(D), ptr(y), c_ll(bc),
                  c_int(H), c_int(G), ptr(_lib.status_word("cuda")), stream())
        ys.append(y.view(bc, Q, H, P))
    ops.check_status()
    assert bool((ys[1] == ys[0]).all())
    x = rows[:, :H * P].double().view(Q, H, P)
    Bm, Cm = (rows[:, o:o + G * N].double().view(Q, G, N).repeat_interleave(H // G, 1) for o in (H * P, H * P + G * N))
    M = torch.einsum("lhn,shn->hls", Cm, Bm) * (cs.double()[:, :, None] - cs.double()[:, None]).exp().tril() * dt.double()[:, None]
    terms = [torch.einsum("hls,shp->lhp", M, x), torch.einsum("lhn,hpn->lhp", Cm, state.double()) * cs.double().exp().t()[..., None], D.double()[:, None] * x]
    size = torch.einsum("hls,shp->lhp", M.abs(), x.abs()) + terms[0].abs() + terms[1].abs() + terms[2].abs()
    assert bool(((ys[0][0].double() - sum(terms)).abs() <= 2.0 ** -8 * size + 1e-6).all())


@pytest.mark.parametrize("H,G", [(24, 1), (80, 8)])
def test_ssd_chunk_kernel_repeats_itself(H, G):
    """The skip connection reads x from the tile that TMA brought while other tiles are on their way: calls over rows that change in between, one
    behind the other, give the bits of calls that are waited for. The skip connection outweighs the rest a thousand times, so that a row which came late shows."""
    from sneppx_alg_b200.ops._lib import c_int, c_ll, ptr, stream
    torch.manual_seed(H)
    Q, P, N, bc = 128, 64, 128, 40
    u = [torch.randn(bc * Q, H * P + 2 * G * N, device="cuda").bfloat16() for _ in range(4)]
    W, state = u[0].shape[1], torch.randn(bc, H, P, N, device="cuda").bfloat16()
    dt = torch.rand(bc, H, Q, device="cuda") * 0.1
    cs, D = torch.cumsum(-dt, -1), 1000 * torch.randn(H, device="cuda")
    rows = torch.empty_like(u[0])

    def call(x):
        rows.copy_(x)
        y = torch.empty(bc * Q, H * P, dtype=torch.bfloat16, device="cuda")
        _lib.call("sx_ssd_chunk_fwd", ptr(rows[:, H * P + G * N:]), c_ll(W), ptr(rows[:, H * P:]), c_ll(W), ptr(rows), c_ll(W), ptr(state), ptr(cs), ptr(dt),
                  ptr(D), ptr(y), c_ll(bc), c_int(H), c_int(G), ptr(_lib.status_word("cuda")), stream())
        return y

    want = []
    for x in u:
        want.append(call(x))
        torch.cuda.synchronize()
    got = [call(u[i % 4]) for i in range(24)]
    _lib.check_status()
    assert all(torch.equal(y, want[i % 4]) for i, y in enumerate(got))
    skip = D.repeat_interleave(P) * u[0][:, :H * P].float()
    assert (want[0].float() - skip).norm() < 0.02 * skip.norm()


def test_router_and_moe_layer():
    torch.manual_seed(0)
    T, d, E, k, Fd = 1000, 256, 16, 4, 192
    x = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    logits = torch.randn(T, E, device="cuda")
    idx, w, probs, counts = moe.route(logits, k)
    ref_idx = moe.topk_reference(torch.softmax(logits, -1), k)
    assert torch.equal(idx.sort(-1).values, ref_idx.sort(-1).values)
    assert torch.allclose(w.sum(-1), torch.ones(T, device="cuda"), atol=1e-5)
    assert counts.sum().item() == T * k
    W1 = (0.05 * torch.randn(E, 2 * Fd, d, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    W2 = (0.05 * torch.randn(E, d, Fd, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    w = w.detach().requires_grad_(True)
    y = moe.experts_forward(x, idx, w, W1, W2)
    g = torch.randn_like(y)
    y.backward(g)
    ops.check_status()
    xr, wr, W1r, W2r = [t.detach().float().requires_grad_(True) for t in (x, w, W1, W2)]
    yr = moe.moe_reference(xr, idx, wr, W1r, W2r)
    yr.backward(g.float())
    assert _rel(y, yr) < 3e-2
    assert _rel(x.grad, xr.grad) < 4e-2 and _rel(w.grad, wr.grad) < 4e-2
    assert _rel(W1.grad, W1r.grad) < 4e-2 and _rel(W2.grad, W2r.grad) < 4e-2


def test_quant_roundtrip_and_reference():
    torch.manual_seed(0)
    x = torch.randn(300, 512, device="cuda", dtype=torch.bfloat16) * 3
    q, s = quant.quant_fp8_1x128(x)
    qr, sr = quant.quant_fp8_1x128_reference(x)
    assert torch.allclose(s, sr, rtol=1e-6)
    assert (q.float() - qr.float()).abs().max().item() <= 32.0  # at most one e4m3 step at the top binade
    assert (q.view(torch.uint8) != qr.view(torch.uint8)).float().mean().item() < 0.01
    assert _rel(quant.dequant_fp8(q, s, "1x128"), x) < 0.07
    w = torch.randn(200, 384, device="cuda", dtype=torch.bfloat16)
    qw, sw = quant.quant_fp8_128x128(w)
    qwr, swr = quant.quant_fp8_128x128_reference(w)
    assert torch.allclose(sw, swr, rtol=1e-6)
    assert _rel(quant.dequant_fp8(qw, sw, "128x128"), w) < 0.07
    w4 = torch.randn(128, 256, device="cuda", dtype=torch.bfloat16)
    p, s4 = quant.quant_int4(w4)
    pr, s4r = quant.quant_int4_reference(w4)
    assert torch.allclose(s4, s4r, rtol=1e-6) and (p != pr).float().mean().item() < 0.01
    assert _rel(quant.dequant_int4(p, s4), w4) < 0.2


def test_models_train_on_gpu():
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.training.engine import TrainEngine
    torch.manual_seed(0)
    cfgs = [
        ModelConfig(architecture="mamba2", hidden_size=256, num_hidden_layers=2, vocab_size=1000, ssm_state_size=64,
                    ssm_head_dim=64, ssm_ngroups=1, ssm_chunk_size=64, tie_word_embeddings=True),
        ModelConfig(architecture="hss_ser", hidden_size=256, num_hidden_layers=2, vocab_size=1024, ssm_state_size=64,
                    ssm_head_dim=64, ssm_chunk_size=64, num_experts=8, num_experts_per_token=2,
                    moe_intermediate_size=256, router_aux_loss_coef=0.01, tie_word_embeddings=True),
        ModelConfig(architecture="deepseek_moe", hidden_size=256, num_hidden_layers=2, num_attention_heads=2,
                    head_dim=128, intermediate_size=512, vocab_size=1024, num_experts=8, num_experts_per_token=2,
                    num_shared_experts=1, moe_intermediate_size=128, first_dense_layers=1,
                    router_aux_loss_coef=0.001, max_position_embeddings=256),
    ]
    for cfg in cfgs:
        model = build_model(cfg, dtype=torch.bfloat16, device="cuda")
        eng = TrainEngine(model, lr=2e-3, max_grad_norm=1.0)
        ids = torch.randint(0, 1000, (2, 256), device="cuda")
        first = eng.step(ids, ids).item()
        for _ in range(6):
            last = eng.step(ids, ids).item()
        ops.check_status()
        assert last == last and last < first, (cfg.architecture, first, last)


def test_gemm_fp8_block_scaled():
    """fp8 x fp8 tensor-core GEMM against the fp32 product of the dequantised operands (same quantised inputs, so
    the only differences are accumulation order and the bf16 output rounding)."""
    from sneppx_alg_b200.ops import quant
    torch.manual_seed(0)
    for M, N, K in ((5, 256, 512), (64, 384, 1024), (33, 1000, 256), (200, 128, 2048), (16, 4096, 4096)):
        x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
        w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.05
        bias = torch.randn(N, device="cuda")
        wq, sw = quant.quant_fp8_128x128(w)
        xq, sx = quant.quant_fp8_1x128(x)
        y = quant.gemm_fp8(None, wq, sw, bias=bias, xq=xq, sx=sx)
        ref = quant.gemm_fp8_reference(xq, sx, wq, sw, bias, torch.float32)
        err = (y.float() - ref).abs().max() / ref.abs().max()
        assert err < 1e-2, (M, N, K, float(err))
        # end to end against the unquantised product: fp8 quantisation noise only
        y2 = quant.gemm_fp8(x, wq, sw, bias=bias)
        full = x.float() @ w.float().t() + bias
        assert (y2.float() - full).abs().max() / full.abs().max() < 8e-2
    from sneppx_alg_b200 import ops
    ops.check_status()


@pytest.mark.parametrize("mode", ["fp8", "int4"])
@pytest.mark.parametrize("rows", [64, 300, 2048])
def test_quantized_linear_all_input_sizes(mode, rows):
    """Decode-size inputs take the fp8 x fp8 / in-GEMM dequant paths, prefill-size inputs expand the weight once and
    use the bf16 GEMM; all must agree with the dequantised-weight product."""
    torch.manual_seed(0)
    lin = torch.nn.Linear(512, 384, bias=True, device="cuda", dtype=torch.bfloat16)
    ql = quant.QuantizedLinear.from_linear(lin, mode)
    x = torch.randn(2, rows // 2, 512, device="cuda", dtype=torch.bfloat16)
    y = ql(x)
    if mode == "fp8":
        w = quant.dequant_fp8(ql.qweight.view(torch.float8_e4m3fn), ql.scales, "128x128", torch.float32)
    else:
        w = quant.dequant_int4(ql.qweight, ql.scales, torch.float32)
    ref = x.float() @ w.t() + lin.bias.float()
    assert y.shape == (2, rows // 2, 384)
    # the fp8 x fp8 path also rounds the activations to e4m3 (3 mantissa bits)
    assert _rel(y, ref) < (6e-2 if (mode == "fp8" and rows <= 256) else 2e-2)


def test_grouped_fp8_expert_gemm_and_fp8_moe_layer():
    """Grouped block-scaled fp8 GEMM (expert-sorted rows x stacked expert matrices) against the fp32 product of the
    de-quantised operands; then the SER layer with fp8 forward expert GEMMs against the fp32 dense oracle."""
    from sneppx_alg_b200.ops import quant
    torch.manual_seed(0)
    E, N, K = 5, 384, 512
    groups = [0, 0, 3, -1, 4, 1, 1, 1, -1]
    tg = torch.tensor(groups, dtype=torch.int32, device="cuda")
    rows = 128 * len(groups)
    x = torch.randn(rows, K, device="cuda", dtype=torch.bfloat16)
    W = (torch.randn(E, N, K, device="cuda") * 0.05).to(torch.bfloat16)
    y = quant.gemm_fp8_grouped(x, tg, W)
    ref = quant.gemm_fp8_grouped_reference(x.float(), tg, W.float())
    assert (y.float() - ref.float()).abs().max() / ref.float().abs().max() < 1e-2
    for t, e in enumerate(groups):       # unused tiles are zero, used ones are not
        blk = y[t * 128:(t + 1) * 128].float().abs().max().item()
        assert (blk == 0.0) == (e < 0)
    ops.check_status()
    T, d, Ex, k, Fd = 1000, 256, 8, 2, 128
    xx = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    idx, w, _, _ = moe.route(torch.randn(T, Ex, device="cuda"), k)
    W1 = (0.05 * torch.randn(Ex, 2 * Fd, d, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    W2 = (0.05 * torch.randn(Ex, d, Fd, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    w = w.detach().requires_grad_(True)
    yy = moe.experts_forward(xx, idx, w, W1, W2, fp8=True)
    g = torch.randn_like(yy)
    yy.backward(g)
    ops.check_status()
    xr, wr, W1r, W2r = [t.detach().float().requires_grad_(True) for t in (xx, w, W1, W2)]
    yr = moe.moe_reference(xr, idx, wr, W1r, W2r)
    yr.backward(g.float())
    assert _rel(yy, yr) < 8e-2                       # e4m3 rounding of both operands of both GEMMs
    assert _rel(xx.grad, xr.grad) < 8e-2 and _rel(W1.grad, W1r.grad) < 8e-2 and _rel(W2.grad, W2r.grad) < 8e-2


@pytest.mark.parametrize("B,L,H,P,G,N,K", [
    (2, 256, 8, 64, 1, 128, 4), (1, 500, 8, 64, 2, 128, 4), (3, 129, 8, 64, 8, 128, 4), (2, 127, 8, 64, 1, 128, 4), (2, 1, 8, 64, 1, 128, 4),
    (1, 40, 16, 32, 4, 64, 3), (2, 300, 8, 16, 1, 64, 2), (1, 77, 24, 64, 1, 64, 4), (1, 200, 8, 128, 2, 256, 1)])
def test_mamba2_mixer(B, L, H, P, G, N, K, monkeypatch):
    """The mixer as one node against the plain 32-bit recurrence: chunks that are full, end in padding or shorten with the sequence, one to
    H groups, the fused and the staged output stage, one to four taps. Bound: rounding an operand to bf16 adds 2^-9 relative at random, at
    most about twelve such roundings lie on the way to any result: sqrt(12) 2^-9 = 0.007 of its 2-norm; twice that, and four times for
    the sums of mixed sign over tokens that the step parameters' gradients are."""
    torch.manual_seed(B * L + N)
    di, C = H * P, H * P + 2 * G * N
    zx = torch.randn(B, L, di + C + H, device="cuda")
    zx[..., di + C:] -= 2
    args = [zx.bfloat16(), (0.5 * torch.randn(C, K, device="cuda")).bfloat16(), (0.1 * torch.randn(C, device="cuda")).bfloat16(),
            torch.randn(H, device="cuda") - 1, torch.log(1 + 15 * torch.rand(H, device="cuda")), torch.randn(H, device="cuda")]
    args = [t.requires_grad_() for t in args]
    ref = [t.detach().double().requires_grad_() for t in args]
    z, xbc, dt = torch.split(ref[0], [di, C, H], -1)
    pad = torch.nn.functional.pad(xbc, (0, 0, K - 1, 0))
    xbc = torch.nn.functional.silu(sum(pad[:, k:k + L] * ref[1][:, k] for k in range(K)) + ref[2])
    x, Bm, Cm = torch.split(xbc, [di, G * N, G * N], -1)
    x, Bm, Cm = x.view(B, L, H, P), Bm.view(B, L, G, N).repeat_interleave(H // G, 2), Cm.view(B, L, G, N).repeat_interleave(H // G, 2)
    dt, h, ys = torch.nn.functional.softplus(dt + ref[3]), zx.new_zeros(B, H, P, N, dtype=torch.float64), []
    for t in range(L):
        h = h * torch.exp(-torch.exp(ref[4]) * dt[:, t])[..., None, None] + (dt[:, t, :, None] * x[:, t])[..., None] * Bm[:, t, :, None]
        ys.append((h * Cm[:, t, :, None]).sum(-1) + ref[5][:, None] * x[:, t])
    want = torch.stack(ys, 1).reshape(B, L, di) * torch.nn.functional.silu(z)
    g = torch.randn(B, L, di, device="cuda").bfloat16()
    wgrad = torch.autograd.grad(want, ref, g.double())
    size = (H, P, G, N)
    for fused in ("1", "0"):
        monkeypatch.setenv("SX_SSD_FUSED", fused)
        assert ssm.mixer_ok(*args, *size)
        y = ssm.mamba2_mixer(*args, *size)
        grads = torch.autograd.grad(y, args, g)
        ops.check_status()
        err = lambda a, b: ((a.double() - b).norm() / (b.norm() + 1e-30)).item()  # noqa: E731
        assert y.shape == want.shape and err(y, want) < 0.014
        for got, exp, t, name in zip(grads, wgrad, args, ("zx", "conv", "conv bias", "dt bias", "A_log", "D")):
            if L == 1 and name == "A_log":      # nothing decays before a first token: exactly 0, here 32-bit terms below 100 that cancel
                assert exp.abs().max() == 0 and got.abs().max() < 100 * 2.0 ** -20
                continue
            assert got.shape == t.shape and got.dtype == t.dtype and err(got, exp) < (0.014 if name == "zx" else 0.028), (name, err(got, exp))
        for lo, hi, name in ((0, di, "z"), (di, di + di, "x"), (2 * di, 2 * di + 2 * G * N, "B, C"), (di + C, di + C + H, "dt")):
            assert err(grads[0][..., lo:hi], wgrad[0][..., lo:hi]) < 0.028, (name, err(grads[0][..., lo:hi], wgrad[0][..., lo:hi]))


@pytest.mark.parametrize("B,L,H,P,G,N,fused", [(1, 33, 8, 64, 1, 64, True), (2, 64, 8, 64, 2, 128, True), (1, 65, 8, 64, 1, 128, True), (3, 200, 24, 64, 3, 128, True),
                                               (2, 128, 8, 128, 1, 64, True), (1, 300, 16, 64, 2, 128, False), (40, 128, 8, 64, 1, 128, True)])
def test_mixer_in_one_call_is_the_mixer_by_entry_points(monkeypatch, B, L, H, P, G, N, fused):
    """Chunks of 64 and 128, ragged tails, one and several groups, the fused and the staged output: the same launches in the same order. The same bits
    but where sums are added atomically (the decay's gradient over a state, the taps'), two orders of which are 2^-16 of the sums' terms apart and
    then rounded to bf16 (2^-8 of a value between the two)."""
    from sneppx_alg_b200.ops import _lib
    monkeypatch.setenv("SX_SSD_FUSED", "1" if fused else "0")
    torch.manual_seed(L + H)
    di, C = H * P, H * P + 2 * G * N
    zx = torch.randn(B, L, di + C + H, device="cuda")
    zx[..., di + C:] -= 2
    args = [zx.bfloat16(), (0.5 * torch.randn(C, 4, device="cuda")).bfloat16(), (0.1 * torch.randn(C, device="cuda")).bfloat16(),
            torch.randn(H, device="cuda") - 1, torch.log(1 + 15 * torch.rand(H, device="cuda")), torch.randn(H, device="cuda")]
    args = [t.requires_grad_() for t in args]
    assert ssm.mixer_ok(*args, H, P, G, N)
    g = torch.randn(B, L, di, device="cuda").bfloat16()
    got = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(ssm._MixerFn, "_native", staticmethod(lambda *a: None))
        n = _lib.launch_count
        y = ssm.mamba2_mixer(*args, H, P, G, N)
        assert (_lib.launch_count - n == 1) == native
        got.append((y, *torch.autograd.grad(y, args, g)))
    ops.check_status()
    (y1, z1, *rest1), (y0, z0, *rest0) = got
    assert torch.equal(y1, y0) and torch.equal(z1[..., :di + C], z0[..., :di + C])
    close = lambda a, b: bool(((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 2.0 ** -12 * b.float().abs().max()).all())  # noqa: E731
    assert close(z1, z0) and all(a.dtype == b.dtype and close(a, b) for a, b in zip(rest1, rest0))


def test_mixer_in_one_call_holds_no_more_memory(monkeypatch):
    """Scratch of the pass as one call against that of its entry points one by one, at a size where both are far above the allocator's rounding."""
    torch.manual_seed(0)
    B, L, H, P, G, N = 1, 4096, 40, 64, 4, 128
    di, C = H * P, H * P + 2 * G * N
    zx = torch.randn(B, L, di + C + H, device="cuda").bfloat16().requires_grad_()
    args = [zx, (0.5 * torch.randn(C, 4, device="cuda")).bfloat16(), torch.randn(C, device="cuda").bfloat16(), torch.randn(H, device="cuda") - 3,
            torch.rand(H, device="cuda"), torch.randn(H, device="cuda")]
    g, peaks = torch.randn(B, L, di, device="cuda").bfloat16(), []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(ssm._MixerFn, "_native", staticmethod(lambda *a: None))
        for step in range(2):
            torch.cuda.empty_cache()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            y = ssm.mamba2_mixer(*args, H, P, G, N)
            forward = torch.cuda.max_memory_allocated() - before
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            torch.autograd.grad(y, zx, g)
            backward = torch.cuda.max_memory_allocated() - before
            del y
        peaks.append((forward, backward))
    assert all(a <= b for a, b in zip(*peaks)), peaks


@pytest.mark.parametrize("C,L,Lp,wide", [(64, 1, 1, False), (1536, 1, 1, True), (320, 7, 7, True), (320, 7, 8, True), (64, 33, 64, False)])
def test_gate_mul_padded_rows(C, L, Lp, wide):
    """Dense and wider gradients of z, y with rows behind each sequence that are neither read nor written. 32-bit arithmetic and one bf16 rounding;
    the sigmoid is within 2^-20, which the factor sig (1 + z (1 - sig)) of dz takes up to 1 + 2 |z| < 10 times, against |g y|."""
    from sneppx_alg_b200.ops import _lib
    from sneppx_alg_b200.ops._lib import c_int, c_ll, ptr, stream
    torch.manual_seed(C + L)
    n, bf = 3, torch.bfloat16
    y = torch.full((n, Lp, C), float("nan"), device="cuda", dtype=bf)
    y[:, :L] = torch.randn(n, L, C, device="cuda").to(bf)
    z, g = torch.randn(n, L, C + 64, device="cuda").to(bf), torch.randn(n, L, C, device="cuda").to(bf)
    out, dy = torch.empty(n, L, C, device="cuda", dtype=bf), torch.full_like(y, 3.0)
    dz = torch.full((n, L, C + 64 if wide else C), 3.0, device="cuda", dtype=bf)
    _lib.call("sx_gate_mul_fwd", ptr(y), ptr(z), c_ll(C + 64), ptr(out), c_ll(n * L), c_int(C), c_int(L), c_int(Lp), stream())
    _lib.call("sx_gate_mul_bwd", ptr(g), ptr(y), ptr(z), c_ll(C + 64), ptr(dy), ptr(dz), c_ll(n * L), c_int(C), c_int(L), c_int(Lp), c_ll(dz.shape[-1]),
              stream())
    yr, zr = y[:, :L].double().requires_grad_(), z[..., :C].double().requires_grad_()
    ref = yr * torch.nn.functional.silu(zr)
    grads = torch.autograd.grad(ref, (yr, zr), g.double())
    slack = 1e-5 * (1 + (g.double() * yr.detach()).abs())
    close = lambda a, b: bool(((a.double() - b).abs() <= b.abs() * 2.0 ** -8 + slack).all())  # noqa: E731
    assert close(out, ref.detach()) and close(dy[:, :L], grads[0]) and close(dz[..., :C], grads[1])
    assert bool((dy[:, L:] == 3.0).all()) and bool((dz[..., C:] == 3.0).all())


@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("B,L,C,act", [(2, 77, 72, True), (1, 1, 8, False), (3, 33, 200, True), (1, 300, 320, False), (1, 4856, 6912, True)])
def test_conv1d_taps(K, B, L, C, act):
    """One to four taps, below and above the size from which one and two take wider loads, channels that fill no warp, runs that end in a
    sequence. Products and sums are 32-bit: one bf16
    rounding of outputs, and of gradients (2^-8), with 2^-16 of the sum of magnitudes for sums and for the fast sigmoid."""
    torch.manual_seed(K * C + L)
    x, g = (torch.randn(B, L, C, device="cuda").bfloat16() for _ in range(2))
    w, b = (0.5 * torch.randn(C, K, device="cuda")).bfloat16(), torch.randn(C, device="cuda").bfloat16()
    ins = [t.clone().requires_grad_() for t in (x, w, b)]
    y = ssm.causal_conv1d(*ins, act=act)
    got = torch.autograd.grad(y, ins, g)
    ref = [t.double().requires_grad_() for t in (x, w, b)]
    pad = torch.nn.functional.pad(ref[0], (0, 0, K - 1, 0))
    pre = sum(pad[:, k:k + L] * ref[1][:, k] for k in range(K)) + ref[2]
    yr = torch.nn.functional.silu(pre) if act else pre
    want = torch.autograd.grad(yr, ref, g.double(), retain_graph=True)
    # magnitudes: the same sums over absolute values, the derivative of silu is below 1.1
    up = 1.1 * g.double().abs()
    xa = torch.nn.functional.pad(x.double().abs(), (0, 0, K - 1, 0))
    wa = w.double().abs()
    mag_y = sum(xa[:, k:k + L] * wa[:, k] for k in range(K)) + b.double().abs()
    ua = torch.nn.functional.pad(up, (0, 0, 0, K - 1))
    mag_x = sum(ua[:, K - 1 - k:K - 1 - k + L] * wa[:, k] for k in range(K))
    mag_w = torch.stack([(xa[:, k:k + L] * up).sum((0, 1)) for k in range(K)], 1)
    near = lambda a, e, m: bool(((a.double() - e).abs() <= e.abs() * 2.0 ** -8 + m * 2.0 ** -16 + 1e-30).all())  # noqa: E731
    assert near(y, yr.detach(), mag_y)
    # gradients before their rounding depend on the pre-activation through the sigmoid, which is steepest by |pre| / 4
    k2 = 1 + mag_y.max()
    assert near(got[0], want[0], mag_x * k2) and near(got[1], want[1], mag_w * k2) and near(got[2], want[2], up.sum((0, 1)) * k2)


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("L", [1, 2, 3, 5, 7, 8, 15, 16, 17, 31, 33, 64, 67])
def test_conv1d_forward_runs(K, L, act):
    """Few positions, runs of 16 and runs of 32 (a batch that fills the SMs) give a sequence the same bits, and write the state of its last positions
    and nothing else. Against 64 bits: one rounding to bf16, 2^-8 of the value, and K + 8 roundings to 32 bits of the sum of magnitudes, below 2^-16."""
    torch.manual_seed(100 * L + K)
    C, W = 1024, 1024 + 64
    x = torch.randn(1, L, W, device="cuda").bfloat16()
    prev = torch.randn(1, max(K - 1, 1), C, device="cuda").bfloat16()
    w, b = torch.randn(C, K, device="cuda").bfloat16(), torch.randn(C, device="cuda").bfloat16()

    def run(x, prev, n, state=True):
        B, Ly = x.shape[0], n + 2
        y, s = torch.full((B, Ly, C), 7.0, device="cuda").bfloat16(), torch.full((B, max(K - 1, 1), C), 7.0, device="cuda").bfloat16()
        assert x.is_contiguous() and x.shape[1] == n
        _lib.call("sx_conv1d_fwd", _lib.ptr(x), _lib.ptr(prev if K > 1 else None), _lib.ptr(w), _lib.ptr(b), _lib.ptr(y), _lib.ptr(s if state else None),
                  _lib.c_int(B), _lib.c_int(n), _lib.c_int(C), _lib.c_int(K), _lib.c_int(act), _lib.c_ll(W), _lib.c_int(Ly), _lib.stream())
        assert bool((y[:, n:] == 7.0).all())
        return y[:, :n], s

    y, s = run(x, prev, L)
    ext = torch.cat([prev[:, prev.shape[1] - (K - 1):] if K > 1 else prev[:, :0], x[..., :C]], dim=1).double()
    terms = torch.stack([ext[:, k:k + L] * w[:, k].double() for k in range(K)] + [b.double().expand(1, L, C)])
    want = terms.sum(0)
    want = torch.nn.functional.silu(want) if act else want
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * terms.abs().sum(0)).all())
    for i in range(K - 1):                                      # the state's rows: positions L - (K - 1) + i
        l = L - (K - 1) + i
        assert torch.equal(s[0, i], x[0, l, :C]) if l >= 0 else bool((s[0, i] == 7.0).all())
    n = (2 * 148 * 768 * 4) // (C * ((L + 31) // 32)) + 1       # sequences that make runs of 32
    yb, sb = run(x.repeat(n, 1, 1), prev.repeat(n, 1, 1), L)
    assert bool((yb == y).all()) and bool((sb == s).all())
    assert torch.equal(run(x, prev, L, state=False)[0], y)
    longer = torch.cat([x, torch.randn(1, 40, W, device="cuda").bfloat16()], dim=1)
    assert torch.equal(run(longer, prev, L + 40)[0][:, :L], y)


@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("L", [1, 2, 3, 63, 65, 130])
def test_conv1d_backward_runs(K, L):
    """A batch large enough for runs of 64 positions gives each sequence the bits that runs of 16 give it alone, sequences shorter than the taps and
    ends of runs included; the taps' gradients are sums of 200 equal terms in 32 bits, rounded to bf16."""
    torch.manual_seed(10 * L + K)
    C, n = 1024, 200 * max(1, 128 // L)
    x, g = (torch.randn(1, L, C, device="cuda").bfloat16() for _ in range(2))
    w, b = (0.5 * torch.randn(C, K, device="cuda")).bfloat16(), torch.randn(C, device="cuda").bfloat16()
    grads = []
    for B in (1, n):
        ins = [x.repeat(B, 1, 1).requires_grad_(), w.clone().requires_grad_(), b.clone().requires_grad_()]
        grads.append(torch.autograd.grad(ssm.causal_conv1d(*ins, act=True), ins, g.repeat(B, 1, 1)))
    assert bool((grads[1][0] == grads[0][0]).all())
    for a, e in zip(grads[1][1:], grads[0][1:]):
        assert bool(((a.double() / n - e.double()).abs() <= 2.0 ** -7 * e.double().abs() + 2.0 ** -14 * e.double().abs().max()).all())


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("L,shift", [(16, 0), (33, 0), (100, 0), (33, 4)])
def test_conv1d_one_tap_of_large_inputs(L, shift, act):
    """One tap on inputs that outgrow L2 takes 16-byte loads where the tensors lie on 16 bytes: the bits of a sequence by itself, which takes 8-byte ones."""
    torch.manual_seed(L + shift)
    C = 2048
    n = (1 << 25) // (L * C) + 1
    flat = torch.randn(n * L * C + 8, device="cuda").bfloat16()
    x, w, b = flat[shift:shift + n * L * C].view(n, L, C), torch.randn(C, 1, device="cuda").bfloat16(), torch.randn(C, device="cuda").bfloat16()

    def run(x):
        y = torch.full((x.shape[0], L + 1, C), 7.0, device="cuda").bfloat16()
        _lib.call("sx_conv1d_fwd", _lib.ptr(x), _lib.ptr(None), _lib.ptr(w), _lib.ptr(b), _lib.ptr(y), _lib.ptr(None), _lib.c_int(x.shape[0]), _lib.c_int(L),
                  _lib.c_int(C), _lib.c_int(1), _lib.c_int(act), _lib.c_ll(C), _lib.c_int(L + 1), _lib.stream())
        assert bool((y[:, L:] == 7.0).all())
        return y[:, :L]

    y = run(x)
    assert all(torch.equal(y[i:i + 1], run(x[i:i + 1])) for i in (0, 1, n // 2, n - 1))
    want = x.double() * w[:, 0].double() + b.double()
    want = torch.nn.functional.silu(want) if act else want
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * ((x.double() * w[:, 0].double()).abs() + b.double().abs())).all())
