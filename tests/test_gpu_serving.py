"""Serving kernels on the GPU: KV append + RoPE, paged decode attention, dequant-GEMM, and the paged engine
end to end against plain cached generation."""
import pytest
import torch

from sneppx_alg_b200 import ops
from sneppx_alg_b200.ops import paged, quant
from sneppx_alg_b200.ops.functional import rope_tables

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return (a.float() - b.float()).abs().max().item() / (b.float().abs().max().item() + 1e-6)


def test_kv_append_and_paged_decode():
    torch.manual_seed(0)
    B, Hq, Hkv, D, bs, nblk = 5, 8, 2, 128, 16, 64
    kc = torch.zeros(nblk, bs, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    kc_ref, vc_ref = kc.clone(), vc.clone()
    cos, sin = rope_tables(2048, D, 5e5, "cuda")
    lens = [700, 33, 1, 256, 1500]
    tables = torch.zeros(B, 100, dtype=torch.int32)
    free = list(range(nblk * 0, nblk))
    import random
    random.Random(0).shuffle(free)
    need = sum((n + bs - 1) // bs for n in lens)
    kc = torch.zeros(need + 4, bs, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    kc_ref, vc_ref = kc.clone(), vc.clone()
    nxt = 0
    for b, n in enumerate(lens):
        nb = (n + bs - 1) // bs
        tables[b, :nb] = torch.arange(nxt, nxt + nb, dtype=torch.int32)
        nxt += nb
        qkv = torch.randn(n, (Hq + 2 * Hkv) * D, device="cuda", dtype=torch.bfloat16)
        pos = torch.arange(n, device="cuda", dtype=torch.int32)
        slot = (tables[b, :nb].cuda().repeat_interleave(bs)[:n] * bs + pos % bs).to(torch.int32)
        ref_in = qkv.clone()
        paged.kv_append_(qkv, cos, sin, pos, slot, kc, vc, Hq, Hkv, D)
        ref_f, kc_ref_f, vc_ref_f = ref_in.float(), kc_ref.float(), vc_ref.float()
        paged.kv_append_reference(ref_f, cos, sin, pos, slot, kc_ref_f, vc_ref_f, Hq, Hkv, D)
        kc_ref.copy_(kc_ref_f)
        vc_ref.copy_(vc_ref_f)
        assert _rel(qkv, ref_f) < 1e-2
    assert _rel(kc, kc_ref) < 1e-2 and _rel(vc, vc_ref) < 1e-2
    q = torch.randn(B, Hq, D, device="cuda", dtype=torch.bfloat16)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out = paged.paged_decode(q, kc, vc, tables.cuda(), sl)
    ref = paged.paged_decode_reference(q.float(), kc.float(), vc.float(), tables.cuda(), sl)
    assert _rel(out, ref) < 2e-2


@pytest.mark.parametrize("Hq,Hkv,bs", [(32, 8, 16), (8, 8, 16), (16, 2, 32), (12, 4, 8), (8, 2, 128)])
def test_paged_decode_tensor_core(Hq, Hkv, bs, monkeypatch):
    """Tensor-core decode kernel against the fp32 reference and against the SIMT kernel; cache rows that belong to no
    sequence hold NaN, so any read past a sequence's end that reaches the output fails the test."""
    import random
    torch.manual_seed(1)
    D = 128
    lens = [1, 15, 128, 129, 700, 2304, 0, 1000]
    B = len(lens)
    need = sum((n + bs - 1) // bs for n in lens)
    kc = torch.full((need + 3, bs, Hkv, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    vc = torch.full_like(kc, float("nan"))
    order = list(range(need + 3))
    random.Random(3).shuffle(order)
    width = max((n + bs - 1) // bs for n in lens) + 2
    tables = torch.zeros(B, width, dtype=torch.int32)
    nxt = 0
    for b, n in enumerate(lens):
        nb = (n + bs - 1) // bs
        blocks = order[nxt: nxt + nb]
        nxt += nb
        tables[b, :nb] = torch.tensor(blocks, dtype=torch.int32)
        if n:
            k = torch.randn(n, Hkv, D, device="cuda", dtype=torch.bfloat16)
            v = torch.randn(n, Hkv, D, device="cuda", dtype=torch.bfloat16)
            idx = torch.tensor(blocks, device="cuda").repeat_interleave(bs)[:n] * bs + torch.arange(n, device="cuda") % bs
            kc.view(-1, Hkv, D)[idx] = k
            vc.view(-1, Hkv, D)[idx] = v
    q = (torch.randn(B, Hq, D, device="cuda") * 1.5).to(torch.bfloat16)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    assert paged._use_tc(D, bs, Hq // Hkv)
    out = paged.paged_decode(q, kc, vc, tables.cuda(), sl)
    ops.check_status()
    ref = paged.paged_decode_reference(q.float(), kc.float(), vc.float(), tables.cuda(), sl)
    assert torch.isfinite(out.float()).all()
    assert _rel(out, ref) < 2e-2
    monkeypatch.setenv("SX_PAGED_TC", "0")
    simt = paged.paged_decode(q, kc, vc, tables.cuda(), sl)
    assert _rel(out, simt) < 2e-2


@pytest.mark.parametrize("mode", ["fp8", "int4"])
@pytest.mark.parametrize("M,N,K", [(64, 512, 1024), (300, 1000, 256), (2048, 4096, 4096)])
def test_dequant_gemm(mode, M, N, K):
    torch.manual_seed(0)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    if mode == "fp8":
        q, s = quant.quant_fp8_128x128(w)
        wd = quant.dequant_fp8(q, s, "128x128")
        q = q.view(torch.uint8)
    else:
        q, s = quant.quant_int4(w)
        wd = quant.dequant_int4(q, s)
    bias = torch.randn(N, device="cuda")
    y = quant.gemm_dequant(x, q, s, mode, bias)
    ops.check_status()
    ref = x.float() @ wd.float().t() + bias
    assert _rel(y, ref) < 1.5e-2


@pytest.mark.parametrize("mode", ["fp8", "int4"])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128, 129])
@pytest.mark.parametrize("N,K", [(128, 128), (200, 384), (4096, 4224), (1000, 3968)])
def test_dequant_gemm_tiles(mode, M, N, K):
    """Edges of the row tiles (16 / 32 / 64 / 128), ragged N, one and odd numbers of 128-wide k-blocks (an int4 stage holds two), K split
    over clusters. Products of bf16 inputs with unscaled weight values are exact and summed in 32 bits, so against 64 bits only the
    rounding of the bf16 output remains (8 significant bits: at most 2^-8 relative), plus 2^-20 of the sum of magnitudes for the 32-bit
    sums."""
    torch.manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    if mode == "fp8":
        q, s = quant.quant_fp8_128x128(w)
        wd = q.double() * s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
        q = q.view(torch.uint8)
    else:
        q, s = quant.quant_int4(w)
        wd = torch.stack([q & 15, q >> 4], -1).view(N, K).double() - 8
        wd = wd * s.double().repeat_interleave(128, 1)
    bias = torch.randn(N, device="cuda")
    y = quant.gemm_dequant(x, q, s, mode, bias)
    ops.check_status()
    ref = x.double() @ wd.t() + bias.double()
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ wd.abs().t() + bias.abs().double()) * 2.0 ** -20
    assert bool(((y.double() - ref).abs() <= bound).all())


def _dequant_case(mode, M, N, K, bias=True):
    torch.manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    if mode == "fp8":
        q, s = quant.quant_fp8_128x128(w)
        wd = q.double() * s.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
        q = q.view(torch.uint8)
    else:
        q, s = quant.quant_int4(w)
        wd = (torch.stack([q & 15, q >> 4], -1).view(N, K).double() - 8) * s.double().repeat_interleave(128, 1)
    return x, q, s, wd, torch.randn(N, device="cuda") if bias else None


@pytest.mark.parametrize("mode", ["fp8", "int4"])
@pytest.mark.parametrize("M,N,K,bias", [(148 * 128, 128, 128, True), (149 * 128, 128, 128, False), (19073, 128, 128, True), (2049, 1200, 128, True),
                                        (5000, 1000, 256, True), (38017, 130, 256, False), (4096, 4104, 256, True)])
def test_dequant_gemm_of_many_short_tiles(mode, M, N, K, bias):
    """K of 128 and 256 with up to and more than one wave of tiles: the last rows and columns of ragged tiles, odd numbers of tiles a CTA. The bound is
    that of test_dequant_gemm_tiles; rows in common with a call of few rows agree with it as far as two such results can."""
    x, q, s, wd, b = _dequant_case(mode, M, N, K, bias)
    y = quant.gemm_dequant(x, q, s, mode, b)
    ops.check_status()
    for r in (slice(0, 1024), slice(M - 700, M)):
        ref = x[r].double() @ wd.t() + (b.double() if bias else 0.0)
        mag = x[r].double().abs() @ wd.abs().t() + (b.abs().double() if bias else 0.0)
        assert bool(((y[r].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * 2.0 ** -20).all())
    few = quant.gemm_dequant(x[M - 100:].contiguous(), q, s, mode, b)
    assert bool(((y[M - 100:].double() - few.double()).abs() <= few.double().abs() * 2.0 ** -7 + mag[-100:] * 2.0 ** -19).all())


@pytest.mark.parametrize("mode,M,N,K", [("int4", 16, 28672, 4096), ("int4", 32, 4096, 14336), ("int4", 1, 3584, 18944), ("int4", 128, 6144, 4096),
                                        ("fp8", 16, 4096, 14336), ("fp8", 32, 6144, 4096), ("fp8", 100, 4096, 4096)])
def test_dequant_gemm_repeats_itself(mode, M, N, K):
    """Converters, MMA and promotion warps run ahead of one another by up to the buffers between them, how far depends on what the memory does: calls
    on cold weights, one behind the other, give the same bits each time, and those of the dequantised product (one rounding of 32-bit sums)."""
    x, q, s, wd, _ = _dequant_case(mode, M, N, K, False)
    want = (x.double() @ wd.double().t())
    ws = [(q.clone(), s.clone()) for _ in range(max(2, (200 << 20) // q.numel()))]
    ys = [quant.gemm_dequant(x, *w, mode) for _ in range(3) for w in ws]
    ops.check_status()
    assert (ys[0].double() - want).norm() < 2.0 ** -8 * want.norm()
    assert all(torch.equal(y, ys[0]) for y in ys)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 128), (4, 4, 64)])
@pytest.mark.parametrize("d", [512, 4096, 8704])
def test_kernels_that_start_early_keep_the_order_of_the_stream(d, Hq, Hkv, D):
    """The kernels of a decode step wait for their predecessors inside. Layers of one after the other over the same buffers, for inputs that change,
    give the bits that the same calls give when each is waited for, launched one by one and as a graph: norms of short, ordinary and long rows,
    products of bf16 and int4 weights that are fetched early, KV append, both decode kernels (head size 64: not on tensor cores), their merge, SwiGLU."""
    from sneppx_alg_b200.ops import _lib
    from sneppx_alg_b200.ops._lib import c_float, c_int, c_ll, ptr, stream
    from sneppx_alg_b200.ops.gemm import gemm, static_weights
    torch.manual_seed(d + D)
    B, L, F, bs, n, rounds = 16, 3, 1024, 16, 700, 4
    wide = (Hq + 2 * Hkv) * D
    rand = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    weights = [dict(n1=rand(d), n2=rand(d), qkv=rand(wide, d) * d ** -0.5, o=rand(d, Hq * D) * (Hq * D) ** -0.5, gu=quant.quant_int4(rand(2 * F, d) * d ** -0.5),
                    down=rand(d, F) * F ** -0.5) for _ in range(L)]
    blocks = (n + rounds) // bs + 1
    table = torch.randperm(B * blocks, device="cuda").view(B, blocks).int()
    caches0 = rand(L, 2, B * blocks, bs, Hkv, D)
    cos, sin = rope_tables(1024, D, 1e4, "cuda")
    pos = [torch.full((B,), n + t, dtype=torch.int32, device="cuda") for t in range(rounds)]
    lens = [p + 1 for p in pos]
    slots = [table[:, (n + t) // bs] * bs + (n + t) % bs for t in range(rounds)]
    xs = [rand(B, d) for _ in range(rounds)]
    hn, out, o, qkv, h = rand(B, d), rand(B, d), rand(B, d), rand(B, wide), rand(B, F)
    res = [rand(B, d), rand(B, d)]
    kept, caches = torch.zeros(rounds, 2, B, d, device="cuda").bfloat16(), caches0.clone()

    def run(done):
        def norm(x, r_in, w, r_out):
            _lib.call("sx_rmsnorm_fwd", ptr(x), ptr(r_in), ptr(w), ptr(hn), ptr(r_out), ptr(None), c_ll(B), c_int(d), c_float(1e-5), stream())
            done()
        with static_weights():
            for t in range(rounds):
                out.copy_(xs[t])
                res[0].zero_()
                for w, (kc, vc) in zip(weights, caches):
                    norm(out, res[0], w["n1"], res[1])
                    gemm(hn, w["qkv"], out=qkv)
                    done()
                    paged.kv_append_(qkv, cos, sin, pos[t], slots[t], kc, vc, Hq, Hkv, D)
                    done()
                    a = paged.paged_decode(qkv[:, :Hq * D].view(B, Hq, D), kc, vc, table, lens[t])
                    done()
                    gemm(a.view(B, -1), w["o"], out=o)
                    done()
                    norm(o, res[1], w["n2"], res[0])
                    gu = quant.gemm_dequant(hn, *w["gu"], "int4")
                    done()
                    _lib.call("sx_glu_fwd", ptr(gu), ptr(h), c_ll(B), c_int(F), c_int(0), stream())
                    done()
                    gemm(h, w["down"], out=out)
                    done()
                kept[t, 0].copy_(out)
                kept[t, 1].copy_(res[0])

    def result():
        torch.cuda.synchronize()
        ops.check_status()
        both = kept.clone(), caches.clone()
        kept.zero_()
        caches.copy_(caches0)
        return both

    run(torch.cuda.synchronize)
    want = result()
    assert bool(want[0].isfinite().all())
    for _ in range(3):
        run(lambda: None)
        assert all(torch.equal(a, e) for a, e in zip(result(), want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(lambda: None)
    result()
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(a, e) for a, e in zip(result(), want))


def test_dequant_gemm_of_short_rows_keeps_up_with_its_output():
    """16384 x 4096 outputs of K = 128 are bound by writing 134 MB: two to four times a copy's time, ten when every tile was a CTA of its own."""
    x, q, s, _, _ = _dequant_case("int4", 16384, 4096, 128, False)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    big = torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
    times = []
    for fn in (lambda: quant.gemm_dequant(x, q, s, "int4"), lambda: big[:256 << 20].copy_(big[256 << 20:])):
        ts = []
        for _ in range(9):
            torch.cuda._sleep(400000)
            a.record()
            fn()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b) * 1e3)
        times.append(sorted(ts)[4])
    assert times[0] < 6 * times[1] * (16384 * 4096 * 2 + x.numel() * 2) / (512 << 20), times


@pytest.mark.parametrize("mode", ["fp8", "int4"])
def test_dequant_gemm_of_more_rows_than_a_grid_has_tiles(mode):
    """65535 tiles of 128 rows are one launch; the rows behind them come from a second one."""
    M, N, K = 65535 * 128 + 77, 8, 384
    x, q, s, wd, b = _dequant_case(mode, 256, N, K)
    big = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    big[:128], big[-128:] = x[:128], x[128:]
    y = quant.gemm_dequant(big, q, s, mode, b)
    ops.check_status()
    ref = x.double() @ wd.t() + b.double()
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ wd.abs().t() + b.abs().double()) * 2.0 ** -20
    assert bool(((torch.cat([y[:128], y[-128:]]).double() - ref).abs() <= bound).all())
    assert torch.equal(y[128:-128], b.bfloat16().expand(M - 256, N))


def test_paged_engine_matches_cached_generation_gpu():
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.serving.generation import generate
    from sneppx_alg_b200.serving.llm_engine import LLMEngine, SamplingParams
    torch.manual_seed(0)
    cfg = ModelConfig(hidden_size=256, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                      intermediate_size=512, vocab_size=512, max_position_embeddings=512, rms_norm_eps=1e-5)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda").eval()
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (37, 130, 64, 5)]
    eng = LLMEngine(model, num_blocks=256, block_size=16, max_batch_size=4)
    outs = eng.generate(prompts, SamplingParams(max_new_tokens=12))
    ops.check_status()
    agree = 0
    for p, o in zip(prompts, outs):
        ref = generate(model, torch.tensor([p], device="cuda"), max_new_tokens=12)[0, len(p):].tolist()
        agree += sum(int(a == b) for a, b in zip(o, ref))
        assert o[0] == ref[0]            # first token comes from the same prefill math
    assert agree >= 0.7 * 12 * len(prompts)   # bf16 paths differ in reduction order; most greedy tokens coincide
    # weight-only fp8 serving runs end to end
    quant.quantize_model_(model, "fp8")
    eng2 = LLMEngine(model, num_blocks=256, block_size=16)
    assert len(eng2.generate(prompts[:2], SamplingParams(max_new_tokens=4))[0]) == 4
    ops.check_status()


@pytest.mark.parametrize("hidden,headdim,state,groups,taps,layers,batch", [
    (256, 64, 128, 1, 4, 3, 5), (320, 64, 128, 2, 4, 2, 1), (128, 32, 64, 4, 2, 1, 17), (192, 24, 40, 2, 3, 2, 3), (256, 128, 256, 1, 4, 2, 128),
    (128, 16, 136, 16, 4, 2, 2), (64, 72, 8, 1, 2, 2, 4)])
def test_mamba2_decode_step(hidden, headdim, state, groups, taps, layers, batch):
    """The in-place decode step against the same weights in 32 bits on the CPU: logits and states over steps with a changing batch, state
    rows and columns that do not fill a warp, two to four taps. A handed-out state is not written by later steps, a sequence twice in a
    batch goes through the model's forward. Bound: every activation of a layer is rounded to bf16 (2^-9) about eight times, errors of the
    layers add up; measured 0.003 to 0.012."""
    import copy
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.serving.llm_engine import StatefulRunner
    from sneppx_alg_b200.serving.mamba_states import _Block
    torch.manual_seed(hidden + state)
    inner = 9 * 72 if headdim == 72 else 2 * hidden
    cfg = ModelConfig(architecture="mamba2", hidden_size=hidden if headdim != 72 else 324 * 2, num_hidden_layers=layers, vocab_size=1000,
                      ssm_state_size=state, ssm_expand=2 if headdim != 72 else 1, ssm_head_dim=headdim, ssm_ngroups=groups,
                      ssm_conv_kernel=taps, rms_norm_eps=1e-5, tie_word_embeddings=True)
    assert inner % headdim == 0
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda").eval()
    with torch.no_grad():
        for n, p in model.named_parameters():
            if "conv_bias" in n or n.endswith(".D"):
                p.copy_(torch.randn_like(p.float()))
    plain = copy.deepcopy(model).float().cpu()
    run, ref = StatefulRunner(model), StatefulRunner(plain)
    g = torch.Generator().manual_seed(1)
    for sid in range(batch):
        # the same states on both sides
        st = [{"conv": torch.randn(1, taps - 1, plain.layers[0].mixer.conv_dim, generator=g).bfloat16(),
               "ssm": 0.3 * torch.randn(1, plain.layers[0].mixer.nheads, headdim, state, generator=g)} for _ in range(layers)]
        run.states[sid] = [{k: v.cuda() for k, v in d.items()} for d in st]
        ref.states[sid] = [{k: v.float() for k, v in d.items()} for d in st]

    def close(a, b):
        return (a.cpu().float() - b).norm().item() <= 0.03 * b.norm().item()

    kept = None
    for step in range(4):
        ids = list(range(batch)) if step != 1 else list(range(batch - 1, -1, -2))
        tokens = [(37 * step + 11 * i) % 1000 for i in ids]
        a, b = run.decode(ids, tokens), ref.decode(ids, tokens)
        ops.check_status()
        assert a.shape == (len(ids), 1000) and a.dtype == torch.float32 and close(a, b)
        assert all(isinstance(run.states.entry(i), _Block) for i in ids)
        if step == 1:
            kept = run.states[ids[0]]
            before = [{k: v.clone() for k, v in d.items()} for d in kept]
    for sid in range(batch):
        for x, y in zip(run.states[sid], ref.states[sid]):
            assert close(x["ssm"], y["ssm"]) and close(x["conv"], y["conv"])
    assert all(torch.equal(x[k], y[k]) for x, y in zip(kept, before) for k in x)
    a, b = run.decode([0, 0], [3, 3]), ref.decode([0, 0], [3, 3])
    assert close(a, b) and isinstance(run.states.entry(0), list)


@pytest.mark.parametrize("T,Hq,Hkv,D,rotate", [(1, 4, 1, 128, True), (37, 28, 4, 128, True), (9, 40, 8, 256, True), (50, 6, 2, 16, True),
                                               (50, 6, 2, 24, True), (33, 8, 8, 64, False), (149, 12, 2, 128, True), (131, 1, 1, 16, True),
                                               (160, 32, 32, 128, True), (9, 40, 8, 256, False)])
def test_kv_append_sizes(T, Hq, Hkv, D, rotate):
    """16-byte form (tokens that share a CTA, one CTA or several a token) and the form for head sizes that are no multiple of 16; rows without a slot
    are rotated and written nowhere. Products and sums are 32-bit: one bf16 rounding, 2^-8; copies are exact."""
    torch.manual_seed(T)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda", dtype=torch.bfloat16)
    kc = torch.randn(T // 4 + 2, 4, Hkv, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.randn_like(kc)
    cos, sin = rope_tables(256, D, 1e4, "cuda")
    pos = torch.randint(0, 256, (T,), device="cuda", dtype=torch.int32)
    slot = torch.randperm(T, device="cuda").int() + 3
    slot[::5] = -1
    want = [t.double() for t in (qkv, kc, vc)]
    paged.kv_append_reference(want[0], cos.double(), sin.double(), pos, slot, want[1], want[2], Hq, Hkv, D, rotate)
    paged.kv_append_(qkv, cos, sin, pos, slot, kc, vc, Hq, Hkv, D, rotate)
    for got, ref in zip((qkv, kc, vc), want):
        assert bool(((got.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all())
    assert torch.equal(vc.double(), want[2])


def test_mamba2_decode_step_that_fails(monkeypatch):
    """A launch that fails in the second layer: a sequence whose states were stepped where they lie is dropped, so that a retry fails instead of
    going on from half-advanced states; one whose states came as lists keeps them and steps as if nothing had happened."""
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.ops import _lib
    from sneppx_alg_b200.serving.llm_engine import StatefulRunner
    torch.manual_seed(0)
    cfg = ModelConfig(architecture="mamba2", hidden_size=256, num_hidden_layers=3, vocab_size=500, ssm_state_size=128, ssm_expand=2, ssm_head_dim=64,
                      ssm_ngroups=1, ssm_conv_kernel=4, rms_norm_eps=1e-5, tie_word_embeddings=True)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda").eval()
    run, other = StatefulRunner(model), StatefulRunner(model)
    for r in (run, other):
        for sid in (0, 1, 2):
            r.prefill(sid, [3 + sid, 5, 7], 0)
        r.decode([0, 2], [9, 9])
    real, calls = _lib.call, []

    def failing(name, *args):
        calls.append(name)
        if calls.count("sx_mamba2_step") == 2:
            raise RuntimeError("no launch")
        real(name, *args)

    monkeypatch.setattr(_lib, "call", failing)
    with pytest.raises(RuntimeError, match="no launch"):
        run.decode([0, 1], [11, 12])
    monkeypatch.setattr(_lib, "call", real)
    with pytest.raises(KeyError):
        run.decode([0, 1], [11, 12])
    assert sorted(run.states.keys()) == [1, 2]
    assert torch.equal(run.decode([1, 2], [12, 13]), other.decode([1, 2], [12, 13]))
    assert torch.equal(run.decode([1, 2], [14, 15]), other.decode([1, 2], [14, 15]))
    ops.check_status()


@pytest.mark.parametrize("mode", ["fp8", "int4"])
@pytest.mark.parametrize("M", [1, 17, 64, 128])
@pytest.mark.parametrize("N,K", [(128, 128), (128, 640), (200, 384), (4096, 4224), (1000, 3968)])
def test_dequant_gemm_with_static_weights(mode, M, N, K):
    """Weights and scales read ahead of the kernel that makes X, which lets its dependents start early: the same values as without, over several
    calls in a row; rings of stages that hold all of a CTA's slice and more, slices of K that are empty."""
    from sneppx_alg_b200.ops import functional as F_
    from sneppx_alg_b200.ops.gemm import static_weights
    x, q, s, wd, b = _dequant_case(mode, M, N, K)
    w = torch.ones(K, device="cuda", dtype=torch.bfloat16)
    want, rows = [], [x * (1 + i) for i in range(4)]
    for r in rows:
        h, _ = F_.rmsnorm(r, w)
        want.append((h, quant.gemm_dequant(h, q, s, mode, b)))
    got = []
    with static_weights():
        for r in rows:
            h, _ = F_.rmsnorm(r, w)
            got.append((h, quant.gemm_dequant(h, q, s, mode, b)))
    ops.check_status()
    for (h, y), (hw, yw) in zip(got, want):
        assert torch.equal(h, hw) and torch.equal(y, yw)
    ref = want[0][0].double() @ wd.t() + b.double()
    mag = want[0][0].double().abs() @ wd.abs().t() + b.abs().double()
    assert bool(((want[0][1].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * 2.0 ** -20).all())


def test_captured_decode_with_changing_batches():
    """Rows of the captured step's block table are written when a table changes: sequences that swap rows, leave, come back shorter and grow over
    blocks give the logits of the same steps without capture."""
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.serving.kv_cache import PagedKVCache
    from sneppx_alg_b200.serving.llm_engine import LlamaPagedRunner
    torch.manual_seed(4)
    cfg = ModelConfig(hidden_size=512, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=128, intermediate_size=512,
                      vocab_size=300, max_position_embeddings=256, rms_norm_eps=1e-5)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda").eval()
    runners = []
    for graphs in (True, False):
        cache = PagedKVCache(2, 80, 8, 2, 128, device="cuda", enable_prefix_cache=False)
        runners.append(LlamaPagedRunner(model, cache))
        if graphs:
            runners[0].enable_graphs(6, 128)

    def start(sid, n):
        for r in runners:
            r.cache.add_sequence(sid)
            r.prefill(sid, [(7 * sid + 3 * i) % 300 for i in range(n)], 0)

    def stop(sid):
        for r in runners:
            r.cache.free_sequence(sid)

    def steps(ids, n):
        for t in range(n):
            a, b = (r.decode(ids, [(11 * s + 5 * t) % 300 for s in ids]) for r in runners)
            assert a.shape == b.shape and _rel(a, b) < 2e-2, (ids, t)

    for sid, n in enumerate((5, 40, 17, 63, 8)):
        start(sid, n)
    steps([0, 1, 2, 3], 9)
    steps([3, 0], 10)                 # fewer rows: another captured step
    steps([2, 1, 0, 3, 4], 3)         # more of them, in other rows
    stop(1)
    start(1, 2)                       # a shorter table, of blocks that others have held, in a row that held a longer one
    steps([2, 1, 0, 3, 4], 9)
    stop(3)
    start(5, 30)
    for r in runners:                 # two sequences with one table, then one of them copies its last block
        r.cache.fork(5, 6)
    steps([5, 6, 1, 0], 9)
    steps([6, 5, 2, 1, 0, 4], 4)
    ops.check_status()
