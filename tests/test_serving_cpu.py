"""Paged continuous-batching engine against plain cached generation (CPU, fp32): same greedy tokens, prefix cache
hits, copy-on-write, sampling utilities."""
import torch

from sneppx_alg_b200.models import ModelConfig, build_model
from sneppx_alg_b200.serving.generation import (apply_repetition_penalty, batch_generate, generate,
                                               top_k_top_p_filtering)
from sneppx_alg_b200.serving.kv_cache import KVBlockPool, PagedKVCache
from sneppx_alg_b200.serving.llm_engine import LLMEngine, SamplingParams


def _model():
    torch.manual_seed(0)
    cfg = ModelConfig(hidden_size=64, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                      intermediate_size=128, vocab_size=97, max_position_embeddings=128, rms_norm_eps=1e-5)
    return build_model(cfg).eval()


def test_engine_matches_cached_generation_and_reuses_prefix():
    model = _model()
    g = torch.Generator().manual_seed(1)
    shared = torch.randint(0, 97, (20,), generator=g).tolist()
    prompts = [shared + torch.randint(0, 97, (n,), generator=g).tolist() for n in (3, 9, 5)]
    ref = [generate(model, torch.tensor([p]), max_new_tokens=8)[0, len(p):].tolist() for p in prompts]
    eng = LLMEngine(model, num_blocks=64, block_size=4, max_batch_size=2)
    outs = eng.generate(prompts, SamplingParams(max_new_tokens=8))
    assert outs == ref
    assert eng.cache.pool.num_free + len(eng.cache.prefix.table) == 64      # everything returned except cached blocks
    # a second wave with the same prefix is served from the prefix cache and still matches
    outs2 = eng.generate(prompts[:1], SamplingParams(max_new_tokens=8))
    assert outs2[0] == ref[0] and eng.stats["cached_prefix_tokens"] >= 20


def test_block_pool_refcount_and_cow():
    pool = KVBlockPool(4)
    a = pool.allocate()
    pool.share(a)
    pool.release(a)
    assert pool.num_free == 3
    pool.release(a)
    assert pool.num_free == 4
    cache = PagedKVCache(1, 8, 2, 1, 4, dtype=torch.float32, device="cpu", enable_prefix_cache=False)
    cache.add_sequence(0)
    cache.reserve(0, 3)
    cache.k[0][cache.tables[0][1]].fill_(7.0)
    cache.fork(0, 1)
    slots = cache.reserve(1, 1)            # writes into the shared, half-full block -> copy
    assert cache.tables[1][1] != cache.tables[0][1]
    assert float(cache.k[0][cache.tables[1][1]][0, 0, 0]) == 7.0 and slots[0] == cache.tables[1][1] * 2 + 1


def test_sampling_filters():
    logits = torch.tensor([[1.0, 2.0, 3.0, 4.0]])
    f = top_k_top_p_filtering(logits.clone(), top_k=2)
    assert torch.isinf(f[0, :2]).all() and not torch.isinf(f[0, 2:]).any()
    f = top_k_top_p_filtering(logits.clone(), top_p=0.6)
    assert not torch.isinf(f[0, 3]) and torch.isinf(f[0, 0])
    p = apply_repetition_penalty(torch.tensor([[2.0, -2.0]]), torch.tensor([[0, 1]]), 2.0)
    assert p.tolist() == [[1.0, -4.0]]
    model = _model()
    outs = batch_generate(model, [torch.tensor([1, 2, 3]), torch.tensor([4, 5])], max_new_tokens=3)
    assert len(outs[0]) == 6 and len(outs[1]) == 5


def test_engine_serves_recurrent_state_models():
    """Mamba-2 through the continuous-batching engine: tokens equal the model's own greedy decoding from a full
    re-forward at every step, for requests of different lengths that join and leave the batch at different times."""
    import torch
    from sneppx_alg_b200.models import ModelConfig, build_model
    from sneppx_alg_b200.serving.llm_engine import LLMEngine, SamplingParams, StatefulRunner
    torch.manual_seed(0)
    cfg = ModelConfig(architecture="mamba2", hidden_size=32, num_hidden_layers=2, vocab_size=96, ssm_state_size=8,
                      ssm_conv_kernel=4, ssm_expand=2, ssm_head_dim=8, ssm_ngroups=1, ssm_chunk_size=8, rms_norm_eps=1e-5)
    model = build_model(cfg).eval()
    prompts = [[5, 9, 33, 2, 7], [11, 12], [70, 3, 3, 8, 1, 2, 90, 4, 6]]
    lens = [6, 3, 4]
    eng = LLMEngine(model, max_batch_size=2)   # two slots for three requests: the third joins when one finishes
    assert isinstance(eng.runner, StatefulRunner)
    ids = [eng.submit(p, SamplingParams(max_new_tokens=n)) for p, n in zip(prompts, lens)]
    eng.run_until_done()
    for rid, p, n in zip(ids, prompts, lens):
        seq = list(p)
        with torch.no_grad():
            for _ in range(n):
                seq.append(int(model(torch.tensor([seq]))["logits"][0, -1].argmax()))
        assert eng.finished[rid].output == seq[len(p):]
    assert eng.runner.states == {} and eng.cache.pool.num_free == 2


def test_same_length_prompts_share_one_prefill_pass():
    """Waiting requests whose prompts have the same length are prefilled as one batch (one pass over the weights);
    the tokens are those of one-by-one generation, the prompt of another length still goes alone, and the batch
    respects the token budget."""
    model = _model()
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 97, (12,), generator=g).tolist() for _ in range(5)] + [torch.randint(0, 97, (7,), generator=g).tolist()] + \
              [torch.randint(0, 97, (12,), generator=g).tolist() for _ in range(2)]
    ref = [generate(model, torch.tensor([p]), max_new_tokens=6)[0, len(p):].tolist() for p in prompts]
    eng = LLMEngine(model, num_blocks=128, block_size=4, max_batch_size=8, max_prefill_tokens=40, enable_prefix_cache=False)
    calls = []
    orig = eng.runner.prefill_batch
    eng.runner.prefill_batch = lambda ids, ps: (calls.append(len(ps)), orig(ids, ps))[1]
    out = eng.generate(prompts, SamplingParams(max_new_tokens=6))
    assert out == ref
    assert calls and calls[0] == 3                     # 40-token budget: three 12-token prompts per pass
    assert eng.stats["prefill_tokens"] == sum(len(p) for p in prompts)
    assert not eng.cache.tables and eng.cache.pool.free_count() == 128 if hasattr(eng.cache.pool, "free_count") else True


def test_tensor_parallel_engine_matches_single_rank_tokens():
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, os.path.join(here, "mp_tp_serving_check.py"), "2", str(29820 + os.getpid() % 9)],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "TP_SERVING_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


def test_tensor_parallel_serving_over_http_matches_single_rank_tokens():
    """Rank 0 serves POST /v1/generate, rank 1 mirrors it (requests broadcast once per engine step)."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, os.path.join(here, "mp_tp_http_check.py"), "2", str(29840 + os.getpid() % 9)],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "TP_HTTP_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


def test_prefix_cache_gives_blocks_back_under_pressure():
    """A pool mostly pinned by cached prefixes must still admit new requests (entries nobody shares are evicted,
    least recently used first), never run dry in the middle of a generation, and fail a request that can never
    fit instead of spinning."""
    model = _model()
    g = torch.Generator().manual_seed(3)
    eng = LLMEngine(model, num_blocks=24, block_size=4, max_batch_size=4)
    assert eng.cache.prefix.max_entries <= 12          # capped at a fraction of the pool
    ref_prompts = [torch.randint(0, 97, (17 + i,), generator=g).tolist() for i in range(8)]
    refs = [generate(model, torch.tensor([p]), max_new_tokens=6)[0, len(p):].tolist() for p in ref_prompts]
    # eight different prompts of ~6 blocks each through a 24-block pool: the cache fills, then has to yield
    outs = eng.generate(ref_prompts, SamplingParams(max_new_tokens=6))
    assert outs == refs
    assert not eng.failed
    assert eng.cache.pool.num_free + len(eng.cache.prefix.table) == 24
    # a request larger than the whole pool is rejected at once; the engine goes idle instead of looping
    rid = eng.submit(list(range(90)) + [1] * 30, SamplingParams(max_new_tokens=8))
    done = eng.run_until_done(max_steps=50)
    assert rid in eng.failed and rid in done and not eng.has_work()
    # and the engine still serves afterwards
    assert eng.generate(ref_prompts[:1], SamplingParams(max_new_tokens=6))[0] == refs[0]


def test_recurrent_states_leave_their_block_when_read():
    """Every way of reading a sequence's states gives the ordinary per-layer dicts with the values of the buffer that is current, and
    the sequence keeps what was handed out."""
    import copy
    import pickle
    import torch
    from sneppx_alg_b200.serving.mamba_states import SequenceStates, _Block

    def fresh():
        s, b = SequenceStates(), _Block(torch.arange(2 * 3 * 4 * 8.).view(2, 3, 4, 8), torch.arange(2 * 2 * 3 * 5.).view(2, 2, 3, 5))
        b.cur = 1
        dict.__setitem__(s, 7, b)
        s[8] = [{"conv": None, "ssm": None}]
        return s, b

    reads = [lambda s: s[7], lambda s: s.get(7), lambda s: list(s.values())[0], lambda s: dict(s.items())[7], lambda s: dict(s)[7],
             lambda s: {**s}[7], lambda s: s.copy()[7], lambda s: (s | {})[7], lambda s: copy.copy(s)[7],
             lambda s: pickle.loads(pickle.dumps(s))[7], lambda s: s.setdefault(7), lambda s: s.pop(7)]
    for read in reads:
        s, b = fresh()
        got = read(s)
        assert type(got) is list and len(got) == 2
        for i, layer in enumerate(got):
            assert torch.equal(layer["ssm"], b.ssm[i:i + 1]) and torch.equal(layer["conv"], b.conv[1, i:i + 1])
        assert not any(isinstance(s.entry(k), _Block) for k in s.keys())
    s, b = fresh()
    assert s.entry(7) is b and 7 in s and len(s) == 2 and s.get(9) is None
    assert s != {} and SequenceStates() == {}


def test_paged_decode_deals_its_items_evenly():
    """The decode kernel's CTAs take items c, c + n, ...: every (sequence, KV head, split) exactly once, and with few items a CTA none gets more
    tiles of equal sequences than when the long items are dealt first."""
    import ctypes as C
    from sneppx_alg_b200 import _build
    lib, n_cta = _build.load_cuda(), 148
    for B, Hkv, n in ((16, 4, 1000), (16, 8, 1000), (16, 2, 4000), (128, 2, 4000), (48, 8, 4000), (3, 1, 200), (1, 1, 1), (128, 32, 1000)):
        max_len = (n // 16 + 1) * 16
        ns = lib.sx_paged_decode_tc_splits(C.c_int(max_len), C.c_int(B * Hkv))
        tiles = (n + 127) // 128
        per = -(-tiles // ns)
        count = [max(0, min(tiles, (s + 1) * per) - s * per) for s in range(ns)]
        b, hk, s = C.c_int(), C.c_int(), C.c_int()
        seen, load = set(), [0] * n_cta
        for i in range(B * Hkv * ns):
            lib.sx_paged_decode_tc_item(i, B, Hkv, ns, n_cta, C.byref(b), C.byref(hk), C.byref(s))
            seen.add((b.value, hk.value, s.value))
            load[i % n_cta] += count[s.value]
        assert seen == {(i, j, k) for i in range(B) for j in range(Hkv) for k in range(ns)}
        best, longest = [0] * n_cta, sorted(count, reverse=True)
        for i in range(B * Hkv * ns):
            best[i % n_cta] += longest[i // (B * Hkv)]
        assert max(load) == max(best) or B * Hkv * ns > 7 * n_cta, (B, Hkv, n, max(load), max(best))


def test_prompts_are_uploaded_as_torch_tensor_takes_them():
    """Lists of integers take a shorter way; everything else is what torch.tensor makes of it, refusals included, and arrays and tensors are
    converted at once."""
    import numpy as np
    import pytest
    from sneppx_alg_b200.serving.llm_engine import LlamaPagedRunner, _upload
    dev = torch.device("cpu")
    for values in ([], [3, 1, 2], [True, False], [1.0, 2.0], (4, 5), np.arange(6), np.arange(6, dtype=np.uint8), torch.arange(4), [np.int64(3), 4],
                   [torch.tensor(7), 8], [[1, 2], [3, 4]], np.ones((2, 3), dtype=np.int32)):
        for dtype in (torch.long, torch.int32):
            want, got = torch.tensor(values, dtype=dtype), _upload(values, dtype, dev)
            assert got.dtype == dtype and torch.equal(got, want), values
    for values in ([2 ** 70], [None], ["a"], [torch.arange(3), torch.arange(3)]):
        with pytest.raises(Exception) as ours:
            _upload(values, torch.long, dev)
        with pytest.raises(type(ours.value)):
            torch.tensor(values, dtype=torch.long)

    class Counted(np.ndarray):
        def __iter__(self):
            raise AssertionError("walked one value after another")

    assert _upload(np.arange(5).view(Counted), torch.long, dev).tolist() == [0, 1, 2, 3, 4]
    model, prompts = _model(), [[5, 6, 7, 8, 9], [10, 11, 12, 13, 14]]
    outs = []
    for form in (prompts, np.array(prompts), torch.tensor(prompts), [tuple(p) for p in prompts]):
        cache = PagedKVCache(2, 16, 4, 2, 16, dtype=torch.float32, device="cpu")
        runner = LlamaPagedRunner(model, cache)
        for sid in (0, 1, 2):
            cache.add_sequence(sid)
        outs.append(torch.cat([runner.prefill_batch([0, 1], form), runner.prefill(2, form[0], 0)]))
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_slots_by_block_and_tables_shared_whole():
    """Slots reserved by block against one token at a time, over full, partly filled and shared blocks and an exhausted pool; tables shared and
    released whole against block by block."""
    import random
    import pytest

    class Plain(PagedKVCache):
        def reserve(self, seq_id, n_new):
            table, slots = self.tables[seq_id], []
            for i in range(self.lens[seq_id], self.lens[seq_id] + n_new):
                at, off = divmod(i, self.block_size)
                if at == len(table):
                    table.append(self.pool.allocate())
                elif self.pool.ref[table[at]] > 1:
                    new = self.pool.allocate()
                    self.k[0][new], self.v[0][new] = self.k[0][table[at]].clone(), self.v[0][table[at]].clone()
                    self.pool.release(table[at])
                    table[at] = new
                slots.append(table[at] * self.block_size + off)
            self.lens[seq_id] += n_new
            return slots

        def fork(self, src, dst):
            self.tables[dst] = [self.pool.share(b) for b in self.tables[src]]
            self.lens[dst] = self.lens[src]

        def free_sequence(self, seq_id, tokens=None):
            for b in self.tables.pop(seq_id, []):
                self.pool.release(b)
            self.lens.pop(seq_id, 0)

    rng = random.Random(5)
    for trial in range(20):
        pair = [cls(1, 24, 4, 1, 8, dtype=torch.float32, device="cpu", enable_prefix_cache=False) for cls in (PagedKVCache, Plain)]
        live, nxt = [], 0
        for _ in range(40):
            act = rng.random()
            if act < 0.3 or not live:
                for c in pair:
                    c.add_sequence(nxt)
                live.append(nxt)
                nxt += 1
            elif act < 0.7:
                sid, n = rng.choice(live), rng.choice([0, 1, 3, 4, 5, 9])
                got = []
                for c in pair:
                    try:
                        got.append(c.reserve(sid, n))
                    except MemoryError:
                        got.append("exhausted")
                assert got[0] == got[1]
                if got[0] == "exhausted":
                    break
                for layer, value in (("k", 1.0 + nxt), ("v", 2.0 + nxt)):
                    for c in pair:
                        getattr(c, layer)[0].view(24 * 4, -1)[got[0]] = value
            elif act < 0.85:
                src = rng.choice(live)
                for c in pair:
                    c.fork(src, nxt)
                live.append(nxt)
                nxt += 1
            else:
                sid = live.pop(rng.randrange(len(live)))
                for c in pair:
                    c.free_sequence(sid)
            a, b = pair
            assert a.tables == b.tables and a.lens == b.lens and a.pool.free == b.pool.free and a.pool.ref == b.pool.ref
            assert torch.equal(a.k[0], b.k[0]) and torch.equal(a.v[0], b.v[0])
    pool = KVBlockPool(3)
    blocks = [pool.allocate(), pool.allocate()]
    pool.release_all(pool.share_all(blocks))
    assert pool.num_free == 1
    pool.release_all(blocks)
    assert pool.num_free == 3 and pool.free[-2:] == blocks
    with pytest.raises(RuntimeError, match="double free"):
        pool.release_all(blocks)
