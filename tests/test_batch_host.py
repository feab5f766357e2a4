"""CPU: continuous-batching host logic and sampler / cache bookkeeping against
the reference's own function source (tests/golden/reference_golden.json, generated by
tests/golden/make_golden.py).  The scheduling tests drive `BatchGenerator` with a deterministic
stand-in for the engine (same call surface as mlx_vlm_b200.engine.Engine), so that
time-multiplexing the batch-1 engine over rows is checked against running each row alone."""
import json
import os
import types

import numpy as np
import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
with open(os.path.join(HERE, "golden", "reference_golden.json")) as f:
    GOLD = json.load(f)


# --------------------------------------------------------------------------- goldens
def _filled(n, base):
    from mlx_vlm_b200.models.cache import KVCache
    c = KVCache()
    if n:
        kk = (base + torch.arange(n, dtype=torch.float32)).reshape(1, 1, n, 1) * torch.ones(1, 2, 1, 2)
        c.update_and_fetch(kk, -kk)
    return c


def _check(c, g):
    assert c.left_padding.tolist() == g["left_padding"], g["op"]
    assert c.offset.tolist() == g["offset"], g["op"]
    assert c._idx == g["idx"], g["op"]
    if g["keys"] is None:
        assert c.keys is None
    else:
        assert np.array_equal(c.keys[..., :c._idx, :].numpy(), np.asarray(g["keys"], dtype=np.float32)), g["op"]
        assert np.array_equal(c.values[..., :c._idx, :].numpy(), np.asarray(g["values"], dtype=np.float32)), g["op"]


def test_batch_kv_cache_matches_reference_trace():
    """reference cache.py:972-1201 (merge / append / extract / filter / extend / trim)."""
    from mlx_vlm_b200.models.cache import BatchKVCache, create_causal_mask
    t = GOLD["BatchKVCache_trace"]
    b = BatchKVCache.merge([_filled(5, 100), _filled(2, 200), _filled(7, 300)])
    _check(b, t[0])
    step = (900 + torch.arange(3, dtype=torch.float32)).reshape(3, 1, 1, 1) * torch.ones(1, 2, 1, 2)
    b.update_and_fetch(step, -step)
    _check(b, t[1])
    ex = b.extract(1)
    assert ex.offset == t[2]["offset"]
    assert np.array_equal(ex.keys[..., :ex.offset, :].numpy(), np.asarray(t[2]["keys"], dtype=np.float32))
    b.filter([0, 1])
    _check(b, t[3])
    b.extend(BatchKVCache.merge([_filled(3, 400)]))
    _check(b, t[4])
    assert b.trim(2) == 2
    _check(b, t[5])
    _check(BatchKVCache([1, 3, 0]), t[6])
    assert BatchKVCache([1, 3, 0]).batch_size == 3 and BatchKVCache([0]).is_single_row()
    for c in GOLD["causal_mask_left_padding"]:
        m = create_causal_mask(c["N"], c["offset"], left_padding=c["left_padding"]).int().numpy()
        assert m.tolist() == c["mask"]
    # right padding -> left padding (cache.py:1017-1033): rows rotate right by their padding
    r = BatchKVCache([0, 0])
    kk = torch.arange(8, dtype=torch.float32).reshape(2, 1, 4, 1)
    r.prepare(right_padding=[0, 2])
    r.update_and_fetch(kk, kk)
    r.finalize()
    assert r.left_padding.tolist() == [0, 2] and r.offset.tolist() == [4, 2]
    # (the roll is over the whole 256-step buffer, like the reference's dynamic_roll: the two
    # right-padding slots move out past the write index, zeros move in as left padding)
    assert r.keys[1, 0, :4, 0].tolist() == [0.0, 0.0, 4.0, 5.0] and r.keys[1, 0, 4:6, 0].tolist() == [6.0, 7.0]


def test_prompt_padding_matches_reference():
    from mlx_vlm_b200.generate_batch import _left_pad_prompts, _right_pad_prompts
    g = GOLD["pad_prompts"]
    assert _left_pad_prompts(g["prompts"]).tolist() == g["left"]
    assert _right_pad_prompts(g["prompts"]).tolist() == g["right"]
    assert _left_pad_prompts(g["prompts"], 6).tolist() == g["left_max6"]
    # known answers of the reference's own tests (tests/test_generate.py:478-527)
    assert _left_pad_prompts([[1, 2, 3], [4, 5], [6]]).tolist() == [[1, 2, 3], [0, 4, 5], [0, 0, 6]]
    assert _left_pad_prompts([[1, 2], [3]], max_length=5).tolist() == [[0, 0, 0, 1, 2], [0, 0, 0, 0, 3]]
    assert _left_pad_prompts([[1, 2, 3, 4, 5]]).shape == (1, 5)
    assert _left_pad_prompts([[1, 2], []]).tolist() == [[1, 2], [0, 0]]


def _arr(x):
    return torch.tensor(np.array([[float(v) for v in row] for row in x], dtype=np.float32))


def test_sampler_masks_match_reference_source():
    """sample_utils.py:149-345 executed over numpy vs our torch samplers: same survivors
    (-inf pattern), same surviving values."""
    from mlx_vlm_b200 import sample_utils as SU
    g = GOLD["sampler_masks"]
    lp, lg = _arr(g["logprobs"]), _arr(g["logits"])

    def same(a, want):
        w = _arr(want)
        assert torch.equal(torch.isinf(a), torch.isinf(w))
        fin = ~torch.isinf(w)
        assert torch.allclose(a[fin], w[fin], atol=1e-6)
    same(SU.apply_top_k(lp, 3), g["top_k_3"])
    same(SU.apply_top_p(lp, 0.7), g["top_p_0.7"])
    same(SU.apply_min_p(lp, 0.2), g["min_p_0.2"])
    same(SU.apply_min_p(lp, 0.6, 3), g["min_p_0.6_keep3"])
    same(SU.apply_top_n_sigma(lg, 1.0), g["top_n_sigma_1.0"])
    same(SU.apply_p_less(lg, 0.8), g["p_less_t0.8"])
    same(SU.apply_typical_p(lp, 0.6), g["typical_p_0.6"])
    with pytest.raises(ValueError):
        SU.apply_top_k(lp, 0)
    with pytest.raises(ValueError):
        SU.apply_min_p(lp, 1.5)


def test_stopping_criteria_and_prompt_cache_state():
    """utils.py:2191-2249; generate/common.py:243-263."""
    from mlx_vlm_b200.generate import PromptCacheState
    from mlx_vlm_b200.utils import StoppingCriteria
    tok = types.SimpleNamespace(eos_token_ids=[7], encode=lambda s, add_special_tokens=False: [1, 42])
    sc = StoppingCriteria([2, 3], tok, additional_eos_token_ids=[3, 9, 9])
    assert sc.eos_token_ids == [2, 3, 9] and sc(9) and not sc(4)
    sc.add_eos_token_ids(5)
    sc.add_eos_token_ids(["<end>"])
    assert sc(5) and sc(42)
    sc.reset()
    assert sc.eos_token_ids == [7, 3, 9]
    with pytest.raises(ValueError):
        StoppingCriteria([1]).add_eos_token_ids(3)
    st = PromptCacheState()
    assert st.find_prefix_length([1, 2, 3]) == 0
    st.update([1, 2, 3, 4], kv_cache=["c"])
    assert st.find_prefix_length([1, 2, 9]) == 2 and st.find_prefix_length([1, 2, 3, 4, 5]) == 4


# --------------------------------------------------------------------------- scheduling
V = 97


def _f(tok, ctx, pos):
    return (tok * 31 + ctx * 7 + pos * 3 + 1) % V


class _FakeCache:
    def __init__(self):
        self.offset = 0


class _FakeEngine:
    """Call surface of mlx_vlm_b200.engine.Engine used by BatchGenerator."""

    def __init__(self):
        self.log, self.tokens_launched = [], 0
        self.tok = self.ctx = self.pos = 0
        self.device = "cpu"
        self.stream = types.SimpleNamespace(synchronize=lambda: None)
        self.calls = []

    def set_next(self, tok, ctx, pos):
        self.tok, self.ctx, self.pos = tok, ctx, pos

    def emit(self, tok):
        self.log.append(tok)
        self.tokens_launched += 1

    def decode(self, n):
        for _ in range(n):
            self.tok = _f(self.tok, self.ctx, self.pos)
            self.ctx += 1
            self.pos += 1
            self.emit(self.tok)

    def fetch_tokens(self, start, n, host):
        host[:n] = torch.tensor(self.log[start:start + n], dtype=torch.int32)

    def snapshot(self, name):
        lp = torch.full((V,), -5.0)
        lp[self.log[-1]] = -0.25
        return lp


class _FakeLM:
    def __init__(self, eng):
        self.eng = eng
        self.layers = [0, 1]

    def make_cache(self):
        return [_FakeCache(), _FakeCache()]

    def __call__(self, ids, inputs_embeds=None, cache=None, position_ids=None, rope_deltas=None,
                 logits_to_keep=None, reserve_tokens=0, **kw):
        ids = np.asarray(ids)
        L = ids.shape[1]
        off = cache[0].offset
        delta = int(np.asarray(rope_deltas).reshape(-1)[0]) if rope_deltas is not None else 0
        self.eng.calls.append(("lm", L, off))
        if L == 1 and inputs_embeds is None:   # decode step through __call__
            self.eng.set_next(int(ids[0, 0]), off, off + delta)
            self.eng.decode(1)
        else:                                  # prefill: first token depends on the whole prompt
            first = (int(ids.sum()) * 13 + off + L) % V
            self.eng.set_next(first, off + L, off + L + delta)
            self.eng.emit(first)
        for c in cache:
            c.offset += L
        logits = torch.full((1, 1, V), -3.0)
        logits[0, 0, self.eng.log[-1]] = 4.0
        return types.SimpleNamespace(logits=logits)

    def fused_greedy_decode_n(self, n, cache, reserve_tokens=0):
        assert self.eng.ctx == cache[0].offset, "engine state must be restored for this row"
        self.eng.calls.append(("slice", n, cache[0].offset))
        self.eng.decode(n)
        for c in cache:
            c.offset += n


class _FakeBatchEngine(_FakeEngine):
    """+ the lock-step batched decoder surface (engine.py: set_kv_row / bind_pool / batch_* / kv_copy_row);
    row contents are tracked as (uid-independent) tags so that a wrong row copy shows up as wrong tokens."""

    def __init__(self):
        super().__init__()
        self.row = 0
        self.batch = None
        self.copies = []

    def set_kv_row(self, r):
        self.row = r

    def bind_pool(self, pool):
        self.pool = pool

    def kv_copy_row(self, dst, dst_row, src, src_row, n):
        self.copies.append((dst_row, src_row, n))

    def batch_begin(self, tok, ctx, pos, active):
        self.batch = [list(map(int, x)) for x in (tok, ctx, pos, active)]
        self.blog = []
        self.calls.append(("begin", len(tok)))

    def batch_decode(self, n, want_logprobs=False):
        tok, ctx, pos, act = self.batch
        self.calls.append(("bstep", n, len(tok)))
        for _ in range(n):
            out = []
            for b in range(len(tok)):
                t = _f(tok[b], ctx[b], pos[b])
                out.append(t)
                if act[b]:
                    tok[b], ctx[b], pos[b] = t, ctx[b] + 1, pos[b] + 1
            self.blog.append(out)

    def batch_fetch(self, first, n, toks, lps=None):
        for i in range(n):
            toks[i, :] = torch.tensor(self.blog[first + i], dtype=torch.int32)
            if lps is not None:
                lps[i, :] = -0.25

    def batch_logits_view(self, which="logits"):
        B = len(self.batch[0])
        lg = torch.full((B, V), -3.0)
        for b in range(B):
            lg[b, self.blog[-1][b]] = 4.0
        return lg


def _fake_model(lockstep=False):
    eng = _FakeBatchEngine() if lockstep else _FakeEngine()
    lm = _FakeLM(eng)
    if lockstep:
        lm.args = types.SimpleNamespace(num_hidden_layers=2)
        lm.n_kv_heads, lm.head_dim = 1, 8

        def make_cache_row(pool, row):
            cs = [_FakeCache(), _FakeCache()]
            for c in cs:
                c._row, c._pool = row, pool
            return cs
        lm.make_cache_row = make_cache_row

    def get_input_embeddings(ids, pixel_values=None, mask=None, **kw):
        ids = np.asarray(ids)
        T = ids.shape[1]
        delta = -3 if pixel_values is not None else 0
        return types.SimpleNamespace(inputs_embeds=torch.zeros(1, T, 4), position_ids=None,
                                     rope_deltas=np.asarray([[delta]]))
    model = types.SimpleNamespace(engine=eng, language_model=lm, get_input_embeddings=get_input_embeddings,
                                  config=types.SimpleNamespace(eos_token_id=[V + 1]))
    proc = types.SimpleNamespace(tokenizer=types.SimpleNamespace(stopping_criteria=None))
    return model, proc


def _alone(ids, max_tokens, with_image=False, eos=()):
    """Expected tokens of one request run by itself."""
    model, proc = _fake_model()
    from mlx_vlm_b200.generate_batch import BatchGenerator
    g = BatchGenerator(model, proc, max_tokens=max_tokens, decode_slice=1, stop_tokens=set(eos))
    g.insert([ids], prompt_kwargs=[{"pixel_values": 1} if with_image else {}])
    out = []
    while g.has_work:
        _, rs = g.next()
        out.extend(rs)
    return [r.token for r in out], out[-1].finish_reason


@pytest.mark.parametrize("decode_slice", [1, 4, 16])
def test_batch_generator_time_multiplexing_equals_rows_alone(decode_slice):
    from mlx_vlm_b200.generate_batch import BatchGenerator
    prompts = [[5, 6, 7, 8, 9], [1, 2], [3, 3, 3], [11] * 9]
    images = [True, False, True, False]
    maxes = [7, 12, 1, 9]
    model, proc = _fake_model()
    g = BatchGenerator(model, proc, max_tokens=32, completion_batch_size=3, prefill_batch_size=2,
                       decode_slice=decode_slice)
    uids = g.insert(prompts, maxes, [{"pixel_values": 1} if im else {} for im in images])
    assert uids == [0, 1, 2, 3]
    assert [len(r.ids) for r in g.unprocessed_prompts] == [2, 3, 5, 9]   # shortest first
    got = {u: [] for u in uids}
    fin = {}
    admitted = []
    n_calls = 0
    while g.has_work:
        pr, rs = g.next()
        n_calls += 1
        admitted.extend(p.uid for p in pr)
        assert len(pr) <= 2 and len(g.active_uids) <= 3
        assert len({r.uid for r in rs}) == len(rs), "one token per active row per call"
        for r in rs:
            got[r.uid].append(r.token)
            if r.finish_reason:
                fin[r.uid] = r.finish_reason
    assert admitted == [1, 2, 0, 3]
    for u, (p, im, m) in enumerate(zip(prompts, images, maxes)):
        want, reason = _alone(p, m, im)
        assert got[u] == want, (u, got[u], want)
        assert fin[u] == reason == "length" and len(got[u]) == m
    st = g.stats()
    assert st.prompt_tokens == sum(len(p) for p in prompts) and st.generation_tokens == sum(maxes)
    if decode_slice > 1:
        assert any(c[0] == "slice" and c[1] > 1 for c in model.engine.calls)


@pytest.mark.parametrize("decode_slice", [1, 3, 8])
def test_batch_generator_lock_step_equals_rows_alone(decode_slice):
    """host logic of the lock-step mode over a stand-in of the batched decoder: admission into pool rows,
    slices, rows leaving (EOS / length) with compaction, re-arming only when the row set changes"""
    from mlx_vlm_b200.generate_batch import BatchGenerator
    prompts = [[5, 6, 7, 8, 9], [1, 2], [3, 3, 3], [11] * 9, [2, 4, 6]]
    images = [True, False, True, False, False]
    maxes = [7, 12, 1, 9, 15]
    model, proc = _fake_model(lockstep=True)
    g = BatchGenerator(model, proc, max_tokens=32, completion_batch_size=3, prefill_batch_size=2,
                       decode_slice=decode_slice)
    assert g._lockstep
    uids = g.insert(prompts, maxes, [{"pixel_values": 1} if im else {} for im in images])
    got = {u: [] for u in uids}
    fin = {}
    while g.has_work:
        pr, rs = g.next()
        assert len(g.active_uids) <= 3
        assert len({r.uid for r in rs}) == len(rs), "one token per active row per call"
        for slot, row in enumerate(g._active):
            assert row.cache[0]._row == slot, "live rows stay compact in the pool"
        for r in rs:
            got[r.uid].append(r.token)
            if r.finish_reason:
                fin[r.uid] = r.finish_reason
    for u, (p, im, m) in enumerate(zip(prompts, images, maxes)):
        want, reason = _alone(p, m, im)
        assert got[u] == want, (u, got[u], want)
        assert fin[u] == reason == "length" and len(got[u]) == m
    eng = model.engine
    assert any(c[0] == "bstep" and c[2] > 1 for c in eng.calls), "several rows per device step"
    assert eng.copies, "a finished row is replaced by a row copy"
    n_begin = sum(c[0] == "begin" for c in eng.calls)
    n_step = sum(c[0] == "bstep" for c in eng.calls)
    assert n_begin <= n_step
    if decode_slice == 1:
        assert n_begin < n_step, "the device state is re-armed only when the row set changes"
    # EOS inside a slice: the row stops there, the rest of its slice is dropped
    toks, _ = _alone([4, 4, 2], 10)
    eos = toks[3]
    model, proc = _fake_model(lockstep=True)
    g = BatchGenerator(model, proc, max_tokens=10, decode_slice=8, stop_tokens={eos})
    a, b = g.insert([[4, 4, 2], [9, 9]])
    out = {a: [], b: []}
    while g.has_work:
        for r in g.next()[1]:
            out[r.uid].append((r.token, r.finish_reason))
    assert [t for t, _ in out[a]] == toks[:toks.index(eos) + 1] and out[a][-1][1] == "stop"
    want_b, _ = _alone([9, 9], 10, eos=[eos])
    assert [t for t, _ in out[b]] == want_b


def test_batch_generator_stop_remove_and_logprobs():
    from mlx_vlm_b200.generate_batch import BatchGenerator
    ids = [4, 4, 2]
    toks, _ = _alone(ids, 10)
    eos = toks[3]
    want, reason = _alone(ids, 10, eos=[eos])
    assert reason == "stop" and want == toks[:want.index(eos) + 1]
    model, proc = _fake_model()
    g = BatchGenerator(model, proc, max_tokens=10, compute_logprobs=True)
    a, b = g.insert([ids, [9, 9]])
    assert g.remove(b) and not g.remove(b)
    out = []
    while g.has_work:
        out.extend(g.next()[1])
    assert [r.token for r in out] == toks and all(r.uid == a for r in out)
    assert all(abs(r.token_logprob + 0.25) < 1e-6 for r in out)
    # custom sampler path: argmax sampler must reproduce the greedy tokens
    model, proc = _fake_model()
    g = BatchGenerator(model, proc, max_tokens=10, sampler=lambda lp: torch.argmax(lp, dim=-1))
    g.greedy_sampling = False
    g.insert([ids])
    out = []
    while g.has_work:
        out.extend(g.next()[1])
    assert [r.token for r in out] == toks
    with pytest.raises(NotImplementedError):
        BatchGenerator(model, proc, kv_bits=4)


def test_streaming_detokenizer_matches_reference_trace():
    """tokenizer_utils.py:48-118 executed from the reference's source over a byte-level fake
    tokenizer: multi-byte characters split across tokens are held back, a newline settles the
    pending tokens, skipped special ids never appear."""
    from mlx_vlm_b200.generate import _NaiveDetokenizer
    g = GOLD["detokenizer_trace"]
    pieces = {int(k): bytes.fromhex(v) for k, v in g["pieces_hex"].items()}

    class FakeTok:
        def decode(self, ids):
            return b"".join(pieces[i] for i in ids).decode("utf-8", errors="replace")
    det = _NaiveDetokenizer(FakeTok())
    for st in g["steps"]:
        det.add_token(st["token"], skip_special_token_ids=g["skip"])
        assert det.last_segment == st["segment"], st
        assert list(det.tokens) == st["settled_tokens"], st
    det.finalize()
    assert det.last_segment == g["final_segment"]
    assert det.text == g["final_text"] and list(det.tokens) == g["final_tokens"]


def test_penalty_processors_match_reference_source():
    """sample_utils.py:390-475 from the reference's source: repetition (assign: duplicates once),
    presence (subtract once per distinct token), frequency (scatter-subtract: duplicates add up),
    each over the last `context_size` tokens only."""
    from mlx_vlm_b200 import sample_utils as SU
    g = GOLD["logits_processors"]
    logits, hist = torch.tensor(g["logits"], dtype=torch.float32), g["tokens"]
    for key, want in g.items():
        if "(" not in key:
            continue
        name, rest = key.split("(", 1)
        arg, ctx = rest.split(")")[0].split(",")
        fn = getattr(SU, name)(float(arg), int(ctx))
        tokens = [] if key.endswith("empty history") else list(hist)
        got = fn(tokens, logits.clone())
        assert torch.allclose(got, torch.tensor(want, dtype=torch.float32), atol=1e-6), key
    with pytest.raises(ValueError):
        SU.make_repetition_penalty(-1.0)


def test_vision_feature_cache_lru_and_keys():
    """vision_cache.py:15-79: key derivation (path, list, tobytes hash, identity), LRU order."""
    import hashlib
    from mlx_vlm_b200 import VisionFeatureCache
    c = VisionFeatureCache(max_size=2)
    img = np.arange(12, dtype=np.uint8).reshape(2, 2, 3)
    assert c._make_key("a.png") == "a.png"
    assert c._make_key(img) == "pil:" + hashlib.sha256(img.tobytes()).hexdigest()[:16]
    assert c._make_key(["a.png", img]) == "a.png|" + c._make_key(img)
    o = object()
    assert c._make_key(o) == f"obj:{id(o)}"
    assert c.get("a.png") is None and "a.png" not in c and len(c) == 0
    c.put("a.png", 1)
    c.put("b.png", 2)
    assert c.get("a.png") == 1          # refreshes a.png
    c.put("c.png", 3)                   # evicts b.png (least recently used)
    assert "b.png" not in c and "a.png" in c and "c.png" in c and len(c) == 2
    c.put("a.png", 10)                  # update in place, no eviction
    assert c.get("a.png") == 10 and len(c) == 2
    c.clear()
    assert len(c) == 0


def test_kv_cache_extract_known_answers():
    """reference tests/test_cache.py:14-31, 83-90, 138-142 transcribed: extracting one row of a
    (standalone) KVCache, index validation, the empty cache."""
    from mlx_vlm_b200.models.cache import KVCache
    cache = KVCache()
    keys = torch.arange(2 * 2 * 3 * 4, dtype=torch.float32).reshape(2, 2, 3, 4)
    values = keys + 100
    cache.update_and_fetch(keys, values)
    ex = cache.extract(1)
    assert ex.offset == 3
    assert tuple(ex.keys[..., :3, :].shape) == (1, 2, 3, 4)
    assert torch.equal(ex.keys[..., :3, :], keys[1:2]) and torch.equal(ex.values[..., :3, :], values[1:2])
    assert torch.equal(cache.extract(-1).keys, cache.extract(1).keys)
    with pytest.raises(IndexError):
        cache.extract(2)
    with pytest.raises(IndexError):
        cache.extract(-3)
    empty = KVCache().extract(0)
    assert empty.empty() and empty.offset == 0


def test_batch_generator_api_known_answers(monkeypatch):
    """Behavioural checks of the reference's TestBatchGenerator (tests/test_generate.py:532-683)
    transcribed onto our BatchGenerator: construction, insert bookkeeping, stats arithmetic, and the
    first next() of a request reporting its prompt progress with no generation response yet."""
    import mlx_vlm_b200.generate_batch as gb
    model, proc = _fake_model()
    g = gb.BatchGenerator(model, proc, max_tokens=128, stop_tokens={2, 3})
    assert g.max_tokens == 128 and g.model is model and g.uid_count == 0 and not g.has_work
    assert g.tokenizer.stopping_criteria(2) and g.tokenizer.stopping_criteria(3)
    g = gb.BatchGenerator(model, proc, max_tokens=100)
    uids = g.insert([[1, 2, 3], [4, 5, 6, 7], [8, 9]])
    assert uids == [0, 1, 2] and g.uid_count == 3 and len(g.unprocessed_prompts) == 3
    g = gb.BatchGenerator(model, proc, max_tokens=50)
    assert len(g.insert([[1, 2, 3], [4, 5]], max_tokens=[100, 200])) == 2 and len(g.unprocessed_prompts) == 2
    assert sorted(r.max_tokens for r in g.unprocessed_prompts) == [100, 200]
    assert len(g.insert([[1, 2, 3], [4, 5]], max_tokens=75)) == 2
    with pytest.raises(ValueError):
        g.insert([[1]], max_tokens=[1, 2])
    g = gb.BatchGenerator(model, proc)
    g._prompt_tokens_counter, g._prompt_time_counter, g._gen_tokens_counter = 100, 0.5, 50
    st = g.stats()
    assert st.prompt_tps == 200.0 and st.prompt_tokens == 100 and st.generation_tokens == 50
    # first next(): prompt progress of the admitted request, no generation response yet
    model, proc = _fake_model()
    g = gb.BatchGenerator(model, proc, prefill_batch_size=1, completion_batch_size=1, prefill_step_size=None)
    prompt = [1, 2, 3]
    uids = g.insert([prompt], prompt_kwargs=[{"inputs_embeds": torch.zeros(1, 3, 8)}])
    ticks = iter([10.0, 10.2])
    monkeypatch.setattr(gb.time, "perf_counter", lambda: next(ticks))
    pr, gr = g.next()
    assert gr == [] and len(pr) == 1
    assert pr[0].uid == uids[0] and pr[0].prompt_tokens == len(prompt) and pr[0].cached_tokens == 0
    assert pr[0].prompt_tps == pytest.approx(15.0) and pr[0].prompt_time == pytest.approx(0.2)


def test_generation_batch_filter_extend_rope_deltas():
    """Bookkeeping of the reference's GenerationBatch (tests/test_generate.py:319-400): filter keeps
    uids / max_tokens / token counts / per-row rope deltas aligned, extend concatenates them, an empty
    accumulator absorbs the other side, mixing M-RoPE and non-M-RoPE rows is an error."""
    from mlx_vlm_b200.generate_batch import GenerationBatch, _Row

    def rows(uids, deltas, ntok=None, maxes=None):
        out = []
        for i, (u, d) in enumerate(zip(uids, deltas)):
            r = _Row(u, [1, 2], (maxes or [10] * len(uids))[i], {})
            r.delta, r.n_tokens = d, (ntok or [0] * len(uids))[i]
            out.append(r)
        return out
    e = GenerationBatch.empty(None, None, None)
    assert len(e) == 0 and e.uids == [] and e.max_tokens == [] and e._rope_deltas is None
    b = GenerationBatch(rows([0, 1, 2], [0, 0, 0], ntok=[5, 10, 15], maxes=[50, 60, 70]))
    b.filter([0, 2])
    assert b.uids == [0, 2] and b.max_tokens == [50, 70] and b._num_tokens == [5, 15] and len(b) == 2
    a = GenerationBatch(rows([0, 1], [5, 7]))
    a.extend(GenerationBatch(rows([2], [0])))
    assert a._rope_deltas.tolist() == [[5], [7], [0]]
    a.filter([0, 2])
    assert a.uids == [0, 2] and a._rope_deltas.tolist() == [[5], [0]]
    with pytest.raises(RuntimeError, match="MRoPE"):
        GenerationBatch(rows([0], [3])).extend(GenerationBatch(rows([1], [None])))
    e.extend(GenerationBatch(rows([0, 1], [5, 7])))
    assert e._rope_deltas.tolist() == [[5], [7]] and e.uids == [0, 1]


def test_qwen2_vl_config_schema_and_from_dict():
    """models/qwen2_vl/config.py: the reference's schema (field names / order / defaults as recorded
    from its dataclasses by tests/golden/make_golden.py), kv-head default, rope_scaling validation,
    and `ModelConfig.from_dict` copying the root-level text parameters into text_config."""
    import dataclasses
    from mlx_vlm_b200.models.qwen2_vl.config import (ModelConfig, TextConfig, VisionConfig,
                                                     qwen2_vl_2b_config, qwen2_vl_7b_config)
    g = GOLD["qwen2_vl_config_schema"]
    for cls in (VisionConfig, TextConfig, ModelConfig):
        got = [[f.name, None if f.default is dataclasses.MISSING else f.default] for f in dataclasses.fields(cls)]
        assert got == g[cls.__name__], cls.__name__
    t = TextConfig(model_type="qwen2_vl", hidden_size=64, num_hidden_layers=1, intermediate_size=64,
                   num_attention_heads=4, rms_norm_eps=1e-6, vocab_size=100, num_key_value_heads=None)
    assert t.num_key_value_heads == 4 and t.mrope_section == [24, 20, 20]
    with pytest.raises(ValueError, match="rope_scaling"):
        TextConfig(model_type="qwen2_vl", hidden_size=64, num_hidden_layers=1, intermediate_size=64,
                   num_attention_heads=4, rms_norm_eps=1e-6, vocab_size=100, rope_scaling={"type": "mrope"})
    with pytest.raises(ValueError, match="type"):
        TextConfig(model_type="qwen2_vl", hidden_size=64, num_hidden_layers=1, intermediate_size=64,
                   num_attention_heads=4, rms_norm_eps=1e-6, vocab_size=100,
                   rope_scaling={"type": "yarn", "mrope_section": [1, 1, 1]})
    raw = {"model_type": "qwen2_vl", "hidden_size": 1536, "num_hidden_layers": 28, "intermediate_size": 8960,
           "num_attention_heads": 12, "num_key_value_heads": 2, "rms_norm_eps": 1e-6, "vocab_size": 151936,
           "rope_scaling": {"type": "mrope", "mrope_section": [16, 24, 24]}, "tie_word_embeddings": True,
           "image_token_id": 151655, "unknown_key": 1,
           "vision_config": {"depth": 32, "embed_dim": 1280, "hidden_size": 1536, "num_heads": 16, "extra": 2}}
    mc = ModelConfig.from_dict(raw)
    assert isinstance(mc.text_config, TextConfig) and isinstance(mc.vision_config, VisionConfig)
    assert mc.text_config.hidden_size == 1536 and mc.text_config.mrope_section == [16, 24, 24]
    assert mc.text_config.tie_word_embeddings and mc.vision_config.embed_dim == 1280 and mc.vocab_size == 151936
    assert "text_config" not in raw, "from_dict must not mutate its argument"
    two, seven = qwen2_vl_2b_config(), qwen2_vl_7b_config()
    assert (two.text_config.hidden_size, two.text_config.num_key_value_heads) == (1536, 2)
    assert (seven.text_config.hidden_size, seven.text_config.intermediate_size) == (3584, 18944)
