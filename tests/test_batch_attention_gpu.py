"""The lock-step rows' attention (csrc/decode_batch.cu: a cluster per row and key/value head shares the row's keys) at the edges
of its split: rows whose keys leave CTAs of the cluster empty, end inside a group of 16 or a slot of 128, and take several slots."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(hidden, heads, kv, inter=256):
    from mlx_vlm_b200.models.qwen2_vl import Model
    from mlx_vlm_b200.models.qwen2_vl.config import ModelConfig, TextConfig, VisionConfig
    text = TextConfig(model_type="qwen2_vl", hidden_size=hidden, num_hidden_layers=2, intermediate_size=inter, num_attention_heads=heads,
                      rms_norm_eps=1e-6, vocab_size=512, num_key_value_heads=kv, rope_theta=1000000.0,
                      rope_scaling={"type": "mrope", "mrope_section": [hidden // heads // 2 - 8, 4, 4]}, tie_word_embeddings=True)
    vis = VisionConfig(depth=1, embed_dim=128, hidden_size=hidden, num_heads=2)
    return Model(ModelConfig(text_config=text, vision_config=vis, model_type="qwen2_vl", vocab_size=512), device="cuda:0").init_random(1, 0.04)


def _rotate(x, pos, d):
    inv = 1000000.0 ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
    c, s = (pos * inv).cos(), (pos * inv).sin()
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _want(model, ids, pool, lens):
    """one decode step of every row in float64"""
    w = {n: t.double() for n, t in model.engine.weights.items() if n.startswith("lm.")}
    t = model.config.text_config
    H, nh, nkv = t.hidden_size, t.num_attention_heads, t.num_key_value_heads
    d = H // nh

    def rms(x, g):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * g
    out = []
    for b, n in enumerate(lens):
        x = w["lm.embed"][int(ids[b, 0])]
        for i in range(2):
            qkv = w[f"lm.{i}.wqkv"] @ rms(x, w[f"lm.{i}.ln1"]) + w[f"lm.{i}.bqkv"]
            q, k, v = qkv[:H].view(nh, d), qkv[H:H + nkv * d].view(nkv, d), qkv[H + nkv * d:].view(nkv, d)
            q, k = _rotate(q, n, d), _rotate(k, n, d)
            K = torch.cat([pool[i, 0, b, :, :n].double(), k[:, None]], 1).repeat_interleave(nh // nkv, 0)
            V = torch.cat([pool[i, 1, b, :, :n].double(), v[:, None]], 1).repeat_interleave(nh // nkv, 0)
            p = torch.softmax((K @ q[:, :, None])[..., 0] * d ** -0.5, -1)
            x = x + w[f"lm.{i}.wo"] @ (p[:, None] @ V)[:, 0].reshape(-1)
            g = w[f"lm.{i}.wgu"] @ rms(x, w[f"lm.{i}.ln2"])
            x = x + w[f"lm.{i}.wd"] @ (torch.nn.functional.silu(g[:g.shape[0] // 2]) * g[g.shape[0] // 2:])
        out.append(w["lm.embed"] @ rms(x, w["lm.norm"]))
    return torch.stack(out)


# (head size, heads, kv heads): 7 and 6 and 1 heads to a group, more heads than a CTA takes, both head sizes
@pytest.mark.parametrize("hd,nh,nkv", [(128, 14, 2), (128, 12, 2), (64, 4, 4), (64, 18, 2), (128, 8, 1)])
@pytest.mark.parametrize("lens", [(1, 15, 16, 17), (127, 128, 129, 255, 640), (1023, 1024, 1025), (3, 2500), (90,) * 16])
def test_rows_of_any_length(hd, nh, nkv, lens):
    model = _model(hd * nh, nh, nkv)
    lm = model.language_model
    rows, caches = lm.make_batch_cache(len(lens), max(lens) + 8)
    rows.lengths = list(lens)
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    pool = rows.pool.buf
    pool.copy_(torch.randn(pool.shape, generator=g, device="cuda"))
    for b, n in enumerate(lens):
        pool[:, :, b, :, n:] = float("nan")        # rows that are not cached yet are never part of a result
    before = pool.clone()
    ids = np.random.default_rng(3).integers(0, 512, size=(len(lens), 1))
    got = lm(ids, cache=caches).logits
    model.engine.stream.synchronize()       # (the logits are the engine stream's: nothing else waits for it)
    got = got[:, 0].double()
    want = _want(model, ids, before, lens)
    # two layers of bf16 roundings (2^-9 each at about ten places a layer): measured 0.008 - 0.02
    err = ((got - want).norm(dim=1) / want.norm(dim=1)).max().item()
    print(f"{lens} hd={hd}: {err:.4f}")
    assert err <= 0.05
    for b, n in enumerate(lens):
        assert torch.equal(pool[:, :, b, :, :n], before[:, :, b, :, :n])
        assert not bool(torch.isnan(pool[:, :, b, :, n].float()).any())
        assert bool(torch.isnan(pool[:, :, b, :, n + 1:].float()).all())


def _boundaries(n):
    """keys of a row of n cached ones at the edges of every split: first and last key of each CTA of 1, 2, 4 and 8, the ends of
    their 128-key slots, the last key"""
    at = {0, n - 1}
    for ranks in (1, 2, 4, 8):
        share = -(-(n + 1) // (16 * ranks)) * 16
        for r in range(ranks):
            at |= {j for j in (r * share, r * share + 127, r * share + 128, (r + 1) * share - 1)}
    return sorted(j for j in at if 0 <= j < n)


# rows for the kernel of short rows (up to 256 keys of 128 dims, 768 of 64) and for clusters; one more key than it takes
@pytest.mark.parametrize("hd,nh,nkv", [(128, 14, 2), (64, 4, 4), (64, 18, 2), (128, 40, 8)])
@pytest.mark.parametrize("lens", [(2, 17, 255), (256, 5), (127, 767), (768, 33, 130), (1023, 1024, 1025), (40,) * 16])
@pytest.mark.parametrize("what", ["cached", "new"])
def test_every_key_counts(hd, nh, nkv, lens, what):
    """cached: nearly equal weights and values of n times the size at the edges of the splits, so that one of these keys left out
    or counted twice moves the result by more than a tenth; new: the step's own key takes nearly all of the weight"""
    model = _model(hd * nh, nh, nkv)
    model.engine.stream.synchronize()
    lm = model.language_model
    rows, caches = lm.make_batch_cache(len(lens), max(lens) + 8)
    rows.lengths = list(lens)
    g = torch.Generator(device="cuda").manual_seed(len(lens) + hd)
    pool = rows.pool.buf
    pool.copy_(torch.randn(pool.shape, generator=g, device="cuda"))
    pool[:, 0] *= 0.02 if what == "cached" else 0.0
    H = hd * nh
    for i in range(2):
        b = model.engine.weights[f"lm.{i}.bqkv"]
        b.copy_(torch.randn(b.shape, generator=g, device="cuda"))
        b[:H + nkv * hd] = 0.0 if what == "cached" else 1.0     # (q . k = hd at the same position: weight e^(sqrt hd))
    for b, n in enumerate(lens):
        if what == "cached":
            pool[:, 1, b, :, _boundaries(n)] *= n
        pool[:, :, b, :, n:] = float("nan")
    before = pool.clone()
    torch.cuda.synchronize()
    ids = np.random.default_rng(5).integers(0, 512, size=(len(lens), 1))
    got = lm(ids, cache=caches).logits
    model.engine.stream.synchronize()       # (the logits are the engine stream's: nothing else waits for it)
    got = got[:, 0].double()
    want = _want(model, ids, before, lens)
    err = ((got - want).norm(dim=1) / want.norm(dim=1)).max().item()
    print(f"{what} {lens} hd={hd}: {err:.4f}")
    assert err <= 0.05        # the roundings of test_rows_of_any_length


def test_rows_grow_from_one_kernel_to_the_other():
    """a generation whose rows pass the longest that the kernel of short rows takes, in chunks: the graphs of both kernels give the
    tokens of single steps"""
    model = _model(128 * 4, 4, 2)
    eng, lm = model.engine, model.language_model
    ids = np.random.default_rng(6).integers(0, 512, size=(2, 1))

    def run(chunks):
        rows, caches = lm.make_batch_cache(2, 512)
        rows.lengths = [210, 230]
        rows.pool.buf.copy_(torch.randn(rows.pool.buf.shape, generator=torch.Generator(device="cuda").manual_seed(7), device="cuda"))
        torch.cuda.synchronize()
        lm(ids, cache=caches)
        for n in chunks:
            eng.batch_decode(n)
        eng.stream.synchronize()
        return eng.batch_token_log_view()[:1 + sum(chunks), :2].clone(), rows.pool.buf.clone()
    ones, pool1 = run([1] * 48)
    many, pool2 = run([12, 4, 8, 8, 16])
    again, _ = run([48])
    assert torch.equal(ones, many)
    assert torch.equal(pool1[:, :, :, :, 210:220], pool2[:, :, :, :, 210:220])
    assert torch.equal(ones[:1], again[:1])
