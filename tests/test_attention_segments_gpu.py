"""The pipelined attention on segments that start anywhere (frames and pictures of any size in one launch) and on later
portions of a prompt (keys and values read from the cache), at the edges of its 128-key tiles."""
import numpy as np
import pytest
import torch

from _util import cmp_noise, rl2
from test_engine_gpu import _build

pytestmark = pytest.mark.gpu


def _pictures(c, sizes, seed=3):
    from oracle import qwen2vl as O
    rng = np.random.default_rng(seed)
    pvs, grids = zip(*[O.preprocess_image(rng.integers(0, 256, size=(3,) + s, dtype=np.uint8), c.vision) for s in sizes])
    return list(pvs), [list(g) for g in grids]


# patches per picture: 36 | 128 (one whole tile) | 132 (four keys in the second tile), so that segments start at patches
# 36 and 164 (neither a multiple of 8); then 156 (28 in the second tile) before 12
@pytest.mark.parametrize("sizes", [((84, 84), (112, 224), (28, 924)), ((84, 364), (28, 84)), ((28, 28),)])
def test_pictures_of_any_size_share_a_launch(sizes):
    from oracle import qwen2vl as O
    c, W, model, _ = _build("tiny", 8, (56, 56))
    pvs, grids = _pictures(c, sizes)
    ids = [5]
    for _ in sizes:
        ids += [c.vision_start_token_id, c.image_token_id, c.vision_end_token_id, 7]
    ids = np.asarray([O.expand_image_tokens(ids, grids, c)], dtype=np.int64)
    pv, grid = np.concatenate(pvs, axis=0), np.asarray(grids, dtype=np.int64)
    ref = O.greedy_generate(c, W, ids, pv, grid, 1)["prefill"]
    ex = O.greedy_generate(c, W, ids, pv, grid, 1, dtype="f32")["prefill"]
    feats = model.vision_tower(torch.from_numpy(pv).cuda(), grid)
    model.engine.stream.synchronize()
    cmp_noise(feats, ref.image_features, ex.image_features, f"features of {sizes}")


def test_a_picture_of_nans_stays_alone():
    """the rows behind a segment's last key are cleared before they meet its zero weights"""
    c, _, model, _ = _build("tiny", 8, (56, 56))
    pvs, grids = _pictures(c, ((84, 84), (56, 56)))
    grid = np.asarray(grids, dtype=np.int64)
    good = torch.from_numpy(np.concatenate(pvs, axis=0)).cuda()
    bad = good.clone()
    bad[36:] = float("nan")
    a, b = model.vision_tower(good, grid), model.vision_tower(bad, grid)
    model.engine.stream.synchronize()
    assert torch.equal(a[:9], b[:9]) and bool(torch.isnan(b[9:].float()).all())


@pytest.mark.parametrize("first,total", [(1, 130), (127, 128), (128, 257), (129, 160), (200, 201), (20, 51), (13, 15), (100, 129)])
def test_a_later_portion_reads_the_cache(first, total):
    """two portions == one, at the real head size: same kernel, same keys and values, same order of sums"""
    from mlx_vlm_b200.models.cache import make_prompt_cache
    _, _, model, _ = _build("wide1", 8, (56, 56))
    ids = np.random.default_rng(total).integers(0, 900, size=(1, total))
    emb = model.get_input_embeddings(ids, None)
    lm = model.language_model
    kw = dict(position_ids=emb.position_ids, logits_to_keep=1, reserve_tokens=total + 64)
    c1, c2 = make_prompt_cache(lm), make_prompt_cache(lm)
    one = lm(ids, inputs_embeds=emb.inputs_embeds, cache=c1, **kw).logits
    c2[0]._pool.reserve(total + 64)
    c2[0]._pool.buf.fill_(float("nan"))        # unused rows of a cache are never part of a result
    lm(ids[:, :first], inputs_embeds=emb.inputs_embeds[:, :first], cache=c2, **kw)
    two = lm(ids[:, first:], inputs_embeds=emb.inputs_embeds[:, first:], cache=c2, **kw).logits
    model.engine.stream.synchronize()
    # the GEMMs of the portions may sum their splits in another order: one bf16 rounding (2^-9) of the last hidden state
    assert rl2(two[0, -1], one[0, -1]) <= 2.0 ** -8
    a, b = c1[0]._pool.buf[0, :, :, :, :total], c2[0]._pool.buf[0, :, :, :, :total]
    assert rl2(b, a) <= 2.0 ** -9
