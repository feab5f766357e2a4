"""A prompt long enough for GEMMs that add the residual in place (csrc/engine.cu: v2_linear_residual_norm): the first pass, in which
the GEMM configurations are measured, must leave the residual stream alone.  The same kernels on the same data: equal bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# 3584 wide: 1281 tokens and more fill the SMs without split-K; 3700 x 3584 fp32 is more than the partial-tile region holds
@pytest.mark.parametrize("T", [1290, 3700])
def test_first_pass_equals_later_ones(T):
    from mlx_vlm_b200.models.cache import make_prompt_cache
    from mlx_vlm_b200.models.qwen2_vl import Model
    from oracle import qwen2vl as O
    from test_engine_gpu import _to_model_config
    from test_gate_gpu import _cfg_7b_geometry
    c = _cfg_7b_geometry()
    model = Model(_to_model_config(c), device="cuda:0")
    model.load_weights(O.init_weights(c, 0, norm_jitter=0.05))
    ids = np.random.default_rng(T).integers(0, 900, size=(1, T))
    emb = model.get_input_embeddings(ids, None)
    got = []
    for _ in range(2):
        cache = make_prompt_cache(model.language_model)
        model.language_model(ids, inputs_embeds=emb.inputs_embeds, cache=cache, position_ids=emb.position_ids,
                             rope_deltas=emb.rope_deltas)
        model.engine.stream.synchronize()
        got.append((cache[1].keys[0, :, :T].clone(), model.engine.logits_view().clone()))
    assert model.engine.device_error() == 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
