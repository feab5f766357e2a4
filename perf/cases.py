"""The work that a program built on mlx_vlm_b200 has it do, as cases that can be timed and compared.

A case is one call (or the few calls that belong together) through the package's own entry points, at the layer sizes
of the package's configurations: the vision towers (`vision_tower`, `encode_image`), a prompt's prefill (fresh, a later
portion, several prompts at once), one decode step (one request, lock-step rows), and an attention block of a decoder
that is assembled layer by layer.  Most cases hold a few layers of the geometry that they name, with a vocabulary cut
in proportion, so that a rounding that falls the other way does not travel through a whole model; one is a whole model.

`exact` restates each case in float64 with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

STD = 0.03          # of every random weight: scores and activations of the size that trained layers have

# decoder geometries of the package's configurations: hidden, mlp, heads, kv heads
GEOMETRY = {
    "qwen2-vl-2b": (1536, 8960, 12, 2),
    "qwen2-vl-7b": (3584, 18944, 28, 4),
    "llama-7b": (4096, 11008, 32, 32),      # LLaVA-1.5-7B
    "mistral-7b": (4096, 14336, 32, 8),     # Idefics2-8B
}
VIT = dict(embed_dim=1280, num_heads=16, hidden_size=1536)   # Qwen2-VL's tower


def listed():
    return [
        # one photo at the size of the headline benchmark, through some blocks of the Qwen2-VL tower
        {"name": "vit_one_image", "kind": "vit", "grids": "1x24x24", "depth": 4},
        # a message with several pictures of uneven shapes and a short clip (one attention segment per frame)
        {"name": "vit_mixed", "kind": "vit", "grids": "1x38x26,1x22x34,4x18x30,1x46x46", "depth": 2},
        # the headline benchmark's prompt: 128 text tokens and one image, first chunk of a request
        {"name": "prefill_short", "kind": "prefill", "geometry": "qwen2-vl-2b", "layers": 4, "vocab": 16384, "tokens": 272, "ctx": 0},
        # a long document: the second portion of a prompt that is taken in steps of 2048 tokens
        {"name": "prefill_portion", "kind": "prefill", "geometry": "qwen2-vl-7b", "layers": 2, "vocab": 16384, "tokens": 2048, "ctx": 2048},
        # eight image prompts of uneven length admitted to a batch together
        {"name": "prefill_batch", "kind": "prefill_rows", "geometry": "llama-7b", "layers": 2, "vocab": 2048,
         "lengths": "608,601,617,608,590,633,608,612"},
        # one decoded token of the whole 2B model, late in the headline benchmark's answer
        {"name": "decode_whole_2b", "kind": "decode", "geometry": "qwen2-vl-2b", "layers": 28, "vocab": 151936, "ctx": 700},
        # one decoded token at the end of a long conversation, some layers of the Mistral geometry
        {"name": "decode_long", "kind": "decode", "geometry": "mistral-7b", "layers": 4, "vocab": 8192, "ctx": 6000},
        # continuous batching: eight requests of uneven age advance by one token
        {"name": "rows_eight", "kind": "rows", "geometry": "qwen2-vl-7b", "layers": 4, "vocab": 16384,
         "lengths": "300,784,412,655,272,530,701,333"},
        # the same with the small model, fewer rows and long conversations
        {"name": "rows_long", "kind": "rows", "geometry": "qwen2-vl-2b", "layers": 4, "vocab": 16384, "lengths": "2900,1025,3777,2048,3301"},
        # LLaVA-1.5: eight pictures through blocks of the CLIP tower (fp32 arithmetic) and the projector
        {"name": "clip_images", "kind": "clip", "images": 8, "side": 336, "layers": 3},
        # Idefics2: four pictures, one of them padded, through blocks of the SigLIP tower, MLP and resampler
        {"name": "siglip_images", "kind": "siglip", "images": 4, "side": 448, "cut": 1, "layers": 2},
        # the attention block of a decoder assembled layer by layer, on a prompt
        {"name": "latent_prompt", "kind": "latent", "heads": 16, "tokens": 2048, "ctx": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vit", "vit", "prefill", "prefill", "prefill_rows", "decode", "decode", "rows", "rows", "clip", "siglip", "latent"])
    if kind == "vit":
        left, grids = _log(rng, 200, 7000), []
        while left > 60 and len(grids) < 6:
            h = 2 * rng.randint(4, max(4, min(40, int(math.sqrt(left)) // 2)))
            w = 2 * max(2, min(40, round(h * rng.uniform(0.6, 1.7) / 2)))
            t = rng.choice([1, 1, 1, 2, 3])
            grids.append((t, h, w))
            left -= t * h * w
        return {"kind": kind, "grids": ",".join("x".join(map(str, g)) for g in grids), "depth": rng.choice([1, 2])}
    if kind == "prefill":
        geo = rng.choice(sorted(GEOMETRY))
        ctx = rng.choice([0, 0, 0, 2048, _log(rng, 1, 4000)])
        return {"kind": kind, "geometry": geo, "layers": 2, "vocab": 8192, "tokens": _log(rng, 1, 2048), "ctx": ctx}
    if kind == "prefill_rows":
        n = rng.randint(2, 8)
        return {"kind": kind, "geometry": rng.choice(sorted(GEOMETRY)), "layers": 2, "vocab": 2048,
                "lengths": ",".join(str(_log(rng, 16, 520)) for _ in range(n))}
    if kind == "decode":
        return {"kind": kind, "geometry": rng.choice(sorted(GEOMETRY)), "layers": rng.randint(2, 4), "vocab": 8192,
                "ctx": _log(rng, 8, 8000)}
    if kind == "rows":
        top = rng.choice([800, 4000])
        return {"kind": kind, "geometry": rng.choice(["qwen2-vl-2b", "qwen2-vl-7b", "mistral-7b"]), "layers": 2, "vocab": 8192,
                "lengths": ",".join(str(_log(rng, 20, top)) for _ in range(rng.randint(2, 16)))}
    if kind == "clip":
        return {"kind": kind, "images": rng.randint(1, 8), "side": 336, "layers": rng.choice([2, 3])}
    if kind == "siglip":
        return {"kind": kind, "images": rng.randint(1, 4), "side": 14 * rng.randint(12, 32), "cut": rng.randint(0, 1), "layers": rng.choice([1, 2])}
    return {"kind": "latent", "heads": rng.choice([16, 32]), "tokens": _log(rng, 8, 1400), "ctx": rng.choice([0, _log(rng, 1, 600)])}


# ---------------------------------------------------------------------------------------------- inputs and weights
class _Rand:
    """seeded device tensors, in the order in which they are asked for"""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def __call__(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        t = torch.randn(shape, generator=self.g, device="cuda", dtype=torch.float32)
        return t.mul_(std).add_(mean).to(dtype)

    def weight(self, *shape):
        return self(*shape, std=STD, dtype=torch.bfloat16)

    def norm(self, n):
        return self(n, std=0.1, mean=1.0, dtype=torch.bfloat16)

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device="cuda").cpu().numpy()


def _grids(case):
    return [tuple(int(v) for v in g.split("x")) for g in case["grids"].split(",")]


def _lengths(case):
    return [int(v) for v in case["lengths"].split(",")]


def _vit_weights(r, depth, E, out):
    p, w = "vision_tower.", {}
    w[p + "patch_embed.proj.weight"] = r.weight(E, 3, 2, 14, 14)
    for i in range(depth):
        q = f"{p}blocks.{i}."
        for n in ("norm1", "norm2"):
            w[q + n + ".weight"], w[q + n + ".bias"] = r.norm(E), r.weight(E)
        for n, (o, k) in {"attn.qkv": (3 * E, E), "attn.proj": (E, E), "mlp.fc1": (4 * E, E), "mlp.fc2": (E, 4 * E)}.items():
            w[q + n + ".weight"], w[q + n + ".bias"] = r.weight(o, k), r.weight(o)
    w[p + "merger.ln_q.weight"], w[p + "merger.ln_q.bias"] = r.norm(E), r.weight(E)
    for n, o in (("mlp.0", 4 * E), ("mlp.2", out)):
        w[p + f"merger.{n}.weight"], w[p + f"merger.{n}.bias"] = r.weight(o, 4 * E), r.weight(o)
    return w


def _lm_weights(r, geometry, layers, vocab):
    H, I, nh, nkv = GEOMETRY[geometry]
    kv = nkv * (H // nh)
    p, w = "language_model.model.", {}
    w[p + "embed_tokens.weight"], w[p + "norm.weight"] = r.weight(vocab, H), r.norm(H)
    for i in range(layers):
        q = f"{p}layers.{i}."
        for n in ("input_layernorm", "post_attention_layernorm"):
            w[q + n + ".weight"] = r.norm(H)
        for n, o in (("q", H), ("k", kv), ("v", kv)):
            w[q + f"self_attn.{n}_proj.weight"], w[q + f"self_attn.{n}_proj.bias"] = r.weight(o, H), r.weight(o)
        for n, (o, k) in {"self_attn.o": (H, H), "mlp.gate": (I, H), "mlp.up": (I, H), "mlp.down": (H, I)}.items():
            w[q + n + "_proj.weight"] = r.weight(o, k)
    return w


def _qwen_model(r, geometry="qwen2-vl-2b", layers=1, vocab=64, depth=1):
    """(model with seeded weights, the same weights by their checkpoint names)"""
    from mlx_vlm_b200.models.qwen2_vl import Model
    from mlx_vlm_b200.models.qwen2_vl.config import ModelConfig, TextConfig, VisionConfig
    H, I, nh, nkv = GEOMETRY[geometry]
    text = TextConfig(model_type="qwen2_vl", hidden_size=H, num_hidden_layers=layers, intermediate_size=I, num_attention_heads=nh,
                      rms_norm_eps=1e-6, vocab_size=vocab, num_key_value_heads=nkv, rope_theta=1000000.0,
                      rope_scaling={"type": "mrope", "mrope_section": [16, 24, 24]}, tie_word_embeddings=True)
    vision = VisionConfig(depth=depth, embed_dim=VIT["embed_dim"], hidden_size=H, num_heads=VIT["num_heads"])
    w = _lm_weights(r, geometry, layers, vocab)
    w.update(_vit_weights(r, depth, VIT["embed_dim"], H))
    model = Model(ModelConfig(text_config=text, vision_config=vision, model_type="qwen2_vl", vocab_size=vocab), device="cuda:0")
    model.load_weights(w)
    return model, w


def _prompt_positions(T, ctx):
    """(3, 1, T) positions of a prompt portion: some text, an image's rows and columns where it fits, text"""
    pos = np.tile(np.arange(ctx, ctx + T), (3, 1))
    if ctx == 0 and T >= 200:
        a, side = 15, 12
        g = np.indices((1, side, side)).reshape(3, -1) + a
        pos[:, a:a + side * side] = g
        pos[:, a + side * side:] -= side * side - side
    return pos[:, None]


def _clip_setup(case, seed):
    r = _Rand(seed)
    from mlx_vlm_b200.models.llava.config import ModelConfig, TextConfig, VisionConfig
    from mlx_vlm_b200.models.llava.weights import weight_shapes
    cfg = ModelConfig(text_config=TextConfig(num_hidden_layers=1, intermediate_size=1024, vocab_size=64),
                      vision_config=VisionConfig(num_hidden_layers=case["layers"], image_size=case["side"]), vocab_size=64)
    w = {n: r.norm(*s) if "norm" in n and n.endswith(".weight") else r.weight(*s) for n, s in weight_shapes(cfg).items()}
    return cfg, w, r(case["images"], 3, case["side"], case["side"])


def _siglip_setup(case, seed):
    r = _Rand(seed)
    from mlx_vlm_b200.models.idefics2.config import ModelConfig, PerceiverConfig, TextConfig, VisionConfig
    from mlx_vlm_b200.models.idefics2.weights import weight_shapes
    cfg = ModelConfig(text_config=TextConfig(num_hidden_layers=1, vocab_size=64),
                      vision_config=VisionConfig(hidden_size=1152, intermediate_size=4304, num_hidden_layers=case["layers"],
                                                 num_attention_heads=16, image_size=980, patch_size=14),
                      perceiver_config=PerceiverConfig(resampler_depth=1), vocab_size=64)
    w = {n: r.norm(*s) if "norm" in n and n.endswith(".weight") else r.weight(*s) for n, s in weight_shapes(cfg).items()
         if not n.startswith("language_model.layers.0.mlp")}
    w.update({n: torch.zeros(s, device="cuda", dtype=torch.bfloat16) for n, s in weight_shapes(cfg).items() if n not in w})
    n, side = case["images"], case["side"]
    pixels = r(1, n, 3, side, side).cpu().numpy()        # the processor hands host arrays over
    mask = np.ones((1, n, side, side), dtype=bool)
    if case["cut"]:                                      # the last picture is smaller and padded with zeros
        cut = side - 14 * max(1, side // 56)
        mask[0, -1, cut:] = False
        pixels[0, -1, :, cut:] = 0
    return cfg, w, pixels, mask


LATENT = dict(width=2048, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=1536)


def _latent_setup(case, seed):
    r, z, H = _Rand(seed), LATENT, case["heads"]
    cfg = dict(heads=H, dim=z["dim"], rot_dim=z["rot_dim"], vdim=z["vdim"], kv_rank=z["kv_rank"], q_rank=z["q_rank"],
               rot={"base": 10000.0, "dims": z["rot_dim"]}, scale=(z["dim"] + z["rot_dim"]) ** -0.5)
    W, dn, dr, dv, kr, qr = z["width"], z["dim"], z["rot_dim"], z["vdim"], z["kv_rank"], z["q_rank"]
    w = {"dq": r.weight(qr, W), "dq.norm": r.norm(qr), "uq": r.weight(H * (dn + dr), qr), "dkv": r.weight(kr + dr, W),
         "dkv.norm": r.norm(kr), "uk": r.weight(H * dn, kr), "uv": r.weight(H * dv, kr), "o": r.weight(W, H * dv)}
    rows = r(case["ctx"], kr + dr, dtype=torch.bfloat16)     # what earlier portions of the prompt cached
    return cfg, w, rows, r(case["tokens"], W)


# ------------------------------------------------------------------------------------------------------- the cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "vit":
        r = _Rand(seed)
        model, _ = _qwen_model(r, depth=case["depth"])
        grid = np.asarray(_grids(case))
        return {"case": case, "model": model, "grid": grid, "pixels": r(int(grid.prod(1).sum()), 3 * 2 * 14 * 14)}
    if kind == "clip":
        from mlx_vlm_b200.models.llava import Model
        cfg, w, pixels = _clip_setup(case, seed)
        model = Model(cfg, device="cuda:0")
        model.load_weights(w)
        return {"case": case, "model": model, "pixels": pixels}
    if kind == "siglip":
        from mlx_vlm_b200.models.idefics2 import Model
        cfg, w, pixels, mask = _siglip_setup(case, seed)
        model = Model(cfg, device="cuda:0")
        model.load_weights(w)
        return {"case": case, "model": model, "pixels": pixels, "mask": mask}
    if kind == "latent":
        return _latent_prepare(case, seed)
    r = _Rand(seed)
    model, _ = _qwen_model(r, case["geometry"], case["layers"], case["vocab"])
    lm, H = model.language_model, GEOMETRY[case["geometry"]][0]
    s = {"case": case, "model": model}
    if kind == "prefill":
        T, ctx = case["tokens"], case["ctx"]
        s["cache"] = lm.make_cache()
        pool = s["cache"][0]._pool
        pool.reserve(ctx + T + 512)
        pool.buf[..., :ctx, :] = r(*pool.buf[..., :ctx, :].shape, dtype=torch.bfloat16)
        s["ids"], s["embeds"] = r.ints(0, case["vocab"], 1, T), r(1, T, H, std=STD, dtype=torch.bfloat16)
        s["positions"] = _prompt_positions(T, ctx)
    elif kind == "prefill_rows":
        lens = _lengths(case)
        s["batch"], _ = lm.make_batch_cache(len(lens), max(lens) + 8)
        s["ids"] = [r.ints(0, case["vocab"], 1, n) for n in lens]
        s["embeds"] = [r(1, n, H, std=STD, dtype=torch.bfloat16) for n in lens]
    elif kind == "decode":
        s["cache"] = lm.make_cache()
        pool = s["cache"][0]._pool
        pool.reserve(case["ctx"] + 256)
        pool.buf.copy_(r(*pool.buf.shape, dtype=torch.bfloat16))
        s["ids"] = r.ints(0, case["vocab"], 1, 1)
    else:
        lens = _lengths(case)
        s["batch"], s["cache"] = lm.make_batch_cache(len(lens), max(lens) + 256)
        s["batch"].lengths = list(lens)
        pool = s["batch"].pool
        pool.buf.copy_(r(*pool.buf.shape, dtype=torch.bfloat16))
        s["ids"] = r.ints(0, case["vocab"], len(lens), 1)
    torch.cuda.synchronize()
    return s


def _latent_prepare(case, seed):
    from mlx_vlm_b200.models.cache import LatentPool
    from mlx_vlm_b200.models.decoder_blocks import LatentAttention
    from mlx_vlm_b200.models.layer_ops import LayerOps
    cfg, w, rows, x = _latent_setup(case, seed)
    T, ctx = case["tokens"], case["ctx"]
    block = LatentAttention(0, cfg, LATENT["width"])
    block.cache_index = 0
    arena = {n: torch.empty(s, device="cuda", dtype=torch.bfloat16) for n, s in block.manifest("")}
    block.pack("", w, arena.__getitem__)
    pool = LatentPool(1, block.row_dim, torch.device("cuda", 0), batch=1, capacity=T + ctx + 64)
    pool.buf[0, 0, :ctx] = rows
    ops = LayerOps("cuda:0", torch.cuda.Stream(device="cuda:0"))
    slot = torch.zeros(T, dtype=torch.int32, device="cuda")
    pos = torch.arange(ctx, ctx + T, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return {"case": case, "block": block, "pool": pool, "ops": ops, "slot": slot, "pos": pos, "x": x}


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "vit":
        return s["model"].vision_tower(s["pixels"], s["grid"])
    if kind == "clip":
        return s["model"].encode_image(s["pixels"])
    if kind == "siglip":
        return s["model"].encode_image(s["pixels"], s["mask"])
    if kind == "latent":
        from mlx_vlm_b200.models.decoder_blocks import StepCtx
        ops = s["ops"]
        ctx = StepCtx(ops, s["slot"], s["pos"], s["pool"], 1e-5, segments=[(0, case["tokens"], 0, case["ctx"])])
        with ops.on_stream():
            y = s["block"].forward(ctx, s["x"])
        return {"y": y, "rows": s["pool"].buf[0, 0, case["ctx"]:case["ctx"] + case["tokens"]]}
    lm = s["model"].language_model
    if kind == "prefill":
        T, ctx, cache = case["tokens"], case["ctx"], s["cache"]
        for c in cache:
            c.offset = ctx
        out = lm(s["ids"], inputs_embeds=s["embeds"], cache=cache, position_ids=s["positions"], rope_deltas=np.zeros((1, 1)),
                 logits_to_keep=1, reserve_tokens=ctx + T + 256)
        return {"logits": out.logits, "kv": cache[0]._pool.buf[:, :, 0, :, ctx:ctx + T]}
    if kind == "prefill_rows":
        pool = s["batch"].pool
        caches = [lm.make_cache_row(pool, b) for b in range(len(s["ids"]))]
        lm.prefill_rows(s["ids"], s["embeds"], caches)
        return {"logits": s["model"].engine.snapshot("logits"),
                "kv": [pool.buf[:, :, b, :, :n] for b, n in enumerate(_lengths(case))]}
    if kind == "decode":
        cache, ctx = s["cache"], case["ctx"]
        for c in cache:
            c.offset = ctx
        out = lm(s["ids"], cache=cache, position_ids=np.full((3, 1, 1), ctx), rope_deltas=np.zeros((1, 1)))
        return {"logits": out.logits, "kv": cache[0]._pool.buf[:, :, 0, :, ctx]}
    lens = _lengths(case)
    s["batch"].lengths = list(lens)
    out = lm(s["ids"], cache=s["cache"])
    return {"logits": out.logits, "kv": [s["batch"].pool.buf[:, :, b, :, n] for b, n in enumerate(lens)]}


# ------------------------------------------------------------------------------------------- what a pass cannot avoid
def _lm_work(geometry, layers, vocab, spans, head_rows):
    """spans: (new tokens, cached tokens before them) per request.  Weights once, cached keys and values once, the new
    ones written, the tokens' embeddings and logits; causal attention counts the visible keys."""
    H, I, nh, nkv = GEOMETRY[geometry]
    kv = 2 * nkv * (H // nh)
    per_layer = H * (2 * H + kv + 3 * I)
    T = sum(n for n, _ in spans)
    seen = sum(n * c + n * (n + 1) / 2 for n, c in spans)
    return {"bytes": 2.0 * (layers * per_layer + vocab * H + layers * kv * sum(n + c for n, c in spans) + T * H + head_rows * vocab),
            "flops": 2.0 * (layers * (T * per_layer + 2 * seen * H) + head_rows * vocab * H)}


def work(case):
    kind = case["kind"]
    if kind == "vit":
        E, out, n = VIT["embed_dim"], VIT["hidden_size"], case["depth"]
        N = sum(t * h * w for t, h, w in _grids(case))
        pairs = sum(t * (h * w) ** 2 for t, h, w in _grids(case))
        wts = 1176 * E + n * 12 * E * E + 16 * E * E + 4 * E * out
        return {"bytes": 2.0 * wts + 4.0 * N * 1176 + 2.0 * N / 4 * out,
                "flops": 2.0 * (N * (1176 * E + n * 12 * E * E) + n * 2 * pairs * E + N / 4 * (16 * E * E + 4 * E * out))}
    if kind == "clip":
        B, L, E, I, H, n = case["images"], (case["side"] // 14) ** 2 + 1, 1024, 4096, 4096, case["layers"] - 1
        wts = 588 * E + n * (4 * E * E + 2 * E * I) + E * H + H * H
        return {"bytes": 2.0 * (wts + L * E) + 4.0 * B * 3 * case["side"] ** 2 + 2.0 * B * (L - 1) * H,
                "flops": 2.0 * B * (n * (L * (4 * E * E + 2 * E * I) + 2 * L * L * E) + L * 588 * E + (L - 1) * (E * H + H * H))}
    if kind == "siglip":
        B, P, E, I, n, H, Im, nl = case["images"], (case["side"] // 14) ** 2, 1152, 4304, case["layers"], 4096, 14336, 64
        tower = 588 * E + n * (4 * E * E + 2 * E * I) + 2 * E * Im + Im * H
        latent = 2 * 1536 * H + 12 * H * H
        keys = P + nl
        return {"bytes": 2.0 * (tower + latent + 2 * 384 * H + P * E) + 4.0 * B * 3 * case["side"] ** 2 + 2.0 * B * nl * H,
                "flops": 2.0 * B * (P * tower + n * 2 * P * P * E + nl * latent + keys * 2 * 384 * H + 2 * nl * keys * 1536)}
    if kind == "latent":
        z, H, T, ctx = LATENT, case["heads"], case["tokens"], case["ctx"]
        W, qk, dv, kr, qr = z["width"], z["dim"] + z["rot_dim"], z["vdim"], z["kv_rank"], z["q_rank"]
        row = kr + z["rot_dim"]
        wts = W * (qr + row) + qr * H * qk + kr * H * (z["dim"] + dv) + W * H * dv
        seen = T * ctx + T * (T + 1) / 2
        # keys and values per head are expanded from the cached rows once for every cached token
        return {"bytes": 2.0 * (wts + row * (T + ctx)) + 8.0 * T * W,
                "flops": 2.0 * (T * (W * (qr + row) + qr * H * qk + W * H * dv) + (T + ctx) * kr * H * (z["dim"] + dv) + seen * H * (qk + dv))}
    if kind == "prefill":
        return _lm_work(case["geometry"], case["layers"], case["vocab"], [(case["tokens"], case["ctx"])], 1)
    if kind == "prefill_rows":
        return _lm_work(case["geometry"], case["layers"], case["vocab"], [(n, 0) for n in _lengths(case)], len(_lengths(case)))
    if kind == "decode":
        return _lm_work(case["geometry"], case["layers"], case["vocab"], [(1, case["ctx"])], 1)
    return _lm_work(case["geometry"], case["layers"], case["vocab"], [(1, n) for n in _lengths(case)], len(_lengths(case)))


def tolerance(case):
    """about four times the distance from `exact` that the bf16 roundings of these layers give: measured 0.016 - 0.036 for
    the decoder slices, 0.06 for the whole model, 0.009 for the bf16 tower, 0.0017 for the fp32 towers (the rounding of their
    features to bf16) and 0.005 for the latent block (bf16 operands, fp32 sums)"""
    kind = case["kind"]
    if kind == "vit":
        return {"rel": 0.03}
    if kind in ("clip", "siglip"):
        return {"rel": 0.006}
    if kind == "latent":
        return {"rel": 0.02}
    return {"rel": 0.2 if case["layers"] > 8 else 0.1}


# ----------------------------------------------------------------------------------------------------- float64
def _d(w, name):
    return w[name].double()


def _lin(w, name, x):
    y = x @ _d(w, name + ".weight").T
    return y + _d(w, name + ".bias") if name + ".bias" in w else y


def _ln(w, name, x, eps):
    y = torch.nn.functional.layer_norm(x, x.shape[-1:], eps=eps)
    return y * _d(w, name + ".weight") + _d(w, name + ".bias")


def _rms(x, weight, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * weight.double()


def _rotate(x, ang):
    """rotate-half: x (..., T, d), ang (T, d / 2)"""
    a, b = x.chunk(2, -1)
    c, s = ang.cos(), ang.sin()
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, scale, visible=None):
    """q (h, T, d), k / v (h, S, d), a few heads at a time; visible (T,): number of keys that each query sees"""
    out = []
    for a in range(0, q.shape[0], 4):
        s = q[a:a + 4] @ k[a:a + 4].transpose(1, 2) * scale
        if visible is not None:
            s = s.masked_fill(torch.arange(k.shape[1], device=s.device) >= visible[:, None], float("-inf"))
        out.append(torch.softmax(s, -1) @ v[a:a + 4])
    return torch.cat(out)


def _exact_lm(case, w, spans):
    """spans: (embeddings (T, H), positions (3, T), cached k and v (layers, 2, kv heads, ctx, d)) per request ->
    per request (logits of the last token, new rows (layers, 2, kv heads, T, d))"""
    H, I, nh, nkv = GEOMETRY[case["geometry"]]
    hd = H // nh
    inv = 1000000.0 ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
    axis = torch.cat([torch.full((n,), i, device="cuda") for i, n in enumerate((16, 24, 24))])
    xs = [e.double() for e, _, _ in spans]
    angs = [torch.as_tensor(np.ascontiguousarray(p), device="cuda").double()[axis].T * inv for _, p, _ in spans]
    news = [[] for _ in spans]
    for i in range(case["layers"]):
        q_ = f"language_model.model.layers.{i}."
        lw = {n[len(q_):]: t.double() for n, t in w.items() if n.startswith(q_)}
        for j, (_, _, old) in enumerate(spans):
            x = xs[j]
            T = x.shape[0]
            n1 = _rms(x, lw["input_layernorm.weight"], 1e-6)
            heads = {n: _lin(lw, f"self_attn.{n}_proj", n1).view(T, -1, hd).transpose(0, 1) for n in "qkv"}
            q, k, v = _rotate(heads["q"], angs[j]), _rotate(heads["k"], angs[j]), heads["v"]
            news[j].append(torch.stack([k, v]))
            k, v = torch.cat([old[i, 0].double(), k], 1), torch.cat([old[i, 1].double(), v], 1)
            ctx = k.shape[1] - T
            rep = nh // nkv
            o = _attend(q, k.repeat_interleave(rep, 0), v.repeat_interleave(rep, 0), hd ** -0.5,
                        torch.arange(ctx + 1, ctx + T + 1, device="cuda"))
            x = x + _lin(lw, "self_attn.o_proj", o.transpose(0, 1).reshape(T, H))
            n2 = _rms(x, lw["post_attention_layernorm.weight"], 1e-6)
            m = torch.nn.functional.silu(_lin(lw, "mlp.gate_proj", n2)) * _lin(lw, "mlp.up_proj", n2)
            xs[j] = x + _lin(lw, "mlp.down_proj", m)
    head, norm = _d(w, "language_model.model.embed_tokens.weight"), w["language_model.model.norm.weight"]
    return [(_rms(x[-1:], norm, 1e-6) @ head.T, torch.stack(n)) for x, n in zip(xs, news)]


def _exact_vit(case, seed):
    r = _Rand(seed)
    E, nh, n = VIT["embed_dim"], VIT["num_heads"], case["depth"]
    w = _lm_weights(r, "qwen2-vl-2b", 1, 64)
    w = _vit_weights(r, n, E, GEOMETRY["qwen2-vl-2b"][0])
    grids = _grids(case)
    N, hd, p = sum(t * h * g for t, h, g in grids), E // nh, "vision_tower."
    x = r(N, 1176).double() @ _d(w, p + "patch_embed.proj.weight").reshape(E, -1).T
    pos, cuts = [], []
    for t, h, g in grids:
        at = np.indices((h, g)).reshape(2, h // 2, 2, g // 2, 2).transpose(0, 1, 3, 2, 4).reshape(2, -1).T
        pos += [at] * t
        cuts += [h * g] * t
    pos = torch.as_tensor(np.concatenate(pos), device="cuda").double()
    inv = 10000.0 ** (-torch.arange(0, hd // 2, 2, device="cuda", dtype=torch.float64) / (hd // 2))
    ang = (pos[:, :, None] * inv).reshape(N, -1)
    for i in range(n):
        q_ = f"{p}blocks.{i}."
        qkv = _lin(w, q_ + "attn.qkv", _ln(w, q_ + "norm1", x, 1e-6)).view(N, 3, nh, hd).permute(1, 2, 0, 3)
        q, k, v = _rotate(qkv[0], ang), _rotate(qkv[1], ang), qkv[2]
        o = torch.cat([_attend(a, b, c, hd ** -0.5) for a, b, c in zip(q.split(cuts, 1), k.split(cuts, 1), v.split(cuts, 1))], 1)
        x = x + _lin(w, q_ + "attn.proj", o.transpose(0, 1).reshape(N, E))
        m = _lin(w, q_ + "mlp.fc1", _ln(w, q_ + "norm2", x, 1e-6))
        x = x + _lin(w, q_ + "mlp.fc2", m * torch.sigmoid(1.702 * m))
    m = _lin(w, p + "merger.mlp.0", _ln(w, p + "merger.ln_q", x, 1e-6).view(N // 4, 4 * E))
    return _lin(w, p + "merger.mlp.2", torch.nn.functional.gelu(m))


def _tower_blocks(w, prefix, n, x, nh, eps):
    """pre-norm blocks on x (images, tokens, E), full attention inside each image"""
    B, L, E = x.shape
    hd = E // nh
    for i in range(n):
        q_ = f"{prefix}encoder.layers.{i}."
        y = _ln(w, q_ + "layer_norm1", x, eps)
        q, k, v = (_lin(w, q_ + f"self_attn.{c}_proj", y).view(B, L, nh, hd).transpose(1, 2).reshape(B * nh, L, hd) for c in "qkv")
        o = _attend(q, k, v, hd ** -0.5).view(B, nh, L, hd).transpose(1, 2).reshape(B, L, E)
        x = x + _lin(w, q_ + "self_attn.out_proj", o)
        m = _lin(w, q_ + "mlp.fc1", _ln(w, q_ + "layer_norm2", x, eps))
        x = x + _lin(w, q_ + "mlp.fc2", m * torch.sigmoid(1.702 * m))
    return x


def _patches(pixels, ps):
    """(B, C, H, W) -> (B, patches, ps * ps * C)"""
    B, C, H, W = pixels.shape
    return pixels.double().view(B, C, H // ps, ps, W // ps, ps).permute(0, 2, 4, 3, 5, 1).reshape(B, -1, ps * ps * C)


def _exact_clip(case, seed):
    cfg, w, pixels = _clip_setup(case, seed)
    p, E = "vision_tower.vision_model.", 1024
    x = _patches(pixels, 14) @ _d(w, p + "embeddings.patch_embedding.weight").reshape(E, -1).T
    x = torch.cat([_d(w, p + "embeddings.class_embedding").expand(x.shape[0], 1, E), x], 1)
    x = _ln(w, p + "pre_layrnorm", x + _d(w, p + "embeddings.position_embedding.weight"), 1e-5)
    x = _tower_blocks(w, p, case["layers"] - 1, x, 16, 1e-5)[:, 1:]
    m = torch.nn.functional.gelu(_lin(w, "multi_modal_projector.linear_1", x))
    return _lin(w, "multi_modal_projector.linear_2", m)


def _exact_siglip(case, seed):
    cfg, w, pixels, mask = _siglip_setup(case, seed)
    E, side, n, p = 1152, case["side"] // 14, case["images"], "vision_model."
    x = _patches(torch.as_tensor(pixels[0], device="cuda"), 14) @ _d(w, p + "embeddings.patch_embedding.weight").reshape(E, -1).T
    # position buckets of a picture's valid rows and columns on the 70 x 70 grid; bucket -1 counts from the table's end
    ids, edges = np.zeros((n, side, side), dtype=np.int64), np.linspace(1 / 70, 1.0, 70, endpoint=False)
    for b in range(n):
        ok = mask[0, b].reshape(side, 14, side, 14).any((1, 3))
        nr, nc = int(ok[:, 0].sum()), int(ok[0].sum())
        row, col = (np.digitize(np.linspace(0, 1, m, endpoint=False), edges, right=True) - 1 for m in (nr, nc))
        ids[b, :nr, :nc] = row[:, None] * 70 + col
    pos = _d(w, p + "embeddings.position_embedding.weight")
    x = x + _d(w, p + "embeddings.patch_embedding.bias") + pos[torch.as_tensor(ids.reshape(n, -1) % pos.shape[0], device="cuda")]
    x = _ln(w, p + "post_layernorm", _tower_blocks(w, p, case["layers"], x, 16, 1e-6), 1e-5)

    def glu(q_, t):
        return _lin(w, q_ + "down_proj", torch.nn.functional.silu(_lin(w, q_ + "gate_proj", t)) * _lin(w, q_ + "up_proj", t))

    x = glu("connector.modality_projection.", x)
    r_ = "connector.perceiver_resampler."
    h, q_ = _d(w, r_ + "latents").expand(n, -1, -1), r_ + "layers.0."
    a = _rms(h, w[q_ + "input_latents_norm.weight"], 1e-5)
    both = torch.cat([_rms(x, w[q_ + "input_context_norm.weight"], 1e-5), a], 1)

    def split(t, heads):
        return t.view(n, t.shape[1], heads, 96).transpose(1, 2)

    q = split(_lin(w, q_ + "self_attn.q_proj", a), 16).reshape(n * 16, -1, 96)
    k, v = (split(_lin(w, q_ + f"self_attn.{c}_proj", both), 4).repeat_interleave(4, 1).reshape(n * 16, -1, 96) for c in "kv")
    o = _attend(q, k, v, 96 ** -0.5).view(n, 16, -1, 96).transpose(1, 2).reshape(n, -1, 1536)
    h = h + _lin(w, q_ + "self_attn.o_proj", o)
    h = h + glu(q_ + "mlp.", _rms(h, w[q_ + "post_attention_layernorm.weight"], 1e-5))
    return _rms(h, w[r_ + "norm.weight"], 1e-5).reshape(-1, h.shape[-1])


def _exact_latent(case, seed):
    cfg, w, rows, x = _latent_setup(case, seed)
    z, H, T, ctx = LATENT, case["heads"], case["tokens"], case["ctx"]
    dn, dr, dv, kr = z["dim"], z["rot_dim"], z["vdim"], z["kv_rank"]
    pos = torch.arange(ctx, ctx + T, device="cuda", dtype=torch.float64)
    ang = pos[:, None] * 10000.0 ** (-torch.arange(0, dr, 2, device="cuda", dtype=torch.float64) / dr)
    x, d = x.double(), {n: t.double() for n, t in w.items()}
    q = (_rms(x @ d["dq"].T, d["dq.norm"], 1e-5) @ d["uq"].T).view(T, H, dn + dr).transpose(0, 1)
    kv = x @ d["dkv"].T
    new = torch.cat([_rms(kv[:, :kr], d["dkv.norm"], 1e-5), _rotate(kv[:, kr:], ang)], -1)
    full = torch.cat([rows.double(), new])
    k = (full[:, :kr] @ d["uk"].T).view(-1, H, dn).transpose(0, 1)
    k = torch.cat([k, full[:, kr:].expand(H, -1, -1)], -1)
    v = (full[:, :kr] @ d["uv"].T).view(-1, H, dv).transpose(0, 1)
    q = torch.cat([q[..., :dn], _rotate(q[..., dn:], ang)], -1)
    o = _attend(q, k, v, cfg["scale"], torch.arange(ctx + 1, ctx + T + 1, device="cuda"))
    return {"y": o.transpose(0, 1).reshape(T, H * dv) @ d["o"].T, "rows": new}


def exact(case, seed):
    kind = case["kind"]
    if kind == "vit":
        return _exact_vit(case, seed)
    if kind == "clip":
        return _exact_clip(case, seed)
    if kind == "siglip":
        return _exact_siglip(case, seed)
    if kind == "latent":
        return _exact_latent(case, seed)
    r = _Rand(seed)
    H, I, nh, nkv = GEOMETRY[case["geometry"]]
    hd, layers, vocab = H // nh, case["layers"], case["vocab"]
    w = _lm_weights(r, case["geometry"], layers, vocab)
    _vit_weights(r, 1, VIT["embed_dim"], H)                      # the generator goes on where `prepare` does
    if kind == "prefill":
        T, ctx = case["tokens"], case["ctx"]
        old = r(layers, 2, 1, nkv, ctx, hd, dtype=torch.bfloat16)[:, :, 0]
        r.ints(0, vocab, 1, T)
        (logits, new), = _exact_lm(case, w, [(r(T, H, std=STD, dtype=torch.bfloat16), _prompt_positions(T, ctx)[:, 0], old)])
        return {"logits": logits[None], "kv": new}
    embed = w["language_model.model.embed_tokens.weight"]
    if kind == "prefill_rows":
        lens = _lengths(case)
        for n in lens:
            r.ints(0, vocab, 1, n)
        none = torch.zeros(layers, 2, nkv, 0, hd, device="cuda")
        got = _exact_lm(case, w, [(r(n, H, std=STD, dtype=torch.bfloat16), np.tile(np.arange(n), (3, 1)), none) for n in lens])
        return {"logits": got[-1][0][0], "kv": [new for _, new in got]}
    lens = [case["ctx"]] if kind == "decode" else _lengths(case)
    step = 256                                                   # capacity of the package's pools grows in such steps
    cap = -(-(max(lens) + 256) // step) * step
    pool = r(layers, 2, len(lens), nkv, cap, hd, dtype=torch.bfloat16)
    ids = torch.as_tensor(r.ints(0, vocab, len(lens), 1), device="cuda")
    got = _exact_lm(case, w, [(embed[ids[b]], np.full((3, 1), n), pool[:, :, b, :, :n]) for b, n in enumerate(lens)])
    if kind == "decode":
        return {"logits": got[0][0][None], "kv": got[0][1][..., 0, :]}
    return {"logits": torch.stack([lg for lg, _ in got]), "kv": [new[..., 0, :] for _, new in got]}
