"""One decoded token of one layer against float64, for every form of the decode kernels: two q heads a CTA (Mistral), three and four of
four slots (Qwen2-VL-2B, 7B), the per-phase kernels (32 kv heads); contexts at which a CTA's trips over keys and values begin and end
(its share is an eighth of the keys, a trip 64 or 128 of them); a vocabulary whose tiles fill no whole batch of any CTA.

Bound: the bf16 roundings of such layers leave 0.016 - 0.036 of the result over two to four of them; 0.04 here."""
import pytest
import torch

from perf import cases as C

pytestmark = pytest.mark.gpu
CONTEXTS = {"mistral-7b": (1, 8, 1023, 1024, 1025, 2049, 5000), "qwen2-vl-2b": (1, 7, 511, 513, 1030, 2600),
            "qwen2-vl-7b": (3, 512, 1100), "llama-7b": (1, 300, 4500)}


@pytest.mark.parametrize("geometry,ctx", [(g, c) for g, cs in CONTEXTS.items() for c in cs])
def test_token(geometry, ctx):
    case = {"kind": "decode", "geometry": geometry, "layers": 1, "vocab": 10661, "ctx": ctx}
    got = C.run(C.prepare(case, ctx))
    want = C.exact(case, ctx)
    for name in ("logits", "kv"):
        a, b = got[name].double(), want[name].double().reshape(got[name].shape)
        assert float((a - b).norm() / b.norm()) <= 0.04, name
