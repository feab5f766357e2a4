"""The expanded form of latent attention on a prompt portion (csrc/attention_latent.cu, LatentAttention._expanded): the kernel alone
against float64 on the same operands, the layer against its absorbed form, and a wait that runs out."""
import os
import subprocess
import sys
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S,H,dn,dr,dv", [
    (1, 1, 1, 64, 0, 64), (128, 128, 2, 128, 64, 128), (129, 129, 2, 128, 64, 128), (127, 256, 3, 128, 64, 128), (128, 257, 2, 128, 0, 128),
    (300, 300, 2, 64, 32, 72), (2, 391, 2, 72, 8, 8), (257, 640, 1, 192, 0, 128), (255, 1023, 2, 128, 64, 120), (16, 16, 2, 16, 64, 16),
    (390, 900, 2, 8, 8, 24), (700, 701, 1, 64, 64, 64)])
@pytest.mark.parametrize("out_type", [torch.float32, torch.bfloat16])
def test_kernel(n, S, H, dn, dr, dv, out_type):
    """tile and group edges; rows behind the last key are NaN, as a cache's unused rows may be.  Bound: a weight is rounded
    to bf16 (2^-9), the sums are fp32: |error| <= 2^-8 sum p |v|, and the rounding of a bf16 output"""
    from mlx_vlm_b200 import _native as N
    lib = N.lm_lib()
    g = torch.Generator(device="cuda").manual_seed(n + S + dn)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    pad = S + 9
    q = mk(n, H, dn + dr)
    kv = torch.full((pad, H * (dn + dv) + 8), float("nan"), device="cuda", dtype=torch.bfloat16)
    kv[:S, :H * (dn + dv)] = mk(S, H * (dn + dv))
    rows = torch.full((pad, 24 + dr), float("nan"), device="cuda", dtype=torch.bfloat16)
    rows[:S] = mk(S, 24 + dr)
    q[n // 2] *= 6.0           # sharp rows: weights that grow along the keys move the reference of the row
    scale = 1.3 * (dn + dr) ** -0.5
    out = torch.full((n + 3, H * dv), 9.0, device="cuda", dtype=out_type)
    kr = rows[:, 24:]
    rc = lib.b200_lm_latent_expanded_attention(q.data_ptr(), H * (dn + dr), kv.data_ptr(), kv.stride(0), kr.data_ptr() if dr else 0,
                                               rows.stride(0), kv[:, H * dn:].data_ptr(), kv.stride(0), out.data_ptr(), H * dv,
                                               int(out_type == torch.float32), H, dn, dr, dv, n, S, scale, 0, 0)
    N.check(rc, "attention", lib)
    torch.cuda.synchronize()
    k = torch.cat([kv[:S, :H * dn].double().view(S, H, dn), rows[:S, None, 24:].double().expand(S, H, dr)], -1)
    v = kv[:S, H * dn:H * (dn + dv)].double().view(S, H, dv)
    s = torch.einsum("thd,shd->hts", q.double(), k) * scale
    seen = torch.arange(S, device="cuda")[None, :] <= torch.arange(S - n, S, device="cuda")[:, None]
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
    want = torch.einsum("hts,shd->thd", p, v).reshape(n, -1)
    bound = 2.0 ** -8 * torch.einsum("hts,shd->thd", p, v.abs()).reshape(n, -1)
    if out_type == torch.bfloat16:
        bound = bound + 2.0 ** -8 * want.abs()
    assert bool(((out[:n].double() - want).abs() <= bound + 1e-6).all())
    assert bool((out[n:] == 9.0).all())


@pytest.mark.parametrize("n,S", [(140, 140), (130, 400)])
def test_scores_that_are_not_finite(n, S):
    """infinities and NaN in a query or a key: NaN exactly where float64's softmax gives it (a row whose scores hold +inf or NaN, or
    nothing but -inf), the other rows untouched; a key behind a query's last visible one does not reach it"""
    from mlx_vlm_b200 import _native as N
    lib = N.lm_lib()
    H, dn, dr, dv = 2, 64, 0, 64
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = mk(n, H, dn), mk(S, H, dn), mk(S, H, dv)
    q[:, :, 0] = q[:, :, 0].abs() + 0.1
    q[n // 3, 0, 5] = float("nan")
    q[n // 2, 1, 7] = float("inf")
    k[S - 60, 0, 0] = float("-inf")            # weight 0 for every query that sees it
    k[S - 20, 0, 0] = float("inf")
    k[S - 2, 1, 3] = float("nan")
    if n == S:
        k[0, 1, 0] = float("-inf")             # the first query's only key
    out = torch.empty(n, H * dv, device="cuda")
    N.check(lib.b200_lm_latent_expanded_attention(q.data_ptr(), H * dn, k.data_ptr(), H * dn, 0, 0, v.data_ptr(), H * dv, out.data_ptr(),
                                                  H * dv, 1, H, dn, dr, dv, n, S, 0.11, 0, 0), "attention", lib)
    torch.cuda.synchronize()
    s = torch.einsum("thd,shd->hts", q.double(), k.double()) * 0.11
    seen = torch.arange(S, device="cuda")[None, :] <= torch.arange(S - n, S, device="cuda")[:, None]
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
    want = torch.einsum("hts,shd->thd", p, v.double()).reshape(n, -1)
    bound = 2.0 ** -8 * torch.einsum("hts,shd->thd", p, v.double().abs()).reshape(n, -1) + 1e-6     # as in test_kernel
    bad = torch.isnan(want)
    # two queries; the 20 that see key S - 20 and the 2 that see S - 2, each in its head; the first query where all it sees is -inf
    assert torch.equal(torch.isnan(out), bad) and int(bad.sum()) == (24 + (n == S)) * dv
    assert bool(((out.double() - want).abs() <= bound)[~bad].all())


def _layer(H, dn, dr, dv, r, q_rank, pairs, gated, pool_extra, seed, kv_from=None):
    from mlx_vlm_b200.models.cache import LatentPool
    from mlx_vlm_b200.models.decoder_blocks import LatentAttention
    W = 256
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s: (0.06 * torch.randn(*s, device="cuda", generator=g)).to(torch.bfloat16)
    m = LatentAttention(0, {"heads": H, "dim": dn, "rot_dim": dr, "vdim": dv, "kv_rank": r, "q_rank": q_rank, "scale": (dn + dr) ** -0.5,
                            "rot": {"base": 10000.0, "dims": dr}, "kv_from": kv_from}, W, rotation="pairs" if pairs else "half", gated=gated)
    m.cache_index = 0
    w = {n: 1 + mk(*s) if n.endswith("norm") else mk(*s) for n, s in m.checkpoint_tensors("").items()}
    arena = {n: torch.empty(s, device="cuda", dtype=torch.bfloat16) for n, s in m.manifest("")}
    m.pack("", w, arena.__getitem__)
    pool = LatentPool(1, r + dr + pool_extra, torch.device("cuda", 0), batch=3, capacity=2048)
    pool.buf.copy_(torch.randn(pool.buf.shape, device="cuda", generator=g))
    return m, pool, torch.randn(1200, W, device="cuda", generator=g)


@pytest.mark.parametrize("H,dn,dr,dv,r,q_rank,pairs,gated,pool_extra", [
    (4, 128, 64, 128, 512, 96, False, False, 0), (3, 64, 32, 64, 64, 0, True, False, 8), (2, 64, 0, 128, 128, 64, False, "head", 0),
    (4, 128, 64, 64, 192, 0, False, "element", 0), (3, 64, 64, 72, 64, 32, True, False, 0)])
@pytest.mark.parametrize("segs", [[(0, 128, 1, 0)], [(0, 333, 0, 77)], [(0, 130, 2, 0), (130, 256, 0, 1030)]])
def test_layer_against_its_absorbed_form(H, dn, dr, dv, r, q_rank, pairs, gated, pool_extra, segs):
    """the same cached rows and, from float64's view, no further from the absorbed form on the row kernels (fp32 queries, weights
    and sums) than the absorbed form on the tensor cores is"""
    from mlx_vlm_b200.models.decoder_blocks import StepCtx
    from mlx_vlm_b200.models.layer_ops import LayerOps
    m, pool, x = _layer(H, dn, dr, dv, r, q_rank, pairs, gated, pool_extra, H + dn + r)
    assert m.expands
    T = sum(n for _, n, _, _ in segs)
    slot = torch.cat([torch.full((n,), s, dtype=torch.int32) for _, n, s, _ in segs]).cuda()
    pos = torch.cat([torch.arange(p, p + n, dtype=torch.int32) for _, n, _, p in segs]).cuda()
    cached = pool.buf.clone()
    got = {}
    for form in ("expanded", "absorbed", "rows"):
        pool.buf.copy_(cached)
        ops = LayerOps("cuda:0", torch.cuda.Stream())
        ops.tc_enabled = form != "rows"
        m.expands = form == "expanded"
        torch.cuda.synchronize()
        with ops.on_stream():
            y = m.forward(StepCtx(ops, slot, pos, pool, 1e-5, segments=segs), x[:T].contiguous())
        torch.cuda.synchronize()
        assert ops.tc_enabled == (form != "rows")
        got[form] = (y.double(), pool.buf.clone())
    assert torch.equal(got["expanded"][1], got["absorbed"][1])
    err = lambda f: float((got[f][0] - got["rows"][0]).norm() / got["rows"][0].norm())
    assert err("expanded") < max(1.1 * err("absorbed"), 2.0 ** -8), (err("expanded"), err("absorbed"))


@pytest.mark.parametrize("segs", [[(0, 128, 1, 0)], [(0, 130, 2, 0), (130, 256, 0, 1030)]])
def test_a_layer_that_borrows_its_latent(segs):
    """own rows are neither normed nor written: the slots stay as they are, the launches go out in one call"""
    from mlx_vlm_b200.models.decoder_blocks import StepCtx
    from mlx_vlm_b200.models.layer_ops import LayerOps
    m, pool, x = _layer(4, 128, 64, 128, 512, 96, False, False, 0, 3, kv_from=0)
    assert m.expands and not m.own_kv
    T = sum(n for _, n, _, _ in segs)
    slot = torch.cat([torch.full((n,), s, dtype=torch.int32) for _, n, s, _ in segs]).cuda()
    pos = torch.cat([torch.arange(p, p + n, dtype=torch.int32) for _, n, _, p in segs]).cuda()
    cached = pool.buf.clone()
    got = {}
    for form in ("expanded", "absorbed", "rows"):
        ops = LayerOps("cuda:0", torch.cuda.Stream())
        ops.tc_enabled = form != "rows"
        m.expands = form == "expanded"
        torch.cuda.synchronize()
        with ops.on_stream():
            y = m.forward(StepCtx(ops, slot, pos, pool, 1e-5, segments=segs), x[:T].contiguous())
        torch.cuda.synchronize()
        assert ops.tc_enabled == (form != "rows") and torch.equal(pool.buf, cached)
        got[form] = y.double()
    err = lambda f: float((got[f] - got["rows"]).norm() / got["rows"].norm())
    assert err("expanded") < max(1.1 * err("absorbed"), 2.0 ** -8), (err("expanded"), err("absorbed"))


@pytest.mark.parametrize("gated", [False, "head"])
def test_operand_rows_written_by_the_norm_before(gated):
    """where the norm ahead left the step's bf16 operand rows (StepCtx.x_operand) they are read instead of x: the same sums"""
    from mlx_vlm_b200.models.decoder_blocks import StepCtx
    from mlx_vlm_b200.models.layer_ops import LayerOps
    m, pool, x = _layer(4, 128, 64, 128, 512, 96, False, gated, 0, 5)
    T, x = 300, x[:300].contiguous()
    slot, pos = torch.zeros(T, dtype=torch.int32).cuda(), torch.arange(T, dtype=torch.int32).cuda()
    ops, got = LayerOps("cuda:0", torch.cuda.Stream()), []
    torch.cuda.synchronize()
    with ops.on_stream():
        for xb in (None, ops.to_bf16(x, x.shape[1])):
            got.append(m.forward(StepCtx(ops, slot, pos, pool, 1e-5, segments=[(0, T, 0, 0)], x_operand=xb),
                                 x if xb is None else torch.full_like(x, float("nan"))))
    torch.cuda.synchronize()
    assert ops.tc_enabled and torch.equal(*got)


def test_what_keeps_the_absorbed_form():
    from mlx_vlm_b200.models.decoder_blocks import EXPANDED_MAX, LatentAttention
    base = {"heads": 4, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 64, "scale": 0.1}
    assert LatentAttention(0, base, 64).expands
    for change in ({"mask": {"size": 9}}, {"dim": 60}, {"dim": 136}, {"rot_dim": 72}, {"vdim": 136}, {"vdim": 4}, {"kv_rank": 68}, {"scale": -1.0}):
        m = LatentAttention(0, {**base, **change}, 64)
        assert not m.expands and any(n == "uv" for n, _ in m.manifest("")), change
    assert not LatentAttention(0, base, 64, split_weights=True).expands
    m = LatentAttention(0, base, 64)
    ops = types.SimpleNamespace(tc_ok=lambda n, *k: n >= 128 and all(v % 8 == 0 for v in k))
    rows = torch.empty(2, 4, 96, dtype=torch.bfloat16, device="cuda")
    per = 4 * 128
    assert m._expand_portions(ops, [(0, 200, 0, 0)], rows)
    assert not m._expand_portions(ops, [(0, 200, 0, 0), (200, 100, 1, 0)], rows)             # a short portion
    assert not m._expand_portions(ops, [(0, 200, 0, EXPANDED_MAX // per)], rows)             # too long a context
    assert m._expand_portions(ops, [(0, 200, 0, 8192 - 200)], rows) and m._expand_portions(ops, [(0, 512, 0, 100000)], rows)
    assert not m._expand_portions(ops, [(0, 200, 0, 8193 - 200)], rows)                      # few heads and tokens, many keys
    assert not m._expand_portions(ops, [(0, 512, 0, 100000), (512, 511, 1, 8192)], rows)
    assert not m._expand_portions(ops, None, rows) and not m._expand_portions(ops, [(0, 200, 0, 0)], rows.float())
    assert not m._expand_portions(ops, [(0, 200, 0, 0)], rows[..., 4:])                       # rows that do not start on 16 bytes


_CHILD = """
import sys, ctypes as C, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lm_lib()
def state():
    v = C.c_int(-1)
    N.check(lib.b200_wait_error(C.byref(v)), "wait", lib)
    return v.value
T, S = {T}, {S}
q, k, kr, v = (torch.randn(n, d, device="cuda").to(torch.bfloat16) for n, d in ((T, 192), (S, 128), (S, 64), (S, 128)))
out = torch.zeros(T, 128, device="cuda")
def run(flags):
    out.zero_()
    torch.cuda.synchronize()
    N.check(lib.b200_lm_latent_expanded_attention(q.data_ptr(), 192, k.data_ptr(), 128, kr.data_ptr(), 64, v.data_ptr(), 128, out.data_ptr(),
                                                  128, 1, 1, 128, 64, 128, T, S, 0.1, flags, 0), "attention", lib)
    torch.cuda.synchronize()
    return out.clone()
a = run(0)
assert bool(torch.isfinite(a).all()) and state() == 0
b = run(1)                            # nothing is loaded: the waits run out after a second
assert bool(torch.isnan(b).all()) and state() == 8, (b, state())
assert torch.equal(run(0), a) and state() == 8
"""


@pytest.mark.parametrize("T,S", [(5, 7), (300, 700)])
def test_a_wait_that_runs_out_is_told(T, S):
    """in a process of its own: NaN, the word that the host reads, and the next launch as if nothing had been"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, T=T, S=S)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
