"""The row kernels of the fp32 towers (csrc/tower_f32.cu) at the edges of their forms: LayerNorm with a CTA or a warp per row, pixels of
any strides, rows without their class token, sums rounded once to bf16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def eng():
    import types
    from mlx_vlm_b200 import _native as N
    stream = torch.cuda.Stream()      # (the default stream cannot be captured, and a GEMM's first call measures in captures)
    with torch.cuda.stream(stream):
        yield types.SimpleNamespace(lib=N.lib(), stream=stream, device=torch.device("cuda", 0), s=stream.cuda_stream)


def _parts(buf):
    t = buf.t.double()
    return t[:, :buf.n] + t[:, buf.n_pad:buf.n_pad + buf.n], t


@pytest.mark.parametrize("T,n", [(1183, 1024), (1184, 1024), (1191, 1152), (1200, 1028), (1185, 4), (1186, 2048), (1184, 2052), (1, 1024), (1187, 1280), (1190, 1284)])
def test_layer_norm(eng, T, n):
    """Bound: the mean and the differences round at the size of the row's numbers, at most 8 x 2^-24 of the largest, which a
    division by the deviation makes larger (rows of four numbers may hardly deviate); the rest is a few roundings of the
    result.  The split keeps 16 mantissa bits"""
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    g = torch.Generator(device="cuda").manual_seed(T + n)
    wide = torch.randn(T, n + 4, device="cuda", generator=g) * 2 + 3
    x = wide[:, :n]
    w, b = (torch.randn(n, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    out32, sp = torch.full((T + 2, n), 7.0, device="cuda"), SplitBuf(eng, T, n)
    TowerOps(eng).layer_norm(x, w, b, 1e-5, out32=out32[:T], out_split=sp)
    torch.cuda.synchronize()
    want = torch.nn.functional.layer_norm(x.double(), (n,), eps=1e-5) * w.double() + b.double()
    xd = x.double()
    rstd = 1.0 / (xd.var(1, unbiased=False, keepdim=True) + 1e-5).sqrt()
    bound = 2.0 ** -21 * (xd.abs().amax(1, keepdim=True) * rstd * w.double().abs() + want.abs() + b.double().abs())
    assert bool(((out32[:T].double() - want).abs() <= bound).all()) and bool((out32[T:] == 7.0).all())
    both, raw = _parts(sp)
    assert bool(((both - want).abs() <= bound + 2.0 ** -16 * want.abs()).all())
    assert not raw[:, n:sp.n_pad].any() and not raw[:, sp.n_pad + n:].any()


@pytest.mark.parametrize("B,H,W,C,ps", [(1, 14, 14, 3, 14), (3, 28, 126, 3, 14), (2, 30, 50, 3, 10), (1, 16, 272, 1, 16), (2, 21, 7, 4, 7)])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (0, 3, 1, 2), (3, 2, 1, 0)])
def test_patches_of_pixels_in_any_order(eng, B, H, W, C, ps, order):
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    pix = torch.randn(B, H, W, C, device="cuda")
    lie = pix.permute(order).contiguous()                       # how the pixels lie; read through a view
    view = lie.permute([order.index(i) for i in range(4)])
    assert torch.equal(view, pix)
    K = ps * ps * C
    sp = SplitBuf(eng, B * (H // ps) * (W // ps), K, padded=True)
    sp.t.fill_(float("nan"))
    TowerOps(eng).patchify(view, ps, sp)
    torch.cuda.synchronize()
    want = pix.view(B, H // ps, ps, W // ps, ps, C).permute(0, 1, 3, 2, 4, 5).reshape(-1, K)
    hi = want.to(torch.bfloat16)
    lo = (want - hi.float()).to(torch.bfloat16)
    pad = torch.zeros(want.shape[0], sp.n_pad - K, device="cuda", dtype=torch.bfloat16)
    assert torch.equal(sp.t, torch.cat([hi, pad, lo, pad], 1))


@pytest.mark.parametrize("n_seg,seg,skip,n", [(1, 5, 1, 8), (3, 577, 1, 1024), (4, 16, 0, 100), (2, 9, 8, 4)])
def test_rows_without_their_first(eng, n_seg, seg, skip, n):
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    x = torch.randn(n_seg * seg, n, device="cuda")
    sp = SplitBuf(eng, n_seg * (seg - skip), n)
    TowerOps(eng).split_segments(x, seg, skip, sp)
    torch.cuda.synchronize()
    want = x.view(n_seg, seg, n)[:, skip:].reshape(-1, n)
    hi = want.to(torch.bfloat16)
    assert torch.equal(sp.t[:, :n], hi) and torch.equal(sp.t[:, sp.n_pad:sp.n_pad + n], (want - hi.float()).to(torch.bfloat16))
    assert not sp.t[:, n:sp.n_pad].any()


@pytest.mark.parametrize("T,n,K", [(130, 256, 128), (577, 200, 1000), (1, 8, 64)])
def test_sums_rounded_once(eng, T, n, K):
    """the bf16 rows are the fp32 rows of the same sums, rounded (another tile order may move a sum by an fp32 ulp)"""
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    ops, x = TowerOps(eng), torch.randn(T, K, device="cuda")
    w, b = (0.1 * torch.randn(n, K, device="cuda")).to(torch.bfloat16), torch.randn(n, device="cuda").to(torch.bfloat16)
    sp, o32, o16 = SplitBuf(eng, T, K), torch.empty(T, n, device="cuda"), torch.empty(T, n, device="cuda", dtype=torch.bfloat16)
    ops.split(x, sp)
    ops.linear(sp, w, b, out32=o32)
    ops.linear_bf16(sp, w, b, o16)
    torch.cuda.synchronize()
    assert ((o16.float() - o32).abs() <= 2.0 ** -8 * o32.abs() + 1e-5).all()
    assert (o16 != o32.to(torch.bfloat16)).float().mean() < 0.01


@pytest.mark.parametrize("T", [1, 63, 130, 600, 2500])
@pytest.mark.parametrize("inter,K,bias", [(64, 64, False), (132, 200, True), (4, 128, True), (3420, 1280, True), (1000, 320, False)])
def test_swiglu_in_the_product(eng, T, inter, K, bias):
    """against float64 on the same operands.  x keeps 16 mantissa bits (2^-17 of each term), the sums are fp32 (truncated: 2^-23
    a step), the logistic function is good to a few fp32 ulps, the result keeps 16 mantissa bits"""
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    g = torch.Generator(device="cuda").manual_seed(T + inter)
    ops, x = TowerOps(eng), torch.randn(T, K, device="cuda", generator=g)
    w = (torch.randn(2 * inter, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    b = torch.randn(2 * inter, device="cuda", generator=g).to(torch.bfloat16) if bias else None
    sp, out = SplitBuf(eng, T, K), SplitBuf(eng, T, inter)
    ops.split(x, sp)
    ops.linear_swiglu(sp, w, b, out)
    torch.cuda.synchronize()
    wd, bd = w.double(), b.double() if bias else torch.zeros(2 * inter, device="cuda", dtype=torch.float64)
    y, size = x.double() @ wd.T + bd, x.double().abs() @ wd.abs().T + bd.abs()
    gate, up = y[:, :inter], y[:, inter:]
    want = torch.nn.functional.silu(gate) * up
    err = (2.0 ** -17 + (K / 16 + 8) * 2.0 ** -23) * size          # of the two sums
    bound = 1.1 * err[:, :inter] * (up.abs() + err[:, inter:]) + gate.abs() * err[:, inter:] + 2.0 ** -16 * want.abs() + 1e-30
    both, raw = _parts(out)
    assert bool(((both - want).abs() <= bound).all())
    assert not raw[:, inter:out.n_pad].any() and not raw[:, out.n_pad + inter:].any()


@pytest.mark.parametrize("T,inter", [(1, 4), (577, 1028), (130, 4304)])
def test_swiglu_of_rows(eng, T, inter):
    """the C entry for gate and up rows that lie in memory: fp32 arithmetic (a few ulps), the result keeps 16 mantissa bits"""
    from mlx_vlm_b200 import _native as N
    from mlx_vlm_b200.models.tower_ops import SplitBuf
    gu = 3 * torch.randn(T, 2 * inter + 4, device="cuda")
    out = SplitBuf(eng, T, inter)
    N.check(eng.lib.b200_f32_swiglu_split(gu.data_ptr(), gu.stride(0), out.t.data_ptr(), out.ld, out.n_pad, T, inter, eng.s), "swiglu")
    torch.cuda.synchronize()
    want = torch.nn.functional.silu(gu[:, :inter].double()) * gu[:, inter:2 * inter].double()
    both, raw = _parts(out)
    assert bool(((both - want).abs() <= (2.0 ** -16 + 2.0 ** -20) * want.abs() + 1e-30).all())
    assert not raw[:, inter:out.n_pad].any() and not raw[:, out.n_pad + inter:].any()


def test_patches_of_channel_last_pixels(eng):
    """the C entry without strides reads (B, H, W, C) as it lies"""
    from mlx_vlm_b200 import _native as N
    from mlx_vlm_b200.models.tower_ops import SplitBuf, TowerOps
    pix = torch.randn(2, 28, 42, 3, device="cuda")
    a, b = (SplitBuf(eng, 2 * 2 * 3, 588, padded=True) for _ in range(2))
    TowerOps(eng).patchify(pix, 14, a)
    N.check(eng.lib.b200_clip_patchify(pix.data_ptr(), 2, 28, 42, 3, 14, b.t.data_ptr(), b.n_pad, eng.s), "clip_patchify")
    torch.cuda.synchronize()
    assert torch.equal(a.t, b.t)
