"""The GEMM of CTA pairs (csrc/gemm_wt.cu: gemm_wt_pair_kernel) at the edges of its tiles: 256 weight rows (128 / SwiGLU: 64 channels
per CTA of the pair), token tiles of 128 .. 256, k-blocks of 64, one and several tiles per pair, split-K.

Bound: bf16 products are exact in fp32, sums of K of them err by less than 2^-20 here, outputs are rounded to bf16 (2^-9): the
relative L2 distance from the rounded float64 result stays below 1e-3 (single roundings that fall the other way)."""
import os
import subprocess
import sys

import pytest
import torch

from _util import rl2

pytestmark = pytest.mark.gpu
PAIR = 8          # B200_WT_FLAG_PAIR


@pytest.fixture(scope="module")
def lib():
    from mlx_vlm_b200 import _native as N
    return N.lib()


def _rand(*shape, seed, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * std).to(torch.bfloat16)


def _call(lib, x, w, bias, res, out, part, N, epi, mode, inter, cfg):
    import ctypes
    from mlx_vlm_b200 import _native as Nn
    T, K = x.shape
    c = (ctypes.c_int * 4)(*cfg)
    Nn.check(lib.b200_gemm_wt(x.data_ptr(), K, w.data_ptr(), Nn.ptr(bias), Nn.ptr(res), 0 if res is None else res.shape[1],
                              Nn.ptr(out), 0 if out is None else out.shape[1], Nn.ptr(part), T, N, K, epi, mode, inter, c, PAIR, 0),
             "gemm_wt")
    torch.cuda.synchronize()


# (T, N, K, TN, stages): one tile and less | ragged tokens, rows and k | more tiles than pairs | an odd row count
@pytest.mark.parametrize("T,N,K,TN,stages", [(1, 8, 64, 64, 2), (128, 256, 64, 128, 4), (129, 257, 72, 128, 3), (300, 520, 1000, 224, 6),
                                             (1000, 3000, 256, 256, 6), (2100, 2600, 192, 160, 5), (513, 131, 4096, 192, 2)])
def test_bf16_with_bias_and_residual(lib, T, N, K, TN, stages):
    x, w, b, r = _rand(T, K, seed=1), _rand(N, K, seed=2, std=K ** -0.5), _rand(N, seed=3), _rand(T, N, seed=4)
    y = x.double() @ w.double().T
    ldn = (N + 7) // 8 * 8
    plain = torch.full((T, ldn), 9.0, dtype=torch.bfloat16, device="cuda")
    _call(lib, x, w, None, None, plain, None, N, 0, 0, 0, (TN, 1, stages, 1))
    assert rl2(plain[:, :N], y.to(torch.bfloat16)) <= 1e-3 and bool((plain[:, N:] == 9.0).all())
    got = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    _call(lib, x, w, b, r, got, None, N, 0, 0, 0, (TN, 1, stages, 1))
    want = ((y + b.double()).to(torch.bfloat16).double() + r.double()).to(torch.bfloat16)
    assert rl2(got, want) <= 1e-3


@pytest.mark.parametrize("T,inter,K,TN", [(128, 64, 64, 128), (257, 200, 320, 256), (700, 1032, 128, 192), (64, 4096, 64, 64)])
def test_swiglu(lib, T, inter, K, TN):
    x, w = _rand(T, K, seed=5), _rand(2 * inter, K, seed=6, std=K ** -0.5)
    got = torch.full((T, inter), 9.0, dtype=torch.bfloat16, device="cuda")
    _call(lib, x, w, None, None, got, None, 2 * inter, 0, 2, inter, (TN, 1, 4, 1))
    g, u = ((x.double() @ w.double().T).to(torch.bfloat16).double()).split(inter, 1)
    # three roundings of the unit, one of each product: 4 x 2^-9, most of them shared with the reference's
    assert rl2(got, torch.nn.functional.silu(g) * u) <= 2.0 ** -8


@pytest.mark.parametrize("T,N,K,TN,split", [(200, 300, 512, 128, 2), (600, 1280, 5120, 192, 4), (33, 64, 192, 64, 3), (900, 640, 64, 256, 1)])
def test_split_k_partials(lib, T, N, K, TN, split):
    x, w = _rand(T, K, seed=7), _rand(N, K, seed=8, std=K ** -0.5)
    part = torch.full((split, T, N), float("nan"), device="cuda")
    _call(lib, x, w, None, None, None, part, N, 0, 1, 0, (TN, 1, 4, split))
    assert rl2(part.double().sum(0), x.double() @ w.double().T) <= 1e-5


_CHILD = """
import sys, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
g = torch.Generator(device="cuda").manual_seed(9)
for T, n, K, mode, epi in {cases!r}:
    kp = (K + 63) // 64 * 64
    x = torch.randn(T, K, generator=g, device="cuda")
    xs = torch.zeros(T, 2 * kp, dtype=torch.bfloat16, device="cuda")
    xs[:, :K] = x.to(torch.bfloat16); xs[:, kp:kp + K] = (x - xs[:, :K].float()).to(torch.bfloat16)
    w = (torch.randn(n, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    b = torch.randn(n, generator=g, device="cuda").to(torch.bfloat16)
    r = torch.randn(T, n, generator=g, device="cuda")
    y = (xs[:, :K].double() + xs[:, kp:kp + K].double()) @ w.double().T + b.double()
    if epi == 2: y = torch.nn.functional.gelu(y)
    npad = (n + 63) // 64 * 64
    o32, osp = torch.zeros(T, n, device="cuda"), torch.zeros(T, 2 * npad, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        N.check(lib.b200_gemm_wt_f32(xs.data_ptr(), 2 * kp, w.data_ptr(), K, b.data_ptr(), r.data_ptr() if mode == 3 else 0, n,
                                     o32.data_ptr(), n, osp.data_ptr(), 2 * npad, npad, T, n, K, 2, epi, mode, 0), "f32")
    torch.cuda.synchronize()
    got = o32.double() - r.double() if mode == 3 else osp[:, :n].double() + osp[:, npad:npad + n].double()
    e = float((got - y).norm() / y.norm())
    print(T, n, K, mode, e)
    assert e <= (2e-6 if mode == 3 else 2.0 ** -17), e
"""


def test_fp32_outputs_of_split_operands(tmp_path):
    """the fp32-accurate modes, with the configuration given by a file of measured choices (k-blocks per stage 0: pairs)"""
    cases = [(300, 264, 128, 3, 0), (577, 1152, 584, 3, 2), (640, 520, 72, 4, 2), (200, 256, 1152, 4, 0)]
    lines = []
    for T, n, K, mode, _ in cases:
        lines.append(f"{(T + 63) // 64} {n} {2 * ((K + 63) // 64 * 64)} {mode} 0 160 0 4 1")
    path = tmp_path / "choices.txt"
    path.write_text("\n".join(lines) + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, cases=cases)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200_WT_TUNE_FILE=str(path)))
    assert r.returncode == 0, r.stdout + r.stderr
    assert path.read_text() == "\n".join(lines) + "\n"        # nothing was measured: the file's choices ran


_CHILD_HEADS = """
import sys, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
T, n, K, heads = 300, 256, 64, 3
g = torch.Generator(device="cuda").manual_seed(10)
x = torch.randn(T, heads * K, generator=g, device="cuda").to(torch.bfloat16)
w = (torch.randn(heads, n, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
one, out = torch.zeros(T, n, device="cuda"), torch.zeros(T, heads * n, device="cuda")
torch.cuda.synchronize()
stream = torch.cuda.Stream()       # (choices are measured under capture, which the default stream does not take)
for _ in range(2):
    N.check(lib.b200_gemm_wt_f32(x.data_ptr(), heads * K, w.data_ptr(), K, 0, 0, 0, one.data_ptr(), n, 0, 0, 0, T, n, K, 1, 0, 3,
                                 stream.cuda_stream), "f32")
    N.check(lib.b200_gemm_wt_f32_heads(x.data_ptr(), heads * K, heads * K, K, w.data_ptr(), K, out.data_ptr(), heads * n, n, T, heads,
                                       n, K, 1, 0, stream.cuda_stream), "heads")
torch.cuda.synchronize()
want = torch.einsum("thk,hnk->thn", x.double().view(T, heads, K), w.double())
for got, ref in ((one, want[:, 0]), (out.view(T, heads, n), want)):
    e = float((got.double() - ref).norm() / ref.norm())
    print(e)
    assert e <= 2e-6, e
"""


@pytest.mark.parametrize("line", ["5 256 64 3 0 160 0 4 1", "5 256 64 3 0 160 0 4 1\n5 256 64 3 0 160 0 4 1 3"])
def test_column_groups_beside_a_plain_product_of_pairs(tmp_path, line):
    """a per-head product of the tokens, rows and k of a plain one that runs on pairs keeps a choice of its own; a file's line that
    gives pairs to column groups is passed over"""
    path = tmp_path / "choices.txt"
    path.write_text(line + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD_HEADS.format(root=root)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200_WT_TUNE_FILE=str(path)))
    assert r.returncode == 0, r.stdout + r.stderr
    added = path.read_text()[len(line) + 1:].split()
    assert added[:5] == ["5", "256", "64", "3", "0"] and int(added[6]) >= 1 and added[9] == "3" and len(added) == 10


_CHILD_WAIT = """
import sys, ctypes as C, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
def state():
    v = C.c_int(-1)
    N.check(lib.b200_wait_error(C.byref(v)))
    return v.value
T, n, K = {T}, {n}, {K}
x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
w = torch.randn(n, K, device="cuda").to(torch.bfloat16)
cfg = (C.c_int * 4)(128, 1, 4, 1)
out = torch.zeros(T, n, device="cuda", dtype=torch.bfloat16)
def run(flags):
    out.zero_()
    torch.cuda.synchronize()
    N.check(lib.b200_gemm_wt(x.data_ptr(), K, w.data_ptr(), 0, 0, 0, out.data_ptr(), n, 0, T, n, K, 0, 0, 0, cfg, 8 | flags, 0))
    torch.cuda.synchronize()
want = (x.double() @ w.double().T).to(torch.bfloat16)
run(0)
assert torch.allclose(out.float(), want.float(), atol=0.5) and state() == 0
run(2)                                # nothing is loaded: the waits run out after a second
assert bool(torch.isnan(out.float()).all()) and state() == 5, (out, state())
run(0)
assert torch.allclose(out.float(), want.float(), atol=0.5) and state() == 5
"""


# fewer k-blocks than the ring has stages; several tiles of a pair and several rounds of the ring
@pytest.mark.parametrize("T,n,K", [(128, 256, 64), (1300, 4096, 640)])
def test_a_wait_that_runs_out_is_told(T, n, K):
    """in a process of its own: NaN instead of an accumulator that is not whole, the word that the host reads, and the next launch
    as if nothing had been"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD_WAIT.format(root=root, T=T, n=n, K=K)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


# ---- wide pairs: 512 weight rows (SwiGLU: 256 channels) a pair, the second half's products a few k-blocks behind the first's
WIDE = 16         # B200_WT_FLAG_WIDE


# one k-block and fewer of them than twice the lag | one row more or less than a half, a tile | more tiles than pairs, several
# rounds of the ring
@pytest.mark.parametrize("T,N,K,TN,stages", [(1, 8, 64, 64, 3), (129, 256, 128, 128, 4), (130, 257, 200, 256, 4), (256, 520, 320, 224, 3),
                                             (300, 1030, 392, 192, 2), (2100, 10000, 576, 256, 4), (513, 131, 4096, 192, 4)])
def test_wide_pairs_give_what_pairs_give(lib, T, N, K, TN, stages):
    """the same sums in the same order: bit for bit the output of the pairs of 256 rows, which the tests above hold to float64"""
    import ctypes
    from mlx_vlm_b200 import _native as Nn
    x, w, b, r = _rand(T, K, seed=11), _rand(N, K, seed=12, std=K ** -0.5), _rand(N, seed=13), _rand(T, N, seed=14)
    ld = (N + 7) // 8 * 8
    for epi, mode, inter, bias, res in ((0, 0, 0, b, r), (1, 0, 0, b, None), (2, 0, 0, None, None), (0, 2, N // 16 * 8, None, None)):
        n = 2 * inter if mode == 2 else N
        if n == 0:
            continue
        outs = []
        for flag in (PAIR, WIDE):
            out = torch.full((T, ld), 9.0, dtype=torch.bfloat16, device="cuda")
            Nn.check(lib.b200_gemm_wt(x.data_ptr(), K, w.data_ptr(), Nn.ptr(bias), Nn.ptr(res), N if res is not None else 0, out.data_ptr(),
                                      ld, 0, T, n, K, epi, mode, inter, (ctypes.c_int * 4)(TN, 1, stages, 1), flag, 0), "gemm_wt")
            outs.append(out)
        torch.cuda.synchronize()
        assert torch.equal(*outs), (epi, mode)
        assert bool((outs[1][:, inter or N:] == 9.0).all()) and not bool((outs[1][:, :inter or N] == 9.0).all())


def test_wide_pairs_take_no_partials(lib):
    import ctypes
    x, w = _rand(64, 128, seed=15), _rand(64, 128, seed=16)
    part = torch.empty(2, 64, 64, device="cuda")
    assert lib.b200_gemm_wt(x.data_ptr(), 128, w.data_ptr(), 0, 0, 0, 0, 0, part.data_ptr(), 64, 64, 128, 0, 1, 0,
                            (ctypes.c_int * 4)(64, 1, 4, 2), WIDE, 0) != 0


def test_fp32_outputs_of_wide_pairs(tmp_path):
    """as test_fp32_outputs_of_split_operands, with a file that gives wide pairs (k-blocks per stage -1)"""
    cases = [(300, 264, 128, 3, 0), (577, 1152, 584, 3, 2), (640, 520, 72, 4, 2), (200, 1000, 1152, 4, 0)]
    lines = [f"{(T + 63) // 64} {n} {2 * ((K + 63) // 64 * 64)} {mode} 0 {tn} -1 4 1" for (T, n, K, mode, _), tn in zip(cases, (160, 256, 224, 96))]
    path = tmp_path / "choices.txt"
    path.write_text("\n".join(lines) + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, cases=cases)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200_WT_TUNE_FILE=str(path)))
    assert r.returncode == 0, r.stdout + r.stderr
    assert path.read_text() == "\n".join(lines) + "\n"


@pytest.mark.parametrize("T,n,K", [(128, 512, 64), (1300, 8192, 640)])
def test_a_wait_of_wide_pairs_that_runs_out_is_told(T, n, K):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    child = _CHILD_WAIT.replace("cfg, 8 | flags", "cfg, 16 | flags")
    r = subprocess.run([sys.executable, "-c", child.format(root=root, T=T, n=n, K=K)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


_CHILD_LINES = """
import sys, torch
sys.path.insert(0, {root!r})
sys.path.insert(0, {root!r} + "/tests")
from mlx_vlm_b200 import _native as N
lib = N.lib()
stream = torch.cuda.Stream()       # (choices are measured under capture, which the default stream does not take)
g = torch.Generator(device="cuda").manual_seed(21)
for T, n, K in ((300, 264, 128), (577, 1152, 640), (130, 136, 192)):
    x = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    out = torch.zeros(T, n, device="cuda")
    torch.cuda.synchronize()
    N.check(lib.b200_gemm_wt_f32(x.data_ptr(), K, w.data_ptr(), K, 0, 0, 0, out.data_ptr(), n, 0, 0, 0, T, n, K, 1, 0, 3, stream.cuda_stream), "f32")
    torch.cuda.synchronize()
    want = x.double() @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) <= 2e-6
from test_engine_gpu import _build
c, W, model, req = _build("wide1", 20, (56, 56))
lm = model.language_model
ids = torch.arange(20)[None].numpy()
logits = lm(ids, inputs_embeds=model.get_input_embeddings(ids).inputs_embeds, cache=lm.make_cache(), logits_to_keep=1).logits
torch.cuda.synchronize()
assert bool(torch.isfinite(logits.float()).all())
"""


def test_lines_that_no_call_takes_are_passed_over(tmp_path):
    """a file of choices may name what gemm_wt refuses: splits outside the partial mode, more shared memory than there is, splits without a
    k-block, wide pairs that would write partial tiles; such products are measured, the others' lines are kept"""
    bad = ["5 264 128 3 0 160 -1 4 2", "10 1152 640 3 0 256 2 6 1", "3 136 192 3 0 96 1 4 3", "1 1536 1536 1 1 64 -1 4 1"]
    good = "1 1536 8960 1 1 32 1 4 3"
    path = tmp_path / "choices.txt"
    path.write_text("\n".join(bad + [good]) + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD_LINES.format(root=root)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200_WT_TUNE_FILE=str(path)))
    assert r.returncode == 0, r.stdout + r.stderr
    added = [line.split()[:5] for line in path.read_text().splitlines()[len(bad) + 1:]]
    assert all(line.split()[:5] in added for line in bad) and good.split()[:5] not in added, added


@pytest.mark.parametrize("ks,tn", [(1, 128), (2, 96), (0, 160), (-1, 192)])
def test_split_outputs_of_an_odd_number_of_rows(tmp_path, ks, tn):
    """[hi | lo] pairs whose rows are written feature by feature: one CTA, pairs and wide pairs, configurations given by a file"""
    cases = [(300, 263, 128, 4, 0), (577, 131, 584, 4, 2), (65, 77, 72, 4, 0), (200, 999, 1152, 4, 2)]
    lines = [f"{(T + 63) // 64} {n} {2 * ((K + 63) // 64 * 64)} {mode} 0 {tn} {ks} 3 1" for T, n, K, mode, _ in cases]
    path = tmp_path / "choices.txt"
    path.write_text("\n".join(lines) + "\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, cases=cases)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, B200_WT_TUNE_FILE=str(path)))
    assert r.returncode == 0, r.stdout + r.stderr
    assert path.read_text() == "\n".join(lines) + "\n"        # nothing was measured: the file's choices ran


@pytest.mark.parametrize("T,N,K,cfg,flag", [(1, 65, 64, (16, 1, 3, 1), 0), (65, 77, 72, (96, 2, 2, 1), 0), (300, 263, 192, (128, 1, 3, 1), 0),
                                            (300, 257, 192, (160, 1, 4, 1), PAIR), (577, 1031, 128, (224, 1, 4, 1), WIDE)])
@pytest.mark.parametrize("epi,even", [(0, True), (1, True), (2, True), (0, False), (1, False), (2, False)])
def test_rows_of_an_odd_number_of_features(lib, T, N, K, cfg, flag, epi, even):
    """even row strides: two features to a word, the last one alone; odd ones: feature by feature; with and without a residual, in place,
    and nothing behind the last feature is written or taken"""
    import ctypes
    from mlx_vlm_b200 import _native as Nn
    x, w, b = _rand(T, K, seed=31), _rand(N, K, seed=32, std=K ** -0.5), _rand(N, seed=33)
    y = (x.double() @ w.double().T + b.double()).to(torch.bfloat16).double()
    if epi == 1:
        y = y * torch.sigmoid((1.703125 * y).to(torch.bfloat16).double()).to(torch.bfloat16).double()
    if epi == 2:
        y = torch.nn.functional.gelu(y)
    ld = N + 1 + T % 2 * 2 if even else N + T % 2 * 2
    for res in (None, _rand(T, ld, seed=34)):
        out = torch.full((T, ld), 9.0, dtype=torch.bfloat16, device="cuda")
        if res is not None:
            res[:, N:] = float("nan")
            out[:, :N] = res[:, :N]
        r = None if res is None else out                  # (the output is its own residual)
        Nn.check(lib.b200_gemm_wt(x.data_ptr(), K, w.data_ptr(), b.data_ptr(), Nn.ptr(r), ld, out.data_ptr(), ld, 0, T, N, K, epi, 0, 0,
                                  (ctypes.c_int * 4)(*cfg), flag, 0), "gemm_wt")
        torch.cuda.synchronize()
        want = y if res is None else y.to(torch.bfloat16).double() + res[:, :N].double()
        # the unit's own roundings to bf16: the exact GELU has five, the fast one three, most of them shared with the reference's
        assert rl2(out[:, :N], want) <= (2.0 ** -8 if epi == 0 else 2.0 ** -7)
        assert bool((out[:, N:] == 9.0).all())
