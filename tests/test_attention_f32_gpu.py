"""fp32 attention of the towers (csrc/attention_f32_tc.cu) against float64 at the edges of its tiles: 128 query rows, 64 keys,
groups of 16 keys, head sizes padded to 32 / 64 / 80 / 96.

Bound: a score is a sum of at most 96 products with 24 bits each (relative error about 1e-7 of |q||k|, |scores| <= ~6 here, so
6e-7 in the exponent), the exponential 2^-22, sums and outputs 2^-24 a step: 2e-6 of the output's size."""
import os
import subprocess
import sys

import pytest
import torch

from _util import rl2

pytestmark = pytest.mark.gpu
BOUND = 2e-6


@pytest.fixture(scope="module")
def lib():
    from mlx_vlm_b200 import _native as N
    return N.lib()


def _rand(*shape, seed):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def _want(q, k, v, nh, nkv, hd, keep=None):
    q = q.double().view(-1, nh, hd).transpose(0, 1)
    k, v = (x.double().view(-1, nkv, hd).transpose(0, 1).repeat_interleave(nh // nkv, 0) for x in (k, v))
    s = q @ k.transpose(1, 2) * hd ** -0.5
    if keep is not None:
        s = s.masked_fill(~keep, float("-inf"))
    return (torch.softmax(s, -1) @ v).transpose(0, 1).reshape(-1, nh * hd)


def _split_value(t, n, n_pad):
    return t[:, :n].double() + t[:, n_pad:n_pad + n].double()


@pytest.mark.parametrize("nh,nkv,hd,Lq,S", [
    (2, 2, 64, 128, 64), (2, 2, 64, 129, 65), (1, 1, 64, 127, 63), (2, 1, 64, 1, 1), (2, 2, 64, 5, 16), (2, 2, 64, 130, 17),
    (3, 3, 72, 64, 128), (2, 2, 72, 200, 129), (4, 1, 96, 64, 113), (2, 2, 80, 33, 49), (2, 2, 20, 70, 100), (1, 1, 4, 3, 80),
    (2, 2, 32, 40, 192)])
@pytest.mark.parametrize("aligned", [True, False])
def test_tile_edges(lib, nh, nkv, hd, Lq, S, aligned):
    """two segments, both outputs; unaligned output addresses are stored element by element"""
    from mlx_vlm_b200 import _native as N
    q, k, v = _rand(2 * Lq, nh * hd, seed=1), _rand(2 * S, nkv * hd, seed=2), _rand(2 * S, nkv * hd, seed=3)
    E, n_pad, off = nh * hd, (nh * hd + 63) // 64 * 64, 0 if aligned else 1
    o32 = torch.full((2 * Lq * E + 2,), 7.0, device="cuda")
    osp = torch.full((2 * Lq * 2 * n_pad + 2,), 7.0, device="cuda", dtype=torch.bfloat16)
    N.check(lib.b200_attention_f32(q.data_ptr(), E, hd, k.data_ptr(), nkv * hd, hd, v.data_ptr(), nkv * hd, hd,
                                   o32[off:].data_ptr(), E, osp[off:].data_ptr(), 2 * n_pad, n_pad, nh, nkv, hd, Lq, S, 2, Lq, S, 0,
                                   hd ** -0.5, 0), "attention_f32")
    torch.cuda.synchronize()
    want = torch.cat([_want(q[s * Lq:(s + 1) * Lq], k[s * S:(s + 1) * S], v[s * S:(s + 1) * S], nh, nkv, hd) for s in (0, 1)])
    assert rl2(o32[off:off + 2 * Lq * E].view(2 * Lq, E).double(), want) <= BOUND
    got = _split_value(osp[off:off + 2 * Lq * 2 * n_pad].view(2 * Lq, 2 * n_pad), E, n_pad)
    assert rl2(got, want) <= BOUND + 2.0 ** -17
    assert float(o32[-1]) == 7.0 and float(osp[-1]) == 7.0


def test_masked_keys_and_ragged_segments(lib):
    from mlx_vlm_b200 import _native as N
    nh, hd, S = 2, 64, 200
    q, k, v = (_rand(2 * S, nh * hd, seed=s) for s in (4, 5, 6))
    mask = torch.rand(2, S, generator=torch.Generator().manual_seed(7)) > 0.4
    mask[0, :64], mask[1, 64:130], mask[0, 199] = False, False, True       # whole tiles without a key
    m = mask.to(device="cuda", dtype=torch.uint8)
    out = torch.empty(2 * S, nh * hd, device="cuda")
    args = (q.data_ptr(), nh * hd, hd, k.data_ptr(), nh * hd, hd, v.data_ptr(), nh * hd, hd, out.data_ptr(), nh * hd, 0, 0, 0, nh,
            nh, hd)
    N.check(lib.b200_attention_f32(*args, S, S, 2, S, S, m.data_ptr(), hd ** -0.5, 0), "attention_f32")
    torch.cuda.synchronize()
    for s in (0, 1):
        sl = slice(s * S, (s + 1) * S)
        assert rl2(out[sl].double(), _want(q[sl], k[sl], v[sl], nh, nh, hd, m[s].bool())) <= BOUND
    cuts = [0, 1, 65, 65, 193, 400]
    cu = torch.tensor(cuts, dtype=torch.int32, device="cuda")
    N.check(lib.b200_attention_f32_varlen(*args, cu.data_ptr(), len(cuts) - 1, 207, hd ** -0.5, 0), "attention_f32_varlen")
    torch.cuda.synchronize()
    for a, b in zip(cuts, cuts[1:]):
        if b > a:
            assert rl2(out[a:b].double(), _want(q[a:b], k[a:b], v[a:b], nh, nh, hd)) <= BOUND


def _inf_case(kind, q, k, v, hd):
    if kind == "value":              # stays in its own dimension
        v[70, 3], v[5, hd + 1] = float("inf"), float("-inf")
    elif kind == "key":              # every query of head 0 scores -inf: weight 0; head 1 half +inf (NaN), half -inf
        q[:, 2] = q[:, 2].abs() + 0.1
        k[66, 2], k[100, hd] = float("-inf"), float("inf")
    elif kind == "first_tile":       # the whole first tile scores -inf
        q[:, 2] = q[:, 2].abs() + 0.1
        k[:64, 2] = float("-inf")
    elif kind == "query":
        q[3, 1] = float("inf")
    elif kind == "large":            # finite in fp32, not in bf16
        v[7, 0], v[100, hd + 4] = 3.4e38, -3.4e38
    elif kind == "nan":
        v[9, 9] = float("nan")


@pytest.mark.parametrize("kind", ["value", "key", "first_tile", "query", "large", "nan"])
@pytest.mark.parametrize("hd,Lq,S", [(64, 130, 200), (72, 40, 129), (96, 128, 131)])
def test_numbers_that_bf16_parts_do_not_hold(lib, kind, hd, Lq, S):
    """infinities, NaN and magnitudes above the largest bf16 reach the results that the formula gives them and no others"""
    from mlx_vlm_b200 import _native as N
    nh = 2
    q, k, v = _rand(Lq, nh * hd, seed=11), _rand(S, nh * hd, seed=12), _rand(S, nh * hd, seed=13)
    _inf_case(kind, q, k, v, hd)
    out = torch.empty(Lq, nh * hd, device="cuda")
    N.check(lib.b200_attention_f32(q.data_ptr(), nh * hd, hd, k.data_ptr(), nh * hd, hd, v.data_ptr(), nh * hd, hd, out.data_ptr(),
                                   nh * hd, 0, 0, 0, nh, nh, hd, Lq, S, 1, Lq, S, 0, hd ** -0.5, 0), "attention_f32")
    torch.cuda.synchronize()
    want, got = _want(q, k, v, nh, nh, hd), out.double()
    assert bool(torch.isfinite(want).any()) and (kind in ("first_tile", "large") or not bool(torch.isfinite(want).all()))
    odd = ~torch.isfinite(want)
    assert torch.equal(torch.nan_to_num(got[odd], 1.0, 2.0, 3.0), torch.nan_to_num(want[odd], 1.0, 2.0, 3.0))
    # column by column: a large value's dimension does not hide the others
    err = ((got - want).masked_fill(odd, 0.0).norm(dim=0) / want.masked_fill(odd, 0.0).norm(dim=0).clamp_min(1e-300)).max().item()
    print(kind, hd, err)
    assert bool(torch.isfinite(got[~odd]).all()) and err <= 2 * BOUND


_CHILD = """
import sys, ctypes as C, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
def state():
    v = C.c_int(-1)
    N.check(lib.b200_wait_error(C.byref(v)))
    return v.value
T, S, hd = {T}, {S}, 64
g = torch.Generator(device="cuda").manual_seed(1)
q, k, v = (torch.randn(n, hd, device="cuda", generator=g) for n in (T, S, S))
out = torch.zeros(T, hd, device="cuda")
def run(flags):
    out.zero_()
    torch.cuda.synchronize()
    N.check(lib.b200_attention_f32_debug(q.data_ptr(), hd, hd, k.data_ptr(), hd, hd, v.data_ptr(), hd, hd, out.data_ptr(), hd, 1, 1, hd,
                                         T, S, 1.0, flags, 0))
    torch.cuda.synchronize()
    return out.clone()
want = torch.softmax(q.double() @ k.double().T, -1) @ v.double()
a = run(0)
assert float((a - want).norm() / want.norm()) < 1e-5 and state() == 0
b = run(1)                            # nothing is loaded: the waits run out after a second
assert bool(torch.isnan(b).all()) and state() == 7, (b, state())
assert torch.equal(run(0), a) and state() == 7
"""


@pytest.mark.parametrize("T,S", [(5, 7), (300, 700)])
def test_a_wait_that_runs_out_is_told(T, S):
    """in a process of its own: NaN, the word that the host reads, and the next launch as if nothing had been"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, T=T, S=S)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
