"""The activations that the GEMM epilogues compute on bf16 pairs (csrc/common.cuh: gelu_fast_bf2, swiglu_bf2) against the scalar chain of
roundings, over every finite bf16 number: an identity weight makes the products the numbers themselves."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _all_bf16(n_cols=64):
    """every finite bf16 number, zeros behind the last"""
    x = torch.arange(0, 65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = x[torch.isfinite(x.float())]
    return torch.nn.functional.pad(x, (0, -x.numel() % n_cols)).view(-1, n_cols).cuda()


def _call(x, w, epi, mode, inter, pair):
    import ctypes
    from mlx_vlm_b200 import _native as N
    lib = N.lib()
    T, K = x.shape
    out = torch.empty(T, inter or w.shape[0], dtype=torch.bfloat16, device="cuda")
    N.check(lib.b200_gemm_wt(x.data_ptr(), K, w.data_ptr(), 0, 0, 0, out.data_ptr(), out.shape[1], 0, T, w.shape[0], K, epi, mode, inter,
                             (ctypes.c_int * 4)(128, 1, 4, 1), 8 if pair else 0, 0), "gemm_wt")
    torch.cuda.synchronize()
    return out


def _sigmoid(x):
    return torch.sigmoid(x.double()).to(torch.bfloat16)


def _close(got, want):
    """The exponential and the reciprocal err by some 2^-22 (more where the exponent is large: 2^-24 of it): where the logistic function
    lies that close to the middle of two bf16 numbers it may round the other way, one unit (2^-7 at most), which the one or two
    products behind it hand on and may round once more each: below 2^-6.  A logistic function below 2^-126 counts as 0: it
    belongs to arguments between 87 and 89, so 3 x 89 x 2^-126 < 2^-117 of the result.  What overflows is the same infinity."""
    g, w = got.double(), want.double()
    assert bool(((g == w) | ((g - w).abs() <= 2.0 ** -6 * w.abs().clamp(max=3.4e38) + 2.0 ** -117)).all())
    assert float((g != w).double().mean()) < 5e-3


@pytest.mark.parametrize("pair", [False, True])
def test_fast_gelu(pair):
    x = _all_bf16()
    got = _call(x, torch.eye(64, device="cuda", dtype=torch.bfloat16), 1, 0, 0, pair)
    u = (x.double() * 1.703125).to(torch.bfloat16)
    _close(got, (x.double() * _sigmoid(u).double()).to(torch.bfloat16))


@pytest.mark.parametrize("pair", [False, True])
def test_swiglu(pair):
    """gate: every number; up: 1.5, and 3 for the odd channels (the second product rounds)"""
    x = _all_bf16(56)
    T = x.shape[0]
    x = torch.cat([x, torch.ones(T, 8, device="cuda", dtype=torch.bfloat16)], 1)
    w = torch.zeros(112, 64, device="cuda", dtype=torch.bfloat16)
    w[torch.arange(56), torch.arange(56)] = 1.0
    w[56::2, 56] = 1.5
    w[57::2, 56] = 3.0
    got = _call(x, w, 0, 2, 56, pair)
    g = x[:, :56]
    s = (g.double() * _sigmoid(g).double()).to(torch.bfloat16).double()
    up = torch.where(torch.arange(56, device="cuda") % 2 == 0, 1.5, 3.0).double()
    _close(got, (s * up).to(torch.bfloat16))
