"""The pipelined attention as the engine runs it (csrc/attention_fa.cu, values as rows), alone, against the same oracle and bound as
its form with transposed values in test_kernels2_gpu.py: whole and ragged tiles of 128 queries and keys, keys that end inside a
group of 16, later portions of a prompt, tables of segments, unused rows full of NaN."""
import os
import subprocess
import sys

import pytest
import torch

from test_kernels2_gpu import R, cmp_bf16, rnd, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from mlx_vlm_b200 import _native as N
    return N.lib()


def _call(lib, q, k, v, out, nh, nkv, hd, Lq, S, causal, segs=None):
    from mlx_vlm_b200 import _native as N
    N.check(lib.b200_attention_fa_rows(q.data_ptr(), q.stride(0), hd, k.data_ptr(), k.stride(0), hd, v.data_ptr(), v.stride(0), hd,
                                       out.data_ptr(), nh * hd, nh, nkv, hd, Lq, S, int(causal), q.shape[0], k.shape[0],
                                       N.ptr(segs), 0 if segs is None else segs.shape[0], 0, 0), "attention_fa_rows")
    torch.cuda.synchronize()


def _want(q, k, v, causal):
    """q pre-scaled: (queries, heads, hd), k / v (keys, kv heads, hd)"""
    from oracle import mlx_semantics as S
    q, k, v = (x.transpose(0, 1)[None] for x in (q, k, v))
    return S.sdpa(R(), q, k, v, 1.0, bool(causal))[0].transpose(0, 1)


@pytest.mark.parametrize("Lq,S,nh,nkv,hd,causal", [
    (576, 576, 16, 16, 80, 0), (272, 272, 12, 2, 128, 1), (17, 17, 4, 2, 64, 1), (300, 300, 28, 4, 128, 1), (33, 33, 4, 4, 72, 0),
    (577, 577, 16, 16, 64, 0), (1, 1, 2, 1, 128, 1), (128, 129, 2, 2, 64, 0), (129, 144, 2, 2, 80, 0),
    (1, 200, 4, 2, 128, 1), (130, 391, 4, 2, 128, 1), (255, 513, 6, 2, 64, 1)])
def test_values_as_rows(lib, Lq, S, nh, nkv, hd, causal):
    """q, k and v side by side in one buffer, the rows behind the last key NaN"""
    rows = max(Lq, S) + 40
    buf = torch.full((rows, (nh + 2 * nkv) * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    q, k, v = rnd(Lq, nh, hd, scale=hd ** -0.5, seed=12), rnd(S, nkv, hd, seed=13), rnd(S, nkv, hd, seed=14)
    buf[:Lq, :nh * hd] = to_dev(q).view(Lq, -1)
    buf[:S, nh * hd:(nh + nkv) * hd] = to_dev(k).view(S, -1)
    buf[:S, (nh + nkv) * hd:] = to_dev(v).view(S, -1)
    out = torch.full((rows, nh * hd), 9.0, dtype=torch.bfloat16, device="cuda")
    _call(lib, buf, buf[:, nh * hd:], buf[:, (nh + nkv) * hd:], out, nh, nkv, hd, Lq, S, causal)
    cmp_bf16(out[:Lq].view(Lq, nh, hd), _want(q, k, v, causal), f"Lq={Lq} S={S} hd={hd}")
    assert bool((out[Lq:] == 9.0).all())


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("lens", [(1, 130, 15, 128, 257), (36, 128, 132), (300,)])
def test_a_table_of_segments(lib, lens, causal):
    """a segment of NaN between the others stays alone"""
    nh, nkv, hd = 4, 2, 128
    T = sum(lens)
    q, k, v = rnd(T, nh, hd, scale=hd ** -0.5, seed=15), rnd(T, nkv, hd, seed=16), rnd(T, nkv, hd, seed=17)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    bad = 1 if len(lens) > 2 else -1
    dq, dk, dv = (to_dev(x).view(T, -1) for x in (q, k, v))
    if bad >= 0:
        for x in (dq, dk, dv):
            x[starts[bad]:starts[bad] + lens[bad]] = float("nan")
    segs = torch.tensor([[a, n, a, n] for a, n in zip(starts, lens)], dtype=torch.int32, device="cuda")
    out = torch.full((T, nh * hd), 9.0, dtype=torch.bfloat16, device="cuda")
    _call(lib, dq, dk, dv, out, nh, nkv, hd, max(lens), max(lens), causal, segs)
    for i, (a, n) in enumerate(zip(starts, lens)):
        sl = slice(a, a + n)
        if i == bad:
            assert bool(torch.isnan(out[sl].float()).all())
        else:
            cmp_bf16(out[sl].view(n, nh, hd), _want(q[sl], k[sl], v[sl], causal), f"segment {i} of {lens}")


_CHILD = """
import sys, ctypes as C, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
def state():
    v = C.c_int(-1)
    N.check(lib.b200_wait_error(C.byref(v)))
    return v.value
T, S = {T}, {S}
g = torch.Generator(device="cuda").manual_seed(1)
q, k, v = (torch.randn(n, 128, device="cuda", generator=g).to(torch.bfloat16) for n in (T, S, S))
out = torch.zeros(T, 128, device="cuda", dtype=torch.bfloat16)
def run(flags):
    out.zero_()
    torch.cuda.synchronize()
    N.check(lib.b200_attention_fa_rows(q.data_ptr(), 128, 128, k.data_ptr(), 128, 128, v.data_ptr(), 128, 128, out.data_ptr(), 128, 1, 1,
                                       128, T, S, 0, T, S, 0, 0, flags, 0))
    torch.cuda.synchronize()
    return out.float().clone()
want = torch.softmax(q.double() @ k.double().T, -1) @ v.double()
a = run(0)
assert float((a - want).norm() / want.norm()) < 0.05 and state() == 0
b = run(1)                            # nothing is loaded: the waits run out after a second
assert bool(torch.isnan(b).all()) and state() == 6, (b, state())
assert torch.equal(run(0), a) and state() == 6
"""


@pytest.mark.parametrize("T,S", [(5, 7), (300, 700)])
def test_a_wait_that_runs_out_is_told(T, S):
    """in a process of its own: NaN, the word that the host reads, and the next launch as if nothing had been"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, T=T, S=S)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


_CHILD_THREADS = """
import sys, threading, torch
sys.path.insert(0, {root!r})
from mlx_vlm_b200 import _native as N
lib = N.lib()
n, hd = 200, 64
x = torch.randn(3, n, hd, device="cuda").to(torch.bfloat16)
f = torch.randn(3, n, hd, device="cuda")
streams = [torch.cuda.Stream() for _ in range(16)]
outs = [(torch.zeros(n, hd, device="cuda", dtype=torch.bfloat16), torch.zeros(n, hd, device="cuda")) for _ in streams]
torch.cuda.synchronize()
gate, bad = threading.Barrier(len(streams)), []
def go(s, o):
    with torch.cuda.stream(s): torch.zeros(1, device="cuda")      # (the thread has a context)
    s.synchronize()
    gate.wait()
    a = lib.b200_attention_fa_rows(x[0].data_ptr(), hd, hd, x[1].data_ptr(), hd, hd, x[2].data_ptr(), hd, hd, o[0].data_ptr(), hd, 1, 1, hd,
                                   n, n, 0, n, n, 0, 0, 0, s.cuda_stream)
    b = lib.b200_attention_f32(f[0].data_ptr(), hd, hd, f[1].data_ptr(), hd, hd, f[2].data_ptr(), hd, hd, o[1].data_ptr(), hd, 0, 0, 0, 1,
                               1, hd, n, n, 1, n, n, 0, 0.1, s.cuda_stream)
    if a or b: bad.append((a, b, lib.b200_last_error()))
ts = [threading.Thread(target=go, args=a) for a in zip(streams, outs)]
[t.start() for t in ts]
[t.join() for t in ts]
torch.cuda.synchronize()
assert not bad, bad
assert all(torch.equal(o[i], outs[0][i]) and bool(o[i].any()) for o in outs for i in (0, 1))
"""


def test_first_calls_of_many_threads():
    """none of the threads launches before the kernel's shared memory is allowed for"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD_THREADS.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
