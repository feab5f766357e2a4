"""Order of tensor-memory accesses in the attention kernels, read from their source.

A wait on an mbarrier or a barrier of threads orders a tensor-memory access behind another thread's products only together with
tcgen05.fence::after_thread_sync (and, ahead of a barrier of threads, fence::before_thread_sync); timing usually hides a
missing one, so nothing that runs could show it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlx_vlm_b200", "csrc")
KERNELS = [("attention_fa.cu", "attention_fa_kernel"), ("attention_f32_tc.cu", "attention_f32_tc_kernel"),
           ("attention_latent.cu", "attention_latent_kernel")]


def _body(name, kernel):
    """the kernel's text without comments, and without the helpers before it"""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    at = text.index("{", text.index(kernel + "(", text.index("__global__", text.index(kernel + "(") - 120)))
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at:i]
    raise AssertionError(f"{name}: {kernel} does not end")


def _events(body):
    kinds = [("wait", r"mbar_wait(?:_issuer)?\("), ("after", r"\b[flt]_fence_after\(\)"), ("before", r"\b[flt]_fence_before\(\)"),
             ("barrier", r"bar\.sync 1|\b[fl]_s?bar(?:256)?\(\)|__syncthreads\(\)"),
             ("access", r"\b(?!t_ld16\(t_o)(?:f_st16|f_tmem_ld16|f_scores|f_umma(?:_ts)?|[lt]_(?:ld16|st16|st8|mma_ss|mma_ts)|add_tile)(?:<\w+>)?\(|tcgen05\.dealloc")]
    out = []      # (the loads of the lambda add_tile count where it is called)
    for kind, pattern in kinds:
        out += [(m.start(), kind) for m in re.finditer(pattern, body)]
    return sorted(out)


@pytest.mark.parametrize("name,kernel", KERNELS)
def test_an_access_behind_a_wait_is_fenced(name, kernel):
    body = _body(name, kernel)
    state, barrier_fenced, fenced_before, seen = None, True, True, 0
    for at, kind in _events(body):
        where = f"{name}: ...{body[max(0, at - 60):at + 60]!r}"
        if kind in ("wait", "barrier"):
            if kind == "barrier":
                barrier_fenced = fenced_before or (state == "barrier" and barrier_fenced)    # (a second one needs no fence of its own)
            state = kind
        elif kind == "after":
            assert state != "barrier" or barrier_fenced, f"no fence before the barrier: {where}"
            state = "after"
            fenced_before = False
        elif kind == "before":
            fenced_before = True
        else:
            assert state in ("after", None), f"an access behind a {state} without a fence: {where}"
            fenced_before = False
            seen += 1
    assert seen >= 6


@pytest.mark.parametrize("name,kernel", KERNELS + [("gemm_wt.cu", "gemm_wt_pair_kernel")])
def test_columns_are_allocated_before_the_next_kernel_may_start(name, kernel):
    """A kernel that asks for all 512 columns and lets its dependent start first could find columns taken by a CTA that waits for it"""
    body = _body(name, kernel)
    alloc = body.index("tcgen05.alloc")
    assert "512u" in body[alloc:alloc + 200]
    signals = [m.start() for m in re.finditer(r"griddepcontrol\.launch_dependents|w_pdl_launch\(\)", body)]
    assert len(signals) == 1 and signals[0] > body.index("__syncthreads()", alloc), name


@pytest.mark.parametrize("kernel,reads", [("gemm_wt_kernel", r"wt_bias<|p\.(?:bias|residual|res32)\b"), ("gemm_wt_pair_kernel", r"wt_bias<|p\.(?:bias|residual|res32)\b"),
                                          ("finish_rows_kernel", r"\b(?:P|bias|resid|nw|nb)\b")])
def test_operands_of_the_epilogue_are_read_behind_the_kernel_before(kernel, reads):
    """A kernel that starts while the one before it still runs reads nothing that a caller may have made on the device right ahead of the
    call until griddepcontrol.wait, whatever role its warps have (only the weight matrices are requested earlier)"""
    body = _body("gemm_wt.cu", kernel)
    waits = [m.start() for m in re.finditer(r"w_pdl_wait\(\)", body)]
    seen = [m.start() for m in re.finditer(reads, body)]
    assert waits and seen and min(seen) > max(waits), kernel


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith(".cu")))
def test_register_shares_are_checked_before_a_launch(name):
    """setmaxnreg.inc waits without end for registers that the block was not launched with; launch bounds are only an upper limit, so
    the host asks what the kernel was compiled with, and a refusal is not remembered as a first use"""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    if "setmaxnreg.inc" not in text:
        return
    launches = [m.start() for m in re.finditer(r"<<<", text)]
    assert len(launches) == 1
    asked, refused, unset = (text.index(w) for w in (".numRegs", "B200_REQUIRE(tc_shares_fit(", "first.bit = 0ull"))
    assert text.index("cudaFuncGetAttributes") < asked < unset < refused < launches[0]
