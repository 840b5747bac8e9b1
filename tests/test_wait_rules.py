"""Reads of what the kernel before wrote come after the wait for it.  The compiler takes loads through a const __restrict__ parameter for
loads of what nobody writes and may move them up across the wait, so every such pointer to another kernel's results is named in the
call of pdl_wait, which hands it back as a new one.  Checked on the sources: no run shows a load that is early only sometimes."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocmforge_b200", "csrc")

# what no kernel of a step writes: weights, frequency tables, the step descriptor, block and chunk tables
CONSTANT = {"tok_seq", "tok_pos", "seq_slot", "block_table", "cu_q", "cu", "tiles", "seq_start", "seq_nnew", "rows", "table", "inv_freq",
            "pos_table", "w", "W", "b", "bias", "w0", "w1", "w_next", "b_next", "w_post", "norm_w", "q_norm_w", "k_norm_w", "skip",
            "slopes", "sinks", "dt_bias", "a_log", "correction"}
# the same name for another thing: alpha is a weight of Dynamic Tanh and of the scaled update, decay one of retention
ALSO_CONSTANT = {("dyt_rows_kernel", "alpha"), ("scaled_add_kernel", "alpha"), ("retention_scan_kernel", "decay"),
                 ("retention_chunk_state_kernel", "decay"), ("retention_chunk_carry_kernel", "decay"), ("retention_chunk_out_kernel", "decay")}
WRITTEN_ALL_THE_SAME = {("moe_sort_kernel", "w"), ("moe_combine_kernel", "w"), ("gemm_simt_kernel", "tiles")}


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^{;]*?\{", text, re.S):
            end, depth = m.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            name = next(n for n in re.findall(r"(\w+)\s*\(", m.group(0)) if n != "__launch_bounds__")
            yield name, m.group(0), text[m.end():end]


def unguarded(name, signature, body):
    """The const __restrict__ parameters that another kernel may have written and that the wait does not hand back."""
    waits = re.findall(r"pdl_wait\(([^)]*)\)", body)
    if not waits:
        return []
    named = {n.strip() for w in waits for n in w.split(",")}
    before = body[:body.index("pdl_wait(")]
    found = []
    for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", signature):
        constant = (p in CONSTANT or (name, p) in ALSO_CONSTANT) and (name, p) not in WRITTEN_ALL_THE_SAME
        derived = re.findall(r"\*\s*(\w+)\s*=[^;]*\b%s\b" % p, before)         # pointers formed from it before the wait
        if not constant and not (set(derived) <= named if derived else p in named):
            found.append(p)
    return found


@pytest.mark.parametrize("name,signature,body", [pytest.param(*k, id=k[0]) for k in kernels() if "pdl_wait" in k[2]])
def test_results_of_the_kernel_before_are_read_after_the_wait(name, signature, body):
    assert unguarded(name, signature, body) == []


def test_the_check_sees_what_is_left_out():
    sig = "__global__ void k(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y) {"
    assert unguarded("k", sig, "pdl_wait(); y[0] = x[0] * w[0]; }") == ["x"]
    assert unguarded("k", sig, "pdl_wait(x); y[0] = x[0] * w[0]; }") == []
    assert unguarded("k", sig, "const float* at = x + 4; pdl_wait(x); y[0] = at[0]; }") == ["x"]
    assert unguarded("k", sig, "const float* at = x + 4; pdl_wait(at); y[0] = at[0]; }") == []
