"""Kernels of a dependent-launch chain read what earlier kernels of the chain wrote from L2 only.

A block launched that way may be resident before its input is written, so a line it finds in L1, or gets through the
read-only path that a `const __restrict__` pointer allows, can be older than its wait.  The kernels therefore take
such arrays as ``Fresh<T>``, which has no plain reads; what remains as a plain `const` pointer has to be constant.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "async-gpu_b200", "csrc")
# weights, tables and host-written indexes: nothing on the device writes them
CONSTANT = {"w", "gamma", "beta", "norm", "q_norm", "kv_norm", "wte", "wpe", "table", "pos_table", "rope", "tab", "tiles", "scales", "idx", "g"}
WAITS = ("pdl_wait()", "norm_rows_to_smem")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _block(s, i, open_, close):
    """The text between the bracket at or after i and the one that closes it, and where that is."""
    i = s.index(open_, i)
    depth, j = 0, i
    while True:
        depth += (s[j] == open_) - (s[j] == close)
        if depth == 0:
            return s[i + 1:j], j
        j += 1


def _kernels():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        s = _text(name)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\()?", s):
            i = m.end()
            if s[m.start():i].rstrip().endswith("("):
                i = _block(s, i - 1, "(", ")")[1] + 1
            kernel = re.compile(r"\s*(\w+)").match(s, i).group(1)
            params, j = _block(s, i, "(", ")")
            out[kernel] = (name, [" ".join(p.split()) for p in re.split(r",(?![^<]*>)", params)], _block(s, j, "{", "}")[0])
    return out


KERNELS = _kernels()
CHAIN = sorted(k for k, (_, _, body) in KERNELS.items() if any(w in body for w in WAITS))


def test_the_chain_is_found():
    assert {"rmsnorm_kernel", "layernorm_kernel", "glu_kernel", "delta_step_kernel", "f32_gemv_kernel", "decode_attn_kernel"} <= set(CHAIN)


@pytest.mark.parametrize("kernel", CHAIN)
def test_chain_kernels_take_written_arrays_as_fresh(kernel):
    name, params, body = KERNELS[kernel]
    plain = [re.search(r"(\w+)$", p).group(1) for p in params if re.match(r"const [\w:]+ \*", p)]
    assert set(plain) <= CONSTANT, f"{name}: {kernel} reads {sorted(set(plain) - CONSTANT)} plainly"
    assert "__ldcs" not in body, f"{name}: {kernel}"


def test_kernels_that_read_through_l1_start_behind_everything_before_them():
    chain, ordered = set(), set()
    for name in os.listdir(CSRC):
        if name.endswith(".cu"):
            chain |= set(re.findall(r"launch_pdl\(ctx, (\w+)", _text(name)))
            ordered |= set(re.findall(r"launch_ordered\(ctx, (\w+)", _text(name)))
    assert not chain & ordered
    assert {"delta_conv_kernel", "delta_scan_kernel", "mlstm_scan_kernel", "latent_prefill_simple_kernel", "latent_decode_simple_kernel",
            "diff_simple_kernel"} <= ordered
    assert not ordered & set(CHAIN)
