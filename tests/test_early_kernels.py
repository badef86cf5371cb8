"""Kernels that may begin while the kernel before still runs: what that kernel writes is read through plain pointers.  Loads through `const __restrict__` pointers and
`__ldg` count as loads of memory that nobody writes, which the compiler may move up past `griddepcontrol.wait`."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rexl3_b200", "ops", "csrc")


@pytest.mark.parametrize("source,kernel,inputs", [
    ("attention.cu", "attn_merge_few_kernel", ["part_o", "part_ml", "ctx_len"]),
    ("moe.cu", "moe_gather_rot_rows_kernel", ["x", "ids", "pos_of_pair"]),
    ("moe.cu", "moe_combine_rows_kernel", ["part", "ids", "w", "pos_of_pair", "shared"]),
    ("exl3_aux.cu", "rot_in_rows_kernel", ["x"]),
    ("exl3_aux.cu", "finish_add_norm_rot_rows_kernel", ["part", "h"]),
])
def test_inputs_of_early_kernels_are_plain_pointers(source, kernel, inputs):
    text = open(os.path.join(CSRC, source)).read()
    m = re.search(r"\b" + kernel + r"\((.*?)\)\s*\{\n(.*?)\n\}\n", text, re.S)
    params, body = m.group(1), m.group(2)
    assert body.index("pdl_wait();") >= 0
    for name in inputs:
        p = next(p for p in params.split(",") if re.search(r"\b" + name + r"$", p.strip()))
        assert "__restrict__" not in p, p
    assert not any(re.search(r"\b(" + "|".join(inputs) + r")\b", load) for load in re.findall(r"__ldg\((.*?)\);", body)), body
