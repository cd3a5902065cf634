"""Programmatic launches: which kernels may let a dependent start early.

A kernel that triggers lets the next kernel of the stream start beside it, if that one was launched as a programmatic
dependent.  Inside a call that is the library's own next kernel, which allocates tensor memory only after its wait.  After
the last kernel of a call it would be somebody else's, which may allocate first and then wait for good.  So a trigger
stands only in kernels that another launch of the same call always follows, or behind the condition that one does.
"""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turboquant-pytorch_b200", "csrc")
ALWAYS_FOLLOWED = {
    "k_project_rows_two": "k_qjl_score_packed",
    "k_qjl_query_operand": "k_umma_qjl_scores",
    "k_v2_operand_image": "k_umma_v2_stage",
    "k_decode_attn": "k_decode_finish",
}
FOLLOWED_IF = {"k_project_rows": "if (followed)", "k_score_mma": "if (stats != nullptr)", "k_umma_v2_stage": "if constexpr (STAGE != 3)"}


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            kernel = re.search(r"\b(k_\w+)\s*\(", text[a:b])
            yield kernel.group(1), text[a:b]


TRIGGERING = {name: body for name, body in _kernels() if "pdl_trigger()" in body}


def test_the_kernels_that_trigger_are_known():
    assert set(TRIGGERING) == set(ALWAYS_FOLLOWED) | set(FOLLOWED_IF)


@pytest.mark.parametrize("name", sorted(FOLLOWED_IF))
def test_the_last_kernel_of_a_call_does_not_trigger(name):
    assert re.search(re.escape(FOLLOWED_IF[name]) + r"\s*pdl_trigger\(\);", TRIGGERING[name])


@pytest.mark.parametrize("name", sorted(n for n, body in _kernels() if "pdl_wait()" in body and "tmem_alloc(" in body))
def test_tensor_memory_is_allocated_after_the_wait(name):
    body = dict(_kernels())[name]
    assert body.index("pdl_wait()") < body.index("tmem_alloc(")
