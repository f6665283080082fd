"""Orders in the kernels' sources that no run can show to be wrong without hanging a GPU."""
import os
import re

from conftest import cg

CSRC = os.path.join(os.path.dirname(cg.__file__), "csrc")


def kernel(file, name):
    """The source of one kernel's definition."""
    text = open(os.path.join(CSRC, file)).read()
    begin = re.search(rf"\b{name}\(const __grid_constant__", text).start()
    return text[begin:text.index("\n}\n", begin)]


def places(body, *instructions):
    """Where each stands; all must stand there exactly once."""
    assert all(body.count(i) == 1 for i in instructions), [body.count(i) for i in instructions]
    return [body.index(i) for i in instructions]


def test_prompt_attention_takes_tmem_between_its_dependency_and_its_trigger():
    """A CTA that wants most of an SM's TMEM: after the wait no earlier kernel holds columns, and before the trigger no later
    kernel runs.  The other way round a dependent's CTA could hold columns and wait for a kernel that waits for them."""
    for name in ("k_attn_fa", "k_attn_fq"):
        wait, alloc, trigger = places(kernel("attention_fa.cu", name), "griddepcontrol.wait;", "tcgen05.alloc.", "griddepcontrol.launch_dependents;")
        assert wait < alloc < trigger
