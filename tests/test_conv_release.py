"""Programmatic dependent launch of the tensor-core kernels, by their source: a
CTA releases the next kernel only behind the barrier that follows its own TMEM
allocation.  A release before it could let the next kernel's CTAs, which wait
for this grid, take the columns that this grid waits for.  Needs no GPU."""
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).parents[1] / "phasefield_coarsening_gb300" / "csrc" / "ppf_nn_conv.cu"


@pytest.mark.parametrize("kernel", ["conv_kernel", "wgrad_kernel"])
def test_release_follows_the_allocation(kernel):
    text = re.sub(r"//[^\n]*", "", SRC.read_text())
    inline = dict(re.findall(r"__forceinline__ void (grid_\w+)\(\) \{(.*?)\n?\}\n", text, re.S))
    body = text[text.index(" " + kernel + "(const"):]
    body = body[:body.index("tmem_dealloc")]
    for name, code in inline.items():
        body = body.replace(name + "()", code)
    alloc, release = body.index("tmem_alloc("), body.index("griddepcontrol.launch_dependents")
    assert body.count("griddepcontrol.launch_dependents") == 1
    assert alloc < body.index("__syncthreads()", alloc) < release
    assert body.index("griddepcontrol.wait") < release
