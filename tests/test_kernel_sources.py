"""Rules of programmatic dependent launch that a kernel's source has to keep; a broken one shows on the device now and then
only, so it is looked for in the text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tinyserve_b200", "csrc")


def kernels():
    """{(file, kernel): (parameters, body)} of every __global__ function."""
    found = {}
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        with open(os.path.join(CSRC, name)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__", text):
            brace = text.index("{", m.start())
            semicolon = text.find(";", m.start())
            if 0 <= semicolon < brace:
                continue
            head = re.sub(r"__(?:launch_bounds|maxnreg)__\s*\((?:[^()]|\([^()]*\))*\)", "", text[m.start():brace])
            depth, end = 0, brace
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
                end += 1
            found[(name, re.search(r"(\w+)\s*\(", head).group(1))] = (head[head.index("("):], text[brace:end])
    return found


def test_every_kernel_is_found():
    names = kernels()
    assert len(names) > 70 and ("gemv_mma.cu", "gemv_mma_kernel") in names


# the kernels that write lengths, positions, slots or block tables, which attention kernels read ahead of their wait
@pytest.mark.parametrize("kernel", ["block_table_gather_kernel", "sanitize_step_kernel", "sanitize_group_kernel"])
def test_nothing_is_launched_ahead_of_the_step_indices(kernel):
    _, body = kernels()[("elementwise.cu", kernel)]
    assert "pdl_wait();" in body and "pdl_trigger" not in body
    assert body.rstrip().endswith("__threadfence();")


# what no kernel of a step writes: the embedding, tables of angles, logits of attention sinks
CONSTANTS = {"table", "cos", "sin", "vcos", "vsin", "sinks"}


def test_what_a_predecessor_wrote_is_not_declared_constant():
    """A load through a `const ... __restrict__` parameter may be brought forward over the dependency wait."""
    for (name, kernel), (parameters, body) in kernels().items():
        declared = set(re.findall(r"const\s+[\w:<>]+\s*\*\s*__restrict__\s+(\w+)", parameters))
        assert declared <= CONSTANTS, f"{name}: {kernel} declares {sorted(declared - CONSTANTS)} constant"
        assert "griddepcontrol" not in body        # (kernels wait through pdl_wait)
