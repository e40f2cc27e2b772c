"""Order of the programmatic-launch instructions in the kernel sources (csrc/launch.cuh has the rules). A wrong order is a race
that timing may hide, so it is looked for in the text."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "csrc"
TEXT = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu"))}


def _kernels():
    """name -> body of every __global__ function."""
    out = {}
    for text in TEXT.values():
        text = re.sub(r"__(?:launch_bounds|cluster_dims)__\([^()]*\)", "", text)
        for m in re.finditer(r"__global__\s+void\s+(\w+)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            out[m.group(1)] = text[m.end():i]
    return out


KERNELS = _kernels()


def test_kernels_that_let_their_successor_start_wait_themselves():
    found = [name for name, body in KERNELS.items() if "pdl_launch_dependents" in body]
    assert len(found) >= 10
    assert not [name for name in found if "pdl_wait" not in KERNELS[name]]


def test_programmatic_launches_are_of_kernels_that_wait():
    launched = {m for text in TEXT.values() for m in re.findall(r"launch_(?:early|pdl)\(cb::(\w+)", text)}
    assert len(launched) >= 10
    assert not [name for name in launched if "pdl_wait" not in KERNELS[name]]


@pytest.mark.parametrize("name", ["decode_begin_kernel"])
def test_the_start_of_a_decode_step_is_a_full_dependency(name):
    """The GEMMs of a step request weights ahead of their own wait. They may start only when everything that ran before the step is
    complete, so the step's first kernel lets them start behind its wait."""
    body = KERNELS[name]
    assert body.index("pdl_wait()") < body.index("pdl_launch_dependents()")


def test_kernels_that_wait_for_a_peer_trigger_on_request_only():
    """Outside the layers of a decode step nothing starts behind a kernel that still waits for its peers."""
    waiting = [name for name, body in KERNELS.items() if "barrier_device" in body and "pdl_launch_dependents" in body]
    assert waiting == ["allreduce_norm_kernel"]
    for name in waiting:
        assert re.search(r"if \(early\) pdl_launch_dependents\(\);", KERNELS[name]) and KERNELS[name].count("pdl_launch_dependents") == 1
