"""Shared memory of another CTA of a cluster may be touched only once that CTA has started.  Read from the source, because a
kernel that breaks this is not something to run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flintnsteel_b200", "csrc")


def kernel(file, name):
    """The kernel's text without comments."""
    with open(os.path.join(CSRC, file)) as f:
        text = f.read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    return text[text.index(f" {name}(const SelectArgs a)"):]


@pytest.mark.parametrize("file, name", [("fns_cluster.cuh", "k_cluster"), ("fns_rows.cuh", "k_rows")])
def test_a_cluster_barrier_lies_before_the_first_access_to_another_cta(file, name):
    text = kernel(file, name)
    pointers = re.findall(r"(\w+) = cluster\.map_shared_rank\(", text)  # only an address until it is indexed
    touches = [m.start() for m in re.finditer(r"map_shared_rank\([^;]*?\)->", text)]
    for p in pointers:
        touches += [m.start() for m in re.finditer(rf"\b{p}\[", text)]
    arrive, wait = text.index("cluster.barrier_arrive()"), text.index("cluster.barrier_wait()")
    assert arrive < text.index("griddepcontrol.wait") < wait < min(touches)
    assert "cluster.sync()" not in text[arrive:wait]
