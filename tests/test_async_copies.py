"""Asynchronous copies into shared memory are waited for, on every lane.

A lane's `cp.async` copies that were never committed to a group are not
covered by `cp.async.wait_group`, so a kernel in which some lanes copy and
then wait without a commit between reads what has not arrived.  No result
shows that reliably; the rule is checked on the source: the wait that ends
every use takes in uncommitted copies, and no kernel copies without a commit
of its own before the next wait."""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hamstr_oop_gb300", "csrc")


def _source():
    with open(os.path.join(CSRC, "mixed.cu")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_final_wait_takes_in_uncommitted_copies():
    body = re.search(r"void cp_async_wait_all\(\)\s*\{(.*?)\}", _source(), re.S).group(1)
    assert "cp.async.wait_all;" in body


def test_copies_shared_between_lanes_are_committed_by_every_lane():
    """The boundary system's factors are copied by all lanes, also by those
    without a segment, which take no other path to a commit."""
    src = _source()
    kernel = src[src.index("void __launch_bounds__(32) mx_spike_solve_kernel"):]
    copies = [m.end() for m in re.finditer(r"cp_async16_cg\(red_s[^;]*;", kernel)]
    assert copies
    assert kernel[copies[-1]:].lstrip().startswith("cp_async_commit();")
