"""Kernels launched so that they may be scheduled before their predecessor has
finished (launch_pdl, launch_pdl_if) wait for it first, and what their addresses
are formed from -- the thread's index, or every pointer they read through the
read-only path -- is tied to that wait: such a load could otherwise be moved
ahead of it by the compiler."""
import re

import pytest

from conftest import ROOT

CSRC = ROOT / "high_precision_blas1_b200" / "csrc"


def sources():
    return {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}


def early_kernels():
    """(file, kernel) of every kernel given to launch_pdl or launch_pdl_if."""
    names = set()
    for text in sources().values():
        for call in re.finditer(r"launch_pdl(?:_if)?\(([^;]*);", text):
            names |= set(re.findall(r"\b(\w+_kernel)\b", call.group(1)))
        # kernels handed to a local launcher: go(kernel<...>)
        if "launch_pdl" in text:
            names |= set(re.findall(r"\bgo\((\w+_kernel)<", text))
    return [(f, k) for k in sorted(names) for f, text in sources().items()
            if re.search(r"\b" + k + r"\(\s*int", text)]


def test_there_are_such_kernels():
    assert {k for _, k in early_kernels()} >= {"reduce_kernel", "map_kernel", "csr_row_kernel", "csr_row_dot_kernel"}


@pytest.mark.parametrize("name,kernel", early_kernels())
def test_reads_follow_the_wait(name, kernel):
    text = sources()[name]
    at = re.search(r"\b" + kernel + r"\((\s*int[^{]*)\)\s*\{", text)
    params, body = at.group(1), text[at.end():]
    body = body[:re.search(r"^}", body, re.M).start()]
    wait = re.search(r"\bpdl_\w+_for\(([^)]*)\)", body)
    before, after = body[:wait.start()], body[wait.end():]
    assert not re.search(r"__ldg|ld\w*E\(|ld_\w+<|ld16|\w\[\w", before), "a load before the wait"
    tied = {a.strip() for a in wait.group(1).split(",")}
    read_only = {re.search(r"(\w+)\s*(?:=.*)?$", p.strip(), re.S).group(1) for p in params.split(",")
                 if "const" in p and "*" in p}
    assert read_only
    if len(tied) == 1:
        index = tied.pop()
        assert re.search(index + r" = [^;]*blockIdx\.x[^;]*threadIdx\.x", before), "the thread's index"
        # no other index is formed from the block's and the thread's numbers
        assert not re.search(r"blockIdx\.x\s*\)?\s*\*", after)
        assert not re.search(r"\bt = (?:int\()?threadIdx|\bld\w*(?:<\w+>)?\(\w+, (?:int\()?threadIdx", after)
    else:
        assert read_only <= tied


def test_the_wait_is_not_made_without_pointers():
    for name, text in sources().items():
        assert not re.search(r"\bpdl_enter\(\)", text), name
        if name != "hpb_common.cuh":
            assert "cudaGridDependencySynchronize" not in text, name
