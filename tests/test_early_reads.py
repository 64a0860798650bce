"""Kernels that may start while the one ahead still runs read what it wrote past L1 (``fresh`` and its like in
``csrc/common.cuh``): a race cannot be made to show, so the sources are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ginfer_b200", "csrc")


def code_of(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


# operands that the kernel ahead made and scratch that goes from kernel to kernel, by the names they have there
@pytest.mark.parametrize("name, pointers, shared", [
    ("decay_chunk.cu", "q k v g c starts nstarts scores gains src S from gain n0 slot", ("a", "b + 64 * n + 4 * tx"))])
def test_operands_and_scratch_are_read_past_l1(name, pointers, shared):
    code = code_of(name)
    for p in pointers.split():
        plain = [m for m in re.findall(r"[^\n]*(?<![\w.>])%s\s*\[[^\n]*" % p, code)
                 if not re.search(r"(?<![\w.>])%s\s*\[[^\]]*\]\s*=[^=]" % p, m)]        # (stores may be plain)
        assert not plain, (p, plain)
    quads = re.findall(r"(?<!__ldcg\()reinterpret_cast<const float4\*>\(([^;]*?)\);", code)
    assert set(quads) == set(shared)                 # four at once without __ldcg: out of shared memory only
