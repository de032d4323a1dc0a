"""CPU check of the kernels' sources: a role that touches tensor memory after a barrier wait has a
``tcgen05.fence::after_thread_sync`` in between.  Without it the access is not ordered behind the tcgen05
operations that the barrier reports as done (the previous readers of the columns, for a store)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "b12x_b200" / "csrc"
ACCESS = re.compile(r"\b(sf_atoms_to_tmem<|tc_st_32x32b_x\d+\(|tc_ld_32x32b_x\d+\(|epilogue_tile<|mma_\w+\()")
WAIT = re.compile(r"\bmbar_wait_\w+\(")


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_tensor_memory_is_fenced_after_a_wait(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for kernel in re.finditer(r"__global__.*?\n}\n", text, re.S):
        body = kernel.group(0)
        for hit in ACCESS.finditer(body):
            waits = [m.end() for m in WAIT.finditer(body, 0, hit.start())]
            if waits:
                between = body[waits[-1]:hit.start()]
                assert "tc_fence_after()" in between, f"{name}: {hit.group(0)} with no fence after the wait: ...{between[-200:]}"
