"""What a kernel that gave up a wait leaves in the status word, and what the user reads of it (no device)."""
import glob
import os
import re

import pytest
import torch

from bitnet_c_b200.csrc import build, ops


def _codes():
    for path in sorted(glob.glob(os.path.join(os.path.dirname(build.__file__), "*.cu"))):
        with open(path) as f:
            for name, code in re.findall(r"#define (\w+_ERR_\w*WAIT) (\d+)", f.read()):
                yield os.path.basename(path)[:-3], name, int(code)


def test_codes_are_distinct():
    codes = [code for *_, code in _codes()]
    assert len(codes) >= 8 and len(set(codes)) == len(codes)


@pytest.mark.parametrize("family,name,code", list(_codes()))
def test_every_code_names_its_kernel(monkeypatch, family, name, code):
    cpu = torch.device("cpu")
    monkeypatch.setattr(ops, "_tc_status", {})
    monkeypatch.setattr(ops, "_scratch", {})
    monkeypatch.setattr(ops, "_SCRATCH_FLOATS", 1)
    ops.check_tc_status(cpu)
    ops.tc_status(cpu).fill_(code)
    with pytest.raises(ops.KernelError, match=rf"^{family}: "):
        ops.check_tc_status(cpu)
    ops.check_tc_status(cpu)  # reported once


def test_loads_of_tensor_memory_wait_in_their_own_statement():
    """A load's registers are valid behind its wait only, and nothing ties a use of them to a wait in a statement of its own."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(os.path.dirname(build.__file__), "*.cu*"))):
        with open(path) as f:
            for statement in re.findall(r"asm volatile\((.*?)\);", f.read(), re.S):
                if "tcgen05.ld" in statement or "tcgen05.wait::ld" in statement:
                    seen += 1
                    assert "tcgen05.ld" in statement and "tcgen05.wait::ld" in statement, (os.path.basename(path), statement[:80])
    assert seen >= 3
