"""A kernel's shared-memory limit belongs to a device: on a second device in
the same process it has to be raised again, so no source raises one in an
initialiser that runs once per process."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nasoq_gb300", "csrc")


@pytest.mark.parametrize("name", ["mlp.cu"])
def test_not_once_per_process(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    assert "cudaFuncSetAttribute" in text
    assert not re.search(r"static[^;{}]*=\s*cudaFuncSetAttribute", text)
    assert not re.search(r"static\s+bool[^;]*;[^{}]*\{\s*[A-Z_]*\(?cudaFuncSetAttribute", text)
