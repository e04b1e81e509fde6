"""A kernel's shared-memory limit belongs to one device of the process, so no
launcher may remember that it has raised it (jqc.h: contexts are independent,
also those of different devices and host threads)."""

from __future__ import annotations

import glob
import os
import re

import pytest

import jax_examples_b200

CSRC = os.path.join(os.path.dirname(jax_examples_b200.__file__), "csrc")
SOURCES = [f for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))) if "cudaFuncSetAttribute" in open(f).read()]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_shared_memory_limit_is_set_by_every_launch(path):
    text = open(path).read()
    for m in re.finditer(r"cudaFuncSetAttribute\(", text):
        start = text.rfind("\n}", 0, m.start())  # the enclosing function's text before the call
        body = text[start:m.start()]
        kept = re.findall(r"^\s+static (?!constexpr|const )\w[\w ]*", body, re.M)
        assert not kept, f"{os.path.basename(path)}: {kept} outlives the launch"
