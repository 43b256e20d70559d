"""Dynamic shared memory that is read or written in 16-byte pieces says so: its
start is only as aligned as its declaration asks for, and static shared
variables of any size come before it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvdbm-jax_gb300", "csrc")
DECLARED = re.compile(r"extern\s+__shared__\s+(?:__align__\((\d+)\)\s+)?([\w ]+?)\s+(\w+)\[\]")
WIDE = re.compile(r"float4|uint4|int4|cp_async16|cp\.async|tcgen05")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_dynamic_shared_memory_alignment(path):
    src = open(path).read()
    for align, kind, name in DECLARED.findall(src):
        if kind == "double":  # (read as doubles alone)
            continue
        if WIDE.search(src):
            assert align and int(align) >= 16, f"{os.path.basename(path)}: {kind} {name}[] is declared without 16-byte alignment"
