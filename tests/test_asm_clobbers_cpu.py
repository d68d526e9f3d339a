"""Inline assembly that orders memory says so.  A barrier (or an asynchronous
copy and its wait) whose asm names no "memory" leaves the compiler free to move
the loads and stores of other variables across it."""
from __future__ import annotations

import re

import pytest

from conftest import ROOT

CSRC = ROOT / "barnes-hut_gb300" / "csrc"


def statements():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for m in re.finditer(r"\basm\b[^;{}]*?\((?:[^()\"]|\"(?:[^\"\\]|\\.)*\"|\([^()]*(?:\([^()]*\)[^()]*)*\))*\)\s*;",
                             path.read_text()):
            yield path.name, m.group(0)


@pytest.mark.parametrize("mnemonic", ["bar.", "griddepcontrol.", "cp.async."])
def test_ordering_asm_clobbers_memory(mnemonic):
    found = [(name, s) for name, s in statements() if mnemonic in s]
    assert found
    bare = [f"{name}: {s}" for name, s in found if '"memory"' not in s or "volatile" not in s]
    assert not bare, bare
