"""Every entry point that launches a walk reads the device's error word before
it returns (a walk that gave up leaves truncated sums and says so there only)."""
from __future__ import annotations

import re

import pytest

from conftest import ROOT

CSRC = ROOT / "barnes-hut_gb300" / "csrc"
WALKS = re.compile(r"\b(?:launch_traverse|launch_exact_walk|launch_collect|step_once|step_graph)\(")


def entry_points():
    """(name, body) of the C entry points that launch walks."""
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"^(?:extern \"C\" )?int (bh_\w+)\([^;{]*?\)\n\{\n(.*?)^\}", text, re.S | re.M):
            if WALKS.search(m.group(2)):
                yield m.group(1), m.group(2)


@pytest.mark.parametrize("name", sorted(name for name, _ in entry_points()))
def test_reads_the_error_word(name):
    body = dict(entry_points())[name]
    after = body[max(m.end() for m in WALKS.finditer(body)):]
    # past the last launch nothing returns but a failure, the error word's
    # status (finish, bh_context_sync), or success after the word was copied
    # back and looked at
    checked = "kErrOverflow" in after
    reads = ("finish(", "bh_context_sync(")
    for ret in re.findall(r"return ([^;]*);", after):
        assert ret == "rc" or "bh_fail" in ret or any(r in ret for r in reads) or checked, f"{name}: return {ret}"
    assert checked or any(r in after for r in reads)
