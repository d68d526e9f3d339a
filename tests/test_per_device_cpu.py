"""What is asked of a device once is kept for that device, not for the process:
the cache (csrc/bh_per_device.h), and no other process-wide answer from the CUDA
runtime in the sources."""
from __future__ import annotations

import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "barnes-hut_gb300" / "csrc"
SOURCE = r"""
#include "bh_per_device.h"
int main()
{
    static bh::PerDevice p;
    int asked = 0;
    auto ask = [&](int v) { return [&asked, v] { ++asked; return v; }; };
    int bad = 0;
    bad += p.get(0, 8, ask(16)) != 16;
    bad += p.get(1, 8, ask(8)) != 8;      // another device, another answer
    bad += p.get(0, 8, ask(4)) != 16;     // kept
    bad += asked != 2;
    bad += p.get(2, 8, ask(0)) != 8;      // cannot be had: not kept
    bad += p.get(2, 8, ask(16)) != 16;
    bad += p.get(-1, 8, ask(3)) != 3;     // outside the table: asked each time
    bad += p.get(64, 8, ask(0)) != 8;
    return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_kept_per_device(tmp_path):
    src, exe = tmp_path / "per.cpp", tmp_path / "per"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_process_wide_answers():
    """No function-local static is initialised by a call (lambda or runtime)."""
    found = [f"{p.name}: {m.group(0)}" for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.cpp")])
             for m in re.finditer(r"^\s+static (?:const )?(?:int|bool|int64_t|size_t) \w+ = (?:\[|\w+\().*$",
                                  p.read_text(), re.M)]
    assert not found, found
