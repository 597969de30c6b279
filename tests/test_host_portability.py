"""The library's host code names no instruction of one CPU outside a check for
it (GPU hosts are x86 and Arm)."""
import platform
import re
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "turbogp_b200" / "csrc"


def test_cpu_builtins_stand_in_one_checked_place():
    users = [p.name for p in sorted(CSRC.iterdir())
             if re.search(r"__builtin_ia32|_mm_pause|immintrin|x86intrin|cpuid", p.read_text())]
    assert users == ["cpu_relax.hpp"]


@pytest.mark.skipif(platform.machine() != "x86_64", reason="compiles for x86 and pretends to be another")
@pytest.mark.parametrize("flags", [[], ["-U__x86_64__", "-U__i386__"], ["-U__x86_64__", "-U__i386__", "-D__aarch64__"]])
def test_spin_step_compiles_for(tmp_path, flags):
    src = tmp_path / "relax.cpp"
    src.write_text('#include "cpu_relax.hpp"\nvoid f() { tgp::cpu_relax(); }\n')
    asm = tmp_path / "relax.s"
    subprocess.run(["g++", "-std=c++17", "-O2", "-S", *flags, f"-I{CSRC}", str(src), "-o", str(asm)], check=True)
    text = asm.read_text()
    assert bool(re.search(r"\bpause\b|\brep;?\s*nop", text)) == (not flags) and ("yield" in text) == ("-D__aarch64__" in flags)
