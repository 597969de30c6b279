"""The Rust build script compiles every CUDA source that the Python build does and
rebuilds when any of their headers changes."""
import re

from conftest import ROOT
from turbogp_b200 import build

SCRIPT = (ROOT / "integration" / "rust" / "build.rs").read_text()


def names(pattern):
    return re.findall(r'"([^"]+)"', re.search(pattern, SCRIPT, re.S).group(1))


def test_sources():
    assert names(r"const SOURCES: \[&str; \d+\] = \[(.*?)\];") == build.SOURCES
    assert int(re.search(r"const SOURCES: \[&str; (\d+)\]", SCRIPT).group(1)) == len(build.SOURCES)


def test_headers():
    want = sorted(p.name for p in build.CSRC.iterdir() if p.suffix in (".hpp", ".cuh"))
    assert sorted(names(r"for header in \[(.*?)\]")) == want
