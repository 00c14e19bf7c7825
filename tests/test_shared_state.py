"""Host state of the native code: what a function remembers between calls is
shared by all threads and devices of a process, so it is constant, or one of the
types that carry their own lock (the engines' register is guarded beside it).
Anything else belongs to an engine, a plan or a server."""
import re

from conftest import ROOT

ALLOWED = re.compile(r"const\b|constexpr\b|std::mutex\b|AttrCache\b|std::vector<std::unique_ptr<Engine>> engines;")


def test_functions_keep_no_unguarded_state():
    found = []
    for f in sorted((ROOT / "voss_gb300" / "csrc").iterdir()):
        if f.suffix not in (".cpp", ".cu", ".h", ".cuh"):
            continue
        for i, line in enumerate(f.read_text().splitlines(), 1):
            m = re.match(r"\s+static\s+(.*)", line)
            if m and "(" not in m[1].split("=")[0] and not ALLOWED.match(m[1]):
                found.append(f"{f.name}:{i}: {line.strip()}")
    assert not found, found
