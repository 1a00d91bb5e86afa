"""What the library keeps for the whole process is read and written by several host threads at once: function-local statics
are constants, atomics, per-device records of atomics, or guarded by a mutex beside them."""
import pathlib
import re

CSRC = pathlib.Path(__file__).parents[1] / "stokesflow.jl_b200" / "csrc"


def test_no_unguarded_function_local_statics():
    bad = []
    for f in sorted(CSRC.glob("*.cu*")):
        lines = f.read_text().splitlines()
        for n, line in enumerate(lines):
            # an indented static variable (functions and file-scope state are not indented)
            if not re.match(r"\s+static\s", line) or re.match(r"\s+static\s+(const|constexpr)\b", line):
                continue
            if re.match(r"\s+static\s+(PerDevice|std::atomic<.*>|std::mutex)\s", line) or re.search(r"\)\s*(const)?\s*{", line):
                continue
            if "std::lock_guard" in "\n".join(lines[n:n + 4]):
                continue
            bad.append(f"{f.name}:{n + 1}: {line.strip()}")
    assert not bad, "\n".join(bad)
