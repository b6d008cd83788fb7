"""Rules of the kernels' inline loads that no run would show: a load of memory
that kernels write is volatile, so that the compiler keeps it behind barriers
and behind the wait of a kernel launched ahead.  Only loads through the
read-only path (.nc), of tables that no kernel writes in a run, may be moved."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fundem_b200", "csrc")


def test_loads_of_written_memory_are_volatile():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        for m in re.finditer(r"\basm(\s+volatile)?\s*\(\s*\"ld\.global([^ ]*) ", text):
            found += 1
            assert m.group(1) or ".nc" in m.group(2), (name, m.group(0))
    assert found >= 4
