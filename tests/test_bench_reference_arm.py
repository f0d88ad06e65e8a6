"""The benchmark's reference arm where the reference is not built: the contract's one line, exit code 0."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unavailable_line():
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libqsr_cpu_ref.so")):
        pytest.skip("reference CPU build present")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300, env=dict(os.environ, RANK="0", WORLD_SIZE="1"))
    assert r.returncode == 0, r.stderr[-2000:]
    (line,) = [x for x in r.stdout.splitlines() if x.startswith("{")]
    d = json.loads(line)
    assert d["impl"] == "reference" and "not built" in d["unavailable"] and set(d) == {"impl", "unavailable"}
