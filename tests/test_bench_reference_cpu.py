"""CPU: bench.py's reference arm where the reference's kernels are not built says so in one line and ends well."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(os.path.isdir(os.path.join(ROOT, "oracle", "_ref")), reason="the reference's kernels are built")
@pytest.mark.parametrize("rank", [0, 1])
def test_unavailable(rank):
    env = dict(os.environ, RANK=str(rank), WORLD_SIZE="2")
    p = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2", "--steps",
                        "1", "--warmup", "3"], capture_output=True, text=True, timeout=300, cwd=ROOT, env=env)
    assert p.returncode == 0, p.stderr[-2000:]
    lines = p.stdout.splitlines()
    if rank:
        assert not lines
    else:
        assert len(lines) == 1
        d = json.loads(lines[0])
        assert d["impl"] == "reference" and d["unavailable"] and "\n" not in d["unavailable"]
