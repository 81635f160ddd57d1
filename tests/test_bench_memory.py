"""CPU: the benchmark's end-to-end leg leaves C on the device where host memory does not hold it."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    sys.path.insert(0, ROOT)
    import bench
    return bench


def _root(tmp_path, available_kb, groups):
    (tmp_path / "proc").mkdir()
    (tmp_path / "proc" / "meminfo").write_text("MemTotal: 99999999 kB\nMemAvailable:   %d kB\n" % available_kb)
    for name, text in groups.items():
        f = tmp_path / "sys" / "fs" / "cgroup" / name
        f.parent.mkdir(parents=True, exist_ok=True)
        f.write_text(text)
    return str(tmp_path)


@pytest.mark.parametrize("groups,want", [
    ({}, 1000 << 10), ({"memory.max": "max\n", "memory.current": "5\n"}, 1000 << 10),
    ({"memory.max": "600000\n", "memory.current": "100000\n"}, 500000),
    ({"memory.max": "60\n", "memory.current": "100\n"}, 0),
    ({"memory/memory.limit_in_bytes": "9223372036854771712", "memory/memory.usage_in_bytes": "7"}, 1000 << 10),
    ({"memory/memory.limit_in_bytes": "700000", "memory/memory.usage_in_bytes": "200000"}, 500000)])
def test_host_memory(bench, tmp_path, groups, want):
    assert bench.host_memory(_root(tmp_path, 1000, groups)) == want


def test_this_host(bench):
    assert bench.host_memory() > 0


@pytest.mark.parametrize("have,want", [(196e9, True), (115e9, True), (112e9, False), (62e9, False)])
def test_headline_output(bench, have, want):
    c, a = 12 * 8583661418 + 8 * 2097153, 12 * 134217728 + 8 * 2097153  # 103 GB and 1.6
    assert bench.output_in_host_memory(c, a, have) is want
