"""populate_pages: a host array's pages made resident without a change of its contents."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("offset,size", [(0, 0), (5, 1), (0, 4 << 20), (16, (4 << 20) - 1), (24, (9 << 20) + 3),
                                         (8, 70 << 20)])
def test_contents_and_residency(tmp_path, offset, size):
    exe = tmp_path / "host_pages_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-o", str(exe), os.path.join(HERE, "host_pages_check.cpp")],
                   check=True)
    r = subprocess.run([str(exe), str(offset), str(size)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    n, pages, resident, page = map(int, r.stdout.split())
    if size >= 70 << 20 and tuple(map(int, os.uname().release.split("-")[0].split(".")[:2])) >= (5, 14):
        assert resident == pages
