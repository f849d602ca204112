"""The host side of the split engine's buffers (ballasim_b200/csrc/split_bufs.h), built with g++ over a fake device memory
that refuses allocations."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = tmp_path_factory.mktemp("split_bufs") / "split_bufs"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=address", f"-I{ROOT / 'ballasim_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "split_bufs.cc"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("check", ["refused_list", "captured_addresses", "gives_way"])
def test_split_buffers(exe, check):
    r = subprocess.run([str(exe), check], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
