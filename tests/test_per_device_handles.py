"""Streams and events that a thread keeps between calls are kept per device: a
thread that changes its device gets others (an event made on one device cannot
be recorded on another's streams).  CPU only.
"""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rtdl_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <stdexcept>
#include "per_device.cuh"
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
  int made = 0;
  rtdl_b200::PerDevice<int> handles;
  auto get = [&](int device, int which) { return handles.get(device, which, [&] { return ++made; }); };
  const int a = get(0, 0), b = get(0, 1), c = get(1, 0);
  CHECK(a != b && a != c && b != c && made == 3);
  CHECK(get(0, 0) == a && get(0, 1) == b && get(1, 0) == c && made == 3);
  bool threw = false;
  try { handles.get(2, 0, []() -> int { throw std::runtime_error("no device"); }); } catch (const std::exception&) { threw = true; }
  CHECK(threw);
  const int d = get(2, 0);
  CHECK(d == 4 && get(2, 0) == d);
  return 0;
}
"""


def test_handles_are_kept_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / "per_device.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(src), "-o", str(tmp_path / "per_device")], check=True)
    done = subprocess.run([str(tmp_path / "per_device")], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def test_no_stream_or_event_is_kept_without_its_device():
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        kept = re.findall(r"\b(?:static|thread_local)\s[^;(]*cuda(?:Event|Stream)_t[^;]*;", path.read_text())
        bare = [k for k in kept if "PerDevice<" not in k and "std::map<int, cudaStream_t>" not in k]
        assert not bare, (path.name, bare)
