"""What the library sets once per device (csrc/per_device.cuh, compiled for the host): each device that comes is set, whichever came first, once; a failure
is answered and tried again, and stays with its device; a device past the table is set every time; threads that come at once all find it set.
And every kernel attribute that the sources set is set that way: attributes hold for the device that is current."""
import re
import subprocess

from tinygpt_b200 import build

MAIN = """
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.cuh"
int main() {
  b200::OncePerDevice<int, 8> once;
  int set[16] = {};
  for (int d : {1, 0, 1, 7, 0, 8, 8, 7, -1, -1}) {
    const int e = once(d, [&] { ++set[d + 1]; return 0; });
    if (e != 0) return printf("device %d: %d\\n", d, e), 1;
  }
  if (set[2] != 1 || set[1] != 1 || set[8] != 1 || set[9] != 2 || set[0] != 2) return printf("sets %d %d %d %d %d\\n", set[2], set[1], set[8], set[9], set[0]), 1;
  int tries = 0;
  for (int i = 0; i < 4; ++i) {
    const int e = once(3, [&] { return ++tries < 3 ? 700 : 0; });
    if (e != (i < 2 ? 700 : 0)) return printf("try %d: %d\\n", i, e), 1;
  }
  if (tries != 3) return printf("%d tries\\n", tries), 1;
  for (int round = 0; round < 200; ++round) {
    b200::OncePerDevice<int> fresh;
    std::atomic<int> is_set{0}, bad{0};
    std::vector<std::thread> all;
    for (int t = 0; t < 4; ++t)
      all.emplace_back([&] {
        if (fresh(2, [&] { is_set.store(1); return 0; }) != 0 || is_set.load() != 1) ++bad;
      });
    for (auto& t : all) t.join();
    if (bad.load() != 0) return printf("a thread went on before the device was set\\n"), 1;
  }
  return 0;
}
"""


def test_once_per_device(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(build.CSRC), str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_attributes_are_set_per_device():
    seen = 0
    for src in sorted(build.CSRC.glob("*.cu")):
        text = src.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            before = text[:m.start()]
            start = before.rfind("attrs([] {")   # the function that is handed to the PerDevice is still open here
            assert start >= 0 and "}));" not in before[start:], f"{src.name}:{before.count(chr(10)) + 1}"
            seen += 1
    assert seen > 10
