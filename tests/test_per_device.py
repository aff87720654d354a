"""Per-device values of kernels (d3_per_device.h) and the kernels whose function attributes need them, on the CPU."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "simple-dftd3_b200" / "csrc"

PROGRAM = r"""
#include "d3_per_device.h"
#include <atomic>
#include <thread>
#include <vector>
int main()
{
    d3::PerDevice<int> values;
    int k1, k2;
    std::atomic<int> made{0};
    auto make = [&](int& v) { v = ++made; return true; };
    // once for each device and kernel
    if (values.get(0, &k1, make) != 1 || values.get(0, &k1, make) != 1) return 1;
    if (values.get(1, &k1, make) != 2 || values.get(0, &k2, make) != 3 || values.get(1, &k1, make) != 2) return 2;
    // a failure is not kept
    if (values.get(2, &k1, [](int&) { return false; }) != 0 || values.get(2, &k1, make) != 4) return 3;
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; t++) threads.emplace_back([&] { values.get(3, &k1, make); });
    for (auto& t : threads) t.join();
    return made == 5 ? 0 : 4;
}
"""


def test_values_belong_to_device_and_kernel(tmp_path):
    (tmp_path / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), "-o", str(tmp_path / "p"), str(tmp_path / "p.cpp")],
                   check=True)
    assert subprocess.run([str(tmp_path / "p")]).returncode == 0


def test_attributes_are_set_through_it():
    for path in CSRC.glob("*.cu"):
        text = path.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            before = text[:m.start()]
            assert before.rfind("PerDevice<") > before.rfind("\n}\n"), path.name
