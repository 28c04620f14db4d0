"""What a host thread keeps of a device's answers (dem_device.cuh) is kept per device: the header compiled
for the host with a counter in place of the device."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "cabanadem_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "dem_device.cuh"
int main() {
    b200dem::PerDevice kept;
    int asked = 0;
    auto ask = [&](int dev) { ++asked; return 100 + dev; };
    bool ok = kept.get(0, ask) == 100 && kept.get(3, ask) == 103 && asked == 2;      // each device asked once
    ok = ok && kept.get(0, ask) == 100 && kept.get(3, ask) == 103 && asked == 2;
    ok = ok && kept.get(b200dem::kMaxDevices, ask) == 164 && kept.get(b200dem::kMaxDevices, ask) == 164 && asked == 4;
    ok = ok && kept.get(-1, ask) == 99 && asked == 5;
    std::printf("%s %d\n", ok ? "ok" : "bad", asked);
    return ok ? 0 : 1;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="no host compiler")
def test_each_device_is_asked_once(tmp_path):
    src = tmp_path / "dev.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "dev"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def test_kernels_with_raised_shared_memory_are_asked_per_device():
    """A kernel whose dynamic shared memory is raised once and then launched from a kept grid size."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"static thread_local int [^;]*;", text):
            body = text[m.end():m.end() + 900].split("\n}\n")[0]
            assert "cudaFuncSetAttribute" not in body, (name, m.group(0))
