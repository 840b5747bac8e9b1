"""What the launchers remember of a kernel's attributes holds for one device: a second device of the process must be set up too."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocmforge_b200", "csrc")


def sources():
    return [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))]


@pytest.mark.parametrize("path", sources(), ids=os.path.basename)
def test_no_launcher_remembers_attributes_for_all_devices(path):
    with open(path) as f:
        text = f.read()
    assert not re.findall(r"^ +static (?:bool|size_t|int) .*;", text, flags=re.M)


def test_each_device_has_a_note_of_its_own(tmp_path):
    with open(os.path.join(CSRC, "common.cuh")) as f:
        text = f.read()
    struct = re.search(r"template <typename T>\nstruct PerDevice \{.*?\n\};\n", text, flags=re.S).group(0)
    src = tmp_path / "t.cpp"
    src.write_text("""
#include <cstddef>
static int current = 0;
static int cudaGetDevice(int* d) { *d = current; return 0; }
""" + struct + """
static int asked = 0;
static void launch(size_t smem) {
    static PerDevice<size_t> devices;
    size_t& configured = devices.here();
    if (smem > configured) { ++asked; configured = smem; }
}
int main() {
    launch(100); launch(100); launch(50);
    if (asked != 1) return 1;
    current = 1; launch(100); launch(100);
    if (asked != 2) return 2;
    current = 0; launch(100); launch(200);
    if (asked != 3) return 3;
    current = 1; launch(150);
    return asked == 4 ? 0 : 4;
}
""")
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
