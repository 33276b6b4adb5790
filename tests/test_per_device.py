"""What a launcher does once per device is done on every device of a process: the header that says so, on the host."""
import shutil
import subprocess

import pytest

from quicknn_b200.kernels.build import CSRC

PROGRAM = r"""
#include <initializer_list>
#include "per_device.h"
int main() {
    static qnn::OncePerDevice once;
    int calls[70] = {};
    auto at = [&](int d, int rc) { return once.run(d, [&] { ++calls[d < 0 ? 69 : d]; return rc; }); };
    if (at(1, 7) != 7 || calls[1] != 1) return 1;                // what failed is tried again
    for (int round = 0; round < 3; ++round)
        for (int d : {0, 1, 7, 63}) if (at(d, 0) != 0) return 2;
    if (calls[0] != 1 || calls[1] != 2 || calls[7] != 1 || calls[63] != 1) return 3;
    for (int round = 0; round < 3; ++round) { at(64, 0); at(-1, 0); }
    return calls[64] == 3 && calls[69] == 3 ? 0 : 4;             // beyond what is counted: every time
}
"""


def test_once_on_every_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "a.cpp", tmp_path / "a"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.parametrize("name", ["moe.cu", "memory_chunks.cu"])
def test_experts_and_memories_ask_per_device(name):
    """Their kernels need more shared memory than a kernel has unasked, on whichever device they run."""
    with open(f"{CSRC}/{name}") as f:
        text = f.read()
    assert "static bool" not in text and text.count("cudaFuncSetAttribute") == 0 and "allow_shared(" in text
