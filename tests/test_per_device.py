"""What a launcher does once per device is done on every device of a process: the header that says so, on the host."""
import os
import re
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


KNOWN = r"""
#include "per_device.h"
int main() {
    static qnn::KnownPerDevice known;
    int calls = 0;
    auto at = [&](int d, unsigned key, int answer) { return known.get(d, key, [&] { ++calls; return answer; }); };
    if (at(0, 0, 7) != 7 || at(1, 0, -1) != -1 || calls != 2) return 1;              // every device is asked
    if (at(0, 0, 9) != 7 || at(1, 0, 9) != -1 || calls != 2) return 2;               // once
    if (at(0, 4096, 5) != 5 || at(0, 4096, 6) != 5 || calls != 3) return 3;          // and again for another question
    if (at(0, 0xfffffffeu, 0) != 0 || at(0, 0xfffffffeu, 1) != 0 || calls != 4) return 4;
    if (at(64, 0, 1) != 1 || at(64, 0, 2) != 2 || at(-1, 0, 3) != 3 || calls != 7) return 5;      // beyond what is counted: every time
    return 0;
}
"""


def test_what_a_device_holds_is_known_per_device_and_question(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "a.cpp", tmp_path / "a"
    src.write_text(KNOWN)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_no_launcher_keeps_a_flag_or_an_occupancy_for_the_process(name):
    """Attributes of a kernel, SM counts and occupancies are a device's: a flag for the process would leave the second device without."""
    with open(f"{CSRC}/{name}") as f:
        text = f.read()
    assert not re.search(r"static (bool|int) (configured|set|known|fits|sm_count|max_pairs|split_ok)\b", text)
