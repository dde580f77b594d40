"""What is set once for each device is set for each: host logic alone, built without a GPU."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neurogrid_b200", "csrc")
PROGRAM = r"""
#include "ng_device_once.h"
#include <cstdio>
int main() {
    static std::atomic<unsigned long long> done{0};
    int calls[3] = {0, 0, 0};
    bool works = true;
    auto ask = [&](int device) { return ng_once_per_device(done, device, [&] { ++calls[device]; return works; }); };
    works = false;
    if (ask(1)) return 1;                                   // a failure is reported ...
    works = true;
    for (int i = 0; i < 3; ++i)
        if (!ask(0) || !ask(1) || !ask(2)) return 2;
    printf("%d %d %d", calls[0], calls[1], calls[2]);       // ... and tried again; every device once
    return 0;
}
"""


def test_every_device_is_set_once(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "1 2 1"


def test_float32_path_keeps_no_flag_of_the_process():
    """The libraries that LFM2 runs in float32 on whatever device is current: no limit that only the first device gets."""
    for name in ("gemm_f32", "elementwise", "shortconv", "rope_cache", "attention_generic", "sampling"):
        text = open(os.path.join(CSRC, name + ".cu")).read()
        assert "static bool" not in text and "cudaFuncSetAttribute" not in text, name
