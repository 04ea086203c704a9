"""The window count behind the waits between the streams of the pipelined PCA windows, run past 2^31 and 2^32 windows:
compiled from the pipe's own header."""

import pathlib
import subprocess

from holovibes_gb300 import _build

PROGRAM = r"""
#include "pipe_internal.h"
#include <cstdio>
#include <type_traits>
int main()
{
    using Count = std::remove_reference_t<decltype(hv_pipe{}.pp_w)>;
    for (unsigned long long start : {0ull, (1ull << 31) - 3, (1ull << 32) - 3, (1ull << 40)})
    {
        Count w;
        w.n = start;
        for (unsigned long long k = start; k < start + 9; ++k, ++w.n)
            for (unsigned back = 0; back <= 4; ++back)
            {
                if (w.has(back) != (k >= back))
                    return std::printf("window %llu: has(%u)\n", k, back), 1;
                for (unsigned slots : {2u, 4u})
                    if (k >= back && w.slot(back, slots) != (k - back) % slots)
                        return std::printf("window %llu: slot(%u, %u)\n", k, back, slots), 1;
            }
    }
    return 0;
}
"""


def test_count_past_32_bits(tmp_path):
    src, exe = tmp_path / "count.cpp", tmp_path / "count"
    src.write_text(PROGRAM)
    cuda = pathlib.Path(_build.nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{_build.CSRC}", f"-I{_build.INCLUDE}", f"-I{cuda}", str(src), "-o", str(exe)],
                   check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
