"""CPU test of the scanning sweeps' block size (pbf_gb300/csrc/scan_block.h): a
size that the caller chose is kept at every particle count, 256 too; the
library's own choice is 256 threads below 1,572,864 particles, and at every count
for the sweeps that record no pair lists."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <initializer_list>
#include "scan_block.h"
using namespace pbf;
int main() {
    int bad = 0;
    const uint32_t sizes[] = {1u, 1572863u, 1572864u, 4194303u, 4194304u, 1u << 29};
    const unsigned own[] = {256, 256, 512, 512, 1024, 1024};
    for (int k = 0; k < 6; ++k) {
        for (uint32_t asked : {32u, 96u, 128u, 256u})
            for (unsigned largest : {512u, 1024u})
                for (bool pairs : {false, true})
                    bad += scan_block(asked, sizes[k], pairs, largest) != asked;
        bad += scan_block(0, sizes[k], true, 1024) != own[k];
        bad += scan_block(0, sizes[k], true, 512) != (own[k] < 512 ? own[k] : 512);
        bad += scan_block(0, sizes[k], false, 1024) != 256;
    }
    std::printf("%d bad\n", bad);
    return bad;
}
"""


def test_block_size_rule(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "pbf_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
