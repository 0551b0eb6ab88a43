"""Host checks of counts against the 32-bit offsets they are stored in
(tsr_b200/csrc/limits.h), compiled on their own: the sizes where they decide
are beyond what a test can build."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tsr_b200" / "csrc"

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "limits.h"
int main(int argc, char **argv) {
    for (int i = 1; i < argc; ++i) {
        uint32_t entries = 0;
        if (tsr::neighbor_entries(std::strtoull(argv[i], nullptr, 10), &entries)) std::printf("%u\\n", entries);
        else std::printf("refused\\n");
    }
}
"""


def test_neighbor_entries_that_32_bits_cannot_address_are_refused(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no host compiler")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    subprocess.run([cc, "-std=c++17", "-I", str(CSRC), str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    # the largest number of edges the events allow is six a leaf, 2^32 - 2; a
    # 32-bit sum of the row lengths wraps from 2^31 edges on
    edges = [0, 1, 6 * 89335, 2**31 - 1, 2**31, 2**31 + 1, 2**32 - 2]
    r = subprocess.run([str(tmp_path / "p")] + [str(e) for e in edges], capture_output=True, text=True, check=True)
    want = [str(2 * e) if 2 * e < 2**32 - 1 else "refused" for e in edges]
    assert r.stdout.split() == want

