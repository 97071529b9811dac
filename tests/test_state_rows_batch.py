"""The batches of the state transfers' row kernels on domains whose rows 32 bits
cannot number: compiled for the host, every batch's row numbers and the step past
its last stay below 2^32, for the largest domains the checks accept."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freeshearlayer_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "fsl_internal.h"
using namespace fsl;
int main()
{
    // LEN, HIG of 2^31 cells with DEP = 2 and 3, from long to wide
    for (int D = 2; D <= 3; D++)
        for (long long H = 2; H <= (1LL << 31) / (2 * D); H *= 2) {
            const long long L = (1LL << 31) / (D * H);
            const long long batch = rows_batch((int)H);
            long long planes = 0, launches = 0;
            if (batch < 1) return 1;
            for (long long b = 0; b < L; b += batch, launches++) {
                const long long ni = L - b < batch ? L - b : batch;
                // the largest row number a warp reaches, its last step past the end included
                if (ni * H * 5 + 8LL * kRowBlocks > 0xffffffffLL) return 2;
                planes += ni;
            }
            if (planes != L) return 3;
            std::printf("%d %lld %lld\n", D, H, launches);
        }
    return 0;
}
"""


def test_row_numbers_fit_in_32_bits(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "rows.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "rows"
    subprocess.run([nvcc, "-std=c++17", "-I" + CSRC, "-I" + os.path.join(CSRC, "..", "..", "include"), "-o", str(exe),
                    str(src)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    launches = [int(line.split()[2]) for line in out.stdout.splitlines()]
    assert max(launches) >= 2  # some domain needs more than one launch
