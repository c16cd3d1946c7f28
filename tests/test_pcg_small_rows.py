"""Small rows of the persistent PCG over its CTAs: a launch is made only with as many
CTAs as hold the coupled levels.  CTA b of c keeps levels b, b + c, ... in kPcgOwnRows
places of shared memory; the header is compiled here for its host side and the
dispatch's rule compared with that count for every number of CTAs and levels."""

import subprocess

import __graft_entry__ as ge

SOURCE = r"""
#include <cstdio>
#include "pcg_kernels.cuh"
using namespace b200fe;
int main() {
    int wrong = 0, refused = 0;
    for (int ctas = 1; ctas <= 160; ++ctas)
        for (int SG = 0; SG <= kPcgMaxSG + 2; ++SG) {
            int most = 0;  // levels of the CTA with the most
            for (int b = 0; b < ctas; ++b) {
                int k = 0;
                for (int h = b; h < SG; h += ctas) ++k;
                most = k > most ? k : most;
            }
            const bool fit = most <= kPcgOwnRows && SG <= kPcgMaxSG;
            wrong += pcg_rows_fit(ctas, SG) != fit;
            refused += !fit && SG <= kPcgMaxSG;
            if (ctas >= kPcgMinCtas && SG <= kPcgMaxSG && !fit) ++wrong;
        }
    std::printf("%d %d\n", wrong, refused);
    return 0;
}
"""


def test_launches_hold_every_small_row(tmp_path):
    build = ge.load_module("build")
    src = tmp_path / "rows.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "rows"
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    f"-I{build.CSRC}", f"-I{build.ROOT / 'include'}", "-o", str(exe), str(src)], check=True)
    wrong, refused = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert int(wrong) == 0 and int(refused) > 0
