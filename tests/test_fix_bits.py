"""The range of the mixed form's fixed-point accumulator (csrc/tdp_host.h): the adds that a tile's words
get, counted from the kernels' enumeration of items, and as many bits as those leave."""
import os
import subprocess

from tholedipoleplugin_b200 import build as B

SOURCE = r"""
#include "tdp_host.h"

int main() {
    for (long tiles : {1, 2, 3, 13, 33, 64, 125, 384, 1000, 1296, 2031, 3072})
        for (long group : {1, 2})
            for (long chunk : {1, 2, 4, 8, 16})
                for (long parts : {1, 2, 8}) {
                    // Square blocks of max(group, chunk) tiles, p <= q; an item is one group against one chunk.
                    const long side = std::max(group, chunk), nb = (tiles + side - 1) / side;
                    std::vector<long> count(tiles, 0);
                    for (long q = 0; q < nb; q++)
                        for (long p = 0; p <= q; p++)
                            for (long i0 = p * side; i0 < std::min(tiles, (p + 1) * side); i0 += group)
                                for (long j0 = q * side; j0 < std::min(tiles, (q + 1) * side); j0 += chunk) {
                                    const long j1 = std::min(tiles, j0 + chunk), first = std::max(j0, i0);
                                    if (j1 <= first) continue;
                                    for (long j = first; j < j1; j++) count[j] += parts;
                                    for (long i = i0; i < std::min(tiles, i0 + group); i++) count[i] += parts;
                                }
                    long most = 1;
                    for (long c : count) most = std::max(most, c);
                    const long adds = tdp::fix_adds(tiles, group, chunk, parts);
                    const int bits = tdp::fix_bits(adds);
                    if (adds != most || bits > 32 || adds > 1L << (40 - bits) || (bits < 32 && adds <= 1L << (39 - bits))) {
                        printf("%ld tiles, groups of %ld, chunks of %ld, %ld parts: %ld adds, counted %ld, %d bits\n",
                               tiles, group, chunk, parts, adds, most, bits);
                        return 1;
                    }
                }
    return 0;
}
"""


def test_range(tmp_path):
    src, exe = tmp_path / "bits.cpp", tmp_path / "bits"
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", cuda, "-I", os.path.join(B.ROOT, "include"), "-I", B.CSRC, "-o",
                    str(exe), str(src)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
