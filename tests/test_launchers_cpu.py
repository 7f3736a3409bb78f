"""Launch shape of the launchers' SpMV (host code, no device): split_launch in
csrc/compat.cuh.  The kernel learns the mean segment length on the device and
goes by groups of lanes or by stream; the grid has to serve both.

* by groups: a warp for every segment, up to the 64 warps an SM holds and not
  past them (a second wave);
* by stream (from 32,768 segments on): a warp for every 32 segments;
* no count up to the largest int gives an empty or a negative grid."""
import os
import subprocess

from conftest import PKG_DIR, REPO

HARNESS = r"""
#include <cstdio>

#include "compat.cuh"

int main() {
    int nseg, sms;
    while (std::scanf("%d %d", &nseg, &sms) == 2) {
        const sihg::SplitLaunch g = sihg::split_launch(nseg, sms);
        std::printf("%d %d %d %d %d\n", g.blocks, g.threads, g.smem, g.group_blocks, sihg::kStreamSegs);
    }
    return 0;
}
"""

SEGMENTS = [1, 3, 4, 5, 31, 500, 9727, 9728, 9729, 32767, 32768, 32769, 40000, 100000, 300000, 311296, 311297,
            1000000, 2**31 - 128, 2**31 - 1]


def test_grid_serves_groups_and_stream(tmp_path):
    src, exe = tmp_path / "grid.cu", tmp_path / "grid"
    src.write_text(HARNESS)
    subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(PKG_DIR, "csrc"), "-I", os.path.join(REPO, "include"),
                    str(src), "-o", str(exe)], check=True)
    for sms in (1, 152):
        text = "".join(f"{n} {sms}\n" for n in SEGMENTS)
        lines = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
        assert len(lines) == len(SEGMENTS)
        for n, line in zip(SEGMENTS, lines):
            blocks, threads, smem, group_blocks, stream_from = map(int, line.split())
            warps = blocks * threads // 32
            assert threads in (128, 256) and blocks >= 1
            group_warps = group_blocks * threads // 32
            assert 1 <= group_blocks <= blocks and min(n, 64 * sms) <= group_warps <= 64 * sms + 7
            # a window for every warp of a block that starts on a unit of 32 segments
            units = -(-n // 32)
            windows = max((units - b + blocks - 1) // blocks for b in (0, blocks - 1)) if n >= stream_from else 0
            assert smem == 2048 * windows <= 2048 * (threads // 32)
            if n >= stream_from:
                assert 32 * warps >= n
