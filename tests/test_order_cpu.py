"""Order of the plain algorithm's segments (host code, no device): by lanes, then
by descending length, stable, with the pointers and lanes in that order
(order_by_lanes in csrc/layout.cu), against numpy's stable sort."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, REPO

HARNESS = r"""
#include <cstdio>
#include <vector>

#include "mixed.h"

int main() {
    int cnt;
    if (std::fread(&cnt, 4, 1, stdin) != 1) return 2;
    std::vector<int> ptr(cnt + 1), order, new_ptr;
    std::vector<uint8_t> lanes(cnt);
    if (std::fread(ptr.data(), 4, cnt + 1, stdin) != (size_t)cnt + 1) return 2;
    if (cnt && std::fread(lanes.data(), 1, cnt, stdin) != (size_t)cnt) return 2;
    sihg::order_by_lanes(ptr, lanes, order, new_ptr);
    std::fwrite(order.data(), 4, cnt, stdout);
    std::fwrite(new_ptr.data(), 4, cnt + 1, stdout);
    std::fwrite(lanes.data(), 1, cnt, stdout);
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    from sih_pdhg import _lib

    if not os.path.exists(_lib.LIB_PATH):
        pytest.fail(f"{_lib.LIB_PATH} is missing: build the library first")
    d = tmp_path_factory.mktemp("order")
    src = d / "order_check.cu"
    src.write_text(HARNESS)
    exe = d / "order_check"
    lib_dir = os.path.dirname(_lib.LIB_PATH)
    subprocess.check_call(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(PKG_DIR, "csrc"), "-I",
                           os.path.join(REPO, "include"), str(src), "-o", str(exe), "-L", lib_dir, "-lsih_pdhg",
                           "-Xlinker", "-rpath", "-Xlinker", lib_dir])
    return str(exe)


# empty; one; one thread's most segments and one more than that; several threads
@pytest.mark.parametrize("cnt", [0, 1, 40, 131071, 131072, 300007])
@pytest.mark.parametrize("kind", ["few", "many"])
def test_order_is_the_stable_sort_by_lanes_and_length(harness, cnt, kind):
    """Equal lengths many times over, and lengths around and past the last bucket
    (2,047) some of them twice."""
    rng = np.random.default_rng(cnt)
    lens = rng.integers(0, 7, cnt) if kind == "few" else rng.integers(0, 2050, cnt) * (rng.random(cnt) < 0.01)
    if cnt > 40:
        lens[rng.choice(cnt, 30, replace=False)] = np.repeat([2046, 2047, 2048, 5000, 40000], 6)
    lanes = rng.choice([1, 2, 4, 8, 16, 32], cnt).astype(np.uint8)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    data = np.int32(cnt).tobytes() + ptr.tobytes() + lanes.tobytes()
    out = subprocess.run([harness], input=data, capture_output=True, timeout=60, check=True).stdout
    order = np.frombuffer(out, np.int32, cnt)
    new_ptr = np.frombuffer(out, np.int32, cnt + 1, 4 * cnt)
    new_lanes = np.frombuffer(out, np.uint8, cnt, 8 * cnt + 4)
    ref = np.lexsort((-lens, -lanes.astype(int)))  # stable, the last key first
    np.testing.assert_array_equal(order, ref)
    np.testing.assert_array_equal(new_ptr, np.concatenate([[0], np.cumsum(lens[ref])]))
    np.testing.assert_array_equal(new_lanes, lanes[ref])
