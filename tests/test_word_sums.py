"""The GEMM epilogue's word sums with two 32-bit steps, restated with integers: exact up to the K that
csrc/gemm_tc.cuh allows for gathered operand rows, and not a step of 128 bytes beyond."""
import os
import re

from conftest import PACKAGE_DIR

M32 = (1 << 32) - 1


def short_word_sum(v):
    return ((v[2] + v[3] * 256) & M32) * 65536 + ((v[0] + v[1] * 256) & M32)


def test_short_word_sums_are_exact_up_to_the_gathered_row():
    with open(os.path.join(PACKAGE_DIR, "csrc", "gemm_tc.cuh")) as f:
        k_bytes = int(re.search(r"constexpr uint32_t kGatherRowBytes = (\d+);", f.read()).group(1))
    top = k_bytes * 255 * 255
    for v in ([top] * 4, [top, 0, top, 0], [0, top, 0, top], [1, 2, 3, 4]):
        assert short_word_sum(v) == sum(x << (8 * d) for d, x in enumerate(v))
    beyond = [(k_bytes + 128) * 255 * 255] * 4
    assert short_word_sum(beyond) != sum(x << (8 * d) for d, x in enumerate(beyond))
