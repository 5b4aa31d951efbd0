"""Kernels of a chain of launches may start before the kernel ahead of them has written its results
(csrc/launch.cuh), so they may promise the compiler constant memory (const __restrict__, __ldg) for a
plan's tables only. Checked on the source."""
import glob
import os
import re

from conftest import PACKAGE_DIR

# pointers to tables that a plan builds before its first product
TABLES = {"primes", "fwd", "inv", "zeta", "table", "stage", "forward", "inverse", "q"}


def functions(text):
    """(head, body) of every function definition at namespace level."""
    for match in re.finditer(r"^(?!namespace|struct|class|enum|extern|constexpr|#)(?:[^\n;{}]*\n)*?[^\n;{}]*\)[^\n;{}]*\{\n",
                             text, re.M):
        end = text.find("\n}\n", match.end())
        yield match.group(0), text[match.end():end]


def test_only_tables_are_promised_constant():
    chained = 0
    for path in sorted(glob.glob(os.path.join(PACKAGE_DIR, "csrc", "*.cu*"))):
        for head, body in functions(open(path).read()):
            kernel = "__global__" in head
            if kernel and "chain_enter()" not in body and "chain_wait()" not in body:
                continue  # launched in plain stream order
            chained += kernel
            if not kernel and "__device__" not in head:
                continue
            names = set(re.findall(r"const \w+\* __restrict__ (\w+)", head + body))
            assert names <= TABLES, (os.path.basename(path), head.split("(")[0], names - TABLES)
            loads = re.findall(r"__ldg\(([^;]*);", body)
            assert all(re.search(r"primes|prm\.(q|minus_p)|stage", x) for x in loads), (path, head, loads)
    assert chained >= 12
