// CPU check of csrc/residue_index.h at the widest points that build_host_plan accepts (run by
// tests/test_residue_index.py): the residues of consecutive columns, primes and operands are
// consecutive words, the last of them ends the buffer of 2 r N words, and that buffer is over 4 GB.
#include <cstdio>
#include <vector>

#include "../../fherma-polynomial-cuda_b200/csrc/host_plan.h"
#include "../../fherma-polynomial-cuda_b200/csrc/residue_index.h"

using namespace negacyclic;

static int failures = 0;
#define EXPECT(cond)                                                          \
    do {                                                                      \
        if (!(cond)) {                                                        \
            std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);   \
            ++failures;                                                       \
        }                                                                     \
    } while (0)

static void check(uint32_t n, uint32_t limbs, uint32_t split) {
    HostPlan plan;
    std::string error;
    int status = 0;
    const std::vector<uint32_t> q(limbs, 0xffffffffu);
    const bool accepted = build_host_plan(n, limbs, q.data(), split, plan, error, status);
    EXPECT(accepted);
    if (!accepted) return;
    const uint32_t r = uint32_t(plan.primes.size());
    const unsigned __int128 words = static_cast<unsigned __int128>(2) * r * n;
    EXPECT(words * 4 > 0xffffffffu);
    EXPECT(residue_index(1, r - 1, n - 1, r, n) == words - 1);
    for (uint32_t op = 0; op < 2; ++op)
        for (uint32_t k = 0; k < r; ++k) {
            const unsigned __int128 row = (static_cast<unsigned __int128>(op) * r + k) * n;
            EXPECT(residue_index(op, k, 0, r, n) == row && residue_index(op, k, n - 1, r, n) == row + n - 1);
        }
    std::printf("N=%u L=%u r=%u: %.2f GB\n", n, limbs, r, double(words) * 4e-9);
}

int main() {
    check(131072, 2000, 0);
    check(131072, 2900, 0);
    check(65536, 3950, 0);
    std::printf("%d failures\n", failures);
    return failures != 0;
}
