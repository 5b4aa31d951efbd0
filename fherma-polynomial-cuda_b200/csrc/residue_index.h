// Where a residue is kept: [2][r][N] words, operand by operand and prime by prime. Free of CUDA types,
// so that tests/native/residue_index_check.cpp checks it on the CPU at the widest points.
#pragma once

#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define NEGACYCLIC_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define NEGACYCLIC_HOST_DEVICE inline
#endif

namespace negacyclic {

// Word index of operand op's residue mod prime k at `column` (t*N' + j). 64 bits: the 2 r N words pass
// 4 GB from r = 4097 on at N = 131072 and from r = 8193 on at N = 65536 (6.37 GB at N = 131072, L = 2900).
NEGACYCLIC_HOST_DEVICE size_t residue_index(uint32_t op, uint32_t k, uint32_t column, uint32_t r, uint32_t n) {
    return (size_t(op) * r + k) * n + column;
}

}  // namespace negacyclic
