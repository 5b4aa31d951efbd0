// Byte-sliced u8 x u8 -> s32 GEMM on the 5th-generation tensor cores (sm_100a).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <string>

#include "kernels.cuh"

namespace negacyclic {

struct TensorGemmPlan {
    CUtensorMap a_map;   // 2-D view of A: (K bytes, rows),          box (128, 128),   128B swizzle
    CUtensorMap b_map;   // 2-D view of B: (K bytes, columns),       box (128, 256),   128B swizzle
    CUtensorMap b_map_half;  // same view, box (128, 128): one CTA's half of a pair tile
    uint32_t m = 0, columns = 0, k_bytes = 0;
    uint32_t m_tiles = 0, n_tiles = 0, k_tiles = 0;
    RowMap rows{};
    uint32_t* tile_counter = nullptr;  // device word the CTA-pair kernel claims tiles from; GEMMs that
                                       // share one may not run at the same time
    uint32_t sm_count = 148;          // persistent grid size
    uint64_t a_tile_bytes = 0;        // bytes of one 128-row A tile (raster group sizing)
    bool pairs = false;               // 2-CTA (cta_group::2) 256x256 tiles
    bool narrow = false;              // fewer columns than one tile: TMA fills the rest of B with zeros
    int source = 0;                   // GemmSource of the A tiles
    bool ready = false;
};

// Where the single-CTA kernel's A tiles come from.
//  kSourceTma:      operand rows of k_bytes in memory, through the plan's tensor map.
//  kSourceRows:     the unpadded operands: row m is coefficient i = s*j + t of operand op, L words
//                   (zeros above) at rows[op] + i*L.
//  kSourceResidues: the residues: byte 4k + d of row m is byte d of residues[k*n + t*N' + j], k < r
//                   (zeros above).
enum GemmSource : int { kSourceTma = 0, kSourceRows = 1, kSourceResidues = 2 };

// Longest K, in bytes, of a GEMM that gathers operand rows: its epilogue forms v_0 + 256 v_1 of two byte
// dots in 32 bits, exact while 257 K 255^2 < 2^32.
constexpr uint32_t kGatherRowBytes = 256;
static_assert(257ull * kGatherRowBytes * 255 * 255 < 1ull << 32, "two byte dots in 32 bits");

struct GatherSource {
    const uint32_t* rows[2];
    uint32_t limbs;
    bool aligned;  // both operands start on 16 bytes and L is a multiple of 4
    const uint32_t* residues;
    uint32_t r, n;
};

// A GEMM whose A operand is gathered by warps (GatherSource) instead of read by TMA: `rows` is the
// split row map of the whole shape, k_bytes a multiple of 128, and of operand rows at most
// kGatherRowBytes. False (with `why`) outside that.
bool prepare_gemm_gather(TensorGemmPlan& plan, GemmSource source, RowMap rows, uint32_t m, const uint8_t* b, uint32_t columns,
                         uint32_t k_bytes, std::string& why);
void launch_gemm_gather(const TensorGemmPlan& plan, const GatherSource& source, const Epilogue& epilogue,
                        cudaStream_t stream, const RowMap& rows, uint32_t m);

// Builds the tensor maps; false (with `why`) when the shape is outside what the
// kernel handles (then the SIMT kernel is used).
bool prepare_gemm_tensor(TensorGemmPlan& plan, const uint8_t* a, uint64_t a_pitch, RowMap rows, uint32_t m,
                         const uint8_t* b, uint32_t columns, uint32_t k_bytes, std::string& why);

constexpr uint32_t kNoWithheldStep = 0xffffffffu;
// K steps (of 128 bytes) from which the CTA-pair kernel is the faster one: it halves the B bytes each
// SM reads, but a tile costs it a claim from the global counter and twice the tile. Conversion and
// CRT stages, us, pairs against single CTAs: 2 steps 59 / 40 and 4 steps 28.5 / 20.5 (N=65536, L=55),
// 10 steps 95.5 / 88 and 20 steps 54.7 / 50.6 (N=16384, L=301), 28 steps 1100 / 1115 and 57 steps
// 547 / 573 (N=32768, L=868), 55 steps 8950 / 9580 (N=65536, L=1747).
constexpr uint32_t kPairMinSteps = 24;
struct TensorGemmOptions {
    bool allow_pairs = true;      // false: the single-CTA kernel
    uint32_t pair_min_steps = kPairMinSteps;  // CTA pairs from this many K steps on
    bool counter_cleared = false; // an earlier kernel of the stream has zeroed plan.tile_counter
    long long limit_cycles = 0;   // bound of every pipeline wait (0: about 2 s of SM clock)
    // diagnostics only: the producer of the first CTA (pair) stops before this pipeline step, so that
    // its consumer's wait runs out
    uint32_t withheld = kNoWithheldStep;
};

// A launch over the plan's rows or part of them (a chunk of coefficients): `rows`/`m` describe the
// chunk within the shape the plan was prepared for (see gemm_tensor_accepts).
void launch_gemm_tensor(const TensorGemmPlan& plan, const Epilogue& epilogue, cudaStream_t stream, const RowMap& rows,
                        uint32_t m, const TensorGemmOptions& options = {});
bool gemm_tensor_accepts(const TensorGemmPlan& plan, const RowMap& rows, uint32_t m);

// Device word that records pipeline-wait timeouts of the tensor GEMM (0 = none).
uint32_t* tensor_gemm_error_flag();

}  // namespace negacyclic
