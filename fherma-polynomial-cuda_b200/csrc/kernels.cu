// SIMT stages of the negacyclic product and the parameter-only table builders.
//
// Data layout in HBM (one plan, r primes, ring split s, N' = N/s):
//   operands   [2][N][Lp] u32      a then b, limbs padded to Lp = roundup(L, 32) (128-byte rows),
//                                  split-major: row op*N + t*N' + j holds coefficient s*j + t
//   residues   [2][r][N]  u32      per (operand, prime): s transforms of N' values,
//                                  transform t holds coefficients i = s*j + t at j
//   crt_in     [N][r']    u32      coefficient-major residues v_k (r' = roundup(r, 32))
//   dots       [N][L+5]   u64      word sums of the byte-sliced CRT product
//   twiddles   [r][N']    uint2    {w, floor(w 2^32/p)}: forward psi^brv(m), inverse psi^-brv(m),
//                                  zeta psi^(2 brv(m)+1) (evaluation point at output m)
#include "kernels.cuh"

#include "launch.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <type_traits>

namespace negacyclic {

namespace {

// One padded row: Lp words (16-byte aligned) from `limbs` words, zeros above.
__device__ __forceinline__ void pad_row(const uint32_t* src, uint32_t* __restrict__ dst, uint32_t limbs,
                                        uint32_t padded, uint32_t lane) {
    uint4* out = reinterpret_cast<uint4*>(dst);
    for (uint32_t c = lane; c < padded / 4; c += 32) {
        const uint32_t w = 4 * c;
        uint4 v;
        v.x = w < limbs ? src[w] : 0u;
        v.y = w + 1 < limbs ? src[w + 1] : 0u;
        v.z = w + 2 < limbs ? src[w + 2] : 0u;
        v.w = w + 3 < limbs ? src[w + 3] : 0u;
        out[c] = v;
    }
}

// [N][L] a and b -> [2][N][Lp] split-major: output row op*N + t*N' + j holds coefficient
// s*j + t of operand op. One warp per output row. Also clears the GEMMs' tile counters, so that no
// memset node stands in the product's chain.
__global__ void pad_operands_kernel(const uint32_t* a, const uint32_t* b, uint32_t* __restrict__ out, uint32_t n, uint32_t limbs, uint32_t padded,
                                    uint32_t log_split, uint32_t log_n_sub, uint32_t* tile_counters) {
    chain_enter();
    if (blockIdx.x == 0 && threadIdx.x < kTileCounters) tile_counters[threadIdx.x] = 0;
    const uint32_t lane = threadIdx.x % 32, warps = gridDim.x * (blockDim.x / 32);
    const uint32_t n_sub_mask = (1u << log_n_sub) - 1;
    for (uint32_t w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < 2 * n; w += warps) {
        const uint32_t op = w >= n ? 1 : 0, row = w - op * n;
        const uint32_t i = ((row & n_sub_mask) << log_split) + (row >> log_n_sub);
        pad_row((op ? b : a) + size_t(i) * limbs, out + size_t(w) * padded, limbs, padded, lane);
    }
}

// Rows [first, first + count) of operands [op_first, op_first + op_count) (operand stride N rows)
// from an unpadded [2][N][L] array into the padded split-major layout. Staged rows are either
// already split-major (log_split = 0: row = position) or in coefficient order (row i goes to
// t*N' + j, i = s*j + t). One warp per row.
__global__ void pad_rows_kernel(const uint32_t* staged, uint32_t* __restrict__ out, uint32_t n,
                                uint32_t limbs, uint32_t padded, uint32_t log_split, uint32_t log_n_sub,
                                uint32_t first, uint32_t count, uint32_t op_first, uint32_t op_count) {
    chain_enter();
    const uint32_t lane = threadIdx.x % 32, warps = gridDim.x * (blockDim.x / 32);
    const uint32_t split_mask = (1u << log_split) - 1;
    for (uint32_t w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < op_count * count; w += warps) {
        const uint32_t local_op = w / count, op = op_first + local_op, i = first + (w - local_op * count);
        const uint32_t row = ((i & split_mask) << log_n_sub) + (i >> log_split);
        pad_row(staged + (size_t(op) * n + i) * limbs, out + (size_t(op) * n + row) * padded, limbs, padded, lane);
    }
}

__device__ __forceinline__ uint32_t bit_reverse(uint32_t x, uint32_t bits) {
    return bits ? (__brev(x) >> (32 - bits)) : 0u;
}

__device__ uint32_t twiddle_place(uint32_t m, uint32_t log_n);

__global__ void twiddles_kernel(const DevicePrime* __restrict__ primes, uint32_t r, uint32_t n_sub,
                                uint32_t log_n, uint2* fwd, uint2* inv, uint2* zeta) {
    uint32_t k = blockIdx.y;
    if (k >= r) return;
    const DevicePrime f = primes[k];
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < n_sub; m += gridDim.x * blockDim.x) {
        uint32_t e = bit_reverse(m, log_n);
        uint32_t w_fwd = pow_mod(f.psi, e, f);
        uint32_t w_inv = pow_mod(f.psi, 2ull * n_sub - e, f);
        uint32_t w_zeta = pow_mod(f.psi, 2ull * e + 1, f);
        size_t at = size_t(k) * n_sub + m;
        const size_t placed = size_t(k) * n_sub + twiddle_place(m, log_n);
        fwd[placed] = make_uint2(w_fwd, shoup_quotient(w_fwd, f.p));
        inv[placed] = make_uint2(w_inv, shoup_quotient(w_inv, f.p));
        zeta[at] = make_uint2(w_zeta, shoup_quotient(w_zeta, f.p));
    }
}

// B_conv[4k+d][j] = byte_d(256^j mod p_k); zero for padded primes and j >= 4L.
__global__ void convert_weights_kernel(const DevicePrime* __restrict__ primes, uint32_t r,
                                       uint32_t padded_r, uint32_t limbs, uint32_t k_bytes,
                                       uint8_t* out) {
    uint32_t k = blockIdx.y;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < k_bytes; j += gridDim.x * blockDim.x) {
        uint32_t w = 0;
        if (k < r && j < 4 * limbs) w = pow_mod(256, j, primes[k]);
        for (uint32_t d = 0; d < 4; ++d) out[(size_t(k) * 4 + d) * k_bytes + j] = uint8_t(w >> (8 * d));
    }
}

// B_crt[c][4k+d] = byte_{c-d}(W_k), W_k given as `words` u32 words; zero outside.
__global__ void crt_weights_kernel(const uint32_t* __restrict__ weights, uint32_t r, uint32_t padded_r,
                                   uint32_t words, uint32_t columns, uint8_t* out) {
    uint32_t c = blockIdx.y;
    const uint32_t k_bytes = 4 * padded_r;
    for (uint32_t kd = blockIdx.x * blockDim.x + threadIdx.x; kd < k_bytes; kd += gridDim.x * blockDim.x) {
        uint32_t k = kd / 4, d = kd % 4;
        uint8_t value = 0;
        if (k < r && c < columns && c >= d) {
            uint32_t at = c - d;  // byte position within W_k
            if (at < 4 * words) value = uint8_t(weights[size_t(k) * words + at / 4] >> (8 * (at % 4)));
        }
        out[size_t(c) * k_bytes + kd] = value;
    }
}

// ---------------------------------------------------------------------------
// SIMT byte GEMM: D[m][c] = sum_j A[m][j] * B[c][j] with dp4a, 64x64 tiles,
// 256 threads, each thread a 4-row x 4-column (one column group) micro-tile.
constexpr int kTile = 64, kTileK = 64;

__global__ void __launch_bounds__(256) gemm_simt_kernel(const uint8_t* a, uint64_t a_pitch, RowMap rows,
                                                        uint32_t m_total, const uint8_t* b, uint32_t columns,
                                                        uint32_t k_bytes, Epilogue epi) {
    chain_enter();
    __shared__ uint32_t as[kTile][kTileK / 4 + 1];
    __shared__ uint32_t bs[kTile][kTileK / 4 + 1];
    const uint32_t tid = threadIdx.x, tr = tid / 16, tc = tid % 16;
    const uint32_t m0 = blockIdx.x * kTile, c0 = blockIdx.y * kTile;
    const uint32_t load_row = tid / 4, load_part = tid % 4;
    const uint32_t am = m0 + load_row, bc = c0 + load_row;
    const uint8_t* arow = am < m_total ? a + rows.row(am) * a_pitch : nullptr;
    const uint8_t* brow = bc < columns ? b + size_t(bc) * k_bytes : nullptr;
    uint32_t acc[4][4] = {};  // unsigned byte dot products (u8 x u8)
    for (uint32_t k0 = 0; k0 < k_bytes; k0 += kTileK) {
        uint32_t kk = k0 + load_part * 16;
        uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
        if (arow && kk < k_bytes) va = *reinterpret_cast<const uint4*>(arow + kk);
        if (brow && kk < k_bytes) vb = *reinterpret_cast<const uint4*>(brow + kk);
        as[load_row][load_part * 4 + 0] = va.x;
        as[load_row][load_part * 4 + 1] = va.y;
        as[load_row][load_part * 4 + 2] = va.z;
        as[load_row][load_part * 4 + 3] = va.w;
        bs[load_row][load_part * 4 + 0] = vb.x;
        bs[load_row][load_part * 4 + 1] = vb.y;
        bs[load_row][load_part * 4 + 2] = vb.z;
        bs[load_row][load_part * 4 + 3] = vb.w;
        __syncthreads();
#pragma unroll
        for (int kw = 0; kw < kTileK / 4; ++kw) {
            uint32_t ra[4], rb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) ra[i] = as[tr * 4 + i][kw];
#pragma unroll
            for (int j = 0; j < 4; ++j) rb[j] = bs[tc * 4 + j][kw];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __dp4a(ra[i], rb[j], acc[i][j]);
        }
        __syncthreads();
    }
    const uint32_t group = (c0 / 4) + tc;  // column group index (4 columns)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t m = m0 + tr * 4 + i;
        if (m >= m_total) continue;
        if (epi.mode == kEpilogueRaw) {
            const uint64_t out_row = rows.row(m);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t c = c0 + tc * 4 + j;
                if (c < columns) epi.raw[out_row * epi.raw_ld + c] = int32_t(acc[i][j]);
            }
            continue;
        }
        uint64_t s = uint64_t(uint32_t(acc[i][0])) + (uint64_t(uint32_t(acc[i][1])) << 8) +
                     (uint64_t(uint32_t(acc[i][2])) << 16) + (uint64_t(uint32_t(acc[i][3])) << 24);
        if (epi.mode == kEpilogueConvert) {
            if (group >= epi.r) continue;
            const DevicePrime f = epi.primes[group];
            uint32_t op, column;
            rows.residue(m, op, column);
            epi.residues[residue_index(op, group, column, epi.r, epi.n)] = redc(s, f.p, f.pinv);
        } else {
            if (group < epi.words) epi.dots[rows.row(m) * epi.dots_stride + group] = s;
        }
    }
}

// ---------------------------------------------------------------------------
// NTT: one CTA per length-N' transform, whole transform in shared memory.

__global__ void __launch_bounds__(512) ntt_forward_kernel(uint32_t* residues, const DevicePrime* __restrict__ primes,
                                                          const uint2* __restrict__ fwd, uint32_t r, uint32_t n,
                                                          uint32_t n_sub, uint32_t t_first, uint32_t op_first) {
    chain_enter();
    extern __shared__ uint32_t x[];
    const uint32_t t_index = t_first + blockIdx.x, k = blockIdx.y, op = op_first + blockIdx.z;
    const uint32_t p = primes[k].p;
    uint32_t* data = residues + (size_t(op) * r + k) * n + size_t(t_index) * n_sub;
    const uint2* table = fwd + size_t(k) * n_sub;
    for (uint32_t j = threadIdx.x; j < n_sub; j += blockDim.x) x[j] = data[j];
    __syncthreads();
    for (uint32_t m = 1, t = n_sub; m < n_sub; m *= 2) {
        t /= 2;
        for (uint32_t bfly = threadIdx.x; bfly < n_sub / 2; bfly += blockDim.x) {
            uint32_t i = bfly / t, jj = bfly - i * t, j = 2 * i * t + jj;
            uint2 w = table[m + i];
            uint32_t u = x[j], v = shoup(x[j + t], w.x, w.y, p);
            x[j] = add_mod(u, v, p);
            x[j + t] = sub_mod(u, v, p);
        }
        __syncthreads();
    }
    for (uint32_t j = threadIdx.x; j < n_sub; j += blockDim.x) data[j] = x[j];
}

__global__ void __launch_bounds__(512) ntt_inverse_kernel(uint32_t* residues, const DevicePrime* __restrict__ primes,
                                                          const uint2* __restrict__ inv, uint32_t r, uint32_t n,
                                                          uint32_t n_sub, uint32_t v_first) {
    chain_enter();
    extern __shared__ uint32_t x[];
    const uint32_t v_index = v_first + blockIdx.x, k = blockIdx.y;
    const DevicePrime f = primes[k];
    uint32_t* data = residues + size_t(k) * n + size_t(v_index) * n_sub;
    const uint2* table = inv + size_t(k) * n_sub;
    for (uint32_t j = threadIdx.x; j < n_sub; j += blockDim.x) x[j] = data[j];
    __syncthreads();
    for (uint32_t m = n_sub, t = 1; m > 1; m /= 2, t *= 2) {
        const uint32_t h = m / 2;
        for (uint32_t bfly = threadIdx.x; bfly < n_sub / 2; bfly += blockDim.x) {
            uint32_t i = bfly / t, jj = bfly - i * t, j = 2 * i * t + jj;
            uint2 w = table[h + i];
            uint32_t u = x[j], v = x[j + t];
            x[j] = add_mod(u, v, f.p);
            x[j + t] = shoup(sub_mod(u, v, f.p), w.x, w.y, f.p);
        }
        __syncthreads();
    }
    for (uint32_t j = threadIdx.x; j < n_sub; j += blockDim.x) data[j] = shoup(x[j], f.finish, f.finish_q, f.p);
}

// ---------------------------------------------------------------------------
// Register-blocked NTT for N' >= 256 (from 64 in the kernels that do whole products): 16 values per thread (32 at N' = 8192), up to four (five)
// butterfly stages per pass between shared-memory exchanges.
// A pass of R stages on group g (2^R values spaced t_min apart, t_min = the
// smallest half-size in the pass) covers indices base + k*t_min, k < 2^R, with
// base = (g / t_min) * 2^R * t_min + g % t_min.
//
// What bounds it, at N' = 8192: issue slots, the multiply pipe and the ALU are each about half used,
// and shared-memory and twiddle loads take the rest. 32 values per thread take 5 + 4 + 4 stages in
// three passes, one exchange fewer than 4 + 4 + 4 + 1, in four CTAs of 256 threads per SM instead of
// two of 512, so that one CTA's loads and barriers fall into another's arithmetic; twiddles are loaded in
// pairs, and those of the unit-stride pass from a table laid out for it. 16450 warp instructions per
// transform instead of 18600. Forward 2010 -> 1810 us and inverse 1226 -> 890 us (961 before its scaling
// went into the last stage) at N = 65536, L = 1747 (58176 and 29088 transforms; 2.1 TB/s). Keeping the next transform's input on its way into
// shared memory (persistent CTAs), or 16 values per thread with three CTAs of 512, were slower.

constexpr uint32_t per_thread(uint32_t log) { return log == 13 ? 32 : 16; }  // values per thread

// Shared-memory layout of a length-2^kLog transform: word i is stored at i ^ M(i >> 5), where M
// XORs column b into the bank bits when bit 5 + b of i is set. A pass's warp accesses vary five bits
// of i; they are free of bank conflicts when the images of those bits are linearly independent. The
// columns up to 2^12 were found by an exhaustive check of every warp access of every pass (forward
// and inverse). At 2^13 the passes vary bits 0-4, bits 0-3 and 8, and bits 4-8, which the columns
// below keep independent. M is linear, and a pass's per-value
// offsets k t_min share no bits with its group base, so the swizzle of base + k t_min is the
// swizzle of base (once per group) XOR a compile-time constant.
template <uint32_t kLog>
__host__ __device__ constexpr uint32_t swizzle_column(int b) {
    constexpr uint32_t c6[] = {1}, c7[] = {1, 2};  // short transforms share a warp; any column does
    constexpr uint32_t c8[] = {30, 1, 4};
    constexpr uint32_t c9[] = {7, 9, 27, 13};
    constexpr uint32_t c10[] = {27, 13, 8, 26, 8};
    constexpr uint32_t c11[] = {11, 1, 14, 20, 24, 27};
    constexpr uint32_t c12[] = {17, 26, 2, 21, 24, 25, 27};
    constexpr uint32_t c13[] = {1, 2, 4, 24, 0, 0, 0, 0};
    return kLog == 6 ? c6[b] : kLog == 7 ? c7[b] : kLog == 8 ? c8[b] : kLog == 9 ? c9[b] : kLog == 10 ? c10[b] : kLog == 11 ? c11[b] : kLog == 12 ? c12[b] : c13[b];
}

template <uint32_t kLog>
__host__ __device__ constexpr uint32_t swizzle(uint32_t i) {
    uint32_t m = 0;
    for (int b = 0; b < int(kLog) - 5; ++b)
        if ((i >> (5 + b)) & 1u) m ^= swizzle_column<kLog>(b);
    return i ^ m;
}

// Twiddle b of the `blocks` that a group uses in one stage; `stage` points at the stage's table
// (entries m .. 2m of the prime's row), which serves groups 0 .. m / blocks. Twiddles come two at a
// time, the odd one with the even one before it (rows and stages start on 16-byte boundaries).
// In table order a group's twiddles are consecutive. In the unit-stride pass of length 8192, where
// every lane has a group of its own, the table is laid out pair by pair instead (twiddle_place), so
// that a warp's load is 512 consecutive bytes and not 32 pieces 64 bytes apart.
constexpr uint32_t kPairedGroups = 512;  // groups of 16 in the unit-stride pass of length 8192

template <int blocks, bool kPaired>
__device__ __forceinline__ uint2 stage_twiddle(const uint2* __restrict__ stage, uint32_t group, int b) {
    if constexpr (blocks == 1) return __ldg(stage + group);
    const uint32_t at = kPaired ? uint32_t(b / 2) * kPairedGroups + group : (group * blocks + b) / 2;
    const uint4 pair = __ldg(reinterpret_cast<const uint4*>(stage) + at);
    return b % 2 ? make_uint2(pair.z, pair.w) : make_uint2(pair.x, pair.y);
}

// Where twiddle m of a length-2^log_n table is stored in the prime's row.
__device__ uint32_t twiddle_place(uint32_t m, uint32_t log_n) {
    if (log_n != 13 || m < 2 * kPairedGroups) return m;
    const uint32_t stage = 1u << (31 - __clz(m)), blocks = stage / kPairedGroups, e = m - stage;
    const uint32_t group = e / blocks, b = e % blocks;
    return stage + ((b / 2) * kPairedGroups + group) * 2 + b % 2;
}

// Cooley-Tukey stages with half-sizes t_min*2^(R-1) .. t_min (forward, merged psi twiddles) on
// one group of 2^R values. With j = base + k*t_min and base = group_hi * 2^(log t_min + R) + off
// (off < t_min), butterfly (k, k + half) of stage r has twiddle m + (j >> (log t + 1))
// = m + group_hi * 2^r + (k >> (R - r)): the 2^(R-1-r) butterflies of block b = k >> (R - r)
// share one twiddle, so a pass loads 2^R - 1 twiddles for its R * 2^(R-1) butterflies.
// Values between stages are kept in [0, 2p) (2p < 2^32): each butterfly reduces its two inputs
// once, so that u + v and u - v + p stay below 2p, and multiplies by the twiddle without
// Shoup's final correction. Canonical inputs are a special case; the last pass reduces.
template <int R, bool kPaired, int r = 0>
__device__ __forceinline__ void ct_stages(uint32_t (&x)[1 << R], uint32_t group_hi, uint32_t log_t_min,
                                          uint32_t log_n, const uint2* __restrict__ table, uint32_t p) {
    constexpr int half = 1 << (R - 1 - r), blocks = 1 << r;
    const uint32_t log_t = log_t_min + (R - 1 - r);  // this stage's half-size t = 2^log_t
    const uint32_t m = 1u << (log_n - 1 - log_t);     // number of groups: n / (2t)
    const uint2* stage = table + m;
#pragma unroll
    for (int b = 0; b < blocks; ++b) {
        const uint2 w = stage_twiddle<blocks, kPaired>(stage, group_hi, b);
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const int k = b * 2 * half + j;
            const uint32_t u = reduce_once(x[k], p);
            const uint32_t v = reduce_once(shoup_lazy(x[k + half], w.x, w.y, p), p);
            x[k] = u + v;
            x[k + half] = u - v + p;
        }
    }
    if constexpr (r + 1 < R) ct_stages<R, kPaired, r + 1>(x, group_hi, log_t_min, log_n, table, p);
}

// Gentleman-Sande stages with half-sizes t_min .. t_min*2^(R-1) (inverse). Stage r's butterflies
// (k, k + 2^r) in block b = k >> (r + 1) share twiddle h + group_hi * 2^(R-1-r) + b.
// Values between stages are in [0, 2p), as in ct_stages.
// kScale: the pass ends the transform, and its last stage scales (Finish) to canonical values.
template <int R, bool kPaired, bool kScale = false, int r = 0>
__device__ __forceinline__ void gs_stages(uint32_t (&x)[1 << R], uint32_t group_hi, uint32_t log_t_min,
                                          uint32_t log_n, const uint2* __restrict__ table, uint32_t p,
                                          const Finish& finish = Finish{}) {
    constexpr int half = 1 << r;
    if constexpr (kScale && r == R - 1) {
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const uint32_t u = reduce_once(x[k], p), v = reduce_once(x[k + half], p);
            x[k] = shoup(u + v, finish.f, finish.f_q, p);
            x[k + half] = shoup(u - v + p, finish.w, finish.w_q, p);
        }
        return;
    }
    const uint32_t log_t = log_t_min + r;
    const uint32_t h = 1u << (log_n - 1 - log_t);
    constexpr int blocks = 1 << (R - 1 - r);
    const uint2* stage = table + h;
#pragma unroll
    for (int b = 0; b < blocks; ++b) {
        const uint2 w = stage_twiddle<blocks, kPaired>(stage, group_hi, b);
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const int k = b * 2 * half + j;
            const uint32_t u = reduce_once(x[k], p), v = reduce_once(x[k + half], p);
            x[k] = u + v;
            x[k + half] = shoup_lazy(u - v + p, w.x, w.y, p);
        }
    }
    if constexpr (r + 1 < R) gs_stages<R, kPaired, kScale, r + 1>(x, group_hi, log_t_min, log_n, table, p, finish);
}

// One pass of R stages over all of this thread's groups (transform length 2^kLog). src/dst are shared (swizzled index) or global (plain index);
// kScale: the last inverse pass, whose last stage scales.
template <int R, bool kForward, bool kFromGlobal, bool kToGlobal, bool kScale, uint32_t kLogTMin, uint32_t kLog>
__device__ __forceinline__ void ntt_pass(uint32_t tid, const uint32_t* src, uint32_t* dst,
                                         const uint2* __restrict__ table, uint32_t p,
                                         const Finish& finish = Finish{}) {
    constexpr int G = per_thread(kLog) >> R;  // groups per thread
    constexpr uint32_t kThreads = (1u << kLog) / per_thread(kLog);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t group = tid + g * kThreads;
        const uint32_t off = group & ((1u << kLogTMin) - 1);
        const uint32_t base = ((group >> kLogTMin) << (kLogTMin + R)) + off;
        const uint32_t placed = swizzle<kLog>(base);  // shared-memory place of the group's first word
        // with t_min = 1 a group is 2^R consecutive words (base a multiple of 2^R): global
        // accesses go four words at a time (two in a one-stage pass), so a warp instruction
        // covers 16-byte (8-byte) pieces
        constexpr bool kVector = kLogTMin == 0 && R >= 2;
        constexpr bool kPair = kLogTMin == 0 && R == 1;
        uint32_t x[1 << R];
        if constexpr (kFromGlobal && kPair) {
            const uint2 w = *reinterpret_cast<const uint2*>(src + base);
            x[0] = w.x;
            x[1] = w.y;
        } else if constexpr (kFromGlobal && kVector) {
#pragma unroll
            for (int q = 0; q < (1 << R) / 4; ++q) {
                const uint4 w = reinterpret_cast<const uint4*>(src + base)[q];
                x[4 * q] = w.x;
                x[4 * q + 1] = w.y;
                x[4 * q + 2] = w.z;
                x[4 * q + 3] = w.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < (1 << R); ++k) {
                const uint32_t i = base + (uint32_t(k) << kLogTMin);
                x[k] = kFromGlobal ? src[i] : src[placed ^ swizzle<kLog>(uint32_t(k) << kLogTMin)];
            }
        }
        constexpr bool kPaired = kLog == 13 && kLogTMin == 0;
        if (kForward)
            ct_stages<R, kPaired>(x, group >> kLogTMin, kLogTMin, kLog, table, p);
        else
            gs_stages<R, kPaired, kScale>(x, group >> kLogTMin, kLogTMin, kLog, table, p, finish);
        if constexpr (kToGlobal && !kScale) {
#pragma unroll
            for (int k = 0; k < (1 << R); ++k) x[k] = reduce_once(x[k], p);  // [0, 2p) -> canonical
        }
        if constexpr (kToGlobal && kPair) {
            *reinterpret_cast<uint2*>(dst + base) = make_uint2(x[0], x[1]);
        } else if constexpr (kToGlobal && kVector && R == 4 && kThreads >= 32) {
            // neighbouring lanes trade quarters of their 16 words, so that the two of them fill
            // whole 32-byte sectors with each store
            const bool odd = tid & 1;
            uint32_t* to = dst + base - (odd ? 16 - 4 : 0);
#pragma unroll
            for (int q = 0; q < 16; q += 8) {
                uint32_t first[4], second[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? x[q + i] : x[q + 4 + i], 1);
                    first[i] = odd ? got : x[q + i];
                    second[i] = odd ? x[q + 4 + i] : got;
                }
                *reinterpret_cast<uint4*>(to + q) = make_uint4(first[0], first[1], first[2], first[3]);
                *reinterpret_cast<uint4*>(to + q + 16) = make_uint4(second[0], second[1], second[2], second[3]);
            }
        } else if constexpr (kToGlobal && kVector) {
#pragma unroll
            for (int q = 0; q < (1 << R) / 4; ++q)
                reinterpret_cast<uint4*>(dst + base)[q] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < (1 << R); ++k) {
                const uint32_t i = base + (uint32_t(k) << kLogTMin);
                if (kToGlobal)
                    dst[i] = x[k];
                else
                    dst[placed ^ swizzle<kLog>(uint32_t(k) << kLogTMin)] = x[k];
            }
        }
    }
}

// Passes kDone.. of a length-2^kLog transform: four stages per pass, and a shorter pass for the
// remainder at the unit-stride end, where it touches global memory 2 consecutive words per
// thread instead of 16: last in the forward transform (half-sizes large -> small), first in the
// inverse (small -> large, which also scales its output). Length 8192 takes five stages at the
// large-stride end instead (its global accesses there are whole 128-byte lines), and four at the
// unit-stride end, where lanes trade words so that their stores fill sectors.
constexpr int ntt_pass_stages(bool forward, uint32_t log, uint32_t done) {
    if (log == 13) return (forward ? done == 0 : done == 8) ? 5 : 4;
    if (!forward && done == 0 && log % 4 != 0) return int(log % 4);
    return log - done < 4 ? int(log - done) : 4;
}

// `tid`: the thread's number among the transform's.
template <bool kForward, uint32_t kLog, uint32_t kDone>
__device__ __forceinline__ void ntt_passes(uint32_t tid, uint32_t* data, uint32_t* xs, const uint2* __restrict__ table,
                                           uint32_t p, const Finish& finish = Finish{}) {
    constexpr int R = ntt_pass_stages(kForward, kLog, kDone);
    constexpr uint32_t kLogTMin = kForward ? kLog - kDone - R : kDone;
    constexpr bool kFirst = kDone == 0, kLast = kDone + R == kLog;
    ntt_pass<R, kForward, kFirst, kLast, kLast && !kForward, kLogTMin, kLog>(tid, kFirst ? data : xs, kLast ? data : xs,
                                                                              table, p, finish);
    if constexpr (!kLast) {
        __syncthreads();
        ntt_passes<kForward, kLog, kDone + R>(tid, data, xs, table, p, finish);
    }
}

// grid (op_count t_count, r): x = (op - op_first)*t_count + (t - t_first), y = prime, so a prime's
// transforms share its twiddles in L2
template <uint32_t kLog>
__global__ void __launch_bounds__((1u << kLog) / per_thread(kLog), 4) ntt_forward_blocked_kernel(
    uint32_t* residues, const DevicePrime* __restrict__ primes, const uint2* __restrict__ fwd, uint32_t r, uint32_t n,
    uint32_t t_first, uint32_t t_count, uint32_t op_first) {
    chain_enter();
    extern __shared__ uint32_t xs[];
    constexpr uint32_t kN = 1u << kLog;
    const uint32_t local_op = blockIdx.x / t_count, op = op_first + local_op;
    const uint32_t t_index = t_first + blockIdx.x - local_op * t_count, k = blockIdx.y;
    uint32_t* data = residues + (size_t(op) * r + k) * n + size_t(t_index) * kN;
    ntt_passes<true, kLog, 0>(threadIdx.x, data, xs, fwd + size_t(k) * kN, primes[k].p);
}

template <uint32_t kLog>
__global__ void __launch_bounds__((1u << kLog) / per_thread(kLog), 4) ntt_inverse_blocked_kernel(
    uint32_t* residues, const DevicePrime* __restrict__ primes, const uint2* __restrict__ inv, uint32_t r, uint32_t n,
    uint32_t v_first, uint32_t v_count, uint32_t /*op_first: the inverse works on operand row 0 only*/) {
    chain_enter();
    extern __shared__ uint32_t xs[];
    constexpr uint32_t kN = 1u << kLog;
    const uint32_t v_index = v_first + blockIdx.x, k = blockIdx.y;
    const DevicePrime f = primes[k];
    uint32_t* data = residues + size_t(k) * n + size_t(v_index) * kN;
    ntt_passes<false, kLog, 0>(threadIdx.x, data, xs, inv + size_t(k) * kN, f.p, finish_of(f));
}

// Unsplit rings (s = 1): both operands' forward transforms, their product and its inverse in one CTA
// per prime; only the inputs are read and only the result is written (over operand a's residues).
// One half of the block transforms a, the other b. The forward's last pass and the inverse's first
// work on the same groups of consecutive values, so a's are still in registers when b's come
// through shared memory, are multiplied, and enter the inverse, which the first half finishes.
// Two launches and two round trips through L2 less. Product, us, three kernels / one: 17.7 / 12.4 at
// N = 256, L = 2; 17.5 / 14.5 at N = 2048, L = 13; 38.5 / 34.8 at N = 4096, L = 64; 85.6 / 74.0 at
// N = 8192, L = 128; 791 / 721 at N = 8192, L = 868 (33.0 / 33.6 at N = 2048, L = 94: 197 CTAs).
template <uint32_t kLog, uint32_t kDone, bool kGlobalInput>
__device__ __forceinline__ void forward_to_middle(bool active, uint32_t tid, uint32_t* data, uint32_t* xs,
                                                  const uint2* __restrict__ table, uint32_t p) {
    constexpr int R = ntt_pass_stages(true, kLog, kDone);
    constexpr bool kGlobal = kGlobalInput && kDone == 0;
    if constexpr (kDone + R < kLog) {
        if (active)
            ntt_pass<R, true, kGlobal, false, false, kLog - kDone - R, kLog>(tid, kGlobal ? data : xs, xs, table, p);
        __syncthreads();
        forward_to_middle<kLog, kDone + R, kGlobalInput>(active, tid, data, xs, table, p);
    }
}

template <uint32_t kLog, uint32_t kDone>
__device__ __forceinline__ void inverse_from_middle(bool active, uint32_t tid, uint32_t* data, uint32_t* xs,
                                                    const uint2* __restrict__ table, uint32_t p,
                                                    const Finish& finish) {
    if constexpr (kDone < kLog) {
        constexpr int R = ntt_pass_stages(false, kLog, kDone);
        constexpr bool kLast = kDone + R == kLog;
        __syncthreads();
        if (active) ntt_pass<R, false, false, kLast, kLast, kDone, kLog>(tid, xs, kLast ? data : xs, table, p, finish);
        inverse_from_middle<kLog, kDone + R>(active, tid, data, xs, table, p, finish);
    }
}

template <uint32_t kLog>
__global__ void __launch_bounds__(2 * (1u << kLog) / per_thread(kLog), (kLog >= 12 ? 2 : 4))
    ntt_product_kernel(uint32_t* residues, const DevicePrime* __restrict__ primes, const uint2* __restrict__ fwd,
                       const uint2* __restrict__ inv, uint32_t r) {
    extern __shared__ uint32_t xs[];
    constexpr uint32_t kN = 1u << kLog, kThreads = kN / per_thread(kLog);
    // the prime's twiddles into L1 while the conversion finishes: one load per 128-byte line
    for (uint32_t i = threadIdx.x * 16; i < 2 * kN; i += 2 * kThreads * 16) {
        const uint2* line = (i < kN ? fwd : inv) + size_t(blockIdx.x) * kN + i % kN;
        uint32_t unused;
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(unused) : "l"(line));
    }
    chain_enter();
    constexpr int R = kLog % 4 && kLog != 13 ? int(kLog % 4) : 4;  // of the forward's last and the inverse's first pass
    constexpr int G = per_thread(kLog) >> R;
    const uint32_t k = blockIdx.x, op = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
    const DevicePrime f = primes[k];
    uint32_t* data = residues + (size_t(op) * r + k) * kN;
    uint32_t* own = xs + op * kN;
    const uint2 *forward = fwd + size_t(k) * kN, *inverse = inv + size_t(k) * kN;
    forward_to_middle<kLog, 0, true>(true, tid, data, own, forward, f.p);
    constexpr bool kPaired = kLog == 13;
    uint32_t x[G][1 << R];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t group = tid + g * kThreads, placed = swizzle<kLog>(group << R);
#pragma unroll
        for (int i = 0; i < (1 << R); ++i) x[g][i] = own[placed ^ swizzle<kLog>(uint32_t(i))];
        ct_stages<R, kPaired>(x[g], group, 0, kLog, forward, f.p);
#pragma unroll
        for (int i = 0; i < (1 << R); ++i) {
            x[g][i] = reduce_once(x[g][i], f.p);
            if (op == 1) own[placed ^ swizzle<kLog>(uint32_t(i))] = x[g][i];
        }
    }
    __syncthreads();
    if (op == 0) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t group = tid + g * kThreads, placed = swizzle<kLog>(group << R);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i)
                x[g][i] = mont(x[g][i], xs[kN + (placed ^ swizzle<kLog>(uint32_t(i)))], f.p, f.pinv);
            gs_stages<R, kPaired>(x[g], group, 0, kLog, inverse, f.p);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i) xs[placed ^ swizzle<kLog>(uint32_t(i))] = x[g][i];
        }
    }
    inverse_from_middle<kLog, R>(op == 0, tid, data, xs, inverse, f.p, finish_of(f));
}

// ntt_product_kernel's middle, from the forward transforms' last pass through the products to the
// inverse's first, for a block of several primes' transforms (as one function for both, the kernel
// above spills and takes 4 % longer). `a` and b are
// the operands' transforms in shared memory, b's b_offset words after a's, of which this thread works
// on number `op`.
template <uint32_t kLog>
__device__ __forceinline__ void middle_passes(bool active, uint32_t tid, uint32_t op, uint32_t* a, uint32_t b_offset,
                                              const uint2* __restrict__ forward, const uint2* __restrict__ inverse,
                                              const DevicePrime& f) {
    uint32_t* own = a + op * b_offset;
    constexpr uint32_t kThreads = (1u << kLog) / per_thread(kLog);
    constexpr int R = ntt_pass_stages(false, kLog, 0);  // of the forward's last and the inverse's first pass
    constexpr int G = per_thread(kLog) >> R;
    constexpr bool kPaired = kLog == 13;
    uint32_t x[G][1 << R];
    if (active) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t group = tid + g * kThreads, placed = swizzle<kLog>(group << R);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i) x[g][i] = own[placed ^ swizzle<kLog>(uint32_t(i))];
            ct_stages<R, kPaired>(x[g], group, 0, kLog, forward, f.p);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i) {
                x[g][i] = reduce_once(x[g][i], f.p);
                if (op == 1) own[placed ^ swizzle<kLog>(uint32_t(i))] = x[g][i];
            }
        }
    }
    __syncthreads();
    if (active && op == 0) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t group = tid + g * kThreads, placed = swizzle<kLog>(group << R);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i)
                x[g][i] = mont(x[g][i], a[b_offset + (placed ^ swizzle<kLog>(uint32_t(i)))], f.p, f.pinv);
            gs_stages<R, kPaired>(x[g], group, 0, kLog, inverse, f.p);
#pragma unroll
            for (int i = 0; i < (1 << R); ++i) a[placed ^ swizzle<kLog>(uint32_t(i))] = x[g][i];
        }
    }
}

// A whole product of a small unsplit ring in one CTA: conversion, transforms, CRT and reduction. Such a
// product is bound by its launches (three cost the host 9 to 13 us, more than the device needs), so all
// of it is one. The conversion and the CRT are plain sums here: residue = sum_j REDC(limb_j c_j) with
// c_j = 2^(32j) mod p, and the words of sum_k v_k W_k by a 96-bit accumulator per coefficient.
// N = 256, L = 2: 12.0 -> 8.9 us; N = 64, L = 2: 19.7 -> 7.4 us. At least 512 threads, for the conversion
// (256: 9.6 us).
constexpr uint32_t kSmallPrimes = 64;
template <uint32_t kLog>
__global__ void __launch_bounds__(512) small_product_kernel(SmallProduct prm) {
    extern __shared__ uint32_t xs[];
    constexpr uint32_t kN = 1u << kLog, kThreads = kN / per_thread(kLog);
    const uint32_t r = prm.r, limbs = prm.reduce.limbs, words = limbs + 5;
    uint32_t* const v = xs + r * kN;             // operand b's transforms, later the residues v_k
    uint32_t* const rows = v + r * kN;           // [2][N][limbs] operands
    uint32_t* const digits = rows;               // [words][N] of the CRT sum, later
    uint32_t* const c = rows + max(2 * limbs, words) * kN;  // [r][limbs]
    uint32_t* const crt = c + r * limbs;                    // [r][words]
    uint32_t* const tables = crt + r * words;               // q, then -P mod q: limbs + 2 words each
    __shared__ DevicePrime primes[kSmallPrimes];
    // constants first: the kernel before may still be running
    for (uint32_t i = threadIdx.x; i < r * limbs; i += blockDim.x) {
        const uint8_t* w = prm.convert_weights + size_t(4 * (i / limbs)) * prm.k_bytes + 4 * (i % limbs);
        c[i] = w[0] | uint32_t(w[prm.k_bytes]) << 8 | uint32_t(w[2 * prm.k_bytes]) << 16 | uint32_t(w[3 * prm.k_bytes]) << 24;
    }
    for (uint32_t i = threadIdx.x; i < r * words; i += blockDim.x) crt[i] = prm.crt_words[i];
    for (uint32_t i = threadIdx.x; i < limbs + 2; i += blockDim.x) {
        tables[i] = prm.reduce.q[i];
        tables[limbs + 2 + i] = prm.reduce.minus_p[i];
    }
    if (threadIdx.x < r) primes[threadIdx.x] = prm.primes[threadIdx.x];
    for (uint32_t i = threadIdx.x * 16; i < 2 * r * kN; i += blockDim.x * 16) {  // twiddles into L1
        const uint2* line = i < r * kN ? prm.fwd + i : prm.inv + (i - r * kN);
        uint32_t unused;
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(unused) : "l"(line));
    }
    chain_enter();
    for (uint32_t i = threadIdx.x; i < kN * limbs; i += blockDim.x) {
        rows[i] = prm.a[i];
        rows[kN * limbs + i] = prm.b[i];
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < 2 * r * kN; i += blockDim.x) {
        const uint32_t row = i / kN, op = row >= r ? 1 : 0, k = row - op * r;
        const uint32_t p = primes[k].p, pinv = primes[k].pinv;
        const uint32_t* x = rows + (op * kN + i % kN) * limbs;
        uint32_t sum = 0;
        for (uint32_t j = 0; j < limbs; ++j) sum = add_mod(sum, redc(uint64_t(x[j]) * c[k * limbs + j], p, pinv), p);
        xs[row * kN + swizzle<kLog>(i % kN)] = sum;
    }
    __syncthreads();
    {
        const uint32_t team = threadIdx.x / (2 * kThreads), op = threadIdx.x / kThreads % 2, tid = threadIdx.x % kThreads;
        const bool active = team < r;
        const uint32_t k = active ? team : 0;
        const DevicePrime f = primes[k];
        const uint2 *forward = prm.fwd + k * kN, *inverse = prm.inv + k * kN;
        uint32_t *a = xs + k * kN, *b = v + k * kN;
        forward_to_middle<kLog, 0, false>(active, tid, nullptr, op ? b : a, forward, f.p);
        middle_passes<kLog>(active, tid, op, a, r * kN, forward, inverse, f);
        // the last pass writes v_k in plain order over b's transform
        inverse_from_middle<kLog, ntt_pass_stages(false, kLog, 0)>(active && op == 0, tid, b, a, inverse, f.p,
                                                                    finish_of(f));
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < r * kN; i += blockDim.x) prm.residues[i] = v[i];
    ReduceParams red = prm.reduce;
    red.q = tables;
    red.minus_p = tables + limbs + 2;
    for (uint32_t i = threadIdx.x; i < kN; i += blockDim.x) {
        uint64_t low = 0;  // the running sum from word w up: 96 bits
        uint32_t high = 0;
        for (uint32_t w = 0; w < words; ++w) {
#pragma unroll 4
            for (uint32_t k = 0; k < r; ++k) {
                const uint64_t product = uint64_t(v[k * kN + i]) * crt[k * words + w];
                low += product;
                high += low < product ? 1 : 0;
            }
            digits[w * kN + i] = uint32_t(low);
            low = (low >> 32) | (uint64_t(high) << 32);
            high = 0;
        }
        const uint64_t x[3] = {digits[(limbs + 2) * kN + i], digits[(limbs + 3) * kN + i], digits[(limbs + 4) * kN + i]};
        uint64_t window[kWindow];
#pragma unroll
        for (int j = 0; j < kWindow; ++j) {
            uint32_t w;
            window[j] = window_word(red, j, w) ? digits[w * kN + i] : 0;
        }
        const RowQuotient f = row_quotient(x, window, red);
        RowState st;
        uint32_t* out = red.out + i * limbs;
        for (uint32_t w = 0; w < limbs + 2; ++w) {
            const uint32_t o = st.word(f, digits[w * kN + i], red.minus_p[w], red.q[w]);
            st.note(o, w, red);
            if (w < limbs) out[w] = o;
        }
        st.finish(out, red);
    }
}

// C_v = sum_{t+u=v} A_t B_u + zeta * sum_{t+u=v+s} A_t B_u at every evaluation point,
// written over A_v. Products are Montgomery (x y 2^-32). Each thread takes V consecutive
// evaluation points (V = 2: 8-byte accesses, n_sub even).
template <int S, int V>
__global__ void pointwise_kernel(uint32_t* residues, const DevicePrime* __restrict__ primes,
                                 const uint2* __restrict__ zeta, uint32_t r, uint32_t n, uint32_t n_sub) {
    chain_enter();
    using Word = std::conditional_t<V == 2, uint2, uint32_t>;
    const uint32_t k = blockIdx.y;
    const uint32_t m = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (m >= n_sub) return;
    const DevicePrime f = primes[k];
    Word* a = reinterpret_cast<Word*>(residues + size_t(k) * n + m);
    const Word* b = reinterpret_cast<const Word*>(residues + (size_t(r) + k) * n + m);
    const size_t step = n_sub / V;  // one transform, in Words
    uint32_t av[V][S], bv[V][S];
#pragma unroll
    for (int t = 0; t < S; ++t) {
        const Word x = a[t * step], y = b[t * step];
        if constexpr (V == 2) {
            av[0][t] = x.x, av[1][t] = x.y, bv[0][t] = y.x, bv[1][t] = y.y;
        } else {
            av[0][t] = x, bv[0][t] = y;
        }
    }
    uint2 z[V];
    if constexpr (V == 2) {
        const uint4 zz = *reinterpret_cast<const uint4*>(zeta + size_t(k) * n_sub + m);
        z[0] = make_uint2(zz.x, zz.y), z[1] = make_uint2(zz.z, zz.w);
    } else {
        z[0] = zeta[size_t(k) * n_sub + m];
    }
    // two products per Montgomery reduction: a b + a' b' < 2 p^2 < p 2^32
#pragma unroll
    for (int v = 0; v < S; ++v) {
        uint32_t out[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
            uint32_t low = 0, wrap = 0;
#pragma unroll
            for (int t = 0; t <= v; t += 2) {
                uint64_t pair = uint64_t(av[e][t]) * bv[e][v - t];
                if (t + 1 <= v) pair += uint64_t(av[e][t + 1]) * bv[e][v - t - 1];
                low = add_mod(low, redc(pair, f.p, f.pinv), f.p);
            }
#pragma unroll
            for (int t = v + 1; t < S; t += 2) {
                uint64_t pair = uint64_t(av[e][t]) * bv[e][v + S - t];
                if (t + 1 < S) pair += uint64_t(av[e][t + 1]) * bv[e][v + S - t - 1];
                wrap = add_mod(wrap, redc(pair, f.p, f.pinv), f.p);
            }
            out[e] = add_mod(low, shoup(wrap, z[e].x, z[e].y, f.p), f.p);
        }
        if constexpr (V == 2)
            a[v * step] = make_uint2(out[0], out[1]);
        else
            a[v * step] = out[0];
    }
}

// residues[0][k][v*N' + j] -> crt_in[s*j + v][k] (coefficient-major) for every transform v and
// j in [j_first, j_first + j_count), i.e. coefficients [s j_first, s (j_first + j_count)); zero for
// k in [r, r'). Block x covers up to 64 consecutive j of one transform and block y 64 primes, so
// every global access is a 256-byte run (two warp instructions of 128 bytes); the tile's rows are
// padded to 65 words, which keeps both the row-wise writes and the column-wise reads free of bank
// conflicts. 256 threads: 16 loads in flight per thread.
constexpr uint32_t kTransposeTile = 64;
__global__ void __launch_bounds__(256) transpose_kernel(const uint32_t* residues,
                                                        uint32_t* __restrict__ crt_in, uint32_t r, uint32_t padded_r,
                                                        uint32_t n, uint32_t log_split, uint32_t log_n_sub,
                                                        uint32_t j_first, uint32_t j_count) {
    chain_enter();
    __shared__ uint32_t tile[kTransposeTile][kTransposeTile + 1];
    const uint32_t blocks_per_v = (j_count + kTransposeTile - 1) / kTransposeTile, v = blockIdx.x / blocks_per_v;
    const uint32_t j0 = j_first + (blockIdx.x - v * blocks_per_v) * kTransposeTile, k0 = blockIdx.y * kTransposeTile;
    const uint32_t j_end = j_first + j_count, rho0 = (v << log_n_sub) + j0;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;  // 8 warps
#pragma unroll
    for (uint32_t row = warp; row < kTransposeTile; row += 8) {  // row = prime offset
        const uint32_t k = k0 + row;
#pragma unroll
        for (uint32_t half = 0; half < kTransposeTile; half += 32) {
            const uint32_t j = j0 + half + lane;
            tile[row][half + lane] = (k < r && j < j_end) ? residues[size_t(k) * n + rho0 + half + lane] : 0u;
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t row = warp; row < kTransposeTile; row += 8) {  // row = position offset
        const uint32_t j = j0 + row;
        if (j >= j_end) continue;
        uint32_t* out = crt_in + ((size_t(j) << log_split) + v) * padded_r;
#pragma unroll
        for (uint32_t half = 0; half < kTransposeTile; half += 32) {
            const uint32_t k = k0 + half + lane;
            if (k < padded_r) out[k] = tile[half + lane][row];
        }
    }
}

// ---------------------------------------------------------------------------
// CRT quotient, carries and reduction mod q (csrc/reduce.cuh): one thread per coefficient.
//
// What bounds it: reading 8 (L+5) and writing 4 L bytes per coefficient. A thread's carry chain is
// three dependent instructions per word, and 32 rows advance per warp instruction; a warp per
// coefficient with a warp-wide carry resolution (the earlier form) issued 554 instructions per
// coefficient at L = 55, 70 % of the issue slots, and took 50 us at N = 65536, L = 55 and 0.62 ms
// at L = 1747.
// Rows are read in chunks of 16 or 64 words through shared memory (16-byte cp.async, whole
// 128-byte lines), two chunks ahead of the arithmetic. A pitch of 16 bytes over a multiple of 128
// keeps the threads' 16-byte reads of their own rows free of bank conflicts, and the results go
// back through the same slot, so that global stores are runs of 64 or 128 bytes. Measured against
// the earlier form (stage between events): 624 -> 362 us at N = 65536, L = 1747 (1.38 GB, 3.8 TB/s),
// 142 -> 90 us at N = 32768, L = 868, 49 -> 20.5 us at N = 65536, L = 55.
//
// Few rows: a thread's chain of L + 2 words is then all there is to wait for, so a row is cut into
// kSegments segments, one lane each. A segment starts with no carry; afterwards each passes its carry
// up, where it is added to the stored words and almost always ends in the first one. N = 256, L =
// 1747: product 187 -> 131 us.

// A row's step: kChunk words of every lane's segment, with the same words of q and R behind them.
template <uint32_t kChunk, uint32_t kSegments>
struct ReduceSlot {
    static constexpr uint32_t kPitch = kChunk * 8 + 16;       // bytes per lane
    static constexpr uint32_t kTablePitch = kChunk * 8 + (kSegments > 1 ? 16 : 0);  // bytes per segment: q, then R
    static constexpr uint32_t kBytes = 32 * kPitch + kSegments * kTablePitch;
};
constexpr uint32_t kReduceSlots = 3;

template <uint32_t kChunk, uint32_t kSegments>
__global__ void reduce_kernel(ReduceParams prm) {
    chain_enter();
    using Slot = ReduceSlot<kChunk, kSegments>;
    constexpr uint32_t kPitch = Slot::kPitch, kRows = 32 / kSegments;
    extern __shared__ __align__(16) uint8_t reduce_smem[];
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint8_t* slots = reduce_smem + warp * (kReduceSlots * Slot::kBytes);
    const uint32_t slots_addr = uint32_t(__cvta_generic_to_shared(slots));
    const uint32_t row0 = (blockIdx.x * (blockDim.x / 32) + warp) * kRows;
    if (row0 >= prm.n) return;  // warp-uniform
    const uint32_t limbs = prm.limbs, tlen = limbs + 2, rows = min(kRows, prm.n - row0);
    // segment g of a row is its words [g span, (g + 1) span)
    const uint32_t chunks = ((tlen + kSegments - 1) / kSegments + kChunk - 1) / kChunk, span = chunks * kChunk;
    const uint32_t own_row = lane / kSegments, own_segment = lane % kSegments;
    const uint64_t* d0 = prm.dots + size_t(row0) * prm.dots_stride;

    // chunk c of every lane's segment, and of q and R, into slot c % kReduceSlots
    auto fetch = [&](uint32_t c) {
        if (c < chunks) {
            constexpr uint32_t kLanes = kChunk / 2;  // per segment, 16 bytes each
            const uint32_t slot = slots_addr + (c % kReduceSlots) * Slot::kBytes;
            const uint32_t w = c * kChunk + 2 * (lane % kLanes);
#pragma unroll 8
            for (uint32_t i = 0; i < kLanes; ++i) {
                const uint32_t r = i * (32 / kLanes) + lane / kLanes, at = (r % kSegments) * span + w;
                if (r / kSegments < rows && at < prm.dots_stride)
                    cp_async_16(slot + r * kPitch + (lane % kLanes) * 16, d0 + size_t(r / kSegments) * prm.dots_stride + at);
            }
            constexpr uint32_t kPieces = kChunk / 2;  // of a segment's tables: q, then R
            for (uint32_t i = lane; i < kSegments * kPieces; i += 32) {
                const uint32_t g = i / kPieces, piece = i % kPieces, at = g * span + c * kChunk + piece % (kPieces / 2) * 4;
                if (at < reduce_table_words(limbs))
                    cp_async_16(slot + 32 * kPitch + g * Slot::kTablePitch + piece * 16,
                                (piece < kPieces / 2 ? prm.q : prm.minus_p) + at);
            }
        }
        cp_async_commit();
    };
    for (uint32_t c = 0; c < kReduceSlots; ++c) fetch(c);

    const uint64_t* d = d0 + size_t(min(own_row, rows - 1)) * prm.dots_stride;
    const uint64_t x[3] = {d[limbs + 2], d[limbs + 3], d[limbs + 4]};
    uint64_t window[kWindow];
#pragma unroll
    for (int j = 0; j < kWindow; ++j) {
        uint32_t w;
        window[j] = window_word(prm, j, w) ? d[w] : 0;
    }
    const RowQuotient f = row_quotient(x, window, prm);
    RowState st;
    uint64_t above = 0;  // what the segment adds to the words from L up (in units of word L)
    if (kSegments > 1 && own_segment > 0 && own_segment * span <= limbs) st.start(f, prm.q[own_segment * span - 1]);
    for (uint32_t c = 0; c < chunks; ++c) {
        cp_async_wait<kReduceSlots - 1>();
        __syncwarp();
        uint8_t* slot = slots + (c % kReduceSlots) * Slot::kBytes;
        uint8_t* own = slot + lane * kPitch;
        const uint4* q4 = reinterpret_cast<const uint4*>(slot + 32 * kPitch + own_segment * Slot::kTablePitch);
        const uint4* r4 = q4 + kChunk / 4;
        const uint32_t base = own_segment * span + c * kChunk;
#pragma unroll 1
        for (uint32_t part = 0; part < kChunk; part += 16) {  // 16 words at a time through registers
            if (kSegments == 1 && base + part >= tlen) break;
            uint64_t sums[16];
            uint4 q[4], r[4];
            const bool table = base + part < tlen;  // past a row's end there is nothing (and nothing was fetched)
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g) {
                q[g] = table ? q4[part / 4 + g] : make_uint4(0, 0, 0, 0);
                r[g] = table ? r4[part / 4 + g] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t g = 0; g < 8; ++g) {
                const ulonglong2 pair = *reinterpret_cast<const ulonglong2*>(own + part * 8 + g * 16);
                sums[2 * g] = pair.x;
                sums[2 * g + 1] = pair.y;
            }
            uint32_t o[16];
            st.words16(f, sums, q, r, base + part, prm, o);
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g)  // over words that this thread has already read
                *reinterpret_cast<uint4*>(own + part * 4 + g * 16) =
                    make_uint4(o[4 * g], o[4 * g + 1], o[4 * g + 2], o[4 * g + 3]);
            if (kSegments > 1 && base + part + 16 > limbs) {
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i) {
                    if (base + part + i == limbs) above += o[i];
                    if (base + part + i == limbs + 1) above += uint64_t(o[i]) << 32;
                }
            }
        }
        __syncwarp();
        if constexpr (kChunk == 16) {
            // two lanes' words per instruction (r and r + 4: their banks do not meet), 64 bytes each
#pragma unroll
            for (uint32_t i = 0; i < 16; ++i) {
                const uint32_t r = (i / 4) * 8 + i % 4 + (lane / 16) * 4;
                const uint32_t w = (r % kSegments) * span + c * kChunk + lane % 16;
                if (r / kSegments < rows && w < limbs)
                    prm.out[size_t(row0 + r / kSegments) * limbs + w] =
                        reinterpret_cast<const uint32_t*>(slot + r * kPitch)[lane % 16];
            }
        } else {
            static_assert(kChunk == 16 || kSegments == 1, "wide chunks go with whole rows");
#pragma unroll
            for (uint32_t part = 0; part < kChunk; part += 32) {
                if (base + part + lane >= limbs) continue;
                uint32_t* out = prm.out + size_t(row0) * limbs + base + part + lane;
#pragma unroll 8
                for (uint32_t r = 0; r < rows; ++r)
                    out[size_t(r) * limbs] = reinterpret_cast<const uint32_t*>(slot + r * kPitch)[part + lane];
            }
        }
        __syncwarp();
        fetch(c + kReduceSlots);
    }
    uint32_t* row = prm.out + size_t(row0 + min(own_row, rows - 1)) * limbs;
    if constexpr (kSegments == 1) {
        if (lane < rows) st.finish(row, prm);
    } else {
        // carries between segments; above word L they are summed up instead
        const uint32_t start = own_segment * span, end = start + span;
        int64_t up = own_row < rows ? st.carry : 0;
        if (end >= limbs) {
            if (end < limbs + 2) above += uint64_t(up) << (32 * (end - limbs));
            up = 0;
        }
        while (__any_sync(0xffffffffu, up != 0)) {
            int64_t carry = __shfl_up_sync(0xffffffffu, up, 1, kSegments);
            if (own_segment == 0) carry = 0;
            up = 0;
            uint32_t w = start;
            for (; carry != 0 && w < min(end, limbs); ++w) {
                const int64_t t = int64_t(row[w]) + carry;
                row[w] = uint32_t(t);
                carry = t >> 32;
            }
            if (w < limbs)
                up = carry;
            else
                above += uint64_t(carry);
        }
#pragma unroll
        for (uint32_t i = 1; i < kSegments; i *= 2) above += __shfl_xor_sync(0xffffffffu, above, i, kSegments);
        __syncwarp();
        if (own_segment == 0 && own_row < rows) RowState::finish_in_memory(row, uint32_t(above), prm);
    }
}

uint32_t log2_u32(uint32_t x) { return x ? 31 - __builtin_clz(x) : 0; }

}  // namespace

void launch_pad_operands(const uint32_t* a, const uint32_t* b, uint32_t* out, uint32_t n, uint32_t limbs,
                         uint32_t padded_limbs, uint32_t split, uint32_t* tile_counters, cudaStream_t stream) {
    const uint32_t log_split = log2_u32(split), log_n_sub = log2_u32(n) - log_split;
    const uint32_t blocks = std::min<uint32_t>((2 * n + 7) / 8, 148 * 16);  // 8 rows (warps) per block
    launch_chained(pad_operands_kernel, blocks, 256, 0, stream, a, b, out, n, limbs, padded_limbs, log_split, log_n_sub,
                   tile_counters);
}

void launch_pad_rows(const uint32_t* staged, uint32_t* out, uint32_t n, uint32_t limbs, uint32_t padded_limbs,
                     uint32_t split, uint32_t first_row, uint32_t count, cudaStream_t stream, uint32_t op_first,
                     uint32_t op_count) {
    const uint32_t log_split = log2_u32(split), log_n_sub = log2_u32(n) - log_split;
    const uint32_t blocks = std::min<uint32_t>((op_count * count + 7) / 8, 148 * 16);
    launch_chained(pad_rows_kernel, blocks, 256, 0, stream, staged, out, n, limbs, padded_limbs, log_split, log_n_sub, first_row,
                                                count, op_first, op_count);
}

void launch_twiddles(const DevicePrime* primes, uint32_t r, uint32_t n_sub, uint2* fwd, uint2* inv, uint2* zeta,
                     cudaStream_t stream) {
    dim3 grid((n_sub + 255) / 256, r);
    twiddles_kernel<<<grid, 256, 0, stream>>>(primes, r, n_sub, log2_u32(n_sub), fwd, inv, zeta);
}

void launch_convert_weights(const DevicePrime* primes, uint32_t r, uint32_t padded_r, uint32_t limbs,
                            uint32_t k_bytes, uint8_t* out, cudaStream_t stream) {
    dim3 grid((k_bytes + 255) / 256, padded_r);
    convert_weights_kernel<<<grid, 256, 0, stream>>>(primes, r, padded_r, limbs, k_bytes, out);
}

void launch_crt_weights(const uint32_t* weights_words, uint32_t r, uint32_t padded_r, uint32_t words,
                        uint32_t columns, uint8_t* out, cudaStream_t stream) {
    dim3 grid((4 * padded_r + 255) / 256, columns);
    crt_weights_kernel<<<grid, 256, 0, stream>>>(weights_words, r, padded_r, words, columns, out);
}

void launch_gemm_simt(const uint8_t* a, uint64_t a_pitch, RowMap rows, uint32_t m, const uint8_t* b,
                      uint32_t columns, uint32_t k_bytes, const Epilogue& epilogue, cudaStream_t stream) {
    dim3 grid((m + kTile - 1) / kTile, (columns + kTile - 1) / kTile);
    launch_chained(gemm_simt_kernel, grid, 256, 0, stream, a, a_pitch, rows, m, b, columns, k_bytes, epilogue);
}

static uint32_t ntt_threads(uint32_t n_sub) {
    uint32_t half = n_sub / 2;
    return half >= 512 ? 512 : (half >= 32 ? half : 32);
}

template <bool kForward, uint32_t kLog>
static void launch_blocked(uint32_t* residues, const DevicePrime* primes, const uint2* table, uint32_t r, uint32_t n,
                           uint32_t first, uint32_t count, cudaStream_t stream, uint32_t op_first, uint32_t op_count) {
    constexpr uint32_t kN = 1u << kLog;
    const size_t smem = kN * sizeof(uint32_t);
    auto kernel = kForward ? ntt_forward_blocked_kernel<kLog> : ntt_inverse_blocked_kernel<kLog>;
    static bool configured = false;
    if (!configured) {  // room for several transforms per SM
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        configured = true;
    }
    dim3 grid(kForward ? op_count * count : count, r);
    launch_chained(kernel, grid, kN / per_thread(kLog), smem, stream, residues, primes, table, r, n, first, count, op_first);
}

template <bool kForward>
static bool launch_blocked_any(uint32_t n_sub, uint32_t* residues, const DevicePrime* primes, const uint2* table,
                               uint32_t r, uint32_t n, uint32_t first, uint32_t count, cudaStream_t stream,
                               uint32_t op_first = 0, uint32_t op_count = 2) {
#define NEGACYCLIC_BLOCKED(LOG) \
    launch_blocked<kForward, LOG>(residues, primes, table, r, n, first, count, stream, op_first, op_count)
    switch (n_sub) {
        case 256: NEGACYCLIC_BLOCKED(8); return true;
        case 512: NEGACYCLIC_BLOCKED(9); return true;
        case 1024: NEGACYCLIC_BLOCKED(10); return true;
        case 2048: NEGACYCLIC_BLOCKED(11); return true;
        case 4096: NEGACYCLIC_BLOCKED(12); return true;
        case 8192: NEGACYCLIC_BLOCKED(13); return true;
        default: return false;
    }
#undef NEGACYCLIC_BLOCKED
}

void launch_ntt_forward(uint32_t* residues, const DevicePrime* primes, const uint2* fwd, uint32_t r, uint32_t n,
                        uint32_t n_sub, uint32_t t_first, uint32_t t_count, cudaStream_t stream, uint32_t op_first,
                        uint32_t op_count) {
    if (launch_blocked_any<true>(n_sub, residues, primes, fwd, r, n, t_first, t_count, stream, op_first, op_count))
        return;
    dim3 grid(t_count, r, op_count);
    launch_chained(ntt_forward_kernel, grid, ntt_threads(n_sub), n_sub * sizeof(uint32_t), stream, residues, primes, fwd, r,
                   n, n_sub, t_first, op_first);
}

void launch_ntt_inverse(uint32_t* residues, const DevicePrime* primes, const uint2* inv, uint32_t r, uint32_t n,
                        uint32_t n_sub, uint32_t v_first, uint32_t v_count, cudaStream_t stream) {
    if (launch_blocked_any<false>(n_sub, residues, primes, inv, r, n, v_first, v_count, stream)) return;
    dim3 grid(v_count, r);
    launch_chained(ntt_inverse_kernel, grid, ntt_threads(n_sub), n_sub * sizeof(uint32_t), stream, residues, primes, inv, r,
                   n, n_sub, v_first);
}

template <uint32_t kLog>
static void launch_product(uint32_t* residues, const DevicePrime* primes, const uint2* fwd, const uint2* inv, uint32_t r,
                           cudaStream_t stream) {
    constexpr uint32_t kN = 1u << kLog;
    constexpr int kSmem = 2 * kN * sizeof(uint32_t);
    if (kSmem > 48 * 1024)  // per device; cheap enough to repeat
        cudaFuncSetAttribute(ntt_product_kernel<kLog>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    launch_chained(ntt_product_kernel<kLog>, r, 2 * kN / per_thread(kLog), kSmem, stream, residues, primes, fwd, inv, r);
}

static uint32_t small_threads(uint32_t n, uint32_t r) { return std::max(512u, (n / 8 * r + 31) / 32 * 32); }

static size_t small_smem(uint32_t n, uint32_t r, uint32_t limbs) {
    return (size_t(n) * (2 * r + std::max(2 * limbs, limbs + 5)) + size_t(r) * (2 * limbs + 5) + 2 * (limbs + 2)) *
           sizeof(uint32_t);
}

// The line lies where the three kernels catch up. Product, us, one kernel / three, at N r L of:
// 2560 (N=256, L=2) 8.9 / 12.0, 4608 (N=128, L=4) 8.5 / 12.3, 9216 (N=256, L=4) 14.1 / 12.0, 16384 (N=128,
// L=8) 15.5 / 12.3, 5120 (N=512, L=2) 16.0 / 12.0. At N=64 the tensor GEMMs do not apply: 6272 (L=7) 11.3 /
// 19.8, 16896 (L=11) 18.1 / 20. With few primes (q much shorter than its limbs) the L + 5 words that a thread
// takes one after another count instead: N=64, one prime, 14.9 at L=48, 20.5 at 64, 46.9 at 160 and 55.6 at
// 192 against 20 at 64, 27 at 160 and 29 at 192.
// The launch stays within the 48 KB of static and dynamic shared memory that need no attribute (43 KB
// at most under the other bounds): an attribute would belong to the kernel, not to the plan, and plans on
// other threads set theirs.
bool small_product_takes(uint32_t n, uint32_t r, uint32_t limbs) {
    return n >= 64 && n <= 256 && r <= kSmallPrimes && small_threads(n, r) <= 512 && limbs <= 48 &&
           uint64_t(n) * r * limbs <= (n == 64 ? 12288 : 5000) &&
           small_smem(n, r, limbs) + kSmallPrimes * sizeof(DevicePrime) <= 48 * 1024;
}

template <uint32_t kLog>
static void launch_small(const SmallProduct& params, cudaStream_t stream) {
    constexpr uint32_t kN = 1u << kLog;
    launch_chained(small_product_kernel<kLog>, 1, small_threads(kN, params.r),
                   small_smem(kN, params.r, params.reduce.limbs), stream, params);
}

void launch_small_product(const SmallProduct& params, cudaStream_t stream) {
    switch (params.reduce.n) {
        case 64: launch_small<6>(params, stream); break;
        case 128: launch_small<7>(params, stream); break;
        default: launch_small<8>(params, stream); break;
    }
}

bool launch_ntt_product(uint32_t* residues, const DevicePrime* primes, const uint2* fwd, const uint2* inv, uint32_t r,
                        uint32_t n, cudaStream_t stream) {
    switch (n) {
        case 64: launch_product<6>(residues, primes, fwd, inv, r, stream); return true;
        case 128: launch_product<7>(residues, primes, fwd, inv, r, stream); return true;
        case 256: launch_product<8>(residues, primes, fwd, inv, r, stream); return true;
        case 512: launch_product<9>(residues, primes, fwd, inv, r, stream); return true;
        case 1024: launch_product<10>(residues, primes, fwd, inv, r, stream); return true;
        case 2048: launch_product<11>(residues, primes, fwd, inv, r, stream); return true;
        case 4096: launch_product<12>(residues, primes, fwd, inv, r, stream); return true;
        case 8192: launch_product<13>(residues, primes, fwd, inv, r, stream); return true;
        default: return false;
    }
}

void launch_pointwise(uint32_t* residues, const DevicePrime* primes, const uint2* zeta, uint32_t r, uint32_t n,
                      uint32_t n_sub, uint32_t split, cudaStream_t stream) {
#define NEGACYCLIC_POINTWISE(S, V) \
    launch_chained(pointwise_kernel<S, V>, grid, 128, 0, stream, residues, primes, zeta, r, n, n_sub)
    if (n_sub % 2 == 0) {  // two evaluation points per thread
        dim3 grid((n_sub / 2 + 127) / 128, r);
        switch (split) {
            case 1: NEGACYCLIC_POINTWISE(1, 2); break;
            case 2: NEGACYCLIC_POINTWISE(2, 2); break;
            case 4: NEGACYCLIC_POINTWISE(4, 2); break;
            case 8: NEGACYCLIC_POINTWISE(8, 2); break;
            default: NEGACYCLIC_POINTWISE(16, 2); break;
        }
        return;
    }
    dim3 grid((n_sub + 127) / 128, r);
    switch (split) {
        case 1: NEGACYCLIC_POINTWISE(1, 1); break;
        case 2: NEGACYCLIC_POINTWISE(2, 1); break;
        case 4: NEGACYCLIC_POINTWISE(4, 1); break;
        case 8: NEGACYCLIC_POINTWISE(8, 1); break;
        default: NEGACYCLIC_POINTWISE(16, 1); break;
    }
#undef NEGACYCLIC_POINTWISE
}

void launch_transpose(const uint32_t* residues, uint32_t* crt_in, uint32_t r, uint32_t padded_r, uint32_t n,
                      uint32_t split, uint32_t j_first, uint32_t j_count, cudaStream_t stream) {
    const uint32_t log_split = log2_u32(split), log_n_sub = log2_u32(n) - log_split;
    dim3 grid(split * ((j_count + kTransposeTile - 1) / kTransposeTile), (padded_r + kTransposeTile - 1) / kTransposeTile);
    launch_chained(transpose_kernel, grid, 256, 0, stream, residues, crt_in, r, padded_r, n, log_split, log_n_sub, j_first,
                   j_count);
}

template <uint32_t kChunk, uint32_t kSegments>
static void launch_reduce_chunks(const ReduceParams& params, uint32_t warps, cudaStream_t stream) {
    const size_t smem = size_t(warps) * kReduceSlots * ReduceSlot<kChunk, kSegments>::kBytes;
    if (smem > 48 * 1024)  // per device; cheap enough to repeat
        cudaFuncSetAttribute(reduce_kernel<kChunk, kSegments>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    const uint32_t rows = 32 / kSegments, groups = (params.n + rows - 1) / rows;  // of `rows` rows, a warp each
    launch_chained(reduce_kernel<kChunk, kSegments>, (groups + warps - 1) / warps, warps * 32, smem, stream, params);
}

void launch_reduce(const ReduceParams& params, cudaStream_t stream) {
    // Segments for fewer rows than a warp of them on every other SM: as many as leave 16 words each.
    // Product, us, whole rows / segments: 186.8 / 131.3 (N = 256, L = 1747), 358.5 / 324.7 (N = 1024),
    // 44.3 / 36.4 (N = 256, L = 313); from 4096 rows on they lose: 45.8 / 48.0 (L = 94), 893 / 909
    // (N = 16384, L = 625).
    uint32_t segments = 1;
    if (params.n < 16 * 148)
        while (segments < 16 && params.limbs / (2 * segments) >= 16) segments *= 2;
    switch (segments) {
        case 2: launch_reduce_chunks<16, 2>(params, 1, stream); return;
        case 4: launch_reduce_chunks<16, 4>(params, 1, stream); return;
        case 8: launch_reduce_chunks<16, 8>(params, 1, stream); return;
        case 16: launch_reduce_chunks<16, 16>(params, 1, stream); return;
        default: break;
    }
    // Chunks of 64 words (512-byte runs per row) read DRAM better than chunks of 16 (128-byte runs
    // of rows 14 KB apart): 362 against 432 us at N = 65536, L = 1747, 22.5 against 30.4 at N = 16384,
    // L = 301. A row of up to 64 words is better read in four steps, with more warps per SM: 20.5
    // against 24.6 us at N = 65536, L = 55. (us of the stage between events, about 5 of them launch.)
    if (params.limbs + 2 <= 64)
        launch_reduce_chunks<16, 1>(params, params.n > 32 * 148 * 2 ? 2 : 1, stream);
    else
        launch_reduce_chunks<64, 1>(params, 1, stream);
}

}  // namespace negacyclic
