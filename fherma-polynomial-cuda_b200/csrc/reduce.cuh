// CRT quotient, carries and reduction mod q of one coefficient by one thread, shared by the reduce
// kernel (word sums in global memory) and the CRT GEMM that reduces in its epilogue (word sums in
// TMEM).
//
// The CRT word sums split cleanly: words [0, L+2) are a carry-save form of
// T = sum v_k M_k (< 2^(32(L+2)), so nothing carries out of them), words
// L+2..L+4 a carry-save form of D = sum v_k floor(2^64/p_k). Hence
//   K  = (D + 2^63) >> 64 straight from three word sums,
//   T' = T + K R (R = -P mod q), T' = x (mod q), T' < 2^48 q,
//   c  = T' - quotient q, then at most three q's off.
// The quotient is known before the carries are: Barrett needs the 128 bits of T' from top_shift
// up, and the words below the window carry less than 2^26 into it. Starting the window two words
// lower bounds the missing carry by one unit of the window's lowest bit, which can only make the
// quotient smaller, by less than 2^-62 before the floor. So one pass over the row, lowest word
// first, forms d[w] + K R[w] - quotient q and its carries at once.
#pragma once
#include "kernels.cuh"

namespace negacyclic {

struct RowQuotient {
    uint32_t k;          // CRT quotient K < 2r
    uint32_t low, high;  // Barrett quotient of T' by q, < 2^48
};

constexpr int kWindow = 7;  // word sums of T that the quotient reads: ws - 2 .. ws + 4, ws = floor(top_shift / 32)

// Whether word ws - 2 + j of a row belongs to T (others count as zero).
__device__ __forceinline__ bool window_word(const ReduceParams& prm, int j, uint32_t& w) {
    const int32_t at = (prm.top_shift >> 5) - 2 + j;
    w = uint32_t(at);
    return at >= 0 && at < int32_t(prm.limbs) + 2;
}

// K and the Barrett quotient of a row: x[i] = d[L+2+i], window[j] = d[ws-2+j] (zero outside T); the
// word sums are below 2^56.
__device__ __forceinline__ RowQuotient row_quotient(const uint64_t (&x)[3], const uint64_t (&window)[kWindow],
                                                    const ReduceParams& prm) {
    // K = (D + 2^63) >> 64, D = x[0] + x[1] 2^32 + x[2] 2^64
    const uint64_t low = x[0] + (x[1] << 32);
    const uint64_t high = (x[1] >> 32) + x[2] + (low < x[0] ? 1 : 0);  // D = high 2^64 + low
    const uint32_t k = uint32_t(high + ((low + (1ull << 63)) < low ? 1 : 0));
    const uint32_t offset = uint32_t(prm.top_shift) & 31u;
    uint32_t z[5];  // T' words at ws .. ws+4
    uint64_t acc = 0;
#pragma unroll
    for (int j = 0; j < kWindow; ++j) {
        uint32_t w;
        if (window_word(prm, j, w)) acc += window[j] + uint64_t(k) * prm.minus_p[w];
        if (j >= 2) z[j - 2] = uint32_t(acc);
        acc >>= 32;
    }
    const uint64_t tl = uint64_t(__funnelshift_r(z[0], z[1], offset)) |
                        (uint64_t(__funnelshift_r(z[1], z[2], offset)) << 32);
    const uint64_t th = uint64_t(__funnelshift_r(z[2], z[3], offset)) |
                        (uint64_t(__funnelshift_r(z[3], z[4], offset)) << 32);
    const uint64_t prod_l_hi = __umul64hi(tl, prm.mu_low);
    const uint64_t prod_h_lo = th * prm.mu_low, prod_h_hi = __umul64hi(th, prm.mu_low);
    const uint64_t word1 = prod_l_hi + prod_h_lo;
    const uint64_t word2 = prod_h_hi + (word1 < prod_l_hi ? 1 : 0);
    const uint64_t quotient = th + word2 + ((tl + word1 < tl) ? 1 : 0);
    return RowQuotient{k, uint32_t(quotient), uint32_t(quotient >> 32)};
}

// Takes q off a row (limbs words in global memory, `over` above them) while it is not below q;
// returns false if more than three subtractions were needed.
static __device__ __noinline__ bool correct_row(uint32_t* row, uint32_t over, const uint32_t* __restrict__ q,
                                                uint32_t limbs) {
    for (int corrections = 0;; ++corrections) {
        if (over == 0) {
            uint32_t w = limbs;
            while (w > 0 && row[w - 1] == q[w - 1]) --w;
            if (w > 0 && row[w - 1] < q[w - 1]) return true;
        }
        if (corrections == 3) return false;
        uint32_t borrow = 0;
        for (uint32_t w = 0; w < limbs; ++w) {
            const uint64_t t = uint64_t(row[w]) - q[w] - borrow;
            row[w] = uint32_t(t);
            borrow = uint32_t(t >> 63);
        }
        over -= borrow;
    }
}

// Running state of one row's pass.
// (A row may be cut into segments that start with no carry; they start with start().)
struct RowState {
    int64_t carry = 0;   // signed carry into the next word
    uint64_t below = 0;  // hi(ql q[w-1]) + qh q[w-1], subtracted at word w
    // of the result: words at and above q's (or-ed), and the two below
    uint32_t over = 0, top1 = 0, top0 = 0;

    // Before a first word above word 0: `q_below` is the word of q under it.
    __device__ __forceinline__ void start(const RowQuotient& f, uint32_t q_below) {
        below = ((uint64_t(f.low) * q_below) >> 32) + uint64_t(f.high) * q_below;
    }

    // Word w of T' - quotient q: d + K R - lo(ql q) - below + carry. d < 2^56, K R < 2^46 and
    // below < 2^49, so the sum stays within int64.
    __device__ __forceinline__ uint32_t word(const RowQuotient& f, uint64_t d, uint32_t r, uint32_t q) {
        const uint64_t a = uint64_t(f.low) * q;
        const int64_t y = int64_t(d + uint64_t(f.k) * r) - int64_t(uint32_t(a)) - int64_t(below);
        below = (a >> 32) + uint64_t(f.high) * q;
        const int64_t z = y + carry;
        carry = z >> 32;
        return uint32_t(z);
    }

    // Words base .. base + 15 of the row from their word sums (zeroed here from L+2 up, which are not
    // part of T) and the same words of q and R, four per vector.
    __device__ __forceinline__ void words16(const RowQuotient& f, uint64_t (&d)[16], const uint4 (&q)[4],
                                            const uint4 (&r)[4], uint32_t base, const ReduceParams& prm,
                                            uint32_t (&o)[16]) {
        if (base + 16 > prm.limbs + 2) {
#pragma unroll
            for (uint32_t i = 0; i < 16; ++i)
                if (base + i >= prm.limbs + 2) d[i] = 0;
        }
#pragma unroll
        for (uint32_t g = 0; g < 4; ++g) {
            o[4 * g] = word(f, d[4 * g], r[g].x, q[g].x);
            o[4 * g + 1] = word(f, d[4 * g + 1], r[g].y, q[g].y);
            o[4 * g + 2] = word(f, d[4 * g + 2], r[g].z, q[g].z);
            o[4 * g + 3] = word(f, d[4 * g + 3], r[g].w, q[g].w);
        }
        if (base + 16 + 2 > prm.q_words) {  // some of the top words
#pragma unroll
            for (uint32_t i = 0; i < 16; ++i) note(o[i], base + i, prm);
        }
    }

    // Keeps what finish() needs of word w of the result.
    __device__ __forceinline__ void note(uint32_t o, uint32_t w, const ReduceParams& prm) {
        if (w + 2 == prm.q_words) top0 = o;
        if (w + 1 == prm.q_words) top1 = o;
        if (w >= prm.q_words) over |= o;
    }

    // The same for a row whose words are only in global memory, `above` standing over them.
    static __device__ __forceinline__ void finish_in_memory(uint32_t* row, uint32_t above, const ReduceParams& prm) {
        RowState st;
        st.over = above | (prm.q_words < prm.limbs ? row[prm.q_words] : 0u);
        st.top1 = row[prm.q_words - 1];
        st.top0 = prm.q_words >= 2 ? row[prm.q_words - 2] : 0u;
        st.finish(row, prm);
    }

    // After the row is in global memory: a result whose top two words are below q's is canonical; the
    // rest compare whole rows.
    __device__ __forceinline__ void finish(uint32_t* row, const ReduceParams& prm) const {
        const uint64_t top = (uint64_t(top1) << 32) | top0;
        const uint64_t q_top = (uint64_t(prm.q[prm.q_words - 1]) << 32) |
                               (prm.q_words >= 2 ? prm.q[prm.q_words - 2] : 0u);
        if (over == 0 && top < q_top) return;
        if (!correct_row(row, prm.q_words < prm.limbs ? 0u : over, prm.q, prm.limbs)) atomicOr(prm.error_flag, 1u);
    }
};

}  // namespace negacyclic
