// Sizes and places of the small device buffers of a Lanczos run (one allocation), by the largest number of
// basis vectors and the number of SMs, and the rule for the precision of its correction.  Plain C++ too: the
// host tests compile it without CUDA.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define EDGPU_HOST_DEVICE __host__ __device__ inline
#else
#define EDGPU_HOST_DEVICE inline
#endif

namespace edgpu {

constexpr int RED_BLOCKS = 1024;      // blocks of a norm
constexpr int LZ_THREADS = 256;
constexpr int LZ_G = 16;              // basis vectors per block of the projections (accumulators in registers)
constexpr int LZ_AXPY_THREADS = 128;
constexpr int LZ_MAX_BLOCKS = 4096;

// Groups of at most LZ_G vectors that the projections of k vectors are taken in.
inline int lz_groups(int k) { return std::max(1, (k + LZ_G - 1) / LZ_G); }

// Row blocks of the projections: two blocks per SM (all that fit) over all groups of vectors.
inline int lz_row_blocks(int64_t n, int groups, int sms) {
    const int64_t need = (n + LZ_THREADS - 1) / LZ_THREADS;
    return (int)std::max<int64_t>(1, std::min<int64_t>(need, 2ll * std::max(1, sms) / groups));
}

// Doubles of partial sums: those of the projections (2 LZ_G doubles a block, at most two blocks per SM or one
// row block per group, and a norm per row block) and those of the other kernels.
inline size_t lanczos_scratch_doubles(int kmax, int sms) {
    const size_t blocks = std::max<size_t>((size_t)lz_groups(kmax), 2 * (size_t)std::max(1, sms));
    const size_t need = std::max<size_t>({2 * LZ_G * blocks + blocks, 2 * (size_t)LZ_MAX_BLOCKS, 2 * (size_t)RED_BLOCKS});
    return (need + 15) / 16 * 16;   // (what follows is read 16 bytes at a time)
}

// Offsets in doubles for at most m steps.
struct LanczosSmall {
    size_t scal = 0;       // 16 scalars
    size_t scratch, h, hmax, tickets, total;   // h: m + 1 complex numbers, read and written as double2
    size_t n_groups;
};
inline LanczosSmall lanczos_small(int m, int sms) {
    LanczosSmall o;
    o.n_groups = (size_t)m / LZ_G + 2;
    o.scratch = o.scal + 16;
    o.h = o.scratch + lanczos_scratch_doubles(m + 1, sms);
    o.hmax = o.h + 2 * (size_t)(m + 1);
    o.tickets = o.hmax + o.n_groups;
    o.total = o.tickets + o.n_groups;
    return o;
}

// Whether the sum of K basis vectors of norm 1 with coefficients h_k, taken off a vector of squared norm nrm2, may
// be formed in single precision: |Re h_k|, |Im h_k| <= hmax.  Each component is a chain of at most two FMAs per
// vector and LZ_CHUNK vectors (the chunks add up in FP64), of coefficients rounded to 24 bits and vectors cut to
// 24 bits: a relative error of at most (2 min(K, LZ_CHUNK) + 4) 2^-24 in every term, so 2 (that) K hmax in the norm
// of the sum.  The rule keeps it below 2^-54 of the vector's norm, half of a double's rounding.  Not for NaN,
// infinities, or coefficients below 2^-900 (whose scale is not a double).
constexpr int LZ_CHUNK = 256;
EDGPU_HOST_DEVICE bool lz_single_precision(int K, double hmax, double nrm2) {
    const double reach = hmax * (double)K * (double)(2 * (K < LZ_CHUNK ? K : LZ_CHUNK) + 4) * 2147483648.0;
    return reach * reach <= nrm2 && hmax >= 0x1p-900;
}

}  // namespace edgpu
