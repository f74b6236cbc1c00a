// Vector kernels around the product: seeded start vectors, precision conversion, deterministic FP64
// reductions (dots, norms, Gram-Schmidt projections) and the Lanczos three-term update.
// All reductions use a fixed grid and a fixed second-stage order, so results are reproducible.
#include <algorithm>
#include <array>
#include <cmath>
#include <type_traits>
#include <utility>

#include "edgpu_internal.h"
#include "lanczos_layout.h"

namespace edgpu {

namespace {

constexpr int RED_THREADS = 256;

unsigned grid_for(int64_t n, int threads = 256) {
    int64_t b = (n + threads - 1) / threads;
    if (b > 1048576) b = 1048576;
    if (b < 1) b = 1;
    return (unsigned)b;
}

__device__ __forceinline__ unsigned long long splitmix64_at(unsigned long long seed, unsigned long long k) {
    unsigned long long z = seed + (k + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_random_c128(long long n, unsigned long long seed, double2* dst) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double u = (double)(splitmix64_at(seed, 2ull * i) >> 11) * (1.0 / 9007199254740992.0);
        const double u2 = (double)(splitmix64_at(seed, 2ull * i + 1ull) >> 11) * (1.0 / 9007199254740992.0);
        const double u1 = 1.0 - u;
        const double r = sqrt(-2.0 * log(u1));
        const double ang = 2.0 * M_PI * u2;
        const double s = 0.70710678118654752440;   // 1/sqrt(2)
        dst[i] = make_double2(r * cos(ang) * s, r * sin(ang) * s);
    }
}

__global__ void k_c128_to_c64(long long n, const double2* src, float2* dst) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double2 v = src[i];
        dst[i] = make_float2((float)v.x, (float)v.y);
    }
}

__global__ void k_c64_to_c128(long long n, const float2* src, double2* dst, int accumulate) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float2 v = src[i];
        double2 o = make_double2((double)v.x, (double)v.y);
        if (accumulate) {
            const double2 a = dst[i];
            o.x += a.x;
            o.y += a.y;
        }
        dst[i] = o;
    }
}

__global__ void k_conj_c128(long long n, double2* v) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[i].y = -v[i].y;
}

__device__ __forceinline__ double2 block_sum2(double2 v, double2* sh) {
    for (int d = 16; d > 0; d >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, d);
        v.y += __shfl_down_sync(0xffffffffu, v.y, d);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double2 r = make_double2(0.0, 0.0);
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            r.x += sh[w].x;
            r.y += sh[w].y;
        }
    __syncthreads();
    return r;
}

// Norm, stage 1: |a_i|^2 over a grid-stride slice; partial per block.
__global__ void k_norm_stage1(long long n, const double2* a, double2* partial) {
    __shared__ double2 sh[32];
    double2 s = make_double2(0.0, 0.0);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double2 u = a[i];
        s.x += u.x * u.x + u.y * u.y;
    }
    const double2 r = block_sum2(s, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

// Stage 2: fixed-order sum of the partials; out = the norm and its inverse.
__global__ void k_norm_stage2(int nparts, const double2* partial, double* out) {
    __shared__ double2 sh[32];
    double2 s = make_double2(0.0, 0.0);
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) s.x += partial[i].x;
    const double2 r = block_sum2(s, sh);
    if (threadIdx.x == 0) {
        out[0] = sqrt(r.x);
        out[1] = 1.0 / out[0];
    }
}

// out[c] = sum over the blocks of partial[b][c]: a warp per coupling, lane l adds the blocks l, l + 32, ...,
// then a butterfly (a fixed order; one thread per coupling took 24 us for 304 blocks).
__global__ void k_reduce_grad(int nblocks, int ncoupl, const double* partial, double* out) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (c >= ncoupl) return;
    double s = 0.0;
    for (int b = lane; b < nblocks; b += 32) s += partial[(size_t)b * ncoupl + c];
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) out[c] = s;
}

// ---- one Lanczos step (launch_lanczos_*): alpha, recurrence and projections, correction, next vector ----
// A step on a stored basis of K = j + 1 vectors costs 8 N K double-precision FMAs, which the FP64 pipe of
// the SMs (two FMAs a cycle each) takes longer over than the memory takes to deliver the basis twice; so
// the projections are computed once per step, on the recurrence's result, which is orthogonal to the
// basis up to rounding, and a second time only when they took away most of it (the caller's test).
// Sums run in a fixed order: per thread, per block, then the last block of a group to finish adds the
// blocks' partial sums (a ticket counter tells it; no block waits).  Sector of 112,720 rows, 100 steps:
// 42.8 -> 11.1 ms a run (before: two passes of a dot kernel with a block row per vector and a subtraction
// kernel, separate reductions, a synchronisation per step).
__device__ __forceinline__ double2 lz_load(const double2* p) { return *p; }
__device__ __forceinline__ double2 lz_load(const float2* p) {
    const float2 v = *p;
    return make_double2((double)v.x, (double)v.y);
}

// a += conj(u) w
__device__ __forceinline__ void cdot_acc(double2& a, const double2& u, const double2& w) {
    a.x = fma(u.x, w.x, a.x);
    a.x = fma(u.y, w.y, a.x);
    a.y = fma(u.x, w.y, a.y);
    a.y = fma(-u.y, w.x, a.y);
}

// Whether this block is the last of n to arrive at the ticket counter (which it resets); its threads then
// see what the others wrote before they arrived.
__device__ __forceinline__ bool last_block(unsigned* ticket, unsigned n) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(ticket, 1u) == n - 1;
        if (last) *ticket = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// alpha = <v, w>; y32 != null: w is first written as the widened complex64 product y32
__global__ void __launch_bounds__(LZ_THREADS) k_lz_alpha(long long n, const double2* v, double2* w, const float2* y32,
                                                         double2* partial, double* alpha, unsigned* ticket) {
    __shared__ double2 sh[32];
    double2 s = make_double2(0.0, 0.0);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double2 x;
        if (y32) {
            x = lz_load(y32 + i);
            w[i] = x;
        } else {
            x = w[i];
        }
        cdot_acc(s, v[i], x);
    }
    double2 r = block_sum2(s, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
    if (!last_block(ticket, gridDim.x)) return;
    s = make_double2(0.0, 0.0);
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
        const double2 q = __ldcg(partial + b);
        s.x += q.x;
        s.y += q.y;
    }
    r = block_sum2(s, sh);
    if (threadIdx.x == 0) {
        alpha[0] = r.x;
        alpha[1] = r.y;
    }
}

// h_k = <V_k, w1> for the K vectors of the basis and w1 = w - alpha v - beta u, hmax = the largest of a group's
// |Re h|, |Im h|, nrm2 = |w1|^2.  Grid (row blocks, groups of at most LZ_G vectors): every group forms w1 for
// itself, and so does the correction.
template <typename VT, int S>
__global__ void __launch_bounds__(LZ_THREADS, 2)
k_lz_project(long long n, int K, const VT* V, long long ldv, const double2* w, const double2* v, const double2* u,
             const double* alpha, const double* beta, double2* partial, double2* h, double* hmax, double* nrm2,
             unsigned* ticket) {
    __shared__ double red[LZ_THREADS / 32][2 * LZ_G];
    __shared__ double nsum[LZ_THREADS / 32];
    const int KG = gridDim.y, RB = gridDim.x, grp = blockIdx.y;
    const int k0 = (int)((long long)K * grp / KG), nk = (int)((long long)K * (grp + 1) / KG) - k0;
    const double a = v ? alpha[0] : 0.0, b = u ? beta[0] : 0.0;
    double2 acc[LZ_G];   // (the first S)
#pragma unroll
    for (int g = 0; g < LZ_G; ++g) acc[g] = make_double2(0.0, 0.0);
    double nn = 0.0;
    const VT* Vk = V + (size_t)k0 * ldv;
    // the rows evenly to the row blocks (a block's last warps then idle together, not whole lanes' worth of
    // double-precision instructions)
    const long long r1 = n * (blockIdx.x + 1) / RB;
    for (long long i = n * blockIdx.x / RB + threadIdx.x; i < r1; i += LZ_THREADS) {
        double2 x = w[i];
        if (v) {
            const double2 t = v[i];
            x.x = fma(-a, t.x, x.x);
            x.y = fma(-a, t.y, x.y);
        }
        if (u) {
            const double2 t = u[i];
            x.x = fma(-b, t.x, x.x);
            x.y = fma(-b, t.y, x.y);
        }
        if (grp == 0) nn = fma(x.x, x.x, fma(x.y, x.y, nn));
        // (the groups have S or S - 1 vectors)
#pragma unroll
        for (int g = 0; g < S - 1; ++g) cdot_acc(acc[g], lz_load(Vk + (size_t)g * ldv + i), x);
        if (nk == S) cdot_acc(acc[S - 1], lz_load(Vk + (size_t)(S - 1) * ldv + i), x);
    }
    // sums over the warp, halving the values as the lanes pair up: lane l ends with component l of the
    // 2 LZ_G = 32 sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s[2 * LZ_G];
#pragma unroll
    for (int g = 0; g < LZ_G; ++g) {
        s[2 * g] = acc[g].x;
        s[2 * g + 1] = acc[g].y;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const bool up = (lane & d) != 0;
#pragma unroll
        for (int j = 0; j < d; ++j) {
            const double keep = up ? s[j + d] : s[j], give = up ? s[j] : s[j + d];
            s[j] = keep + __shfl_xor_sync(0xffffffffu, give, d);
        }
    }
    red[warp][lane] = s[0];
    if (grp == 0) {
        for (int d = 16; d > 0; d >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, d);
        if (lane == 0) nsum[warp] = nn;
    }
    __syncthreads();
    double* part = (double*)(partial + ((size_t)grp * RB + blockIdx.x) * LZ_G);
    double* npart = (double*)(partial + (size_t)KG * RB * LZ_G);
    if (threadIdx.x < 2 * LZ_G) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < LZ_THREADS / 32; ++q) t += red[q][threadIdx.x];
        part[threadIdx.x] = t;
    } else if (threadIdx.x == 2 * LZ_G && grp == 0) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < LZ_THREADS / 32; ++q) t += nsum[q];
        npart[blockIdx.x] = t;
    }
    if (!last_block(ticket + grp, (unsigned)RB)) return;
    // component c of the group's sums: warp w takes the blocks w, w + 8, ..., then the warps are added
    double t = 0.0;
#pragma unroll 8
    for (int q = warp; q < RB; q += LZ_THREADS / 32)
        t += __ldcg((const double*)(partial + ((size_t)grp * RB + q) * LZ_G) + lane);
    red[warp][lane] = t;
    if (grp == 0 && warp == 0) {
        double z = 0.0;
#pragma unroll 8
        for (int q = lane; q < RB; q += 32) z += __ldcg(npart + q);
        for (int d = 16; d > 0; d >>= 1) z += __shfl_xor_sync(0xffffffffu, z, d);
        if (lane == 0) nrm2[0] = z;
    }
    __syncthreads();
    if (warp == 0) {
        double z = 0.0;
#pragma unroll
        for (int q = 0; q < LZ_THREADS / 32; ++q) z += red[q][lane];
        if (lane < 2 * nk) ((double*)(h + k0))[lane] = z;
        z = lane < 2 * nk ? fabs(z) : 0.0;
        for (int d = 16; d > 0; d >>= 1) z = fmax(z, __shfl_xor_sync(0xffffffffu, z, d));
        if (lane == 0) hmax[grp] = z;
    }
}

// The upper 24 bits of a double's significand as a float (0 below the normal floats), by its bits: a
// conversion would go through the FP64 pipe.
__device__ __forceinline__ float top_float(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned f = (__funnelshift_l(lo, hi, 3) - (896u << 23)) & 0x7fffffffu;
    return (hi & 0x7fffffffu) < (897u << 20) ? 0.f : __uint_as_float(f | (hi & 0x80000000u));
}
__device__ __forceinline__ float2 lz_top(const double2& v) { return make_float2(top_float(v.x), top_float(v.y)); }
__device__ __forceinline__ float2 lz_top(const float2& v) { return v; }

// w = w1 - alpha v - beta u - sum_k h_k V_k, beta_out = |w|; slot != null: alpha, beta_out and nrm2 for the
// host.  After the recurrence the projections are at the level of rounding errors (1e-15 |w1|), so the
// sum over k needs no more than a few digits beside w1: with hmax given and small enough for that
// (lz_single_precision: its error is then below 2^-54 |w1|), it is taken in single precision, with h scaled by a
// power of two near 1 / hmax; otherwise in FP64.  Basis vectors have elements of at most 1.
// At K = 90 on 112,720 rows: 88 us in FP64, 28 us so.
template <typename VT>
__global__ void __launch_bounds__(LZ_AXPY_THREADS, 8)
k_lz_correct(long long n, int K, const VT* V, long long ldv, const double2* h, const double* hmax, const double2* w1,
             const double2* v, const double2* u, const double* alpha, const double* beta, double2* w, double* partial,
             double* beta_out, const double* nrm2, double* slot, unsigned* ticket) {
    __shared__ double2 hs[LZ_CHUNK];
    __shared__ float2 hf[LZ_CHUNK];
    __shared__ double red[LZ_AXPY_THREADS / 32];
    __shared__ double sc[2];   // the scale of the single-precision sum and its inverse; 0: in FP64
    if (threadIdx.x == 0) {
        double big = 0.0;
        if (hmax)
            for (int g = 0; g < (K + LZ_G - 1) / LZ_G; ++g) big = fmax(big, hmax[g]);
        const bool ok = hmax && lz_single_precision(K, big, nrm2[0]);
        const int e = ok ? ilogb(big) : 0;
        sc[0] = ok ? scalbn(1.0, -e) : 0.0;
        sc[1] = scalbn(1.0, e);
    }
    __syncthreads();
    const double scale = sc[0];
    const bool single = __double2hiint(scale) != 0;
    const double a = v ? alpha[0] : 0.0, b = u ? beta[0] : 0.0;
    double nn = 0.0;
    for (long long i0 = (long long)blockIdx.x * LZ_AXPY_THREADS; i0 < n; i0 += (long long)gridDim.x * LZ_AXPY_THREADS) {
        const long long i = i0 + threadIdx.x;
        const bool act = i < n;
        double2 x = act ? w1[i] : make_double2(0.0, 0.0);
        if (v && act) {
            const double2 t = v[i];
            x.x = fma(-a, t.x, x.x);
            x.y = fma(-a, t.y, x.y);
        }
        if (u && act) {
            const double2 t = u[i];
            x.x = fma(-b, t.x, x.x);
            x.y = fma(-b, t.y, x.y);
        }
        for (int k0 = 0; k0 < K; k0 += LZ_CHUNK) {
            const int nk = min(LZ_CHUNK, K - k0);
            if (K > LZ_CHUNK || i0 == (long long)blockIdx.x * LZ_AXPY_THREADS) {
                __syncthreads();
                for (int k = threadIdx.x; k < nk; k += LZ_AXPY_THREADS) {
                    const double2 c = h[k0 + k];
                    hs[k] = c;
                    if (single) hf[k] = make_float2((float)(c.x * scale), (float)(c.y * scale));
                }
                __syncthreads();
            }
            if (!act) continue;
            const VT* Vk = V + (size_t)k0 * ldv + i;
            if (single) {
                float2 c = make_float2(0.f, 0.f);
                auto add = [&](const VT& t, int k) {
                    const float2 f = hf[k], u1 = lz_top(t);
                    c.x = fmaf(f.x, u1.x, c.x);
                    c.x = fmaf(-f.y, u1.y, c.x);
                    c.y = fmaf(f.x, u1.y, c.y);
                    c.y = fmaf(f.y, u1.x, c.y);
                };
                int k = 0;
                for (; k + 8 <= nk; k += 8) {   // eight loads in flight per thread
                    VT t[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) t[q] = __ldcs(Vk + (size_t)(k + q) * ldv);
#pragma unroll
                    for (int q = 0; q < 8; ++q) add(t[q], k + q);
                }
                for (; k < nk; ++k) add(Vk[(size_t)k * ldv], k);
                x.x = fma(-sc[1], (double)c.x, x.x);
                x.y = fma(-sc[1], (double)c.y, x.y);
                continue;
            }
#pragma unroll 8
            for (int k = 0; k < nk; ++k) {
                const double2 t = lz_load(Vk + (size_t)k * ldv), c = hs[k];
                x.x = fma(-c.x, t.x, x.x);
                x.x = fma(c.y, t.y, x.x);
                x.y = fma(-c.x, t.y, x.y);
                x.y = fma(-c.y, t.x, x.y);
            }
        }
        if (act) w[i] = x;
        nn = fma(x.x, x.x, fma(x.y, x.y, nn));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_sum = [&](double t) {
        for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
        __syncthreads();
        if (lane == 0) red[warp] = t;
        __syncthreads();
        t = 0.0;
        for (int q = 0; q < LZ_AXPY_THREADS / 32; ++q) t += red[q];
        return t;
    };
    nn = block_sum(nn);
    if (threadIdx.x == 0) partial[blockIdx.x] = nn;
    if (!last_block(ticket, gridDim.x)) return;
    double z = 0.0;
#pragma unroll 8
    for (int q = threadIdx.x; q < (int)gridDim.x; q += LZ_AXPY_THREADS) z += __ldcg(partial + q);
    z = block_sum(z);
    if (threadIdx.x == 0) {
        const double be = sqrt(z);
        beta_out[0] = be;
        beta_out[1] = 1.0 / be;
        if (slot) {
            slot[0] = alpha ? alpha[0] : 0.0;
            slot[1] = be;
            slot[2] = nrm2 ? nrm2[0] : z;
        }
    }
}

__global__ void k_normalize(long long n, const double2* w, const double* beta, double2* v, float2* v32) {
    const double inv = beta[1];   // 1 / beta, computed once (a division is a dozen FP64 instructions)
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double2 a = w[i];
        const double2 o = make_double2(a.x * inv, a.y * inv);
        v[i] = o;
        if (v32) v32[i] = make_float2((float)o.x, (float)o.y);
    }
}

__global__ void k_axpy_real(long long n, double a, const double2* x, double2* y) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double2 u = x[i];
        double2 v = y[i];
        v.x += a * u.x;
        v.y += a * u.y;
        y[i] = v;
    }
}

}  // namespace

void launch_random_c128(int64_t n, uint64_t seed, double* dst, cudaStream_t st) {
    if (n <= 0) return;
    k_random_c128<<<grid_for(n), 256, 0, st>>>(n, seed, (double2*)dst);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_c128_to_c64(int64_t n, const double* src, float* dst, cudaStream_t st) {
    if (n <= 0) return;
    k_c128_to_c64<<<grid_for(n), 256, 0, st>>>(n, (const double2*)src, (float2*)dst);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_c64_to_c128(int64_t n, const float* src, double* dst, int accumulate, cudaStream_t st) {
    if (n <= 0) return;
    k_c64_to_c128<<<grid_for(n), 256, 0, st>>>(n, (const float2*)src, (double2*)dst, accumulate);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_conj_c128(int64_t n, double* v, cudaStream_t st) {
    if (n <= 0) return;
    k_conj_c128<<<grid_for(n), 256, 0, st>>>(n, (double2*)v);
    EDGPU_CUDA(cudaGetLastError());
}

size_t dot_scratch_doubles() { return 2 * (size_t)RED_BLOCKS; }

void launch_norm2_c128(int64_t n, const double* a, double* scratch, double* out_dev, cudaStream_t st) {
    k_norm_stage1<<<RED_BLOCKS, RED_THREADS, 0, st>>>(n, (const double2*)a, (double2*)scratch);
    k_norm_stage2<<<1, 1024, 0, st>>>(RED_BLOCKS, (const double2*)scratch, out_dev);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_reduce_grad(int nblocks, int ncoupl, const double* partial, double* out_dev, cudaStream_t st) {
    if (ncoupl <= 0) return;
    k_reduce_grad<<<(ncoupl + 3) / 4, 128, 0, st>>>(nblocks, ncoupl, partial, out_dev);
    EDGPU_CUDA(cudaGetLastError());
}

static unsigned lz_correct_blocks(int64_t n) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + LZ_AXPY_THREADS - 1) / LZ_AXPY_THREADS, LZ_MAX_BLOCKS));
}

void launch_lanczos_alpha(int64_t n, const double* v, double* w, const float* y32, double* scratch, unsigned* tickets,
                          double* alpha_dev, cudaStream_t st) {
    const int64_t need = (n + LZ_THREADS - 1) / LZ_THREADS, most = (n < (1 << 20) ? 1ll : 4ll) * std::max(1, sm_count());
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(need, most));
    k_lz_alpha<<<blocks, LZ_THREADS, 0, st>>>(n, (const double2*)v, (double2*)w, (const float2*)y32, (double2*)scratch,
                                             alpha_dev, tickets);
    EDGPU_CUDA(cudaGetLastError());
}

template <typename VT, int... S>
static constexpr std::array<void (*)(long long, int, const VT*, long long, const double2*, const double2*, const double2*,
                                     const double*, const double*, double2*, double2*, double*, double*, unsigned*),
                            sizeof...(S)>
lz_project_table(std::integer_sequence<int, S...>) {
    return {k_lz_project<VT, S + 1>...};
}

void launch_lanczos_project(int64_t n, int k, const void* V, bool c64, int64_t ldv, const double* w, const double* v,
                            const double* u, const double* alpha_dev, const double* beta_dev, double* scratch,
                            unsigned* tickets, double* h_dev, double* hmax_dev, double* nrm2_dev, cudaStream_t st) {
    const int groups = lz_groups(k);
    const dim3 grid((unsigned)lz_row_blocks(n, groups, sm_count()), (unsigned)groups);
    auto go = [&](auto kern, auto* basis) {
        kern<<<grid, LZ_THREADS, 0, st>>>(n, k, basis, ldv, (const double2*)w, (const double2*)v, (const double2*)u,
                                          alpha_dev, beta_dev, (double2*)scratch, (double2*)h_dev, hmax_dev, nrm2_dev,
                                          tickets);
        EDGPU_CUDA(cudaGetLastError());
    };
    const int most = (k + groups - 1) / groups;   // vectors of the largest group
    auto pick = [&](auto* basis) {
        typedef typename std::remove_const<typename std::remove_pointer<decltype(basis)>::type>::type VT;
        static constexpr auto table = lz_project_table<VT>(std::make_integer_sequence<int, LZ_G>());
        go(table[most - 1], basis);
    };
    if (c64) pick((const float2*)V);
    else pick((const double2*)V);
}

void launch_lanczos_correct(int64_t n, int k, const void* V, bool c64, int64_t ldv, const double* h_dev,
                            const double* hmax_dev, const double* w1, const double* v, const double* u,
                            const double* alpha_dev, const double* beta_dev, double* w, double* scratch, unsigned* tickets, double* beta_out,
                            const double* nrm2_dev, double* slot, cudaStream_t st) {
    const dim3 grid(lz_correct_blocks(n));
    auto go = [&](auto* basis, auto kern) {
        kern<<<grid, LZ_AXPY_THREADS, 0, st>>>(n, k, basis, ldv, (const double2*)h_dev, hmax_dev, (const double2*)w1,
                                               (const double2*)v, (const double2*)u, alpha_dev, beta_dev, (double2*)w,
                                               scratch, beta_out, nrm2_dev, slot, tickets);
        EDGPU_CUDA(cudaGetLastError());
    };
    if (c64) go((const float2*)V, k_lz_correct<float2>);
    else go((const double2*)V, k_lz_correct<double2>);
}

void launch_normalize(int64_t n, const double* w, const double* beta_dev, double* v_next, float* v32, cudaStream_t st) {
    if (n <= 0) return;
    k_normalize<<<grid_for(n), 256, 0, st>>>(n, (const double2*)w, beta_dev, (double2*)v_next, (float2*)v32);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_axpy_real(int64_t n, double a, const double* x, double* y, cudaStream_t st) {
    if (n <= 0) return;
    k_axpy_real<<<grid_for(n), 256, 0, st>>>(n, a, (const double2*)x, (double2*)y);
    EDGPU_CUDA(cudaGetLastError());
}

}  // namespace edgpu
