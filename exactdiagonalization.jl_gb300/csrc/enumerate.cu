// Sector basis and representative enumeration on the GPU.
//
// Replaces hs_get_basis_list(::HilbertSpaceSector) (hilbert_space_representation.jl:127-206) and the
// representative sweep of symmetry_reduce (symmetry_reduce_generic.jl:22-106).  Candidates are
// scanned in increasing order, 1024 per warp (one bitmap word per thread, written coalesced);
// a predicate marks the kept ones, per-block popcounts are scanned into offsets, and a second pass
// regenerates the candidates and writes the kept ones in order: the output is sorted by
// construction.  Candidate sources:
//   RANGE  every word below 2^nbits (general sites: local-code validity + QN sum in the allowed set)
//   COMBO  every nbits-bit word with k set bits, by combinatorial unranking + Gosper's next-
//          combination step (spin-1/2 2Sz sectors; the parent basis then needs no predicate)
//   LIST   a materialised parent basis
#include <algorithm>
#include <cmath>
#include <memory>
#include <mutex>

#include "edgpu_internal.h"
#include "edgpu_device.cuh"

namespace edgpu {

namespace {

constexpr int ENUM_THREADS = 256;

unsigned long long* binomial_table() {
    // C(i, j) for 0 <= i, j <= 64 (row stride 65); C(64, 32) < 2^63 so no entry overflows.
    static unsigned long long* d_tab = nullptr;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (!d_tab) {
        std::vector<unsigned long long> h(65 * 65, 0ull);
        for (int i = 0; i <= 64; ++i) {
            h[i * 65] = 1;
            for (int j = 1; j <= i; ++j) h[i * 65 + j] = h[(i - 1) * 65 + j - 1] + (j <= i - 1 ? h[(i - 1) * 65 + j] : 0ull);
        }
        EDGPU_CUDA(cudaMalloc(&d_tab, h.size() * sizeof(unsigned long long)));
        EDGPU_CUDA(cudaMemcpy(d_tab, h.data(), h.size() * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    }
    return d_tab;
}

unsigned long long host_binom(int n, int k) {
    if (k < 0 || k > n) return 0;
    unsigned long long r = 1;
    for (int i = 1; i <= k; ++i) r = r * (unsigned long long)(n - k + i) / (unsigned long long)i;
    return r;
}

template <typename W>
__device__ __forceinline__ int ctz_w(W v);
template <>
__device__ __forceinline__ int ctz_w<uint32_t>(uint32_t v) { return __ffs((int)v) - 1; }
template <>
__device__ __forceinline__ int ctz_w<unsigned long long>(unsigned long long v) { return __ffsll((long long)v) - 1; }

// Colex unranking: the rank-r word with k set bits among n (rank order == numeric order).
template <typename W>
__device__ __forceinline__ W unrank_combo(unsigned long long r, int n, int k, const unsigned long long* C) {
    W v = 0;
    int c = n;
    for (int i = k; i >= 1; --i) {
        do { --c; } while (C[c * 65 + i] > r);
        v |= (W)1 << c;
        r -= C[c * 65 + i];
    }
    return v;
}

// Next word with the same popcount (Gosper).
template <typename W>
__device__ __forceinline__ W gosper_next(W v) {
    const W t = v | (v - 1);
    return (W)((t + 1) | (((~t & (t + 1)) - 1) >> (ctz_w<W>(v) + 1)));
}

enum { SRC_RANGE = 0, SRC_COMBO = 1, SRC_LIST = 2 };

struct EnumParams {
    int src;
    long long total;
    int n, k;
    const unsigned long long* C;
    const void* list;
    int list_w32;
    int check_sector;
    SectorDev sec;
    int check_rep;
    GroupDev grp;
    unsigned* bitmap;
    long long* block_counts;
    long long* block_offsets;
    void* out;
};

template <typename W>
__device__ __forceinline__ bool sector_ok(W s, const SectorDev& d) {
    long long acc[4] = {0, 0, 0, 0};
    for (int i = 0; i < d.n_sites; ++i) {
        const int c = (int)((s >> d.off[i]) & (W)(((W)1 << d.bw[i]) - 1));
        if (c >= d.dims[i]) return false;
        const long long* q = d.qn + (size_t)(d.qbase[i] + c) * d.qlen;
        for (int k = 0; k < d.qlen; ++k) acc[k] += q[k];
    }
    if (d.all_sectors) return true;
    for (int a = 0; a < d.n_allowed; ++a) {
        bool m = true;
        for (int k = 0; k < d.qlen; ++k) m = m && (d.allowed[a * d.qlen + k] == acc[k]);
        if (m) return true;
    }
    return false;
}

// Stages the row-rotation masks of a torus group in shared memory (keep[64]); the block synchronises.
template <typename W>
__device__ __forceinline__ void stage_keep(W* keep, const GroupDev& g) {
    if (threadIdx.x < 64) keep[threadIdx.x] = g.kind == GK_TORUS && (int)threadIdx.x < g.L1 ? (W)g.keep[threadIdx.x] : (W)0;
    __syncthreads();
}

// A ring of 1-bit (or wider) sites in a 32-bit word, whose rotations are funnel shifts.
template <typename W>
__device__ __forceinline__ bool ring32(const GroupDev& g) {
    return sizeof(W) == 4 && g.kind == GK_TORUS && g.L2 == 1 && g.nbits <= 31;
}

// Whether a rotation other than the identity leaves the ring state q unchanged: then one by L1 / p sites
// does, p a prime divisor of L1.
__device__ __forceinline__ bool ring_periodic(unsigned q, const GroupDev& g) {
    const unsigned full = (unsigned)g.full;
    int m = g.L1;
    for (int p = 2; p * p <= m; ++p) {
        if (m % p) continue;
        const int s = g.L1 / p * g.w;
        if ((((q << s) | (q >> (g.nbits - s))) & full) == q) return true;
        while (m % p == 0) m /= p;
    }
    if (m > 1 && g.L1 > 1) {
        const int s = g.L1 / m * g.w;
        if (s < g.nbits ? (((q << s) | (q >> (g.nbits - s))) & full) == q : false) return true;
    }
    return false;
}

template <typename W>
__device__ __forceinline__ bool rep_ok(W s, const GroupDev& g, const W* keep) {
    if (ring32<W>(g)) {
        // the smallest rotation by unrolled shifts, two instructions each; the characters on the
        // stabiliser only for a representative that has one
        unsigned rep;
        int e;
        canon_ring((unsigned)s, g.nbits, g.L1, g.w, 0, false, rep, e);
        if (rep != (unsigned)s) return false;
        return !ring_periodic((unsigned)s, g) ||
               is_rep_torus<W>(s, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, g.num);
    }
    if (g.kind == GK_TORUS) return is_rep_torus<W>(s, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, g.num);
    if (g.kind == GK_GENERIC) {
        for (int e = 1; e < g.G; ++e) {
            W t = 0;
            const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
            for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((s >> (4 * c)) & 15u)];
            t ^= (W)g.flips[e];
            if (t < s) return false;
            if (t == s && g.num[e] != 0) return false;
        }
        return true;
    }
    return true;
}

template <typename W>
__device__ __forceinline__ W first_candidate(const EnumParams& p, long long r0) {
    if (p.src == SRC_RANGE) return (W)r0;
    if (p.src == SRC_COMBO) return unrank_combo<W>((unsigned long long)r0, p.n, p.k, p.C);
    return p.list_w32 ? (W)((const unsigned*)p.list)[r0] : (W)((const unsigned long long*)p.list)[r0];
}

template <typename W>
__device__ __forceinline__ W next_candidate(const EnumParams& p, W v, long long r) {
    if (p.src == SRC_RANGE) return (W)(v + 1);
    if (p.src == SRC_COMBO) return gosper_next<W>(v);
    return p.list_w32 ? (W)((const unsigned*)p.list)[r] : (W)((const unsigned long long*)p.list)[r];
}

// Bit j of bitmap word t: candidate 32 t + j is kept.  A listed candidate is read by the lane that tests
// it, 32 neighbours at a time (a word is a ballot); the others are generated one after the other.  Bound by
// the rotations' instructions: 10.4 million states of the chain L = 26 take 66 us, 212 with 32 consecutive
// states per thread, rotations in a loop and the masks in local memory.
template <typename W>
__global__ void __launch_bounds__(ENUM_THREADS) k_mark(EnumParams p) {
    __shared__ long long tmp[32];
    __shared__ W keep[64];
    if (p.check_rep) stage_keep<W>(keep, p.grp);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long r0 = t * 32;
    unsigned word = 0;
    if (p.src == SRC_LIST) {
        const int lane = threadIdx.x & 31;
        const long long w0 = (t - lane) * 32;   // the warp's 1024 candidates
#pragma unroll 2
        for (int j = 0; j < 32; ++j) {
            const long long r = w0 + 32 * j + lane;
            bool ok = r < p.total;
            if (ok) {
                const W v = first_candidate<W>(p, r);
                if (p.check_sector) ok = sector_ok<W>(v, p.sec);
                if (ok && p.check_rep) ok = rep_ok<W>(v, p.grp, keep);
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (lane == j) word = m;
        }
        if (r0 < p.total) p.bitmap[t] = word;
    } else if (r0 < p.total) {
        const int cnt = (int)min(32LL, p.total - r0);
        W v = first_candidate<W>(p, r0);
        for (int j = 0; j < cnt; ++j) {
            bool ok = true;
            if (p.check_sector) ok = sector_ok<W>(v, p.sec);
            if (ok && p.check_rep) ok = rep_ok<W>(v, p.grp, keep);
            if (ok) word |= 1u << j;
            if (j + 1 < cnt) v = next_candidate<W>(p, v, r0 + j + 1);
        }
        p.bitmap[t] = word;
    }
    long long tot = 0;
    block_exclusive_scan((long long)__popc(word), tmp, &tot);
    if (threadIdx.x == 0) p.block_counts[blockIdx.x] = tot;
}

__global__ void k_scan_counts(const long long* counts, long long n, long long* offsets, long long* total) {
    __shared__ long long tmp[32];
    const long long per = (n + blockDim.x - 1) / blockDim.x;
    const long long beg = min(n, (long long)threadIdx.x * per), end = min(n, beg + per);
    long long s = 0;
    for (long long i = beg; i < end; ++i) s += counts[i];
    long long tot = 0;
    long long ex = block_exclusive_scan(s, tmp, &tot);
    for (long long i = beg; i < end; ++i) {
        offsets[i] = ex;
        ex += counts[i];
    }
    if (threadIdx.x == 0) *total = tot;
}

template <typename W>
__global__ void __launch_bounds__(ENUM_THREADS) k_compact(EnumParams p) {
    __shared__ long long tmp[32];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long r0 = t * 32;
    const unsigned word = (r0 < p.total) ? p.bitmap[t] : 0u;
    long long pos = block_exclusive_scan((long long)__popc(word), tmp, nullptr) + p.block_offsets[blockIdx.x];
    if (word) {
        const int cnt = (int)min(32LL, p.total - r0);
        W v = first_candidate<W>(p, r0);
        W* out = (W*)p.out;
        for (int j = 0; j < cnt; ++j) {
            if ((word >> j) & 1u) out[pos++] = v;
            if (j + 1 < cnt) v = next_candidate<W>(p, v, r0 + j + 1);
        }
    }
}

// The words of a popcount, ascending: a thread unranks one in sixteen, the block writes them in order
// (10.4 million words: 30 us, 81 with each thread writing its own run).
constexpr int COMBO_RUN = 16;
template <typename W>
__global__ void __launch_bounds__(256) k_combo_write(long long total, int n, int k, const unsigned long long* C, W* out) {
    __shared__ W st[256 * COMBO_RUN + 256 * COMBO_RUN / 32];   // (one word in 33 spare: no bank conflicts)
    const long long base = (long long)blockIdx.x * (256 * COMBO_RUN);
    const long long i0 = base + (long long)threadIdx.x * COMBO_RUN;
    W v = i0 < total ? unrank_combo<W>((unsigned long long)i0, n, k, C) : (W)0;
#pragma unroll
    for (int j = 0; j < COMBO_RUN; ++j) {
        const int at = threadIdx.x * COMBO_RUN + j;
        st[at + at / 32] = v;
        if (i0 + j + 1 < total) v = gosper_next<W>(v);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < COMBO_RUN; ++j) {
        const int at = j * 256 + threadIdx.x;
        if (base + at < total) out[base + at] = st[at + at / 32];
    }
}

// Device copies of the sector definition for the RANGE predicate.
struct SectorBuffers {
    SectorDev dev{};
    std::vector<void*> ptrs;
    template <typename T>
    const T* put(const std::vector<T>& v) {
        if (v.empty()) return nullptr;
        void* d = nullptr;
        EDGPU_CUDA(cudaMalloc(&d, v.size() * sizeof(T)));
        ptrs.push_back(d);
        EDGPU_CUDA(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
        return (const T*)d;
    }
    explicit SectorBuffers(const Layout& lay) {
        std::vector<int32_t> qbase(lay.n_sites);
        int acc = 0;
        for (int i = 0; i < lay.n_sites; ++i) { qbase[i] = acc; acc += lay.dims[i]; }
        std::vector<long long> qn(lay.state_qn.begin(), lay.state_qn.end());
        std::vector<long long> al(lay.allowed.begin(), lay.allowed.end());
        dev.n_sites = lay.n_sites;
        dev.qlen = lay.qlen;
        dev.n_allowed = lay.qlen ? (int)(lay.allowed.size() / lay.qlen) : 0;
        dev.all_sectors = lay.all_sectors ? 1 : 0;
        dev.off = put(lay.off);
        dev.bw = put(lay.bw);
        dev.dims = put(lay.dims);
        dev.qbase = put(qbase);
        dev.qn = put(qn);
        dev.allowed = put(al);
    }
    ~SectorBuffers() {
        for (void* p : ptrs) cudaFree(p);
    }
};

template <typename W>
int64_t run_filtered(EnumParams p, void** out_keys, bool write, cudaStream_t st) {
    const long long n_words = (p.total + 31) / 32;
    const long long n_blocks = (n_words + ENUM_THREADS - 1) / ENUM_THREADS;
    if (n_blocks > 0x7fffffffLL) throw Error(EDGPU_ERR_ARG, "enumeration too large");
    // one allocation: block counts, block offsets, the total, the bitmap
    long long* d_counts = nullptr;
    int64_t total = 0;
    try {
        EDGPU_CUDA(cudaMalloc(&d_counts, (size_t)(2 * n_blocks + 1) * sizeof(long long) + (size_t)n_words * sizeof(unsigned)));
        long long* d_offsets = d_counts + n_blocks;
        long long* d_total = d_offsets + n_blocks;
        unsigned* d_bitmap = (unsigned*)(d_total + 1);
        p.bitmap = d_bitmap;
        p.block_counts = d_counts;
        p.block_offsets = d_offsets;
        if (n_blocks > 0) {
            k_mark<W><<<(unsigned)n_blocks, ENUM_THREADS, 0, st>>>(p);
            EDGPU_CUDA(cudaGetLastError());
            k_scan_counts<<<1, 1024, 0, st>>>(d_counts, n_blocks, d_offsets, d_total);
            EDGPU_CUDA(cudaGetLastError());
            long long h_total = 0;
            EDGPU_CUDA(cudaMemcpyAsync(&h_total, d_total, sizeof(long long), cudaMemcpyDeviceToHost, st));
            EDGPU_CUDA(cudaStreamSynchronize(st));
            total = h_total;
        }
        if (write) {
            void* keys = nullptr;
            EDGPU_CUDA(cudaMalloc(&keys, std::max<int64_t>(total, 1) * sizeof(W)));
            p.out = keys;
            if (total > 0) {
                k_compact<W><<<(unsigned)n_blocks, ENUM_THREADS, 0, st>>>(p);
                cudaError_t e = cudaGetLastError();
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) {
                    cudaFree(keys);
                    throw Error(EDGPU_ERR_CUDA, std::string("k_compact: ") + cudaGetErrorString(e));
                }
            }
            *out_keys = keys;
        }
    } catch (...) {
        cudaFree(d_counts);
        throw;
    }
    cudaFree(d_counts);
    return total;
}

template <typename W>
void enumerate_parent_t(Space& s, cudaStream_t st) {
    const Layout& lay = s.lay;
    if (lay.popcount >= 0) {
        const long long total = (long long)host_binom(lay.nbits, lay.popcount);
        s.dim = total;
        if (s.lazy) return;
        EDGPU_CUDA(cudaMalloc(&s.d_keys, std::max<long long>(total, 1) * sizeof(W)));
        if (total > 0) {
            const long long blocks = (total + 256 * COMBO_RUN - 1) / (256 * COMBO_RUN);
            k_combo_write<W><<<(unsigned)blocks, 256, 0, st>>>(total, lay.nbits, lay.popcount, binomial_table(),
                                                              (W*)s.d_keys);
            EDGPU_CUDA(cudaGetLastError());
            EDGPU_CUDA(cudaStreamSynchronize(st));
        }
        return;
    }
    if (lay.nbits > 34)
        throw Error(EDGPU_ERR_ARG, "sector enumeration over a generic site layout is limited to 34 bits "
                                   "(spin-1/2 single-sector spaces have no limit)");
    SectorBuffers sb(lay);
    EnumParams p{};
    p.src = SRC_RANGE;
    p.total = 1LL << lay.nbits;
    p.check_sector = 1;
    p.sec = sb.dev;
    p.check_rep = 0;
    s.dim = run_filtered<W>(p, &s.d_keys, !s.lazy, st);
}

// key = (state << sb) | index of the stabiliser size among the divisors of G
template <typename W>
__global__ void k_embed(W* keys, long long n, int sb, GroupDev g, const int32_t* divi) {
    __shared__ W keep[64];
    stage_keep<W>(keep, g);
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const W q = keys[i];
    int stab = 1;
    if (g.kind == GK_TORUS) {
        W rep;
        int gb;
        canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, false, true, rep, gb, stab);
    } else if (g.kind == GK_GENERIC) {
        stab = 0;
        for (int e = 0; e < g.G; ++e) {
            W t = 0;
            const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
            for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
            t ^= (W)g.flips[e];
            stab += (t == q);
        }
    }
    keys[i] = (W)((q << sb) | (W)divi[stab]);
}

template <typename W>
void enumerate_reps_t(Space& red, const Space& parent, cudaStream_t st) {
    const Layout& lay = parent.lay;
    GroupBuffers gb;
    gb.upload(red.group, lay);
    EnumParams p{};
    p.check_rep = 1;
    p.grp = gb.dev;
    if (parent.d_keys) {
        p.src = SRC_LIST;
        p.list = parent.d_keys;
        p.list_w32 = parent.w32 ? 1 : 0;
        p.total = parent.dim;
        red.dim = run_filtered<W>(p, &red.d_keys, true, st);
    } else if (lay.popcount >= 0) {
        p.src = SRC_COMBO;
        p.total = (long long)host_binom(lay.nbits, lay.popcount);
        p.n = lay.nbits;
        p.k = lay.popcount;
        p.C = binomial_table();
        red.dim = run_filtered<W>(p, &red.d_keys, true, st);
    } else {
        if (lay.nbits > 34) throw Error(EDGPU_ERR_ARG, "lazy generic sector limited to 34 bits");
        SectorBuffers sb(lay);
        p.src = SRC_RANGE;
        p.total = 1LL << lay.nbits;
        p.check_sector = 1;
        p.sec = sb.dev;
        red.dim = run_filtered<W>(p, &red.d_keys, true, st);
    }
    if (red.sb > 0 && red.dim > 0) {
        k_embed<W><<<(unsigned)((red.dim + 255) / 256), 256, 0, st>>>((W*)red.d_keys, red.dim, red.sb, gb.dev, gb.divi);
        EDGPU_CUDA(cudaGetLastError());
        EDGPU_CUDA(cudaStreamSynchronize(st));
    }
}

// basis_mapping_index / basis_mapping_amplitude for every parent word: orbit minimum, its index in
// the representative table (-1 when the orbit is incompatible), chi(h)/sqrt(|O|) with h.p = rep.
template <typename W, typename PW>
__global__ void k_mapping(const PW* parent, long long n_parent, const W* reps, long long n_reps, int sb, GroupDev g,
                          const double2* phase, long long* index_out, double2* ampl_out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_parent) return;
    const W q = (W)parent[i];
    W rep = q;
    int gb = 0, stab = 1;
    if (g.kind == GK_TORUS) {
        W keep[64];
        for (int a = 0; a < g.L1; ++a) keep[a] = (W)g.keep[a];
        canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, true, true, rep, gb, stab);
    } else if (g.kind == GK_GENERIC) {
        rep = q; gb = 0; stab = 0;
        for (int e = 0; e < g.G; ++e) {
            W t = 0;
            const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
            for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
            t ^= (W)g.flips[e];
            if (t < rep) { rep = t; gb = e; }
            stab += (t == q);
        }
    }
    const long long c = key_find<W>(reps, n_reps, rep, sb, nullptr);
    index_out[i] = c;
    double2 a = make_double2(0.0, 0.0);
    if (c >= 0) {
        const double s = sqrt((double)stab / (double)g.G);
        const double2 ph = phase[g.num[gb]];
        a = make_double2(ph.x * s, ph.y * s);
    }
    ampl_out[i] = a;
}

template <typename W>
__global__ void k_orbit_sizes(const W* reps, long long n, int sb, GroupDev g, int32_t* out) {
    __shared__ W keep[64];
    stage_keep<W>(keep, g);
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const W q = reps[i] >> sb;
    int stab = 1;
    if (g.kind == GK_TORUS) {
        W rep;
        int gb;
        canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, false, true, rep, gb, stab);
    } else if (g.kind == GK_GENERIC) {
        stab = 0;
        for (int e = 0; e < g.G; ++e) {
            W t = 0;
            const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
            for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
            t ^= (W)g.flips[e];
            stab += (t == q);
        }
    }
    out[i] = g.G / stab;
}

template <typename W>
__global__ void k_lookup(const W* keys, long long n, int sb, const unsigned long long* q, long long m, long long* out,
                         unsigned long long smax) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const unsigned long long k = q[i];
    out[i] = (k > smax) ? -1 : key_find<W>(keys, n, (W)k, sb, nullptr);
}

template <typename W>
__global__ void k_get_states(const W* keys, long long n, int sb, unsigned long long* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (unsigned long long)(keys[i] >> sb);
}

// Bucket width of a search directory: for every candidate shift s in [s_lo, s_lo + n_shift) count
// the keys whose bucket (state >> s) holds at most K(s) keys, K(s) = min(4, 28 / (s + sb)) (the keys
// a bucket summary can carry).  A bucket holds more than K keys exactly when some K+1 consecutive
// keys around key i share its bucket.
// Two keys share a bucket of width 2^s exactly when their difference has at most s bits, so a window's lane
// needs one difference per K; which keys lie in a shared window follows from a ballot's bits.  A warp
// loads 32 keys, SURVEY_LOADS groups ahead, and counts the middle 24 (bound by the latency of the loads
// and the instructions per shift: 10.4 million keys, two shifts, 61 us; 92 with every thread comparing all
// windows at each shift).
constexpr int SURVEY_RUN = 8, SURVEY_LOADS = 4;   // 24-key groups per warp and load phase, load phases

template <typename W>
__global__ void __launch_bounds__(256) k_dir_survey(const W* keys, long long n, int sb, int s_lo, int n_shift,
                                                    unsigned long long* counts) {
    __shared__ unsigned part[64];
    __shared__ int members[64];   // K of shift s_lo + j
    if (threadIdx.x < 64) {
        const int mb = s_lo + (int)threadIdx.x + sb;
        part[threadIdx.x] = 0u;
        members[threadIdx.x] = mb == 0 ? 4 : min(4, 28 / mb);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long g0 = ((long long)blockIdx.x * 8 + threadIdx.x / 32) * SURVEY_RUN;
    unsigned mine[2] = {0u, 0u};   // counts of shifts s_lo + lane and s_lo + lane + 32
#pragma unroll 1
    for (int c = 0; c < SURVEY_RUN; c += SURVEY_LOADS) {
        W v[SURVEY_LOADS];
#pragma unroll
        for (int h = 0; h < SURVEY_LOADS; ++h) {   // the lane's window starts at key w and, as a key, is key w
            const long long w = (g0 + c + h) * 24 - 4 + lane;
            v[h] = w >= 0 && w < n ? (W)(keys[w] >> sb) : (W)0;
        }
#pragma unroll
        for (int h = 0; h < SURVEY_LOADS; ++h) {
            const long long w0 = (g0 + c + h) * 24 - 4, w = w0 + lane;
            const bool inner = w0 >= 0 && w0 + 36 <= n;   // every window of the warp lies in the table
            if (w0 + 4 >= n) break;
            const unsigned valid = inner ? 0x0ffffff0u : __ballot_sync(0xffffffffu, lane >= 4 && lane < 28 && w < n);
            int K = -1, len = 0;   // bits of the difference of the window's ends (64: no window)
            for (int j = 0; j < n_shift; ++j) {
                if (members[j] != K) {
                    // (K = 0: buckets too wide for any member; a window of one key is always shared)
                    K = members[j];
                    const W x = v[h] ^ __shfl_down_sync(0xffffffffu, v[h], K);
                    len = sizeof(W) == 8 ? 64 - __clzll((long long)x) : 32 - __clz((int)x);
                    if (!inner && (w < 0 || w + K >= n)) len = 64;
                }
                const unsigned f = __ballot_sync(0xffffffffu, len <= s_lo + j);
                unsigned bad = f;
                if (K == 4) {
                    bad |= bad << 1;
                    bad |= bad << 2;
                    bad |= f << 4;
                } else {
                    for (int d = 1; d <= K; ++d) bad |= f << d;
                }
                const unsigned cnt = __popc(valid & ~bad);
                if (lane == (j & 31)) mine[j >> 5] += cnt;
            }
        }
    }
    if (mine[0]) atomicAdd(&part[lane], mine[0]);
    if (mine[1]) atomicAdd(&part[lane + 32], mine[1]);
    __syncthreads();
    if ((int)threadIdx.x < n_shift && part[threadIdx.x]) atomicAdd(&counts[threadIdx.x], (unsigned long long)part[threadIdx.x]);
}

// Search directory, one entry per bucket b in [0, nb) plus the sentinel dir[nb] = n:
// dir[b] = start | min(count, 15) << 32 | the low mb bits of each key << (36 + k*mb) when the bucket
// holds at most K keys (start = index of the bucket's first key, or of the next key when empty).
// A block builds DIR_CHUNK consecutive buckets, DIR_STEP at a time: the keys from the step's first on are
// staged in shared memory (one search in the table per block), counted by bucket, the counts scanned into
// starts, and neighbouring threads write neighbouring entries.  Bound by instructions: 33.5 million buckets of
// 10.4 million keys (chain L = 26) take 90 us, 180 with a thread per 128 buckets, whose writes lay 1 KB apart
// within a warp.  stats[0] receives the largest bucket and
// stats[1] the number of keys answered by their bucket summary.
constexpr int DIR_STEP = 2048, DIR_TILE = 4096, DIR_CHUNK = 4 * DIR_STEP;

template <typename W>
__global__ void __launch_bounds__(256) k_dir_build(const W* keys, long long n, int sb, int shift, long long nb, int mb,
                                                   int K, unsigned long long* dir, unsigned long long* stats) {
    constexpr int E = DIR_STEP / 256;
    __shared__ W tile[DIR_TILE];
    __shared__ unsigned cell[DIR_STEP + 256];   // bucket r's count, then start | count << 16, at r + r / E
    __shared__ unsigned sums[8];
    const unsigned mbmask = mb >= 32 ? ~0u : (1u << mb) - 1u;   // (a summary's fields have 28 bits at most)
    auto bucket = [&](W key) { return (long long)((unsigned long long)(key >> sb) >> shift); };
    // first of the m keys at k with a bucket >= b
    auto lower = [&](const W* k, long long m, long long b) {
        long long lo = 0;
        while (m > 0) {
            const long long half = m >> 1;
            if (bucket(k[lo + half]) < b) {
                lo += half + 1;
                m -= half + 1;
            } else {
                m = half;
            }
        }
        return lo;
    };
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned mx = 0u, inl = 0u;
    const long long c0 = (long long)blockIdx.x * DIR_CHUNK, c1 = min(c0 + DIR_CHUNK, nb);
    long long cur = lower(keys, n, c0), b1;   // the step's first key and the end of its buckets, alike in all threads
    for (long long b0 = c0; b0 < c1; b0 = b1) {
        b1 = min(b0 + DIR_STEP, c1);
        const int have = (int)min((long long)DIR_TILE, n - cur);
        __syncthreads();
        for (int i = threadIdx.x; i < have; i += 256) tile[i] = keys[cur + i];
#pragma unroll
        for (int j = 0; j < E + 1; ++j) cell[j * 256 + threadIdx.x] = 0u;
        __syncthreads();
        if (cur + have < n) {
            const long long last = bucket(tile[have - 1]);
            if (last == b0) {
                // one bucket fills the tile: count it in the table
                const long long m = lower(keys + cur, n - cur, b0 + 1);
                if (threadIdx.x == 0) {
                    mx = max(mx, (unsigned)m);
                    dir[b0] = (unsigned long long)cur | (15ull << 32);   // (more than K keys: no members)
                }
                cur += m;
                b1 = b0 + 1;
                continue;
            }
            b1 = min(b1, last);   // the buckets before the last key's are whole
        }
        const unsigned nbk = (unsigned)(b1 - b0);
        for (int i = threadIdx.x; i < have; i += 256) {
            const W r = (W)((W)(tile[i] >> sb) >> shift) - (W)b0;
            if (r < nbk) atomicAdd(&cell[(unsigned)r + (unsigned)r / E], 1u);
        }
        __syncthreads();
        unsigned c[E], sum = 0;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            c[j] = cell[threadIdx.x * (E + 1) + j];
            sum += c[j];
        }
        unsigned inc = sum;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += o;
        }
        if (lane == 31) sums[wid] = inc;
        __syncthreads();
        unsigned at = inc - sum, all = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned o = sums[j];
            if (j < wid) at += o;
            all += o;
        }
#pragma unroll
        for (int j = 0; j < E; ++j) {
            cell[threadIdx.x * (E + 1) + j] = at | (c[j] << 16);
            at += c[j];
        }
        __syncthreads();
#pragma unroll 2
        for (unsigned r = threadIdx.x; r < nbk; r += 256) {
            const unsigned v = cell[r + r / E], first = v & 0xffffu, cnt = v >> 16;
            unsigned hi = min(cnt, 15u);   // the entry's upper word; the start is its lower one
            if ((int)cnt <= K) {
                for (unsigned k = 0; k < cnt; ++k) hi |= ((unsigned)tile[first + k] & mbmask) << (4 + (int)k * mb);
                inl += cnt;
            }
            mx = max(mx, cnt);
            dir[b0 + r] = (unsigned long long)((unsigned)cur + first) | ((unsigned long long)hi << 32);
        }
        cur += all;
    }
    if (c1 == nb && threadIdx.x == 0) dir[nb] = (unsigned long long)n;
    for (int d = 16; d > 0; d >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
        inl += __shfl_xor_sync(0xffffffffu, inl, d);
    }
    if ((threadIdx.x & 31) == 0) {
        if (mx > 1) atomicMax(stats, mx);
        if (inl) atomicAdd(stats + 1, inl);
    }
}

template <typename W>
__global__ void k_count_nnz(const W* keys, long long n, int sb, GroupDev g, int T, const unsigned long long* masks,
                            const unsigned long long* rows, const unsigned long long* flips,
                            unsigned long long* counts /* [0] targets, [1] found */) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long nt = 0, nf = 0;
    if (r < n) {
        const W b = keys[r] >> sb;
        for (int t = 0; t < T; ++t) {
            if ((b & (W)masks[t]) != (W)rows[t]) continue;
            const W q = b ^ (W)flips[t];
            ++nt;
            W rep = q;
            int gb = 0, stab = 1;
            if (g.kind == GK_TORUS) {
                W keep[64];
                for (int a = 0; a < g.L1; ++a) keep[a] = (W)g.keep[a];
                canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, false, false, rep, gb, stab);
            } else if (g.kind == GK_GENERIC) {
                for (int e = 0; e < g.G; ++e) {
                    W tt = 0;
                    const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
                    for (int c = 0; c < g.nchunks; ++c) tt |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
                    tt ^= (W)g.flips[e];
                    if (tt < rep) rep = tt;
                }
            }
            nf += (key_find<W>(keys, n, rep, sb, nullptr) >= 0);
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        nt += __shfl_down_sync(0xffffffffu, nt, d);
        nf += __shfl_down_sync(0xffffffffu, nf, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(counts, nt);
        atomicAdd(counts + 1, nf);
    }
}

template <typename W>
void count_nnz_t(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const uint64_t* flips,
                 int64_t* n_targets, int64_t* n_found, cudaStream_t st) {
    GroupBuffers gb;
    gb.upload(s.group, s.lay);
    unsigned long long* d = nullptr;
    const size_t tb = std::max(T, 1) * sizeof(unsigned long long);
    EDGPU_CUDA(cudaMalloc(&d, 3 * tb + 2 * sizeof(unsigned long long)));
    unsigned long long* dm = d;
    unsigned long long* dr = d + std::max(T, 1);
    unsigned long long* df = d + 2 * std::max(T, 1);
    unsigned long long* dc = d + 3 * std::max(T, 1);
    cudaError_t e = cudaSuccess;
    unsigned long long h[2] = {0, 0};
    if (T > 0) e = cudaMemcpyAsync(dm, masks, T * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && T > 0) e = cudaMemcpyAsync(dr, rows, T * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && T > 0) e = cudaMemcpyAsync(df, flips, T * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(dc, 0, 2 * sizeof(unsigned long long), st);
    if (e == cudaSuccess && s.dim > 0) {
        k_count_nnz<W><<<(unsigned)((s.dim + 255) / 256), 256, 0, st>>>((const W*)s.d_keys, s.dim, s.sb, gb.dev, T, dm, dr, df, dc);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, dc, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("count_nnz: ") + cudaGetErrorString(e));
    *n_targets = (int64_t)h[0];
    *n_found = (int64_t)h[1];
}

}  // namespace

// ---- host side ----------------------------------------------------------------------------------

std::vector<unsigned long long> torus_keep_masks(const Group& g, int nbits) {
    const int rowbits = g.L1 * g.w;
    std::vector<unsigned long long> keep(g.L1);
    for (int a = 0; a < g.L1; ++a) {
        const int s = a * g.w;
        const unsigned long long row_keep = (rowbits - s >= 64) ? ~0ull : ((1ull << (rowbits - s)) - 1ull);
        unsigned long long m = 0;
        for (int r = 0; r < g.L2; ++r) m |= row_keep << (r * rowbits);
        keep[a] = m;
    }
    (void)nbits;
    return keep;
}

std::vector<unsigned long long> generic_luts(const Group& g, const Layout& lay, int* nchunks) {
    const int nc = (lay.nbits + 3) / 4;
    *nchunks = nc;
    std::vector<unsigned long long> lut((size_t)g.G * nc * 16, 0ull);
    for (int e = 0; e < g.G; ++e) {
        const int32_t* map = g.maps.data() + (size_t)e * lay.n_sites;
        for (int c = 0; c < nc; ++c) {
            for (int v = 0; v < 16; ++v) {
                const unsigned long long word = (unsigned long long)v << (4 * c);
                unsigned long long out = 0;
                for (int i = 0; i < lay.n_sites; ++i) {
                    const unsigned long long m = (lay.bw[i] >= 64) ? ~0ull : ((1ull << lay.bw[i]) - 1ull);
                    out |= ((word >> lay.off[i]) & m) << lay.off[map[i]];
                }
                lut[((size_t)e * nc + c) * 16 + v] = out;
            }
        }
    }
    return lut;
}

void GroupBuffers::upload(const Group& g, const Layout& lay) {
    release();
    dev = GroupDev{};
    dev.kind = g.kind;
    dev.G = g.G;
    dev.den = g.den;
    dev.L1 = g.L1;
    dev.L2 = g.L2;
    dev.w = g.w;
    dev.rowbits = g.L1 * g.w;
    dev.nbits = lay.nbits;
    dev.full = (lay.nbits >= 64) ? ~0ull : ((1ull << lay.nbits) - 1ull);
    // one allocation: 64-bit tables, then the character numerators and divisor indices
    std::vector<unsigned long long> h;
    size_t o_flips = 0;
    if (g.kind == GK_TORUS) {
        h = torus_keep_masks(g, lay.nbits);
    } else if (g.kind == GK_GENERIC) {
        int nc = 0;
        h = generic_luts(g, lay, &nc);
        dev.nchunks = nc;
        o_flips = h.size();
        h.insert(h.end(), g.flips.begin(), g.flips.end());
        h.resize(o_flips + g.G, 0ull);
    }
    const size_t o_num = h.size();
    h.resize(o_num + (g.num.size() + 1) / 2 + 1, 0ull);
    memcpy(h.data() + o_num, g.num.data(), g.num.size() * sizeof(int32_t));
    const size_t o_divi = h.size();
    std::vector<int32_t> di(g.G + 1, 0);
    for (int d = 1, k = 0; d <= g.G; ++d)
        if (g.G % d == 0) di[d] = k++;
    h.resize(o_divi + di.size() / 2 + 1, 0ull);
    memcpy(h.data() + o_divi, di.data(), di.size() * sizeof(int32_t));
    EDGPU_CUDA(cudaMalloc(&d_all, h.size() * sizeof(unsigned long long)));
    EDGPU_CUDA(cudaMemcpy(d_all, h.data(), h.size() * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    dev.num = (const int32_t*)(d_all + o_num);
    divi = (const int32_t*)(d_all + o_divi);
    if (g.kind == GK_TORUS) dev.keep = d_all;
    if (g.kind == GK_GENERIC) {
        dev.lut = d_all;
        dev.flips = d_all + o_flips;
    }
}

void GroupBuffers::release() {
    cudaFree(d_all);
    d_all = nullptr;
}

Space::~Space() {
    if (d_keys) cudaFree(d_keys);
    if (d_dir) cudaFree(d_dir);
    if (d_map) cudaFree(d_map);
    if (d_rank) cudaFree(d_rank);
    if (d_vec_rank) cudaFree(d_vec_rank);
    delete vec;
}

VectorTables::~VectorTables() {
    if (d_ampl) cudaFree(d_ampl);
    if (d_inv) cudaFree(d_inv);
}

void enumerate_parent(Space& s, cudaStream_t st) {
    if (s.w32) enumerate_parent_t<uint32_t>(s, st);
    else enumerate_parent_t<unsigned long long>(s, st);
}

void enumerate_reps(Space& red, const Space& parent, cudaStream_t st) {
    if (red.w32) enumerate_reps_t<uint32_t>(red, parent, st);
    else enumerate_reps_t<unsigned long long>(red, parent, st);
}

namespace {
template <typename W>
void build_mapping_t(const Space& red, const Space& parent, int64_t* index_out, double* ampl_out, cudaStream_t st) {
    GroupBuffers gb;
    gb.upload(red.group, parent.lay);
    std::vector<double> ph(2 * (size_t)red.group.den);
    for (int j = 0; j < red.group.den; ++j) {
        const double ang = 2.0 * M_PI * (double)j / (double)red.group.den;
        ph[2 * j] = std::cos(ang);
        ph[2 * j + 1] = std::sin(ang);
    }
    double2* d_ph = nullptr;
    long long* d_idx = nullptr;
    double2* d_amp = nullptr;
    const long long n = parent.dim;
    try {
        EDGPU_CUDA(cudaMalloc(&d_ph, ph.size() * sizeof(double)));
        EDGPU_CUDA(cudaMemcpy(d_ph, ph.data(), ph.size() * sizeof(double), cudaMemcpyHostToDevice));
        EDGPU_CUDA(cudaMalloc(&d_idx, std::max<long long>(n, 1) * sizeof(long long)));
        EDGPU_CUDA(cudaMalloc(&d_amp, std::max<long long>(n, 1) * sizeof(double2)));
        if (n > 0) {
            if (parent.w32)
                k_mapping<W, unsigned><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
                    (const unsigned*)parent.d_keys, n, (const W*)red.d_keys, red.dim, red.sb, gb.dev, d_ph, d_idx, d_amp);
            else
                k_mapping<W, unsigned long long><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
                    (const unsigned long long*)parent.d_keys, n, (const W*)red.d_keys, red.dim, red.sb, gb.dev, d_ph,
                    d_idx, d_amp);
            EDGPU_CUDA(cudaGetLastError());
            EDGPU_CUDA(cudaMemcpyAsync(index_out, d_idx, n * sizeof(long long), cudaMemcpyDeviceToHost, st));
            EDGPU_CUDA(cudaMemcpyAsync(ampl_out, d_amp, n * sizeof(double2), cudaMemcpyDeviceToHost, st));
            EDGPU_CUDA(cudaStreamSynchronize(st));
        }
    } catch (...) {
        cudaFree(d_ph);
        cudaFree(d_idx);
        cudaFree(d_amp);
        throw;
    }
    cudaFree(d_ph);
    cudaFree(d_idx);
    cudaFree(d_amp);
}

// Parent-state map over the fixed-popcount parent sector (see Space::d_map): one thread per colex rank
// r: the parent state q = unrank(r), its orbit minimum and an element reaching it, the representative's
// index by the search directory, packed into one entry (all ones when the orbit is not in the table).
template <typename W, typename E>
__global__ void k_build_map(long long n_parent, int n, int k, const unsigned long long* C, const W* reps,
                            DirSearch ds, GroupDev g, int cb, int direct, E* out) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n_parent;
         r += (long long)gridDim.x * blockDim.x) {
        const W q = unrank_combo<W>((unsigned long long)r, n, k, C);
        W rep = q;
        int gb = 0, stab = 1;
        if (g.kind == GK_TORUS) {
            W keep[64];
            for (int a = 0; a < g.L1; ++a) keep[a] = (W)g.keep[a];
            canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, true, false, rep, gb, stab);
        } else if (g.kind == GK_GENERIC) {
            for (int e = 0; e < g.G; ++e) {
                W t = 0;
                const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
                for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
                t ^= (W)g.flips[e];
                if (t < rep) {
                    rep = t;
                    gb = e;
                }
            }
        }
        W reps2[2] = {rep, rep};
        const bool act[2] = {true, false};
        long long c[2];
        int sx[2];
        key_find_sum2<W>(reps, ds, reps2, act, c, sx);
        E e = (E)~(E)0;
        if (c[0] >= 0) e = (E)c[0] | ((E)sx[0] << cb) | (g.den > 1 ? (E)gb << (cb + ds.sb) : (E)0);
        out[direct ? (long long)q : r] = e;
    }
}

template <typename W>
void orbit_sizes_t(const Space& red, int32_t* out_host, cudaStream_t st) {
    GroupBuffers gb;
    gb.upload(red.group, red.lay);
    int32_t* d = nullptr;
    const long long n = red.dim;
    EDGPU_CUDA(cudaMalloc(&d, std::max<long long>(n, 1) * sizeof(int32_t)));
    if (n > 0) {
        k_orbit_sizes<W><<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const W*)red.d_keys, n, red.sb, gb.dev, d);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(out_host, d, n * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            cudaFree(d);
            throw Error(EDGPU_ERR_CUDA, std::string("orbit sizes: ") + cudaGetErrorString(e));
        }
    }
    cudaFree(d);
}

template <typename W>
void lookup_t(const Space& s, const uint64_t* keys_host, int64_t n, int64_t* out_host, cudaStream_t st) {
    unsigned long long* dq = nullptr;
    long long* dout = nullptr;
    try {
        EDGPU_CUDA(cudaMalloc(&dq, std::max<int64_t>(n, 1) * sizeof(unsigned long long)));
        EDGPU_CUDA(cudaMalloc(&dout, std::max<int64_t>(n, 1) * sizeof(long long)));
        EDGPU_CUDA(cudaMemcpyAsync(dq, keys_host, n * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        const unsigned long long smax = (s.lay.nbits >= 64) ? ~0ull : ((1ull << s.lay.nbits) - 1ull);
        k_lookup<W><<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const W*)s.d_keys, s.dim, s.sb, dq, n, dout, smax);
        EDGPU_CUDA(cudaGetLastError());
        EDGPU_CUDA(cudaMemcpyAsync(out_host, dout, n * sizeof(long long), cudaMemcpyDeviceToHost, st));
        EDGPU_CUDA(cudaStreamSynchronize(st));
    } catch (...) {
        cudaFree(dq);
        cudaFree(dout);
        throw;
    }
    cudaFree(dq);
    cudaFree(dout);
}
}  // namespace

void build_mapping(const Space& red, const Space& parent, int64_t* index_out, double* ampl_out, cudaStream_t st) {
    if (red.w32) build_mapping_t<uint32_t>(red, parent, index_out, ampl_out, st);
    else build_mapping_t<unsigned long long>(red, parent, index_out, ampl_out, st);
}

void orbit_sizes(const Space& red, int32_t* out_host, cudaStream_t st) {
    if (red.w32) orbit_sizes_t<uint32_t>(red, out_host, st);
    else orbit_sizes_t<unsigned long long>(red, out_host, st);
}

void lookup_keys(const Space& s, const uint64_t* keys_host, int64_t n, int64_t* out_host, cudaStream_t st) {
    if (n <= 0) return;
    if (s.w32) lookup_t<uint32_t>(s, keys_host, n, out_host, st);
    else lookup_t<unsigned long long>(s, keys_host, n, out_host, st);
}

}  // namespace edgpu

namespace edgpu {
void count_nnz(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const uint64_t* flips,
               int64_t* n_targets, int64_t* n_found, cudaStream_t st) {
    if (s.w32) count_nnz_t<uint32_t>(s, T, masks, rows, flips, n_targets, n_found, st);
    else count_nnz_t<unsigned long long>(s, T, masks, rows, flips, n_targets, n_found, st);
}
}  // namespace edgpu

namespace edgpu {

int orbit_index_bits(int G) {
    int nd = 0;
    for (int d = 1; d <= G; ++d) nd += (G % d == 0);
    int b = 0;
    while ((1 << b) < nd) ++b;
    return b;
}

namespace {
template <typename W>
void dir_t(Space& s, cudaStream_t st) {
    const long long n = s.dim;
    if (n >= (1ll << 32)) throw Error(EDGPU_ERR_ARG, "tables of 2^32 or more rows are not supported");
    unsigned long long max_state = 0;
    if (n > 0) {
        W last;
        EDGPU_CUDA(cudaMemcpy(&last, (const W*)s.d_keys + (n - 1), sizeof(W), cudaMemcpyDeviceToHost));
        max_state = (unsigned long long)(last >> s.sb);
    }
    int bitlen = 0;
    while (bitlen < 64 && (max_state >> bitlen) != 0ull) ++bitlen;
    int nbits_n = 0;
    while ((1ll << nbits_n) < std::max<long long>(n, 1)) ++nbits_n;
    // the directory may use up to 16x the key table (HBM is plentiful; a clustered table needs small
    // buckets before most of its keys fit in their bucket summaries)
    const size_t cap_bytes = std::max<size_t>((size_t)512 << 20, 16 * (size_t)n * sizeof(W));
    // candidate shifts: from about one bucket per key (s_hi) down to the smallest the cap allows
    // bucket summaries need member fields of at least one bit (shift + sb >= 1): a dense table of
    // unreduced keys (every state present) gets buckets of two states
    const int min_shift = s.sb == 0 ? 1 : 0;
    const int s_hi = std::max(min_shift, bitlen - std::max(1, std::min(nbits_n, bitlen)));
    int s_lo = s_hi;
    while (s_lo > min_shift && s_hi - s_lo < 63 &&
           (size_t)((max_state >> (s_lo - 1)) + 2) * sizeof(unsigned long long) <= cap_bytes)
        --s_lo;
    const int n_shift = s_hi - s_lo + 1;
    unsigned long long* d_stats = nullptr;   // survey counts [n_shift], then [largest bucket, inline keys]
    EDGPU_CUDA(cudaMalloc(&d_stats, (n_shift + 2) * sizeof(unsigned long long)));
    std::vector<unsigned long long> cnt(n_shift + 2, 0ull);
    cudaError_t e = cudaMemsetAsync(d_stats, 0, (n_shift + 2) * sizeof(unsigned long long), st);
    if (e == cudaSuccess && n > 0) {
        const long long per_block = 8 * SURVEY_RUN * 24;
        k_dir_survey<W><<<(unsigned)((n + per_block - 1) / per_block), 256, 0, st>>>((const W*)s.d_keys, n, s.sb, s_lo, n_shift, d_stats);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(cnt.data(), d_stats, n_shift * sizeof(unsigned long long),
                                              cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        cudaFree(d_stats);
        throw Error(EDGPU_ERR_CUDA, std::string("search directory survey: ") + cudaGetErrorString(e));
    }
    // the widest buckets whose summaries answer at least 98% of the keys, else the best fraction
    int shift = s_hi;
    double best = -1.0;
    for (int sh = s_hi; sh >= s_lo; --sh) {
        const double f = n > 0 ? (double)cnt[sh - s_lo] / (double)n : 1.0;
        if (f > best) {
            best = f;
            shift = sh;
        }
        if (f >= 0.98) break;
    }
    const long long nb = (bitlen == 0) ? 1 : ((long long)(max_state >> shift) + 1);
    const int mb = shift + s.sb;
    const int K = mb == 0 ? 4 : std::min(4, 28 / mb);
    if (s.d_dir) cudaFree(s.d_dir);
    s.d_dir = nullptr;
    e = cudaMalloc(&s.d_dir, (nb + 1) * sizeof(unsigned long long));
    if (e == cudaSuccess) {
        k_dir_build<W><<<(unsigned)((nb + DIR_CHUNK - 1) / DIR_CHUNK), 256, 0, st>>>((const W*)s.d_keys, n, s.sb, shift,
                                                                                   nb, mb, K, s.d_dir, d_stats + n_shift);
        e = cudaGetLastError();
    }
    unsigned long long hs[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(hs, d_stats + n_shift, sizeof(hs), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_stats);
    if (e != cudaSuccess) {
        if (s.d_dir) cudaFree(s.d_dir);
        s.d_dir = nullptr;
        throw Error(e == cudaErrorMemoryAllocation ? EDGPU_ERR_OOM : EDGPU_ERR_CUDA,
                    std::string("search directory: ") + cudaGetErrorString(e));
    }
    s.dir_shift = shift;
    s.dir_nb = nb;
    s.dir_K = K;
    s.dir_inline = n > 0 ? (double)hs[1] / (double)n : 1.0;
    int steps = 0;
    while ((1ull << steps) < std::max<unsigned long long>(hs[0], 1ull)) ++steps;
    s.dir_steps = steps;
}

template <typename W>
void states_t(const Space& s, uint64_t* out_host, cudaStream_t st) {
    unsigned long long* d = nullptr;
    EDGPU_CUDA(cudaMalloc(&d, std::max<int64_t>(s.dim, 1) * 8));
    k_get_states<W><<<(unsigned)((s.dim + 255) / 256), 256, 0, st>>>((const W*)s.d_keys, s.dim, s.sb, d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_host, d, s.dim * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("get_states: ") + cudaGetErrorString(e));
}
}  // namespace

DirSearch dir_search_of(const Space& s) {
    DirSearch d{};
    d.dir = s.d_dir;
    d.nb = s.dir_nb;
    d.shift = s.dir_shift;
    d.mb = s.dir_shift + s.sb;
    d.K = s.dir_K;
    d.steps = s.dir_steps;
    d.sb = s.sb;
    const unsigned mbmask = d.mb >= 32 ? 0xffffffffu : ((1u << d.mb) - 1u);
    const unsigned smask = (1u << d.sb) - 1u;
    for (int k = 0; k < d.K; ++k) {
        const int o = k * d.mb;
        d.unit |= 1u << o;
        d.keybits |= (mbmask & ~smask) << o;
        d.low |= (mbmask >> 1) << o;
        d.top |= (1u << (d.mb - 1)) << o;
    }
    return d;
}

void build_search_directory(Space& s, cudaStream_t st) {
    if (s.w32) dir_t<uint32_t>(s, st);
    else dir_t<unsigned long long>(s, st);
}

namespace {
int bitlen_u64(unsigned long long v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0ull) ++b;
    return b;
}

// Split colex rank tables of the n-bit words of popcount k: A over the high n - n / 2 bits, then B over the
// low n / 2 (see build_parent_map).
constexpr int RANK_SPLIT_BITS = 44;
std::vector<unsigned long long> split_rank_table(int n, int k) {
    const int lb = n / 2, hb = n - lb;
    std::vector<unsigned long long> T(((size_t)1 << hb) + ((size_t)1 << lb), 0ull);
    unsigned long long acc = 0;
    for (size_t h = 0; h < ((size_t)1 << hb); ++h) {
        T[h] = acc;
        const int need = k - __builtin_popcountll(h);
        acc += (need >= 0 && need <= lb) ? host_binom(lb, need) : 0ull;
    }
    std::vector<unsigned long long> cnt(lb + 1, 0ull);
    for (size_t l = 0; l < ((size_t)1 << lb); ++l) T[((size_t)1 << hb) + l] = cnt[__builtin_popcountll(l)]++;
    return T;
}

template <typename W>
void build_map_t(Space& red, cudaStream_t st) {
    const Layout& L = red.lay;
    const int n = L.nbits, k = L.popcount;
    const long long np = (long long)host_binom(n, k);   // parent states (the map may be larger when direct)
    GroupBuffers gb;
    gb.upload(red.group, L);
    const DirSearch ds = dir_search_of(red);
    const unsigned blocks = (unsigned)std::min<long long>((np + 255) / 256, 152ll * 64);
    if (red.map_wide)
        k_build_map<W, unsigned long long><<<blocks, 256, 0, st>>>(np, n, k, binomial_table(), (const W*)red.d_keys, ds,
                                                                  gb.dev, red.map_cb, red.map_direct,
                                                                  (unsigned long long*)red.d_map);
    else
        k_build_map<W, unsigned><<<blocks, 256, 0, st>>>(np, n, k, binomial_table(), (const W*)red.d_keys, ds, gb.dev,
                                                        red.map_cb, red.map_direct, (unsigned*)red.d_map);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("parent map: ") + cudaGetErrorString(e));
}
}  // namespace

void free_parent_map(Space& red) {
    if (red.d_map) cudaFree(red.d_map);
    if (red.d_rank) cudaFree(red.d_rank);
    red.d_map = nullptr;
    red.d_rank = nullptr;
    red.map_n = 0;
    ++red.map_gen;
}

bool build_parent_map(Space& red, int64_t max_bytes, cudaStream_t st) {
    const Layout& L = red.lay;
    if (!red.reduced || L.popcount < 0 || L.nbits > 64 || red.dim == 0 || !red.d_keys || !red.d_dir) return false;
    const int n = L.nbits, k = L.popcount;
    const unsigned long long np = host_binom(n, k);
    const int cb = bitlen_u64((unsigned long long)red.dim);
    // the element is needed only for characters other than 1
    const int gbits = red.group.den > 1 ? bitlen_u64((unsigned long long)std::max(red.group.G - 1, 0)) : 0;
    const int wide = (cb + red.sb + gbits <= 32) ? 0 : 1;
    if (cb + red.sb + gbits > 64) return false;
    const double bytes = (double)np * (wide ? 8.0 : 4.0);
    if (bytes > (double)max_bytes) return false;
    // direct indexing (entry index = the state itself, no rank) when the whole state range is small:
    // at most 2^30 entries and 4 GB, within the limit
    const double dbytes = n <= 30 ? (double)(1ull << n) * (wide ? 8.0 : 4.0) : 1e300;
    const bool direct = dbytes <= std::min((double)max_bytes, 4.0 * (1ull << 30));
    // Colex rank tables.  Split form (n <= 44): with lb = n / 2 low bits, the rank of q = (H << lb) | L
    // is A[H] + B[L], where A[H] counts the sector's states whose high part is below H (sum over
    // H' < H of C(lb, k - popc(H'))) and B[L] is the rank of L among the lb-bit words of its popcount.
    // Chunk form (larger n): T[(c * (k + 1) + j) * 64 + v] = sum over the set bits b of v, in ascending
    // order t = 0, 1, ..., of C(6c + b, j + t + 1).
    const int rank_wide = np > 0xffffffffull ? 1 : 0;
    const int split = n <= RANK_SPLIT_BITS ? n / 2 : 0;
    std::vector<unsigned long long> T;
    if (split) {
        T = split_rank_table(n, k);
    } else {
        const int nc = (n + RANK_CHUNK - 1) / RANK_CHUNK;
        T.assign((size_t)nc * (k + 1) * 64, 0ull);
        for (int c = 0; c < nc; ++c)
            for (int j = 0; j <= k; ++j)
                for (int v = 0; v < 64; ++v) {
                    unsigned long long sum = 0;
                    int t = 0;
                    for (int bb = 0; bb < RANK_CHUNK; ++bb)
                        if ((v >> bb) & 1) {
                            sum += host_binom(RANK_CHUNK * c + bb, j + t + 1);
                            ++t;
                        }
                    T[((size_t)c * (k + 1) + j) * 64 + v] = sum;
                }
    }
    free_parent_map(red);
    std::vector<unsigned> T32;
    if (!rank_wide) T32.assign(T.begin(), T.end());
    const size_t tbytes = T.size() * (rank_wide ? 8 : 4);
    cudaError_t e = cudaMalloc(&red.d_rank, tbytes);
    if (e == cudaSuccess)
        e = cudaMemcpy(red.d_rank, rank_wide ? (const void*)T.data() : (const void*)T32.data(), tbytes,
                       cudaMemcpyHostToDevice);
    const size_t entries = direct ? ((size_t)1 << n) : (size_t)np;
    if (e == cudaSuccess) e = cudaMalloc(&red.d_map, entries * (wide ? 8 : 4));
    if (e == cudaSuccess && direct) e = cudaMemsetAsync(red.d_map, 0xff, entries * (wide ? 8 : 4), st);   // invalid
    if (e != cudaSuccess) {
        free_parent_map(red);
        if (e == cudaErrorMemoryAllocation) return false;
        throw Error(EDGPU_ERR_CUDA, std::string("parent map: ") + cudaGetErrorString(e));
    }
    red.map_direct = direct ? 1 : 0;
    red.map_n = (int64_t)entries;
    red.map_wide = wide;
    red.map_cb = cb;
    red.rank_wide = rank_wide;
    red.rank_split = split;
    try {
        if (red.w32) build_map_t<uint32_t>(red, st);
        else build_map_t<unsigned long long>(red, st);
    } catch (...) {
        free_parent_map(red);
        throw;
    }
    ++red.map_gen;
    return true;
}

void get_states(const Space& s, uint64_t* out_host, cudaStream_t st) {
    if (s.dim == 0) return;
    if (s.w32) states_t<uint32_t>(s, out_host, st);
    else states_t<unsigned long long>(s, out_host, st);
}

}  // namespace edgpu

namespace edgpu {
namespace {
template <typename W>
__global__ void k_diag(const W* keys, long long n, int sb, int T, const unsigned long long* masks,
                       const unsigned long long* rows, const double2* amps, double2* out64, float2* out32) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const W b = keys[i] >> sb;
    double2 e = make_double2(0.0, 0.0);
    for (int t = 0; t < T; ++t)
        if ((b & (W)masks[t]) == (W)rows[t]) {
            e.x += amps[t].x;
            e.y += amps[t].y;
        }
    if (out64) out64[i] = e;
    if (out32) out32[i] = make_float2((float)e.x, (float)e.y);
}

template <typename W>
void diag_t(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const double* amps, double* out64,
            float* out32, unsigned long long* scratch, cudaStream_t st) {
    unsigned long long* d = scratch;
    const size_t Tm = std::max(T, 1);
    if (!scratch) EDGPU_CUDA(cudaMalloc(&d, Tm * (8 + 8 + 16)));
    unsigned long long* dm = d;
    unsigned long long* dr = d + Tm;
    double2* da = (double2*)(d + 2 * Tm);
    cudaError_t e = cudaSuccess;
    if (T > 0) {
        e = cudaMemcpyAsync(dm, masks, T * 8, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dr, rows, T * 8, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(da, amps, T * 16, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess && s.dim > 0) {
        k_diag<W><<<(unsigned)((s.dim + 255) / 256), 256, 0, st>>>((const W*)s.d_keys, s.dim, s.sb, T, dm, dr, da,
                                                                  (double2*)out64, (float2*)out32);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (!scratch) cudaFree(d);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("diagonal: ") + cudaGetErrorString(e));
}
}  // namespace

void compute_diagonal(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const double* amps,
                      double* out64, float* out32, unsigned long long* scratch, cudaStream_t st) {
    if (s.w32) diag_t<uint32_t>(s, T, masks, rows, amps, out64, out32, scratch, st);
    else diag_t<unsigned long long>(s, T, masks, rows, amps, out64, out32, scratch, st);
}
}  // namespace edgpu

// ---- vectors between the parent space and the reduced space, on the device -----------------------
// symmetry_unreduce(rhsr, small) and symmetry_reduce(rhsr, large) (symmetry_reduce.jl:208-225 and
// :38-56): the reference reads its parent-sized tables basis_mapping_index / basis_mapping_amplitude;
// here every parent entry's representative, stabiliser and group element are recomputed, so they run
// for parents whose tables do not fit (a parent vector of 9.1e9 entries for the 6x6 torus does).
// Parent index i <-> state: the materialised parent's sorted basis, or for a lazy popcount sector the
// colex rank (rank = sum over the set bits, lowest first, of C(position, count so far)).
namespace edgpu {
namespace {

// g.q for element e of the group (T(a, b) with e = a + L1 b for a torus: rows rotated left by a sites,
// then the rows moved up by b; the chunk tables and flip mask for a general group).
template <typename W>
__device__ __forceinline__ W group_elem_apply(W q, int e, const GroupDev& g) {
    if (g.kind == GK_TORUS) {
        const int a = e % g.L1, b = e / g.L1;
        const W full = (W)g.full;
        W v = q;
        if (a) {
            const int s = a * g.w;
            const W keep = (W)g.keep[a];
            v = (W)(((v & keep) << s) | ((v & ~keep & full) >> (g.rowbits - s)));
        }
        const int sr = b * g.rowbits;
        if (sr) v = (W)(((v << sr) | (v >> (g.nbits - sr))) & full);
        return v;
    }
    if (g.kind == GK_GENERIC) {
        W t = 0;
        const unsigned long long* L = g.lut + (size_t)e * g.nchunks * 16;
        for (int c = 0; c < g.nchunks; ++c) t |= (W)L[c * 16 + (int)((q >> (4 * c)) & 15u)];
        return t ^ (W)g.flips[e];
    }
    return q;
}

template <typename W>
__device__ __forceinline__ long long colex_rank(W q, const unsigned long long* C) {
    long long r = 0;
    int j = 0;
    while (q) {
        const int pos = (sizeof(W) == 8) ? __ffsll((long long)q) - 1 : __ffs((int)q) - 1;
        ++j;
        r += (long long)C[pos * 65 + j];
        q &= q - 1;
    }
    return r;
}

// Colex rank through the split tables (rank_tables) or bit by bit.
template <typename W>
__device__ __forceinline__ long long parent_rank(W q, const VectorTables::Dev& t, const unsigned long long* C) {
    if (t.rank_split) {
        const unsigned long long hi = (unsigned long long)(q >> t.rank_split);
        const unsigned long long lo = (unsigned long long)q & ((1ull << t.rank_split) - 1ull);
        if (t.rank_wide) {
            const unsigned long long* A = (const unsigned long long*)t.rank;
            return (long long)(__ldg(A + hi) + __ldg(A + t.rank_hi + lo));
        }
        const unsigned* A = (const unsigned*)t.rank;
        return (long long)(__ldg(A + hi) + __ldg(A + t.rank_hi + lo));
    }
    return colex_rank<W>(q, C);
}

constexpr int UNRED_E = 16;   // consecutive parent states per thread and round

// large[i] = ampl(p_i) small[c(p_i)] (0 where the orbit has no representative), the parent index i
// running over [0, n_parent).  The amplitude chi(g) sqrt(|stab| / |G|) comes from a table by the key's
// orbit-size index and the character (the square root and division it replaces kept the FP64 pipe busy
// for most of the kernel), rings are canonicalised by funnel shifts, the representative's row comes from
// the search directory, and a thread unranks one state in sixteen (the others are the next words), handed
// to the block through shared memory so that large is written in order.  10.4 million states of
// chain L = 26 at k = 1, complex128, this kernel and k_reduce, calls included: 892 -> 272 us; what is left
// here is the ring search and the FP64 pipe (four FMAs a state: 66 us).
template <typename W, typename PW, typename V>
__global__ void __launch_bounds__(256, 4) k_unreduce(const PW* parent, long long n_parent, int n, int k,
                                                  const unsigned long long* C, const W* reps, DirSearch ds, GroupDev g,
                                                  VectorTables::Dev t, const V* small, V* large) {
    __shared__ W st[256 * UNRED_E + 256 * UNRED_E / 32];   // (one word in 33 spare: no bank conflicts)
    __shared__ W keep[64];
    stage_keep<W>(keep, g);
    const bool want_arg = g.den > 1;
    const bool ring = ring32<W>(g);
    const int pb = t.elem_bits;
    for (long long base = (long long)blockIdx.x * (256 * UNRED_E); base < n_parent;
         base += (long long)gridDim.x * (256 * UNRED_E)) {
        if (!parent) {
            const long long i0 = base + (long long)threadIdx.x * UNRED_E;
            W q = i0 < n_parent ? unrank_combo<W>((unsigned long long)i0, n, k, C) : (W)0;
#pragma unroll
            for (int j = 0; j < UNRED_E; ++j) {
                const int at = threadIdx.x * UNRED_E + j;
                st[at + at / 32] = q;
                if (i0 + j + 1 < n_parent) q = gosper_next<W>(q);
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int j = 0; j < UNRED_E; j += 2) {
            W rep[2];
            int gb[2] = {0, 0}, sx[2];
            bool act[2];
            long long c[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int at = (j + h) * 256 + threadIdx.x;
                const long long i = base + at;
                act[h] = i < n_parent;
                W q = 0;
                if (act[h]) q = parent ? (W)parent[i] : st[at + at / 32];
                rep[h] = q;
                if (g.kind == GK_TORUS) {
                    if (ring) {
                        unsigned m;
                        canon_ring((unsigned)q, g.nbits, g.L1, g.w, pb, want_arg, m, gb[h]);
                        rep[h] = (W)m;
                    } else {
                        int stab;
                        canon_torus<W>(q, g.L1, g.L2, g.w, g.rowbits, g.nbits, (W)g.full, keep, want_arg, false, rep[h],
                                       gb[h], stab);
                    }
                } else if (g.kind == GK_GENERIC) {
                    for (int e = 0; e < g.G; ++e) {
                        const W u = group_elem_apply<W>(q, e, g);
                        if (u < rep[h]) {
                            rep[h] = u;
                            gb[h] = e;
                        }
                    }
                }
            }
            if (ds.dir) {
                key_find_sum2<W>(reps, ds, rep, act, c, sx);
            } else {
                c[0] = c[1] = -1;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const long long i = base + (j + h) * 256 + threadIdx.x;
                if (!act[h]) continue;
                V out;
                out.x = 0;
                out.y = 0;
                if (c[h] >= 0) {
                    const double2 a = __ldg(t.ampl + (size_t)sx[h] * g.den + (want_arg ? __ldg(g.num + gb[h]) : 0));
                    const V v = small[c[h]];
                    out.x = (decltype(out.x))(a.x * (double)v.x - a.y * (double)v.y);
                    out.y = (decltype(out.y))(a.x * (double)v.y + a.y * (double)v.x);
                }
                large[i] = out;
            }
        }
        if (!parent) __syncthreads();
    }
}

// small[c] = sum over the orbit members p of rep_c of conj(ampl(p)) large[i(p)].  Every element e of
// the group gives the member e.rep_c with ampl = conj(chi(e)) sqrt(|stab| / |G|); each distinct
// member occurs |stab| times among the |G| elements, so the sum over all elements is divided by
// |stab|.  One thread per representative, elements in a fixed order (reproducible, no atomics); the
// parent index of a member by the split rank tables instead of a sum over its bits.  Bound by the FP64 pipe (four FMAs
// a member: 66 us of the above) and by random sectors of large.
template <typename W, typename PW, typename V>
__global__ void __launch_bounds__(256) k_reduce(const PW* parent, long long n_parent, const unsigned long long* C,
                                                const W* reps, long long n_reps, int sb, GroupDev g,
                                                VectorTables::Dev t, const V* large, V* small) {
    const int L1 = g.kind == GK_TORUS ? g.L1 : 1, L2 = g.kind == GK_TORUS ? g.L2 : 1;
    const int G = g.kind == GK_TORUS ? L1 * L2 : g.G;
    const W full = (W)g.full;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n_reps;
         c += (long long)gridDim.x * blockDim.x) {
        const W key = reps[c], rep = key >> sb;
        const double s = __ldg(t.inv_norm + (int)(key & (W)((((W)1) << sb) - 1)));
        double ar = 0.0, ai = 0.0;
        int a = 0;
        W row = rep;   // TORUS: the rows moved up by b
#pragma unroll 4
        for (int e = 0; e < G; ++e) {
            W m;
            if (g.kind == GK_TORUS) {
                m = a ? torus_row_rotate<W>(row, a * g.w, (W)__ldg(g.keep + a), full, g.rowbits) : row;
                if (++a == L1) {
                    a = 0;
                    if (L2 > 1) row = (W)(((row << g.rowbits) | (row >> (g.nbits - g.rowbits))) & full);
                }
            } else {
                m = group_elem_apply<W>(rep, e, g);
            }
            long long i;
            if (t.by_rank) {
                // (a flip may take a member out of the parent's sector)
                if (__popcll((unsigned long long)m) != t.popcount) continue;
                i = parent_rank<W>(m, t, C);
            } else {
                long long lo = 0, len = n_parent;
                while (len > 0) {   // searchsortedfirst over the parent basis
                    const long long half = len >> 1;
                    if ((W)parent[lo + half] < m) {
                        lo += half + 1;
                        len -= half + 1;
                    } else {
                        len = half;
                    }
                }
                i = (lo < n_parent && (W)parent[lo] == m) ? lo : -1;
            }
            if (i < 0) continue;
            // conj(ampl) = chi(e) sqrt(|stab| / |G|); chi(e) = phase[num[e]]
            const double2 ph = __ldg(t.phase + __ldg(g.num + e));
            const V v = large[i];
            ar = fma(ph.x, (double)v.x, fma(-ph.y, (double)v.y, ar));
            ai = fma(ph.x, (double)v.y, fma(ph.y, (double)v.x, ai));
        }
        V out;
        out.x = (decltype(out.x))(ar * s);
        out.y = (decltype(out.y))(ai * s);
        small[c] = out;
    }
}

// The tables of a reduced space's vector maps: built on first use (the caller holds the space's lock) and
// kept with the space.
const VectorTables& vector_tables(const Space& red, const Space& parent) {
    if (red.vec) return *red.vec;
    std::unique_ptr<VectorTables> v(new VectorTables);
    v->gb.upload(red.group, parent.lay);
    const int den = red.group.den, G = red.group.G;
    std::vector<int> divs;
    for (int d = 1; d <= G; ++d)
        if (G % d == 0) divs.push_back(d);
    const size_t nd = divs.size();
    std::vector<double2> h((size_t)den * (nd + 1));   // amplitudes by (orbit-size index, character), then phases
    std::vector<double> inv(nd);
    for (int j = 0; j < den; ++j) {
        const double ang = 2.0 * M_PI * (double)j / (double)den;
        h[nd * den + j] = make_double2(std::cos(ang), std::sin(ang));
        for (size_t x = 0; x < nd; ++x) {
            const double f = std::sqrt((double)divs[x] / (double)G);
            h[x * den + j] = make_double2(h[nd * den + j].x * f, h[nd * den + j].y * f);
        }
    }
    for (size_t x = 0; x < nd; ++x) inv[x] = std::sqrt((double)divs[x] / (double)G) / (double)divs[x];
    EDGPU_CUDA(cudaMalloc(&v->d_ampl, h.size() * sizeof(double2)));
    EDGPU_CUDA(cudaMemcpy(v->d_ampl, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice));
    EDGPU_CUDA(cudaMalloc(&v->d_inv, inv.size() * sizeof(double)));
    EDGPU_CUDA(cudaMemcpy(v->d_inv, inv.data(), inv.size() * sizeof(double), cudaMemcpyHostToDevice));
    VectorTables::Dev& t = v->dev;
    t.ampl = v->d_ampl;
    t.phase = v->d_ampl + nd * den;
    t.inv_norm = v->d_inv;
    // the element index beside a 32-bit ring state (canon_ring)
    int pb = 0;
    while ((1 << pb) < red.group.L1) ++pb;
    t.elem_bits = red.lay.nbits + pb <= 32 ? pb : 0;
    // the parent index is the colex rank where the parent is all words of a popcount
    t.by_rank = parent.lay.popcount >= 0 ? 1 : 0;
    t.popcount = parent.lay.popcount;
    EDGPU_CUDA(cudaStreamSynchronize(nullptr));   // copies from pageable memory may return before they end
    red.vec = v.release();
    return *red.vec;
}

// Fills in the rank tables of a popcount parent.  They depend on the parent alone (64 MB at 44 bits), so they are
// built for the first reduction from it and kept with it; without room for them the kernel adds up the rank
// bit by bit.
void parent_rank_table(const Space& parent, VectorTables::Dev& t) {
    const int n = parent.lay.nbits;
    if (!t.by_rank || n < 2 || n > RANK_SPLIT_BITS) return;
    const int wide = host_binom(n, parent.lay.popcount) > 0xffffffffull ? 1 : 0;
    std::lock_guard<std::mutex> lk(parent.vec_rank_mu);
    if (!parent.d_vec_rank) {
        const std::vector<unsigned long long> T = split_rank_table(n, parent.lay.popcount);
        const std::vector<unsigned> T32(T.begin(), T.end());
        const size_t bytes = T.size() * (wide ? 8 : 4);
        void* d = nullptr;
        if (cudaMalloc(&d, bytes) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        cudaError_t e = cudaMemcpy(d, wide ? (const void*)T.data() : (const void*)T32.data(), bytes, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
        if (e != cudaSuccess) {
            cudaFree(d);
            throw Error(EDGPU_ERR_CUDA, std::string("rank table: ") + cudaGetErrorString(e));
        }
        parent.d_vec_rank = d;
    }
    t.rank_split = n / 2;
    t.rank_hi = 1ll << (n - n / 2);
    t.rank_wide = wide;
    t.rank = parent.d_vec_rank;
}

template <typename W, typename PW, typename V>
void reduce_vector_t(const Space& red, const Space& parent, bool unreduce, const void* in, void* out,
                     cudaStream_t st) {
    const VectorTables& vt = vector_tables(red, parent);
    const PW* pk = parent.d_keys ? (const PW*)parent.d_keys : nullptr;
    const long long n_parent = parent.d_keys ? parent.dim : (long long)host_binom(parent.lay.nbits, parent.lay.popcount);
    if (unreduce) {
        const long long need = (n_parent + 256 * UNRED_E - 1) / (256 * UNRED_E);
        const int blocks = (int)std::max<long long>(1, std::min<long long>(need, (long long)sm_count() * 16));
        DirSearch ds{};
        if (red.dim > 0) ds = dir_search_of(red);
        k_unreduce<W, PW, V><<<blocks, 256, 0, st>>>(pk, n_parent, parent.lay.nbits, parent.lay.popcount,
                                                     binomial_table(), (const W*)red.d_keys, ds, vt.gb.dev, vt.dev,
                                                     (const V*)in, (V*)out);
    } else if (red.dim > 0) {
        const int blocks = (int)std::max<long long>(1, std::min<long long>((red.dim + 255) / 256, (long long)sm_count() * 16));
        VectorTables::Dev t = vt.dev;
        parent_rank_table(parent, t);
        k_reduce<W, PW, V><<<blocks, 256, 0, st>>>(pk, n_parent, binomial_table(), (const W*)red.d_keys, red.dim, red.sb,
                                                   vt.gb.dev, t, (const V*)in, (V*)out);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("vector reduction: ") + cudaGetErrorString(e));
}

}  // namespace

int64_t parent_dimension(const Space& parent) {
    return parent.d_keys ? parent.dim : (int64_t)host_binom(parent.lay.nbits, parent.lay.popcount);
}

void reduce_vector(const Space& red, const Space& parent, int prec, bool unreduce, const void* in, void* out,
                   cudaStream_t st) {
    if (!parent.d_keys && parent.lay.popcount < 0)
        throw Error(EDGPU_ERR_STATE, "a lazy parent must be one popcount sector of 1-bit sites");
    const bool pw32 = parent.d_keys && parent.w32;
#define EDGPU_RV(W)                                                                                         \
    if (prec == EDGPU_FP64) {                                                                              \
        if (pw32) reduce_vector_t<W, uint32_t, double2>(red, parent, unreduce, in, out, st);                \
        else reduce_vector_t<W, unsigned long long, double2>(red, parent, unreduce, in, out, st);           \
    } else {                                                                                                \
        if (pw32) reduce_vector_t<W, uint32_t, float2>(red, parent, unreduce, in, out, st);                 \
        else reduce_vector_t<W, unsigned long long, float2>(red, parent, unreduce, in, out, st);            \
    }
    if (red.w32) {
        EDGPU_RV(uint32_t)
    } else {
        EDGPU_RV(unsigned long long)
    }
#undef EDGPU_RV
}

}  // namespace edgpu
