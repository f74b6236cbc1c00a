// Column-slab table of the pair-flip schedule and its multi-pass product (both precisions).
//
// On a large sector the target-table product (hx_bond.cuh, GK_TABLE) gathers x at random: with x
// many times the size of L2, nearly every gather is a DRAM sector of 32 bytes for 8 bytes of x.  The
// slab table regroups the same entries by the column slab their target lies in.  Pass q of the
// product reads only the entries whose columns lie in slab q, so while it runs the gathers hit a
// window of x small enough to stay in L2; its share is added to y.  y is then read and written once
// per pass, which is streamed traffic, instead of one random DRAM sector per target.
//
// The entries are those of the target table (itself the (row, target) form of the reference's
// basis_mapping_index, symmetry_reduce_generic.jl:33-35), with the coefficient of each element
// (amplitude x character x orbit-size ratio, reduced_operator_representation.jl:57-85) replaced by an
// index into a small table of the distinct coefficients.  Within a pass and a warp tile of 32 rows they
// are laid out in steps of at most one entry per row, so that the lanes of a warp read neighbouring
// entries and, because the targets of one bond are kept together, gather from few lines of x
// (hx_slab_fill_kernel).  Within a pass every row adds its entries in a fixed order and the passes are
// added in order, so results are reproducible run to run; they differ from the one-pass product by the
// order of the additions.  A scaled table's index leaves the orbit-size ratio sqrt(|O_c| / |O_r|) out: x
// is scaled by sqrt(|O_c|) before the passes (k_slab_xscale) and each row's result by 1 / sqrt(|O_r|) in
// the last pass.
//
// What bounds the product, and what the steps gave (complex64, H x in device time, before -> now;
// before, every lane walked its own row's run of entries): triangular 6x5, 5.2 million rows, one pass,
// 1168 -> 674 us; square 4x8, 18.8 million rows, two passes, 2963 -> 1715 us; square 6x6, 252 million
// rows, 18 passes, 70.6 -> 64.0 ms; chain L = 24, 112,720 rows, 5.6 -> 4.0 us.  It was bound by the L1
// data pipe (every entry load and every gather a line of its own); now a gather touches 0.2 (chains) to
// 0.5 (tori) lines per entry, and the L1 tag lookups of those lines and the L2 requests behind them
// share the limit (24 sectors of the triangular 6x4, 113,000 rows each: 352 us of tag lookups in 376 us;
// one launch over all of them, or more padding, gained nothing).  In FP64 the FP64 pipe sets the pace,
// before and now (chain L = 28 106.7 -> 100.9 us, triangular 6x5 at k = 1 3502 -> 3448, 6x6 130.1 -> 128.4 ms): a
// double-precision FMA occupies it for 16 cycles of an SM per warp, so the mean filling of the steps counts
// there.
#include "hx_bond.cuh"

#include <algorithm>
#include <type_traits>

namespace edgpu {

namespace {

// Shared-memory scratch of the fill pass: words per warp, and the most bytes of a block.
__host__ __device__ constexpr size_t slab_fill_words(int cap, int n_pass) { return (size_t)33 * cap + n_pass + 1; }
constexpr size_t SLAB_FILL_SMEM = 200 * 1024;

// Pass 1 counts every tile's entries and steps per slab: a step holds at most one entry of a row, so a
// tile has as many steps as the row with the most entries (rounded up to a multiple of four).
template <typename W, int PREC>
__global__ void __launch_bounds__(HX_THREADS) hx_slab_count_kernel(const HxParams p, const SlabBuild s) {
    extern __shared__ __align__(16) unsigned char sm[];
    {
        const int4* src = (const int4*)p.blob;
        int4* dst = (int4*)sm;
        for (int i = threadIdx.x; i < p.blob_words16; i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    const BondTables<W, PREC> bt(p, sm);
    RowsSector<PREC> sc{};
    sc.tab = p.tab;
    sc.tile_off = p.tile_off;
    sc.tab_wide = p.tab_wide;
    sc.tab_cb = p.tab_cb;
    const W* __restrict__ keys = (const W*)p.keys;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const W smask = (W)((((W)1) << p.sb) - 1);
    const unsigned wc = (unsigned)s.wc;
    unsigned char* ctr = sm + s.o_scratch;   // [n_pass][thread]
    for (long long tile = (long long)blockIdx.x * wpb + warp; tile < s.n_tiles; tile += (long long)gridDim.x * wpb) {
        const long long row = tile * 32 + lane;
        const bool act = row < p.n_rows;
        const W kr = act ? keys[row] : (W)0;
        const int cnt = bond_row_count<W, PREC>(kr >> p.sb, bt, act ? p.bond_ncls : 0, p.nbits, (W)p.full);
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        const long long tpos = p.tile_off[tile] + (incl - cnt);
        if (s.cls && act) s.cls[row] = (unsigned char)(kr & smask);
        for (int q = 0; q < s.n_pass; ++q) ctr[q * HX_THREADS + threadIdx.x] = 0;
        for (int t = 0; t < cnt; ++t) {
            long long c;
            int sx, g;
            table_entry<PREC>(sc, tpos + t, true, p.sb, c, sx, g);
            if (c >= 0) ++ctr[((unsigned)c / wc) * HX_THREADS + threadIdx.x];
        }
        for (int q = 0; q < s.n_pass; ++q) {
            const unsigned v = ctr[q * HX_THREADS + threadIdx.x];
            const unsigned sum = __reduce_add_sync(0xffffffffu, v), most = __reduce_max_sync(0xffffffffu, v);
            if (lane == 0) {
                s.tile_sum[(size_t)q * s.n_tiles + tile] = sum;
                s.tile_steps[(size_t)q * s.n_tiles + tile] = (most + 3u) & ~3u;
            }
        }
    }
}

// Pass 2 lays out every tile's steps and writes their row masks and entries.  The targets of one bond
// pair, of the tile's rows that have one in the slab, are placed together: into the step where most of
// these rows are still free, what is left of them into the next best, and so on (a row's entries fit,
// whatever their order, because the tile has a step for each).  Neighbouring rows' targets by one bond
// are often neighbours too (they are when the targets are representatives themselves), so a step's
// gathers share lines of x; taking every row's next entry instead (in_order) touches 1.3 to 1.5 times the
// lines.
// One warp per tile; scratch: per warp s.cap steps of 32 entries, their masks and the slabs' first
// steps; the slabs are taken in runs whose steps fit there.
template <typename W, int PREC>
__global__ void __launch_bounds__(HX_THREADS) hx_slab_fill_kernel(const HxParams p, const SlabBuild s) {
    extern __shared__ __align__(16) unsigned char sm[];
    {
        const int4* src = (const int4*)p.blob;
        int4* dst = (int4*)sm;
        for (int i = threadIdx.x; i < p.blob_words16; i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    const BondTables<W, PREC> bt(p, sm);
    RowsSector<PREC> sc{};
    sc.tab = p.tab;
    sc.tile_off = p.tile_off;
    sc.tab_wide = p.tab_wide;
    sc.tab_cb = p.tab_cb;
    const int* num = (const int*)(sm + p.o_num);
    const W* __restrict__ keys = (const W*)p.keys;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const W smask = (W)((((W)1) << p.sb) - 1);
    const W full = (W)p.full;
    const int n = p.nbits;
    const unsigned wc = (unsigned)s.wc;
    const size_t stride = (size_t)s.n_tiles + 1;   // of the tile offsets of one pass
    unsigned* ent = (unsigned*)(sm + s.o_scratch) + (size_t)warp * slab_fill_words(s.cap, s.n_pass);
    unsigned* occ = ent + 32 * s.cap;   // row masks of the steps
    unsigned* first = occ + s.cap;      // [n_pass + 1] first step of each slab of the run
    for (long long tile = (long long)blockIdx.x * wpb + warp; tile < s.n_tiles; tile += (long long)gridDim.x * wpb) {
        const long long row = tile * 32 + lane;
        const bool act = row < p.n_rows;
        const W kr = act ? keys[row] : (W)0;
        const W b = kr >> p.sb;
        const int ri = (int)(kr & smask);
        const int cnt = bond_row_count<W, PREC>(b, bt, act ? p.bond_ncls : 0, n, full);
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        const long long tpos0 = p.tile_off[tile] + (incl - cnt);
        for (int qa = 0; qa < s.n_pass;) {
            // the run of slabs [qa, qb) whose steps fit in the scratch (a slab's always do)
            int qb = qa;
            unsigned used = 0;
            __syncwarp();
            for (; qb < s.n_pass; ++qb) {
                const unsigned* mo = s.moff + qb * stride + tile;
                const unsigned S = mo[1] - mo[0];
                if (used + S > (unsigned)s.cap) break;
                if (lane == 0) first[qb - qa] = used;
                used += S;
            }
            if (lane == 0) first[qb - qa] = used;
            for (unsigned j = lane; j < used; j += 32) occ[j] = 0u;
            __syncwarp();
            long long tpos = tpos0;
            unsigned mine = 0;   // in_order: this row's entries so far
            for (int cls = 0; cls < p.bond_ncls; ++cls) {
                const W m = act ? bond_class_mask<W, PREC>(b, bt, cls, n, full) : (W)0;
                const bool cpar = (bt.ninfo[cls] >> 8) != 0;
                W u = warp_or<W>(m);
                while (u) {
                    const int i = lowest_bit<W>(u);
                    u &= u - 1;
                    const bool on = (m >> i) & 1;
                    const int ti = cls * n + i;
                    int v = (int)(b >> i) & 1;
                    if (cpar) v |= (__popcll((unsigned long long)(b & bt.flip[ti])) != 1) << 1;
                    long long c;
                    int sx, g;
                    table_entry<PREC>(sc, tpos, on, p.sb, c, sx, g);
                    tpos += on ? 1 : 0;
                    const bool has = on && c >= 0;
                    const int q = has ? (int)((unsigned)c / wc) : -1;
                    unsigned entry = 0;
                    if (has) {
                        const unsigned ph = p.want_arg ? (unsigned)num[g] : 0u;
                        const unsigned ap = (unsigned)__ldg(s.amp_id + ((ti << 2) | v)) * (unsigned)p.den + ph;
                        const unsigned nd = (unsigned)p.nd;
                        const unsigned id = s.scaled ? ap : (ap * nd + (unsigned)ri) * nd + (unsigned)sx;
                        entry = ((unsigned)c - (unsigned)q * wc) | (id << s.colbits);
                    }
                    if (s.in_order) {   // (one slab)
                        if (has) ent[mine++ * 32 + lane] = entry;
                        continue;
                    }
                    unsigned pending = __ballot_sync(0xffffffffu, q >= qa && q < qb);
                    if (s.counted) {
                        if ((pending >> lane) & 1u) {
                            unsigned k = first[q - qa];
                            while ((occ[k] >> lane) & 1u) ++k;
                            ent[k * 32 + lane] = entry;
                            atomicOr(&occ[k], 1u << lane);
                        }
                        __syncwarp();
                        continue;
                    }
                    while (pending) {
                        const int q0 = __shfl_sync(0xffffffffu, q, __ffs((int)pending) - 1);
                        unsigned rest = __ballot_sync(0xffffffffu, q == q0);
                        pending &= ~rest;
                        const unsigned f0 = first[q0 - qa], S = first[q0 - qa + 1] - f0;
                        while (rest) {
                            // the step with the most of these rows free (the lowest of them)
                            unsigned best = 0;
                            for (unsigned k = lane; k < S; k += 32)
                                best = max(best, ((unsigned)__popc(rest & ~occ[f0 + k]) << 16) | (0xffffu - k));
                            best = __reduce_max_sync(0xffffffffu, best);
                            const unsigned k = f0 + (0xffffu - (best & 0xffffu));
                            const unsigned o = occ[k], got = rest & ~o;
                            if ((got >> lane) & 1u) ent[k * 32 + lane] = entry;
                            __syncwarp();
                            if (lane == 0) occ[k] = o | got;
                            __syncwarp();
                            rest &= ~got;
                        }
                    }
                }
            }
            if (s.in_order) {
                for (unsigned k = 0; k < used; ++k) {
                    const unsigned o = __ballot_sync(0xffffffffu, k < mine);
                    if (lane == 0) occ[k] = o;
                }
                __syncwarp();
            }
            for (int q = qa; q < qb; ++q) {
                const unsigned f0 = first[q - qa], S = first[q - qa + 1] - f0;
                if (s.padded) {
                    // 32 entries a step, four steps of a lane side by side; a row without one gets a padding
                    // entry on the column of another row's in the step
                    const unsigned pad = (unsigned)s.n_ids << s.colbits, colmask = (1u << s.colbits) - 1u;
                    uint4* tab = (uint4*)(s.tab + s.base[q] + (size_t)s.moff[q * stride + tile] * 32) + lane;
                    for (unsigned k = 0; k < S; k += 4, tab += 32) {
                        unsigned v[4];
                        for (int h = 0; h < 4; ++h) {
                            const unsigned o = occ[f0 + k + h];
                            const int src = o ? __ffs((int)o) - 1 : 0;
                            v[h] = (o >> lane) & 1u ? ent[(f0 + k + h) * 32 + lane]
                                                    : pad | (o ? ent[(f0 + k + h) * 32 + src] & colmask : 0u);
                        }
                        *tab = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                    continue;
                }
                unsigned* tab = s.tab + s.base[q] + s.off[q * stride + tile];
                if (s.counted) {
                    unsigned c = 0;
                    while (c < S && ((occ[f0 + c] >> lane) & 1u)) ++c;
                    if (act) s.cnt[(size_t)q * p.n_rows + row] = (unsigned char)c;
                } else {
                    unsigned* mask = s.mask + s.mbase[q] + s.moff[q * stride + tile];
                    for (unsigned k = lane; k < S; k += 32) mask[k] = occ[f0 + k];
                }
                for (unsigned k = 0; k < S; ++k) {
                    const unsigned o = occ[f0 + k];
                    if ((o >> lane) & 1u) tab[__popc(o & below)] = ent[(f0 + k) * 32 + lane];
                    tab += __popc(o);
                }
            }
            qa = qb;
        }
    }
}

// Exclusive scan of the tile sums of every pass, in chunks of SLAB_CHUNK per block (blockIdx.y =
// pass): chunk totals, then a scan of the chunk totals per pass, then the offsets.
constexpr int SLAB_CHUNK = HX_THREADS * 16;

__global__ void k_slab_scan_part(const unsigned* ts, long long n_tiles, unsigned long long* part, int nb) {
    __shared__ long long tmp[32];
    const int q = blockIdx.y;
    const unsigned* a = ts + (size_t)q * n_tiles;
    const long long beg = (long long)blockIdx.x * SLAB_CHUNK + (long long)threadIdx.x * 16;
    long long s = 0;
    for (long long i = beg; i < min(n_tiles, beg + 16); ++i) s += a[i];
    long long tot = 0;
    block_exclusive_scan(s, tmp, &tot);
    if (threadIdx.x == 0) part[(size_t)q * nb + blockIdx.x] = (unsigned long long)tot;
}

__global__ void k_slab_scan_mid(unsigned long long* part, int nb, unsigned long long* totals) {
    __shared__ long long tmp[32];
    unsigned long long* a = part + (size_t)blockIdx.x * nb;
    long long carry = 0;
    for (int b0 = 0; b0 < nb; b0 += blockDim.x) {
        const int i = b0 + threadIdx.x;
        const long long v = i < nb ? (long long)a[i] : 0;
        long long tot = 0;
        const long long ex = block_exclusive_scan(v, tmp, &tot);
        if (i < nb) a[i] = (unsigned long long)(carry + ex);
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = (unsigned long long)carry;
}

__global__ void k_slab_scan_out(const unsigned* ts, long long n_tiles, const unsigned long long* part, int nb,
                                unsigned* off) {
    __shared__ long long tmp[32];
    const int q = blockIdx.y;
    const unsigned* a = ts + (size_t)q * n_tiles;
    unsigned* o = off + (size_t)q * (n_tiles + 1);
    const long long beg = (long long)blockIdx.x * SLAB_CHUNK + (long long)threadIdx.x * 16;
    const long long end = min(n_tiles, beg + 16);
    long long s = 0;
    for (long long i = beg; i < end; ++i) s += a[i];
    long long ex = block_exclusive_scan(s, tmp, nullptr) + (long long)part[(size_t)q * nb + blockIdx.x];
    for (long long i = beg; i < end; ++i) {
        o[i] = (unsigned)ex;
        ex += a[i];
    }
    if (beg < n_tiles && end == n_tiles) o[n_tiles] = (unsigned)ex;   // the pass's total
}

// acc += c x with explicit fused multiply-adds (the same roundings in every kernel of this file)
template <typename V>
__device__ __forceinline__ V cfma_acc(V acc, V c, V x) {
    acc.x = fma_r(c.x, x.x, acc.x);
    acc.x = fma_r(-c.y, x.y, acc.x);
    acc.y = fma_r(c.x, x.y, acc.y);
    acc.y = fma_r(c.y, x.x, acc.y);
    return acc;
}

// The entries, masks and y are read (and written) once per pass: evict-first, so that the slab of x
// keeps its place in L1 and L2 (18.8 million rows in two passes: 2.00 -> 1.72 ms).
template <typename T>
__device__ __forceinline__ T ld_stream(const T* p) {
    return __ldcs(p);
}
template <typename T>
__device__ __forceinline__ void st_stream(T* p, T v) {
    __stcs(p, v);
}

// The masks of the steps [k, k + 4) (k a multiple of four), 0 from k1 on.
__device__ __forceinline__ void ld_masks(const unsigned* __restrict__ mask, unsigned k, unsigned k1, unsigned* m) {
    const uint4 v = k < k1 ? ld_stream((const uint4*)(mask + k)) : make_uint4(0u, 0u, 0u, 0u);
    m[0] = v.x;
    m[1] = v.y;
    m[2] = v.z;
    m[3] = v.w;
}

// This lane's entries of four steps with the row masks m, the first of them at e0 (moved past them);
// below: the bits of the lanes before this one.  A lane without an entry reads that of the next row
// that has one (every pass ends with a padding entry).
__device__ __forceinline__ void ld_entries(const unsigned* __restrict__ tab, const unsigned* m, unsigned below,
                                           unsigned& e0, unsigned* e) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        e[h] = ld_stream(tab + (e0 + (unsigned)__popc(m[h] & below)));
        e0 += (unsigned)__popc(m[h]);
    }
}

// Adds a row's sum over this pass to y; some: the row has entries in the pass.  Passes add their sums in
// order: the first writes y, the last adds the diagonal term diag x too (so that a pass needs only its
// own slab of x, the last one all of it) and may write complex128 to y_c128 instead.
template <int PREC>
__device__ __forceinline__ void finish_row(const SlabRun& r, long long row, typename Cx<PREC>::V acc, bool some) {
    typedef typename Cx<PREC>::V V;
    typedef typename Cx<PREC>::R R;
    if (row >= r.n_rows) return;
    V* y = (V*)r.y;
    V t;
    if (r.first) {
        if (r.accumulate) {
            V yo = ld_stream(y + row);
            if (r.scaled) {
                // y += H x on a scaled table: the old y_r enters the row's scaled sum as sqrt(|O_r|) y_r
                const R sr = __ldg((const R*)r.scale + r.cls[row]);
                yo.x *= sr;
                yo.y *= sr;
            }
            t = cadd(yo, acc);
        } else {
            t = acc;
        }
    } else {
        if (!some && !r.last) return;   // nothing to add to this row
        t = cadd(ld_stream(y + row), acc);
    }
    if (r.last) {
        t = cfma_acc(t, ld_stream((const V*)r.diag + row), ld_stream((const V*)r.x + row));
        if (r.scaled) {
            const R rs = __ldg((const R*)r.scale + r.nd + r.cls[row]);
            t.x *= rs;
            t.y *= rs;
        }
    }
    if (r.last && r.y_c128 != nullptr) {
        double2 o = make_double2((double)t.x, (double)t.y);
        double2* yc = (double2*)r.y_c128;
        if (r.acc_c128) {
            const double2 old = yc[row];
            o.x += old.x;
            o.y += old.y;
        }
        yc[row] = o;
    } else {
        st_stream(y + row, t);
    }
}

// The coefficient table of a launch: in registers (LUTM 2: real, at most 4), or in shared memory, a copy
// per bank group (1) or one (0), with room for the id after the last (a padding entry's).
template <int PREC, bool REAL, int LUTM>
struct SlabLut {
    typedef typename Cx<PREC>::V V;
    typedef typename Cx<PREC>::R R;
    typedef typename std::conditional<REAL, R, V>::type T;
    static constexpr int REPS = LUTM == 1 ? 128 / (int)sizeof(T) : 1;   // copies per coefficient
    R c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    const T* sm;
    __device__ __forceinline__ SlabLut(const SlabRun& r, unsigned char* smem) : sm((const T*)smem) {
        const T* src = (const T*)r.lut;
        if constexpr (LUTM == 2) {
            const R* lr0 = (const R*)r.lut;
            c0 = __ldg(lr0);
            c1 = __ldg(lr0 + min(1, r.n_lut - 1));
            c2 = __ldg(lr0 + min(2, r.n_lut - 1));
            c3 = __ldg(lr0 + min(3, r.n_lut - 1));
        } else if constexpr (LUTM == 1) {
            for (int i = threadIdx.x; i < r.n_lut * REPS; i += blockDim.x) ((T*)smem)[i] = src[i / REPS];
            __syncthreads();
            sm += threadIdx.x & (REPS - 1);
        } else {
            for (int i = threadIdx.x; i < r.n_lut; i += blockDim.x) ((T*)smem)[i] = src[i];
            __syncthreads();
        }
    }
    __device__ __forceinline__ T operator()(unsigned id) const {
        if constexpr (LUTM == 2) return (id & 2u) ? ((id & 1u) ? c3 : c2) : ((id & 1u) ? c1 : c0);
        else return sm[id * REPS];
    }
};

// acc += c x when e < lim (predicated, without a branch)
__device__ __forceinline__ void fma_if(float2& a, float c, float2 x, unsigned e, unsigned lim) {
    asm("{.reg .pred p; setp.lt.u32 p, %5, %6; @p fma.rn.f32 %0, %2, %3, %0; @p fma.rn.f32 %1, %2, %4, %1;}"
        : "+f"(a.x), "+f"(a.y) : "f"(c), "f"(x.x), "f"(x.y), "r"(e), "r"(lim));
}
__device__ __forceinline__ void fma_if(double2& a, double c, double2 x, unsigned e, unsigned lim) {
    asm("{.reg .pred p; setp.lt.u32 p, %5, %6; @p fma.rn.f64 %0, %2, %3, %0; @p fma.rn.f64 %1, %2, %4, %1;}"
        : "+d"(a.x), "+d"(a.y) : "d"(c), "d"(x.x), "d"(x.y), "r"(e), "r"(lim));
}
__device__ __forceinline__ void fma_if(float2& a, float2 c, float2 x, unsigned e, unsigned lim) {
    fma_if(a, c.x, x, e, lim);
    fma_if(a, c.y, make_float2(-x.y, x.x), e, lim);
}
__device__ __forceinline__ void fma_if(double2& a, double2 c, double2 x, unsigned e, unsigned lim) {
    fma_if(a, c.x, x, e, lim);
    fma_if(a, c.y, make_double2(-x.y, x.x), e, lim);
}

// One pass of the product through a padded table: one lane per row, one warp per tile of 32 rows and
// r.chunk consecutive tiles, four steps at a time: a lane's four entries are one 16-byte load.  While a
// group's gathers are under way, the entries of the group after the next are read, on through the
// warp's tiles.  SUMS: partial sums per row, by the entry's place in its group; mixed precision takes
// four (a row of 93 terms is half as far from its 64-bit sum as with one) or two (SlabRun::two_sums).
// FP64 takes four on small by-bond tables (SLAB_FP64_SUMS; mostly by place), else one, and does not add up a
// step without entries (the last ones of a tile may be), since the FP64 pipe sets the pace (a warp's
// double-precision FMA takes 16 cycles of an SM).  To keep it busy, the gathers run a
// group ahead of the additions there (complex128, chain L = 27 at k = 1 98.3 -> 94.5 us, L = 28 104.3 -> 101.1;
// triangular 6x5 at k = 1 3596 -> 3451, square 4x8 in two passes 5321 -> 5125); in mixed precision the registers
// for that cost more than it gives (chain L = 24 5.5 -> 6.9 us).
template <int PREC, bool REAL, int LUTM, int SUMS>
__global__ void __launch_bounds__(HX_THREADS, PREC == 0 ? 3 : 4) hx_slab_pad_kernel(const SlabRun r) {
    typedef typename Cx<PREC>::V V;
    constexpr bool AHEAD = PREC == 0;
    extern __shared__ __align__(16) unsigned char sm[];
    if (r.early) pdl_launch_dependents();
    const SlabLut<PREC, REAL, LUTM> lut(r, sm);
    pdl_wait();
    const V* __restrict__ xs = (const V*)r.xs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const unsigned lim = (unsigned)r.n_lut << r.colbits;   // padding entries: from here on
    auto gather = [&](const uint4& g, V* x) {
        x[0] = xs[g.x & r.colmask];
        x[1] = xs[g.y & r.colmask];
        x[2] = xs[g.z & r.colmask];
        x[3] = xs[g.w & r.colmask];
    };
    auto add = [&](V& acc, unsigned g, const V& x, bool may_be_empty) {
        if (PREC == 0 && may_be_empty && !__any_sync(0xffffffffu, g < lim)) return;
        fma_if(acc, lut(g >> r.colbits), x, g, lim);
    };
    // (rows are below 2^32, so tiles below 2^27)
    const unsigned tile_end = (unsigned)(r.tile0 + r.n_tiles), hop = gridDim.x * wpb * r.chunk;
    for (unsigned c0 = (unsigned)r.tile0 + (blockIdx.x * wpb + warp) * r.chunk; c0 < tile_end; c0 += hop) {
        unsigned tile = c0;
        const unsigned t1 = min(c0 + r.chunk, tile_end);
        unsigned q = r.moff[tile] >> 2, qt = r.moff[tile + 1] >> 2;   // groups of four steps
        const uint4* __restrict__ tp = (const uint4*)r.tab + ((size_t)q * 32 + lane);
        uint4 e = ld_stream(tp), en = ld_stream(tp + 32);
        V x[4];
        if (AHEAD) gather(e, x);
        for (; tile < t1; ++tile) {
            const unsigned qn = tile + 1 < t1 ? r.moff[tile + 2] >> 2 : qt;
            V acc = czero<V>(), acc1 = acc, acc2 = acc, acc3 = acc;
            for (; q < qt; ++q) {
                V xn[4];
                if (AHEAD) gather(en, xn);
                else gather(e, x);
                tp += 32;
                const uint4 e2 = ld_stream(tp + 32);
                const bool tail = q + 1 == qt;   // (only a tile's last group may have empty steps)
                add(acc, e.x, x[0], false);
                add(SUMS == 1 ? acc : acc1, e.y, x[1], tail);
                add(SUMS == 4 ? acc2 : acc, e.z, x[2], tail);
                add(SUMS == 4 ? acc3 : SUMS == 2 ? acc1 : acc, e.w, x[3], tail);
                e = en;
                en = e2;
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    if (AHEAD) x[h] = xn[h];
            }
            if (SUMS == 4) acc = cadd(cadd(acc, acc1), cadd(acc2, acc3));
            if (SUMS == 2) acc = cadd(acc, acc1);
            finish_row<PREC>(r, (long long)tile * 32 + lane, acc, true);
            qt = qn;
        }
    }
    if (!r.early) pdl_launch_dependents();
}

// Small sectors (SLAB_SPLIT): WAYS warps share a tile, each taking every WAYS-th group of steps, so that a row's
// chain of gathers and additions is that much shorter; their sums are added in order.
template <int PREC, bool REAL, int LUTM, int WAYS>
__global__ void __launch_bounds__(HX_THREADS, 2) hx_slab_split_kernel(const SlabRun r) {
    typedef typename Cx<PREC>::V V;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ V part[HX_THREADS];
    if (r.early) pdl_launch_dependents();
    const SlabLut<PREC, REAL, LUTM> lut(r, sm);
    pdl_wait();
    const V* __restrict__ xs = (const V*)r.xs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lim = (unsigned)r.n_lut << r.colbits;
    const unsigned tile = (unsigned)r.tile0 + blockIdx.x * (HX_THREADS / 32 / WAYS) + warp / WAYS;
    const bool act = tile < (unsigned)(r.tile0 + r.n_tiles);
    V sum[4] = {};
    if (act) {
        const unsigned q1 = r.moff[tile + 1] >> 2;
        unsigned q = (r.moff[tile] >> 2) + warp % WAYS;
        const uint4* __restrict__ tp = (const uint4*)r.tab + ((size_t)q * 32 + lane);
        uint4 e = q < q1 ? ld_stream(tp) : make_uint4(0u, 0u, 0u, 0u);
        while (q < q1) {
            const V x0 = xs[e.x & r.colmask], x1 = xs[e.y & r.colmask];
            const V x2 = xs[e.z & r.colmask], x3 = xs[e.w & r.colmask];
            tp += 32 * WAYS;
            q += WAYS;
            const uint4 en = q < q1 ? ld_stream(tp) : e;
            fma_if(sum[0], lut(e.x >> r.colbits), x0, e.x, lim);
            fma_if(sum[1], lut(e.y >> r.colbits), x1, e.y, lim);
            fma_if(sum[2], lut(e.z >> r.colbits), x2, e.z, lim);
            fma_if(sum[3], lut(e.w >> r.colbits), x3, e.w, lim);
            e = en;
        }
    }
    part[threadIdx.x] = cadd(cadd(sum[0], sum[1]), cadd(sum[2], sum[3]));
    __syncthreads();
    if (act && warp % WAYS == 0) {
        V acc = part[threadIdx.x];
        for (int w = 1; w < WAYS; ++w) acc = cadd(acc, part[threadIdx.x + 32 * w]);
        finish_row<PREC>(r, (long long)tile * 32 + lane, acc, true);
    }
    if (!r.early) pdl_launch_dependents();
}

// Four warps share a tile, warp w of them taking every group's step w: the sums per row of hx_slab_pad_kernel with
// four partial sums, bit for bit, in chains a quarter as long (slab_split).
template <int PREC, bool REAL, int LUTM>
__global__ void __launch_bounds__(HX_THREADS, 2) hx_slab_place_kernel(const SlabRun r) {
    typedef typename Cx<PREC>::V V;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ V part[HX_THREADS];
    if (r.early) pdl_launch_dependents();
    const SlabLut<PREC, REAL, LUTM> lut(r, sm);
    pdl_wait();
    const V* __restrict__ xs = (const V*)r.xs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lim = (unsigned)r.n_lut << r.colbits;
    const unsigned tile = (unsigned)r.tile0 + blockIdx.x * (HX_THREADS / 128) + warp / 4;
    const bool act = tile < (unsigned)(r.tile0 + r.n_tiles);
    V sum = czero<V>();
    if (act) {
        unsigned q = r.moff[tile] >> 2;
        const unsigned q1 = r.moff[tile + 1] >> 2;
        const unsigned* __restrict__ tp = r.tab + ((size_t)q * 32 + lane) * 4 + (warp & 3);
        unsigned e = *tp;   // (a pass ends with two groups of padding entries)
        for (; q < q1; ++q) {
            const V x0 = xs[e & r.colmask];
            tp += 128;
            const unsigned en = *tp;
            fma_if(sum, lut(e >> r.colbits), x0, e, lim);
            e = en;
        }
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    if (act && (warp & 3) == 0) {
        const V* p = part + threadIdx.x;
        finish_row<PREC>(r, (long long)tile * 32 + lane, cadd(cadd(p[0], p[32]), cadd(p[64], p[96])), true);
    }
    if (!r.early) pdl_launch_dependents();
}

// The same through a table with masks (large sectors in many passes, where padding would double the
// table: on 6x6 it would take 54 ms instead of 64, and 164 GB instead of 80): a lane finds its entry of a
// step by counting the rows before it, and the pipeline reads the next group's entries and the masks
// after those; in FP64 all of it a group earlier, for the gathers (6x6 131.4 -> 128.3 ms).
template <int PREC, bool REAL, int LUTM>
__global__ void __launch_bounds__(HX_THREADS, PREC == 0 ? 3 : 4) hx_slab_kernel(const SlabRun r) {
    typedef typename Cx<PREC>::V V;
    constexpr bool AHEAD = PREC == 0;
    extern __shared__ __align__(16) unsigned char sm[];
    if (r.early) pdl_launch_dependents();
    const SlabLut<PREC, REAL, LUTM> lut(r, sm);
    pdl_wait();
    const V* __restrict__ xs = (const V*)r.xs;
    const unsigned* __restrict__ tab = r.tab;
    const unsigned* __restrict__ mask = r.mask;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const unsigned bit = 1u << lane, below = bit - 1u;
    // (rows are below 2^32, so tiles below 2^27)
    const unsigned tile_end = (unsigned)(r.tile0 + r.n_tiles), hop = gridDim.x * wpb * r.chunk;
    for (unsigned c0 = (unsigned)r.tile0 + (blockIdx.x * wpb + warp) * r.chunk; c0 < tile_end; c0 += hop) {
        unsigned tile = c0;
        const unsigned t1 = min(c0 + r.chunk, tile_end);
        unsigned e0 = ld_stream(r.off + tile);
        unsigned k = r.moff[tile], kt = r.moff[tile + 1];
        const unsigned k1 = r.moff[t1];   // the tiles' steps (each tile has a multiple of four)
        // m: the masks of this group, mn: of the next ones; x: the elements of this group (AHEAD) and
        // id: their coefficients; e: the entries of this group, or (AHEAD) of the next
        constexpr int NEXT = AHEAD ? 2 : 1;
        unsigned m[4], mn[NEXT][4], e[4], id[4];
        V x[4];
        ld_masks(mask, k, k1, m);
#pragma unroll
        for (int d = 0; d < NEXT; ++d) ld_masks(mask, k + 4 * (d + 1), k1, mn[d]);
        ld_entries(tab, m, below, e0, e);
        if (AHEAD) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                x[h] = xs[e[h] & r.colmask];
                id[h] = e[h] >> r.colbits;
            }
            ld_entries(tab, mn[0], below, e0, e);
        }
        for (; tile < t1; ++tile) {
            const unsigned kn = tile + 1 < t1 ? r.moff[tile + 2] : kt;
            V sums[PREC == 0 ? 1 : 4] = {};   // partial sums, as hx_slab_pad_kernel's
            unsigned rows_on = 0;             // rows of the tile with entries in this pass
            for (; k < kt; k += 4) {
                V xn[4];
                unsigned idn[4], m2[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    xn[h] = xs[e[h] & r.colmask];
                    idn[h] = e[h] >> r.colbits;
                }
                ld_entries(tab, mn[NEXT - 1], below, e0, e);
                ld_masks(mask, k + 4 * (NEXT + 1), k1, m2);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    rows_on |= m[h];
                    if (PREC == 0 && h > 0 && m[h] == 0u) continue;
                    fma_if(sums[PREC == 0 ? 0 : h], lut(AHEAD ? id[h] : idn[h]), AHEAD ? x[h] : xn[h], ~m[h] & bit, 1u);
                }
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    x[h] = xn[h];
                    id[h] = idn[h];
                    m[h] = mn[0][h];
#pragma unroll
                    for (int d = 0; d + 1 < NEXT; ++d) mn[d][h] = mn[d + 1][h];
                    mn[NEXT - 1][h] = m2[h];
                }
            }
            V acc = sums[0];
            if constexpr (PREC != 0) acc = cadd(cadd(acc, sums[1]), cadd(sums[2], sums[3]));
            finish_row<PREC>(r, (long long)tile * 32 + lane, acc, (rows_on & bit) != 0u);
            kt = kn;
        }
    }
    if (!r.early) pdl_launch_dependents();
}

// The same through a table with the rows' counts (where the caller's limit has no room for masks): step k's
// rows are those with more than k entries, so the masks come from ballots.  Its targets do not lie by bond
// (triangular 6x5 at k = 1, complex64 905 us, 674 padded by bond; complex128, where the FP64 pipe sets the pace,
// 3443 and 3448, 3554 without the gathers ahead).
template <int PREC, bool REAL, int LUTM>
__global__ void __launch_bounds__(HX_THREADS, PREC == 0 ? 3 : 4) hx_slab_counted_kernel(const SlabRun r) {
    typedef typename Cx<PREC>::V V;
    constexpr bool AHEAD = PREC == 0;
    extern __shared__ __align__(16) unsigned char sm[];
    if (r.early) pdl_launch_dependents();
    const SlabLut<PREC, REAL, LUTM> lut(r, sm);
    pdl_wait();
    const V* __restrict__ xs = (const V*)r.xs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const unsigned bit = 1u << lane, below = bit - 1u;
    const long long tile_end = r.tile0 + r.n_tiles, hop = (long long)gridDim.x * wpb;
    for (long long tile = r.tile0 + (long long)blockIdx.x * wpb + warp; tile < tile_end; tile += hop) {
        const long long row = tile * 32 + lane;
        const unsigned cnt = row < r.n_rows ? ld_stream(r.cnt + row) : 0u;
        const unsigned steps = __reduce_max_sync(0xffffffffu, cnt);
        unsigned e0 = ld_stream(r.off + tile);
        // this row's entry of step k, moving e0 past the step (0 without one)
        auto next = [&](unsigned k) {
            const unsigned m = __ballot_sync(0xffffffffu, k < cnt);
            const unsigned e = k < cnt ? ld_stream(r.tab + e0 + (unsigned)__popc(m & below)) : 0u;
            e0 += (unsigned)__popc(m);
            return e;
        };
        V sums[PREC == 0 ? 1 : 4] = {};   // partial sums, as hx_slab_pad_kernel's
        // (AHEAD as in the masked kernel: x and id of this group, e the entries of the next)
        V x[4];
        unsigned e[4], id[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) e[h] = next(h);
        if (AHEAD) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                x[h] = xs[e[h] & r.colmask];
                id[h] = e[h] >> r.colbits;
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) e[h] = next(4 + h);
        }
        for (unsigned k = 0; k < steps; k += 4) {
            V xn[4];
            unsigned idn[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                xn[h] = xs[e[h] & r.colmask];
                idn[h] = e[h] >> r.colbits;
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) e[h] = next(k + (AHEAD ? 8 : 4) + h);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (PREC == 0 && h > 0 && k + h >= steps) continue;
                fma_if(sums[PREC == 0 ? 0 : h], lut(AHEAD ? id[h] : idn[h]), AHEAD ? x[h] : xn[h], k + h, cnt);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                x[h] = xn[h];
                id[h] = idn[h];
            }
        }
        V acc = sums[0];
        if constexpr (PREC != 0) acc = cadd(cadd(acc, sums[1]), cadd(sums[2], sums[3]));
        finish_row<PREC>(r, row, acc, cnt != 0u);
    }
    if (!r.early) pdl_launch_dependents();
}

// x_c -> sqrt(|O_c|) x_c over the columns [c0, c1)
template <typename V, typename R>
__global__ void k_slab_xscale(const V* __restrict__ x, const unsigned char* __restrict__ cls,
                              const R* __restrict__ scale, V* __restrict__ out, long long c0, long long c1) {
    for (long long c = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < c1;
         c += (long long)gridDim.x * blockDim.x) {
        const R f = scale[cls[c]];
        V v = x[c];
        v.x *= f;
        v.y *= f;
        out[c] = v;
    }
}

// the same from complex128 to complex64: x_c rounded to complex64, then scaled in FP32 (as the
// device-buffer path scales a complex64 x)
__global__ void k_slab_xscale_c128_c64(const double2* __restrict__ x, const unsigned char* __restrict__ cls,
                                       const float* __restrict__ scale, float2* __restrict__ out, long long c0,
                                       long long c1) {
    for (long long c = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x; c < c1;
         c += (long long)gridDim.x * blockDim.x) {
        const float f = scale[cls[c]];
        const double2 v = x[c];
        out[c] = make_float2((float)v.x * f, (float)v.y * f);
    }
}

int xscale_blocks(long long n) {
    const long long need = (n + 255) / 256;
    return (int)std::max<long long>(1, std::min<long long>(need, (long long)sm_count() * 8));
}

template <typename K>
void slab_pdl_launch(K kern, const SlabRun& r, int blocks, int threads, size_t smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EDGPU_CUDA(cudaLaunchKernelEx(&cfg, kern, r));
}

// A launch over n_warps warps of work.  With blocks_per_sm the block has half its usual size, so that an SM's
// share can be cut finely: four blocks of 256 fit, and one of them is too much to leave free (6x6 from host
// buffers, two row blocks: 89.5 ms, 103 with blocks of 256).
template <typename K>
void slab_go(K kern, SlabRun r, size_t smem, long long n_warps, cudaStream_t st) {
    const int threads = r.blocks_per_sm ? HX_THREADS / 2 : HX_THREADS;
    int own = 0, *occ = r.blocks_per_sm ? &own : r.occ;   // (the query costs a microsecond of the host's five per launch)
    if (*occ == 0) {
        raise_smem_limit((const void*)kern, smem);
        EDGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, threads, smem));
        *occ = std::max(1, *occ);
    }
    int n = *occ;
    if (r.blocks_per_sm > 0) n = std::min(n, r.blocks_per_sm);
    else if (r.blocks_per_sm < 0) n = std::max(1, n + r.blocks_per_sm);
    const long long need = (n_warps + threads / 32 - 1) / (threads / 32);
    const int blocks = (int)std::max<long long>(1, std::min<long long>(need, (long long)n * sm_count()));
    r.early = pdl_early(blocks);
    slab_pdl_launch(kern, r, blocks, threads, smem, st);
}

template <typename W, int PREC>
void slab_build_t(int pass, const HxParams& p, const SlabBuild& s, cudaStream_t st) {
    int threads = HX_THREADS;
    if (pass == 2)   // as many warps as have room for their scratch (one always has)
        while (threads > 32 && (size_t)s.o_scratch + threads / 32 * slab_fill_words(s.cap, s.n_pass) * 4 > SLAB_FILL_SMEM)
            threads /= 2;
    const size_t smem = (size_t)s.o_scratch + (pass == 1 ? (size_t)s.n_pass * HX_THREADS
                                                         : threads / 32 * slab_fill_words(s.cap, s.n_pass) * 4);
    auto k = pass == 1 ? hx_slab_count_kernel<W, PREC> : hx_slab_fill_kernel<W, PREC>;
    raise_smem_limit((const void*)k, smem);
    const long long warps = threads / 32;
    const long long need = (s.n_tiles + warps - 1) / warps;
    const int blocks = (int)std::max<long long>(1, std::min<long long>(need, (long long)sm_count() * 16));
    k<<<blocks, threads, smem, st>>>(p, s);
    EDGPU_CUDA(cudaGetLastError());
}

}  // namespace

void hx_slab_build(bool w32, int prec, int pass, const HxParams& p, const SlabBuild& s, cudaStream_t st) {
    if (w32) {
        if (prec == 0) slab_build_t<unsigned, 0>(pass, p, s, st);
        else slab_build_t<unsigned, 1>(pass, p, s, st);
    } else {
        if (prec == 0) slab_build_t<unsigned long long, 0>(pass, p, s, st);
        else slab_build_t<unsigned long long, 1>(pass, p, s, st);
    }
}

void hx_slab_scan(const unsigned* tile_sum, unsigned* off, int n_pass, long long n_tiles,
                  std::vector<unsigned long long>& totals, cudaStream_t st) {
    totals.assign((size_t)n_pass, 0);
    if (n_pass == 0 || n_tiles == 0) return;
    const int nb = (int)((n_tiles + SLAB_CHUNK - 1) / SLAB_CHUNK);
    unsigned long long* part = nullptr;
    unsigned long long* tot = nullptr;
    EDGPU_CUDA(cudaMalloc(&part, (size_t)nb * n_pass * sizeof(unsigned long long)));
    cudaError_t e = cudaMalloc(&tot, (size_t)n_pass * sizeof(unsigned long long));
    if (e != cudaSuccess) {
        cudaFree(part);
        throw Error(EDGPU_ERR_OOM, std::string("slab scan: ") + cudaGetErrorString(e));
    }
    const dim3 grid((unsigned)nb, (unsigned)n_pass);
    k_slab_scan_part<<<grid, HX_THREADS, 0, st>>>(tile_sum, n_tiles, part, nb);
    k_slab_scan_mid<<<n_pass, 1024, 0, st>>>(part, nb, tot);
    k_slab_scan_out<<<grid, HX_THREADS, 0, st>>>(tile_sum, n_tiles, part, nb, off);
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(totals.data(), tot, (size_t)n_pass * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(part);
    cudaFree(tot);
    if (e != cudaSuccess) throw Error(EDGPU_ERR_CUDA, std::string("slab scan: ") + cudaGetErrorString(e));
}

template <int PREC, bool REAL, int LUTM>
void slab_launch_k(const SlabRun& r, size_t smem, cudaStream_t st) {
    const long long warps = (r.n_tiles + r.chunk - 1) / r.chunk;
    if (r.padded) {
        // a block per HX_THREADS / (32 ways) tiles
        auto shared_tiles = [&](auto k, int ways) {
            if (*r.occ == 0) {
                raise_smem_limit((const void*)k, smem);
                *r.occ = 1;
            }
            SlabRun s = r;
            const int blocks = (int)((r.n_tiles * 32 * ways + HX_THREADS - 1) / HX_THREADS);
            s.early = pdl_early(blocks);
            slab_pdl_launch(k, s, blocks, HX_THREADS, smem, st);
        };
        if (r.split == SLAB_BY_PLACE) {
            shared_tiles(hx_slab_place_kernel<PREC, REAL, LUTM>, 4);
            return;
        }
        if (r.split) {
            constexpr int WAYS = PREC == 0 ? 8 : 4;
            shared_tiles(hx_slab_split_kernel<PREC, REAL, LUTM, WAYS>, WAYS);
            return;
        }
        auto go = [&](auto k) { slab_go(k, r, smem, warps, st); };
        if constexpr (PREC == 0) {
            if (!r.in_order && r.n_rows <= SLAB_FP64_SUMS * 32) go(hx_slab_pad_kernel<PREC, REAL, LUTM, 4>);
            else go(hx_slab_pad_kernel<PREC, REAL, LUTM, 1>);
        } else if (r.two_sums) go(hx_slab_pad_kernel<PREC, REAL, LUTM, 2>);
        else go(hx_slab_pad_kernel<PREC, REAL, LUTM, 4>);
    } else if (r.cnt) {
        slab_go(hx_slab_counted_kernel<PREC, REAL, LUTM>, r, smem, r.n_tiles, st);
    } else {
        slab_go(hx_slab_kernel<PREC, REAL, LUTM>, r, smem, warps, st);
    }
}

template <int PREC>
void slab_launch_p(const SlabRun& r, size_t smem, cudaStream_t st) {
    if (r.lut_real) {
        if (r.lut_mode == 2) slab_launch_k<PREC, true, 2>(r, 0, st);
        else slab_launch_k<PREC, true, 0>(r, smem, st);
    } else {
        if (r.lut_mode == 1) slab_launch_k<PREC, false, 1>(r, smem, st);
        else slab_launch_k<PREC, false, 0>(r, smem, st);
    }
}

void hx_slab_launch(int prec, const SlabRun& run, cudaStream_t st) {
    if (run.n_tiles == 0) return;
    SlabRun r = run;
    // Consecutive tiles of a warp: about 128 steps together (the pipeline fills once for them), but at
    // least four chunks for every warp that fits, so that none is left with the last long one.
    r.chunk = (int)std::max<long long>(1, std::min<long long>({16, 128 / std::max(1, r.tile_steps),
                                                              r.n_tiles / ((long long)sm_count() * 48 * 4)}));
    const size_t csize = (size_t)(r.lut_real ? 1 : 2) * (prec == 0 ? 8 : 4);
    const size_t smem = (size_t)(r.n_lut + 1) * (r.lut_mode == 1 ? 128 : csize);   // (and a padding entry's id)
    // (by the table's tiles, not the launch's: row blocks add up alike)
    if (r.padded)
        r.split = slab_split(prec, r.in_order, r.first && r.last, (r.n_rows + 31) / 32, r.tile_steps, r.lut_real, smem);
    if (prec == 0) slab_launch_p<0>(r, smem, st);
    else slab_launch_p<1>(r, smem, st);
}

void launch_slab_xscale(int prec, const void* x, const unsigned char* cls, const void* scale, void* out,
                        int64_t c0, int64_t c1, cudaStream_t st) {
    if (c1 <= c0) return;
    const int blocks = xscale_blocks(c1 - c0);
    if (prec == 0)
        k_slab_xscale<double2, double><<<blocks, 256, 0, st>>>((const double2*)x, cls, (const double*)scale,
                                                              (double2*)out, c0, c1);
    else
        k_slab_xscale<float2, float><<<blocks, 256, 0, st>>>((const float2*)x, cls, (const float*)scale,
                                                            (float2*)out, c0, c1);
    EDGPU_CUDA(cudaGetLastError());
}

void launch_slab_xscale_c128_c64(const double* x, const unsigned char* cls, const float* scale, float* out,
                                 int64_t c0, int64_t c1, cudaStream_t st) {
    if (c1 <= c0) return;
    k_slab_xscale_c128_c64<<<xscale_blocks(c1 - c0), 256, 0, st>>>((const double2*)x, cls, scale, (float2*)out,
                                                                  c0, c1);
    EDGPU_CUDA(cudaGetLastError());
}

}  // namespace edgpu
