// Internal declarations shared by the translation units of libedgpu.so.
#pragma once

#include <cstdint>
#include <cstddef>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/edgpu.h"

namespace edgpu {

struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define EDGPU_CUDA(call)                                                                               \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess)                                                                         \
            throw ::edgpu::Error(e_ == cudaErrorMemoryAllocation ? EDGPU_ERR_OOM : EDGPU_ERR_CUDA,     \
                                 std::string(#call) + ": " + cudaGetErrorString(e_));                 \
    } while (0)

enum GroupKind { GK_TRIVIAL = 0, GK_TORUS = 1, GK_GENERIC = 2, GK_RING = 3 };
// Product-kernel flavour for targets looked up in a parent-state map (no canonicalisation code).
constexpr int GK_MAP = 4;
// Pair-flip product flavour that reads every target's map-format entry from the operator's target
// table (row after row, in the schedule's order) instead of looking it up.
constexpr int GK_TABLE = 5;

// Symmetry group acting on basis words: element g maps word q to g.q.
//  TRIVIAL  the identity only (unreduced representation).
//  TORUS    translations T(a,b) of an L1 x L2 torus of w-bit sites numbered x + L1*y;
//           g = a + L1*b; T(a,b).q rotates every row of L1*w bits left by a*w and the rows
//           up by b rows.  num[] is in this order.
//  GENERIC  arbitrary site permutations (+ XOR flip), applied through 4-bit chunk tables.
//  RING     (product kernel only) a TORUS with L2 == 1 in 32-bit words: funnel-shift rotations.
struct Group {
    int kind = GK_TRIVIAL;
    int G = 1;
    int den = 1;
    std::vector<int32_t> num{0};     // character numerators: chi(g) = exp(2 pi i num[g] / den)
    int L1 = 1, L2 = 1, w = 1;       // TORUS
    std::vector<int32_t> maps;       // GENERIC: [G][n_sites] site maps in user order
    std::vector<uint64_t> flips;     // GENERIC: [G]
};

struct Layout {
    int n_sites = 0, nbits = 0, qlen = 0;
    std::vector<int32_t> dims, bw, off;
    std::vector<int64_t> state_qn;   // [sum(dims)][qlen], site-major
    std::vector<int64_t> allowed;    // [n_allowed][qlen]
    bool all_sectors = false;
    int popcount = -1;               // >= 0: spin-1/2-like sector = all words of nbits with this popcount
};

struct VectorTables;

struct Space {
    Layout lay;
    bool reduced = false;
    bool lazy = false;
    Space* parent = nullptr;         // reduced: the parent representation (not owned)
    Group group;
    int64_t dim = 0;
    bool w32 = false;                // keys are uint32 (nbits + sb <= 32) else uint64
    int sb = 0;                      // low key bits holding the orbit-size index (0: unreduced)
    void* d_keys = nullptr;          // sorted keys: (state << sb) | orbit-size index
    unsigned long long* d_dir = nullptr;   // search directory of bucket summaries (see DirSearch)
    int dir_shift = 0;               // bucket of a state = state >> dir_shift
    long long dir_nb = 0;            // number of buckets (entry dir_nb is a sentinel)
    int dir_steps = 0;               // ceil(log2(largest bucket)) for buckets searched in the keys
    int dir_K = 0;                   // keys summarised inline per bucket
    double dir_inline = 0.0;         // fraction of keys in buckets answered by their summary
    // Parent-state map of a reduced table whose parent is one fixed-popcount sector (optional):
    // entry r, for the parent state q of colex rank r (its index in the sorted parent basis; or r = q
    // itself when the map is direct), holds the
    // index c of q's representative | orbit-size index << map_cb | group element g (g.q = rep)
    // << (map_cb + sb), or all ones when q's orbit has no representative in the table.
    void* d_map = nullptr;
    int map_wide = 0;                // entries are uint64 (else uint32)
    int map_cb = 0;                  // bits of the index field
    int map_direct = 0;              // entries indexed by the state itself (2^nbits entries), not the rank
    int64_t map_n = 0;               // entries: C(nbits, popcount), or 2^nbits when direct
    void* d_rank = nullptr;          // colex rank chunk table [chunk][ones before][64 values]
    int rank_wide = 0;               // rank table entries are uint64 (else uint32)
    int rank_split = 0;              // > 0: split rank tables A (high bits) and B (rank_split low bits)
    uint64_t map_gen = 0;            // bumped whenever the map is built or freed
    mutable VectorTables* vec = nullptr;   // tables of the vector maps to and from the parent (on first use)
    // a parent's split colex rank tables for the vector maps of all its reduced spaces (parent_rank_table)
    mutable void* d_vec_rank = nullptr;
    mutable std::mutex vec_rank_mu;
    ~Space();
};
// Build (or free) the parent-state map of a reduced space; false when it does not apply or would
// exceed max_bytes.
bool build_parent_map(Space& red, int64_t max_bytes, cudaStream_t st);
void free_parent_map(Space& red);
constexpr int RANK_CHUNK = 6;      // bits per chunk of the colex rank tables

// ---- device-side descriptors -------------------------------------------------------------------

struct GroupDev {
    int kind, G, den;
    int L1, L2, w, rowbits, nbits, nchunks;
    unsigned long long full;
    const int32_t* num;              // [G]
    const unsigned long long* keep;  // [L1] TORUS row-rotation masks (bits that do not wrap)
    const unsigned long long* lut;   // [G][nchunks][16] GENERIC
    const unsigned long long* flips; // [G] GENERIC
};

struct SectorDev {
    int n_sites, qlen, n_allowed, all_sectors;
    const int32_t* off;
    const int32_t* bw;
    const int32_t* dims;
    const int32_t* qbase;            // [n_sites] first local-state row of each site in qn
    const long long* qn;             // [sum dims][qlen]
    const long long* allowed;        // [n_allowed][qlen]
};

// Device copy of a Group (owned).
struct GroupBuffers {
    GroupDev dev{};
    unsigned long long* d_all = nullptr;
    const int32_t* divi = nullptr;   // [d]: index of d among the divisors of G
    void upload(const Group& g, const Layout& lay);
    void release();
    ~GroupBuffers() { release(); }
};

// Device tables of a reduced space's vector maps (reduce_vector): amplitudes chi sqrt(|stab| / |G|) by
// (orbit-size index, character numerator), phases by numerator and sqrt(|stab| / |G|) / |stab| by orbit-size
// index.
struct VectorTables {
    struct Dev {
        const double2* ampl;
        const double2* phase;
        const double* inv_norm;
        const void* rank;              // the parent's split rank tables (set for a reduction only)
        long long rank_hi;             // entries of the high part's table
        int rank_split, rank_wide;     // low bits (0: no tables), 64-bit entries
        int by_rank;                   // a parent index is the state's colex rank
        int popcount;                  // by_rank: the parent's words are all those of this many set bits
        int elem_bits;                 // index bits beside a 32-bit ring state
    };
    GroupBuffers gb;
    double2* d_ampl = nullptr;
    double* d_inv = nullptr;
    Dev dev{};
    VectorTables() = default;
    VectorTables(const VectorTables&) = delete;
    ~VectorTables();
};

// Host helpers used by several units.
std::vector<unsigned long long> torus_keep_masks(const Group& g, int nbits);
std::vector<unsigned long long> generic_luts(const Group& g, const Layout& lay, int* nchunks);

// ---- enumeration (enumerate.cu) ---------------------------------------------------------------
cudaStream_t lib_stream();
// Raise a kernel's dynamic shared-memory limit to at least smem bytes, never lowering it, under a
// process-wide lock (launches from several host threads must not leave a smaller limit in place).
void raise_smem_limit(const void* kern, size_t smem);
int sm_count();
void enumerate_parent(Space& s, cudaStream_t st);
void enumerate_reps(Space& red, const Space& parent, cudaStream_t st);
void build_mapping(const Space& red, const Space& parent, int64_t* index_out, double* ampl_out, cudaStream_t st);
void orbit_sizes(const Space& red, int32_t* out_host, cudaStream_t st);
void lookup_keys(const Space& s, const uint64_t* keys_host, int64_t n, int64_t* out_host, cudaStream_t st);
// Number of index bits for the divisors of G, and the divisor index of every stabiliser size.
int orbit_index_bits(int G);
// Builds the search directory of any table.
void build_search_directory(Space& s, cudaStream_t st);
void get_states(const Space& s, uint64_t* out_host, cudaStream_t st);
// Vectors between a reduced space and its parent on the device (symmetry_unreduce / symmetry_reduce):
// unreduce: out[n_parent] from in[dim]; reduce: out[dim] from in[n_parent].  complex128 (EDGPU_FP64) or
// complex64 (EDGPU_MIXED) vectors; the parent is materialised or a lazy popcount sector.
void reduce_vector(const Space& red, const Space& parent, int prec, bool unreduce, const void* in, void* out,
                   cudaStream_t st);
int64_t parent_dimension(const Space& parent);
// Diagonal element of every row: sum of the amplitudes of the row == col terms matching the row's state
// (FP64), written as complex128 (out64) and/or complex64 (out32).  scratch: device room for the T terms
// (4 words each), or null to allocate it for the call.
void compute_diagonal(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const double* amps,
                      double* out64, float* out32, unsigned long long* scratch, cudaStream_t st);
// Off-diagonal targets of every row (T terms: masks/rows/flips = row ^ col) and how many land in the table.
void count_nnz(const Space& s, int T, const uint64_t* masks, const uint64_t* rows, const uint64_t* flips,
               int64_t* n_targets, int64_t* n_found, cudaStream_t st);

constexpr int TORUS_MAXR = 8;      // most rows of a torus canonicalised with top-row pruning

// Search directory of a key table (bucket summaries; see key_find_sum2 in edgpu_device.cuh) with the
// constants of the in-register compare of a bucket's K member fields (mb bits each):
// unit = 1 in the lowest bit of every field, keybits = the state bits of every field (above the sb
// orbit-index bits), low = all but the top bit of every field, top = the top bit of every field.
struct DirSearch {
    const unsigned long long* dir;
    long long nb;
    int shift, mb, K, steps, sb;
    unsigned unit, keybits, low, top;
};
DirSearch dir_search_of(const Space& s);

// ---- matrix-free product (hx*.cu) ----------------------------------------------------------------
struct HxParams {
    const void* keys;
    long long n_rows;
    const void* x;
    void* y;
    const void* gy;
    double* grad_partial;
    int accumulate, rows_per_tile, n_coupl;
    const void* blob;
    int blob_words16;
    int o_om, o_or, o_of, o_oa, o_ou, o_oc;   // off-diagonal terms: mask,row,flip,amp,unit amp,coupling id
    int o_dm, o_dr, o_da, o_du, o_dc;         // diagonal terms
    DirSearch ds;                             // the search directory of the table
    const void* diag;                         // per-row diagonal element (V), product mode
    int o_ph, o_num, o_ratio, o_keep, o_lut, o_flip, o_grad;
    const void* lut_g;                        // GENERIC permutation tables in global memory (o_lut < 0)
    int o_rlut;                               // torus row table for top-row pruning, -1 when absent
    unsigned l1inv;                           // ceil(2^16 / L1) (candidate bit -> row of the pruned torus search)
    int rlut_pair;                            // the row table holds pairs of rows (rowbits <= 6)
    int o_keep32;                             // the torus keep masks as 32-bit words (states of <= 32 bits)
    int T_o, T_d, G, den, nd;
    int L1, L2, w, rowbits, nbits, nchunks;
    int sb, pb, want_arg, lpr;
    unsigned long long full;
    int warp_base;
    int o_sec, n_sec;                         // batched launch: shared-memory offset and count of SectorDesc
    long long n_tiles;                        // batched launch: warp tiles over all sectors
    // parent-state map (replaces canonicalisation and search when map != null)
    const void* map;
    int map_wide, map_cb, map_direct;
    const void* rank_tab;                     // colex rank chunk table
    int rank_wide, rank_k, rank_nc;           // entry width, popcount of the parent sector, chunks
    int rank_split;                           // > 0: rank = A[q >> rank_split] + B[q & low bits]
    // pair-flip schedule (hx_bond.cuh): bond classes of the off-diagonal terms, 0 when the terms are not
    // all two-site flips of 1-bit sites
    int bond_ncls;
    int o_bcomp, o_binfo, o_bflip, o_bamp;    // shared-memory offsets of the class tables
    int bond_real;                            // every pair amplitude is real
    int bond_slot;                            // >= 0: every pair that can match has this slot's amplitude, whatever
                                              // the couplings (its value is read from the image, which a change of
                                              // couplings rewrites under launches already captured)
    int bond_nt;                              // targets per lane and step: 2, or 4 (parent-state map only)
    int bond_pf;                              // target tables: x prefetched this many steps ahead (0: none)
    int bond_uni;                             // target tables: warp-uniform pair steps (bond_tile UNI)
    // gradient mode of the pair-flip kernel (offsets into its shared-memory image, -1 when absent): the
    // slots' unit amplitudes and coupling ids, and the diagonal term records
    int o_bunit, o_bcid, o_pdm, o_pdr, o_pdu, o_pdc;
    int bunit_real;                           // every unit pair amplitude is real
    // the diagonal records by site pair (n_pdb entries; -1: a record has a mask of more than two bits):
    // i | j << 8 | coupling id << 16, and per entry the unit amplitudes of the pair's four bit patterns
    int o_pdb, o_pdv, n_pdb;
    // FP64 gradient with one unit amplitude (build_blob): amplitude, the diagonal terms' change on a match over
    // it, offset of their value without one by coupling; no_y: only the gradient is wanted
    int early;                 // the next launch may start with this one (set by the launch, see pdl_early)
    int grad_one, o_gbase, no_y;
    double grad_u, grad_kz;
    // adjoint target table (column-sorted; built by the ADJ passes of bond_tile): per column the
    // count, the offset of its run, a fill cursor, and the entries (row << 32 | slot << 19 |
    // row's orbit-size index << 14 | group element)
    unsigned* adj_cnt;
    const long long* adj_off;
    unsigned* adj_cur;
    unsigned long long* adj_tab;
    // target table of the pair-flip schedule (GK_TABLE launches and the table's build pass)
    const void* tab;
    const long long* tile_off;
    int tab_wide, tab_cb;
    void* y_c128;                             // mixed precision: write y as complex128 here instead (or null)
};

// One sector of a batched launch (hx_multi_kernel), kept in shared memory after the common tables.
// The term, group and orbit-normalisation tables are common to all sectors; the basis table, its
// search directory, the diagonal, the vectors and the character table belong to the sector.
struct __align__(16) SectorDesc {
    const void* keys;
    const void* x;
    void* y;
    const void* diag;
    long long n_rows;
    long long tile_end;                       // cumulative warp tiles through this sector
    DirSearch ds;
    const void* map;                          // the sector's parent-state map (or null)
    int map_wide, map_cb, map_direct;
    int o_ph, o_num, want_arg;
    const void* tab;                          // the sector's target table (pair-flip schedule, or null)
    const long long* tile_off;
    int tab_wide, tab_cb;
};

constexpr int BOND_MAXC = 4;       // rotation components per bond class of the pair-flip schedule
constexpr int BOND_MAXCLS = 24;    // bond classes at most (more: the term-matching schedule)

constexpr size_t GENERIC_SMEM_LUT = 64 * 1024;   // larger GENERIC permutation tables stay in global memory
constexpr int HX_QCAP = 128;         // per-warp target queue capacity (entries; 2 batches of 32 + 31)
constexpr int HX_THREADS = 256;      // threads per block of the product kernel
int hx_warp_bytes(bool w32);

// Launch the product kernel for (word width, group kind, precision, gradient mode).
void hx_launch_w32(int gk, int prec, int mode, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_launch_w64(int gk, int prec, int mode, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_max_blocks_per_sm(bool w32, int gk, int prec, int mode, size_t smem);
// Row-per-lane strategy (hx_rows.cuh), product mode only.
void hx_rows_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_rows_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_rows_occupancy_w32(int gk, int prec, size_t smem);
int hx_rows_occupancy_w64(int gk, int prec, size_t smem);
// Sparse assembly of a representation in FP64 (hx_rows.cuh, hx_sparse_kernel); shared memory:
// the blob's warp_base plus 4 warps x (T_o + 1) x 48 bytes.
void hx_sparse_launch_w32(int gk, const HxParams& p, long long row0, long long n_run, int conj_vals, double tol,
                          long long* counts, const long long* row_ptr, long long* cols, double2* vals, size_t smem,
                          cudaStream_t st);
void hx_sparse_launch_w64(int gk, const HxParams& p, long long row0, long long n_run, int conj_vals, double tol,
                          long long* counts, const long long* row_ptr, long long* cols, double2* vals, size_t smem,
                          cudaStream_t st);
// Row-per-lane gradient mode (hx_rows_kernel MODE 1): shared memory o_grad + n_coupl x HX_THREADS x 8.
void hx_rows_grad_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_rows_grad_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_rows_grad_occupancy_w32(int gk, int prec, size_t smem);
int hx_rows_grad_occupancy_w64(int gk, int prec, size_t smem);
// Adjoint of the product's matrix by scatter (hx_rows.cuh, hx_scatter_adjoint_kernel): p.gy = input,
// p.y = output (zeroed or accumulated by the caller); shared memory as the row-per-lane kernel.
void hx_scatter_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_scatter_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
// Batched sectors in one persistent launch (hx_rows.cuh, hx_multi_kernel), product mode only.
void hx_multi_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_multi_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_multi_occupancy_w32(int gk, int prec, size_t smem);
int hx_multi_occupancy_w64(int gk, int prec, size_t smem);

// Pair-flip schedule (hx_bond.cuh), product mode only: one sector, and all sectors of a batch.
void hx_bond_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_bond_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_bond_occupancy_w32(int gk, int prec, int nt, size_t smem);
int hx_bond_occupancy_w64(int gk, int prec, int nt, size_t smem);
void hx_bond_multi_launch_w32(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
void hx_bond_multi_launch_w64(int gk, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_bond_multi_occupancy_w32(int gk, int prec, int nt, size_t smem);
int hx_bond_multi_occupancy_w64(int gk, int prec, int nt, size_t smem);

// Target table of the pair-flip schedule (hxtable.cu): count the targets of every warp tile of 32 rows,
// scan the counts into tile offsets (returns the total), and write every target's map-format entry,
// looked up with flavour gk (GK_MAP or a canonicalising kind).  p: the pair-flip launch template with
// lpr = 1; p.tab / p.tile_off / p.tab_wide / p.tab_cb set for the fill.
void hx_table_count(bool w32, const HxParams& p, long long n_tiles, long long* tile_cnt, size_t smem, cudaStream_t st);
long long hx_table_scan(const long long* tile_cnt, long long n_tiles, long long* tile_off, cudaStream_t st);
void hx_table_fill(bool w32, int gk, const HxParams& p, long long n_tiles, size_t smem, cudaStream_t st);
// The product through the table (GK_TABLE), one sector and all sectors of a batch.
void hx_table_launch(bool w32, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_table_occupancy(bool w32, int prec, int nt, size_t smem, bool uni = false);
void hx_table_multi_launch(bool w32, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_table_multi_occupancy(bool w32, int prec, int nt, size_t smem);
// The product fused with the coupling gradient on the pair-flip schedule (hx_bond.cuh, GRAD mode):
// targets from the target table (table) or the parent-state map, four per lane and step.  Shared
// memory: the pair-flip image up to p.o_grad, then n_couplings x HX_THREADS doubles.
void hx_bond_grad_launch(bool w32, bool table, int prec, const HxParams& p, int blocks, size_t smem, cudaStream_t st);
int hx_bond_grad_occupancy(bool w32, bool table, int prec, size_t smem);
// Adjoint target table (hxtable.cu): pass 1 counts every column's targets (p.adj_cnt), pass 2 writes
// each target's entry into its column's run (p.adj_off, p.adj_cur, p.adj_tab); the runs are then
// sorted so that the summation order is fixed.  p: the table-flavour pair-flip template (lpr = 1).
void hx_adj_pass(bool w32, int pass, const HxParams& p, long long n_tiles, size_t smem, cudaStream_t st);
void hx_adj_sort(const long long* off, unsigned long long* tab, long long n, cudaStream_t st);
// y = H^dagger x through the adjoint target table: one lane per column, its run in order; p.gy = x.
void hx_adj_launch(bool w32, int prec, const HxParams& p, size_t smem, cudaStream_t st);

// ---- column-slab table of the pair-flip schedule (hxslab.cu) -------------------------------------
// The target table's entries regrouped by column slab: slab q holds the columns [q wc, (q + 1) wc).
// Pass q of the product gathers only from slab q (sized to stay in L2 while the pass runs) and adds
// its share to y.  Within a pass and a warp tile of 32 rows the entries lie in steps of at most one entry
// per row: per tile as many as the row with the most entries, rounded up to a multiple of four.  An entry
// is (column - q wc) | id << colbits.  Two forms: padded, 32 entries per step (a row without one has a
// padding entry of id n_ids), four steps of a row side by side; or per step a 32-bit mask of the rows that
// have an entry, and their entries in row order.  Per pass and tile a 32-bit offset of its first step and
// (with masks) of its first entry, relative to the pass ([n_tiles + 1], the last one the total).  Where neither
// fits the caller's limit, a third form: step k holds every row's k-th entry, so that a byte per row and pass, its
// number of entries, takes the masks' place (one pass over long rows has more than eight steps a tile and
// pass, whose masks take more than that); with an offset per tile and pass ([n_tiles]).
// id indexes the coefficient table: id = ((amplitude id x den + character index) x nd +
// orbit-size index of the row) x nd + orbit-size index of the column.
struct SlabBuild {
    long long wc;                   // columns per slab
    int n_pass;
    long long n_tiles;
    unsigned* tile_sum;             // [n_pass][n_tiles] entries (written by the count pass)
    unsigned* tile_steps;           // [n_pass][n_tiles] steps (written by the count pass)
    const unsigned* off;            // [n_pass][n_tiles + 1] first entries relative to the pass (fill pass)
    const unsigned* moff;           // [n_pass][n_tiles + 1] first steps relative to the pass (fill pass)
    const long long* base;          // [n_pass] first entry of each pass (fill pass)
    const long long* mbase;         // [n_pass] first step of each pass (fill pass)
    unsigned* tab;                  // the entries (fill pass)
    unsigned* mask;                 // the steps' row masks (fill pass)
    const unsigned short* amp_id;   // [n_slots] amplitude id of every pair-flip slot (fill pass)
    unsigned char* cls;             // [n_rows] every row's orbit-size index (count pass; null: not kept)
    int n_slots;
    int colbits;
    int scaled;                     // ids without the orbit-size indices (amplitude id x den + character)
    int padded;                     // every step has 32 entries (no masks)
    int in_order;                   // one slab: step k holds every row's k-th entry, in the target table's order
    int counted;                    // the same for any number of slabs, and the rows' counts kept (no masks)
    unsigned char* cnt;             // [n_pass][n_rows] entries of a row in a pass (fill pass, counted)
    int n_ids;                      // coefficient ids (a padding entry has the id n_ids)
    int cap;                        // steps a warp of the fill pass lays out at a time (>= the most of one tile)
    int o_scratch;                  // shared-memory offset of the passes' scratch
};
struct SlabRun {
    const unsigned* off;            // this pass's first entries by tile [n_tiles + 1]
    const unsigned* moff;           // this pass's first steps by tile [n_tiles + 1]
    const unsigned* tab;            // this pass's entries
    const unsigned* mask;           // this pass's steps (null on a padded or counted table)
    const unsigned char* cnt;       // this pass's rows' counts (counted table, whose off is [n_tiles])
    int padded;
    int two_sums;                   // mixed precision, padded: two partial sums per row (else four)
    int in_order;                   // the rows' entries are in the target table's order
    int split;                      // several warps per tile: SLAB_BY_GROUP or SLAB_BY_PLACE (set by hx_slab_launch)
    int early;                      // the next launch may start with this one (set by hx_slab_launch)
    const void* xs;                 // x from the slab's first column
    const void* x;                  // x (first pass: the diagonal's product)
    void* y;
    const void* diag;
    const void* lut;                // coefficients by id: V, or R when lut_real
    void* y_c128;                   // last pass: complex128 output instead of y (host buffers)
    long long n_rows, n_tiles;
    unsigned colmask;
    int colbits, n_lut, lut_real;
    int first, last, accumulate, acc_c128;
    int tile_steps;                 // mean steps of a tile in a pass
    int lut_mode;                   // 0: one shared-memory copy of the coefficients; 1: a copy per
                                    // bank group (conflict-free lookups); 2: real, at most 4, in registers
    // scaled tables: xs and x hold sqrt(|O_c|) x_c; the last pass multiplies row r by 1/sqrt(|O_r|)
    // (and the first pass of y += H x the old y_r by sqrt(|O_r|))
    int scaled;
    const unsigned char* cls;       // [n_rows] orbit-size index of every row
    const void* scale;              // R[2 nd]: sqrt(|O|) by orbit-size index, then 1 / sqrt(|O|)
    int nd;
    long long tile0;                // the launch covers the tiles [tile0, tile0 + n_tiles)
    int chunk;                      // consecutive tiles of a warp (set by hx_slab_launch)
    int* occ;                       // host: resident blocks per SM of the table's kernel (0: not known yet)
    int blocks_per_sm;              // 0: as many as fit; > 0: at most that many; < 0: leave -blocks_per_sm free
};
// A table is padded (32 entries in every step, no masks) where that takes at most this many entries per
// target: the padded product takes a third of the instructions per step (4x8: 1.72 against 2.16 ms, 6x5:
// 0.68 against 0.75 ms), and one pass over a sector needs 1.1 to 1.4; at 18 passes of a few entries per
// row it is above 2, which would double the memory of the largest tables.
// Tables below SLAB_PAD_SMALL steps (2 MB) are always padded.
constexpr double SLAB_PAD_MOST = 1.5;
constexpr int64_t SLAB_PAD_SMALL = 1 << 14;
// One slab of short rows (at most this many steps per tile on average: chains): the rows' entries stay in
// the target table's order.  That fills the steps better, which FP64 gains by (complex128, in order and by bond:
// chain L = 24 9.65 and 11.2 us, L = 26 30.4 and 35.0, L = 28 101 and 104), and costs mixed precision, which reads
// the same table, gathers that share fewer lines (complex64: 4.0 and 3.8 us, 9.6 and 8.9, 31.9 and 30.2).  In
// mixed precision such a row has four partial sums, two from SLAB_TWO_SUMS rows on (chain L = 24 4.0 us, 4.1 with
// four; L = 28 31.9 and 33.3; for 14 to 28 random terms two sums are 9 to 17% further from the 64-bit sum than four,
// and one 21 to 28% further than two).
constexpr int SLAB_IN_ORDER = 32;
constexpr int64_t SLAB_TWO_SUMS = 1 << 16;
// Several warps share a tile of a padded table where the table leaves most of the chip empty and a row's chain
// of gathers and additions sets the time.
// By group, by-bond tables of up to SLAB_SPLIT tiles: each warp takes every fourth (mixed) or eighth (FP64) group of
// steps (triangular 4x4, 28 tiles, complex64 3.6 -> 2.3 us, complex128 11.5 -> 3.9; 5x4, 290 tiles, 5.4 -> 3.6 and
// 23 -> 11).
// By place: four warps, each one step of every group, with the sums of one warp's four partial sums.  In-order
// tables in complex128 up to 1024 tiles (chain L = 14 2.6 us, 4.1 with a warp per tile; L = 20 3.0 and 5.0, 22 4.8
// and 5.4; at 1838 tiles, L = 23, 7.3 and 7.2), in complex64 from 4 to 600 (L = 12, three tiles, 1.95 us and 1.86;
// L = 18 2.1 and 2.3, 21 2.4 and 2.6; at 1003, L = 22, 3.7 and 2.9).  In FP64 with complex coefficients and more
// than 16 steps by group there too (triangular 4x3 at k = 1 3.6 us, 4.1 by place).
// By-bond tables of one pass in complex128 up to SLAB_FP64_SUMS tiles, whose rows have four partial sums: square
// 5x5 48.0 us, 52.8 with a warp per tile and four sums, 49.6 with one sum; triangular 6x4 at k = 1 68.3, 70.1 and
// 67.9.  Larger ones have one sum (7x4, 44600 tiles: 477 us by place, 468 with a warp per tile and one sum).
// A block copies the coefficients for two tiles: only up to 16 KB of them.
enum { SLAB_BY_GROUP = 1, SLAB_BY_PLACE = 2 };
constexpr int64_t SLAB_SPLIT = 400;
constexpr int64_t SLAB_FP64_SUMS = 1 << 14;
inline int slab_split(int prec, bool in_order, bool one_pass, int64_t tiles, int tile_steps, bool real,
                      size_t lut_bytes) {
    const bool few = lut_bytes <= 16 * 1024;
    if (prec != 0 && in_order) return few && tiles >= 4 && tiles <= 600 ? SLAB_BY_PLACE : 0;
    if (in_order && few && tiles <= 1024 && (real || tile_steps <= 16)) return SLAB_BY_PLACE;
    if (tiles <= SLAB_SPLIT) return SLAB_BY_GROUP;
    return prec == 0 && !in_order && one_pass && few && tiles <= SLAB_FP64_SUMS ? SLAB_BY_PLACE : 0;
}
// Coefficient tables of at most this many entries go to registers (real) or to one copy per shared-
// memory bank group (SLAB_REP_BYTES in all, which keeps eight blocks of the slab kernel per SM).
constexpr int SLAB_REG_LUT = 4;
constexpr int SLAB_REP_BYTES = 24 * 1024;
// x_c -> sqrt(|O_c|) x_c for the columns [c0, c1) of x (R = float for complex64, double for complex128;
// scale = the column scales by orbit-size index), written to out at the same columns.  From a complex128
// source to a complex64 result (mixed precision from host buffers) x_c is rounded to complex64 first.
void launch_slab_xscale(int prec, const void* x, const unsigned char* cls, const void* scale, void* out,
                        int64_t c0, int64_t c1, cudaStream_t st);
void launch_slab_xscale_c128_c64(const double* x, const unsigned char* cls, const float* scale, float* out,
                                 int64_t c0, int64_t c1, cudaStream_t st);
// Count pass (1) or fill pass (2) of the slab table from the target table.  p: the table-flavour
// pair-flip template (tab, tile_off set; lpr = 1), whose image ends at s.o_scratch.
void hx_slab_build(bool w32, int prec, int pass, const HxParams& p, const SlabBuild& s, cudaStream_t st);
// Per pass: exclusive scan of the tile sums [n_pass][n_tiles] into 32-bit offsets relative to the
// pass [n_pass][n_tiles + 1]; totals[q] = sum of pass q (host, after a synchronisation).
void hx_slab_scan(const unsigned* tile_sum, unsigned* off, int n_pass, long long n_tiles,
                  std::vector<unsigned long long>& totals, cudaStream_t st);
// One pass of the slab product.
void hx_slab_launch(int prec, const SlabRun& r, cudaStream_t st);

// ---- the coupling-gradient launch for callers that cannot allocate (noalloc.cu) -----------------
// The fused product and coupling gradient exactly as edgpu_coupling_grad_device launches it (same
// kernel choice), with the per-block partial sums written to partial[blocks][n_couplings] and at most
// cap_blocks blocks.  False, with nothing launched or allocated, when the operator's tables for this
// precision (gradient and product mode) have not been built yet.
bool coupling_grad_launch_built(edgpu_op op, int prec, const void* x, const void* gy, void* y, double* partial,
                                int cap_blocks, cudaStream_t st, int* blocks_used);
int coupling_count(edgpu_op op);
int64_t op_dimension(edgpu_op op);
// The call lock of an operator handle (calls on one handle are serialised).
std::unique_lock<std::mutex> lock_op(edgpu_op op);
// Record an error message for edgpu_last_error() and return code.
int record_api_error(int code, const std::string& msg);

// ---- vector kernels (linalg.cu) ------------------------------------------------------------------
void launch_random_c128(int64_t n, uint64_t seed, double* dst, cudaStream_t st);
void launch_c128_to_c64(int64_t n, const double* src, float* dst, cudaStream_t st);
void launch_c64_to_c128(int64_t n, const float* src, double* dst, int accumulate, cudaStream_t st);
void launch_conj_c128(int64_t n, double* v, cudaStream_t st);
// Deterministic FP64 reductions through a per-call scratch buffer of at least dot_scratch_doubles().
size_t dot_scratch_doubles();
// (a norm: |a|, 1 / |a|)
void launch_norm2_c128(int64_t n, const double* a, double* scratch, double* out_dev, cudaStream_t st);
void launch_reduce_grad(int nblocks, int ncoupl, const double* partial, double* out_dev, cudaStream_t st);
// One Lanczos step.  scratch, tickets (one zeroed counter per 16 basis vectors, which each launch leaves
// zero): lanczos_layout.h.  Every null vector or scalar drops its term.
// alpha = <v, w> (re, im); with y32, w is first written as the widened complex64 vector y32.
void launch_lanczos_alpha(int64_t n, const double* v, double* w, const float* y32, double* scratch, unsigned* tickets,
                          double* alpha_dev, cudaStream_t st);
// h = V^H w1 for w1 = w - alpha v - beta u (k vectors, complex128 or complex64), hmax = largest |Re h|, |Im h| of
// every group of vectors (room for one per 16 vectors), nrm2 = |w1|^2; w1 itself is not kept
void launch_lanczos_project(int64_t n, int k, const void* V, bool c64, int64_t ldv, const double* w, const double* v,
                            const double* u, const double* alpha_dev, const double* beta_dev, double* scratch,
                            unsigned* tickets, double* h_dev, double* hmax_dev, double* nrm2_dev, cudaStream_t st);
// w = w1 - alpha v - beta u - V h (w1 may be w), beta_out = |w|, 1 / |w| (hmax, nrm2: those of the projections, null
// for other coefficients h); slot (host memory the device can address): alpha, |w| and
// nrm2 (without one: |w|^2)
void launch_lanczos_correct(int64_t n, int k, const void* V, bool c64, int64_t ldv, const double* h_dev,
                            const double* hmax_dev, const double* w1, const double* v, const double* u,
                            const double* alpha_dev, const double* beta_dev, double* w, double* scratch, unsigned* tickets, double* beta_out,
                            const double* nrm2_dev, double* slot, cudaStream_t st);
// v_next = w / beta (beta_dev: beta, 1 / beta); also writes a complex64 copy when v32 != null
void launch_normalize(int64_t n, const double* w, const double* beta_dev, double* v_next, float* v32,
                      cudaStream_t st);
void launch_axpy_real(int64_t n, double a, const double* x, double* y, cudaStream_t st);

}  // namespace edgpu
