// spg_lock.cu — lock(): merge one epoch of staged inserts into the CSR.
//
// Spira's lock (matrix.hpp:277-342) sorts and dedups every row buffer keeping
// the last write and keeping zeros (aos_array_buffer.hpp:76-101: reverse +
// stable_sort + first-of-run), then either builds the CSR dropping zeros
// (csr_build.hpp:32-98) or two-pointer-merges each dirty row with its old CSR
// slice, the buffer winning on equal columns and a zero deleting
// (csr_build.hpp:126-488). The GPU formulation computes the same CSR:
//
//   1. one pass checks the ranges, tells how the inserts are ordered and samples
//      the rows' lengths and how scattered their columns are;
//   2. inserts in any row order are sorted stably by row (spg_rowsort.cu);
//   3. a first lock sorts, dedups and compacts the grouped rows into the CSR, in
//      one pass over tiles of rows (spg_rowtiles.cu) or by row classes
//      (spg_prims.cu). Rows of more than 12 288 inserts fit neither: they are
//      sorted apart for the tiles, or, where they are most of the inserts, all
//      goes through a global stable radix sort of the keys (row << cbits | col),
//      in which the last element of a run of equal keys is the last write;
//   4. a later epoch of few inserts goes insert by insert (spg_delta.cu); any
//      other becomes a sorted delta (zeros kept) and is merged into the old
//      CSR tile by tile (spg_merge.cu): an equal column takes the delta's
//      value, a zero of the delta deletes.
// Everything is integer work or a copy of the value bits, so structure and
// values are bit-exact against Spira. Capacity follows Spira's rule: the first
// build is tight; a merge keeps the old capacity when old nnz + |D| fits, else grows to 1.5x
// that bound (csr_build.hpp:139-145).
#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int LB = 256;

__global__ void lock_make_keys(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ cols,
                               uint64_t m, int cbits, uint64_t *__restrict__ keys,
                               uint32_t *__restrict__ idx) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        keys[i] = ((uint64_t)rows[i] << cbits) | cols[i];
        idx[i] = (uint32_t)i;
    }
}

// One pass over the staged inserts, which counts (the last block stores the
// counts for the host):
// stats[0] = max row, stats[1] = max column (range check), stats[2] = 1 if
// some key is greater than its successor (not sorted), stats[3] = 1 if some
// row is (rows not grouped), stats[4] = 1 if some key is not below its
// successor (not strictly increasing: duplicates or unsorted).
// Runs of more than GAP_LONG row offsets with one value (empty rows) are
// listed for offsets_fill_gaps (up to GAP_SLOTS of them) rather than written
// by one thread.
constexpr uint64_t GAP_LONG = 4096;
constexpr unsigned GAP_SLOTS = 1024;

struct RowGap {
    uint64_t lo, hi, pos;
};

// With off (a first lock), the pass also writes the staged rows' offsets, in
// case the rows turn out to be grouped: at a step from row r1 up to row r2
// after insert i, off[r1 + 1 .. r2] = i + 1. Only steps of at most OFF_STEP
// rows are written: inserts in random order, whose steps are long, then write
// next to nothing (writing every rising step's rows took ~m n / 3 stores
// there); a longer one sets stats[6], and launch_row_offsets writes the
// offsets after all (in a matrix of few rows, where short steps are common in
// random order too, steps of one row only). A pass of its own over the 64 M
// inserts' rows of the 4M-row Zipf matrix took 106 us, the stores here 32
// (lock 1.64 -> 1.54 ms).
constexpr uint32_t OFF_STEP = 8;

__device__ __forceinline__ bool offsets_step(uint64_t *__restrict__ off, uint64_t lo, uint64_t hi, uint64_t n_rows,
                                             uint64_t pos) {  // off[lo .. hi] = pos; true if left to the other pass
    if (hi > n_rows || hi - lo >= (n_rows < (1u << 16) ? 1u : OFF_STEP)) return true;  // (rows are not range-checked yet)
    off[hi] = pos;
    for (uint64_t r = lo; r < hi; ++r) off[r] = pos;  // (steps of one row, by far the most: none)
    return false;
}

__device__ __forceinline__ uint32_t column_gap(uint32_t a, uint32_t b) { return a < b ? b - a : a - b; }

// VEC: rows and cols 16-byte aligned; each thread reads 4 rows and 4
// columns per step in two 16-byte loads (the successor of its last pair
// comes from the next lane, or one more load at the warp's edge).
// stats[5] += a sample of the inserts that 32 others of their row follow: every
// fourth insert, by 24 lanes of each warp's 32 (3 / 16 of all). stats[7] += a
// sample of the inserts whose successor in the row is nearer than `near`
// columns, less those whose successor is not: every fourth insert. stats[8] += a
// sample of the inserts that are of one row with the 32nd and the 64th after
// them (an eighth of all), stats[9] += a sample of those whose successor is of an
// earlier row (every fourth): what they say of inserts in no order, hub_rows below.
// Both with HUBS only, for up to FEW_STAGED inserts and for later epochs: the
// registers that they take cost 18 us of 132 for 64 M inserts, and nothing while
// the blocks are few.
constexpr int N_STATS = 10;

template <bool VEC, bool HUBS>
__global__ void lock_prepare(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ cols, uint64_t m,
                             int cbits, uint64_t n_rows, uint32_t near, uint64_t *__restrict__ off,
                             unsigned *__restrict__ stats,
                             unsigned long long *__restrict__ words) {
    unsigned mr = 0, mc = 0, hits = 0, triples = 0, falls = 0;
    int score = 0;
    bool d = false, g = false, e = false, gap = false;
    if (off && blockIdx.x == 0 && threadIdx.x == 0) {  // the rows up to the first insert's and after the last one's
        gap |= offsets_step(off, 0, rows[0], n_rows, 0);
        gap |= offsets_step(off, (uint64_t)rows[m - 1] + 1, n_rows, n_rows, m);
    }
    if constexpr (VEC) {
        const uint64_t n4 = m / 4;  // whole groups of 4; the tail below
        const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
        const uint64_t n_iter = (n4 + stride - 1) / stride;  // warp-uniform: shuffles below
        for (uint64_t it = 0; it < n_iter; ++it) {
            const uint64_t q = it * stride + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
            const bool ok = q < n4;
            uint4 r4 = make_uint4(0, 0, 0, 0), c4 = make_uint4(0, 0, 0, 0);
            if (ok) {
                r4 = reinterpret_cast<const uint4 *>(rows)[q];
                c4 = reinterpret_cast<const uint4 *>(cols)[q];
            }
            const uint32_t r32 = __shfl_down_sync(0xffffffffu, r4.x, 8);
            if (4 * q + 32 < 4 * n4 && (threadIdx.x & 31) < 24) hits += r32 == r4.x ? 1u : 0u;
            if constexpr (HUBS) {
                const uint32_t r64 = __shfl_down_sync(0xffffffffu, r4.x, 16);
                if (4 * q + 64 < 4 * n4 && (threadIdx.x & 31) < 16) triples += r32 == r4.x && r64 == r4.x ? 1u : 0u;
                falls += r4.x > r4.y ? 1u : 0u;
            }
            uint32_t rn = __shfl_down_sync(0xffffffffu, r4.x, 1), cn = __shfl_down_sync(0xffffffffu, c4.x, 1);
            const bool have_next = ok && 4 * q + 4 < m;
            if (have_next && ((threadIdx.x & 31) == 31 || q + 1 >= n4)) {
                rn = rows[4 * q + 4];
                cn = cols[4 * q + 4];
            }
            if (ok && r4.x == r4.y) score += column_gap(c4.x, c4.y) < near ? 1 : -1;
            if (ok) {
                const uint32_t rr[5] = {r4.x, r4.y, r4.z, r4.w, rn}, cc[5] = {c4.x, c4.y, c4.z, c4.w, cn};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    mr = max(mr, rr[k]);
                    mc = max(mc, cc[k]);
                    if (k < 3 || have_next) {
                        const uint64_t k1 = ((uint64_t)rr[k] << cbits) | cc[k];
                        const uint64_t k2 = ((uint64_t)rr[k + 1] << cbits) | cc[k + 1];
                        d |= k1 > k2;
                        e |= k1 >= k2;
                        g |= rr[k] > rr[k + 1];
                        if (off && rr[k] < rr[k + 1])
                            gap |= offsets_step(off, (uint64_t)rr[k] + 1, rr[k + 1], n_rows, 4 * q + k + 1);
                    }
                }
            }
        }
    }
    for (uint64_t i = (VEC ? (m & ~3ull) : 0) + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = rows[i], c = cols[i];
        mr = max(mr, r);
        mc = max(mc, c);
        if (!VEC && (i & 3) == 0 && ((i >> 2) & 31) < 24 && i + 32 < m && rows[i + 32] == r) {
            ++hits;
            if (HUBS && ((i >> 2) & 31) < 16 && i + 64 < m) triples += rows[i + 64] == r ? 1u : 0u;
        }
        if (i + 1 < m) {
            const uint32_t r2 = rows[i + 1], c2 = cols[i + 1];
            const uint64_t k = ((uint64_t)r << cbits) | c, k2 = ((uint64_t)r2 << cbits) | c2;
            if (HUBS && !VEC && (i & 3) == 0 && r > r2) ++falls;
            if (!VEC && (i & 3) == 0 && r == r2) score += column_gap(c, c2) < near ? 1 : -1;
            d |= k > k2;
            e |= k >= k2;
            g |= r > r2;
            if (off && r < r2) gap |= offsets_step(off, (uint64_t)r + 1, r2, n_rows, i + 1);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, o));
        mc = max(mc, __shfl_xor_sync(0xffffffffu, mc, o));
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if constexpr (HUBS) {
        triples = __reduce_add_sync(0xffffffffu, triples);
        falls = __reduce_add_sync(0xffffffffu, falls);
    }
    score = __reduce_add_sync(0xffffffffu, score);
    const unsigned flags = (__any_sync(0xffffffffu, d) ? 1u : 0u) | (__any_sync(0xffffffffu, g) ? 2u : 0u) |
                           (__any_sync(0xffffffffu, e) ? 4u : 0u) | (__any_sync(0xffffffffu, gap) ? 8u : 0u);
    // one set of atomics per block: per-warp atomics on the same two words
    // serialise at L2 and cost more than the pass itself
    __shared__ unsigned s_mr[LB / 32], s_mc[LB / 32], s_fl[LB / 32], s_hits[LB / 32], s_triples[LB / 32], s_falls[LB / 32];
    __shared__ int s_score[LB / 32];
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_mr[w] = mr;
        s_mc[w] = mc;
        s_fl[w] = flags;
        s_hits[w] = hits;
        s_score[w] = score;
        if constexpr (HUBS) {
            s_triples[w] = triples;
            s_falls[w] = falls;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned bm = 0, bc = 0, bf = 0, bh = 0, bt = 0, bd = 0;
        int bs = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            bm = max(bm, s_mr[i]);
            bc = max(bc, s_mc[i]);
            bf |= s_fl[i];
            bh += s_hits[i];
            bs += s_score[i];
            if constexpr (HUBS) {
                bt += s_triples[i];
                bd += s_falls[i];
            }
        }
        atomicMax(stats, bm);
        atomicMax(stats + 1, bc);
        if (bh) atomicAdd(stats + 5, bh);
        if (bs) atomicAdd(reinterpret_cast<int *>(stats) + 7, bs);
        if (bf & 1u) stats[2] = 1u;
        if (bf & 2u) stats[3] = 1u;
        if (bf & 4u) stats[4] = 1u;
        if (bf & 8u) stats[6] = 1u;
        if (bt) atomicAdd(stats + 8, bt);
        if (bd) atomicAdd(stats + 9, bd);
        if (last_block(stats + N_STATS)) store_counters<N_STATS>(words, stats);
    }
}

// Moves the kept entries of a row-grouped first lock from their rows' input
// positions (row r's at [s_off[r], s_off[r] + kept)) to their CSR positions
// (off: the exclusive scan of the kept counts). The staged rows name each
// position's row, as the rows are grouped.
__global__ void first_grouped_compact(const uint32_t *__restrict__ rows, const uint64_t *__restrict__ s_off,
                                      const uint64_t *__restrict__ off, const uint32_t *__restrict__ scols,
                                      const double *__restrict__ svals, uint64_t m, uint32_t *__restrict__ ocols,
                                      double *__restrict__ ovals) {
    // four positions per thread, their loads issued together: the row, the
    // entry and then the row's offsets are a chain of dependent loads
    constexpr int U = 4;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t e0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e0 < m; e0 += U * stride) {
        uint32_t r[U], c[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t e = e0 + u * stride;
            if (e < m) {
                r[u] = rows[e];
                c[u] = scols[e];
                v[u] = svals[e];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t e = e0 + u * stride;
            if (e < m) {
                const uint64_t k = e - s_off[r[u]], o0 = off[r[u]];
                if (k < off[r[u] + 1] - o0) {
                    ocols[o0 + k] = c[u];
                    ovals[o0 + k] = v[u];
                }
            }
        }
    }
}

// First lock of inserts in strictly increasing (row, col) order: the CSR is
// the staged arrays themselves unless a value is zero (*zero = 1; then the
// caller takes the general path).
__global__ void first_direct_copy(const uint32_t *__restrict__ cols, const double *__restrict__ vals, uint64_t m,
                                  uint32_t *__restrict__ out_cols, double *__restrict__ out_vals,
                                  unsigned *__restrict__ zero, unsigned long long *__restrict__ words) {
    bool z = false;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double v = vals[i];
        z |= is_zero(v);
        out_cols[i] = cols[i];
        out_vals[i] = v;
    }
    const bool any = __syncthreads_or(z);
    if (threadIdx.x == 0) {
        if (any) zero[0] = 1u;
        if (last_block(zero + 1)) store_word(words, 0, *(volatile unsigned *)zero);
    }
}

// flag[i] = 1 iff sorted key i is the last of its run (the last write).
__global__ void lock_last_flags(const uint64_t *__restrict__ keys, uint64_t m, uint64_t *__restrict__ flag) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x)
        flag[i] = (i + 1 == m || keys[i] != keys[i + 1]) ? 1 : 0;
}

__global__ void lock_gather_delta(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx,
                                  const uint64_t *__restrict__ pos, uint64_t m, int cbits,
                                  const double *__restrict__ vals, uint32_t *__restrict__ drow,
                                  uint32_t *__restrict__ dcol, double *__restrict__ dval) {
    const uint64_t cmask = cbits ? ((1ull << cbits) - 1) : 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (i + 1 == m || keys[i] != keys[i + 1]) {
            const uint64_t j = pos[i];
            drow[j] = (uint32_t)(keys[i] >> cbits);
            dcol[j] = (uint32_t)(keys[i] & cmask);
            dval[j] = vals[idx[i]];
        }
    }
}

// off[r] = lower_bound(sorted_rows[0..u), r) for r in [0, n_rows], from the
// row boundaries: position i (i == u standing for row n_rows) is the first
// position of rows srows[i - 1] + 1 .. srows[i], so it writes those offsets.
// One pass over the rows, coalesced, no searches. Runs of up to GAP_LONG
// empty rows are written by the thread at their boundary; longer ones are
// listed in `gaps` (up to GAP_SLOTS of them) for offsets_fill_gaps to spread
// over the grid, and written by their thread once the list is full. A
// decreasing step (never in the sorted input) writes nothing, so every write
// stays inside [0, n_rows].

constexpr int OFF_T = 256;

// Block steps over tiles of OFF_T * OFF_E positions (OFF_E = 1 for few
// positions, whose rows lie far apart: 100 k into 2 M rows 26 us with 8): the tile's rows (and the one
// before it) are staged in shared memory with coalesced loads, then thread t
// checks positions t, t + OFF_T, ... against their predecessors, so a
// position costs a few instructions and only row boundaries write.
template <int OFF_E>
__global__ void __launch_bounds__(OFF_T)
offsets_from_sorted_rows(const uint32_t *__restrict__ srows, uint64_t u, uint64_t n_rows,
                         uint64_t *__restrict__ off, RowGap *__restrict__ gaps, unsigned *__restrict__ n_gaps) {
    constexpr int OFF_TILE = OFF_T * OFF_E;
    __shared__ uint32_t s_row[OFF_TILE + 1];  // s_row[j] = row at position tile + j - 1 (when < u)
    for (uint64_t tile = blockIdx.x * (uint64_t)OFF_TILE; tile <= u; tile += (uint64_t)gridDim.x * OFF_TILE) {
        // all loads of a thread issued before any is stored (HBM needs many
        // bytes in flight per SM)
        uint32_t v[OFF_E + 1];
#pragma unroll
        for (int k = 0; k <= OFF_E; ++k) {
            const int j = threadIdx.x + k * OFF_T;
            const uint64_t p = tile + j - 1;  // tile == 0, j == 0: never read
            v[k] = (j <= OFF_TILE && tile + j >= 1 && p < u) ? srows[p] : 0u;
        }
#pragma unroll
        for (int k = 0; k <= OFF_E; ++k) {
            const int j = threadIdx.x + k * OFF_T;
            if (j <= OFF_TILE) s_row[j] = v[k];
        }
        __syncthreads();
        const int lim = (int)min((uint64_t)OFF_TILE, u + 1 - tile);  // positions tile .. u of this tile
#pragma unroll
        for (int k = 0; k < OFF_E; ++k) {
            const int j = threadIdx.x + k * OFF_T;
            if (j >= lim) break;
            const uint64_t i = tile + j;
            const bool at_end = i == u;
            // inside a row: same row as the position before (32-bit fast path)
            if (i != 0 && !at_end && s_row[j + 1] == s_row[j]) continue;
            const uint64_t cur = at_end ? n_rows : min((uint64_t)s_row[j + 1], n_rows);
            const uint64_t lo = i == 0 ? 0 : (uint64_t)s_row[j] + 1;  // rows [lo, cur] start at position i
            if (cur + 1 <= lo) continue;  // a decreasing step (never in sorted input): nothing
            const uint64_t hi = cur + 1;
            if (hi - lo > GAP_LONG) {
                const unsigned slot = atomicAdd(n_gaps, 1u);
                if (slot < GAP_SLOTS) {
                    gaps[slot] = {lo, hi, i};
                    continue;  // listed: written by offsets_fill_gaps
                }
            }
            for (uint64_t r = lo; r < hi; ++r) off[r] = i;
        }
        __syncthreads();
    }
}

// The listed long stretches of empty rows, each spread over the whole grid.
__global__ void offsets_fill_gaps(const RowGap *__restrict__ gaps, const unsigned *__restrict__ n_gaps,
                                  uint64_t *__restrict__ off) {
    const unsigned n = min(*n_gaps, GAP_SLOTS);
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, nt = (uint64_t)gridDim.x * blockDim.x;
    for (unsigned g = 0; g < n; ++g) {
        const RowGap G = gaps[g];
        for (uint64_t r = G.lo + t; r < G.hi; r += nt) off[r] = G.pos;
    }
}

}  // namespace

// off[0..n_rows] from the non-decreasing rows srows[0..u) (stream-ordered).
int launch_row_offsets(Ctx *c, const uint32_t *srows, uint64_t u, uint64_t n_rows, uint64_t *off, cudaStream_t s) {
    DevBuf scratch;  // [counter (16 bytes)] [GAP_SLOTS gaps]
    SPG_TRY(scratch.alloc(16 + GAP_SLOTS * sizeof(RowGap), s));
    unsigned *n_gaps = scratch.as<unsigned>();
    RowGap *gaps = reinterpret_cast<RowGap *>(scratch.as<char>() + 16);
    SPG_CUDA_TRY(cudaMemsetAsync(n_gaps, 0, sizeof(unsigned), s));
    const unsigned cap = (unsigned)c->n_sms * 8;
    if (u < (1u << 20))
        offsets_from_sorted_rows<1><<<grid_for(u + 1, OFF_T, cap), OFF_T, 0, s>>>(srows, u, n_rows, off, gaps, n_gaps);
    else
        offsets_from_sorted_rows<8><<<grid_for(u + 1, OFF_T * 8, cap), OFF_T, 0, s>>>(srows, u, n_rows, off, gaps,
                                                                                   n_gaps);
    offsets_fill_gaps<<<c->n_sms * 4, LB, 0, s>>>(gaps, n_gaps, off);
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

namespace {

// Explicit zeros of a loaded CSR inside rows the delta touches: Spira's merge
// drops them (csr_build.hpp:274-276, 292-296). They become synthetic zero
// inserts placed before the real ones, so a real insert on the same column
// still wins the last-write dedup.
__global__ void zero_entries_in_dirty_rows(const uint64_t *__restrict__ off, const uint32_t *__restrict__ cols,
                                           const double *__restrict__ vals, uint64_t n_rows,
                                           const uint64_t *__restrict__ doff, uint64_t *__restrict__ flag,
                                           uint32_t *__restrict__ zrow, uint32_t *__restrict__ zcol,
                                           const uint64_t *__restrict__ pos, int pass) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n_rows;
         r += (uint64_t)gridDim.x * blockDim.x) {
        const bool dirty = doff[r] != doff[r + 1];
        for (uint64_t k = off[r]; k < off[r + 1]; ++k) {
            const bool z = dirty && is_zero(vals[k]);
            if (pass == 0) {
                flag[k] = z ? 1 : 0;
            } else if (z) {
                zrow[pos[k]] = (uint32_t)r;
                zcol[pos[k]] = cols[k];
            }
        }
    }
}

__global__ void fill_f64(double *p, uint64_t n, double v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

// Delta arrays (sorted by (row, col), one entry per key, zeros kept).
struct Delta {
    uint64_t u = 0;
    DevBuf row, col, val;
};

// First lock (build_csr, csr_build.hpp:32-98): the CSR is the last write of
// every key with zeros dropped. flag[i] = 1 iff sorted entry i is kept.
// First lock, general path: the sorted entries are compacted in two passes
// over tiles of KTILE entries, without a per-entry position array. Entry i
// is kept when it is the last of its key run (the last write) and its value
// is not +-0. Pass 1 counts the kept entries of every tile; after a scan of
// the counts, pass 2 recomputes the flags, ranks them inside the tile
// (entries k * KT + t, k-major: ballots per warp, warp totals in shared
// memory) and writes row, column and value at tile prefix + rank.
constexpr int KT = 256, KI = 8, KTILE = KT * KI;

__device__ __forceinline__ unsigned lane_lt_mask() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ void keep_flags_of_tile(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx,
                                                   const double *__restrict__ vals, uint64_t m, uint64_t base,
                                                   bool (&f)[KI], uint64_t (&key)[KI], double (&val)[KI]) {
    uint32_t ix[KI];
    uint64_t nxt[KI];
#pragma unroll
    for (int k = 0; k < KI; ++k) {  // loads of all items first
        const uint64_t i = base + (uint64_t)k * KT + threadIdx.x;
        key[k] = i < m ? keys[i] : 0;
        nxt[k] = i + 1 < m ? keys[i + 1] : ~0ull;
        ix[k] = i < m ? idx[i] : 0;
    }
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        const uint64_t i = base + (uint64_t)k * KT + threadIdx.x;
        const bool last = i < m && (i + 1 == m || key[k] != nxt[k]);
        val[k] = last ? vals[ix[k]] : 0.0;
        f[k] = last && !is_zero(val[k]);
    }
}

__global__ void __launch_bounds__(KT)
first_keep_count(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx, const double *__restrict__ vals,
                 uint64_t m, uint64_t *__restrict__ tile_counts) {
    bool f[KI];
    uint64_t key[KI];
    double val[KI];
    keep_flags_of_tile(keys, idx, vals, m, blockIdx.x * (uint64_t)KTILE, f, key, val);
    unsigned c = 0;
#pragma unroll
    for (int k = 0; k < KI; ++k) c += f[k];
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    __shared__ unsigned s_c[KT / 32];
    if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < KT / 32; ++w) t += s_c[w];
        tile_counts[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(KT)
first_keep_gather(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx, const double *__restrict__ vals,
                  uint64_t m, int cbits, const uint64_t *__restrict__ tile_prefix, uint32_t *__restrict__ orow,
                  uint32_t *__restrict__ ocol, double *__restrict__ oval) {
    bool f[KI];
    uint64_t key[KI];
    double val[KI];
    keep_flags_of_tile(keys, idx, vals, m, blockIdx.x * (uint64_t)KTILE, f, key, val);
    __shared__ unsigned s_w[KI][KT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned rank[KI];
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        const unsigned b = __ballot_sync(0xffffffffu, f[k]);
        rank[k] = __popc(b & lane_lt_mask());
        if (lane == 0) s_w[k][warp] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // exclusive prefix over (k, warp): the tile's entry order
        unsigned run = 0;
        for (int k = 0; k < KI; ++k)
            for (int w = 0; w < KT / 32; ++w) {
                const unsigned v = s_w[k][w];
                s_w[k][w] = run;
                run += v;
            }
    }
    __syncthreads();
    const uint64_t base = tile_prefix[blockIdx.x];
    const uint64_t cmask = cbits ? ((1ull << cbits) - 1) : 0;
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        if (!f[k]) continue;
        const uint64_t j = base + s_w[k][warp] + rank[k];
        orow[j] = (uint32_t)(key[k] >> cbits);
        ocol[j] = (uint32_t)(key[k] & cmask);
        oval[j] = val[k];
    }
}

// Order flags of a staged epoch, from lock_prepare beside the range check.
struct Prepared {
    unsigned unsorted = 1, ungrouped = 1, not_strict = 1;
    uint64_t long_hits = 0;  // sampled inserts that 32 others of their row follow (3 / 16 of the inserts looked at)
    int64_t clustered = 0;   // sampled inserts with a near successor in their row, less those with a far one
    double pairs = 0.0, triples = 0.0;  // the chance that two, three inserts are of one row (of inserts in no order)
    bool ready = false;
    DevBuf off;             // a first lock: the staged rows' offsets ...
    bool have_off = false;  // ... when the rows are grouped and no step between them was long
};

// Whether inserts in no order go to the global sort, as rows that no block
// takes hold much of them. With K such rows of equal length, a share f of the
// inserts, and short ones besides, two inserts are of one row with chance f^2 /
// K and three with f^3 / K^2: their square and ratio give f and the rows' length.
// From half of the inserts on, sorting those rows apart is slower than sorting
// all (row sort, attempt and tiles / global, later epochs: 2.5 M in 10 rows 499 /
// 392 us, 3 M in 200 rows 701 / 507), in small epochs from a tenth on (5 rows of
// 13 000 430 / 351, and 100 k others 468 / 393), where launches are what is paid;
// below, it is faster (12 M with one row of 2 M: 979 / 1461). First locks of more
// than 4 M inserts are not sampled: the plan of the tiles finds out.
constexpr uint64_t HUB_FEW = 1u << 19;

bool hub_rows(const Prepared &pre, uint64_t m) {
    if (pre.triples == 0.0) return false;
    const double length = (double)m * pre.triples / pre.pairs, share = pre.pairs * pre.pairs / pre.triples;
    return length > 12288.0 && share > (m <= HUB_FEW ? 0.1 : 0.5);
}

// The staged (grouped) rows' offsets.
int staged_offsets(Ctx *c, Prepared *pre, const uint32_t *rows, uint64_t m, uint64_t n_rows, DevBuf &off,
                   cudaStream_t s) {
    const bool have = pre && pre->off.ptr && pre->have_off;
    if (pre && pre->off.ptr) off = std::move(pre->off);
    else SPG_TRY(off.alloc(csr_off_elems(n_rows) * sizeof(uint64_t), s));
    if (!have) SPG_TRY(launch_row_offsets(c, rows, m, n_rows, off.as<uint64_t>(), s));
    return SPG_OK;
}

constexpr uint64_t FEW_STAGED = 4u << 20;

// A sixteenth of the columns: a successor at random is nearer once in eight.
uint32_t near_columns(uint64_t n_cols) { return (uint32_t)std::min<uint64_t>(n_cols / 16 + 1, 0xFFFFFFFFull); }

// Prepared::long_hits and clustered of rows sorted since lock_prepare, from 2^16 places.
constexpr uint64_t LONG_SAMPLES = 1u << 16;

__global__ void long_rows_sample(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ cols, uint64_t m,
                                 uint32_t near, unsigned *__restrict__ hits, unsigned long long *__restrict__ words) {
    const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, i = k * (m - 32) / LONG_SAMPLES;
    const unsigned n = __popc(__ballot_sync(0xffffffffu, rows[i] == rows[i + 32]));
    const int score = rows[i] != rows[i + 1] ? 0 : column_gap(cols[i], cols[i + 1]) < near ? 1 : -1;
    const int sum = __reduce_add_sync(0xffffffffu, score);
    if ((threadIdx.x & 31) == 0) {
        if (n) atomicAdd(hits, n);
        if (sum) atomicAdd(reinterpret_cast<int *>(hits) + 1, sum);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0 && last_block(hits + 2)) {
        store_word(words, 0, *(volatile unsigned *)hits);
        store_word(words, 1, *(volatile unsigned *)(hits + 1));
    }
}

int sample_long_rows(Ctx *c, const uint32_t *rows, const uint32_t *cols, uint64_t m, uint64_t n_cols, Prepared *pre,
                     cudaStream_t s) {
    DevBuf hits;
    SPG_TRY(hits.alloc(3 * sizeof(unsigned), s));
    SPG_CUDA_TRY(cudaMemsetAsync(hits.ptr, 0, 3 * sizeof(unsigned), s));
    long_rows_sample<<<LONG_SAMPLES / LB, LB, 0, s>>>(rows, cols, m, near_columns(n_cols), hits.as<unsigned>(),
                                                        c->d_words);
    SPG_LAUNCH_CHECK();
    SPG_TRY(c->phase_sync(s));
    pre->clustered = (int)(unsigned)c->word(1);
    pre->long_hits = (uint64_t)((double)c->word(0) / LONG_SAMPLES * 3.0 / 16.0 * (double)m);
    return SPG_OK;
}

// Keys (row << cbits | col) of the staged inserts sorted stably, with their
// staging indices.
int sort_keys(Ctx *c, const uint32_t *rows, const uint32_t *cols, uint64_t m, uint64_t n_rows, uint64_t n_cols,
              DevBuf &keys, DevBuf &idx, bool sorted, cudaStream_t s) {
    const int cbits = bits_for(n_cols), rbits = bits_for(n_rows);
    const unsigned g = grid_for(m, LB, (unsigned)c->n_sms * 16);
    // Inserts staged already in (row, col) order need no sort: the stable sort
    // of a non-decreasing sequence is the identity.
    SPG_TRY(keys.alloc(m * sizeof(uint64_t), s));
    SPG_TRY(idx.alloc(m * sizeof(uint32_t), s));
    lock_make_keys<<<g, LB, 0, s>>>(rows, cols, m, cbits, keys.as<uint64_t>(), idx.as<uint32_t>());
    SPG_LAUNCH_CHECK();
    if (!sorted) SPG_TRY(radix_sort_pairs_u64(c, keys.as<uint64_t>(), idx.as<uint32_t>(), m, rbits + cbits, s));
    return SPG_OK;
}

int sort_dedup(Ctx *c, const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m,
               uint64_t n_rows, uint64_t n_cols, bool sorted, Delta &D, cudaStream_t s) {
    const int cbits = bits_for(n_cols);
    const unsigned g = grid_for(m, LB, (unsigned)c->n_sms * 16);
    DevBuf keys, idx, pos;
    SPG_TRY(sort_keys(c, rows, cols, m, n_rows, n_cols, keys, idx, sorted, s));
    SPG_TRY(pos.alloc((m + 1) * sizeof(uint64_t), s));
    lock_last_flags<<<g, LB, 0, s>>>(keys.as<uint64_t>(), m, pos.as<uint64_t>());
    SPG_LAUNCH_CHECK();
    SPG_TRY(exclusive_scan_u64(c, pos.as<uint64_t>(), m, pos.as<uint64_t>() + m, s));
    uint64_t u = 0;
    SPG_CUDA_TRY(cudaMemcpyAsync(&u, pos.as<uint64_t>() + m, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    SPG_TRY(c->phase_sync(s));
    D.u = u;
    SPG_TRY(D.row.alloc(u * sizeof(uint32_t), s));
    SPG_TRY(D.col.alloc(u * sizeof(uint32_t), s));
    SPG_TRY(D.val.alloc(u * sizeof(double), s));
    lock_gather_delta<<<g, LB, 0, s>>>(keys.as<uint64_t>(), idx.as<uint32_t>(), pos.as<uint64_t>(), m, cbits,
                                       vals, D.row.as<uint32_t>(), D.col.as<uint32_t>(), D.val.as<double>());
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

// ---- rows that fit no block (HugeRows): gathered, sorted by (row, column) with
// the row sort's passes, their last writes kept by a count, a scan and a gather.
// Entry p of all the huge rows' entries: its row is the last q with g[q] <= p.
// A warp takes 256 neighbours and finds the row of the first by a search.
__global__ void __launch_bounds__(LB) huge_gather(const uint32_t *__restrict__ huge, const uint64_t *__restrict__ g,
                                                  uint64_t n, const uint64_t *__restrict__ s_off,
                                                  const uint32_t *__restrict__ cols, const double *__restrict__ vals,
                                                  int row_shift, uint32_t *__restrict__ col, uint32_t *__restrict__ row,
                                                  double *__restrict__ val) {
    const uint64_t w = (blockIdx.x * (uint64_t)LB + threadIdx.x) >> 5, m = g[n];
    uint64_t p = w * 256 + (threadIdx.x & 31);
    if (p >= m) return;
    uint64_t q = 0, hi = n;
    while (hi - q > 1) {
        const uint64_t mid = (q + hi) >> 1;
        if (g[mid] <= p) q = mid;
        else hi = mid;
    }
    for (int k = 0; k < 8 && p < m; ++k, p += 32) {
        while (g[q + 1] <= p) ++q;
        const uint64_t e = s_off[huge[q]] + (p - g[q]);
        col[p] = cols[e] | (uint32_t)(q << row_shift);
        row[p] = (uint32_t)q;
        val[p] = vals[e];
    }
}

__global__ void huge_lengths(const uint32_t *__restrict__ huge, uint64_t n, const uint64_t *__restrict__ s_off,
                             uint64_t *__restrict__ g) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n; q += (uint64_t)gridDim.x * blockDim.x)
        g[q] = s_off[huge[q] + 1ull] - s_off[huge[q]];
}

__global__ void huge_counts(const uint32_t *__restrict__ huge, uint64_t n, const uint64_t *__restrict__ first,
                            uint64_t *__restrict__ count) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n; q += (uint64_t)gridDim.x * blockDim.x)
        count[huge[q]] = first[q + 1] - first[q];
}

// The sorted entries' last writes, counted per tile of KTILE (out_row null)
// and, tile_vals being the counts' scan, written to their places.
__global__ void __launch_bounds__(KT)
huge_keep(const uint32_t *__restrict__ row, const uint32_t *__restrict__ col, const double *__restrict__ val,
          uint32_t col_mask, uint64_t m, bool keep_zeros, const unsigned long long *__restrict__ abort, uint64_t *__restrict__ tile_vals,
          uint64_t n, uint32_t *__restrict__ out_row, uint32_t *__restrict__ out_col, double *__restrict__ out_val,
          uint64_t *__restrict__ first) {
    if (*abort) return;  // (the rows are places in `first`)
    __shared__ unsigned s_w[KI][KT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = blockIdx.x * (uint64_t)KTILE + threadIdx.x;
    uint32_t r[KI], c[KI], rank[KI];
    double v[KI];
    bool f[KI];
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        const uint64_t i = base + (uint64_t)k * KT;
        r[k] = i < m ? row[i] : 0u;
        c[k] = i < m ? col[i] : 0u;
        v[k] = i < m ? val[i] : 0.0;
        f[k] = i < m && (i + 1 == m || row[i + 1] != r[k] || col[i + 1] != c[k]) && (keep_zeros || !is_zero(v[k]));
    }
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        const unsigned b = __ballot_sync(0xffffffffu, f[k]);
        rank[k] = __popc(b & lane_lt_mask());
        if (lane == 0) s_w[k][warp] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned run = 0;
        for (int k = 0; k < KI; ++k)
            for (int w = 0; w < KT / 32; ++w) {
                const unsigned x = s_w[k][w];
                s_w[k][w] = run;
                run += x;
            }
        if (!out_row) tile_vals[blockIdx.x] = run;
    }
    if (!out_row) return;
    __syncthreads();
    const uint64_t at = tile_vals[blockIdx.x];
#pragma unroll
    for (int k = 0; k < KI; ++k) {
        const uint64_t i = base + (uint64_t)k * KT, j = at + s_w[k][warp] + rank[k];
        if (i < m && (i == 0 || row[i - 1] != r[k])) first[r[k]] = j;
        if (i + 1 == m) first[n] = j + (f[k] ? 1 : 0);
        if (f[k]) {
            out_row[j] = r[k];
            out_col[j] = c[k] & col_mask;
            out_val[j] = v[k];
        }
    }
}

}  // namespace

int fit_arrays(Ctx *c, uint64_t n, uint64_t room, DevBuf &cols, DevBuf &vals, cudaStream_t s) {
    if (n >= room - room / 8) return SPG_OK;
    DevBuf own_cols, own_vals;
    SPG_TRY(own_cols.alloc(csr_alloc_elems(n) * sizeof(uint32_t), s));
    SPG_TRY(own_vals.alloc(csr_alloc_elems(n) * sizeof(double), s));
    SPG_CUDA_TRY(cudaMemcpyAsync(own_cols.ptr, cols.ptr, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    SPG_CUDA_TRY(cudaMemcpyAsync(own_vals.ptr, vals.ptr, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    cols = std::move(own_cols);
    vals = std::move(own_vals);
    return c->phase_sync(s);
}

int order_huge_rows(Ctx *c, const uint32_t *cols, const double *vals, const uint64_t *s_off, const uint32_t *huge,
                    int cbits, bool keep_zeros, HugeRows *H, uint64_t *count, cudaStream_t s) {
    const uint64_t n = H->n, m = H->entries, tiles = (m + KTILE - 1) / KTILE;
    const unsigned gn = grid_for(n, LB, (unsigned)c->n_sms * 8);
    // stably by (row, column): by both at once where they fit 32 bits
    const bool both = bits_for(n) + cbits <= 32;
    const int row_shift = both && n > 1 ? cbits : 63;  // (63: the column alone)
    StagedSorted by_col, by_row;
    {
        DevBuf g, col, row, val;
        SPG_TRY(g.alloc((n + 1) * sizeof(uint64_t), s));
        SPG_TRY(col.alloc(m * sizeof(uint32_t), s));
        SPG_TRY(row.alloc(m * sizeof(uint32_t), s));
        SPG_TRY(val.alloc(m * sizeof(double), s));
        huge_lengths<<<gn, LB, 0, s>>>(huge, n, s_off, g.as<uint64_t>());
        SPG_LAUNCH_CHECK();
        SPG_TRY(exclusive_scan_u64(c, g.as<uint64_t>(), n, g.as<uint64_t>() + n, s));
        huge_gather<<<grid_for(m, LB * 8), LB, 0, s>>>(huge, g.as<uint64_t>(), n, s_off, cols, vals,
                                                     row_shift, col.as<uint32_t>(), row.as<uint32_t>(), val.as<double>());
        SPG_LAUNCH_CHECK();
        SPG_TRY(sort_staged_rows(c, col.as<uint32_t>(), row.as<uint32_t>(), val.as<double>(), m,
                                 both ? bits_for(n) + cbits : cbits, by_col, s));
    }
    const DevBuf *row = &by_col.cols, *col = &by_col.rows, *val = &by_col.vals;
    if (!both) {
        SPG_TRY(sort_staged_rows(c, row->as<uint32_t>(), col->as<uint32_t>(), val->as<double>(), m, bits_for(n), by_row, s,
                                 by_col.abort.as<unsigned long long>()));
        row = &by_row.rows, col = &by_row.cols, val = &by_row.vals;
    }
    H->abort = std::move(both ? by_col.abort : by_row.abort);
    DevBuf tile_vals;
    SPG_TRY(tile_vals.alloc(tiles * sizeof(uint64_t), s));
    SPG_TRY(H->first.alloc((n + 1) * sizeof(uint64_t), s));
    SPG_TRY(H->row.alloc(m * sizeof(uint32_t), s));
    SPG_TRY(H->cols.alloc(m * sizeof(uint32_t), s));
    SPG_TRY(H->vals.alloc(m * sizeof(double), s));
    for (int pass = 0; pass < 2; ++pass) {
        huge_keep<<<(unsigned)tiles, KT, 0, s>>>(row->as<uint32_t>(), col->as<uint32_t>(), val->as<double>(),
                                                 both ? (uint32_t)((1ull << cbits) - 1) : 0xFFFFFFFFu, m, keep_zeros, H->abort.as<unsigned long long>(), tile_vals.as<uint64_t>(), n,
                                                 pass ? H->row.as<uint32_t>() : nullptr, H->cols.as<uint32_t>(),
                                                 H->vals.as<double>(), H->first.as<uint64_t>());
        SPG_LAUNCH_CHECK();
        if (pass == 0) SPG_TRY(exclusive_scan_u64(c, tile_vals.as<uint64_t>(), tiles, nullptr, s));
    }
    huge_counts<<<gn, LB, 0, s>>>(huge, n, H->first.as<uint64_t>(), count);
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

namespace {

// Installs a first lock's CSR built in arrays sized for m entries (build_csr:
// exact capacity).
int first_install(Ctx *c, Csr *A, GroupedOut &&o, uint64_t m, cudaStream_t s) {
    const uint64_t nnz = o.n;
    SPG_TRY(fit_arrays(c, nnz, m, o.cols, o.vals, s));
    A->invalidate_derived();
    A->off = std::move(o.off);
    A->cols = std::move(o.cols);
    A->vals = std::move(o.vals);
    A->nnz = nnz;
    A->capacity = nnz;  // build_csr: exact
    A->built = true;
    A->may_have_zeros = false;
    return SPG_OK;
}

// First lock: sort, keep the last write of every key unless it is zero, and
// take the offsets from the kept rows.
int first_lock(Ctx *c, Csr *A, const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m,
               Prepared *pre, const unsigned long long *abort, cudaStream_t s) {
    const uint64_t n = A->n_rows;
    const int cbits = bits_for(A->n_cols);
    DevBuf keys, idx, pos, orow, out_cols, out_vals, new_off;
    uint64_t nnz = 0;
    if (m && pre && pre->ready && !pre->not_strict) {
        // strictly increasing keys: no duplicates to resolve, nothing to sort;
        // unless a value is zero, the staged arrays are the CSR
        const unsigned g = grid_for(m, LB, (unsigned)c->n_sms * 16);
        DevBuf zero;
        SPG_TRY(zero.alloc(2 * sizeof(unsigned), s));
        SPG_CUDA_TRY(cudaMemsetAsync(zero.ptr, 0, 2 * sizeof(unsigned), s));
        SPG_TRY(out_cols.alloc(csr_alloc_elems(m) * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(csr_alloc_elems(m) * sizeof(double), s));
        first_direct_copy<<<g, LB, 0, s>>>(cols, vals, m, out_cols.as<uint32_t>(), out_vals.as<double>(),
                                           zero.as<unsigned>(), c->d_words);
        SPG_LAUNCH_CHECK();
        // the offsets go out before the zero check comes back: one host sync
        SPG_TRY(staged_offsets(c, pre, rows, m, n, new_off, s));
        SPG_TRY(c->phase_sync(s));
        if (c->word(0) == 0) {
            A->invalidate_derived();
            A->off = std::move(new_off);
            A->cols = std::move(out_cols);
            A->vals = std::move(out_vals);
            A->nnz = m;
            A->capacity = m;  // build_csr: exact
            A->built = true;
            A->may_have_zeros = false;
            return SPG_OK;
        }
        new_off.release();
        out_cols.release();
        out_vals.release();
    }
    if (m && pre && pre->ready && pre->unsorted && !pre->ungrouped) {
        // Row-grouped inserts (rows non-decreasing, columns in any order, as
        // row-by-row assembly stages them). Two ways to the same CSR:
        //   tiles    (spg_rowtiles.cu) sort, reduce and write the CSR in one pass;
        //            rows above 12 288 entries are sorted apart;
        //   classes  every row is sorted, its last write per column kept unless
        //            zero, and compacted by its length class's kernel, in place
        //            at the row's input positions; a scan of the kept counts
        //            gives the offsets, and entries move only if some were
        //            dropped.
        // Tiles are faster where a row's columns spread over the matrix, so that
        // its buckets hold an entry each (1 M rows of 24 uniform columns: 0.45
        // against 0.60 ms; 2 M of 5: 0.26 / 0.30), where rows are long (200 k of
        // 201 in a band: 0.99 / 1.06; 20 k of 1000 on ten columns: 0.48 / 0.61),
        // and below 4 M inserts, where the classes' ten launches are what is paid
        // (600 k rows of 5: 0.15 / 0.18). Short rows of columns close together
        // crowd their buckets and are the networks' case (27-point stencil, 1 M
        // rows in any column order: 0.67 / 0.49; 300 k rows of 64 on 200 columns:
        // 0.54 / 0.43; 2 M of a 5-point stencil 0.27 / 0.23). So: tiles for few
        // inserts, when about 0.7 of the entries have one of their row 32 places
        // on, or when most have their successor a sixteenth of the columns away
        // or more; and for columns wider than the classes take, whose only
        // other way is the global sort (2 M rows of a 5-point stencil in 2^31
        // columns 0.26 / 1.33, shuffled 0.67 / 1.72).
        // Rows of 2 400 to 4 096 inserts on average go to the classes' radix blocks
        // (2 500 rows of 4000 in 1 M columns: 436 tiles / 385 us), and so do rows
        // of 1 536 and more in up to 2^14 columns, which those sort in two or three
        // passes (3 333 rows of 3000 on 4096: 520 / 350; 1 250 of 8000 on 16 384:
        // 498 / 443; 5 000 of 2000 on 4096: 387 / 333).
        const uint64_t mean = m / n;
        const bool radix = (mean >= 2400 && mean <= 4096) || (mean >= 1536 && mean <= 12288 && cbits <= 14);
        const bool tiles = (m <= FEW_STAGED && !radix) || cbits > ROW_CLASS_CBITS || 
                           (!radix && (8 * pre->long_hits > m + m / 32 || pre->clustered < 0));
        DevBuf s_off, kept, scols, svals;
        SPG_TRY(staged_offsets(c, pre, rows, m, n, s_off, s));
        bool done = false;
        if (!tiles) {
            SPG_TRY(kept.alloc(csr_off_elems(n) * sizeof(uint64_t), s));
            SPG_TRY(scols.alloc(csr_alloc_elems(m) * sizeof(uint32_t), s));
            SPG_TRY(svals.alloc(csr_alloc_elems(m) * sizeof(double), s));
            SPG_TRY(dedup_grouped_rows(c, cols, vals, s_off.as<uint64_t>(), m, n, cbits, scols.as<uint32_t>(),
                                       svals.as<double>(), kept.as<uint64_t>(), &nnz, &done, s));
            if (done) {
                if (nnz == m) {  // nothing dropped: the staging arrays are the CSR
                    out_cols = std::move(scols);
                    out_vals = std::move(svals);
                } else {
                    SPG_TRY(out_cols.alloc(csr_alloc_elems(nnz) * sizeof(uint32_t), s));
                    SPG_TRY(out_vals.alloc(csr_alloc_elems(nnz) * sizeof(double), s));
                    first_grouped_compact<<<grid_for(m, LB, (unsigned)c->n_sms * 16), LB, 0, s>>>(
                        rows, s_off.as<uint64_t>(), kept.as<uint64_t>(), scols.as<uint32_t>(), svals.as<double>(), m,
                        out_cols.as<uint32_t>(), out_vals.as<double>());
                    SPG_LAUNCH_CHECK();
                }
                A->invalidate_derived();
                A->off = std::move(kept);
                A->cols = std::move(out_cols);
                A->vals = std::move(out_vals);
                A->nnz = nnz;
                A->capacity = nnz;  // build_csr: exact
                A->built = true;
                A->may_have_zeros = false;
                SPG_TRY(c->phase_sync(s));
                return SPG_OK;
            }
            kept.release();  // (a row too long for the classes)
            scols.release();
            svals.release();
        }
        GroupedOut o;
        SPG_TRY(build_grouped_rows(c, cols, vals, s_off.as<uint64_t>(), m, n, cbits, pre->clustered > 0, false, abort, &o, &done,
                                   s));
        if (done) return first_install(c, A, std::move(o), m, s);
    }
    if (m) {
        const unsigned g = grid_for(m, LB, (unsigned)c->n_sms * 16);
        SPG_TRY(sort_keys(c, rows, cols, m, n, A->n_cols, keys, idx, !pre->unsorted, s));
        const uint64_t tiles = (m + KTILE - 1) / KTILE;
        SPG_TRY(pos.alloc((tiles + 1) * sizeof(uint64_t), s));  // kept entries per tile, then their prefix
        first_keep_count<<<(unsigned)tiles, KT, 0, s>>>(keys.as<uint64_t>(), idx.as<uint32_t>(), vals, m,
                                                        pos.as<uint64_t>());
        SPG_LAUNCH_CHECK();
        SPG_TRY(exclusive_scan_u64(c, pos.as<uint64_t>(), tiles, pos.as<uint64_t>() + tiles, s));
        SPG_CUDA_TRY(cudaMemcpyAsync(&nnz, pos.as<uint64_t>() + tiles, 8, cudaMemcpyDeviceToHost, s));
        SPG_TRY(c->phase_sync(s));
        SPG_TRY(out_cols.alloc(csr_alloc_elems(nnz) * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(csr_alloc_elems(nnz) * sizeof(double), s));
        SPG_TRY(orow.alloc((nnz ? nnz : 1) * sizeof(uint32_t), s));
        first_keep_gather<<<(unsigned)tiles, KT, 0, s>>>(keys.as<uint64_t>(), idx.as<uint32_t>(), vals, m, cbits,
                                                         pos.as<uint64_t>(), orow.as<uint32_t>(),
                                                         out_cols.as<uint32_t>(), out_vals.as<double>());
        SPG_LAUNCH_CHECK();
    } else {
        SPG_TRY(out_cols.alloc(csr_alloc_elems(0) * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(csr_alloc_elems(0) * sizeof(double), s));
    }
    SPG_TRY(new_off.alloc(csr_off_elems(n) * sizeof(uint64_t), s));
    SPG_TRY(launch_row_offsets(c, orow.as<uint32_t>(), nnz, n, new_off.as<uint64_t>(), s));
    A->invalidate_derived();
    A->off = std::move(new_off);
    A->cols = std::move(out_cols);
    A->vals = std::move(out_vals);
    A->nnz = nnz;
    A->capacity = nnz;  // build_csr: exact
    A->built = true;
    A->may_have_zeros = false;
    SPG_TRY(c->phase_sync(s));
    return SPG_OK;
}

// The general merge of an epoch into the old CSR (rows in any order only without
// stored zeros in it).
template <class AllocOut>
int merge_epoch(Ctx *c, const Csr *A, const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m,
                const unsigned long long *abort, AllocOut alloc_out, Prepared *pre, DevBuf &new_off, DevBuf &out_cols,
                DevBuf &out_vals, uint64_t *new_nnz, uint64_t *u, cudaStream_t s) {
    const uint64_t n = A->n_rows;
    DevBuf s_off;
    if (!pre->ungrouped) SPG_TRY(staged_offsets(c, pre, rows, m, n, s_off, s));
    StagedSorted again;
    if (A->may_have_zeros && A->nnz) {
        // Explicit old zeros of dirty rows become deletes staged before the epoch.
        DevBuf zpos;
        SPG_TRY(zpos.alloc((A->nnz + 1) * sizeof(uint64_t), s));
        const unsigned gz = grid_for(n, LB, (unsigned)c->n_sms * 32);
        zero_entries_in_dirty_rows<<<gz, LB, 0, s>>>(A->d_off(), A->d_cols(), A->d_vals(), n, s_off.as<uint64_t>(),
                                                     zpos.as<uint64_t>(), nullptr, nullptr, nullptr, 0);
        SPG_LAUNCH_CHECK();
        SPG_TRY(exclusive_scan_u64(c, zpos.as<uint64_t>(), A->nnz, zpos.as<uint64_t>() + A->nnz, s));
        uint64_t nz = 0;
        SPG_CUDA_TRY(cudaMemcpyAsync(&nz, zpos.as<uint64_t>() + A->nnz, 8, cudaMemcpyDeviceToHost, s));
        SPG_TRY(c->phase_sync(s));
        if (nz) {
            const uint64_t m2 = nz + m;
            if (m2 >= (1ull << 32))
                return set_error(SPG_ERR_UNSUPPORTED, "lock: %llu staged inserts and stored zeros exceed 2^32-1",
                                 (unsigned long long)m2);
            DevBuf zr, zc, zv;
            SPG_TRY(zr.alloc(m2 * sizeof(uint32_t), s));
            SPG_TRY(zc.alloc(m2 * sizeof(uint32_t), s));
            SPG_TRY(zv.alloc(m2 * sizeof(double), s));
            zero_entries_in_dirty_rows<<<gz, LB, 0, s>>>(A->d_off(), A->d_cols(), A->d_vals(), n, s_off.as<uint64_t>(),
                                                         nullptr, zr.as<uint32_t>(), zc.as<uint32_t>(),
                                                         zpos.as<uint64_t>(), 1);
            SPG_LAUNCH_CHECK();
            fill_f64<<<grid_for(nz, LB, 4096), LB, 0, s>>>(zv.as<double>(), nz, 0.0);
            SPG_LAUNCH_CHECK();
            SPG_CUDA_TRY(cudaMemcpyAsync(zr.as<uint32_t>() + nz, rows, m * 4, cudaMemcpyDeviceToDevice, s));
            SPG_CUDA_TRY(cudaMemcpyAsync(zc.as<uint32_t>() + nz, cols, m * 4, cudaMemcpyDeviceToDevice, s));
            SPG_CUDA_TRY(cudaMemcpyAsync(zv.as<double>() + nz, vals, m * 8, cudaMemcpyDeviceToDevice, s));
            SPG_TRY(sort_staged_rows(c, zr.as<uint32_t>(), zc.as<uint32_t>(), zv.as<double>(), m2, bits_for(n), again, s));
            rows = again.rows.as<uint32_t>();
            cols = again.cols.as<uint32_t>();
            vals = again.vals.as<double>();
            abort = again.abort.as<unsigned long long>();
            m = m2;
            SPG_TRY(launch_row_offsets(c, rows, m, n, s_off.as<uint64_t>(), s));
        }
    }
    // the epoch's last writes, zeros kept (they delete), in (row, column) order
    GroupedOut D;
    bool done = false;
    if (!pre->ungrouped)
        SPG_TRY(build_grouped_rows(c, cols, vals, s_off.as<uint64_t>(), m, n, bits_for(A->n_cols), pre->clustered > 0, true,
                                   abort, &D, &done, s));
    if (!done) {  // mostly rows too long for the tiles (or no memory to sort those apart)
        if (!D.off.ptr) SPG_TRY(D.off.alloc(csr_off_elems(n) * sizeof(uint64_t), s));
        Delta d;
        SPG_TRY(sort_dedup(c, rows, cols, vals, m, n, A->n_cols, !pre->unsorted && !again.rows.ptr, d, s));
        SPG_TRY(launch_row_offsets(c, d.row.as<uint32_t>(), d.u, n, D.off.as<uint64_t>(), s));
        D.cols = std::move(d.col);
        D.vals = std::move(d.val);
        D.n = d.u;
    }
    *u = D.n;
    SPG_TRY(alloc_out(D.n));
    return merge_csr(c, {A->d_off(), A->d_cols(), A->d_vals(), A->nnz},
                     {D.off.as<uint64_t>(), D.cols.as<uint32_t>(), D.vals.as<double>(), D.n}, n, MergeMode::Replace,
                     new_off.as<uint64_t>(), out_cols.as<uint32_t>(), out_vals.as<double>(), new_nnz, s);
}

}  // namespace

// The lock proper, on device-resident staging arrays.
static int lock_device_impl(Ctx *c, Csr *A, const uint32_t *rows, const uint32_t *cols, const double *vals,
                            uint64_t m, cudaStream_t s) {
    if (m >= (1ull << 32))
        return set_error(SPG_ERR_UNSUPPORTED, "lock: %llu staged inserts exceed 2^32-1 per epoch",
                         (unsigned long long)m);
    // Range checks first: a failure leaves A untouched (matrix.hpp:161-171).
    // The same pass tells how the inserts are ordered.
    Prepared pre;
    if (m) {
        DevBuf stats;
        SPG_TRY(stats.alloc((N_STATS + 1) * sizeof(unsigned), s));
        SPG_CUDA_TRY(cudaMemsetAsync(stats.ptr, 0, (N_STATS + 1) * sizeof(unsigned), s));
        if (!A->built) SPG_TRY(pre.off.alloc(csr_off_elems(A->n_rows) * sizeof(uint64_t), s));
        const bool vec = ((uintptr_t)rows | (uintptr_t)cols) % 16 == 0, hubs = m <= FEW_STAGED || A->built;
        auto k = vec ? (hubs ? lock_prepare<true, true> : lock_prepare<true, false>)
                     : (hubs ? lock_prepare<false, true> : lock_prepare<false, false>);
        k<<<grid_for(vec ? (m + 3) / 4 : m, LB, (unsigned)c->n_sms * 16), LB, 0, s>>>(
            rows, cols, m, bits_for(A->n_cols), A->n_rows, near_columns(A->n_cols), pre.off.as<uint64_t>(),
            stats.as<unsigned>(), c->d_words);
        SPG_LAUNCH_CHECK();
        SPG_TRY(c->phase_sync(s));
        unsigned h[N_STATS];
        for (int i = 0; i < N_STATS; ++i) h[i] = (unsigned)c->word(i);
        if ((uint64_t)h[0] >= A->n_rows)
            return set_error(SPG_ERR_OUT_OF_RANGE, "spira::matrix: row_index out of range (%u >= %llu)", h[0],
                             (unsigned long long)A->n_rows);
        if ((uint64_t)h[1] >= A->n_cols)
            return set_error(SPG_ERR_OUT_OF_RANGE, "spira::matrix: col_index out of range (%u >= %llu)", h[1],
                             (unsigned long long)A->n_cols);
        pre.unsorted = h[2];
        pre.ungrouped = h[3];
        pre.not_strict = h[4];
        pre.long_hits = h[5];
        pre.clustered = (int)h[7];
        // (fewer than 32 say nothing; in no order every other insert or so is followed
        // by an earlier row's)
        if (h[8] >= 32 && (double)h[9] * 4.0 > 0.25 * (double)m * (1.0 - std::min(1.0, (double)h[5] * 16.0 / 3.0 / (double)m))) {
            pre.pairs = (double)h[5] * 16.0 / 3.0 / (double)m;
            pre.triples = (double)h[8] * 8.0 / (double)m;
        }
        pre.have_off = pre.off.ptr && !h[3] && !h[6];
        pre.ready = true;
    }
    const uint64_t n = A->n_rows;
    const bool has_old = A->built;
    if (has_old && m == 0) return SPG_OK;  // no dirty row: Spira's merge leaves the CSR as it is
    StagedSorted sorted;
    // Rows in any order are sorted by row, and row-grouped from here on; but they
    // go to the global sort where the row kernels cannot take most of them (12 288
    // inserts a row), and no stored zeros ask for the rows' offsets.
    const bool global = pre.ungrouped && (has_old ? !A->may_have_zeros && hub_rows(pre, m) : m > 12288 * n || hub_rows(pre, m));
    if (m && pre.ungrouped && !global) {
        SPG_TRY(sort_staged_rows(c, rows, cols, vals, m, bits_for(n), sorted, s));
        rows = sorted.rows.as<uint32_t>();
        cols = sorted.cols.as<uint32_t>();
        vals = sorted.vals.as<double>();
        pre.unsorted = 1;
        pre.ungrouped = 0;
        pre.not_strict = 1;
        pre.have_off = false;
        if (!has_old && m > FEW_STAGED) SPG_TRY(sample_long_rows(c, rows, cols, m, A->n_cols, &pre, s));
    }
    const unsigned long long *abort = sorted.abort.as<unsigned long long>();
    if (!has_old) return first_lock(c, A, rows, cols, vals, m, &pre, abort, s);

    DevBuf new_off, out_cols, out_vals;
    uint64_t new_nnz = 0, u = 0;
    bool done = false;
    auto alloc_out = [&](uint64_t inserts) -> int {  // for every entry of both sides, or the capacity below
        const uint64_t ub = A->nnz + inserts, elems = csr_alloc_elems(ub <= A->capacity ? A->capacity : ub + ub / 2);
        SPG_TRY(new_off.alloc(csr_off_elems(n) * sizeof(uint64_t), s));
        SPG_TRY(out_cols.alloc(elems * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(elems * sizeof(double), s));
        return SPG_OK;
    };
    // A fifth of the matrix at most goes insert by insert, unless many rows get
    // more than it takes (1 M rows of 10, insert by insert / general merge: 100 k
    // inserts 274 / 385 us, 1.25 M 430 / 507, 2.5 M 551 / 560; 30 k rows of 1000:
    // 300 k 466 / 663; 3 M, 100 to a row, 1216 with the attempt / 862).
    if (!global && !A->may_have_zeros && m <= A->nnz / 5 && m <= 32 * n && 16 * pre.long_hits <= m) {
        SPG_TRY(alloc_out(m));
        SPG_TRY(merge_small_delta(c, {A->d_off(), A->d_cols(), A->d_vals(), A->nnz}, n, rows, cols, vals, m, abort,
                                  new_off.as<uint64_t>(), out_cols.as<uint32_t>(), out_vals.as<double>(), &new_nnz, &u,
                                  &done, s));
    }
    if (!done) SPG_TRY(merge_epoch(c, A, rows, cols, vals, m, abort, alloc_out, &pre, new_off, out_cols, out_vals, &new_nnz, &u, s));
    // Spira's capacity rule (csr_build.hpp:139-145) on the distinct keys
    const uint64_t total_ub = A->nnz + u;
    const uint64_t cap = (total_ub <= A->capacity) ? A->capacity : total_ub + total_ub / 2;
    A->invalidate_derived();
    A->off = std::move(new_off);
    A->cols = std::move(out_cols);
    A->vals = std::move(out_vals);
    A->nnz = new_nnz;
    A->capacity = cap;
    A->built = true;
    // Zeros of dirty rows were consumed; clean rows may still hold loaded zeros.
    return SPG_OK;
}

}  // namespace spg

using namespace spg;

extern "C" {

int spg_lock_device(spg_ctx *c, spg_csr *A, const uint32_t *d_rows, const uint32_t *d_cols, const double *d_vals,
                    uint64_t n_staged) {
    if (!c || !A) return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_lock_device: null handle");
    SPG_CHECK_LIVE(A);
    if (n_staged && (!d_rows || !d_cols || !d_vals))
        return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_lock_device: null staging array");
    SPG_CUDA_TRY(cudaSetDevice(c->device));
    return lock_device_impl(c, A, d_rows, d_cols, d_vals, n_staged, c->stream);
}

int spg_lock(spg_ctx *c, spg_csr *A, const uint32_t *rows, const uint32_t *cols, const double *vals,
             uint64_t n_staged) {
    if (!c || !A) return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_lock: null handle");
    SPG_CHECK_LIVE(A);
    if (n_staged && (!rows || !cols || !vals))
        return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_lock: null staging array");
    SPG_CUDA_TRY(cudaSetDevice(c->device));
    cudaStream_t s = c->stream;
    DevBuf r, cl, v;
    if (n_staged) {
        SPG_TRY(r.alloc(n_staged * sizeof(uint32_t), s));
        SPG_TRY(cl.alloc(n_staged * sizeof(uint32_t), s));
        SPG_TRY(v.alloc(n_staged * sizeof(double), s));
        SPG_CUDA_TRY(cudaMemcpyAsync(r.ptr, rows, n_staged * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
        SPG_CUDA_TRY(cudaMemcpyAsync(cl.ptr, cols, n_staged * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
        SPG_CUDA_TRY(cudaMemcpyAsync(v.ptr, vals, n_staged * sizeof(double), cudaMemcpyHostToDevice, s));
    }
    return lock_device_impl(c, A, r.as<uint32_t>(), cl.as<uint32_t>(), v.as<double>(), n_staged, s);
}

}  // extern "C"
