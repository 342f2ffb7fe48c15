// spg_rowtiles.cu — row-grouped inserts to CSR in one pass: entries whose rows
// are already grouped (row r's are [s_off[r], s_off[r+1]), columns in any
// order) are sorted by (row, column), reduced to the last write of every key
// (aos_array_buffer.hpp:76-101), freed of zeros (csr_build.hpp:32-98) and
// written to their final places, offsets included, by one kernel.
//
// Consecutive rows form tiles of at most RT_CAP entries, one block each:
//   1. a bitmap marks the rows' first entries; an entry's row is a popcount;
//   2. bucket order: row of L entries at local position s, column c goes to
//      bucket s + floor(c * L / 2^cbits), so bucket order is (row, column)
//      order and a bucket of uniform columns holds one entry on average. One
//      shared-memory counter per bucket ranks the arrivals, one scan turns
//      the counters into slots. Buckets of more than RT_LIM entries (columns
//      clustered in a long row, or many duplicates) are split again over
//      their own column range until none is left. A long row with more entries
//      than columns in its range needs none of this: a cell per column takes
//      the last position;
//   3. an entry's sorted place is its bucket's first slot plus the bucket's
//      entries before it by (column, input position): a few compares, for
//      four entries at a time;
//   4. the last entry of a run of equal columns is the last write; its keep
//      bit is a ballot, the tile's kept count goes through an ordered scan
//      (look-back), and the tile writes its rows' offsets and entries into
//      the CSR, consecutive threads on consecutive entries.
// Rows of more than RT_CAP entries are ordered beforehand by larger blocks
// (the same steps, two sizes) into scratch at their input positions; their
// tiles copy. Rows of more than RT_BIG entries fit no block: when the plan
// meets some, the kernels stop, those rows' entries alone are sorted by column
// (order_huge_rows), and a second run gives each its place, where a pass over
// all of them puts their entries (10 M shuffled inserts, five to a row, with one
// row of 20 000: 0.79 ms, 0.70 without it; all of them sorted by (row, column)
// 1.24, and 1.59 when the row sort and the tiles had been tried before that).
//
// Floor: 24 bytes per entry of HBM traffic (12 in, 12 out). Bound: latency
// between the fifteen barriers of a tile, at 60 % of the issue slots: on the
// 64 M entries of the 4M-row Zipf(1.8) matrix 0.75 ms for the tiles, 0.38 for
// the longer rows (0.23 at the copy rate). Hence small blocks, four of 256
// threads an SM: two of 512 threads with 4096 entries took 1.03 + 0.26 ms,
// of which walking one bucket at a time (step 3; four entries' walks now run
// side by side) 0.13 and copying long rows one load at a time 0.06. It
// replaces per-class sorting kernels (a segmented bitonic network up to 32 entries, a warp bitonic network up to
// 512, LSD radix blocks up to 12 288: 145 instructions per entry and radix
// pass) followed by a compaction pass over all entries.
#include <algorithm>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int RT_CAP = 2048;            // entries of a tile
constexpr int RT_T = 256, RT_PER_SM = 4;
constexpr int RT_MID = 4096, RT_MID_T = 512, RT_MID_PER_SM = 2;  // longer rows: blocks for up to RT_MID entries ...
constexpr int RT_BIG = 12288, RT_BIG_T = 1024;                   // ... and for up to RT_BIG, the longest a block takes
// Rows above RT_LONG entries spread over their own column range, which two
// atomics an entry find, shorter ones over the matrix's columns. At 64, rows of
// 33..64 clustered entries split their buckets again and again (60 k rows of 64
// on 200 columns 265 us, 222 at 32; rows of 40 uniform columns 387 / 425).
constexpr int RT_LONG = 32;
constexpr int RT_LIM = 32;              // longest bucket ordered by counting
constexpr int RT_FEW_CBITS = 14;
constexpr unsigned RT_STATUS_TIMEOUT = 0x20u;

// Counters at the head of the scratch words.
enum : int { RC_PLAN_TICKET = 0, RC_TICKET = 1, RC_TILES = 2, RC_BIG = 3, RC_OVERFLOW = 4, RC_MID = 5, RC_MID_TICKET = 6, RC_BIG_TICKET = 7, RC_HUGE = 8, RC_N = 9 };
constexpr int RC_HUGE_BITS = 24;  // RC_HUGE: rows in the low bits (2^32 / 12 289 at most), their entries above

struct RtArgs {
    const uint32_t *cols;
    const double *vals;
    const uint64_t *s_off;
    uint64_t n_rows;
    int cbits;
    bool keep_zeros;
    unsigned long long *ctr;
    unsigned long long *plan_state, *tile_state;
    uint64_t *tile_start;  // first row of each tile, then n_rows (2^32 in the transpose of a matrix of 2^32 columns)
    uint32_t *longer;      // rows of RT_CAP+1 .. RT_MID entries from the front, longer ones from the back
    uint64_t n_longer;
    uint32_t *huge;        // rows of more than RT_BIG entries
    bool huge_ready;       // they are ordered: off[r] holds such a row's kept count
    uint32_t *big_cols;    // their ordered entries, at the rows' input positions
    double *big_vals;
    uint64_t *off;         // out; off[r] holds a big row's kept count until its tile is written
    uint32_t *out_cols;
    double *out_vals;
    const unsigned long long *abort;  // may be null: the inputs are not to be read if set
    unsigned int *status;
    unsigned long long *words;  // [0] 1: rows too long are listed, nothing is built; [1] entries kept, or such rows; [2] their entries
};

// ---------------------------------------------------------------- tile plan
// A block packs RP_ROWS consecutive rows into tiles greedily: a tile takes
// rows while they fit RT_CAP entries; a longer row is a tile of its own. (Tiles
// cut at fixed windows of the entries, with long rows at a window's end set
// apart, were a third full on the Zipf(1.8) matrix.) Blocks with many entries
// cut their rows into up to RP_SUB equal parts, a warp each, so that matrices
// of long rows do not wait for one warp's steps.
constexpr int RP_T = 256, RP_ROWS = 2048, RP_SUB = RP_T / 32;
constexpr uint64_t RP_PART = 16 * RT_CAP;  // entries per part before a block is cut further

__global__ void __launch_bounds__(RP_T) rt_plan(RtArgs a) {
    __shared__ uint64_t s_off[RP_ROWS + 1];
    __shared__ uint16_t s_list[RP_ROWS];  // tile starts, part w's from its first row on
    __shared__ uint32_t s_n[RP_SUB];
    __shared__ uint64_t s_t, s_base;
    __shared__ int s_ok;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (a.abort && *a.abort) {
        a.ctr[RC_OVERFLOW] = 1ull;
        return;
    }
    if (t == 0) s_t = atomicAdd(a.ctr + RC_PLAN_TICKET, 1ull);
    __syncthreads();
    const uint64_t blk = s_t, r0 = blk * RP_ROWS;
    const int nr = (int)min((uint64_t)RP_ROWS, a.n_rows - r0);
    for (int j = t; j <= nr; j += RP_T) s_off[j] = a.s_off[r0 + j];
    __syncthreads();
    const int parts = (int)min((uint64_t)RP_SUB, (s_off[nr] - s_off[0]) / RP_PART + 1);
    const int per = (nr + parts - 1) / parts;
    const int p0 = min(nr, warp * per), p1 = warp < parts ? min(nr, p0 + per) : p0;
    uint32_t n = 0, huge = 0;
    for (int r = p0; r < p1;) {
        if (lane == 0) s_list[p0 + n] = (uint16_t)r;
        ++n;
        // the last end e in (r, p1] with s_off[e] - s_off[r] <= RT_CAP: 32
        // probes 64 rows apart, then 32 two rows apart, then one
        const uint64_t lim = s_off[r] + RT_CAP;
        int e = r;
        e = min(p1, e + 64 * __popc(__ballot_sync(0xffffffffu, e + 64 * (lane + 1) <= p1 && s_off[min(p1, e + 64 * (lane + 1))] <= lim)));
        e = min(p1, e + 2 * __popc(__ballot_sync(0xffffffffu, e + 2 * (lane + 1) <= p1 && s_off[min(p1, e + 2 * (lane + 1))] <= lim)));
        if (e < p1 && s_off[e + 1] <= lim) ++e;
        if (e == r) {  // longer than a tile
            const uint64_t L = s_off[r + 1] - s_off[r];
            if (lane == 0) {
                if (L > (uint64_t)RT_BIG) ++huge;
                else if (L > (uint64_t)RT_MID) a.longer[a.n_longer - 1 - atomicAdd(a.ctr + RC_BIG, 1ull)] = (uint32_t)(r0 + r);
                else a.longer[atomicAdd(a.ctr + RC_MID, 1ull)] = (uint32_t)(r0 + r);
            }
            ++e;
        }
        r = e;
    }
    if (lane == 0) s_n[warp] = n;
    __syncwarp();
    if (!a.huge_ready && __shfl_sync(0xffffffffu, huge, 0)) {  // (listed here, 32 tiles at a time: an atomic each in the loop waits)
        if (lane == 0) a.ctr[RC_OVERFLOW] = 1ull;
        for (uint32_t k0 = 0; k0 < n; k0 += 32) {
            const int r = k0 + lane < n ? s_list[p0 + k0 + lane] : p0;
            const uint64_t L = k0 + lane < n ? s_off[r + 1] - s_off[r] : 0;
            if (L > (uint64_t)RT_BIG) {
                const unsigned long long at = atomicAdd(a.ctr + RC_HUGE, (unsigned long long)L << RC_HUGE_BITS | 1ull);
                a.huge[at & ((1ull << RC_HUGE_BITS) - 1)] = (uint32_t)(r0 + r);
            }
        }
    }
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < RP_SUB; ++w) {
        if (w < warp) before += s_n[w];
        total += s_n[w];
    }
    if (warp == 0) {
        uint64_t b = 0;
        const bool ok = lookback_scan(a.plan_state, blk, total, &b, lane, a.status, RT_STATUS_TIMEOUT, LB_WAIT_CYCLES);
        if (lane == 0) {
            s_ok = ok ? 1 : 0;
            s_base = b;
        }
    }
    __syncthreads();
    if (!s_ok) return;  // (the tile kernel then has no tiles; the status word fails the call)
    for (uint32_t k = lane; k < n; k += 32) a.tile_start[s_base + before + k] = r0 + s_list[p0 + k];
    if (t == 0 && r0 + RP_ROWS >= a.n_rows) {
        a.tile_start[s_base + total] = a.n_rows;
        a.ctr[RC_TILES] = s_base + total;
    }
}

// ------------------------------------------------------------ ordering a tile
// scol / spos: column and input position, by slot. val / col: the kept
// entries in order (APART: they outlive the next tile's slots).
template <int CAP, bool APART>
struct RtArrays {
    uint32_t scol[CAP];
    uint16_t spos[CAP];
    double val[CAP];
    uint32_t col[CAP];
};
template <int CAP>
struct RtArrays<CAP, false> {
    union {
        struct {
            uint32_t scol[CAP];
            uint16_t spos[CAP];
        };
        struct {
            double val[CAP];
            uint32_t col[CAP];
        };
    };
};

template <int T, int CAP, bool APART>
struct RtSmem : RtArrays<CAP, APART> {
    uint32_t cnt[CAP / 2 + 2];     // 16-bit bucket counters, then the buckets' first slots
    uint32_t keep[CAP / 32];       // bit: the entry in place f is kept
    uint16_t kpre[CAP / 32];       // kept entries before place 32 w
    uint32_t head[CAP / 32 + 2];   // bit: a row's first entry
    uint16_t wbeg[CAP / 32 + 2];   // start of the row that entry 32 w continues
    uint16_t wend[CAP / 32 + 2];   // end of the row that holds entry 32 w + 31
    uint32_t wsum[32];
    BlockLookback<T> lb;
    struct Tile {
        uint64_t id, r0, r1, s0, s1;  // its rows and their entries
        uint32_t total;               // kept entries
        uint32_t copied;              // of a longer row: those that its tile copies
    } tile[3];  // this one, the one before (sorted, not yet written) and the next
};

// The block's next tile (one thread): its ticket and the ends of its rows.
template <class Tile>
__device__ __forceinline__ void rt_take(Tile &x, const RtArgs &a, uint64_t n_tiles) {
    const uint64_t id = atomicAdd(a.ctr + RC_TICKET, 1ull);
    x.id = id;
    if (id < n_tiles) {
        x.r0 = a.tile_start[id];
        x.r1 = a.tile_start[id + 1];
        x.s0 = a.s_off[x.r0];
        x.s1 = a.s_off[x.r1];
    }
}

// Marks the non-empty row [b, e) of the tile. A long row's first two cells of
// scol will hold its least and greatest column.
template <class Smem>
__device__ __forceinline__ void rt_mark_row(Smem &S, int b, int e) {
    if (e - b > RT_LONG) {
        S.scol[b] = 0xFFFFFFFFu;
        S.scol[b + 1] = 0;
    }
    atomicOr(&S.head[b >> 5], 1u << (b & 31));
    for (int w = (b >> 5) + 1; 32 * w < e; ++w) S.wbeg[w] = (uint16_t)b;
    for (int w = b >> 5; 32 * w + 32 <= e; ++w) S.wend[w] = (uint16_t)e;
}

// Thread t's columns of a tile: c[i] = that of entry t + i T.
template <int T, int CAP>
__device__ __forceinline__ void rt_load(uint32_t (&c)[CAP / T], const uint32_t *__restrict__ cols, int E) {
#pragma unroll
    for (int i = 0; i < CAP / T; ++i) c[i] = (int)threadIdx.x + i * T < E ? cols[threadIdx.x + i * T] : 0u;
}

// Least and greatest column of the row or bucket at `lo` into its cells; one
// pair of atomics when the whole warp has the same one. All lanes call.
template <class Smem>
__device__ __forceinline__ void rt_minmax(Smem &S, uint32_t lo, bool on, uint32_t c, int lane) {
    if (!__any_sync(0xffffffffu, on)) return;
    const uint32_t lo0 = __shfl_sync(0xffffffffu, lo, 0);
    if (__all_sync(0xffffffffu, on && lo == lo0)) {
        const uint32_t mn = __reduce_min_sync(0xffffffffu, c), mx = __reduce_max_sync(0xffffffffu, c);
        if (lane == 0) {
            atomicMin(&S.scol[lo], mn);
            atomicMax(&S.scol[lo + 1], mx);
        }
    } else if (on) {
        atomicMin(&S.scol[lo], c);
        atomicMax(&S.scol[lo + 1], c);
    }
}

// Orders a tile's E entries, whose columns are c and whose rows are marked in
// S (not yet synchronised; S.cnt is zero up to counter E) by (row, column,
// position), keeps the last of every run of equal columns of a row unless its
// value is zero, and returns the number kept (in every thread). S.keep / kpre
// have the keep bits by sorted place; pk[i] is the kept entry's index among the
// kept ones, or ~0 for a dropped one; v[i] its value. REPEATS: for matrices
// whose long rows may have more entries than columns.
template <bool REPEATS, int T, int CAP, bool APART>
__device__ __forceinline__ uint32_t rt_order(RtSmem<T, CAP, APART> &S, const uint32_t (&c)[CAP / T],
                                             const double *__restrict__ vals, int E, int cbits, bool keep_zeros,
                                             uint32_t (&pk)[CAP / T], double (&v)[CAP / T]) {
    constexpr int I = CAP / T, CW = I / 2, P = CAP / 1024;
    static_assert(CAP % T == 0 && (I % 4 == 0) && CAP % 1024 == 0, "whole words per thread");
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int shift = cbits ? 32 - cbits : 0;  // (cbits == 0: the only column is 0)
    uint16_t *cnt16 = reinterpret_cast<uint16_t *>(S.cnt);
    __syncthreads();
    // the entry's row [lo, hi); a warp's 32 entries are word w's
#pragma unroll
    for (int i = 0; i < I; ++i) {
        if (i * T >= E) break;  // (the same for the whole block)
        const int e = t + i * T, w = e >> 5;
        uint32_t lo = 0, hi = 0;
        if (e < E) {
            const uint32_t m = S.head[w], upto = 0xffffffffu >> (31 - lane), below = m & upto, above = m & ~upto;
            lo = below ? 32 * w + 31 - __clz((int)below) : S.wbeg[w];
            hi = above ? 32 * w + __ffs((int)above) - 1 : 32 * w + 32 >= E ? E : S.wend[w];
        }
        pk[i] = lo << 16 | hi;
        const bool long_row = hi - lo > (uint32_t)RT_LONG;
        if (REPEATS && long_row && e >= (int)lo + 2) S.scol[e] = 0;
        rt_minmax(S, lo, long_row, c[i], lane);
    }
    __syncthreads();
    // bit i: entry i has a later write (found below); bit 16 + i (REPEATS only):
    // its row has more entries than columns in its range, and a cell of S.scol
    // for each of them (from the third on), which takes the greatest position:
    // nothing else of such a row is kept, and its place is its column
    uint32_t flags = 0;
    auto exact = [&](int i) { return REPEATS && ((flags >> (16 + i)) & 1u); };
    static_assert(I <= 16, "two bits per entry");
#pragma unroll
    for (int i = 0; i < I; ++i) {
        const int e = t + i * T;
        if (e < E) {
            const uint32_t lo = pk[i] >> 16, L = (pk[i] & 0xFFFFu) - lo;
            uint32_t x = c[i] << shift;
            if (L > (uint32_t)RT_LONG) {
                const uint32_t mn = S.scol[lo], range = S.scol[lo + 1] - mn;
                if (REPEATS && range < L - 2) {
                    const uint32_t f = lo + (c[i] - mn);
                    atomicMax(&S.scol[f + 2], (uint32_t)e + 1);
                    pk[i] = f << 16 | f;
                    flags |= 0x10000u << i;
                    continue;
                }
                x = (c[i] - mn) << min(31, __clz((int)range));
            }
            pk[i] = lo + __umulhi(x, L);
        }
    }
    // pk: bucket; after counting, bucket << 16 | rank of arrival
    while (true) {
#pragma unroll
        for (int i = 0; i < I; ++i) {
            if (exact(i)) {  // (so that the other rows' slots start at their first entries)
                atomicAdd(&S.cnt[(t + i * T) >> 1], 1u << (((t + i * T) & 1) * 16));
            } else if (t + i * T < E) {
                const uint32_t sh = (pk[i] & 1u) * 16u;
                const uint32_t v = atomicAdd(&S.cnt[pk[i] >> 1], 1u << sh);
                pk[i] = pk[i] << 16 | ((v >> sh) & 0xFFFFu);
            }
        }
        __syncthreads();
        // exclusive scan of the counters, thread t's are [t I, t I + I)
        uint32_t x[CW], sum = 0;
        bool over = false;
#pragma unroll
        for (int j = 0; j < CW; ++j) {
            x[j] = t * I + 2 * j < E ? S.cnt[t * CW + j] : 0u;
            over |= (x[j] & 0xFFFFu) > (uint32_t)RT_LIM || (x[j] >> 16) > (uint32_t)RT_LIM;
            sum += (x[j] & 0xFFFFu) + (x[j] >> 16);
        }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) S.wsum[warp] = inc;
        __syncthreads();
        uint32_t run = inc - sum + __reduce_add_sync(0xffffffffu, lane < warp ? S.wsum[lane] : 0u);
#pragma unroll
        for (int j = 0; j < CW; ++j) {
            const uint32_t first = run;
            run += x[j] & 0xFFFFu;
            if (t * I + 2 * j <= E) S.cnt[t * CW + j] = first | run << 16;  // up to slot E, the end
            run += x[j] >> 16;
        }
        if (t == T - 1 && E == CAP) cnt16[CAP] = (uint16_t)run;
        if (!__syncthreads_or(over)) break;
        // Rare: buckets longer than RT_LIM are spread over their slots again,
        // by their own column range; one of equal columns only keeps every
        // entry but the last write (the largest position) in arrival order.
        // The bucket's cells of S.scol hold its least and greatest column, its
        // last position and that entry's arrival rank.
#pragma unroll
        for (int i = 0; i < I; ++i) {
            if (t + i * T < E && !exact(i) && (pk[i] & 0xFFFFu) == 0) {
                const uint32_t lo = cnt16[pk[i] >> 16], len = cnt16[(pk[i] >> 16) + 1] - lo;
                if (len > (uint32_t)RT_LIM) {
                    S.scol[lo] = 0xFFFFFFFFu;
                    S.scol[lo + 1] = 0;
                    S.scol[lo + 2] = 0;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < I; ++i) {
            uint32_t lo = 0, len = 0;
            if (t + i * T < E && !exact(i)) {
                lo = cnt16[pk[i] >> 16];
                len = cnt16[(pk[i] >> 16) + 1] - lo;
            }
            const bool on = len > (uint32_t)RT_LIM;
            rt_minmax(S, lo, on, c[i], lane);
            // the last position: a lane's is above those of the lanes before it
            const bool more = __shfl_down_sync(0xffffffffu, on ? lo : ~0u, 1) == lo && lane < 31;
            if (on && !more) atomicMax(&S.scol[lo + 2], (uint32_t)(t + i * T));
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < I; ++i) {
            if (t + i * T < E && !exact(i)) {
                const uint32_t lo = cnt16[pk[i] >> 16], len = cnt16[(pk[i] >> 16) + 1] - lo;
                if (len > (uint32_t)RT_LIM && S.scol[lo + 2] == (uint32_t)(t + i * T)) S.scol[lo + 3] = pk[i] & 0xFFFFu;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < I; ++i) {
            if (t + i * T < E && !exact(i)) {
                const uint32_t lo = cnt16[pk[i] >> 16], len = cnt16[(pk[i] >> 16) + 1] - lo;
                uint32_t b = lo;  // a short bucket keeps its slots: they are its own
                if (len > (uint32_t)RT_LIM) {
                    const uint32_t mn = S.scol[lo], mx = S.scol[lo + 1];
                    if (mn < mx) {
                        b = lo + __umulhi((c[i] - mn) << __clz((int)(mx - mn)), len);
                    } else {
                        const uint32_t r = pk[i] & 0xFFFFu, last = S.scol[lo + 3];
                        b = lo + (r == last ? len - 1 : r > last ? r - 1 : r);
                        if (r != last) flags |= 1u << i;
                    }
                }
                pk[i] = b;
            }
        }
        __syncthreads();  // the counters are read
        for (int w = t; w < E / 2 + 1; w += T) S.cnt[w] = 0;
        __syncthreads();
    }
    // slots: the bucket's first plus the rank of arrival; pk: bucket's ends
#pragma unroll
    for (int i = 0; i < I; ++i) {
        const int e = t + i * T;
        if (exact(i)) {
            if (S.scol[(pk[i] & 0xFFFFu) + 2] != (uint32_t)e + 1) flags |= 1u << i;
        } else if (e < E) {
            const uint32_t b = pk[i] >> 16, lo = cnt16[b], hi = cnt16[b + 1];
            S.scol[lo + (pk[i] & 0xFFFFu)] = c[i];
            S.spos[lo + (pk[i] & 0xFFFFu)] = (uint16_t)e;
            pk[i] = lo << 16 | hi;
        }
    }
#pragma unroll
    for (int i = 0; i < I; ++i) v[i] = t + i * T < E ? vals[t + i * T] : 0.0;
    for (int w = t; w < CAP / 32; w += T) S.keep[w] = 0;
    __syncthreads();
    // place: the bucket's first slot plus the bucket's entries before this one;
    // dropped if the bucket has a later write of its column
    // (four entries' walks side by side, as a walk alone waits for every load;
    // but not with the few registers of a thread of RT_BIG_T)
    constexpr int G = T == RT_BIG_T ? 1 : 4;
#pragma unroll
    for (int i0 = 0; i0 < I; i0 += G) {
        uint32_t acc[G], most = 0;  // entries before | entries of the same column << 16
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (t + (i0 + g) * T >= E) pk[i0 + g] = 0;
            const uint32_t len = (pk[i0 + g] & 0xFFFFu) - (pk[i0 + g] >> 16);
            most = max(most, len);
            acc[g] = 0;
        }
        if (G == 1) {
            if (most > 1) {
                for (uint32_t j = pk[i0] >> 16; j < (pk[i0] & 0xFFFFu); ++j) {
                    const uint32_t cj = S.scol[j];
                    acc[0] += cj < c[i0] ? 1u : 0u;
                    acc[0] += cj == c[i0] ? 0x10000u : 0u;
                }
            }
        } else if (most > 1) {
            for (uint32_t j = 0; j < most; ++j) {
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const uint32_t q = (pk[i0 + g] >> 16) + j;
                    if (q < (pk[i0 + g] & 0xFFFFu)) {
                        const uint32_t cj = S.scol[q];
                        acc[g] += cj < c[i0 + g] ? 1u : 0u;
                        acc[g] += cj == c[i0 + g] ? 0x10000u : 0u;
                    }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int i = i0 + g, e = t + i * T;
            if (e < E) {
                const uint32_t lo = pk[i] >> 16, hi = pk[i] & 0xFFFFu;
                uint32_t f = lo + (acc[g] & 0xFFFFu);
                bool kept = !((flags >> i) & 1u) && (keep_zeros || !is_zero(v[i]));
                if (acc[g] >= 0x20000u) {
                    for (uint32_t j = lo; j < hi; ++j) {
                        if (S.scol[j] == c[i]) {
                            f += S.spos[j] < e ? 1u : 0u;
                            kept = kept && S.spos[j] <= e;
                        }
                    }
                }
                pk[i] = kept ? f : ~0u;
                if (kept) atomicOr(&S.keep[f >> 5], 1u << (f & 31));
            }
        }
    }
    __syncthreads();
    // every warp scans the words' counts for itself (lane l has words [l P,
    // l P + P)) and leaves the same prefixes in S.kpre: no barrier
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < P; ++j) sum += __popc(S.keep[lane * P + j]);
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
    }
    uint32_t run = inc - sum;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        S.kpre[lane * P + j] = (uint16_t)run;
        run += __popc(S.keep[lane * P + j]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < I; ++i) {
        if (t + i * T < E && pk[i] != ~0u) {
            const uint32_t f = pk[i];
            pk[i] = S.kpre[f >> 5] + __popc(S.keep[f >> 5] & ((1u << (f & 31)) - 1u));
        }
    }
    return __shfl_sync(0xffffffffu, inc, 31);
}

// Rows longer than a tile, a block each (taken from the list one by one):
// ordered and compacted into scratch at the row's input positions.
template <int T, int CAP, int PER_SM, int COUNT, int TICKET, bool REPEATS>
__global__ void __launch_bounds__(T, PER_SM) rt_long_rows(RtArgs a) {
    constexpr int I = CAP / T;
    __shared__ uint64_t s_next;
    extern __shared__ __align__(16) unsigned char rt_raw[];
    auto &S = *reinterpret_cast<RtSmem<T, CAP, false> *>(rt_raw);
    const int t = threadIdx.x;
    if (a.ctr[RC_OVERFLOW]) return;
    const uint64_t n = a.ctr[COUNT];
    while (true) {
        if (t == 0) s_next = atomicAdd(a.ctr + TICKET, 1ull);
        __syncthreads();
        const uint64_t k = s_next;
        if (k >= n) return;
        const uint64_t r = a.longer[COUNT == RC_BIG ? a.n_longer - 1 - k : k], s0 = a.s_off[r];
        const int E = (int)(a.s_off[r + 1] - s0);
        uint32_t c[I], o[I];
        double v[I];
        rt_load<T, CAP>(c, a.cols + s0, E);
        for (int w = t; w < CAP / 32 + 2; w += T) {
            S.head[w] = w == 0 ? 1u : 0u;
            S.wbeg[w] = 0;
            S.wend[w] = (uint16_t)E;
        }
        if (t < 2) S.scol[t] = t == 0 ? 0xFFFFFFFFu : 0u;  // the row's cells
        for (int w = t; w < E / 2 + 1; w += T) S.cnt[w] = 0;
        const uint32_t total = rt_order<REPEATS, T, CAP, false>(S, c, a.vals + s0, E, a.cbits, a.keep_zeros, o, v);
#pragma unroll
        for (int i = 0; i < I; ++i) {
            if (t + i * T < E && o[i] != ~0u) {
                S.col[o[i]] = c[i];
                S.val[o[i]] = v[i];
            }
        }
        __syncthreads();
        for (uint32_t q = t; q < total; q += T) {
            a.big_cols[s0 + q] = S.col[q];
            a.big_vals[s0 + q] = S.val[q];
        }
        if (t == 0) a.off[r] = total;
        __syncthreads();  // the shared state is rebuilt by the next row
    }
}

// Tiles in ticket order. A tile's place in the CSR is known once every tile
// before it is sorted, and waiting for that idled the block for as long as the
// sort took (tiles differ, and the slowest of all in flight holds up the
// rest). So a block publishes a sorted tile's count, keeps its entries in
// shared memory and sorts the next tile before it writes this one, whose
// place is known by then.
template <bool REPEATS>
__global__ void __launch_bounds__(RT_T, RT_PER_SM) rt_tiles(RtArgs a) {
    constexpr int T = RT_T, CAP = RT_CAP, I = CAP / T;
    extern __shared__ __align__(16) unsigned char rt_raw[];
    auto &S = *reinterpret_cast<RtSmem<T, CAP, true> *>(rt_raw);
    const int t = threadIdx.x;
    if (a.ctr[RC_OVERFLOW]) {
        if (blockIdx.x == 0 && t == 0) {
            store_word(a.words, 0, 1ull);
            store_word(a.words, 1, a.ctr[RC_HUGE] & ((1ull << RC_HUGE_BITS) - 1));
            store_word(a.words, 2, a.ctr[RC_HUGE] >> RC_HUGE_BITS);
        }
        return;
    }
    const uint64_t n_tiles = a.ctr[RC_TILES];
    if (t == 0) rt_take(S.tile[0], a, n_tiles);
    __syncthreads();
    uint32_t row_p = 0;  // the place in its tile of row r0 + t of the tile sorted last
    for (unsigned it = 0;; ++it) {
        auto &cur = S.tile[it % 3], &prev = S.tile[(it + 2) % 3];
        const bool have = cur.id < n_tiles;
        uint32_t c[I], o[I], total = 0, row_b = 0;
        double v[I];
        int E = -1;  // < 0: a row ordered by rt_long_rows, or no tile
        if (have) {
            const uint64_t r0 = cur.r0, r1 = cur.r1, s0 = cur.s0;
            if (cur.s1 - s0 <= (uint64_t)CAP) {
                E = (int)(cur.s1 - s0);
                rt_load<T, CAP>(c, a.cols + s0, E);
                const uint64_t mine = min(r0 + t, r1 - 1), b0 = a.s_off[mine], e0 = a.s_off[mine + 1];
                for (int w = t; w < CAP / 32 + 2; w += T) S.head[w] = 0;
                for (int w = t; w < E / 2 + 1; w += T) S.cnt[w] = 0;
                __syncthreads();
                row_b = (uint32_t)(b0 - s0);
                if (r0 + t < r1 && b0 != e0) rt_mark_row(S, (int)(b0 - s0), (int)(e0 - s0));
                for (uint64_t r = r0 + t + T; r < r1; r += T) {
                    const uint64_t b = a.s_off[r], e = a.s_off[r + 1];
                    if (b != e) rt_mark_row(S, (int)(b - s0), (int)(e - s0));
                }
                total = rt_order<REPEATS, T, CAP, true>(S, c, a.vals + s0, E, a.cbits, a.keep_zeros, o, v);
            } else {
                total = (uint32_t)a.off[r0];
                if (t == 0) cur.copied = cur.s1 - cur.s0 <= (uint64_t)RT_BIG ? total : 0;  // (the others by rt_huge_rows)
            }
            if (t == 0) {
                cur.total = total;
                atomicExch(a.tile_state + cur.id, (cur.id == 0 ? 0ull + LB_PREFIX : 0ull + LB_AGG) | total);
            }
        }
        if (it > 0) {
            uint64_t base = 0;
            if (!block_lookback<T>(S.lb, a.tile_state, prev.id, prev.total, base, a.status, RT_STATUS_TIMEOUT)) return;
            const uint32_t n = prev.total;
            if (prev.s1 - prev.s0 <= (uint64_t)CAP) {
                for (uint32_t k = t; k < n; k += T) {
                    a.out_cols[base + k] = S.col[k];
                    a.out_vals[base + k] = S.val[k];
                }
                if (prev.r0 + t < prev.r1) a.off[prev.r0 + t] = base + row_p;
                for (uint64_t r = prev.r0 + t + T; r < prev.r1; r += T) {
                    const uint64_t p = a.off[r];  // within the tile: this thread's own
                    a.off[r] = p + base;
                }
            } else {  // one row, eight loads of a thread in flight (one pair at a time: 55 us more on the Zipf matrix)
                constexpr int U = 4;
                const uint32_t copied = prev.copied;
                for (uint32_t k0 = t; k0 < copied; k0 += U * T) {
                    uint32_t cc[U];
                    double vv[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t k = k0 + u * T;
                        cc[u] = k < copied ? a.big_cols[prev.s0 + k] : 0u;
                        vv[u] = k < copied ? a.big_vals[prev.s0 + k] : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t k = k0 + u * T;
                        if (k < copied) {
                            a.out_cols[base + k] = cc[u];
                            a.out_vals[base + k] = vv[u];
                        }
                    }
                }
                if (t == 0) a.off[prev.r0] = base;
            }
            if (t == 0 && prev.r1 == a.n_rows) {
                a.off[a.n_rows] = base + n;
                store_word(a.words, 0, 0ull);
                store_word(a.words, 1, base + n);
            }
        }
        if (!have) return;
        if (t == 32) rt_take(S.tile[(it + 1) % 3], a, n_tiles);
        __syncthreads();  // the tile before is written
        if (E >= 0) {
            const uint64_t r0 = cur.r0, r1 = cur.r1, s0 = cur.s0;
#pragma unroll
            for (int i = 0; i < I; ++i) {
                if (t + i * T < E && o[i] != ~0u) {
                    S.col[o[i]] = c[i];
                    S.val[o[i]] = v[i];
                }
            }
            for (uint64_t r = r0 + t; r < r1; r += T) {
                const uint32_t p = r == r0 + t ? row_b : (uint32_t)(a.s_off[r] - s0);
                const uint32_t q = p == (uint32_t)E ? total : S.kpre[p >> 5] + __popc(S.keep[p >> 5] & ((1u << (p & 31)) - 1u));
                if (r == r0 + t) row_p = q;
                else a.off[r] = q;
            }
        }
        __syncthreads();
    }
}

// The kept entries of the rows that fit no block, to their rows' places.
__global__ void __launch_bounds__(256)
rt_huge_rows(const uint32_t *__restrict__ huge, const uint32_t *__restrict__ row, const uint32_t *__restrict__ cols,
             const double *__restrict__ vals, const uint64_t *__restrict__ first, uint64_t n_huge,
             const unsigned int *status, const uint64_t *__restrict__ off, uint32_t *__restrict__ out_cols,
             double *__restrict__ out_vals) {
    __shared__ unsigned int gave_up;
    if (threadIdx.x == 0) gave_up = *(const volatile unsigned int *)status;
    __syncthreads();
    if (gave_up) return;  // a wait of the tiles: not every place is known
    const uint64_t n = first[n_huge];
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t q = row[i];
        const uint64_t o = off[huge[q]] + (i - first[q]);
        out_cols[o] = cols[i];
        out_vals[o] = vals[i];
    }
}

// Plan, longer rows, tiles.
template <bool REPEATS>
int rt_run(Ctx *c, const RtArgs &a, uint64_t plan_tiles, uint64_t t_max, uint64_t m, cudaStream_t s) {
    rt_plan<<<(unsigned)plan_tiles, RP_T, 0, s>>>(a);
    SPG_LAUNCH_CHECK();
    if (m > (uint64_t)RT_CAP) {
        auto k = rt_long_rows<RT_MID_T, RT_MID, RT_MID_PER_SM, RC_MID, RC_MID_TICKET, REPEATS>;
        constexpr size_t smem = sizeof(RtSmem<RT_MID_T, RT_MID, false>);
        SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<(unsigned)std::min<uint64_t>(a.n_longer, (uint64_t)c->n_sms * RT_MID_PER_SM), RT_MID_T, smem, s>>>(a);
        SPG_LAUNCH_CHECK();
    }
    if (m > (uint64_t)RT_MID) {
        auto k = rt_long_rows<RT_BIG_T, RT_BIG, 1, RC_BIG, RC_BIG_TICKET, REPEATS>;
        constexpr size_t smem = sizeof(RtSmem<RT_BIG_T, RT_BIG, false>);
        SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<(unsigned)std::min<uint64_t>(m / (RT_MID + 1), (uint64_t)c->n_sms), RT_BIG_T, smem, s>>>(a);
        SPG_LAUNCH_CHECK();
    }
    constexpr size_t smem = sizeof(RtSmem<RT_T, RT_CAP, true>);
    SPG_CUDA_TRY(cudaFuncSetAttribute(rt_tiles<REPEATS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned blocks = (unsigned)std::min<uint64_t>(t_max, (uint64_t)c->n_sms * RT_PER_SM);
    rt_tiles<REPEATS><<<blocks, RT_T, smem, s>>>(a);
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

}  // namespace

int build_grouped_rows(Ctx *c, const uint32_t *cols, const double *vals, const uint64_t *s_off,
                       uint64_t m, uint64_t n_rows, int cbits, bool near, bool keep_zeros,
                       const unsigned long long *abort, GroupedOut *out, bool *done, cudaStream_t s) {
    *done = false;
    const uint64_t plan_tiles = (n_rows + RP_ROWS - 1) / RP_ROWS;
    // two neighbouring tiles of one part hold more than RT_CAP entries together
    const uint64_t t_max = 2 * (m / RT_CAP) + 2 * (plan_tiles + m / RP_PART) + 4;
    const bool may_long = m > (uint64_t)RT_CAP;
    const uint64_t n_long = m / (RT_CAP + 1) + 1, n_huge = m / (RT_BIG + 1);
    DevBuf state, tiles, longer, big_cols, big_vals;
    // (the outputs first: the scratch below is a little smaller, and took the
    // freed outputs of an earlier lock when it came first, so that the pool
    // mapped new memory for these at every call: 0.5 ms on the 4M-row matrix)
    SPG_TRY(out->off.alloc(csr_off_elems(n_rows) * sizeof(uint64_t), s));
    SPG_TRY(out->cols.alloc(csr_alloc_elems(m) * sizeof(uint32_t), s));
    SPG_TRY(out->vals.alloc(csr_alloc_elems(m) * sizeof(double), s));
    const size_t state_bytes = (RC_N + plan_tiles + t_max) * sizeof(unsigned long long);
    SPG_TRY(state.alloc(state_bytes, s));
    SPG_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, state_bytes, s));
    SPG_TRY(tiles.alloc((t_max + 1) * sizeof(uint64_t), s));
    SPG_TRY(longer.alloc((n_long + n_huge) * sizeof(uint32_t), s));
    if (may_long) {
        SPG_TRY(big_cols.alloc(m * sizeof(uint32_t), s));
        SPG_TRY(big_vals.alloc(m * sizeof(double), s));
    }
    RtArgs a{};
    a.cols = cols;
    a.vals = vals;
    a.s_off = s_off;
    a.n_rows = n_rows;
    a.cbits = cbits;
    a.keep_zeros = keep_zeros;
    a.ctr = state.as<unsigned long long>();
    a.plan_state = a.ctr + RC_N;
    a.tile_state = a.plan_state + plan_tiles;
    a.tile_start = tiles.as<uint64_t>();
    a.longer = longer.as<uint32_t>();
    a.n_longer = n_long;
    a.huge = a.longer + n_long;
    a.big_cols = big_cols.as<uint32_t>();
    a.big_vals = big_vals.as<double>();
    a.off = out->off.as<uint64_t>();
    a.out_cols = out->cols.as<uint32_t>();
    a.out_vals = out->vals.as<double>();
    a.abort = abort;
    a.status = c->d_status;
    a.words = c->d_words;
    // Long rows may have more inserts than columns where the matrix has few
    // columns or the rows' columns lie near each other. (The kernels for that:
    // 2000 inserts a row on 64 columns 573 -> 284 us, 20 k rows of 1000 on 300
    // neighbouring ones 570 -> 396; but 3 % of the 4M-row Zipf matrix's lock.)
    const bool repeats = near || cbits <= RT_FEW_CBITS;
    HugeRows H;
    while (true) {
        SPG_TRY(repeats ? rt_run<true>(c, a, plan_tiles, t_max, m, s) : rt_run<false>(c, a, plan_tiles, t_max, m, s));
        if (a.huge_ready)
            rt_huge_rows<<<grid_for(H.entries, 256, (unsigned)c->n_sms * 8), 256, 0, s>>>(
                a.huge, H.row.as<uint32_t>(), H.cols.as<uint32_t>(), H.vals.as<double>(), H.first.as<uint64_t>(), H.n,
                a.status, a.off, a.out_cols, a.out_vals);
        SPG_LAUNCH_CHECK();
        SPG_TRY(c->phase_sync(s));
        if (c->word(0) == 0) break;
        H.n = c->word(1);
        H.entries = c->word(2);
        // mostly such rows: the global sort (300 rows of 13 000 in 5 M columns 0.45
        // ms, apart 0.58)
        if (2 * H.entries > m) return SPG_OK;
        const int rc = order_huge_rows(c, cols, vals, s_off, a.huge, cbits, keep_zeros, &H, a.off, s);
        if (rc == SPG_ERR_NO_MEMORY) return SPG_OK;  // (the global sort needs less)
        SPG_TRY(rc);
        SPG_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, state_bytes, s));
        a.huge_ready = true;
        a.abort = H.abort.as<unsigned long long>();  // (the staged rows' own is clear, or the wait above had failed)
    }
    *done = true;
    out->n = c->word(1);
    return SPG_OK;
}

}  // namespace spg
