// spg_merge.cu — row-wise merge of two CSRs: A + B (serial/matrix_addition.hpp:
// 34-110, the result locked, csr_build.hpp:49,71) and a later lock's merge of
// the sorted delta into the old CSR (csr_build.hpp:126-488).
//
// Both inputs are in (row, column) order, so the result is one merge of two
// sorted sequences, cut into tiles of equal size whatever the rows' lengths:
// the items are A's entries, B's entries and the row ends, tile t takes the
// items [t MT_TILE, (t + 1) MT_TILE) of their merged order, and a warp per cut
// finds it by two 32-ary searches (the row by its item count off_A + off_B + r,
// then the place inside it). An equal pair is never cut apart. A block takes a
// tile, stages its columns and values in shared memory and
//   1. labels the entries with their rows (a scan over marks at row starts);
//   2. thread by thread, four neighbouring entries of one side, finds each
//      entry's place in the other side's row (one search, then short steps):
//      its merged place is its own index plus that one's, and an equal column
//      there is the collision;
//   3. keep bits by merged place (after adding or replacing values) and their
//      popcounts give the place among the kept entries; the tile's count goes
//      through the ordered scan (look-back), deferred by one tile as in
//      spg_rowtiles.cu, and the tile is written with its rows' offsets.
//
// Bound: 12 bytes per entry read and written. The entry-parallel form it
// replaces searched every entry's partner in global memory from both sides
// (0.28 ms each on the 1M-row Zipf pair), kept 64-bit flags and partners per
// entry, scanned them and moved the entries: 1.04 ms a call, 0.40 now (tiles
// 0.325 ms, cuts 0.028), of which 37 % is the walks of step 2, 14 % the writes,
// the rest waits between the tile's barriers. More entries per thread (8: 351,
// fewer and larger blocks: 382) or smaller blocks (321 + 42 for the cuts) are no
// faster.
#include <algorithm>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int MT_T = 256, MT_PER_SM = 6;  // threads, blocks per SM
constexpr int MT_E = 4;             // entries per thread, of one side
constexpr int MT_CAP = MT_T * MT_E; // staged entries: both sides, A's part padded to whole threads
constexpr int MT_TILE = MT_CAP - MT_E;  // items per tile (one more entry when a pair would be cut)
constexpr int MT_KW = MT_CAP <= 1024 ? 32 : (MT_CAP + 1023) / 1024 * 32;  // keep words, in whole lanes' shares
constexpr unsigned MT_STATUS_TIMEOUT = 0x40u;
static_assert(MT_KW * 32 >= MT_CAP && MT_KW % 32 == 0, "a bit per place");

struct __align__(16) MtSplit {
    uint64_t row, ia, ib;
    uint64_t rf;  // the first row that starts at or after the cut
};

struct MtArgs {
    CsrView A, B;
    uint64_t n_rows, n_tiles;
    const MtSplit *split;  // n_tiles + 1
    unsigned long long *ticket, *state;
    uint64_t *off;
    uint32_t *cols;
    double *vals;
    uint64_t room;  // entries that cols and vals have room for: those beyond are counted, not written
    unsigned int *status;
    unsigned long long *words;  // [0] entries kept
};

// The last row that starts at or before entry e (by a full warp).
__device__ __forceinline__ uint64_t mt_row_of(const uint64_t *__restrict__ off, uint64_t n_rows, uint64_t e, int lane) {
    uint64_t lo = 0, hi = n_rows;
    while (hi - lo > 1) {
        const uint64_t step = (hi - lo + 31) / 32, r = lo + (uint64_t)(lane + 1) * step;
        const unsigned n = __popc(__ballot_sync(0xffffffffu, r < hi && off[r] <= e));
        lo += n * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// How many of MT_SAMPLES entries of X, one from each of as many equal parts at
// a place of its own, are in Y too (a warp each, MT_SAMPLE_BLOCKS blocks): the
// last block stores the count in words[0], then 1 in words[1].
constexpr unsigned MT_SAMPLES = 1024, MT_SAMPLE_BLOCKS = MT_SAMPLES / 8;

__device__ void mt_sample(const CsrView &X, const CsrView &Y, uint64_t n_rows, unsigned long long *ctr,
                          unsigned long long *words) {
    const unsigned k = (blockIdx.x * 256u + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const uint64_t lo = X.nnz / MT_SAMPLES * k, e = lo + (k * 0x9E3779B1ull >> 8) % (X.nnz / MT_SAMPLES);
    const uint64_t row = mt_row_of(X.off, n_rows, e, lane);
    const uint32_t col = X.cols[e];
    uint64_t b = Y.off[row], n = Y.off[row + 1];
    bool hit = false;
    while (b < n && !hit) {  // 32-ary: the probes' columns ascend
        const uint64_t step = (n - b + 31) / 32, p = b + (uint64_t)lane * step;
        const uint32_t y = p < n ? Y.cols[p] : 0xFFFFFFFFu;
        hit = __any_sync(0xffffffffu, p < n && y == col);
        const unsigned le = __popc(__ballot_sync(0xffffffffu, p < n && y < col));
        if (le == 0) break;
        n = min(n, b + le * step);
        b += (le - 1) * step + 1;
    }
    const int hits = __syncthreads_count(hit && lane == 0);
    if (threadIdx.x == 0) {
        if (hits) atomicAdd(ctr, (unsigned long long)hits);
        __threadfence();
        if (atomicAdd(ctr + 1, 1ull) == MT_SAMPLE_BLOCKS - 1) {
            __threadfence();
            store_word(words, 0, *(volatile unsigned long long *)ctr);
            store_word_now(words, 1, 1ull);
        }
    }
}

// Cut t: the row holding item t MT_TILE, and how many of A's and B's entries
// come before it. With a sample wanted, the first blocks take it.
template <bool SAMPLE>
__global__ void __launch_bounds__(256) mt_splits(MtArgs a, MtSplit *__restrict__ split, unsigned long long *ctr) {
    if (SAMPLE && blockIdx.x < MT_SAMPLE_BLOCKS) {
        if (a.A.nnz >= a.B.nnz) mt_sample(a.A, a.B, a.n_rows, ctr, a.words);
        else mt_sample(a.B, a.A, a.n_rows, ctr, a.words);
        return;
    }
    const uint64_t block = blockIdx.x - (SAMPLE ? MT_SAMPLE_BLOCKS : 0u);
    const uint64_t t = (block * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t > a.n_tiles) return;
    if (t == a.n_tiles) {
        if (lane == 0) split[t] = {a.n_rows, a.A.nnz, a.B.nnz, a.n_rows};
        return;
    }
    const uint64_t d = t * MT_TILE;  // < off_A[n] + off_B[n] + n
    // the last row whose first item is at or before d
    uint64_t lo = 0, hi = a.n_rows;
    while (hi - lo > 1) {
        const uint64_t step = (hi - lo + 31) / 32, r = lo + (uint64_t)(lane + 1) * step;
        const unsigned n = __popc(__ballot_sync(0xffffffffu, r < hi && a.A.off[r] + a.B.off[r] + r <= d));
        lo += n * step;
        hi = min(hi, lo + step);
    }
    const uint64_t row = lo, ab = a.A.off[row], bb = a.B.off[row];
    const uint64_t la = a.A.off[row + 1] - ab, lb = a.B.off[row + 1] - bb, k = d - (ab + bb + row);  // <= la + lb
    // A's share of the row's first k merged entries (A before B on equal
    // columns): A[i] is among them if it comes before B[k - 1 - i]
    uint64_t i0 = k > lb ? k - lb : 0, i1 = min(k, la);
    while (i0 < i1) {
        const uint64_t step = (i1 - i0 + 31) / 32, i = i0 + (uint64_t)lane * step;
        const unsigned n = __popc(__ballot_sync(0xffffffffu, i < i1 && a.A.cols[ab + i] <= a.B.cols[bb + k - 1 - i]));
        if (n == 0) break;
        i1 = min(i1, i0 + (uint64_t)n * step);  // the first probe that failed, or the end
        i0 += (uint64_t)(n - 1) * step + 1;
    }
    if (lane == 0) {
        uint64_t ia = ab + i0, ib = bb + k - i0;
        if (i0 > 0 && ib < bb + lb && a.A.cols[ia - 1] == a.B.cols[ib]) ++ib;  // the pair stays together
        split[t] = {row, ia, ib, row + (k == 0 ? 0 : 1)};
    }
}

// A spare slot after every MT_E: threads on their own MT_E neighbours hit
// distinct banks (unpadded, 56 M conflicts and an L1 pipe two thirds busy).
__device__ __forceinline__ int mt_pad(int k) { return k + k / MT_E; }
constexpr int MT_PADDED = MT_CAP + MT_CAP / MT_E;

struct MtSmem {
    double val[MT_PADDED];                 // A's entries, then (from the next whole thread on) B's
    __align__(16) uint32_t col[MT_CAP];
    __align__(16) uint16_t mark[MT_CAP];   // rows starting at each entry
    uint16_t ra[MT_CAP + 2], rb[MT_CAP + 2];  // the tile's rows' first entries on each side
    double oval[MT_PADDED];                // the kept entries in order, until the next tile is merged
    uint32_t ocol[MT_PADDED];
    uint32_t keep[MT_KW];
    uint16_t kpre[MT_KW];
    uint32_t wsum[MT_T / 32];
    uint32_t marks_a;
    BlockLookback<MT_T> lb;
    struct Tile {
        uint64_t id, r0, r1, a0, a1, b0, b1, rf, rl;  // rows and entries; rows [rf, rl) start in the tile
        uint32_t total;
    } tile[3];
};

__device__ __forceinline__ void mt_take(MtSmem::Tile &x, const MtArgs &a) {
    const uint64_t id = atomicAdd(a.ticket, 1ull);
    x.id = id;
    if (id < a.n_tiles) {
        const MtSplit s = a.split[id], e = a.split[id + 1];
        x.r0 = s.row;
        x.r1 = min(e.row, a.n_rows - 1);
        x.a0 = s.ia;
        x.a1 = e.ia;
        x.b0 = s.ib;
        x.b1 = e.ib;
        x.rf = s.rf;
        x.rl = e.rf;
    }
}

__device__ __forceinline__ void cp_async_4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

template <MergeMode MODE>
__global__ void __launch_bounds__(MT_T, MT_PER_SM) mt_tiles(MtArgs a) {
    extern __shared__ __align__(16) unsigned char mt_raw[];
    MtSmem &S = *reinterpret_cast<MtSmem *>(mt_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) mt_take(S.tile[0], a);
    __syncthreads();
    for (unsigned it = 0;; ++it) {
        auto &cur = S.tile[it % 3], &prev = S.tile[(it + 2) % 3];
        const bool have = cur.id < a.n_tiles;
        alignas(16) uint32_t c[MT_E];
        uint32_t o[MT_E], total = 0;
        double v[MT_E];
        if (have) {
            const uint64_t a0 = cur.a0, b0 = cur.b0, r0 = cur.r0;
            const int na = (int)(cur.a1 - a0), nb = (int)(cur.b1 - b0);
            const int nap = (na + MT_E - 1) / MT_E * MT_E;  // B's part starts at a whole thread
            for (int i = t; i < na; i += MT_T) {
                cp_async_4(&S.col[i], a.A.cols + a0 + i);
                cp_async_8(&S.val[mt_pad(i)], a.A.vals + a0 + i);
            }
            for (int i = t; i < nb; i += MT_T) {
                cp_async_4(&S.col[nap + i], a.B.cols + b0 + i);
                cp_async_8(&S.val[mt_pad(nap + i)], a.B.vals + b0 + i);
            }
#pragma unroll
            for (int j = 0; j < MT_E / 2; ++j) reinterpret_cast<uint32_t *>(S.mark)[t + j * MT_T] = 0;
            if (t < MT_KW) S.keep[t] = 0;
            __syncthreads();
            const int nr = (int)(cur.r1 - r0) + 1;  // rows with entries here are among these
            for (int k = t; k <= nr; k += MT_T) {
                const uint64_t pa = a.A.off[r0 + k], pb = a.B.off[r0 + k];
                const int sa = pa <= a0 ? 0 : (int)min(pa - a0, (uint64_t)na), sb = pb <= b0 ? 0 : (int)min(pb - b0, (uint64_t)nb);
                S.ra[k] = (uint16_t)sa;
                S.rb[k] = (uint16_t)sb;
                if (k > 0 && k < nr) {  // (16-bit counters in 32-bit words)
                    if (sa < na) atomicAdd(reinterpret_cast<uint32_t *>(S.mark) + (sa >> 1), 1u << (16 * (sa & 1)));
                    const int q = nap + sb;
                    if (sb < nb) atomicAdd(reinterpret_cast<uint32_t *>(S.mark) + (q >> 1), 1u << (16 * (q & 1)));
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // rows of the thread's MT_E entries: a scan over the marks
            uint32_t mw[MT_E / 2], sum = 0;
#pragma unroll
            for (int j = 0; j < MT_E / 2; ++j) mw[j] = reinterpret_cast<const uint32_t *>(S.mark)[t * (MT_E / 2) + j];
#pragma unroll
            for (int j = 0; j < MT_E / 2; ++j) sum += (mw[j] & 0xFFFFu) + (mw[j] >> 16);
            uint32_t inc = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += x;
            }
            if (lane == 31) S.wsum[warp] = inc;
            __syncthreads();
            uint32_t row = inc - sum + __reduce_add_sync(0xffffffffu, lane < warp ? S.wsum[lane & (MT_T / 32 - 1)] : 0u);
            if (MT_E * t == nap) S.marks_a = row;
            __syncthreads();
            const bool is_a = MT_E * t < nap;
            if (!is_a) row -= S.marks_a;
            const uint16_t *rs = is_a ? S.rb : S.ra;            // the other side's rows ...
            const uint32_t *oc = S.col + (is_a ? nap : 0);      // ... columns ...
            const int first = MT_E * t - (is_a ? 0 : nap), own = (is_a ? na : nb) - first;  // this thread's, and how many
            int j = 0, end = 0;
#pragma unroll
            for (int q = 0; q < MT_E; q += 4) *reinterpret_cast<uint4 *>(c + q) = *reinterpret_cast<const uint4 *>(S.col + MT_E * t + q);
            uint32_t at = 0xFFFFFFFFu;  // row j and end belong to
#pragma unroll
            for (int q = 0; q < MT_E; ++q) {
                o[q] = 0xFFFFFFFFu;
                if (q < own) {
                    row += (mw[q >> 1] >> (16 * (q & 1))) & 0xFFFFu;
                    v[q] = S.val[mt_pad(MT_E * t + q)];
                    if (row != at) {
                        at = row;
                        j = rs[row];
                        end = rs[row + 1];
                    }
                    // A: the first of B's at or after the column; B: of A's after it
                    int near = 0;
                    while (j < end && near < 4 && (oc[j] < c[q] || (!is_a && oc[j] == c[q]))) {
                        ++j;
                        ++near;
                    }
                    if (near == 4) {
                        int hi = end;
                        while (j < hi) {
                            const int mid = (j + hi) >> 1;
                            if (oc[mid] < c[q] || (!is_a && oc[mid] == c[q])) j = mid + 1;
                            else hi = mid;
                        }
                    }
                    bool kept;
                    if (is_a) {
                        const bool hit = j < end && oc[j] == c[q];
                        if constexpr (MODE == MergeMode::Sum) {
                            if (hit) v[q] = __dadd_rn(v[q], S.val[mt_pad(nap + j)]);
                            kept = !is_zero(v[q]);
                        } else {
                            if (hit) v[q] = S.val[mt_pad(nap + j)];
                            kept = !(hit && is_zero(v[q]));
                        }
                    } else {
                        kept = !(j > (int)rs[row] && oc[j - 1] == c[q]) && !is_zero(v[q]);
                    }
                    if (kept) {
                        o[q] = (uint32_t)(first + q + j);  // the merged place
                        atomicOr(&S.keep[o[q] >> 5], 1u << (o[q] & 31));
                    }
                }
            }
            __syncthreads();
            // kept entries before each word: every warp for itself, MT_KW / 32 words a lane
            uint32_t n3 = 0;
#pragma unroll
            for (int k = 0; k < MT_KW / 32; ++k) n3 += __popc(S.keep[lane * (MT_KW / 32) + k]);
            uint32_t pre = n3;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, pre, d);
                if (lane >= d) pre += x;
            }
            total = __shfl_sync(0xffffffffu, pre, 31);
            pre -= n3;
#pragma unroll
            for (int k = 0; k < MT_KW / 32; ++k) {
                S.kpre[lane * (MT_KW / 32) + k] = (uint16_t)pre;  // (the same from every warp)
                pre += __popc(S.keep[lane * (MT_KW / 32) + k]);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < MT_E; ++q)
                if (o[q] != 0xFFFFFFFFu) o[q] = S.kpre[o[q] >> 5] + __popc(S.keep[o[q] >> 5] & ((1u << (o[q] & 31)) - 1u));
            if (t == 0) {
                cur.total = total;
                atomicExch(a.state + cur.id, (cur.id == 0 ? 0ull + LB_PREFIX : 0ull + LB_AGG) | total);
            }
        }
        if (it > 0) {  // the tile before: its place is known by now
            uint64_t base = 0;
            if (!block_lookback<MT_T>(S.lb, a.state, prev.id, prev.total, base, a.status, MT_STATUS_TIMEOUT)) return;
            for (uint32_t k = base + prev.total <= a.room ? t : prev.total; k < prev.total; k += MT_T) {
                a.cols[base + k] = S.ocol[mt_pad(k)];
                a.vals[base + k] = S.oval[mt_pad(k)];
            }
            for (uint64_t r = prev.rf + t; r < prev.rl; r += MT_T) {
                const uint64_t p = a.off[r];  // within the tile: this thread's own
                a.off[r] = p + base;
            }
            if (t == 0 && prev.id + 1 == a.n_tiles) {
                a.off[a.n_rows] = base + prev.total;
                store_word(a.words, 0, base + prev.total);
            }
        }
        if (!have) return;
        if (t == 32) mt_take(S.tile[(it + 1) % 3], a);
        __syncthreads();  // the tile before is written
#pragma unroll
        for (int q = 0; q < MT_E; ++q) {
            if (o[q] != 0xFFFFFFFFu) {
                S.ocol[mt_pad(o[q])] = c[q];
                S.oval[mt_pad(o[q])] = v[q];
            }
        }
        for (uint64_t r = cur.rf + t; r < cur.rl; r += MT_T) {
            const uint32_t p = (uint32_t)(a.A.off[r] - cur.a0 + a.B.off[r] - cur.b0);  // merged place of its start
            a.off[r] = S.kpre[p >> 5] + __popc(S.keep[p >> 5] & ((1u << (p & 31)) - 1u));
        }
        __syncthreads();
    }
}

// The tiles, into arrays with room for `room` entries; the state words are zero.
int mt_run(Ctx *c, MtArgs &a, MergeMode mode, uint32_t *cols, double *vals, uint64_t room, uint64_t *nnz, cudaStream_t s) {
    a.cols = cols;
    a.vals = vals;
    a.room = room;
    auto k = mode == MergeMode::Sum ? mt_tiles<MergeMode::Sum> : mt_tiles<MergeMode::Replace>;
    SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MtSmem)));
    k<<<(unsigned)std::min<uint64_t>(a.n_tiles, (uint64_t)c->n_sms * MT_PER_SM), MT_T, sizeof(MtSmem), s>>>(a);
    SPG_LAUNCH_CHECK();
    SPG_TRY(c->phase_sync(s));
    *nnz = c->word(0);
    return SPG_OK;
}

// The cuts and everything else that the tiles need but C's arrays, and the
// sample in words 0 and 1.
int mt_prepare(Ctx *c, const CsrView &A, const CsrView &B, uint64_t n_rows, uint64_t *off_out, bool sample,
               DevBuf &split, DevBuf &state, MtArgs &a, cudaStream_t s) {
    const uint64_t items = A.nnz + B.nnz + n_rows, tiles = (items + MT_TILE - 1) / MT_TILE;
    SPG_TRY(split.alloc((tiles + 1) * sizeof(MtSplit), s));
    SPG_TRY(state.alloc((tiles + 3) * sizeof(unsigned long long), s));  // ticket, tiles, the sample's counters
    SPG_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, (tiles + 3) * sizeof(unsigned long long), s));
    a.A = A;
    a.B = B;
    a.n_rows = n_rows;
    a.n_tiles = tiles;
    a.split = split.as<MtSplit>();
    a.ticket = state.as<unsigned long long>();
    a.state = a.ticket + 1;
    a.off = off_out;
    a.status = c->d_status;
    a.words = c->d_words;
    const unsigned blocks = (unsigned)((tiles + 1 + 7) / 8);
    if (sample) {
        c->h_words[1] = 0;
        mt_splits<true><<<MT_SAMPLE_BLOCKS + blocks, 256, 0, s>>>(a, split.as<MtSplit>(), a.state + tiles);
    } else {
        mt_splits<false><<<blocks, 256, 0, s>>>(a, split.as<MtSplit>(), nullptr);
    }
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

}  // namespace

int merge_csr(Ctx *c, const CsrView &A, const CsrView &B, uint64_t n_rows, MergeMode mode, uint64_t *off_out,
              uint32_t *cols_out, double *vals_out, uint64_t *nnz, cudaStream_t s) {
    *nnz = 0;
    if (n_rows == 0) {
        SPG_CUDA_TRY(cudaMemsetAsync(off_out, 0, sizeof(uint64_t), s));
        return SPG_OK;
    }
    DevBuf split, state;
    MtArgs a{};
    SPG_TRY(mt_prepare(c, A, B, n_rows, off_out, false, split, state, a, s));
    return mt_run(c, a, mode, cols_out, vals_out, ~0ull, nnz, s);
}

int sum_csr(Ctx *c, const CsrView &A, const CsrView &B, uint64_t n_rows, uint64_t *off_out, DevBuf &cols, DevBuf &vals,
            uint64_t *nnz, cudaStream_t s) {
    const uint64_t both = A.nnz + B.nnz;
    uint64_t room = both;
    auto alloc = [&]() -> int {
        SPG_TRY(vals.alloc(csr_alloc_elems(room) * sizeof(double), s));  // (the larger one first, for the pool)
        return cols.alloc(csr_alloc_elems(room) * sizeof(uint32_t), s);
    };
    // The pairs of equal columns, which a sum has once, in a sample of the larger
    // side, with a sixteenth to spare (four deviations of the sample): the cuts'
    // kernel takes it in its first blocks, and the host reads it while the cuts
    // are made. Arrays for all entries held up to twice what is needed, and moving
    // the entries afterwards is a copy of C (1 M Zipf rows plus 1 %: 60 us of 410).
    const bool sample = n_rows && both > RESULT_BOUND && std::max(A.nnz, B.nnz) >= MT_SAMPLES;
    DevBuf split, state;
    MtArgs a{};
    if (n_rows) SPG_TRY(mt_prepare(c, A, B, n_rows, off_out, sample, split, state, a, s));
    if (sample) {
        SPG_TRY(c->wait_word(1, s));
        const double hits = (double)c->word(0) / MT_SAMPLES;
        const uint64_t pairs = std::min((uint64_t)(hits * (double)std::max(A.nnz, B.nnz)), std::min(A.nnz, B.nnz));
        room = std::min(both, both - pairs + both / 16);
    }
    SPG_TRY(alloc());
    if (n_rows == 0) {
        *nnz = 0;
        SPG_CUDA_TRY(cudaMemsetAsync(off_out, 0, sizeof(uint64_t), s));
        return SPG_OK;
    }
    SPG_TRY(mt_run(c, a, MergeMode::Sum, cols.as<uint32_t>(), vals.as<double>(), room, nnz, s));
    if (*nnz > room) {  // the sample was wrong: again, with what is needed
        room = *nnz;
        SPG_TRY(alloc());
        SPG_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, (a.n_tiles + 1) * sizeof(unsigned long long), s));
        SPG_TRY(mt_run(c, a, MergeMode::Sum, cols.as<uint32_t>(), vals.as<double>(), room, nnz, s));
    }
    return both > RESULT_BOUND ? fit_arrays(c, *nnz, room, cols, vals, s) : SPG_OK;
}

}  // namespace spg
