// spg_delta.cu — a later lock whose delta is small against the matrix
// (csr_build.hpp:126-488: the buffer wins on equal columns, a zero deletes):
// the work beside copying the matrix is done per insert, not per row or entry.
//
// The inserts come with their rows non-decreasing. Each of them
//   1. ranks itself among its row's inserts by (column, order), which tells
//      whether it is the last write of its key (a row has a few of them; more
//      than SD_RUN go the general way, spg_rowtiles.cu and spg_merge.cu);
//   2. searches its place in the row of the old CSR: place[p], the first old
//      entry at or after it, and whether that is its key (hit);
//   3. contributes +1 (new), -1 (deletes) or 0; P, the scan of the
//      contributions in sorted order, is how far everything after it moves.
// Old entry e then goes to e + P[j], j the first insert placed after it, and
// is left out if the insert before that hits it; row r starts at
// off[r] + P[first insert of a row >= r]; an insert's own entry goes to
// place + P. A block copies SD_CHUNK old entries: with no insert among them,
// as most, all by the same distance.
//
// Bound: the copy, 24 bytes per old entry. The general merge finds the place
// of every entry of both sides (110 us for 10 M entries and 100 k inserts,
// where a copy takes 36).
#include <algorithm>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int SD_T = 256;
constexpr int SD_RUN = 64;             // inserts of one row that rank themselves
constexpr int SD_E = 16, SD_CHUNK = SD_T * SD_E;  // old entries per block
constexpr int SD_NEAR = 1024;          // inserts of a chunk staged in shared memory
constexpr int SD_ROWS = SD_T * 8;      // rows per block
constexpr uint32_t SD_HIT = 1u, SD_LAST = 2u;

struct SdArgs {
    CsrView A;
    uint64_t n_rows;
    const uint32_t *rows, *cols;
    const double *vals;
    uint64_t m;
    const unsigned long long *abort;
    unsigned long long *words;  // for the host: ctr[0], ctr[1], entries gained (signed)
    unsigned long long *ctr;   // [0] distinct keys, [1] 1: a row has more than SD_RUN inserts
    uint64_t *place;           // by sorted position, as the next four
    int64_t *P;                // contributions, then their exclusive scan (m + 1)
    uint32_t *row, *col, *flag;
    double *val;
    uint64_t *chunk, *rchunk;  // first insert placed in each chunk or after, first of each row block or after
    uint64_t n_chunks, n_rchunks;
    uint64_t *off;
    uint32_t *out_cols;
    double *out_vals;
};

__device__ __forceinline__ bool sd_off(const SdArgs &a) { return a.ctr[1] != 0 || (a.abort && *a.abort != 0); }

__global__ void __launch_bounds__(SD_T) sd_probe(SdArgs a) {
    if (a.abort && *a.abort) return;
    const uint64_t i = blockIdx.x * (uint64_t)SD_T + threadIdx.x;
    // More than SD_RUN inserts of a row ahead or behind, here or in a block
    // before: the attempt ends. (An epoch in no order shows only now, sorted,
    // how many inserts its rows get: 900 k in 3000 rows of 1 M, thrown away
    // after 64 steps of every insert 456 us, at once 371.)
    const uint32_t r = i < a.m ? a.rows[i] : 0;
    const bool over = i < a.m && ((i >= (uint64_t)SD_RUN && a.rows[i - SD_RUN] == r) ||
                                  (i + SD_RUN < a.m && a.rows[i + SD_RUN] == r));
    if (__syncthreads_or(over || (threadIdx.x == 0 && a.ctr[1]))) {
        if (threadIdx.x == 0) a.ctr[1] = 1ull;
        return;
    }
    bool last = false;
    if (i < a.m) {
        const uint32_t c = a.cols[i];
        uint64_t p = i;  // sorted position
        last = true;
        for (int k = 1; k < SD_RUN; ++k) {  // the row's inserts before this one
            if (i < (uint64_t)k || a.rows[i - k] != r) break;
            if (a.cols[i - k] > c) --p;
        }
        for (int k = 1; k < SD_RUN; ++k) {  // and after it
            if (i + k >= a.m || a.rows[i + k] != r) break;
            const uint32_t o = a.cols[i + k];
            if (o < c) ++p;
            last = last && o != c;
        }
        const double v = a.vals[i];
        const uint64_t rb = a.A.off[r], re = a.A.off[r + 1];
        uint64_t lo = rb, hi = re;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (a.A.cols[mid] < c) lo = mid + 1;
            else hi = mid;
        }
        const bool hit = last && lo < re && a.A.cols[lo] == c, zero = is_zero(v);
        a.place[p] = lo;
        a.row[p] = r;
        a.col[p] = c;
        a.val[p] = v;
        a.flag[p] = (hit ? SD_HIT : 0u) | (last ? SD_LAST : 0u);
        a.P[p] = !last ? 0 : hit ? (zero ? -1 : 0) : (zero ? 0 : 1);
    }
    const unsigned n = __popc(__ballot_sync(0xffffffffu, last));
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(a.ctr, (unsigned long long)n);
}

// First of x[0..m) that is >= key.
template <class T>
__device__ __forceinline__ uint64_t sd_lower(const T *__restrict__ x, uint64_t lo, uint64_t hi, uint64_t key) {
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (x[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(SD_T) sd_chunks(SdArgs a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // final since the probe and the scan
        store_word(a.words, 0, a.ctr[0]);
        store_word(a.words, 1, a.ctr[1]);
        store_word(a.words, 2, (unsigned long long)a.P[a.m]);
    }
    if (sd_off(a)) return;
    const uint64_t k = blockIdx.x * (uint64_t)SD_T + threadIdx.x;
    if (k <= a.n_chunks) a.chunk[k] = sd_lower(a.place, 0, a.m, k * SD_CHUNK);
    const uint64_t q = k - (a.n_chunks + 1);
    if (k > a.n_chunks && q <= a.n_rchunks) a.rchunk[q] = sd_lower(a.row, 0, a.m, q * SD_ROWS);
}

// Blocks [0, n_chunks): old entries; then n_rchunks: row offsets; then the inserts.
__global__ void __launch_bounds__(SD_T) sd_merge(SdArgs a) {
    __shared__ uint32_t s_place[SD_NEAR];  // within the chunk
    __shared__ int32_t s_move[SD_NEAR + 1];  // relative to the chunk's first
    __shared__ uint8_t s_hit[SD_NEAR];
    if (sd_off(a)) return;
    const int t = threadIdx.x;
    uint64_t b = blockIdx.x;
    if (b < a.n_chunks) {
        const uint64_t e0 = b * SD_CHUNK, j0 = a.chunk[b];
        uint64_t j1 = a.chunk[b + 1];
        const int n = (int)min((uint64_t)SD_CHUNK, a.A.nnz - e0);
        const int64_t first = a.P[j0];
        // The inserts of the chunk are those placed in [e0, e0 + n). (One placed
        // at the end of all, at nnz, moves nothing.)
        const uint64_t nj = j1 - j0;
        const bool near = nj <= (uint64_t)SD_NEAR;
        if (nj && near) {
            for (int k = t; k <= (int)nj; k += SD_T) {
                s_move[k] = (int32_t)(a.P[j0 + k] - first);
                if (k < (int)nj) {
                    s_place[k] = (uint32_t)(a.place[j0 + k] - e0);
                    s_hit[k] = (uint8_t)(a.flag[j0 + k] & SD_HIT);
                }
            }
            __syncthreads();
        }
        for (int h = 0; h < SD_E; h += 8) {  // eight entries' loads in flight
            uint32_t c[8];
            double v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = t + (h + i) * SD_T;
                if (e < n) {
                    c[i] = a.A.cols[e0 + e];
                    v[i] = a.A.vals[e0 + e];
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = t + (h + i) * SD_T;
                if (e >= n) continue;
                int64_t move = first;
                if (nj) {
                    bool hit;
                    if (near) {
                        int lo = 0, hi = (int)nj;  // the first insert placed after e
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if (s_place[mid] <= (uint32_t)e) lo = mid + 1;
                            else hi = mid;
                        }
                        hit = lo > 0 && s_hit[lo - 1] && s_place[lo - 1] == (uint32_t)e;
                        move += s_move[lo];
                    } else {
                        const uint64_t j = sd_lower(a.place, j0, j1, e0 + e + 1);
                        hit = j > j0 && (a.flag[j - 1] & SD_HIT) && a.place[j - 1] == e0 + e;
                        move = a.P[j];
                    }
                    if (hit) continue;  // replaced or deleted
                }
                const uint64_t o = (uint64_t)((int64_t)(e0 + e) + move);
                a.out_cols[o] = c[i];
                a.out_vals[o] = v[i];
            }
        }
        return;
    }
    b -= a.n_chunks;
    if (b < a.n_rchunks) {
        const uint64_t j0 = a.rchunk[b], j1 = a.rchunk[b + 1];
#pragma unroll
        for (int i = 0; i < SD_ROWS / SD_T; ++i) {
            const uint64_t r = b * SD_ROWS + t + i * SD_T;
            if (r > a.n_rows) break;
            a.off[r] = (uint64_t)((int64_t)a.A.off[r] + a.P[j0 == j1 ? j0 : sd_lower(a.row, j0, j1, r)]);
        }
        return;
    }
    b -= a.n_rchunks;
    const uint64_t p = b * SD_T + t;
    if (p < a.m && (a.flag[p] & SD_LAST) && !is_zero(a.val[p])) {
        const uint64_t o = (uint64_t)((int64_t)a.place[p] + a.P[p]);
        a.out_cols[o] = a.col[p];
        a.out_vals[o] = a.val[p];
    }
}

}  // namespace

int merge_small_delta(Ctx *c, const CsrView &A, uint64_t n_rows, const uint32_t *rows, const uint32_t *cols,
                      const double *vals, uint64_t m, const unsigned long long *abort, uint64_t *off_out,
                      uint32_t *cols_out, double *vals_out, uint64_t *nnz, uint64_t *u, bool *done, cudaStream_t s) {
    *done = false;
    SdArgs a{};
    a.n_chunks = (A.nnz + SD_CHUNK - 1) / SD_CHUNK;
    a.n_rchunks = (n_rows + 1 + SD_ROWS - 1) / SD_ROWS;
    // one buffer: 8-byte arrays, then 4-byte ones
    DevBuf work;
    const uint64_t words = 2 + m + (m + 1) + m + (a.n_chunks + 1) + (a.n_rchunks + 1);
    SPG_TRY(work.alloc(words * 8 + 3 * m * 4, s));
    SPG_CUDA_TRY(cudaMemsetAsync(work.ptr, 0, 16, s));
    a.ctr = work.as<unsigned long long>();
    a.place = reinterpret_cast<uint64_t *>(a.ctr + 2);
    a.P = reinterpret_cast<int64_t *>(a.place + m);
    a.val = reinterpret_cast<double *>(a.P + m + 1);
    a.chunk = reinterpret_cast<uint64_t *>(a.val + m);
    a.rchunk = a.chunk + a.n_chunks + 1;
    a.row = reinterpret_cast<uint32_t *>(a.rchunk + a.n_rchunks + 1);
    a.col = a.row + m;
    a.flag = a.col + m;
    a.A = A;
    a.n_rows = n_rows;
    a.rows = rows;
    a.cols = cols;
    a.vals = vals;
    a.m = m;
    a.abort = abort;
    a.words = c->d_words;
    a.off = off_out;
    a.out_cols = cols_out;
    a.out_vals = vals_out;
    SPG_CUDA_TRY(cudaMemsetAsync(a.P + m, 0, sizeof(int64_t), s));
    const unsigned gm = (unsigned)((m + SD_T - 1) / SD_T);
    sd_probe<<<gm, SD_T, 0, s>>>(a);
    SPG_LAUNCH_CHECK();
    SPG_TRY(exclusive_scan_i64(c, a.P, m + 1, s));
    sd_chunks<<<(unsigned)((a.n_chunks + a.n_rchunks + 2 + SD_T - 1) / SD_T), SD_T, 0, s>>>(a);
    SPG_LAUNCH_CHECK();
    sd_merge<<<(unsigned)(a.n_chunks + a.n_rchunks + gm), SD_T, 0, s>>>(a);
    SPG_LAUNCH_CHECK();
    SPG_TRY(c->phase_sync(s));
    *u = c->word(0);
    *nnz = (uint64_t)((int64_t)A.nnz + (int64_t)c->word(2));
    *done = c->word(1) == 0;
    return SPG_OK;
}

}  // namespace spg
