// spg_transpose.cu — A^T as a stable counting sort by column.
//
// Spira (serial/transpose.hpp:35-156) histograms the column indices, prefix-
// sums them into the output offsets and scatters row by row through per-
// column cursors, so every output row lists its source rows in ascending
// order; the result is installed with load_csr (capacity == nnz).
//
// Here the same histogram (device atomics) and prefix sum give the output
// offsets. When no output row has more than 32 entries (and no source row,
// which a thread walks alone, more than 256), a scatter runs in
// parallel through atomic per-column cursors, so inside an output row the
// source rows arrive in any order, and each output row is then put in
// source-row order by a sorting network (in one thread's registers, or across
// a warp's lanes); source rows are distinct within a column, so the result is
// unique: Spira's. Otherwise the entries are sorted
// stably by column (spg_rowsort.cu), which keeps the source rows ascending at
// any length. Integer work and value copies only: bit-exact.
#include <algorithm>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int TB = 256;
constexpr unsigned LOOK_SAMPLES = 1024;  // a block
constexpr uint64_t LOOK_FEW = 1u << 20;

// rowid[k] = source row of entry k (eight lanes per row).
__global__ void tr_expand(const uint64_t *__restrict__ off, uint64_t n_rows, uint32_t *__restrict__ rowid) {
    const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 3;
    if (w >= n_rows) return;
    const uint64_t e = off[w + 1];
    for (uint64_t k = off[w] + (threadIdx.x & 7); k < e; k += 8) rowid[k] = (uint32_t)w;
}

__global__ void tr_count(const uint32_t *__restrict__ cols, uint64_t nnz, unsigned long long *__restrict__ cnt) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < nnz; k += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(cnt + cols[k], 1ull);
}

// Whether the source rows repeat each other's pattern: of a row's entry and the
// one in the same place of the next row, in LOOK_SAMPLES rows, words[0] = how
// often the column is the same or one more, words[1] = the samples taken.
__global__ void __launch_bounds__(LOOK_SAMPLES)
tr_sample(const uint64_t *__restrict__ off, const uint32_t *__restrict__ cols, uint64_t m,
          unsigned long long *__restrict__ words) {
    const uint64_t k = threadIdx.x, r = k * (m - 1) / LOOK_SAMPLES;
    const uint64_t b = off[r], e = off[r + 1], f = off[r + 2];
    bool same = false;
    if (e > b) {
        const uint64_t j = k % (e - b);
        same = j < f - e && cols[e + j] - cols[b + j] <= 1u;
    }
    const int hits = __syncthreads_count(same), taken = __syncthreads_count(e > b);
    if (threadIdx.x == 0) {
        store_word(words, 0, (unsigned long long)hits);
        store_word(words, 1, (unsigned long long)taken);
    }
}

// Thread per source row: entry (w, c) goes to toff[c] + (a cursor of column
// c). A row's entries are handled SB at a time with their loads and cursor
// atomics all issued before any result is used (the atomics' round trips
// overlap instead of queueing one after another).
constexpr int SB = 8;

// The sorting-network path runs before the host has seen the longest output
// row: its kernels take the device-side longest row and do nothing when it
// is above 32 (the stable sort by column then runs instead).
constexpr unsigned long long NET_MAX = 32;

__global__ void tr_scatter(const uint64_t *__restrict__ off, const uint32_t *__restrict__ cols,
                           const double *__restrict__ vals, uint64_t m, const uint64_t *__restrict__ toff,
                           unsigned *__restrict__ cursor, uint32_t *__restrict__ tsrc,
                           double *__restrict__ tval, const unsigned long long *__restrict__ longest) {
    const uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (w >= m) return;
    if (*longest > NET_MAX) return;
    const uint64_t e = off[w + 1];
    for (uint64_t k = off[w]; k < e; k += SB) {
        uint32_t col[SB];
        double v[SB];
        uint64_t base[SB];
        unsigned slot[SB];
#pragma unroll
        for (int j = 0; j < SB; ++j) {
            col[j] = k + j < e ? cols[k + j] : 0u;
            v[j] = k + j < e ? vals[k + j] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < SB; ++j)
            if (k + j < e) {
                slot[j] = atomicAdd(cursor + col[j], 1u);
                base[j] = toff[col[j]];
            }
#pragma unroll
        for (int j = 0; j < SB; ++j)
            if (k + j < e) {
                const uint64_t p = base[j] + slot[j];
                tsrc[p] = (uint32_t)w;
                tval[p] = v[j];
            }
    }
}

// Longest output row (for the choice of sort), from the scanned offsets; above
// NET_MAX too if a source row has more than SRC_MAX entries, which a thread of
// the scatter walks alone (a Zipf matrix of 200 k rows: 3.8 ms, 0.27 sorted).
constexpr uint64_t SRC_MAX = 256;

__global__ void tr_max_len(const uint64_t *__restrict__ toff, uint64_t n, const uint64_t *__restrict__ off, uint64_t m,
                           unsigned long long *__restrict__ mx) {
    unsigned long long v = 0;
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < m; r += (uint64_t)gridDim.x * blockDim.x)
        if (off[r + 1] - off[r] > SRC_MAX) v = NET_MAX + 1;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x)
        v = max(v, (unsigned long long)(toff[c + 1] - toff[c]));
#pragma unroll
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ unsigned long long s_v[TB / 32];
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < TB / 32; ++w) v = max(v, s_v[w]);
        atomicMax(mx, v);
    }
}

// Per output row, the scattered entries (source row, value) put in source-row
// order directly when the row is short: rows of at most 16 entries by one
// thread with a bitonic network in registers (source rows are distinct in a
// column, so the order is unique and the network's instability does not
// matter) and rows of 17..32 entries listed for tr_sort_mid. Used when no
// output row is longer than 32.
template <int N>
__device__ __forceinline__ void bitonic_regs(uint32_t (&k)[N], double (&v)[N]) {
#pragma unroll
    for (int size = 2; size <= N; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    if ((k[i] > k[j]) == up) {
                        const uint32_t tk = k[i];
                        k[i] = k[j];
                        k[j] = tk;
                        const double tv = v[i];
                        v[i] = v[j];
                        v[j] = tv;
                    }
                }
            }
}

template <int N>
__device__ __forceinline__ void sort_row_regs(const uint32_t *__restrict__ tsrc, const double *__restrict__ tval,
                                              uint64_t b, uint32_t L, uint32_t *__restrict__ out_cols,
                                              double *__restrict__ out_vals) {
    uint32_t k[N];
    double v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        k[i] = (uint32_t)i < L ? tsrc[b + i] : 0xFFFFFFFFu;
        v[i] = (uint32_t)i < L ? tval[b + i] : 0.0;
    }
    bitonic_regs<N>(k, v);
#pragma unroll
    for (int i = 0; i < N; ++i)
        if ((uint32_t)i < L) {
            out_cols[b + i] = k[i];
            out_vals[b + i] = v[i];
        }
}

__global__ void __launch_bounds__(TB)
tr_sort_short(const uint64_t *__restrict__ toff, uint64_t n, const uint32_t *__restrict__ tsrc,
              const double *__restrict__ tval, uint32_t *__restrict__ out_cols, double *__restrict__ out_vals,
              unsigned long long *__restrict__ n_mid, uint32_t *__restrict__ mid,
              const unsigned long long *__restrict__ longest) {
    if (*longest > NET_MAX) return;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = toff[c];
        const uint64_t L = toff[c + 1] - b;
        if (L <= 1) {
            if (L == 1) {
                out_cols[b] = tsrc[b];
                out_vals[b] = tval[b];
            }
        } else if (L <= 8) {
            sort_row_regs<8>(tsrc, tval, b, (uint32_t)L, out_cols, out_vals);
        } else if (L <= 16) {
            sort_row_regs<16>(tsrc, tval, b, (uint32_t)L, out_cols, out_vals);
        } else {  // 17..32 (longer rows never reach this kernel)
            mid[atomicAdd(n_mid, 1ull)] = (uint32_t)c;
        }
    }
}

// Rows of 17..32 entries: a warp per row, one entry per lane, bitonic sort
// across the lanes by source row.
__global__ void __launch_bounds__(TB)
tr_sort_mid(const uint64_t *__restrict__ toff, const uint32_t *__restrict__ mid,
            const unsigned long long *__restrict__ n_mid, const uint32_t *__restrict__ tsrc,
            const double *__restrict__ tval, uint32_t *__restrict__ out_cols, double *__restrict__ out_vals,
            const unsigned long long *__restrict__ longest, unsigned long long *__restrict__ words) {
    if (blockIdx.x == 0 && threadIdx.x == 0) store_word(words, 0, *longest);
    if (*longest > NET_MAX) return;
    const unsigned lane = threadIdx.x & 31;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t cnt = *n_mid;
    for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w < cnt; w += n_warps) {
        const uint32_t c = mid[w];
        const uint64_t b = toff[c], L = toff[c + 1] - b;
        uint32_t k = lane < L ? tsrc[b + lane] : 0xFFFFFFFFu;
        double v = lane < L ? tval[b + lane] : 0.0;
#pragma unroll
        for (unsigned size = 2; size <= 32; size <<= 1)
#pragma unroll
            for (unsigned stride = size >> 1; stride > 0; stride >>= 1) {
                const uint32_t pk = __shfl_xor_sync(0xffffffffu, k, stride);
                const double pv = __shfl_xor_sync(0xffffffffu, v, stride);
                const bool up = (lane & size) == 0, lower = (lane & stride) == 0;
                // the lower lane of an ascending pair keeps the smaller key
                const bool keep_small = lower == up;
                const bool take = keep_small ? (pk < k) : (pk > k);
                if (take) {
                    k = pk;
                    v = pv;
                }
            }
        if (lane < L) {
            out_cols[b + lane] = k;
            out_vals[b + lane] = v;
        }
    }
}

}  // namespace

int transpose_impl(Ctx *c, const Csr *A, Csr *T, cudaStream_t s) {
    const uint64_t nnz = A->nnz, m = A->n_rows, n = A->n_cols;
    if (nnz >= (1ull << 32))
        return set_error(SPG_ERR_UNSUPPORTED, "transpose: nnz %llu exceeds 2^32-1", (unsigned long long)nnz);
    const unsigned gmax = (unsigned)c->n_sms * 32;
    DevBuf out_off, out_cols, out_vals;
    SPG_TRY(out_off.alloc(csr_off_elems(n) * sizeof(uint64_t), s));
    unsigned long long longest = NET_MAX + 1;
    // Whether the networks may do: source rows below their padding key, and not
    // above 32 entries a column on average. From 16 on it depends on whether the
    // columns are alike: 27 to every column are the networks' case (looked at
    // first / column sort at once: 300 k columns 344 / 363 us, 500 k 514 / 538, 1 M
    // 961 / 1020), random ones have some column above 32, and the look is lost
    // (500k x 200k with 20 to a column 267 / 219, 500k x 500k with 24 568 / 502).
    // A sample of the rows tells, for 10 us: rows that repeat their predecessor's
    // columns, in place or moved by one, as stencils, bands and blocks do. Such
    // matrices are square, so others are not sampled, nor are those of up to 1 M
    // entries, where the column sort is as fast for both (20 k columns of 28: 77 us
    // a band, 79 random ones; looked at 85).
    bool look = nnz && m < 0xFFFFFFFFull && nnz <= NET_MAX * n;
    if (look && nnz > 16 * n) {
        look = false;
        if (m == n && nnz > LOOK_FEW) {
            tr_sample<<<1, LOOK_SAMPLES, 0, s>>>(A->d_off(), A->d_cols(), m, c->d_words);
            SPG_LAUNCH_CHECK();
            SPG_TRY(c->phase_sync(s));
            look = 4 * c->word(0) >= 3 * c->word(1);
        }
    }
    if (look || nnz == 0) SPG_CUDA_TRY(cudaMemsetAsync(out_off.ptr, 0, csr_off_elems(n) * sizeof(uint64_t), s));
    if (look) {
        tr_count<<<grid_for(nnz, TB, gmax), TB, 0, s>>>(A->d_cols(), nnz,
                                                       reinterpret_cast<unsigned long long *>(out_off.ptr));
        SPG_LAUNCH_CHECK();
        SPG_TRY(exclusive_scan_u64(c, out_off.as<uint64_t>(), n + 1, nullptr, s));
        // The longest output row decides: up to 32 entries, an atomic scatter
        // and sorting networks per row. That path is enqueued at once, its
        // kernels checking the longest row on the device, so the common case
        // costs no host round trip before the final one. Where both apply the
        // networks are faster (3D Laplacian 100^3 221 us, 368 by the column sort;
        // 200k x 200k with 12 a row 150 / 170; 1 M with 6 309 / 326).
        DevBuf meta, midbuf, tsrc, tval;
        SPG_TRY(out_cols.alloc(csr_alloc_elems(nnz) * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(csr_alloc_elems(nnz) * sizeof(double), s));
        // [longest row (8 bytes)] [rows of 17..32 entries (8 bytes)] [cursors]
        SPG_TRY(meta.alloc(16 + n * sizeof(unsigned), s));
        SPG_CUDA_TRY(cudaMemsetAsync(meta.ptr, 0, 16 + n * sizeof(unsigned), s));
        unsigned long long *mx = meta.as<unsigned long long>(), *n_mid = mx + 1;
        unsigned *cur = reinterpret_cast<unsigned *>(mx + 2);
        tr_max_len<<<grid_for(std::max(n, m), TB, (unsigned)c->n_sms * 8), TB, 0, s>>>(out_off.as<uint64_t>(), n, A->d_off(),
                                                                         m, mx);
        SPG_LAUNCH_CHECK();
        SPG_TRY(tsrc.alloc(nnz * sizeof(uint32_t), s));
        SPG_TRY(tval.alloc(nnz * sizeof(double), s));
        SPG_TRY(midbuf.alloc(n * sizeof(uint32_t), s));
        tr_scatter<<<grid_for(m, TB), TB, 0, s>>>(A->d_off(), A->d_cols(), A->d_vals(), m, out_off.as<uint64_t>(),
                                                  cur, tsrc.as<uint32_t>(), tval.as<double>(), mx);
        tr_sort_short<<<grid_for(n, TB, gmax), TB, 0, s>>>(out_off.as<uint64_t>(), n, tsrc.as<uint32_t>(),
                                                           tval.as<double>(), out_cols.as<uint32_t>(),
                                                           out_vals.as<double>(), n_mid, midbuf.as<uint32_t>(),
                                                           mx);
        tr_sort_mid<<<(unsigned)c->n_sms * 8, TB, 0, s>>>(out_off.as<uint64_t>(), midbuf.as<uint32_t>(), n_mid,
                                                         tsrc.as<uint32_t>(), tval.as<double>(),
                                                         out_cols.as<uint32_t>(), out_vals.as<double>(), mx, c->d_words);
        SPG_LAUNCH_CHECK();
        SPG_TRY(c->phase_sync(s));
        longest = c->word(0);
    }
    if (nnz && longest > NET_MAX) {
        // (column, source row, value) sorted stably by column: the rows of a
        // column stay in ascending order, whatever its length
        StagedSorted o;
        DevBuf rowid;
        SPG_TRY(rowid.alloc(nnz * sizeof(uint32_t), s));
        tr_expand<<<grid_for(m * 8, TB), TB, 0, s>>>(A->d_off(), m, rowid.as<uint32_t>());
        SPG_LAUNCH_CHECK();
        SPG_TRY(sort_staged_rows(c, A->d_cols(), rowid.as<uint32_t>(), A->d_vals(), nnz, bits_for(n), o, s));
        if (!look) SPG_TRY(launch_row_offsets(c, o.rows.as<uint32_t>(), nnz, n, out_off.as<uint64_t>(), s));
        out_cols = std::move(o.cols);
        out_vals = std::move(o.vals);
        SPG_TRY(c->phase_sync(s));
    } else if (nnz == 0) {
        SPG_TRY(out_cols.alloc(csr_alloc_elems(0) * sizeof(uint32_t), s));
        SPG_TRY(out_vals.alloc(csr_alloc_elems(0) * sizeof(double), s));
        SPG_TRY(c->phase_sync(s));
    }
    T->invalidate_derived();
    T->n_rows = n;
    T->n_cols = m;
    T->off = std::move(out_off);
    T->cols = std::move(out_cols);
    T->vals = std::move(out_vals);
    T->nnz = nnz;
    T->capacity = nnz;
    T->built = true;
    T->may_have_zeros = A->may_have_zeros;
    return SPG_OK;
}

}  // namespace spg

using namespace spg;

extern "C" int spg_transpose(spg_ctx *c, const spg_csr *A, spg_csr *T) {
    if (!c || !A || !T) return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_transpose: null handle");
    SPG_CHECK_LIVE(A);
    SPG_CHECK_LIVE(T);
    if (!A->built) return set_error(SPG_ERR_LOGIC, "transpose: matrix must be locked");
    if (A == T) return set_error(SPG_ERR_INVALID_ARGUMENT, "spg_transpose: output aliases input");
    SPG_CUDA_TRY(cudaSetDevice(c->device));
    return transpose_impl(c, A, T, c->stream);
}
