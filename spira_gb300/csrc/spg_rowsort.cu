// spg_rowsort.cu — staged inserts put in row order: a stable LSD radix sort of
// (row, column, value) by the row's bits, so that every row's inserts keep the
// order they were staged in (the last write of a column is still the last).
// What follows treats them as row-grouped inserts.
//
// One pass per digit of at most 8 bits, one launch per pass: the digits'
// global counts of all passes are taken beforehand in one read of the rows,
// and a tile learns how many of each digit the tiles before it hold by a
// look-back over their published counts (thread d for digit d, RS_LOOK words
// at a time; tiles in ticket order, every wait bounded). Inside a tile the
// digits are ranked with ballots per warp, and the entries are copied straight
// to their digit-ordered places in shared memory (cp.async), from where every
// digit's run goes out on consecutive addresses.
//
// Bound: 32 bytes per entry and pass of HBM traffic, half of the time taken (a
// pass over 10 M entries: 101 us, 47 at the copy rate); the rest is latency
// between the barriers of three blocks an SM. 116 us before the columns and
// values were prefetched into the L2 during the ranking and the digit's bits
// were a constant of the code. Sorting only the row bits
// and leaving each row to the row kernels takes 3 passes for 2 M rows where
// the (row, column) keys took 6, of three launches each and with an index that
// fetched every value at random afterwards.
#include <algorithm>
#include <vector>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int RS_T = 256, RS_RADIX = 256, RS_LOOK = 8;
constexpr int RS_MAX_PASSES = 4;
constexpr int RS_LT = 512, RS_LI = 6, RS_LB = 3;  // large sorts: threads, entries per thread, blocks per SM
constexpr uint64_t RS_LARGE_PER_SM = 2048;
constexpr unsigned RS_STATUS_TIMEOUT = 0x80u;

// Digit counts of every pass (hist[p * RS_RADIX + d]).
__global__ void __launch_bounds__(RS_T) rs_hist(const uint32_t *__restrict__ rows, uint64_t m, int passes, int bits,
                                                unsigned long long *__restrict__ hist) {
    __shared__ uint32_t s_h[RS_MAX_PASSES][RS_RADIX];
    for (int i = threadIdx.x; i < RS_MAX_PASSES * RS_RADIX; i += RS_T) (&s_h[0][0])[i] = 0;
    __syncthreads();
    const uint32_t mask = (1u << bits) - 1u;
    const uint64_t stride = (uint64_t)gridDim.x * RS_T;
    const uint64_t n_iter = (m + 4 * stride - 1) / (4 * stride);  // the same for every thread: votes below
    for (uint64_t it = 0; it < n_iter; ++it) {
        const uint64_t i0 = 4 * it * stride + blockIdx.x * (uint64_t)RS_T + threadIdx.x;
        uint32_t r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) r[u] = i0 + u * stride < m ? rows[i0 + u * stride] : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // one add for a whole warp of one row (runs of a row would serialise)
            const bool in = i0 + u * stride < m;
            const uint32_t r0 = __shfl_sync(0xffffffffu, r[u], 0);
            const bool one = __all_sync(0xffffffffu, in && r[u] == r0);
            if (in && (!one || (threadIdx.x & 31) == 0)) {
                for (int p = 0; p < passes; ++p) atomicAdd(&s_h[p][(r[u] >> (p * bits)) & mask], one ? 32u : 1u);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * RS_RADIX; i += RS_T) {
        const uint32_t n = (&s_h[0][0])[i];
        if (n) atomicAdd(hist + i, (unsigned long long)n);
    }
}

template <int T, int I>
struct RsSmem {
    double val[T * I];
    uint32_t row[T * I], col[T * I];
    uint16_t cnt[T / 32][RS_RADIX];  // per-warp digit counts, then per-warp offsets
    uint32_t loc[RS_RADIX];          // the tile's first place of each digit
    uint64_t gbase[RS_RADIX];        // where that goes, less the place
    uint32_t wsum[RS_RADIX / 32];
    uint64_t wsum64[RS_RADIX / 32];
    uint64_t tile;
};

// TEST: waits end after wait_cycles (the limit is a constant otherwise: 1 % of a pass).
template <int T, int I, int PER_SM, int BITS, bool TEST = false>
__global__ void __launch_bounds__(T, PER_SM)
rs_pass(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ cols, const double *__restrict__ vals,
        uint64_t m, int shift, const unsigned long long *__restrict__ hist,
        unsigned long long *__restrict__ ticket, unsigned long long *__restrict__ state,
        uint32_t *__restrict__ out_rows, uint32_t *__restrict__ out_cols, double *__restrict__ out_vals,
        unsigned int *__restrict__ status, unsigned long long *__restrict__ abort, long long wait_cycles) {
    constexpr int TILE = T * I, W = T / 32;
    static_assert(T >= RS_RADIX && T % 32 == 0, "a thread per digit");
    extern __shared__ __align__(16) unsigned char rs_raw[];
    auto &S = *reinterpret_cast<RsSmem<T, I> *>(rs_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // An earlier pass, or a block of this one, may have given up. The flag can
    // change while the block's threads read it: what thread 0 saw counts for
    // all. (Thread 0 alone reading it cost 3 % of a pass.)
    const bool stop = *abort;
    if (t == 0 && !stop) S.tile = atomicAdd(ticket, 1ull);
    for (int i = t; i < W * RS_RADIX / 2; i += T) reinterpret_cast<uint32_t *>(&S.cnt[0][0])[i] = 0;
    if (__syncthreads_or(t == 0 && stop)) return;
    const uint64_t tile = S.tile, t0 = tile * TILE;
    const int n = (int)min((uint64_t)TILE, m - t0);
    // the columns and values are wanted once the ranks are known: into the L2 meanwhile
    for (int i = t * 32; i < n; i += T * 32) prefetch_l2(cols + t0 + i);
    for (int i = t * 16; i < n; i += T * 16) prefetch_l2(vals + t0 + i);
    constexpr uint32_t mask = (1u << BITS) - 1u;
    // warp w owns entries [w 32 I, (w + 1) 32 I) of the tile and walks them in order
    const int base = warp * (I * 32) + lane;
    uint32_t r[I], rank[I];
#pragma unroll
    for (int j = 0; j < I; ++j) r[j] = base + j * 32 < n ? rows[t0 + base + j * 32] : 0u;
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < I; ++j) {
        const bool ok = base + j * 32 < n;
        const unsigned valid = __ballot_sync(0xffffffffu, ok);
        rank[j] = 0;
        if (!valid) continue;
        const uint32_t d = (r[j] >> shift) & mask;
        unsigned peers = valid;
#pragma unroll
        for (int b = 0; b < BITS; ++b) {
            const unsigned bit = (d >> b) & 1u, bal = __ballot_sync(0xffffffffu, bit);
            peers &= bit ? bal : ~bal;
        }
        uint32_t before = 0;
        if (ok) before = S.cnt[warp][d];
        __syncwarp();
        rank[j] = before + __popc(peers & lt);
        if (ok && (peers & lt) == 0) S.cnt[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // digit t: exclusive prefix over the warps, its tile count published, and
    // exclusive scans over the digits of the tile's and the global counts
    const bool digit = t < max(32, 1 << BITS);  // whole warps
    uint32_t tot = 0, place = 0;
    uint64_t gplace = 0;
    unsigned long long *mine = state + tile * RS_RADIX + t;
    if (digit) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t x = S.cnt[w][t];
            S.cnt[w][t] = (uint16_t)tot;
            tot += x;
        }
        atomicExch(mine, (tile == 0 ? 0ull + LB_PREFIX : 0ull + LB_AGG) | tot);
        const uint64_t g = hist[t];
        uint32_t inc = tot;
        uint64_t ginc = g;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
            const uint64_t gx = __shfl_up_sync(0xffffffffu, ginc, o);
            if (lane >= o) {
                inc += x;
                ginc += gx;
            }
        }
        if (lane == 31) {
            S.wsum[warp] = inc;
            S.wsum64[warp] = ginc;
        }
        place = inc - tot;
        gplace = ginc - g;
    }
    __syncthreads();
    if (digit) {
        for (int w = 0; w < warp; ++w) {
            place += S.wsum[w];
            gplace += S.wsum64[w];
        }
        S.loc[t] = place;
    }
    __syncthreads();
    // the entries to their places in the tile
#pragma unroll
    for (int j = 0; j < I; ++j) {
        if (base + j * 32 < n) {
            const uint32_t d = (r[j] >> shift) & mask, p = S.loc[d] + S.cnt[warp][d] + rank[j];
            const uint64_t k = t0 + base + j * 32;
            S.row[p] = r[j];
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(&S.col[p])),
                         "l"(cols + k));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(&S.val[p])),
                         "l"(vals + k));
        }
    }
    // entries of digit t in the tiles before: RS_LOOK published words at a time
    uint64_t excl = 0;
    bool fail = false;
    if (tile > 0 && digit) {
        const long long c0 = clock64();
        int64_t q = (int64_t)tile - 1;
        bool done = false;
        while (!done && !fail) {
            unsigned long long w[RS_LOOK];
#pragma unroll
            for (int j = 0; j < RS_LOOK; ++j)
                w[j] = q - j >= 0 ? *(volatile unsigned long long *)(state + (q - j) * RS_RADIX + t) : 0ull;
            bool wait = false;
            int used = 0;
#pragma unroll
            for (int j = 0; j < RS_LOOK; ++j) {
                if (!done && !fail && !wait) {
                    const unsigned long long st = w[j] & ~LB_VALUE;
                    if (st == 0) wait = true;  // (tile 0 publishes a prefix: the walk ends there)
                    else if (st == LB_POISON) fail = true;
                    else {
                        excl += w[j] & LB_VALUE;
                        ++used;
                        done = st == LB_PREFIX;
                    }
                }
            }
            q -= used;
            if (wait && clock64() - c0 > (TEST ? wait_cycles : LB_WAIT_CYCLES)) {
                atomicOr(status, RS_STATUS_TIMEOUT);
                *(volatile unsigned long long *)abort = 1ull;
                fail = true;
            }
        }
        atomicExch(mine, fail ? 0ull + LB_POISON : LB_PREFIX | (excl + tot));
    }
    if (digit) S.gbase[t] = gplace + excl - place;
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (__syncthreads_or(fail)) return;  // (the status word fails the call)
    for (int i = t; i < n; i += T) {
        const uint32_t row = S.row[i];
        const uint64_t pos = S.gbase[(row >> shift) & mask] + i;
        out_rows[pos] = row;
        out_cols[pos] = S.col[i];
        out_vals[pos] = S.val[i];
    }
}

template <int T, int I, int PER_SM, int BITS>
int rs_launch(const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m, int shift,
              const unsigned long long *hist, unsigned long long *ticket, unsigned long long *state, uint32_t *orows,
              uint32_t *ocols, double *ovals, unsigned int *status, unsigned long long *abort, cudaStream_t s) {
    auto k = rs_pass<T, I, PER_SM, BITS>;
    constexpr size_t smem = sizeof(RsSmem<T, I>);
    SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t tiles = (m + T * I - 1) / (T * I);
    k<<<(unsigned)tiles, T, smem, s>>>(rows, cols, vals, m, shift, hist, ticket, state, orows, ocols, ovals,
                                       status, abort, LB_WAIT_CYCLES);
    SPG_LAUNCH_CHECK();
    return SPG_OK;
}

using RsLaunch = decltype(&rs_launch<RS_LT, RS_LI, RS_LB, 8>);

template <int T, int I, int PER_SM>
RsLaunch rs_launch_of(int bits) {
    switch (bits) {
        case 5: return rs_launch<T, I, PER_SM, 5>;
        case 6: return rs_launch<T, I, PER_SM, 6>;
        case 7: return rs_launch<T, I, PER_SM, 7>;
        default: return rs_launch<T, I, PER_SM, 8>;
    }
}

}  // namespace

int sort_staged_rows(Ctx *c, const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m, int rbits,
                     StagedSorted &out, cudaStream_t s, const unsigned long long *earlier) {
    const int passes = std::max(1, (rbits + 7) / 8), bits = std::max(5, (rbits + passes - 1) / passes);
    // tiles of RS_LT x RS_LI entries; of 1024 while the larger ones are fewer than
    // two for three SMs (first lock in random order into 1 M rows, large / small:
    // 100 k inserts 153.5 / 152.6 us, 400 k 166 / 173, 1.4 M 220 / 257)
    const bool large = m >= (uint64_t)c->n_sms * RS_LARGE_PER_SM;
    const uint64_t tile = large ? RS_LT * RS_LI : 256 * 4, tiles = (m + tile - 1) / tile;
    DevBuf work, rows2, cols2, vals2;
    const uint64_t words = passes * (RS_RADIX + 1 + tiles * RS_RADIX);
    SPG_TRY(work.alloc(words * sizeof(unsigned long long), s));
    SPG_CUDA_TRY(cudaMemsetAsync(work.ptr, 0, words * sizeof(unsigned long long), s));
    unsigned long long *hist = work.as<unsigned long long>(), *ticket = hist + passes * RS_RADIX,
                       *state = ticket + passes;
    SPG_TRY(out.abort.alloc(sizeof(unsigned long long), s));
    if (earlier) SPG_CUDA_TRY(cudaMemcpyAsync(out.abort.ptr, earlier, sizeof(*earlier), cudaMemcpyDeviceToDevice, s));
    else SPG_CUDA_TRY(cudaMemsetAsync(out.abort.ptr, 0, sizeof(unsigned long long), s));
    SPG_TRY(out.rows.alloc(m * sizeof(uint32_t), s));
    SPG_TRY(out.cols.alloc(csr_alloc_elems(m) * sizeof(uint32_t), s));  // (a CSR's arrays, for the transpose)
    SPG_TRY(out.vals.alloc(csr_alloc_elems(m) * sizeof(double), s));
    if (passes > 1) {
        SPG_TRY(rows2.alloc(m * sizeof(uint32_t), s));
        SPG_TRY(cols2.alloc(m * sizeof(uint32_t), s));
        SPG_TRY(vals2.alloc(m * sizeof(double), s));
    }
    rs_hist<<<grid_for(m, RS_T * 16, (unsigned)c->n_sms * 4), RS_T, 0, s>>>(rows, m, passes, bits, hist);
    SPG_LAUNCH_CHECK();
    const RsLaunch launch = large ? rs_launch_of<RS_LT, RS_LI, RS_LB>(bits) : rs_launch_of<256, 4, 6>(bits);
    const uint32_t *ir = rows, *ic = cols;
    const double *iv = vals;
    for (int p = 0; p < passes; ++p) {
        const bool to_out = (passes - 1 - p) % 2 == 0;  // the last pass ends in the outputs
        uint32_t *orr = (to_out ? out.rows : rows2).as<uint32_t>(), *oc = (to_out ? out.cols : cols2).as<uint32_t>();
        double *ov = (to_out ? out.vals : vals2).as<double>();
        SPG_TRY(launch(ir, ic, iv, m, p * bits, hist + p * RS_RADIX, ticket + p, state + p * tiles * RS_RADIX, orr,
                       oc, ov, c->d_status, out.abort.as<unsigned long long>(), s));
        ir = orr;
        ic = oc;
        iv = ov;
    }
    return SPG_OK;
}

// A pass whose first tile nobody takes: every tile waits for it, gives up after
// wait_cycles and stops the rest, of this pass and of the next one, before
// anything is written. Half of the blocks start when the others have given up.
int rowsort_wait_selftest(Ctx *c, long long wait_cycles, bool *gave_up, cudaStream_t s) {
    constexpr int T = 256, I = 4, PER_SM = 6;
    const uint64_t tiles = 1 + 2 * PER_SM * (uint64_t)c->n_sms, m = tiles * T * I;
    const uint64_t words = RS_RADIX + 3 + 2 * tiles * RS_RADIX;  // digit counts, two tickets, the flag, two passes' states
    DevBuf work, rows, vals, orows, ocols, ovals;
    SPG_TRY(work.alloc(words * sizeof(unsigned long long), s));
    SPG_TRY(rows.alloc(m * sizeof(uint32_t), s));  // (the columns too)
    SPG_TRY(vals.alloc(m * sizeof(double), s));
    SPG_TRY(orows.alloc(m * sizeof(uint32_t), s));
    SPG_TRY(ocols.alloc(m * sizeof(uint32_t), s));
    SPG_TRY(ovals.alloc(m * sizeof(double), s));
    SPG_CUDA_TRY(cudaMemsetAsync(work.ptr, 0, words * sizeof(unsigned long long), s));
    SPG_CUDA_TRY(cudaMemsetAsync(rows.ptr, 0, m * sizeof(uint32_t), s));
    SPG_CUDA_TRY(cudaMemsetAsync(vals.ptr, 0, m * sizeof(double), s));
    SPG_CUDA_TRY(cudaMemsetAsync(orows.ptr, 0xFF, m * sizeof(uint32_t), s));
    unsigned long long *hist = work.as<unsigned long long>(), *ticket = hist + RS_RADIX, *abort = ticket + 2,
                       *state = abort + 1;
    SPG_CUDA_TRY(cudaMemsetAsync(ticket, 1, 1, s));  // the first pass's tickets start at 1
    auto k = rs_pass<T, I, PER_SM, 8, true>;
    constexpr size_t smem = sizeof(RsSmem<T, I>);
    SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (uint64_t p = 0; p < 2; ++p) {
        k<<<(unsigned)(tiles - 1 + p), T, smem, s>>>(rows.as<uint32_t>(), rows.as<uint32_t>(), vals.as<double>(), m, 0,
                                                    hist, ticket + p, state + p * tiles * RS_RADIX,
                                                    orows.as<uint32_t>(), ocols.as<uint32_t>(), ovals.as<double>(),
                                                    c->d_status, abort, wait_cycles);
        SPG_LAUNCH_CHECK();
    }
    std::vector<unsigned long long> w(words);
    std::vector<uint32_t> o(m);
    SPG_CUDA_TRY(cudaMemcpyAsync(w.data(), work.ptr, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    SPG_CUDA_TRY(cudaMemcpyAsync(o.data(), orows.ptr, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    SPG_CUDA_TRY(cudaStreamSynchronize(s));
    const unsigned long long *wt = w.data() + RS_RADIX, *ws = wt + 3;
    bool ok = (*(volatile unsigned *)c->h_status & RS_STATUS_TIMEOUT) && wt[2] == 1 && wt[1] == 0;
    for (uint64_t i = 0; i < RS_RADIX; ++i) ok = ok && ws[i] == 0 && ws[RS_RADIX + i] == LB_POISON;  // tiles 0 and 1
    for (uint64_t i = wt[0] * RS_RADIX; i < 2 * tiles * RS_RADIX; ++i) ok = ok && ws[i] == 0;  // tiles nobody took
    for (uint32_t x : o) ok = ok && x == 0xFFFFFFFFu;
    *gave_up = ok;
    return SPG_OK;
}

}  // namespace spg
