// spg_internal.cuh — shared internals of libspg.so: handles, error plumbing,
// device buffers and the device-wide primitives (scan, radix sort) that the
// lock / transpose / SpGEMM kernels are built from.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <string>
#include <utility>
#include <atomic>
#include <vector>

#include "../../include/spg.h"

namespace spg {

// ---------------------------------------------------------------------------
// Errors. Every C entry point returns a status; the detail text goes to a
// thread-local string read back by spg_last_error().
// ---------------------------------------------------------------------------
int set_error(int code, const char *fmt, ...);
void clear_error();

struct Status {
    int code = SPG_OK;
    bool ok() const { return code == SPG_OK; }
};

#define SPG_CUDA_TRY(expr)                                                          \
    do {                                                                            \
        cudaError_t _e = (expr);                                                    \
        if (_e != cudaSuccess) {                                                    \
            if (_e == cudaErrorMemoryAllocation) {                                  \
                cudaGetLastError();                                                 \
                return ::spg::set_error(SPG_ERR_NO_MEMORY, "%s: %s (%s:%d)", #expr, \
                                        cudaGetErrorString(_e), __FILE__, __LINE__); \
            }                                                                       \
            return ::spg::set_error(SPG_ERR_CUDA, "%s: %s (%s:%d)", #expr,          \
                                    cudaGetErrorString(_e), __FILE__, __LINE__);    \
        }                                                                           \
    } while (0)

#define SPG_TRY(expr)                      \
    do {                                   \
        int _s = (expr);                   \
        if (_s != SPG_OK) return _s;       \
    } while (0)

#define SPG_LAUNCH_CHECK() SPG_CUDA_TRY(cudaPeekAtLastError())

// ---------------------------------------------------------------------------
// Handles
// ---------------------------------------------------------------------------
struct Ctx;

// Stream-ordered device buffer from the context's memory pool.
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaStream_t stream = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept { *this = std::move(o); }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            ptr = o.ptr; bytes = o.bytes; stream = o.stream;
            o.ptr = nullptr; o.bytes = 0;
        }
        return *this;
    }
    ~DevBuf() { release(); }
    int alloc(size_t n, cudaStream_t s);
    void release();
    template <class T> T *as() const { return static_cast<T *>(ptr); }
};

// Cached SpMV plan (row blocks for the stream / merge variants).
struct SpmvPlan {
    int kind = -1;           // variant the plan belongs to
    uint64_t n_items = 0;    // number of work items (blocks / tiles / chunks)
    uint64_t count1 = 0;     // variant-specific count
    DevBuf items;            // variant-specific item descriptors
    DevBuf aux;              // variant-specific scratch (carry-outs)
    DevBuf extra0, extra1, extra2;
    DevBuf extra3, extra4;
    // Host-side block split for the pipelined host SpMV (adaptive variants):
    // host_rows[b] = first row of block b, host_rows[host_nb] = n_rows.
    int host_nb = 0;
    std::vector<uint64_t> host_rows;
};

struct Csr;
struct Batch;
void batch_orphan(Batch *b);  // spg_batch.cu

struct Ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;
    // Live handles created on this context. Destroying the context releases
    // their device memory and orphans them; an orphaned handle can still be
    // destroyed, every other call on it returns SPG_ERR_LOGIC.
    std::vector<Csr *> live_csrs;
    std::vector<Batch *> live_batches;
    int n_sms = 0;
    size_t l2_bytes = 0;
    // Status word written by kernels whose bounded waits ran out; 0 = ok.
    // Mapped pinned memory: h_status is the host view, d_status the device one.
    unsigned int *h_status = nullptr;
    unsigned int *d_status = nullptr;
    // Results of an operation's kernels (counts, flags), in the same mapped
    // memory: the last block or tile stores them there and the host reads them
    // once the stream is synchronised. Copying a word back instead costs 5 us
    // per synchronisation (14.3 against 9.4 us for launch, word and wait). A
    // context runs one operation at a time, and its kernels store all the words
    // that it reads.
    static constexpr int N_WORDS = 16;
    unsigned long long *h_words = nullptr;
    unsigned long long *d_words = nullptr;
    uint64_t word(int k) const { return *(volatile unsigned long long *)(h_words + k); }
    // Waits for a word that was set to 0 before the launch and that a running
    // kernel stores (store_word_now), or for the stream if that is sooner.
    int wait_word(int k, cudaStream_t s);
    // Returns SPG_ERR_DEVICE_TIMEOUT (and clears the word) if a kernel flagged
    // one since the last check; call after a stream synchronisation.
    int take_status() {
        const unsigned v = h_status ? *(volatile unsigned *)h_status : 0u;
        if (!v) return SPG_OK;
        *(volatile unsigned *)h_status = 0;
        return set_error(SPG_ERR_DEVICE_TIMEOUT, "a device-side wait gave up (status 0x%x)", v);
    }
    // Pinned host staging for the *_host entry points.
    void *pinned = nullptr;
    size_t pinned_bytes = 0;
    int ensure_pinned(size_t bytes);
    // Device vectors reused by spg_spmv_host, the stream that copies y back
    // while later row blocks compute, and the events between the two.
    DevBuf xbuf, ybuf;
    cudaStream_t copy_stream = nullptr, upload_stream = nullptr;
    static constexpr int N_HOST_EVENTS = 8;
    cudaEvent_t host_events[N_HOST_EVENTS] = {};
    cudaEvent_t upload_events[N_HOST_EVENTS] = {};
    // Host SpMVs of several matrices in one call (spg_host_multi.cu): per
    // matrix lane a compute, an upload and a download stream and events,
    // created at first use; the recorded graph and what it was recorded for.
    static constexpr int MULTI_MAX = 4;
    cudaStream_t multi_stream[MULTI_MAX][3] = {};
    cudaEvent_t multi_event[MULTI_MAX][2 * N_HOST_EVENTS] = {};
    cudaGraphExec_t multi_graph = nullptr;
    std::vector<uintptr_t> multi_key;
    void drop_multi() {
        if (multi_graph) cudaGraphExecDestroy(multi_graph);
        multi_graph = nullptr;
        multi_key.clear();
    }
    // SpMV variant choice: policy and the loaded selector (spg_tune.cu).
    int spmv_policy = SPG_POLICY_SELECTOR;
    DevBuf model;  // FP32 selector blob
    int model_k = 0;
    // The same for SpGEMM.
    int spgemm_policy = SPG_POLICY_SELECTOR;
    DevBuf gemm_model;
    int gemm_model_k = 0;
    // Device-time accounting of operations that synchronise internally
    // (spg_ctx_timer_start / _stop): each stretch of work on the context
    // stream between two host synchronisations is one phase, timed by an
    // event pair; the host round trips between phases are not counted.
    bool timer_on = false;
    double timer_ms = 0.0;
    cudaEvent_t timer_ev[2] = {nullptr, nullptr};
    // Waits for `s` (the operations' synchronisation point); closes and opens
    // a timed phase when the timer runs on this stream.
    int phase_sync(cudaStream_t s);
};

struct Csr {
    Ctx *ctx = nullptr;
    uint64_t n_rows = 0, n_cols = 0;
    uint64_t nnz = 0, capacity = 0;
    bool built = false;
    // True when load_csr installed explicit +-0.0 values (only load_csr can:
    // lock and SpGEMM never store zeros). The merge then drops them from the
    // rows it touches, as csr_build.hpp:274-301 does.
    bool may_have_zeros = false;
    DevBuf off;   // uint64_t[n_rows + 1]
    DevBuf cols;  // uint32_t[capacity]
    DevBuf vals;  // double[capacity]
    // The longest row, computed lazily by csr_max_row.
    bool stats_valid = false;
    uint64_t max_row = 0;
    int selected_spmv = -1;
    // SpGEMM variant chosen for this matrix times gemm_sel_b (at its epoch).
    int gemm_selected = -1;
    const Csr *gemm_sel_b = nullptr;
    uint64_t gemm_sel_b_epoch = 0;
    SpmvPlan plan_stream, plan_merge, plan_adaptive, plan_inter;
    // For the host-buffer SpMV of row-parallel variants: the largest column
    // each of host_reach.size() equal row blocks reads (-1: empty block), so a
    // block can start once the part of x up to that column has arrived.
    std::vector<int64_t> host_reach;
    // The pipelined host SpMV recorded as a CUDA graph for one pinned (x, y)
    // pair and variant, replayed while the same pair comes back.
    cudaGraphExec_t host_graph = nullptr;
    const double *host_gx = nullptr;  // the pair, the variant and the device staging it was recorded with
    double *host_gy = nullptr;
    const void *host_gdx = nullptr, *host_gdy = nullptr;
    int host_gvariant = -1;
    // Device staging of x and y for host-buffer SpMVs from pinned memory (the
    // matrix's own, so SpMVs of different matrices can be in flight at once).
    DevBuf stage_x, stage_y;
    void drop_host_graph() {
        if (host_graph) cudaGraphExecDestroy(host_graph);
        host_graph = nullptr;
        host_gx = nullptr;
        host_gy = nullptr;
        host_gdx = host_gdy = nullptr;
        host_gvariant = -1;
    }
    ~Csr() { drop_host_graph(); }
    // Renewed whenever the CSR changes, unique across all matrices of the
    // process (keys graphs recorded over the matrix).
    uint64_t epoch = 0;
    static uint64_t next_epoch() {
        static std::atomic<uint64_t> counter{0};
        return ++counter;
    }
    void invalidate_derived() {
        epoch = next_epoch();
        stats_valid = false;
        selected_spmv = -1;
        gemm_selected = -1;
        gemm_sel_b = nullptr;
        plan_stream = SpmvPlan{};
        plan_merge = SpmvPlan{};
        plan_adaptive = SpmvPlan{};
        plan_inter = SpmvPlan{};
        host_reach.clear();
        drop_host_graph();
    }
    const uint64_t *d_off() const { return off.as<uint64_t>(); }
    const uint32_t *d_cols() const { return cols.as<uint32_t>(); }
    const double *d_vals() const { return vals.as<double>(); }
    // Frees the device arrays while the owning context's stream still exists.
    void orphan() {
        invalidate_derived();
        off.release();
        cols.release();
        vals.release();
        stage_x.release();  // every device buffer goes while the context's stream exists
        stage_y.release();
        built = false;
        nnz = capacity = 0;
        ctx = nullptr;
    }
};

// Checks that a handle still belongs to a live context.
#define SPG_CHECK_LIVE(A)                                                                              \
    do {                                                                                               \
        if ((A)->ctx == nullptr)                                                                       \
            return ::spg::set_error(SPG_ERR_LOGIC, "the matrix's context was destroyed");             \
    } while (0)

inline cudaStream_t pick_stream(Ctx *c, void *s) {
    return s ? static_cast<cudaStream_t>(s) : c->stream;
}

inline int bits_for(uint64_t n) {  // bits needed to represent 0..n-1
    int b = 0;
    while (b < 64 && (n - 1) >> b) ++b;
    return n <= 1 ? 0 : b;
}

// Elements to allocate for CSR cols/vals of a given capacity: rounded up to a
// multiple of 16 plus 16 more, so kernels that read whole 16-aligned chunks of
// 16 entries (SPG_SPMV_ADAPTIVE) never touch memory past the allocation.
inline uint64_t csr_alloc_elems(uint64_t cap) { return ((cap + 15) & ~15ull) + 16; }
// Entries to allocate for CSR offsets of n rows: n + 1 plus 2 spare, so a
// 16-byte bulk copy of offsets [r0 & ~1, r1 + 1] rounded to an even count
// stays inside the allocation.
inline uint64_t csr_off_elems(uint64_t n_rows) { return n_rows + 3; }

// Ascending bitonic sort of the 32 * E keys a warp holds, key[e] of lane l
// being element 32 e + l. Partners 32 or more apart share a lane (registers),
// nearer ones are exchanged by shuffles.
// k0 > 2 (warp-uniform) skips the stages below k0: the caller guarantees
// that every block of k0 / 2 network positions is already sorted, ascending
// where (position & k0 / 2) == 0 and descending elsewhere.
template <int E, class K>
__device__ __forceinline__ void warp_bitonic(K (&key)[E], int lane, int k0 = 2) {
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
        if (k < k0) continue;
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int jj = j >> 5;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if ((e & jj) == 0) {
                        const int f = e | jj;
                        const bool up = ((32 * e) & k) == 0;  // k >= 64: the item decides
                        const K a = key[e], b = key[f];
                        const bool sw = up ? (a > b) : (a < b);
                        key[e] = sw ? b : a;
                        key[f] = sw ? a : b;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const K o = __shfl_xor_sync(0xffffffffu, key[e], j);
                    const int i = 32 * e + lane;
                    const bool keep_min = (((i & k) == 0) == ((i & j) == 0));
                    key[e] = keep_min ? (o < key[e] ? o : key[e]) : (o > key[e] ? o : key[e]);
                }
            }
        }
    }
}

// Spira's ValueTraits<double>::is_zero (traits.hpp:73-80): +0 and -0 are
// zero, NaN is not; also exactly Spira's SpGEMM drop test `v != V{}`
// (spgemm.hpp:44) negated. Tested on the bit pattern (every bit but the sign
// clear): integer ALU work instead of an FP64 compare, which costs as much
// FP64 pipe time as a multiply on GB300. The words are taken apart in assembly:
// written as (bits << 1) == 0, the compiler turns the test back into the FP64
// compare (the FP64 pipe of kernels without any arithmetic was 8-22 % busy).
__device__ __forceinline__ bool is_zero(double v) {
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
    return (lo | (hi << 1)) == 0;
}

// Brings p's line into the L2 (no fault, no wait).
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// One thread of every block calls it once the block's results are in global
// memory (atomics or plain stores of that thread): true in the last block of
// the grid, which then sees them all. *done starts at zero.
template <class Count>
__device__ __forceinline__ bool last_block(Count *done) {
    __threadfence();
    if (atomicAdd(done, (Count)1) != (Count)gridDim.x - 1) return false;
    __threadfence();
    return true;
}

__device__ __forceinline__ void store_word(unsigned long long *words, int k, unsigned long long v) {
    *(volatile unsigned long long *)(words + k) = v;
}

// words[0 .. N) from N counters that other blocks added to: all are read before
// the first is stored (one after another, each store waits for its read).
template <int N, class T>
__device__ __forceinline__ void store_counters(unsigned long long *words, const T *ctr) {
    T v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = *(const volatile T *)(ctr + k);
#pragma unroll
    for (int k = 0; k < N; ++k) store_word(words, k, v[k]);
}

// store_word for a host that reads the word while the kernel runs (Ctx::wait_word),
// after what the thread stored before.
__device__ __forceinline__ void store_word_now(unsigned long long *words, int k, unsigned long long v) {
    __threadfence_system();
    store_word(words, k, v);
    __threadfence_system();
}

// Lanes of the (full) warp whose NB-bit value d (a radix digit, or 256 for
// "no key" when NB = 9) equals this lane's: NB ballots on the ALU pipe,
// cheaper on GB300 than match.any, which issues on the narrow
// address-divergence unit.
template <int NB = 9>
__device__ __forceinline__ unsigned warp_match_digit(unsigned d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const unsigned bit = (d >> b) & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Ordered scan of tile counts inside one launch (decoupled look-back): a
// word per tile, zeroed before the launch. Tiles are taken in launch order by
// tickets, so a tile only waits for tiles whose blocks already run; every
// wait is bounded, and a tile that gives up poisons its own word, so later
// tiles stop too.
constexpr unsigned long long LB_AGG = 1ull << 62;      // tile published its own count
constexpr unsigned long long LB_PREFIX = 2ull << 62;   // tile published its inclusive prefix
constexpr unsigned long long LB_POISON = 3ull << 62;   // tile gave up: everything after stops
constexpr unsigned long long LB_VALUE = (1ull << 62) - 1;
constexpr long long LB_WAIT_CYCLES = 1ll << 31;        // ~1 s at 2 GHz

// By one (full) warp: lane l reads the word of tile p - l, so each step covers
// 32 predecessors. (Reading 8 words per lane, 256 per step, measured slower:
// 0.73 against 0.43 ms on the 200k x 8 SpGEMM with 2048-product tiles.)
// Returns false if the tile had to give up (timeout, or an earlier tile gave
// up); on a timeout `status_bit` is set in *status. Lane 0 publishes.
__device__ __forceinline__ bool lookback_scan(unsigned long long *tstate, uint64_t t, uint64_t total, uint64_t *base,
                                              int lane, unsigned int *status, unsigned status_bit,
                                              long long wait_cycles) {
    if (t == 0) {
        if (lane == 0) atomicExch(tstate, LB_PREFIX | total);
        *base = 0;
        return true;
    }
    if (lane == 0) atomicExch(tstate + t, LB_AGG | total);
    uint64_t excl = 0;
    int64_t p = (int64_t)t - 1;  // nearest predecessor of the window
    const long long t0 = clock64();
    while (true) {
        const int64_t q = p - lane;
        const unsigned long long v = q >= 0 ? *(volatile unsigned long long *)(tstate + q) : 0ull;
        const unsigned long long st = v & ~LB_VALUE;
        const unsigned pref = __ballot_sync(0xffffffffu, q >= 0 && st == LB_PREFIX);
        // lanes up to the nearest prefix (tile 0 always publishes one, so a
        // window reaching q < 0 holds it at a lower lane)
        const unsigned need = pref ? (pref & (0u - pref)) * 2u - 1u : 0xffffffffu;
        const unsigned waiting = __ballot_sync(0xffffffffu, q >= 0 && st == 0) & need;
        const unsigned poison = __ballot_sync(0xffffffffu, q >= 0 && st == LB_POISON) & need;
        if (poison) {
            if (lane == 0) atomicExch(tstate + t, LB_POISON);
            return false;
        }
        if (waiting) {
            if (clock64() - t0 > wait_cycles) {
                if (lane == 0) {
                    atomicOr(status, status_bit);
                    atomicExch(tstate + t, LB_POISON);
                }
                return false;
            }
            __nanosleep(32);
            continue;
        }
        unsigned long long add = ((need >> lane) & 1u) ? (v & LB_VALUE) : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        excl += add;
        if (pref) break;
        p -= 32;
    }
    if (lane == 0) atomicExch(tstate + t, LB_PREFIX | (excl + total));
    *base = excl;
    return true;
}

// The same by a whole block of T threads, for a tile whose count is already
// published (its own word holds LB_AGG | total, or LB_PREFIX | total for tile
// 0): thread t reads the word of tile id - 1 - t, so a window covers T tiles,
// about what is in flight, and the nearest published prefix is mostly found in
// one step of one L2 round trip (one warp's windows of 32 took 14 of them in
// the row-tile kernel). Publishes the inclusive prefix. All threads call;
// false in every thread if the tile had to give up.
template <int T>
struct BlockLookback {
    uint64_t sum[T / 32];
    uint32_t state[T / 32];
};

template <int T>
__device__ __forceinline__ bool block_lookback(BlockLookback<T> &S, unsigned long long *tstate, uint64_t id,
                                               uint64_t total, uint64_t &base, unsigned int *status,
                                               unsigned status_bit, long long wait_cycles = LB_WAIT_CYCLES) {
    constexpr int W = T / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    base = 0;
    if (id == 0) return true;
    const long long t0 = clock64();
    int64_t p = (int64_t)id - 1;
    while (true) {
        const int64_t q = p - t;
        const unsigned long long v = q >= 0 ? *(volatile unsigned long long *)(tstate + q) : 0ull + LB_PREFIX;
        const unsigned long long st = v & ~LB_VALUE;
        // up to the warp's nearest prefix (tile 0 always publishes one)
        const unsigned pref = __ballot_sync(0xffffffffu, st == LB_PREFIX);
        const unsigned need = pref ? (pref & (0u - pref)) * 2u - 1u : 0xffffffffu;
        const unsigned waiting = __ballot_sync(0xffffffffu, st == 0) & need;
        const unsigned poison = __ballot_sync(0xffffffffu, st == LB_POISON) & need;
        uint64_t add = (need >> lane) & 1u ? v & LB_VALUE : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        if (lane == 0) {
            S.sum[warp] = add;
            S.state[warp] = (pref ? 1u : 0u) | (waiting ? 2u : 0u) | (poison ? 4u : 0u);
        }
        const bool late = __syncthreads_or(t == 0 && clock64() - t0 > wait_cycles);
        bool found = false, wait = false, bad = false;
        uint64_t sum = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            if (!found) {
                const uint32_t x = S.state[w];
                sum += S.sum[w];
                found = x & 1u;
                wait |= (x & 2u) != 0;
                bad |= (x & 4u) != 0;
            }
        }
        __syncthreads();  // the parts are read
        if (bad || (wait && late)) {
            if (t == 0) {
                if (!bad) atomicOr(status, status_bit);
                atomicExch(tstate + id, 0ull + LB_POISON);
            }
            return false;
        }
        if (wait) continue;
        base += sum;
        if (found) break;
        p -= T;
    }
    if (t == 0) atomicExch(tstate + id, LB_PREFIX | (base + total));
    return true;
}

inline unsigned grid_for(uint64_t n, unsigned block, unsigned cap = 1u << 30) {
    uint64_t g = (n + block - 1) / block;
    if (g == 0) g = 1;
    if (g > cap) g = cap;
    return static_cast<unsigned>(g);
}

// ---------------------------------------------------------------------------
// Device-wide primitives (spg_prims.cu)
// ---------------------------------------------------------------------------
// Exclusive scan of n uint64 values in place; writes the total to *d_total
// (device pointer, may be null). Temporary memory from the context pool.
int exclusive_scan_u64(Ctx *c, uint64_t *d_data, uint64_t n, uint64_t *d_total,
                       cudaStream_t s);
// Exclusive scan of int64 (signed) values in place.
int exclusive_scan_i64(Ctx *c, int64_t *d_data, uint64_t n, cudaStream_t s);
// Stable LSD radix sort of 64-bit keys carrying a 32-bit payload, on the low
// `key_bits` bits. Inputs are consumed; results land in (keys, vals) again.
int radix_sort_pairs_u64(Ctx *c, uint64_t *d_keys, uint32_t *d_vals, uint64_t n,
                         int key_bits, cudaStream_t s);
// A first lock's row-grouped inserts, sorted row by row on chip (rows of up to
// 32 entries in registers, longer ones in shared memory): every row's last
// write per column, unless zero, in column order at the row's first input
// positions (out_cols / out_vals[s_off[r] + k], k < off[r + 1] - off[r]);
// s_off[r] = first position of row r (n_rows + 1 entries), off the scan of the
// rows' kept entries, *nnz of them in all (synchronises the stream). *done =
// false when a row has more than 12 288 entries or columns need more than
// ROW_CLASS_CBITS bits; the outputs are then undefined.
constexpr int ROW_CLASS_CBITS = 26;
int dedup_grouped_rows(Ctx *c, const uint32_t *cols, const double *vals, const uint64_t *s_off, uint64_t m,
                       uint64_t n_rows, int cbits, uint32_t *out_cols, double *out_vals, uint64_t *off, uint64_t *nnz,
                       bool *done, cudaStream_t s);

// A CSR's device arrays.
struct CsrView {
    const uint64_t *off;
    const uint32_t *cols;
    const double *vals;
    uint64_t nnz;
};
// Staged inserts stably sorted by row (spg_rowsort.cu). *abort != 0 (and the
// context's status word is set) if a wait gave up: whatever runs on the outputs
// before the next phase_sync has to look at it first. earlier: the flag of what
// the inputs come from (nothing is sorted if it is set); may be null.
struct StagedSorted {
    DevBuf rows, cols, vals, abort;
};
int sort_staged_rows(Ctx *c, const uint32_t *rows, const uint32_t *cols, const double *vals, uint64_t m, int rbits,
                     StagedSorted &out, cudaStream_t s, const unsigned long long *earlier = nullptr);
// Part of spg_selftest_wait_kinds: the sort's wait for earlier tiles runs out.
int rowsort_wait_selftest(Ctx *c, long long wait_cycles, bool *gave_up, cudaStream_t s);
// off[0..n_rows] from the non-decreasing rows srows[0..u) (spg_lock.cu, stream-ordered).
int launch_row_offsets(Ctx *c, const uint32_t *srows, uint64_t u, uint64_t n_rows, uint64_t *off, cudaStream_t s);
// A later lock's delta, small against the matrix, merged into it
// (spg_delta.cu): rows non-decreasing, the last write of each key wins, zeros
// delete. The outputs have room for nnz(A) + m entries (off_out: n_rows + 1).
// *u = distinct keys of the delta. *done = false when a row has too many of
// the inserts; the outputs are then undefined. abort: as above, may be null.
int merge_small_delta(Ctx *c, const CsrView &A, uint64_t n_rows, const uint32_t *rows, const uint32_t *cols,
                      const double *vals, uint64_t m, const unsigned long long *abort, uint64_t *off_out,
                      uint32_t *cols_out, double *vals_out, uint64_t *nnz, uint64_t *u, bool *done, cudaStream_t s);
// Row-grouped entries (row r's are [s_off[r], s_off[r+1]), columns in any
// order) as CSR: the last write of every key in (row, column) order, zeros
// dropped unless keep_zeros (spg_rowtiles.cu). near: most entries' columns lie
// near their row's others (a choice of kernels). The output arrays are sized
// for m entries; n of them are used. *done = false when there are rows of more
// than 12 288 entries and no memory to sort those apart; the outputs are then
// undefined.
struct GroupedOut {
    DevBuf off, cols, vals;
    uint64_t n = 0;
};
int build_grouped_rows(Ctx *c, const uint32_t *cols, const double *vals, const uint64_t *s_off,
                       uint64_t m, uint64_t n_rows, int cbits, bool near, bool keep_zeros,
                       const unsigned long long *abort, GroupedOut *out, bool *done, cudaStream_t s);

// Its rows of more than 12 288 entries, which no block takes: the n of them in
// huge[], `entries` in all, as (place in huge[], column, value) in order, reduced
// like the others; row q's are [first[q], first[q + 1]), and count[huge[q]] is
// their number (spg_lock.cu). abort: as of StagedSorted.
struct HugeRows {
    uint64_t n = 0, entries = 0;
    DevBuf row, cols, vals, first, abort;
};
int order_huge_rows(Ctx *c, const uint32_t *cols, const double *vals, const uint64_t *s_off, const uint32_t *huge,
                    int cbits, bool keep_zeros, HugeRows *H, uint64_t *count, cudaStream_t s);

// SpGEMM pieces shared by its variants (spg_spgemm.cu, spg_spgemm_sort.cu).
// Expand - sort - compress output: kept entries in (row, column) order.
struct EscOut {
    DevBuf crow, ccol, cval;
    uint64_t n = 0;
};
int spgemm_esc(Ctx *c, const Csr *A, const Csr *B, const uint64_t *hp, uint64_t HP, int rbits, int cbits,
               EscOut *out, cudaStream_t s);
void spgemm_install(Csr *Cm, uint64_t m, uint64_t n, DevBuf &&off, DevBuf &&cols, DevBuf &&vals, uint64_t nnz);
uint64_t read_u64(Ctx *c, const uint64_t *d, cudaStream_t s, int *rc);
// ROWMERGE's way when no row has more than SPGEMM_HASH_MAX products
// (spg_spgemm_hash.cu).
constexpr int SPGEMM_HASH_MAX = 64;
bool spgemm_merges_rows(uint64_t m, uint64_t P, bool near);  // whether a thread's merge per row is the faster way all the same
int spgemm_hash_rows(Ctx *c, const Csr *A, const Csr *B, Csr *Cm, uint64_t P, uint64_t room, cudaStream_t s);
int spgemm_warpsort(Ctx *c, const Csr *A, const Csr *B, Csr *Cm, int variant, cudaStream_t s);
int spgemm_run(Ctx *c, const Csr *A, const Csr *B, Csr *Cm, int variant, cudaStream_t s);
// SPG_SPGEMM_AUTO resolved by the context's policy (spg_tune.cu).
int spgemm_resolve_auto(Ctx *c, const Csr *A, const Csr *B, int *variant);

// C = the row-wise merge of two CSRs of the same shape (spg_merge.cu). Sum: equal
// columns add up (one IEEE add), zeros of the result and stored zeros are
// dropped. Replace: B's entry replaces A's, a zero of B deletes; A's other
// entries stay as they are. off_out has n_rows + 1 entries; cols_out / vals_out
// at least nnz(A) + nnz(B). *nnz is read back (the call synchronises).
enum class MergeMode { Sum, Replace };
int merge_csr(Ctx *c, const CsrView &A, const CsrView &B, uint64_t n_rows, MergeMode mode, uint64_t *off_out,
              uint32_t *cols_out, double *vals_out, uint64_t *nnz, cudaStream_t s);
// C = A + B with C's arrays allocated here: for all entries of both sides when
// they are few, by a sample of the equal pairs otherwise.
int sum_csr(Ctx *c, const CsrView &A, const CsrView &B, uint64_t n_rows, uint64_t *off_out, DevBuf &cols, DevBuf &vals,
            uint64_t *nnz, cudaStream_t s);
// Results up to this size keep arrays of their upper bound; larger ones get
// arrays of about their own size (12 bytes an entry).
constexpr uint64_t RESULT_BOUND = 4u << 20;
// Moves n entries out of arrays for `room` of them when more than an eighth is
// unused (waits for the copy).
int fit_arrays(Ctx *c, uint64_t n, uint64_t room, DevBuf &cols, DevBuf &vals, cudaStream_t s);

// CSR helpers used by several ops (spg_lock.cu).
int csr_alloc(Csr *A, uint64_t capacity, cudaStream_t s);

// SpMV dispatch (spg_spmv.cu).
int spmv_launch(Ctx *c, Csr *A, const double *x, double *y, int variant,
                cudaStream_t s);
int spmv_resolve_auto(Ctx *c, Csr *A, int *variant);
// Loads spg_selector.bin from beside libspg.so (or $SPG_SELECTOR_MODEL) if any.
int selector_load_default(Ctx *c);
// Looks up the device address of spg_spmv_noalloc's scratch array for the
// current device again (spg_spmv.cu); spg_ctx_create calls it.
void noalloc_refresh(int device);
// SPG_SPMV_ADAPTIVE, SPG_SPMV_ADAPTIVE16 and SPG_SPMV_INTERLEAVED
// (spg_spmv_adaptive.cu); each builds and caches its plan on first use.
int spmv_adaptive(Ctx *c, Csr *A, const double *x, double *y, int variant, cudaStream_t s);
int build_adaptive_plan(Ctx *c, Csr *A, int variant, cudaStream_t s);
// Pipelined form for the host entry point: splits the chunks into at most nb
// blocks (fewer if a row could outrun the one-block look-ahead of the fix-up)
// and returns the first row of each block (rows->back() = n_rows). Stage i
// (0 <= i <= blocks) enqueues block i's chunks (i < blocks) and block i-1's
// fix-up (i >= 1): after stage i, rows [rows[i-1], rows[i]) are final.
int spmv_adaptive_blocks(Ctx *c, Csr *A, int variant, int nb, std::vector<uint64_t> *rows, cudaStream_t s);
int spmv_adaptive_stage(Ctx *c, Csr *A, const double *x, double *y, int variant, int i, cudaStream_t s);
// Rows [r0, r1) of a row-parallel variant (SCALAR, VECTOR*); others give
// SPG_ERR_UNSUPPORTED.
int spmv_launch_rows(Ctx *c, Csr *A, const double *x, double *y, int variant, uint64_t r0, uint64_t r1,
                     cudaStream_t s);
// A->host_reach for nb equal row blocks (cached until the next lock).
int spmv_row_block_reach(Ctx *c, Csr *A, int nb, cudaStream_t s);
// Fills A->max_row (the longest row) once per CSR; `known` false while `s`
// is being captured (the count needs a synchronisation).
int csr_max_row(Ctx *c, Csr *A, cudaStream_t s, bool *known);
// Builds whatever plan `variant` needs, so that a later spmv_launch only
// enqueues work (plans synchronise: callers that record a CUDA graph call it
// before the recording).
int spmv_prepare(Ctx *c, Csr *A, int variant, cudaStream_t s);
// Shape of a chunk-kernel variant (ADAPTIVE, ADAPTIVE16, INTERLEAVED and
// their tiles): nonzeros per lane, sub-batch depth, interleaved copy, blocks
// of 256 threads per SM. items == 0 for every other variant.
struct SegShape {
    int items, sub;
    bool inter;
    int minb;
};
inline SegShape seg_shape(int variant) {
    switch (variant) {
        case SPG_SPMV_ADAPTIVE: return {32, 8, false, 4};
        case SPG_SPMV_ADAPTIVE16: return {16, 8, false, 4};
        case SPG_SPMV_INTERLEAVED: return {16, 2, true, 8};
        case SPG_SPMV_INTERLEAVED_S4: return {16, 4, true, 5};
        case SPG_SPMV_INTERLEAVED_S8: return {16, 8, true, 4};
        case SPG_SPMV_ADAPTIVE16_S4: return {16, 4, false, 6};
        case SPG_SPMV_ADAPTIVE_S16: return {32, 16, false, 2};
        default: return {0, 0, false, 0};
    }
}
inline bool spmv_is_seg(int variant) { return seg_shape(variant).items != 0; }
// The cached plan slot of one of those variants (tiles share their base's).
inline SpmvPlan &adaptive_plan_of(Csr *A, int variant) {
    return seg_shape(variant).inter ? A->plan_inter : A->plan_adaptive;
}

}  // namespace spg

// Opaque C handle types are the internal structs.
struct spg_ctx : spg::Ctx {};
struct spg_csr : spg::Csr {};
