// spg_spgemm_hash.cu — the row merge of SPG_SPGEMM_ROWMERGE when no row of A
// has more than SH_H products (and not many rows few): C = A * B in Spira's Gustavson order
// (serial/spgemm.hpp:28-48), written to its final place in one pass.
//
// Eight lanes take a row. They walk its A entries in ascending k, each lane one
// entry of B's row k, and add the products up in a hash table of the row in
// shared memory: the columns of one B row differ, so the eight lanes never
// meet in a slot, and a barrier of the warp between two A entries makes every
// C(i, j) the left-to-right sum over ascending k from its first product (+0.0 +
// p1 = p1 whenever the sum can be kept). The loads of eight A entries' B rows
// are in flight together. The kept sums are then compacted, put in column
// order by a bitonic network over the row's lanes, and the tile of SH_ROWS rows goes straight
// into C through an ordered scan of the tiles' counts.
//
// Bound: the FP64 pipe, one multiply and one add per eight-lane step (0.19 ms
// for the 48 M products of the 3D 7-point Laplacian squared); measured there:
// 0.53 ms, the shared-memory and shuffle pipe 79 % and the issue slots 66 %
// busy. A thread per row merging its B rows in registers and a compaction pass
// took 0.73 ms (dependent loads, 28 sectors per warp load); counting the
// smaller columns instead of the network 0.60.
#include <algorithm>

#include "spg_internal.cuh"

namespace spg {
namespace {

constexpr int SH_T = 128, SH_G = 8;             // threads; lanes per row
constexpr int SH_ROWS = 32;                     // rows per tile
constexpr int SH_H = 64;                        // slots of a row's table
constexpr uint32_t SH_EMPTY = 0xFFFFFFFFu;
constexpr unsigned SH_STATUS_TIMEOUT = 0x200u;

struct ShArgs {
    const uint64_t *aoff;
    const uint32_t *acols;
    const double *avals;
    const uint64_t *boff;
    const uint32_t *bcols;
    const double *bvals;
    uint64_t m, n_tiles;
    unsigned long long *ticket, *state;
    uint64_t *coff;
    uint32_t *ccols;
    double *cvals;
    uint64_t room;  // entries that ccols and cvals have room for: those beyond are counted, not written
    unsigned int *status;
    unsigned long long *words;  // [0] entries of C
};

struct ShSmem {
    double val[SH_ROWS][SH_H];
    __align__(16) uint32_t key[SH_ROWS][SH_H];
    uint8_t slot[SH_ROWS][4 * SH_G];
    BlockLookback<SH_T> lb;
    uint32_t cnt[SH_ROWS];
    uint64_t tile;
};

// Adds p to the sum of column c in the row's table, for the lanes that are on
// (all lanes call). The slots are found first, so that the add is one FP64
// instruction for the whole warp: such an instruction costs the same whatever
// its mask (adding inside the probing loop issued it twice per step).
__device__ __forceinline__ void sh_add(uint32_t *key, double *val, bool on, uint32_t c, double p) {
    static_assert(SH_H == 64, "six hash bits");
    uint32_t h = (c * 0x9E3779B1u) >> 26;
    bool todo = on, first = false;
    while (__any_sync(0xffffffffu, todo)) {
        if (todo) {
            uint32_t k = key[h];
            if (k == SH_EMPTY) {
                k = atomicCAS(&key[h], SH_EMPTY, c);
                if (k == SH_EMPTY) {
                    first = true;
                    k = c;
                }
            }
            todo = k != c;
            if (todo) h = (h + 1) & (SH_H - 1);
        }
    }
    __syncwarp();
    if (on) val[h] = first ? p : __dadd_rn(val[h], p);
}

// Ascending bitonic sort of the group's 8 E keys, element 8 e + l in key[e] of
// lane l (four rows per warp at once).
template <int E, class K>
__device__ __forceinline__ void sh_sort(K (&key)[SH_H / SH_G], int l) {
#pragma unroll
    for (int k = 2; k <= SH_G * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= SH_G) {  // partners in one lane
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int f = e | (j / SH_G);
                    if (f != e) {
                        const bool up = ((SH_G * e) & k) == 0;
                        const K x = min(key[e], key[f]), y = max(key[e], key[f]);
                        key[e] = up ? x : y;
                        key[f] = up ? y : x;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const K o = __shfl_xor_sync(0xffffffffu, key[e], j);
                    const bool low = (((SH_G * e + l) & k) == 0) == ((l & j) == 0);
                    key[e] = low ? min(key[e], o) : max(key[e], o);
                }
            }
        }
    }
}

// Idx: B's entry indices; K: column << 6 | slot.
template <class Idx, class K>
__global__ void __launch_bounds__(SH_T, 8) sh_tiles(ShArgs a) {
    extern __shared__ __align__(16) unsigned char sh_raw[];
    ShSmem &S = *reinterpret_cast<ShSmem *>(sh_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int l = lane % SH_G, g0 = lane - l;  // place in the group, the group's first lane
    if (t == 0) S.tile = atomicAdd(a.ticket, 1ull);
#pragma unroll
    for (int i = 0; i < SH_ROWS * SH_H / 4 / SH_T; ++i)
        reinterpret_cast<uint4 *>(&S.key[0][0])[t + i * SH_T] = make_uint4(SH_EMPTY, SH_EMPTY, SH_EMPTY, SH_EMPTY);
    __syncthreads();
    const uint64_t tile = S.tile, row0 = tile * SH_ROWS;
#pragma unroll 1
    for (int pass = 0; pass < SH_ROWS / (SH_T / SH_G); ++pass) {
        const int j = pass * (SH_T / SH_G) + t / SH_G;  // the group's row of the tile
        const uint64_t row = row0 + j;
        uint32_t *key = S.key[j];
        double *val = S.val[j];
        uint64_t ab = 0;
        uint32_t r = 0;
        if (row < a.m) {
            ab = a.aoff[row];
            r = (uint32_t)(a.aoff[row + 1] - ab);
        }
        const uint32_t rmax = __reduce_max_sync(0xffffffffu, r);  // of the warp's four rows
        for (uint32_t t0 = 0; t0 < rmax; t0 += SH_G) {
            // eight A entries of the row, one per lane
            Idx bs = 0;
            uint32_t len = 0;
            double av = 0.0;
            if (t0 + l < r) {
                const uint32_t k = a.acols[ab + t0 + l];
                av = a.avals[ab + t0 + l];
                bs = (Idx)a.boff[k];
                len = (uint32_t)((Idx)a.boff[k + 1] - bs);
            }
            const bool any_long = __any_sync(0xffffffffu, len > (uint32_t)SH_G);
            uint32_t c[SH_G], on = 0;
            double b[SH_G];
#pragma unroll
            for (int q = 0; q < SH_G; ++q) {
                const Idx s = __shfl_sync(0xffffffffu, bs, g0 + q) + (Idx)l;
                c[q] = 0;
                b[q] = 0.0;
                if ((uint32_t)l < __shfl_sync(0xffffffffu, len, g0 + q)) {
                    on |= 1u << q;
                    c[q] = a.bcols[s];
                    b[q] = a.bvals[s];
                }
            }
#pragma unroll
            for (int q = 0; q < SH_G; ++q) {
                if (t0 + q >= rmax) break;  // (warp-uniform)
                const double x = __shfl_sync(0xffffffffu, av, g0 + q);
                sh_add(key, val, (on >> q) & 1u, c[q], __dmul_rn(x, b[q]));
                if (any_long) {  // B rows of more than eight entries
                    const uint32_t n = __shfl_sync(0xffffffffu, len, g0 + q);
                    const uint32_t nmax = __reduce_max_sync(0xffffffffu, n);
                    const Idx s = __shfl_sync(0xffffffffu, bs, g0 + q);
                    for (uint32_t e = SH_G + l; e - l < nmax; e += SH_G) {
                        const uint32_t cc = e < n ? a.bcols[s + e] : 0u;
                        sh_add(key, val, e < n, cc, __dmul_rn(x, e < n ? a.bvals[s + e] : 0.0));
                    }
                }
                __syncwarp();
            }
        }
        // the kept sums' columns and slots (spgemm.hpp:44: v != V{}), compacted
        // into the key array as far as needed for the sort
        constexpr int Q = SH_H / SH_G;
        K k[Q];
        uint32_t n = 0;
        uint32_t occ = 0;
        {
            uint32_t col[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                col[q] = key[l + q * SH_G];
                const bool keep = col[q] != SH_EMPTY && !is_zero(val[l + q * SH_G]);
                occ |= keep ? 1u << q : 0u;
                n += __popc((__ballot_sync(0xffffffffu, keep) >> g0) & 0xFFu);
            }
            __syncwarp();
            if (__reduce_max_sync(0xffffffffu, n) <= 4 * SH_G) {
                // four keys a lane: the group's lanes take turns by place
                uint32_t mine = __popc(occ), inc = mine;
#pragma unroll
                for (int o = 1; o < SH_G; o <<= 1) {
                    const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
                    if (l >= o) inc += x;
                }
                uint32_t w = inc - mine;
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if ((occ >> q) & 1u) S.slot[j][w] = (uint8_t)(l + q * SH_G), ++w;
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t f = l + e * SH_G, slot = f < n ? S.slot[j][f] : 0u;
                    k[e] = f < n ? (K)key[slot] << 6 | slot : ~(K)0;
                }
                sh_sort<4, K>(k, l);
#pragma unroll
                for (int e = 4; e < Q; ++e) k[e] = ~(K)0;
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q) k[q] = (occ >> q) & 1u ? (K)col[q] << 6 | (K)(l + q * SH_G) : ~(K)0;
                sh_sort<Q, K>(k, l);
            }
        }
        double v[Q];
#pragma unroll
        for (int e = 0; e < Q; ++e)
            if (l + e * SH_G < n) v[e] = val[(uint32_t)k[e] & 63u];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < Q; ++e) {
            if (l + e * SH_G < n) {
                key[l + e * SH_G] = (uint32_t)(k[e] >> 6);
                val[l + e * SH_G] = v[e];
            }
        }
        if (l == 0) S.cnt[j] = n;
        __syncwarp();
    }
    __syncthreads();
    // the rows' places in the tile (every warp for itself), the tile's in C
    const uint32_t cnt = S.cnt[lane];
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
    }
    static_assert(SH_ROWS == 32, "a lane per row");
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31), before = inc - cnt;
    if (t == 0) atomicExch(a.state + tile, (tile == 0 ? 0ull + LB_PREFIX : 0ull + LB_AGG) | total);
    uint64_t base = 0;
    if (!block_lookback<SH_T>(S.lb, a.state, tile, total, base, a.status, SH_STATUS_TIMEOUT)) return;
    if (t < SH_ROWS && row0 + t < a.m) a.coff[row0 + t] = base + before;
    if (t == 0 && tile + 1 == a.n_tiles) {
        a.coff[a.m] = base + total;
        store_word(a.words, 0, base + total);
    }
    for (int j = base + total <= a.room ? warp : SH_ROWS; j < SH_ROWS; j += SH_T / 32) {
        const uint32_t n = __shfl_sync(0xffffffffu, cnt, j), o = __shfl_sync(0xffffffffu, before, j);
        for (uint32_t q = lane; q < n; q += 32) {
            a.ccols[base + o + q] = S.key[j][q];
            a.cvals[base + o + q] = S.val[j][q];
        }
    }
}

}  // namespace

// Every row has at most SPGEMM_HASH_MAX products, P of them in all (0 < P <
// 2^32); B has fewer than 2^32 columns (SH_EMPTY is none of them). C has about
// `room` entries (P at most).
int spgemm_hash_rows(Ctx *c, const Csr *A, const Csr *B, Csr *Cm, uint64_t P, uint64_t room, cudaStream_t s) {
    const uint64_t m = A->n_rows, n = B->n_cols, tiles = (m + SH_ROWS - 1) / SH_ROWS;
    static_assert(SPGEMM_HASH_MAX == SH_H, "a slot per product");
    DevBuf state, off, cols, vals;
    SPG_TRY(off.alloc(csr_off_elems(m) * sizeof(uint64_t), s));
    SPG_TRY(state.alloc((1 + tiles) * sizeof(unsigned long long), s));
    unsigned long long *ticket = state.as<unsigned long long>();
    ShArgs a{A->d_off(), A->d_cols(), A->d_vals(), B->d_off(), B->d_cols(), B->d_vals(), m, tiles, ticket, ticket + 1,
             off.as<uint64_t>(), nullptr, nullptr, 0, c->d_status, c->d_words};
    // 32-bit indices and sort keys (column, six slot bits) where they fit
    const bool i32 = B->nnz <= 0xFFFFFFFFull, k32 = n <= (1ull << 26);
    auto k = i32 ? (k32 ? sh_tiles<uint32_t, uint32_t> : sh_tiles<uint32_t, unsigned long long>)
                 : (k32 ? sh_tiles<unsigned long long, uint32_t> : sh_tiles<unsigned long long, unsigned long long>);
    SPG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ShSmem)));
    uint64_t nnz = 0;
    while (true) {
        // (the larger one first: the smaller one first took a part of the place that
        // a freed result had left for it, and the pool mapped memory at every call)
        SPG_TRY(vals.alloc(csr_alloc_elems(room) * sizeof(double), s));
        SPG_TRY(cols.alloc(csr_alloc_elems(room) * sizeof(uint32_t), s));
        SPG_CUDA_TRY(cudaMemsetAsync(state.ptr, 0, (1 + tiles) * sizeof(unsigned long long), s));
        a.ccols = cols.as<uint32_t>();
        a.cvals = vals.as<double>();
        a.room = room;
        k<<<(unsigned)tiles, SH_T, sizeof(ShSmem), s>>>(a);
        SPG_LAUNCH_CHECK();
        SPG_TRY(c->phase_sync(s));
        nnz = c->word(0);
        if (nnz <= room) break;
        room = nnz;  // more entries than expected: again
    }
    if (P > RESULT_BOUND) SPG_TRY(fit_arrays(c, nnz, room, cols, vals, s));
    spgemm_install(Cm, m, n, std::move(off), std::move(cols), std::move(vals), nnz);
    return SPG_OK;
}

}  // namespace spg
