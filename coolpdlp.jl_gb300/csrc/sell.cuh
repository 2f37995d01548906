// sell.cuh -- the sliced-ELL step engine: one lane per row, 32 rows a slice.
//
// The tile engine (tiles.cuh) computes products nonzero by nonzero, stages them
// in shared memory and sums them row by row: two phases, the second with as
// many lanes as a tile has rows.  Here a lane walks its own row: the row's
// entries are stored column-major in its slice, padded to the slice's longest
// row, so a warp's loads are 128 (indices) and 128 or 256 bytes (values) wide,
// nothing is staged, and the chain is offset -> entries -> gathers -> sum.
// Measured (power-law LP, density order): FP64 6M nonzeros primal step 0.0887 ->
// 0.0376 ms, dual 0.0729 -> 0.0505 ms; FP32 24M nonzeros primal 0.1164 -> 0.0933
// ms, dual 0.1115 -> 0.1096 ms (a quarter of its entries are in long rows).
// It suits the two places where the tile engine is not bound by memory:
//  * FP64 on GB300, whose pipe retires 1.9 lane operations a clock and SM and
//    charges idle lanes like busy ones: products and sums become one fused
//    operation an entry with (nearly) all lanes in use;
//  * small and medium LPs, where a step is the latency of that chain.
// Rows are sorted by length inside windows of SELL_WINDOW rows (a permutation
// kept per slice row, unless it is the identity, as in density order), so that
// the padding stays small.  Rows longer than LONG_ROW are cut into pieces of
// the tile plan's size and reduced by one warp each, like the tile engine's
// long rows; every row sum rounds like the tile engine's in FP32.
#pragma once

#include "tiles.cuh"

namespace cpdlp {

constexpr int SELL_WINDOW = 256;
// the slices may hold this many times the nonzeros; FP32 without the
// autotuner: the share of the nonzeros in rows longer than LONG_ROW
constexpr double SELL_MAX_PADDING = 1.5;
constexpr double SELL_MAX_LONG_F32 = 0.05;
// FP32: a lane walks its row, so a slice takes as long as its longest row has
// entries, while tiles have a lane an entry.  With few rows that chain is the
// kernel: slices take at most this many entries a row, or at least this many rows.
// us a step (tiles, slices; m x m, L entries in every row and column): L = 24: m =
// 500 5.2, 4.5; L = 32: 500 5.3, 5.4, 2,000 6.2, 5.5; L = 48: 2,000 6.2, 7.4, 8,000
// 9.2, 9.1; L = 64: 2,000 6.7, 8.8, 8,000 10.8, 10.3, 16,000 16.9, 14.2.  Narrow
// storage, which reads less: L = 24: 500 4.9, 4.7; L = 32: 2,000 5.9, 5.9, 500 5.1, 5.9;
// L = 48: 8,000 8.4, 9.3, 16,000 14.2, 12.0.  (FP64: slices at all of them: L = 64:
// 500 16.1, 14.7, 8,000 41.5, 17.1.)
constexpr int SELL_F32_ENTRIES = 32, SELL_PM1_ENTRIES = 24;
constexpr int64_t SELL_F32_ROWS = 16000;
constexpr uint8_t SELL_SKIP = 255;  // no row, or a row that the long pieces take

template <class T>
struct SellSide {
    bool on = false;
    bool suits = false;           // sell_suits, of slices that are held
    int32_t nslices = 0, nltasks = 0, npieces = 0, tile = 512;
    int64_t entries = 0;          // with padding
    int64_t long_nnz = 0;         // nonzeros of the rows that the pieces take
    int32_t widest = 0;           // entries of the longest row in a slice
    DBuf<int32_t> off;            // per slice, units of 32 entries
    DBuf<uint8_t> len;            // per slice row
    DBuf<int32_t> perm;           // slice row -> row; empty: the identity
    DBuf<int32_t> idx;
    DBuf<T> val;
    DBuf<int4> ltasks;            // {row, -(piece + 1), id, slot}
    DBuf<int32_t> counters;
    DBuf<T> partials;
    void release() { *this = SellSide(); }
};

// V: the stored values, T: the vectors and sums (FP64 over FP32 values in the
// power method)
template <class V, class T = V>
struct SellView {
    const int32_t* __restrict__ off;
    const uint8_t* __restrict__ len;
    const int32_t* __restrict__ perm;
    const int32_t* __restrict__ idx;
    const V* __restrict__ val;
    const int4* __restrict__ ltasks;
    int32_t* counters;
    T* partials;                       // npieces
    int32_t nslices, nltasks, tile;
    const int32_t* __restrict__ ptr;   // the CSR, for the long rows
    const int32_t* __restrict__ cidx;
    const V* __restrict__ cval;
};

// Whether the products of a side should run on its slices, from its row lengths
// (long_nnz and widest; without the autotuner).  FP64: whenever build_sell keeps them.
template <class T>
bool sell_suits(const SellSide<T>& S, int64_t rows, int64_t nnz, bool narrow) {
    if (sizeof(T) == 8) return true;
    return (double)S.long_nnz <= SELL_MAX_LONG_F32 * (double)nnz &&
           (S.widest <= (narrow ? SELL_PM1_ENTRIES : SELL_F32_ENTRIES) ||
            rows >= SELL_F32_ROWS);
}

// The slices of a CSR (device; hp: its row pointer on the host); tile: the
// piece size of long rows; val null: narrow storage.  False, and nothing kept, when
// they would hold more than SELL_MAX_PADDING times the nonzeros: that is seen
// before they are allocated (a window with one row of 64 entries and 255 empty ones
// pads 32 times).  The same, before any work on the device, where the row lengths
// do not suit (unless `timed`: the autotuner decides).  Leaves S.on false.
template <class T>
bool build_sell(SellSide<T>& S, const std::vector<int32_t>& hp, const int32_t* ptr,
                const int32_t* idx, const T* val, int64_t rows, int tile, bool timed, cudaStream_t s);

template <class V, class T>
SellView<V, T> sell_view(const SellSide<V>& S, const int32_t* ptr, const int32_t* idx, const V* val,
                         T* partials) {
    return SellView<V, T>{S.off.p, S.len.p, S.perm.p, S.idx.p, S.val.p, S.ltasks.p, S.counters.p,
                          partials, S.nslices, S.nltasks, S.tile, ptr, idx, val};
}
template <class V>
SellView<V> sell_view(const SellSide<V>& S, const int32_t* ptr, const int32_t* idx, const V* val) {
    return sell_view<V, V>(S, ptr, idx, val, S.partials.p);
}

__device__ __forceinline__ int ld_cs(const int32_t* p) {
    int v;
    asm volatile("ld.global.cs.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
// N entries of a row from place ip / vp (stride `step`): the loads of all
// entries are in flight together, then, after mid(), all gathers; entries
// beyond the row's length add -0 (its padding has value 0 and index 0).
// COH: the gathered vector may have been written by the kernel before, which ran
// at the same time (a chained launch).
// FUSED: one rounding an entry (FP64 steps), else the product and the sum round.
template <int N, bool COH, bool FUSED, class V, class T, class Mid>
__device__ __forceinline__ T row_chunk(const int32_t* ip, const V* vp, int64_t step, int len,
                                       const T* x, T s, Mid&& mid) {
    int c[N];
    T v[N], g[N];
#pragma unroll
    for (int u = 0; u < N; u++) c[u] = ld_cs(ip + u * step);
    if constexpr (!is_pm1<V>::value) {
#pragma unroll
        for (int u = 0; u < N; u++) v[u] = (T)ld_stream(vp + u * step);
    }
    mid();
#pragma unroll
    for (int u = 0; u < N; u++) g[u] = gather<COH>(x + (is_pm1<V>::value ? pm1_col(c[u]) : c[u]));
#pragma unroll
    for (int u = 0; u < N; u++) {
        if constexpr (is_pm1<V>::value) {
            s = add_rn(s, u < len ? pm1_apply(c[u], g[u]) : T(-0.0));
        } else if constexpr (FUSED) {
            s = __fma_rn(v[u], u < len ? g[u] : T(-0.0), s);
        } else {
            const T p = mul_rn(v[u], g[u]);
            s = add_rn(s, u < len ? p : T(-0.0));
        }
    }
    return s;
}
template <bool COH, bool FUSED, class V, class T, class Mid>
__device__ __forceinline__ T row_rest(const int32_t* ip, const V* vp, int64_t step, int w, int len,
                                      const T* x, T s, Mid&& mid) {
    switch (w) {
        case 8: return row_chunk<8, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 7: return row_chunk<7, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 6: return row_chunk<6, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 5: return row_chunk<5, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 4: return row_chunk<4, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 3: return row_chunk<3, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 2: return row_chunk<2, COH, FUSED>(ip, vp, step, len, x, s, mid);
        case 1: return row_chunk<1, COH, FUSED>(ip, vp, step, len, x, s, mid);
        default: mid(); return s;
    }
}
// A whole row of w stored entries (uniform over the warp), len of them its own;
// mid() runs once, between the first entries' loads and their gathers.
template <bool COH, bool FUSED, class V, class T, class Mid>
__device__ __forceinline__ T row_sum(const int32_t* ip, const V* vp, int64_t step, int w, int len,
                                     const T* x, Mid&& mid) {
    auto none = [] {};
    T s = T(0);
    if (w <= 8) return row_rest<COH, FUSED>(ip, vp, step, w, len, x, s, mid);
    s = row_chunk<8, COH, FUSED>(ip, vp, step, len, x, s, mid);
#pragma unroll 1
    for (;;) {
        w -= 8;
        len -= 8;
        ip += 8 * step;
        if constexpr (!is_pm1<V>::value) vp += 8 * step;
        if (w <= 8) break;
        s = row_chunk<8, COH, FUSED>(ip, vp, step, len, x, s, none);
    }
    return row_rest<COH, FUSED>(ip, vp, step, w, len, x, s, none);
}
// The same with the loads of the next eight entries over the gathers and the sum
// of the ones before: for a product by itself, whose kernel has registers left
// (FP64 power-law 240,000 nonzeros 33 -> 28 us a call).  The step kernels need
// theirs for occupancy: 64-76 registers instead of 40-48 took the FP64 6M-nonzero
// steps from 0.089 to 0.107 ms.
template <bool COH, bool FUSED, class V, class T>
__device__ __forceinline__ T row_sum_ahead(const int32_t* ip, const V* vp, int64_t step, int w,
                                           int len, const T* x) {
    auto none = [] {};
    T s = T(0);
    if (w <= 8) return row_rest<COH, FUSED>(ip, vp, step, w, len, x, s, none);
    int c[8];
    V v[8];
    auto load = [&] {
#pragma unroll
        for (int u = 0; u < 8; u++) c[u] = ld_cs(ip + u * step);
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = ld_stream(vp + u * step);
    };
    load();
#pragma unroll 1
    for (;;) {
        T g[8], a[8];
#pragma unroll
        for (int u = 0; u < 8; u++) g[u] = gather<COH>(x + c[u]);
#pragma unroll
        for (int u = 0; u < 8; u++) a[u] = (T)v[u];
        const int n = len;
        w -= 8;
        len -= 8;
        ip += 8 * step;
        vp += 8 * step;
        const bool full = w >= 8;
        if (full) load();
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if constexpr (FUSED) s = __fma_rn(a[u], u < n ? g[u] : T(-0.0), s);
            else {
                const T p = mul_rn(a[u], g[u]);
                s = add_rn(s, u < n ? p : T(-0.0));
            }
        }
        if (!full) break;
    }
    return row_rest<COH, FUSED>(ip, vp, step, w, len, x, s, none);
}

// epilogues whose FP64 sums round every product and every addition (mul!, whose
// sums of up to LONG_ROW entries are the reference's)
template <class E, class = void>
struct epi_exact : std::false_type {};
template <class E>
struct epi_exact<E, std::enable_if_t<E::EXACT>> : std::true_type {};

// narrow +-1 storage: the signs in the indices, no values
template <class T>
SellView<Pm1, T> sell_view_pm1(const SellSide<T>& S, const int32_t* ptr, const int32_t* idx) {
    return SellView<Pm1, T>{S.off.p, S.len.p, S.perm.p, S.idx.p, nullptr, S.ltasks.p, S.counters.p,
                            S.partials.p, S.nslices, S.nltasks, S.tile, ptr, idx, nullptr};
}

// one piece of a row longer than LONG_ROW (long_piece in tiles.cuh, with the
// piece size at run time and LU entries' loads in flight)
template <bool COH, bool FUSED, int LU = 4, class V, class T, class Epi>
__device__ __forceinline__ void sell_piece(const SellView<V, T>& S, const T* x, Epi& epi,
                                           typename Epi::Acc& acc, int4 t, int lane) {
    const int row = t.x, piece = -t.y - 1, lid = t.z, slot = t.w;
    const int rb = ld_keep(S.ptr + row), re = ld_keep(S.ptr + row + 1);
    const int npieces = (re - rb + S.tile - 1) / S.tile;
    const int a = rb + piece * S.tile, b = min(a + S.tile, re);
    if (COH) {
        grid_wait();
        grid_release();
    }
    T s = T(0);
    for (int e = a + lane; e < b; e += 32 * LU) {
        int c[LU];
        T v[LU], g[LU];
#pragma unroll
        for (int u = 0; u < LU; u++) c[u] = e + 32 * u < b ? ld_cs(S.cidx + e + 32 * u) : 0;
        if constexpr (!is_pm1<V>::value) {
#pragma unroll
            for (int u = 0; u < LU; u++) v[u] = e + 32 * u < b ? (T)ld_stream(S.cval + e + 32 * u) : T(0);
        }
#pragma unroll
        for (int u = 0; u < LU; u++) g[u] = gather<COH>(x + (is_pm1<V>::value ? pm1_col(c[u]) : c[u]));
#pragma unroll
        for (int u = 0; u < LU; u++)
            if (e + 32 * u < b) {
                if constexpr (is_pm1<V>::value) s = add_rn(s, pm1_apply(c[u], g[u]));
                else if constexpr (FUSED) s = __fma_rn(v[u], g[u], s);
                else s = add_rn(s, mul_rn(v[u], g[u]));
            }
    }
    s = warp_sum_tree(s);
    if (npieces == 1) {
        if (lane == 0) epi.row_long(0, row, s, lid, acc);
        return;
    }
    int done = 0;
    if (lane == 0) {
        S.partials[slot + piece] = s;
        __threadfence();
        done = atomicAdd(&S.counters[lid], 1);
    }
    done = __shfl_sync(FULL_MASK, done, 0);
    if (done != npieces - 1) return;
    __threadfence();
    // the partials, 32 at a time: in FP32 added in piece order, like the tile
    // engine, in FP64 by a tree (156 dependent FP64 additions took 5 us)
    T tot = T(0);
    for (int q0 = 0; q0 < npieces; q0 += 32) {
        const T v = q0 + lane < npieces ? __ldcg(S.partials + slot + q0 + lane) : T(0);
        if constexpr (sizeof(T) == 8) tot = add_rn(tot, v);
        else
            for (int q = 0; q < min(32, npieces - q0); q++)
                tot = add_rn(tot, __shfl_sync(FULL_MASK, v, q));
    }
    if constexpr (sizeof(T) == 8) tot = warp_sum_tree(tot);
    if (lane == 0) {
        epi.row_long(0, row, tot, lid, acc);
        S.counters[lid] = 0;
    }
}

// The long pieces first (they take longest), then a warp per slice.  CHAIN: a
// chained launch (grid_wait), which loads the entries and the bounds before it
// waits for the kernel before it.
template <int WARPS, bool CHAIN, class V, class T, class Epi>
__global__ void __launch_bounds__(WARPS * 32)
    k_sell(SellView<V, T> S, const T* x, Epi epi) {
    constexpr bool SPLIT = CHAIN && epi_split<Epi>::value;
    constexpr bool FUSED = sizeof(T) == 8 && !epi_exact<Epi>::value;
    const int lane = threadIdx.x & 31;
    const int task = blockIdx.x * WARPS + (threadIdx.x >> 5);
    typename Epi::Acc acc;
    epi.init(acc);
    if (task < S.nltasks) {
        sell_piece<CHAIN, FUSED>(S, x, epi, acc, S.ltasks[task], lane);
    } else if (task - S.nltasks < S.nslices) {
        const int s = task - S.nltasks, k = s * 32 + lane;
        const int o = ld_keep(S.off + s), w = ld_keep(S.off + s + 1) - o;
        const int len = S.len[k];
        const int r = S.perm ? ld_keep(S.perm + k) : k;
        const bool in = len != SELL_SKIP;
        typename Epi::Pre pre{};
        if (in) {
            if constexpr (SPLIT) pre = epi.pre_static(r);
            else if constexpr (!CHAIN) pre = epi.pre_global(r);
        }
        const int32_t* ip = S.idx + (int64_t)o * 32 + lane;
        const V* vp = nullptr;
        if constexpr (!is_pm1<V>::value) vp = S.val + (int64_t)o * 32 + lane;
        T sum;
        if constexpr (epi_exact<Epi>::value) {  // mul!
            static_assert(!CHAIN, "a product by itself is not chained");
            sum = row_sum_ahead<CHAIN, FUSED>(ip, vp, (int64_t)32, w, in ? len : 0, x);
        } else {
            sum = row_sum<CHAIN, FUSED>(ip, vp, (int64_t)32, w, in ? len : 0, x, [&] {
                if constexpr (CHAIN) {
                    grid_wait();
                    grid_release();
                    if constexpr (SPLIT) {
                        if (in) epi.pre_dynamic(r, pre);
                    } else if (in) pre = epi.pre_global(r);
                }
            });
        }
        if (in) epi.row(0, r, sum, pre, acc);
    }
    epi.finish(acc);
}

// blocks of a launch of eight warps each (the block-partial rows of a reducing
// epilogue; its long-row outputs, one per counter, follow)
template <class V>
int64_t sell_blocks(const SellSide<V>& S) {
    return ((int64_t)S.nslices + S.nltasks + TILE_WARPS - 1) / TILE_WARPS;
}

// Eight warps a block; two, without a reducing epilogue, when the whole grid is
// small, so that it covers all SMs (an FP64 block of eight warps keeps one SM's
// FP64 pipe busy while others are idle).
template <class V, class T, class Epi>
void launch_sell(const SellView<V, T>& S, const T* x, const Epi& epi, cudaStream_t s) {
    const int64_t tasks = (int64_t)S.nslices + S.nltasks;
    if (tasks == 0 || tiles_dry_run()) return;
    constexpr bool REDUCES = !std::is_empty<typename Epi::Acc>::value;
    auto start = [&](auto warps) {
        constexpr int W = decltype(warps)::value;
        const unsigned grid = (unsigned)((tasks + W - 1) / W);
        if constexpr (!epi_exact<Epi>::value) {
            if (chain_this(tasks * 32, is_pm1<V>::value ? 0 : (int)sizeof(T))) {
                launch_chained(k_sell<W, true, V, T, Epi>, grid, W * 32u, s, S, x, epi);
                return;
            }
        }
        k_sell<W, false, V, T, Epi><<<grid, W * 32, 0, s>>>(S, x, epi);
    };
    if constexpr (!REDUCES) {
        if (tasks < 152 * 16) start(std::integral_constant<int, 2>{});
        else start(std::integral_constant<int, TILE_WARPS>{});
    } else {
        start(std::integral_constant<int, TILE_WARPS>{});
    }
    CK_LAUNCH();
}

}  // namespace cpdlp
