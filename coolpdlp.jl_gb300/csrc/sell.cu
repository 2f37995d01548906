// sell.cu -- device build of the sliced-ELL step engine's arrays.
#include "sell.cuh"
#include "sparse_build.cuh"

namespace cpdlp {

namespace {

// One block per window: rows by length (descending, ties in index order) --
// a row's place is the number of rows before it.  Rows longer than LONG_ROW
// keep no entries here and go last.
__global__ void __launch_bounds__(SELL_WINDOW)
    k_sell_sort(const int32_t* __restrict__ ptr, int64_t rows, int32_t* __restrict__ perm,
                uint8_t* __restrict__ len, int32_t* __restrict__ width, int* moved) {
    __shared__ int key[SELL_WINDOW];
    __shared__ int sorted[SELL_WINDOW];
    const int t = threadIdx.x;
    const int64_t r = (int64_t)blockIdx.x * SELL_WINDOW + t;
    int n = -1;  // no row
    if (r < rows) {
        n = ptr[r + 1] - ptr[r];
        if (n > LONG_ROW) n = -1;
    }
    key[t] = n;
    __syncthreads();
    int place = 0;
    for (int q = 0; q < SELL_WINDOW; q++) {
        const int k = key[q];
        place += k > n || (k == n && q < t) ? 1 : 0;
    }
    const int64_t at = (int64_t)blockIdx.x * SELL_WINDOW + place;
    perm[at] = (int32_t)r;
    len[at] = n < 0 ? SELL_SKIP : (uint8_t)n;
    sorted[place] = n;
    if (place != t && n >= 0) *moved = 1;
    __syncthreads();
    if (t % 32 == 0) width[((int64_t)blockIdx.x * SELL_WINDOW + t) / 32] = max(sorted[t], 0);
}

// without the permutation: widths and lengths of the rows in their own order
__global__ void k_sell_plain(const int32_t* __restrict__ ptr, int64_t rows, int64_t padded,
                             uint8_t* __restrict__ len, int32_t* __restrict__ width) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= padded) return;
    int n = -1;
    if (r < rows) {
        n = ptr[r + 1] - ptr[r];
        if (n > LONG_ROW) n = -1;
    }
    len[r] = n < 0 ? SELL_SKIP : (uint8_t)n;
    int w = max(n, 0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(FULL_MASK, w, o));
    if (threadIdx.x % 32 == 0) width[r / 32] = w;
}

template <class T>
__global__ void k_sell_fill(const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            const T* __restrict__ val, const int32_t* __restrict__ off,
                            const uint8_t* __restrict__ len, const int32_t* __restrict__ perm,
                            int64_t padded, int32_t* __restrict__ oidx, T* __restrict__ oval) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= padded) return;
    const int64_t s = k / 32;
    const int o = off[s], w = off[s + 1] - o, n = len[k] == SELL_SKIP ? 0 : len[k];
    const int a = n > 0 ? ptr[perm ? perm[k] : k] : 0;
    for (int q = 0; q < w; q++) {
        const int64_t e = ((int64_t)o + q) * 32 + k % 32;
        oidx[e] = q < n ? idx[a + q] : 0;
        if (oval) oval[e] = q < n ? val[a + q] : T(0);
    }
}

}  // namespace

template <class T>
bool build_sell(SellSide<T>& S, const std::vector<int32_t>& hp, const int32_t* ptr,
                const int32_t* idx, const T* val, int64_t rows, int tile, bool timed, cudaStream_t s) {
    S.release();
    S.tile = tile;
    if (rows <= 0) return true;
    // what the row lengths say (a pass of its own: a matrix that does not suit, or
    // has no long rows, is done with it)
    const int32_t* const p = hp.data();
    int64_t in_long = 0;
    int32_t widest = 0;
    for (int64_t r = 0; r < rows; r++) {
        const int32_t n = p[r + 1] - p[r], own = n > LONG_ROW ? 0 : n;
        in_long += n - own;
        widest = std::max(widest, own);
    }
    S.long_nnz = in_long;
    S.widest = widest;
    S.suits = sell_suits(S, rows, p[rows], val == nullptr);
    if (!timed && !S.suits) {
        S.release();
        return false;
    }
    // the pieces of the rows longer than LONG_ROW
    std::vector<int4> longs;
    int32_t slot = 0, id = 0;
    for (int64_t r = 0; r < rows && in_long > 0; r++) {
        const int32_t n = p[r + 1] - p[r];
        if (n <= LONG_ROW) continue;
        const int32_t np = (n + tile - 1) / tile;
        for (int32_t q = 0; q < np; q++) longs.push_back(make_int4((int32_t)r, -(q + 1), id, slot));
        id++;
        if (np > 1) slot += np;
    }
    S.nltasks = (int32_t)longs.size();
    S.npieces = slot;
    S.ltasks.alloc(std::max<size_t>(longs.size(), 1));
    S.counters.alloc((size_t)std::max(id, 1));
    S.partials.alloc((size_t)std::max(slot, 1));
    if (!longs.empty())
        CK(cudaMemcpyAsync(S.ltasks.p, longs.data(), sizeof(int4) * longs.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(S.counters.p, 0, sizeof(int32_t) * S.counters.n, s));
    // slices
    const int64_t nwin = (rows + SELL_WINDOW - 1) / SELL_WINDOW, padded = nwin * SELL_WINDOW;
    S.nslices = (int32_t)(padded / 32);
    S.len.alloc((size_t)padded);
    S.perm.alloc((size_t)padded);
    S.off.alloc((size_t)S.nslices + 1);
    DBuf<int32_t> width((size_t)S.nslices);
    DBuf<int> moved(1);
    CK(cudaMemsetAsync(moved.p, 0, sizeof(int), s));
    k_sell_sort<<<(unsigned)nwin, SELL_WINDOW, 0, s>>>(ptr, rows, S.perm.p, S.len.p, width.p, moved.p);
    CK_LAUNCH();
    exclusive_scan_i32(width.p, S.off.p, S.nslices, s);
    int32_t sorted_units = 0, plain_units = 0;
    int any = 0;
    CK(cudaMemcpyAsync(&sorted_units, S.off.p + S.nslices, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&any, moved.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    // the rows' own order where it pads hardly more (density order, columns of
    // equal length): no permutation to read, consecutive rows per warp
    DBuf<uint8_t> len2;
    DBuf<int32_t> off2;
    if (any) {
        len2.alloc((size_t)padded);
        off2.alloc((size_t)S.nslices + 1);
        k_sell_plain<<<grid_for(padded, 256), 256, 0, s>>>(ptr, rows, padded, len2.p, width.p);
        CK_LAUNCH();
        exclusive_scan_i32(width.p, off2.p, S.nslices, s);
        CK(cudaMemcpyAsync(&plain_units, off2.p + S.nslices, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
    }
    if (!any || (double)plain_units <= 1.03 * (double)sorted_units) {
        if (any) {
            S.len = std::move(len2);
            S.off = std::move(off2);
            sorted_units = plain_units;
        }
        S.perm.release();
    }
    S.entries = 32 * (int64_t)sorted_units;
    if ((double)S.entries > SELL_MAX_PADDING * (double)hp[(size_t)rows]) {
        CK(cudaStreamSynchronize(s));
        S.release();
        return false;
    }
    S.idx.alloc((size_t)std::max<int64_t>(S.entries, 1));
    if (val) S.val.alloc((size_t)std::max<int64_t>(S.entries, 1));
    k_sell_fill<T><<<grid_for(padded, 256), 256, 0, s>>>(ptr, idx, val, S.off.p, S.len.p, S.perm.p, padded,
                                                         S.idx.p, S.val.p);
    CK_LAUNCH();
    CK(cudaStreamSynchronize(s));  // (the host task list and the temporaries go out of scope)
    return true;
}
template bool build_sell<float>(SellSide<float>&, const std::vector<int32_t>&, const int32_t*,
                                const int32_t*, const float*, int64_t, int, bool, cudaStream_t);
template bool build_sell<double>(SellSide<double>&, const std::vector<int32_t>&, const int32_t*,
                                 const int32_t*, const double*, int64_t, int, bool, cudaStream_t);

}  // namespace cpdlp
