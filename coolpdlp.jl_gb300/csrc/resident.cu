// resident.cu -- host plans and device builds of the slices that resident.cuh
// keeps in shared memory.
#include "resident.cuh"

namespace cpdlp {

namespace {

// Sorts the rows of one LP (blockIdx.x) by length, descending and stable, for
// A (blockIdx.y = 0) or A' (1).  One CTA: the lengths go to shared memory, a
// histogram gives each length's first place, and one warp places the rows in
// order, 32 at a time (rows of equal length by their lane).
__global__ void __launch_bounds__(256)
    k_res_sort(const ResLP* __restrict__ lps, const int32_t* __restrict__ a_ptr,
               const int32_t* __restrict__ at_ptr, int32_t* __restrict__ ordA,
               int32_t* __restrict__ ordAt, uint16_t* __restrict__ invA,
               uint16_t* __restrict__ invAt, uint8_t* __restrict__ lenA,
               uint8_t* __restrict__ lenAt) {
    extern __shared__ uint8_t len[];
    __shared__ int hist[LONG_ROW + 1];
    const ResLP L = lps[blockIdx.x];
    const bool t = blockIdx.y != 0;
    const int rows = t ? L.n : L.m, off = t ? L.col_off : L.row_off;
    const int32_t* ptr = (t ? at_ptr : a_ptr) + off;
    int32_t* ord = (t ? ordAt : ordA) + off;
    uint16_t* inv = (t ? invAt : invA) + off;
    uint8_t* lo = (t ? lenAt : lenA) + off;
    const int loc = res_local(rows, L.cs);
    for (int k = threadIdx.x; k <= LONG_ROW; k += blockDim.x) hist[k] = 0;
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += blockDim.x) {
        const int n = ptr[r + 1] - ptr[r];
        len[r] = (uint8_t)n;
        atomicAdd(&hist[n], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0;
        for (int n = LONG_ROW; n >= 0; n--) {
            const int c = hist[n];
            hist[n] = at;
            at += c;
        }
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    for (int r0 = 0; r0 < rows; r0 += 32) {
        const int r = r0 + lane;
        const bool in = r < rows;
        const int n = in ? len[r] : LONG_ROW + 1;
        const unsigned peers = __match_any_sync(FULL_MASK, n);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        const int at = in ? hist[n] + rank : 0;
        __syncwarp();
        if (in && rank == 0) hist[n] += __popc(peers);
        __syncwarp();
        if (in) {
            // place `at` is row at % 32 of slice at / 32, which is slice
            // (at / 32) / cs of rank (at / 32) % cs; a rank's slices are a block
            const int s = at >> 5;
            ord[at] = r;
            inv[r] = (uint16_t)(((s % L.cs) * loc + s / L.cs) * 32 + (at & 31));
            lo[at] = (uint8_t)n;
        }
    }
}

// Fills the slices of one LP's matrix: thread per slice row, consecutive rows
// write consecutive entries.  Padding: index 0, value 0.
template <class T>
__global__ void __launch_bounds__(256)
    k_res_fill(const ResLP* __restrict__ lps, const int32_t* __restrict__ a_ptr,
               const int32_t* __restrict__ a_idx, const T* __restrict__ a_val,
               const int32_t* __restrict__ at_ptr, const int32_t* __restrict__ at_idx,
               const T* __restrict__ at_val, ResView<T> g, uint16_t* __restrict__ oidxA,
               T* __restrict__ ovalA, uint16_t* __restrict__ oidxAt, T* __restrict__ ovalAt) {
    const ResLP L = lps[blockIdx.x];
    const bool t = blockIdx.y != 0;
    const int rows = t ? L.n : L.m, off = t ? L.col_off : L.row_off, cs = L.cs;
    const int other = t ? L.row_off : L.col_off;
    const int32_t* ptr = (t ? at_ptr : a_ptr) + off;
    const int32_t* idx = t ? at_idx : a_idx;
    const T* val = t ? at_val : a_val;
    const int32_t* ord = (t ? g.ordAt : g.ordA) + off;
    const uint16_t* inv = (t ? g.invA : g.invAt) + other;
    const int32_t* meta = t ? g.metaAt + L.mAt : g.metaA + L.mA;
    uint16_t* oi = t ? oidxAt + L.eAt : oidxA + L.eA;
    T* ov = t ? ovalAt + L.eAt : ovalA + L.eA;
    const int ns = res_slices(rows);
    for (int r = threadIdx.x + blockIdx.z * blockDim.x; r < ns * 32; r += blockDim.x * gridDim.z) {
        const int s = r >> 5, q = s % cs, l = s / cs;
        int list = cs + 1;
        for (int k = 0; k < q; k++) list += (ns - k + cs - 1) / cs + 1;
        const int o = meta[q] + meta[list + l], w = meta[list + l + 1] - meta[list + l];
        int a = 0, n = 0;
        if (r < rows) {
            a = ptr[ord[r]];
            n = ptr[ord[r] + 1] - a;
        }
        for (int k = 0; k < w; k++) {
            const int64_t e = ((int64_t)o + k) * 32 + (r & 31);
            oi[e] = k < n ? inv[idx[a + k] - other] : (uint16_t)0;
            ov[e] = k < n ? val[a + k] : T(0);
        }
    }
}

}  // namespace

bool res_meta(const int32_t* ptr, int rows, int cs, std::vector<int32_t>& meta, int32_t& cap) {
    int32_t hist[LONG_ROW + 1] = {};
    for (int r = 0; r < rows; r++) {
        const int n = ptr[r + 1] - ptr[r];
        if (n > LONG_ROW) return false;
        hist[n]++;
    }
    // widths of the slices: the length of the row at place 32 s
    const int ns = res_slices(rows);
    std::vector<int32_t> width((size_t)ns);
    int n = LONG_ROW, until = hist[LONG_ROW];  // places below `until` have length >= n
    for (int s = 0; s < ns; s++) {
        while (32 * s >= until) until += hist[--n];
        width[(size_t)s] = n;
    }
    meta.assign((size_t)cs + 1, 0);
    cap = 0;
    for (int q = 0; q < cs; q++) {
        int32_t o = 0;
        meta.push_back(0);
        for (int s = q; s < ns; s += cs) {
            o += width[(size_t)s];
            meta.push_back(o);
        }
        meta[(size_t)q + 1] = meta[(size_t)q] + o;
        cap = std::max(cap, o);
    }
    return true;
}

int res_plan(const int32_t* ptrA, const int32_t* ptrAt, int64_t m, int64_t n, int64_t nnz, int sv,
             bool single, ResLP& r, std::vector<int32_t>& metaA, std::vector<int32_t>& metaAt) {
    if (m < 1 || n < 1 || nnz < 1 || m > RES_MAX_DIM || n > RES_MAX_DIM) return 0;
    // FP64 steps are bounded by the SMs' FP64 pipes, so even small LPs are
    // spread over a cluster
    if (single && sv == 8 && nnz > RES_SINGLE_F64_NNZ) return 0;
    int cs = 1;
    if (sv == 8 && nnz >= RES_F64_CLUSTER_NNZ) cs = RES_MAX_CS;
    if (sv == 4 && nnz >= RES_F32_CLUSTER_NNZ) cs = 4;
    if (single && nnz >= RES_SINGLE_CLUSTER_NNZ) cs = RES_MAX_CS;
    r.m = (int32_t)m;
    r.n = (int32_t)n;
    // every rank needs a slice of both matrices: the parts it sends tell the
    // others that it is done with what it received (see ResWait)
    while (cs > 1 && cs > std::min(res_slices(r.m), res_slices(r.n))) cs /= 2;
    for (; cs <= RES_MAX_CS && (cs == 1 || cs <= std::min(res_slices(r.m), res_slices(r.n))); cs *= 2) {
        r.cs = cs;
        // a lower bound first: the unpadded entries
        if ((double)nnz * 2.0 * (2 + sv) > (double)RES_MAX_SMEM * cs) continue;
        if (!res_meta(ptrA, (int)m, cs, metaA, r.capA)) return 0;
        if (!res_meta(ptrAt, (int)n, cs, metaAt, r.capAt)) return 0;
        const ResLayout o = sv == 4 ? res_layout<float>(r) : res_layout<double>(r);
        if (o.total <= RES_MAX_SMEM) return cs;
    }
    return 0;
}

template <class T>
void res_build(ResStore<T>& st, const ResLP* lps_dev, int count, const int32_t* a_ptr,
               const int32_t* a_idx, const T* a_val, const int32_t* at_ptr, const int32_t* at_idx,
               const T* at_val, int64_t max_rows, cudaStream_t s) {
    if (count <= 0) return;
    CK(cudaFuncSetAttribute(k_res_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_MAX_DIM + 1));
    k_res_sort<<<dim3((unsigned)count, 2), 256, (size_t)max_rows, s>>>(
        lps_dev, a_ptr, at_ptr, st.ordA.p, st.ordAt.p, st.invA.p, st.invAt.p, st.lenA.p, st.lenAt.p);
    CK_LAUNCH();
    const unsigned z = (unsigned)std::min<int64_t>(std::max<int64_t>(max_rows / 1024, 1), 64);
    k_res_fill<T><<<dim3((unsigned)count, 2, z), 256, 0, s>>>(
        lps_dev, a_ptr, a_idx, a_val, at_ptr, at_idx, at_val, res_view(st), st.idxA.p, st.valA.p,
        st.idxAt.p, st.valAt.p);
    CK_LAUNCH();
}
template void res_build<float>(ResStore<float>&, const ResLP*, int, const int32_t*, const int32_t*,
                               const float*, const int32_t*, const int32_t*, const float*, int64_t,
                               cudaStream_t);
template void res_build<double>(ResStore<double>&, const ResLP*, int, const int32_t*,
                                const int32_t*, const double*, const int32_t*, const int32_t*,
                                const double*, int64_t, cudaStream_t);

}  // namespace cpdlp
