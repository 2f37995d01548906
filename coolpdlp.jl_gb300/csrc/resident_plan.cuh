// resident_plan.cuh -- the slices of LPs that stay in shared memory: their
// device arrays and the host plans that decide which LPs those are (the kernels
// and the layout's reasons are in resident.cuh).
#pragma once

#include <vector>

#include "cpdlp_common.cuh"

namespace cpdlp {

constexpr int RES_MAX_DIM = 65000;      // padded to whole slices per rank: 16-bit indices
constexpr int RES_MAX_CS = 8;            // portable cluster size
constexpr uint32_t RES_MAX_SMEM = 212 * 1024;  // dynamic shared memory of a CTA
constexpr int RES_COEF = 128;            // averaging coefficients computed at a time
// LPs with at least this many nonzeros take a whole cluster.  FP64 (in a batch
// or alone): a step of 1,978 nonzeros takes 3.9 us on one CTA and 3.1 us on 8,
// 575 nonzeros 2.5 and 3.0 us.  FP32 alone: 8,000 nonzeros 2.7 and 1.5 us, 1,978
// nonzeros 1.14 and 1.27 us.  FP32 in a batch: groups of 4 from 3,000 nonzeros
// (10,000 nonzeros: 1.6 us a step against 3.1 us alone on an SM; the slowest LPs
// of a batch end sooner, and 2,048 LPs together take 571 instead of 550 ms;
// groups of 8 from there 679 ms).
constexpr int64_t RES_F64_CLUSTER_NNZ = 1500;
constexpr int64_t RES_F32_CLUSTER_NNZ = 3000;
constexpr int64_t RES_SINGLE_CLUSTER_NNZ = 3000;
// a single LP with FP64 iterates is resident up to this many nonzeros: above,
// the FP64 pipes of the whole chip beat those of eight SMs
constexpr int64_t RES_SINGLE_F64_NNZ = 32000;

// Device arrays of the slices of a set of LPs (the LPs' rows and columns
// concatenated as in the CSR they are built from).
template <class T>
struct ResStore {
    DBuf<uint16_t> idxA, idxAt;     // entries, 32 per slice and width step
    DBuf<T> valA, valAt;
    DBuf<int32_t> metaA, metaAt;    // per LP: CS + 1 rank starts, then each rank's slice offsets
    DBuf<int32_t> ordA, ordAt;      // slice row -> row of the LP
    DBuf<uint16_t> invA, invAt;     // row of the LP -> slice row
    DBuf<uint8_t> lenA, lenAt;      // length of each slice row
    void release() { *this = ResStore(); }
};

struct ResLP {
    int64_t eA, eAt;      // first entry of the LP in the entry arrays
    int32_t mA, mAt;      // first word of its meta lists
    int32_t capA, capAt;  // largest rank's entries / 32 (the shared-memory layout)
    int32_t row_off, col_off, m, n, cs;
};

template <class T>
struct ResView {
    const uint16_t *idxA, *idxAt;
    const T *valA, *valAt;
    const int32_t *metaA, *metaAt, *ordA, *ordAt;
    const uint16_t *invA, *invAt;
    const uint8_t *lenA, *lenAt;
};
template <class T>
ResView<T> res_view(const ResStore<T>& s) {
    return ResView<T>{s.idxA.p, s.idxAt.p, s.valA.p, s.valAt.p, s.metaA.p, s.metaAt.p, s.ordA.p,
                      s.ordAt.p, s.invA.p, s.invAt.p, s.lenA.p, s.lenAt.p};
}

__host__ __device__ inline int res_slices(int rows) { return (rows + 31) / 32; }
// slices of the rank with most of them
__host__ __device__ inline int res_local(int rows, int cs) { return (res_slices(rows) + cs - 1) / cs; }

// byte offsets in the dynamic shared memory of each CTA (the same in every
// rank, so that an address maps to its copy in another CTA)
struct ResLayout {
    uint32_t valA, valAt, vec, idxA, idxAt, offA, offAt, lenA, lenAt, total;
};
template <class T>
__host__ __device__ inline ResLayout res_layout(const ResLP& r) {
    const uint32_t lr = (uint32_t)res_local(r.m, r.cs), lc = (uint32_t)res_local(r.n, r.cs);
    ResLayout o;
    uint32_t p = 0;
    auto take = [&](uint32_t bytes) {
        const uint32_t at = p;
        p += (bytes + 15u) & ~15u;
        return at;
    };
    o.valA = take((uint32_t)r.capA * 32u * (uint32_t)sizeof(T));
    o.valAt = take((uint32_t)r.capAt * 32u * (uint32_t)sizeof(T));
    // step: y | xbar whole (each rank's slices in a block of its own), x xa c lv
    // uv of the own columns, ya lc uc of the own rows; power method (FP64):
    // x | Ax whole, A'Ax own
    const uint32_t whole = 32u * (uint32_t)r.cs * (lr + lc);
    const uint32_t step = (whole + 32u * (5u * lc + 3u * lr)) * (uint32_t)sizeof(T);
    const uint32_t power = (whole + 32u * lc) * 8u;
    o.vec = take(step > power ? step : power);
    o.idxA = take((uint32_t)r.capA * 64u);
    o.idxAt = take((uint32_t)r.capAt * 64u);
    o.offA = take(lr * 4u);
    o.offAt = take(lc * 4u);
    o.lenA = take(lr * 32u);
    o.lenAt = take(lc * 32u);
    o.total = p;
    return o;
}

// Host: the slice lists of one matrix of one LP for clusters of cs CTAs, from
// the LP's row pointer ptr[0..rows]: CS + 1 rank starts, then for each rank
// the offsets of its slices (units of 32 entries).  False when a row is longer
// than LONG_ROW (its sum would not be the tile engine's).
bool res_meta(const int32_t* ptr, int rows, int cs, std::vector<int32_t>& meta, int32_t& cap);

// Cluster size for an LP of `sv`-byte values, 0 when it does not go to the
// resident path; fills r (offsets aside) and the meta lists.
int res_plan(const int32_t* ptrA, const int32_t* ptrAt, int64_t m, int64_t n, int64_t nnz, int sv,
             bool single, ResLP& r, std::vector<int32_t>& metaA, std::vector<int32_t>& metaAt);

// Device: sorts the rows of each LP in `lps` and fills the slices.
template <class T>
void res_build(ResStore<T>& st, const ResLP* lps_dev, int count, const int32_t* a_ptr,
               const int32_t* a_idx, const T* a_val, const int32_t* at_ptr, const int32_t* at_idx,
               const T* at_val, int64_t max_rows, cudaStream_t s);

}  // namespace cpdlp
