// resident.cuh -- LPs that stay on the chip: one CTA, or a thread-block cluster
// of CS CTAs, holds an LP's two matrices and its iterates in shared memory and
// runs PDHG steps (pdlp.jl:96-136), KKT evaluations (errors.jl:65-109) and the
// power method (linalg.jl:86-96) without touching global memory in between.
//
// What bounds it.  A step of a small LP is a chain of two products with a
// barrier after each.  Over global memory every link of that chain is an L2
// round trip (task, row pointer, entries, gather), 24 us a step for a
// 5,500-nonzero FP32 LP on one CTA; from shared memory it is a few hundred
// cycles.  FP32 steps are then bounded by shared-memory wavefronts (about 3.5
// a gather of 32 random words); FP64 steps by the FP64 pipe, which on GB300
// retires 1.9 lane operations a clock and SM whether lanes are masked or not
// (64 cycles a warp instruction), so idle lanes cost as much as busy ones.
//
// Layout.  The rows of each matrix are sorted by length (descending, stable)
// and cut into slices of 32, one lane per row, stored column-major and padded
// to the slice's longest row: lanes read consecutive words, and because the
// order is by length the lanes of a slice end together (the padding of a whole
// LP is at most 32 x 64 entries).  Slice s belongs to rank s % CS of the
// cluster.  A row's entries keep their column order and are summed one after
// the other, so row sums are those of the tile engine (rows up to LONG_ROW).
// The gathered vectors (y, xbar) are held whole by every CTA: the owner of a
// row stores its new value into every CTA's copy through distributed shared
// memory (a cluster barrier takes 0.24 us whatever the cluster's size).
// Indices are 16 bit: at most 65,535 rows and columns.
#pragma once

#include <cooperative_groups.h>

#include "cpdlp_common.cuh"
#include "epilogues.cuh"
#include "solver.cuh"

namespace cpdlp {

constexpr int RES_MAX_DIM = 65535;
constexpr int RES_MAX_CS = 8;            // portable cluster size
constexpr uint32_t RES_MAX_SMEM = 222 * 1024;  // dynamic shared memory of a CTA
constexpr int RES_COEF = 128;            // averaging coefficients computed at a time
// LPs with at least this many nonzeros take a whole cluster: in a batch with
// FP64 iterates, and alone with either type
constexpr int64_t RES_F64_CLUSTER_NNZ = 1500;
constexpr int64_t RES_SINGLE_CLUSTER_NNZ = 3000;

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
    // step: y (m) | xbar (n) whole, x xa c lv uv of the own columns, ya lc uc
    // of the own rows; power method (FP64): x (n) | Ax (m) whole, A'Ax own
    const uint32_t step = (((uint32_t)(r.m + r.n) + 7u) / 4u * 4u + 32u * (5u * lc + 3u * lr)) *
                          (uint32_t)sizeof(T);
    const uint32_t power = ((uint32_t)(r.m + r.n) + 4u + 32u * lc) * 8u;
    o.vec = take(step > power ? step : power);
    o.idxA = take((uint32_t)r.capA * 64u);
    o.idxAt = take((uint32_t)r.capAt * 64u);
    o.offA = take((lr + 1u) * 2u);
    o.offAt = take((lc + 1u) * 2u);
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

// ---------------------------------------------------------------------------
// device side
// ---------------------------------------------------------------------------
template <int CS>
__device__ __forceinline__ int res_rank() {
    if constexpr (CS == 1) return 0;
    else return (int)cooperative_groups::this_cluster().block_rank();
}
template <int CS>
__device__ __forceinline__ void res_sync() {
    if constexpr (CS == 1) __syncthreads();
    else cooperative_groups::this_cluster().sync();
}
// stores v at the same place of every CTA's shared memory
template <int CS, class T>
__device__ __forceinline__ void res_put(T* p, T v) {
    if constexpr (CS == 1) *p = v;
    else {
#pragma unroll
        for (int q = 0; q < CS; q++) *cooperative_groups::this_cluster().map_shared_rank(p, q) = v;
    }
}

// one row of a slice: entries at ip/vp + 32 k, k < w (the slice's width); the
// row's own length is len <= w, its padding has index 0
template <class V, class T>
__device__ __forceinline__ T slice_sum(const uint16_t* ip, const V* vp, int w, int len,
                                       const T* vec) {
    T s = T(0);
    int k = 0;
#pragma unroll 1
    for (; k + 4 <= w; k += 4) {
        T p[4];
#pragma unroll
        for (int u = 0; u < 4; u++) p[u] = mul_rn((T)vp[(k + u) * 32], vec[ip[(k + u) * 32]]);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (k + u < len) s = add_rn(s, p[u]);
    }
#pragma unroll 1
    for (; k < w; k++) {
        const T p = mul_rn((T)vp[k * 32], vec[ip[k * 32]]);
        if (k < len) s = add_rn(s, p);
    }
    return s;
}

// Sums Q <= 8 values per thread over the group; every thread gets the sums.
// A warp's first three exchanges halve the number of values a lane carries
// (9 additions a lane instead of 5 Q: FP64 additions are what this costs),
// then warps and ranks are added in order.  sh: NW * 8 + 8 doubles.
template <int Q, int CS, int NW>
__device__ __forceinline__ void res_sum(double (&v)[Q], double* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; q++) a[q] = q < Q ? v[q < Q ? q : 0] : 0.0;
    double b[4], c[2], d;
    {
        const bool h = lane & 16;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double send = h ? a[q] : a[q + 4], keep = h ? a[q + 4] : a[q];
            b[q] = keep + __shfl_xor_sync(FULL_MASK, send, 16);
        }
    }
    {
        const bool h = lane & 8;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const double send = h ? b[q] : b[q + 2], keep = h ? b[q + 2] : b[q];
            c[q] = keep + __shfl_xor_sync(FULL_MASK, send, 8);
        }
    }
    {
        const bool h = lane & 4;
        const double send = h ? c[0] : c[1], keep = h ? c[1] : c[0];
        d = keep + __shfl_xor_sync(FULL_MASK, send, 4);
    }
    d += __shfl_xor_sync(FULL_MASK, d, 2);
    d += __shfl_xor_sync(FULL_MASK, d, 1);
    // lane bits 4, 3, 2 chose values +4, +2, +1
    if ((lane & 3) == 0) sh[w * 8 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = d;
    __syncthreads();
    if (threadIdx.x < Q) {
        double s = 0.0;
        for (int ww = 0; ww < NW; ww++) s += sh[ww * 8 + threadIdx.x];
        sh[NW * 8 + threadIdx.x] = s;
    }
    res_sync<CS>();
#pragma unroll
    for (int q = 0; q < Q; q++) {
        if constexpr (CS == 1) v[q] = sh[NW * 8 + q];
        else {
            double s = cooperative_groups::this_cluster().map_shared_rank(sh, 0)[NW * 8 + q];
            for (int r = 1; r < CS; r++)
                s += cooperative_groups::this_cluster().map_shared_rank(sh, r)[NW * 8 + q];
            v[q] = s;
        }
    }
    res_sync<CS>();
}

// the resident LP as one CTA of its group sees it
template <class T, int CS, int NT>
struct ResCtx {
    static constexpr int NW = NT / 32;
    ResLP R;
    int rank, lane, w;
    int LA, LAt;                  // own slices of A's and A''s rows
    int locA, locAt;              // slices of the fullest rank (vector strides)
    const T *valA, *valAt;
    const uint16_t *idxA, *idxAt, *offA, *offAt;
    const uint8_t *lenA, *lenAt;
    T *y, *xb;                    // gathered vectors, whole
    T *x, *xa, *c, *lv, *uv;      // own columns
    T *ya, *lc, *uc;              // own rows
    double *px, *ps, *pax;        // the power method's vectors
    const int32_t *ordA, *ordAt;  // global: slice row -> row of the LP
    const uint16_t *invA, *invAt;

    // reads the matrices into shared memory; ends with a CTA barrier
    __device__ void load(const ResLP& r, const ResView<T>& g, unsigned char* sm) {
        R = r;
        rank = res_rank<CS>();
        lane = threadIdx.x & 31;
        w = threadIdx.x >> 5;
        const ResLayout o = res_layout<T>(r);
        locA = res_local(r.m, CS);
        locAt = res_local(r.n, CS);
        LA = (res_slices(r.m) - rank + CS - 1) / CS;
        LAt = (res_slices(r.n) - rank + CS - 1) / CS;
        one(g.metaA + r.mA, r.m, LA, g.idxA + r.eA, g.valA + r.eA, g.lenA + r.row_off,
            sm + o.valA, sm + o.idxA, sm + o.offA, sm + o.lenA);
        one(g.metaAt + r.mAt, r.n, LAt, g.idxAt + r.eAt, g.valAt + r.eAt, g.lenAt + r.col_off,
            sm + o.valAt, sm + o.idxAt, sm + o.offAt, sm + o.lenAt);
        valA = reinterpret_cast<const T*>(sm + o.valA);
        valAt = reinterpret_cast<const T*>(sm + o.valAt);
        idxA = reinterpret_cast<const uint16_t*>(sm + o.idxA);
        idxAt = reinterpret_cast<const uint16_t*>(sm + o.idxAt);
        offA = reinterpret_cast<const uint16_t*>(sm + o.offA);
        offAt = reinterpret_cast<const uint16_t*>(sm + o.offAt);
        lenA = sm + o.lenA;
        lenAt = sm + o.lenAt;
        T* v = reinterpret_cast<T*>(sm + o.vec);
        y = v;
        xb = v + (r.m + 3) / 4 * 4;
        x = v + (r.m + r.n + 7) / 4 * 4;
        xa = x + 32 * locAt;
        c = xa + 32 * locAt;
        lv = c + 32 * locAt;
        uv = lv + 32 * locAt;
        ya = uv + 32 * locAt;
        lc = ya + 32 * locA;
        uc = lc + 32 * locA;
        px = reinterpret_cast<double*>(sm + o.vec);
        ps = px + (r.n + 1) / 2 * 2;
        pax = ps + (r.m + 1) / 2 * 2;
        ordA = g.ordA + r.row_off;
        ordAt = g.ordAt + r.col_off;
        invA = g.invA + r.row_off;
        invAt = g.invAt + r.col_off;
        __syncthreads();
    }
    __device__ void one(const int32_t* meta, int rows, int L, const uint16_t* gi, const T* gv,
                        const uint8_t* gl, unsigned char* sv, unsigned char* si,
                        unsigned char* so, unsigned char* sl) {
        const int32_t start = meta[rank], units = meta[rank + 1] - start;
        const int ns = res_slices(rows);
        int list = CS + 1;  // this rank's offsets follow those of the lower ranks
        for (int q = 0; q < rank; q++) list += (ns - q + CS - 1) / CS + 1;
        // 32 entries are 64 bytes of indices and 128 or 256 bytes of values
        const int4* a = reinterpret_cast<const int4*>(gi + (int64_t)start * 32);
        const int4* b = reinterpret_cast<const int4*>(gv + (int64_t)start * 32);
        for (int k = threadIdx.x; k < units * 4; k += NT) reinterpret_cast<int4*>(si)[k] = __ldg(a + k);
        for (int k = threadIdx.x; k < units * (int)(2 * sizeof(T)); k += NT)
            reinterpret_cast<int4*>(sv)[k] = __ldg(b + k);
        for (int k = threadIdx.x; k <= L; k += NT)
            reinterpret_cast<uint16_t*>(so)[k] = (uint16_t)meta[list + k];
        for (int k = threadIdx.x; k < L * 32; k += NT) {
            const int r = ((k >> 5) * CS + rank) * 32 + (k & 31);
            sl[k] = r < rows ? gl[r] : 0;
        }
    }

    // own slice l of a matrix: its rows are r = row(l)
    __device__ __forceinline__ int row(int l) const { return (l * CS + rank) * 32 + lane; }
    template <class VT>
    __device__ __forceinline__ VT sumA(int l, const VT* vec) const {
        const int o = offA[l];
        return slice_sum(idxA + o * 32 + lane, valA + o * 32 + lane, offA[l + 1] - o,
                         lenA[l * 32 + lane], vec);
    }
    template <class VT>
    __device__ __forceinline__ VT sumAt(int l, const VT* vec) const {
        const int o = offAt[l];
        return slice_sum(idxAt + o * 32 + lane, valAt + o * 32 + lane, offAt[l + 1] - o,
                         lenAt[l * 32 + lane], vec);
    }

    // costs and bounds of the own rows and columns (global vectors of the LP)
    __device__ void load_bounds(const T* gc, const T* glv, const T* guv, const T* glc, const T* guc) {
        for (int l = w; l < LAt; l += NW) {
            const int r = row(l);
            if (r < R.n) {
                const int j = ordAt[r];
                c[l * 32 + lane] = gc[j];
                lv[l * 32 + lane] = glv[j];
                uv[l * 32 + lane] = guv[j];
            }
        }
        for (int l = w; l < LA; l += NW) {
            const int r = row(l);
            if (r < R.m) {
                const int i = ordA[r];
                lc[l * 32 + lane] = glc[i];
                uc[l * 32 + lane] = guc[i];
            }
        }
    }
    // whole vectors of the LP into the gathered copies
    __device__ void load_y(const T* gy) {
        for (int i = threadIdx.x; i < R.m; i += NT) y[invA[i]] = __ldcg(gy + i);
    }
    __device__ void load_xb(const T* gx) {
        for (int j = threadIdx.x; j < R.n; j += NT) xb[invAt[j]] = __ldcg(gx + j);
    }
    __device__ void load_x(const T* gx) {
        for (int l = w; l < LAt; l += NW) {
            const int r = row(l);
            if (r < R.n) x[l * 32 + lane] = __ldcg(gx + ordAt[r]);
        }
    }
    __device__ void load_xa(const T* gx) {
        for (int l = w; l < LAt; l += NW) {
            const int r = row(l);
            if (r < R.n) xa[l * 32 + lane] = gx ? __ldcg(gx + ordAt[r]) : T(0);
        }
    }
    __device__ void load_ya(const T* gy) {
        for (int l = w; l < LA; l += NW) {
            const int r = row(l);
            if (r < R.m) ya[l * 32 + lane] = gy ? __ldcg(gy + ordA[r]) : T(0);
        }
    }

    // where the last step of a block leaves sol, sol_last and the averages
    struct Dump {
        T *x, *xl, *xa, *xal, *y, *yl, *ya, *yal;
    };

    // One step! (pdlp.jl:96-136), the arithmetic of PrimalEpi and DualEpi.
    // `last`: also write both iterates and both averages to d.
    __device__ __forceinline__ void step(T tau, T sigma, T inv_sigma, T a, T b, bool avg, bool last,
                                         const Dump& d) {
        for (int l = w; l < LAt; l += NW) {
            const T s = sumAt(l, y);
            const int r = row(l), k = l * 32 + lane;
            if (r < R.n) {
                const T xo = x[k];
                const T xp = proj_box(sub_rn(xo, mul_rn(tau, sub_rn(c[k], s))), lv[k], uv[k]);
                res_put<CS>(xb + r, sub_rn(mul_rn(T(2), xp), xo));
                x[k] = xp;
                T xao = T(0), xan = T(0);
                if (avg) {
                    xao = xa[k];
                    xan = add_rn(mul_rn(xp, a), mul_rn(xao, b));
                    xa[k] = xan;
                }
                if (last) {
                    const int j = ordAt[r];
                    d.x[j] = xp;
                    d.xl[j] = xo;
                    if (avg) {
                        d.xa[j] = xan;
                        d.xal[j] = xao;
                    }
                }
            }
        }
        res_sync<CS>();
        for (int l = w; l < LA; l += NW) {
            const T s = sumA(l, xb);
            const int r = row(l), k = l * 32 + lane;
            if (r < R.m) {
                const T yo = y[r];
                const T t2 = sub_rn(yo, mul_rn(sigma, s));
                const T t4 = sub_rn(mul_rn(inv_sigma, yo), s);
                const T yp = sub_rn(t2, mul_rn(sigma, proj_box(t4, -uc[k], -lc[k])));
                res_put<CS>(y + r, yp);
                T yao = T(0), yan = T(0);
                if (avg) {
                    yao = ya[k];
                    yan = add_rn(mul_rn(yp, a), mul_rn(yao, b));
                    ya[k] = yan;
                }
                if (last) {
                    const int i = ordA[r];
                    d.y[i] = yp;
                    d.yl[i] = yo;
                    if (avg) {
                        d.ya[i] = yan;
                        d.yal[i] = yao;
                    }
                }
            }
        }
        res_sync<CS>();
    }

    // averaging coefficients of the next `count` <= RES_COEF steps from the
    // weight sum tab.es (pdlp.jl:126-136): eta/(eta+es), es/(eta+es), es growing
    // by eta a step (a chain of additions, like the host's).  Computed ahead for
    // all steps at once: an FP64 division a step by one thread, as the step
    // loop over global memory has it, would be longer than the step.
    struct Coefs {
        T a[RES_COEF], b[RES_COEF];
        double es;
    };
    __device__ void coefs(double eta, int count, Coefs& tab) {
        __syncthreads();
        const double es = tab.es;
        __syncthreads();
        for (int t = threadIdx.x; t < count; t += NT) {
            double e = es;
            for (int q = 0; q < t; q++) e += eta;
            tab.a[t] = (T)(eta / (eta + e));
            tab.b[t] = (T)(e / (eta + e));
            if (t == count - 1) tab.es = e + eta;
        }
        __syncthreads();
    }

    // `count` steps; tab.es: the weight sum, advanced (averaging only)
    __device__ void steps(double eta, double omega, int count, bool avg, Coefs& tab, const Dump& d) {
        const double sg = eta * omega;
        const T tau = (T)(eta / omega), sigma = (T)sg, inv_sigma = (T)(1.0 / sg);
        for (int k0 = 0; k0 < count; k0 += RES_COEF) {
            const int nk = min(count - k0, RES_COEF);
            if (avg) coefs(eta, nk, tab);
            for (int k = 0; k < nk; k++)
                step(tau, sigma, inv_sigma, avg ? tab.a[k] : T(0), avg ? tab.b[k] : T(0), avg,
                     k0 + k == count - 1, d);
        }
    }

    // FP64 sums of the KKT terms of one iterate (gx, gy), v = {primal^2,
    // row objective, dual^2, column objective, c'x}; overwrites the gathered
    // copies y and xb
    __device__ void kkt(const T* gx, const T* gy, const T* invD1, const T* invD2, double (&v)[5],
                        double* sh) {
        load_xb(gx);
        load_y(gy);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 5; q++) v[q] = 0.0;
        for (int l = w; l < LA; l += NW) {
            const T s = sumA(l, xb);
            const int r = row(l), k = l * 32 + lane;
            if (r < R.m) {
                const T lo = lc[k], up = uc[k], yy = y[r];
                const double dd = (double)mul_rn(invD1[ordA[r]], sub_rn(s, proj_box(s, lo, up)));
                v[0] += __dmul_rn(dd, dd);
                v[1] += (double)sub_rn(safeprod_left(up, pos_part(-yy)), safeprod_left(lo, neg_part(-yy)));
            }
        }
        for (int l = w; l < LAt; l += NW) {
            const T s = sumAt(l, y);
            const int r = row(l), k = l * 32 + lane;
            if (r < R.n) {
                const T cj = c[k], lo = lv[k], up = uv[k];
                const T gg = sub_rn(cj, s);
                const T rr = proj_multiplier(gg, lo, up);
                const double dd = (double)mul_rn(invD2[ordAt[r]], sub_rn(gg, rr));
                v[2] += __dmul_rn(dd, dd);
                v[3] += (double)sub_rn(safeprod_left(up, pos_part(-rr)), safeprod_left(lo, neg_part(-rr)));
                v[4] += (double)mul_rn(cj, xb[r]);
            }
        }
        res_sum<5, CS, NW>(v, sh);
    }

    // powm! iterations (linalg.jl:86-96) in FP64 over the stored values, from
    // the vector px (already loaded): stops after an iteration whose residual
    // is at most tol or rtol * theta, or after iteration `last`.
    // The residual of an iteration needs its theta, so its norm is summed with
    // the next iteration's theta (one exchange an iteration); the extra
    // iteration's own theta is dropped.  it0: iterations already run.
    struct Power {
        double theta, residual;
        int64_t it;
        bool stop;
    };
    __device__ Power power(int64_t it0, int64_t max_here, int64_t maxiter, double tol, double rtol,
                           double theta_prev, double* sh) {
        Power P{theta_prev, INFINITY, it0, false};
        double r2 = 0.0;       // own part of the last iteration's residual^2
        bool pending = false;  // an iteration's residual is not summed yet
        for (;;) {
            // Ax, then A'Ax with the sums of theta, |A'Ax|^2 and the residual
            for (int l = w; l < LA; l += NW) {
                const double s = sumA(l, px);
                const int r = row(l);
                if (r < R.m) res_put<CS>(ps + r, s);
            }
            res_sync<CS>();
            double v[3] = {0.0, 0.0, r2};
            for (int l = w; l < LAt; l += NW) {
                const double s = sumAt(l, ps);
                const int r = row(l);
                if (r < R.n) {
                    pax[l * 32 + lane] = s;
                    v[0] += px[r] * s;
                    v[1] += s * s;
                }
            }
            res_sum<3, CS, NW>(v, sh);
            if (pending) {
                P.residual = sqrt(v[2]);
                P.it++;
                if (P.it > maxiter || P.residual <= tol || (rtol > 0 && P.residual <= rtol * P.theta)) {
                    P.stop = true;
                    return P;
                }
                if (P.it - it0 >= max_here) return P;
            }
            const double theta = v[0], inv = 1.0 / sqrt(v[1]);
            P.theta = theta;
            r2 = 0.0;
            for (int l = w; l < LAt; l += NW) {
                const int r = row(l);
                if (r < R.n) {
                    const double ax = pax[l * 32 + lane];
                    const double rr = add_rn(mul_rn(-theta, px[r]), ax);
                    r2 += rr * rr;
                    res_put<CS>(px + r, mul_rn(ax, inv));
                }
            }
            pending = true;
            res_sync<CS>();
        }
    }
};

}  // namespace cpdlp
