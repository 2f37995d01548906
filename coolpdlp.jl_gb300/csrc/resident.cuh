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

#include "epilogues.cuh"
#include "resident_plan.cuh"
#include "solver.cuh"

namespace cpdlp {

// ---------------------------------------------------------------------------
// device side.  Everything of the LP is addressed by byte offsets into the
// dynamic shared memory (32-bit shared-memory instructions, one register an
// address).  The geometry lives in shared memory too, and steps, checks and
// the power method are functions of their own (not inlined), so that each has
// the registers to itself: inlined into one kernel of 64 registers they spilled
// 900 bytes and a step of a 60-row FP32 LP took 2.8 us.
// ---------------------------------------------------------------------------
extern __shared__ __align__(16) unsigned char res_smem[];

template <class V>
__device__ __forceinline__ V& sm_at(uint32_t off) {
    return *reinterpret_cast<V*>(res_smem + off);
}
template <int CS>
__device__ __forceinline__ int res_rank() {
    if constexpr (CS == 1) return 0;
    else return (int)cooperative_groups::this_cluster().block_rank();
}
// the two halves of a group barrier: work between them that touches only the
// thread's own data overlaps the wait (one CTA: all of it in the second half)
template <int CS>
__device__ __forceinline__ void res_arrive() {
    if constexpr (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
template <int CS>
__device__ __forceinline__ void res_wait() {
    if constexpr (CS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}
template <int CS>
__device__ __forceinline__ void res_sync() {
    res_arrive<CS>();
    res_wait<CS>();
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t map_rank(uint32_t a, int rank) {
    uint32_t b;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
    return b;
}
// stores v at the same place of every CTA's shared memory (ordered by the
// group barrier that follows)
template <int CS>
__device__ __forceinline__ void res_put(double* p, double v, int rank) {
    *p = v;
    if constexpr (CS > 1) {
        const uint32_t a = smem_addr(p);
#pragma unroll
        for (int q = 0; q < CS; q++)
            if (q != rank)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(map_rank(a, q)), "d"(v) : "memory");
    }
}

// ---- exchange of a gathered vector -------------------------------------------
// Every CTA holds the whole vector, each rank's slices in a block of its own.
// A warp that finished a slice stores it locally and sends its 128 or 256
// bytes to every other CTA with 16-byte asynchronous stores that count
// themselves on the receiver's mbarrier; a receiver waits until all bytes of
// the other ranks are there.  Against plain remote stores and a cluster
// barrier (whose release waits for the stores' acknowledgements) a half-step
// on 8 CTAs loses 0.5 us of waiting.
// No second barrier protects the readers of the vector: a rank sends its part
// of y after it gathered the whole xbar for it, so a CTA that has all of y
// knows that every CTA is done with xbar, and the other way round.  This, and
// that no CTA's barrier sees bytes of a later phase, needs every rank to send
// some of both vectors: res_plan gives each at least one slice of A and of A'.
struct ResWait {
    uint64_t bar[2];   // mbarriers: 0 for y (and Ax), 1 for xbar (and x)
    // a wait ran out (never, unless the kernel is wrong): here, or in any CTA of
    // the group before the last sum over the group (res_flag)
    int failed;
};
constexpr int RES_TRIES = 1 << 20;  // of a wait
// one warp sends slice block p[0..32) (whole in local shared memory)
template <int CS, class V>
__device__ __forceinline__ void res_send(const V* p, uint64_t* bar, int rank) {
    if constexpr (CS > 1) {
        __syncwarp();
        constexpr int CH = 32 * (int)sizeof(V) / 16;  // 16-byte chunks of a slice
        const int lane = threadIdx.x & 31;
        const uint32_t a = smem_addr(p), mb = smem_addr(bar);
#pragma unroll
        for (int k = 0; k < CH * CS; k += 32) {
            const int q = (k + lane) / CH, c = (k + lane) % CH;
            if (q < CS && q != rank) {
                const int4 v = reinterpret_cast<const int4*>(p)[c];
                asm volatile(
                    "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                        map_rank(a + 16u * (uint32_t)c, q)),
                    "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(map_rank(mb, q))
                    : "memory");
            }
        }
    }
}
// waits for `bytes` of the other ranks; parity: the barrier's phases so far,
// modulo 2 (advanced), and RES_GAVE_UP once a wait ran out: a phase that did not
// complete takes no second arrival.  Also a CTA barrier.
constexpr unsigned RES_GAVE_UP = 1u << 31;
template <int CS>
__device__ __forceinline__ void res_receive(ResWait& W, int which, uint32_t bytes, unsigned& parity,
                                            int most_tries = RES_TRIES) {
    __syncthreads();
    if constexpr (CS > 1) {
        const uint32_t mb = smem_addr(&W.bar[which]);
        if (threadIdx.x == 0 && !(parity & RES_GAVE_UP))
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes)
                         : "memory");
        const unsigned par = (parity >> which) & 1u;
        uint32_t ok = 0;
        for (int tries = 0; tries < most_tries; tries++) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(mb), "r"(par)
                : "memory");
            if (ok || *(volatile int*)&W.failed) break;
        }
        parity ^= 1u << which;
        if (!ok) {
            W.failed = 1;
            parity |= RES_GAVE_UP;
        }
    }
}
// before the first exchange (thread 0 of every CTA, then a group barrier)
__device__ __forceinline__ void res_wait_init(ResWait& W) {
    for (int k = 0; k < 2; k++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&W.bar[k])) : "memory");
    W.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One row of a slice: entries at ip/vp + 32 k, k < w (the slice's width, uniform
// over the warp); the row's own length is len <= w.  Its padding (index 0, value
// 0) adds -0, which changes nothing, and costs no branch.
// FP32: up to eight entries' loads are in flight together (straight code for
// each remainder: guards around each entry's loads took 1.6 times as long); the
// sum rounds each product and each addition like the tile engine.
template <int N, class V>
__device__ __forceinline__ float slice_chunk(const uint16_t* ip, const V* vp, int len,
                                             const float* vec, float s) {
    float p[N];
#pragma unroll
    for (int u = 0; u < N; u++) p[u] = mul_rn(vp[u * 32], vec[ip[u * 32]]);
#pragma unroll
    for (int u = 0; u < N; u++) s = add_rn(s, u < len ? p[u] : -0.0f);
    return s;
}
template <class V>
__device__ __forceinline__ float slice_sum(const uint16_t* ip, const V* vp, int w, int len,
                                           const float* vec) {
    float s = 0.0f;
#pragma unroll 1
    for (; w > 8; w -= 8, len -= 8, ip += 256, vp += 256) s = slice_chunk<8>(ip, vp, len, vec, s);
    switch (w) {
        case 8: return slice_chunk<8>(ip, vp, len, vec, s);
        case 7: return slice_chunk<7>(ip, vp, len, vec, s);
        case 6: return slice_chunk<6>(ip, vp, len, vec, s);
        case 5: return slice_chunk<5>(ip, vp, len, vec, s);
        case 4: return slice_chunk<4>(ip, vp, len, vec, s);
        case 3: return slice_chunk<3>(ip, vp, len, vec, s);
        case 2: return slice_chunk<2>(ip, vp, len, vec, s);
        case 1: return slice_chunk<1>(ip, vp, len, vec, s);
        default: return s;
    }
}
// FP64: fused operations (one rounding where the product and the sum have two)
// in column order, two entries' loads ahead.  A GB300 sub-partition starts one
// FP64 instruction of a warp every 63 cycles (76 with all four busy), dependent
// or not, so their number per sub-partition is what a step costs; a second
// chain for every other entry only added one.
template <class V>
__device__ __forceinline__ double slice_sum(const uint16_t* ip, const V* vp, int w, int len,
                                            const double* vec) {
    double s = 0.0;
    if (w & 1) {
        s = __fma_rn((double)vp[0], len > 0 ? vec[ip[0]] : -0.0, -0.0);
        ip += 32;
        vp += 32;
        w--;
        len--;
    }
    if (w == 0) return s;
    V v0 = vp[0], v1 = vp[32];
    double g0 = vec[ip[0]], g1 = vec[ip[32]];
#pragma unroll 1
    for (;;) {
        const double a0 = (double)v0, a1 = (double)v1, b0 = len > 0 ? g0 : -0.0,
                     b1 = len > 1 ? g1 : -0.0;
        w -= 2;
        if (w > 0) {
            ip += 64;
            vp += 64;
            len -= 2;
            v0 = vp[0];
            v1 = vp[32];
            g0 = vec[ip[0]];
            g1 = vec[ip[32]];
        }
        s = __fma_rn(a0, b0, s);
        s = __fma_rn(a1, b1, s);
        if (w <= 0) return s;
    }
}
constexpr int RES_SUMS = 5;  // most values of one sum
// Sums Q <= RES_SUMS values per thread over the group; every thread gets the
// sums.  FP64 additions are what this costs (64 cycles each, one after the
// other), so few of them are in a row: a warp's first exchanges halve the
// number of values a lane carries (9 additions a lane for 5 values instead of
// 25), every warp stores its sums into every CTA, and after one group barrier
// warp q of each CTA adds value q of all warps of the group with a tree.  The
// order depends on the group's shape alone.  `busy` is false for a warp whose
// values are all zero (it does no additions).  finish(q, sum), by one lane of warp
// q, gives what the threads receive in place of the sum: what every thread would
// compute alike costs the pipe once per warp.  Both together took an iteration
// of the power method from 7.5 to 4.5 us (1,000 x 2,000, 16 warps a CTA).
// sh: res_sh<CS, NW>() doubles; `phase` alternates the halves, so that a fast
// CTA's next sums do not meet a slow one's reads.
// With the sums every CTA learns whether a wait ran out in any of them: a CTA
// that acted on its own wait alone would leave its loops, and the group's
// barriers, at another point than the others.
template <int CS, int NW>
constexpr int res_slot_size() { return RES_SUMS * CS * NW + CS; }
template <int CS, int NW>
constexpr int res_sh() { return 2 * res_slot_size<CS, NW>() + 8; }
// a warp's part of the sums, stored into every CTA's slots
template <int Q, int CS, int NW>
__device__ __forceinline__ void res_partial(const double (&v)[Q], double* slot, bool busy) {
    static_assert(Q <= RES_SUMS && Q <= NW, "a warp per value");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int P = CS * NW;  // warps of the group
    double d = 0.0;
    int which = lane / (Q <= 4 ? 8 : 4);
    if (!busy) {
    } else if constexpr (Q <= 4) {
        double a[4], c[2];
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = q < Q ? v[q < Q ? q : 0] : 0.0;
        const bool h = lane & 16, h2 = lane & 8;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const double send = h ? a[q] : a[q + 2], keep = h ? a[q + 2] : a[q];
            c[q] = keep + __shfl_xor_sync(FULL_MASK, send, 16);
        }
        const double send = h2 ? c[0] : c[1], keep = h2 ? c[1] : c[0];
        d = keep + __shfl_xor_sync(FULL_MASK, send, 8);
        d += __shfl_xor_sync(FULL_MASK, d, 4);
    } else {
        double a[8], b[4], c[2];
#pragma unroll
        for (int q = 0; q < 8; q++) a[q] = q < Q ? v[q < Q ? q : 0] : 0.0;
        const bool h = lane & 16, h2 = lane & 8, h3 = lane & 4;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double send = h ? a[q] : a[q + 4], keep = h ? a[q + 4] : a[q];
            b[q] = keep + __shfl_xor_sync(FULL_MASK, send, 16);
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const double send = h2 ? b[q] : b[q + 2], keep = h2 ? b[q + 2] : b[q];
            c[q] = keep + __shfl_xor_sync(FULL_MASK, send, 8);
        }
        const double send = h3 ? c[0] : c[1], keep = h3 ? c[1] : c[0];
        d = keep + __shfl_xor_sync(FULL_MASK, send, 4);
    }
    if (busy) {
        d += __shfl_xor_sync(FULL_MASK, d, 2);
        d += __shfl_xor_sync(FULL_MASK, d, 1);
    }
    const int rank = res_rank<CS>();
    if ((lane & (Q <= 4 ? 7 : 3)) == 0 && which < Q)
        res_put<CS>(slot + which * P + rank * NW + w, d, rank);
    __syncwarp();
}
// whether a wait ran out in any CTA of the group before its res_put_flag (one
// warp each, the group barrier between them); the same answer in every CTA
template <int CS, int NW>
__device__ __forceinline__ void res_put_flag(double* slot, const ResWait& W) {
    const int lane = threadIdx.x & 31;
    if (lane < CS) {
        const double f = *(const volatile int*)&W.failed ? 1.0 : 0.0;
        const uint32_t a = smem_addr(slot + RES_SUMS * CS * NW + res_rank<CS>());
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(map_rank(a, lane)), "d"(f) : "memory");
    }
    __syncwarp();
}
template <int CS, int NW>
__device__ __forceinline__ bool res_flag(const double* slot) {
    const int lane = threadIdx.x & 31;
    return __any_sync(FULL_MASK, lane < CS && slot[RES_SUMS * CS * NW + lane] != 0.0);
}
// value q of all warps of the group, by one warp (whole in every lane)
template <int CS, int NW>
__device__ __forceinline__ double res_total(const double* slot, int q) {
    constexpr int P = CS * NW;
    const int lane = threadIdx.x & 31;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < (P + 31) / 32; k++)
        if (k * 32 + lane < P) s = k ? s + slot[q * P + k * 32 + lane] : slot[q * P + lane];
#pragma unroll
    for (int o = (P < 32 ? P : 32) / 2; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
    return s;
}
template <int CS, int NW>
__device__ __forceinline__ double* res_slot(double* sh, int& phase) {
    double* slot = sh + 8 + phase * res_slot_size<CS, NW>();
    phase ^= 1;
    return slot;
}
template <int Q, int CS, int NW, class F>
__device__ __forceinline__ void res_sum(double (&v)[Q], double* sh, int& phase, ResWait& W, bool busy,
                                        F&& finish) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double* slot = res_slot<CS, NW>(sh, phase);
    res_partial<Q, CS, NW>(v, slot, busy);
    if constexpr (CS > 1)
        if (w == NW - 1) res_put_flag<CS, NW>(slot, W);
    res_sync<CS>();
    if constexpr (CS > 1)
        if (w == NW - 1 && res_flag<CS, NW>(slot) && lane == 0) W.failed = 1;
    if (w < Q) {
        const double s = res_total<CS, NW>(slot, w);
        if (lane == 0) sh[w] = finish(w, s);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; q++) v[q] = sh[q];
    // sh[0..7] are rewritten only after the next call's group barrier
}

template <int Q, int CS, int NW>
__device__ __forceinline__ void res_sum(double (&v)[Q], double* sh, int& phase, ResWait& W,
                                        bool busy = true) {
    res_sum<Q, CS, NW>(v, sh, phase, W, busy, [](int, double s) { return s; });
}

// the resident LP as one CTA of its group sees it (in shared memory)
struct ResGeo {
    ResLP R;
    int rank;
    int LA, LAt;                  // own slices of A's and A''s rows
    int baseA, baseAt;            // place of the own block in a gathered vector
    uint32_t remA, remAt;         // rows in the other ranks' slices (with padding)
    ResLayout o;
    uint32_t y, xb;               // gathered vectors, whole
    uint32_t x, xa, c, lv, uv;    // own columns
    uint32_t ya, lc, uc;          // own rows
    uint32_t px, ps, pax;         // the power method's vectors
    const int32_t *ordA, *ordAt;  // global: slice row -> row of the LP
    const uint16_t *invA, *invAt;
};
// averaging coefficients of the next steps and the weight sum (shared memory)
template <class T>
struct ResCoefs {
    T a[RES_COEF], b[RES_COEF];
    T k[3];  // tau, sigma, 1 / sigma
    double es;
};
// where the last step of a block leaves sol, sol_last and the averages
template <class T>
struct ResDump {
    T *x, *xl, *xa, *xal, *y, *yl, *ya, *yal;
};
struct ResPower {
    double theta, residual;
    int64_t it;
    bool stop;
};

// f(l, r) for each own slice l of this warp and this lane's row r of it
template <int CS, int NT, class F>
__device__ __forceinline__ void res_rows(int slices, int rank, int rows, F&& f) {
    const int lane = threadIdx.x & 31;
    for (int l = threadIdx.x >> 5; l < slices; l += NT / 32) {
        const int r = (l * CS + rank) * 32 + lane;
        if (r < rows) f(l * 32 + lane, r);
    }
}

template <class T, int CS, int NT>
__device__ void res_load_side(const ResGeo& G, const int32_t* meta, int rows, int L,
                              const uint16_t* gi, const T* gv, const uint8_t* gl, uint32_t sv,
                              uint32_t si, uint32_t so, uint32_t sl) {
    const int rank = G.rank;
    const int32_t start = meta[rank], units = meta[rank + 1] - start;
    const int ns = res_slices(rows);
    int list = CS + 1;  // this rank's offsets follow those of the lower ranks
    for (int q = 0; q < rank; q++) list += (ns - q + CS - 1) / CS + 1;
    // 32 entries are 64 bytes of indices and 128 or 256 bytes of values
    const int4* a = reinterpret_cast<const int4*>(gi + (int64_t)start * 32);
    const int4* b = reinterpret_cast<const int4*>(gv + (int64_t)start * 32);
    for (int k = threadIdx.x; k < units * 4; k += NT) (&sm_at<int4>(si))[k] = __ldg(a + k);
    for (int k = threadIdx.x; k < units * (int)(2 * sizeof(T)); k += NT)
        (&sm_at<int4>(sv))[k] = __ldg(b + k);
    // offset (units of 32 entries) and width of each slice in one word
    for (int k = threadIdx.x; k < L; k += NT)
        (&sm_at<uint32_t>(so))[k] = (uint32_t)meta[list + k] << 8 | (uint32_t)(meta[list + k + 1] - meta[list + k]);
    for (int k = threadIdx.x; k < L * 32; k += NT) {
        const int r = ((k >> 5) * CS + rank) * 32 + (k & 31);
        (&sm_at<uint8_t>(sl))[k] = r < rows ? gl[r] : 0;
    }
}
// the geometry and the matrices of LP r; ends with a CTA barrier
template <class T, int CS, int NT>
__device__ __noinline__ void res_load(ResGeo& G, const ResLP& r, const ResView<T>& g) {
    if (threadIdx.x == 0) {
        G.R = r;
        G.rank = res_rank<CS>();
        G.LA = (res_slices(r.m) - G.rank + CS - 1) / CS;
        G.LAt = (res_slices(r.n) - G.rank + CS - 1) / CS;
        G.o = res_layout<T>(r);
        const uint32_t S = sizeof(T), cols = 32u * S * (uint32_t)res_local(r.n, CS),
                       rows = 32u * S * (uint32_t)res_local(r.m, CS);
        G.baseA = G.rank * res_local(r.m, CS) * 32;
        G.baseAt = G.rank * res_local(r.n, CS) * 32;
        G.remA = 32u * (uint32_t)(res_slices(r.m) - G.LA);
        G.remAt = 32u * (uint32_t)(res_slices(r.n) - G.LAt);
        G.y = G.o.vec;
        G.xb = G.y + CS * rows;
        G.x = G.xb + CS * cols;
        G.xa = G.x + cols;
        G.c = G.xa + cols;
        G.lv = G.c + cols;
        G.uv = G.lv + cols;
        G.ya = G.uv + cols;
        G.lc = G.ya + rows;
        G.uc = G.lc + rows;
        G.px = G.o.vec;
        G.ps = G.px + CS * 256u * (uint32_t)res_local(r.n, CS);
        G.pax = G.ps + CS * 256u * (uint32_t)res_local(r.m, CS);
        G.ordA = g.ordA + r.row_off;
        G.ordAt = g.ordAt + r.col_off;
        G.invA = g.invA + r.row_off;
        G.invAt = g.invAt + r.col_off;
    }
    __syncthreads();
    res_load_side<T, CS, NT>(G, g.metaA + r.mA, r.m, G.LA, g.idxA + r.eA, g.valA + r.eA,
                             g.lenA + r.row_off, G.o.valA, G.o.idxA, G.o.offA, G.o.lenA);
    res_load_side<T, CS, NT>(G, g.metaAt + r.mAt, r.n, G.LAt, g.idxAt + r.eAt, g.valAt + r.eAt,
                             g.lenAt + r.col_off, G.o.valAt, G.o.idxAt, G.o.offAt, G.o.lenAt);
    __syncthreads();
}
// costs and bounds of the own rows and columns (global vectors of the LP)
template <class T, int CS, int NT>
__device__ __noinline__ void res_bounds(const ResGeo& G, const T* gc, const T* glv, const T* guv,
                                        const T* glc, const T* guc) {
    res_rows<CS, NT>(G.LAt, G.rank, G.R.n, [&](int k, int r) {
        const int j = G.ordAt[r];
        (&sm_at<T>(G.c))[k] = gc[j];
        (&sm_at<T>(G.lv))[k] = glv[j];
        (&sm_at<T>(G.uv))[k] = guv[j];
    });
    res_rows<CS, NT>(G.LA, G.rank, G.R.m, [&](int k, int r) {
        const int i = G.ordA[r];
        (&sm_at<T>(G.lc))[k] = glc[i];
        (&sm_at<T>(G.uc))[k] = guc[i];
    });
}
// whole vectors of the LP (global, the LP's order) into the gathered copies
template <class T, int NT>
__device__ __forceinline__ void res_load_y(const ResGeo& G, const T* gy) {
    T* y = &sm_at<T>(G.y);
    for (int i = threadIdx.x; i < G.R.m; i += NT) y[G.invA[i]] = __ldcg(gy + i);
}
template <class T, int NT>
__device__ __forceinline__ void res_load_xb(const ResGeo& G, const T* gx) {
    T* xb = &sm_at<T>(G.xb);
    for (int j = threadIdx.x; j < G.R.n; j += NT) xb[G.invAt[j]] = __ldcg(gx + j);
}
// sol and the average (null: zero) of the own rows and columns, and y whole
template <class T, int CS, int NT>
__device__ __noinline__ void res_load_iterate(const ResGeo& G, const T* gx, const T* gxa,
                                              const T* gy, const T* gya) {
    res_rows<CS, NT>(G.LAt, G.rank, G.R.n, [&](int k, int r) {
        (&sm_at<T>(G.x))[k] = __ldcg(gx + G.ordAt[r]);
        (&sm_at<T>(G.xa))[k] = gxa ? __ldcg(gxa + G.ordAt[r]) : T(0);
    });
    res_rows<CS, NT>(G.LA, G.rank, G.R.m, [&](int k, int r) {
        (&sm_at<T>(G.ya))[k] = gya ? __ldcg(gya + G.ordA[r]) : T(0);
    });
    res_load_y<T, NT>(G, gy);
}

// `count` steps (pdlp.jl:96-136); FP32: the arithmetic of PrimalEpi and
// DualEpi, FP64: the same with fused operations.  tab.es: the weight sum,
// advanced (averaging only).  The last step also writes both iterates and both
// averages to d; ends with a group barrier.
template <class T, int CS, int NT>
__device__ __noinline__ void res_steps(const ResGeo& G, double eta, double omega, int count,
                                       bool avg, ResCoefs<T>& tab, const ResDump<T>& d, ResWait& W,
                                       unsigned& parity_io) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = G.rank;
    const int LA = G.LA, LAt = G.LAt, m = G.R.m, n = G.R.n;
    const T *valA = &sm_at<T>(G.o.valA) + lane, *valAt = &sm_at<T>(G.o.valAt) + lane;
    const uint16_t *idxA = &sm_at<uint16_t>(G.o.idxA) + lane, *idxAt = &sm_at<uint16_t>(G.o.idxAt) + lane;
    const uint32_t *offA = &sm_at<uint32_t>(G.o.offA), *offAt = &sm_at<uint32_t>(G.o.offAt);
    const uint8_t *lenA = &sm_at<uint8_t>(G.o.lenA) + lane, *lenAt = &sm_at<uint8_t>(G.o.lenAt) + lane;
    const T *y = &sm_at<T>(G.y), *xb = &sm_at<T>(G.xb);
    T *yown = &sm_at<T>(G.y) + G.baseA, *xbown = &sm_at<T>(G.xb) + G.baseAt;
    T *x = &sm_at<T>(G.x) + lane, *xa = &sm_at<T>(G.xa) + lane, *ya = &sm_at<T>(G.ya) + lane;
    const T *c = &sm_at<T>(G.c) + lane, *lv = &sm_at<T>(G.lv) + lane, *uv = &sm_at<T>(G.uv) + lane;
    const T *lc = &sm_at<T>(G.lc) + lane, *uc = &sm_at<T>(G.uc) + lane;
    unsigned parity = parity_io;
    T tau = T(0), sigma = T(0), inv_sigma = T(0);
    for (int k0 = 0; k0 < count; k0 += RES_COEF) {
        const int nk = min(count - k0, RES_COEF);
        // the step sizes, and eta/(eta+es), es/(eta+es) of all nk steps at once,
        // es growing by eta a step (a chain of additions, like the host's): a
        // division a step by one thread would be longer than the step
        __syncthreads();
        const double es = tab.es;
        __syncthreads();
        if (avg)
            for (int t = threadIdx.x; t < nk; t += NT) {
                double e = es;
                for (int q = 0; q < t; q++) e += eta;
                tab.a[t] = (T)(eta / (eta + e));
                tab.b[t] = (T)(e / (eta + e));
                if (t == nk - 1) tab.es = e + eta;
            }
        if (threadIdx.x == NT - 32) {
            const double sg = eta * omega;
            tab.k[0] = (T)(eta / omega);
            tab.k[1] = (T)sg;
            tab.k[2] = (T)(1.0 / sg);
        }
        __syncthreads();
        tau = tab.k[0];
        sigma = tab.k[1];
        inv_sigma = tab.k[2];
#pragma unroll 1
        for (int st = 0; st < nk; st++) {
            const bool last = k0 + st == count - 1;
#pragma unroll 1
            for (int l = w; l < LAt; l += NW) {
                const int k = l * 32, r = (l * CS + rank) * 32 + lane;
                const uint32_t o = offAt[l];
                const T xo = x[k], cj = c[k], lo = lv[k], up = uv[k];
                const T s = slice_sum(idxAt + (o >> 8) * 32, valAt + (o >> 8) * 32, (int)(o & 255u),
                                      lenAt[k], y);
                const T xp = proj_box(mul_add(-tau, sub_rn(cj, s), xo), lo, up);
                xbown[k + lane] = extrapolate(xp, xo);
                x[k] = xp;
                res_send<CS>(xbown + k, &W.bar[1], rank);
                if (last && r < n) {
                    d.x[G.ordAt[r]] = xp;
                    d.xl[G.ordAt[r]] = xo;
                }
            }
            // the averages are formed while the others' parts arrive
            if (avg) {
                const T a = tab.a[st], b = tab.b[st];
#pragma unroll 1
                for (int l = w; l < LAt; l += NW) {
                    const int k = l * 32, r = (l * CS + rank) * 32 + lane;
                    const T xao = xa[k], xan = mul_add(x[k], a, mul_rn(xao, b));
                    xa[k] = xan;
                    if (last && r < n) {
                        d.xa[G.ordAt[r]] = xan;
                        d.xal[G.ordAt[r]] = xao;
                    }
                }
            }
            res_receive<CS>(W, 1, G.remAt * (uint32_t)sizeof(T), parity);
#pragma unroll 1
            for (int l = w; l < LA; l += NW) {
                const int k = l * 32, r = (l * CS + rank) * 32 + lane;
                const uint32_t o = offA[l];
                const T yo = yown[k + lane], lo = lc[k], up = uc[k];
                const T s = slice_sum(idxA + (o >> 8) * 32, valA + (o >> 8) * 32, (int)(o & 255u),
                                      lenA[k], xb);
                const T t2 = mul_add(-sigma, s, yo);
                const T t4 = mul_add(inv_sigma, yo, -s);
                const T yp = mul_add(-sigma, proj_box(t4, -up, -lo), t2);
                yown[k + lane] = yp;
                res_send<CS>(yown + k, &W.bar[0], rank);
                if (last && r < m) {
                    d.y[G.ordA[r]] = yp;
                    d.yl[G.ordA[r]] = yo;
                }
            }
            if (avg) {
                const T a = tab.a[st], b = tab.b[st];
#pragma unroll 1
                for (int l = w; l < LA; l += NW) {
                    const int k = l * 32, r = (l * CS + rank) * 32 + lane;
                    const T yao = ya[k], yan = mul_add(yown[k + lane], a, mul_rn(yao, b));
                    ya[k] = yan;
                    if (last && r < m) {
                        d.ya[G.ordA[r]] = yan;
                        d.yal[G.ordA[r]] = yao;
                    }
                }
            }
            res_receive<CS>(W, 0, G.remA * (uint32_t)sizeof(T), parity);
        }
    }
    parity_io = parity;
    // a check reads what the other CTAs dumped, and overwrites y and xbar
    res_sync<CS>();
}

// FP64 sums of the KKT terms of one iterate (gx, gy): v = {primal^2, row
// objective, dual^2, column objective, c'x}; overwrites the gathered copies
// y and xb
template <class T, int CS, int NT>
__device__ __noinline__ void res_kkt_sums(const ResGeo& G, const T* gx, const T* gy, const T* invD1,
                                          const T* invD2, double (&out)[5], double* sh, int& phase,
                                          ResWait& W) {
    const int lane = threadIdx.x & 31;
    res_load_xb<T, NT>(G, gx);
    res_load_y<T, NT>(G, gy);
    __syncthreads();
    const T *y = &sm_at<T>(G.y), *xb = &sm_at<T>(G.xb);
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    {
        const T *val = &sm_at<T>(G.o.valA) + lane, *lc = &sm_at<T>(G.lc) + lane, *uc = &sm_at<T>(G.uc) + lane;
        const uint16_t* idx = &sm_at<uint16_t>(G.o.idxA) + lane;
        const uint32_t* off = &sm_at<uint32_t>(G.o.offA);
        const uint8_t* len = &sm_at<uint8_t>(G.o.lenA) + lane;
        for (int l = threadIdx.x >> 5; l < G.LA; l += NT / 32) {
            const int k = l * 32, r = (l * CS + G.rank) * 32 + lane;
            const uint32_t o = off[l];
            const T s = slice_sum(idx + (o >> 8) * 32, val + (o >> 8) * 32, (int)(o & 255u), len[k], xb);
            if (r < G.R.m) {
                const T lo = lc[k], up = uc[k], yy = y[G.baseA + k + lane];
                const double dd = (double)mul_rn(invD1[G.ordA[r]], sub_rn(s, proj_box(s, lo, up)));
                v[0] += __dmul_rn(dd, dd);
                v[1] += (double)sub_rn(safeprod_left(up, pos_part(-yy)), safeprod_left(lo, neg_part(-yy)));
            }
        }
    }
    {
        const T *val = &sm_at<T>(G.o.valAt) + lane, *lv = &sm_at<T>(G.lv) + lane,
                *uv = &sm_at<T>(G.uv) + lane, *c = &sm_at<T>(G.c) + lane;
        const uint16_t* idx = &sm_at<uint16_t>(G.o.idxAt) + lane;
        const uint32_t* off = &sm_at<uint32_t>(G.o.offAt);
        const uint8_t* len = &sm_at<uint8_t>(G.o.lenAt) + lane;
        for (int l = threadIdx.x >> 5; l < G.LAt; l += NT / 32) {
            const int k = l * 32, r = (l * CS + G.rank) * 32 + lane;
            const uint32_t o = off[l];
            const T s = slice_sum(idx + (o >> 8) * 32, val + (o >> 8) * 32, (int)(o & 255u), len[k], y);
            if (r < G.R.n) {
                const T cj = c[k], lo = lv[k], up = uv[k];
                const T gg = sub_rn(cj, s);
                const T rr = proj_multiplier(gg, lo, up);
                const double dd = (double)mul_rn(invD2[G.ordAt[r]], sub_rn(gg, rr));
                v[2] += __dmul_rn(dd, dd);
                v[3] += (double)sub_rn(safeprod_left(up, pos_part(-rr)), safeprod_left(lo, neg_part(-rr)));
                v[4] += (double)mul_rn(cj, xb[G.baseAt + k + lane]);
            }
        }
    }
    __syncwarp();
    res_sum<5, CS, NT / 32>(v, sh, phase, W, (int)(threadIdx.x >> 5) < max(G.LA, G.LAt));
#pragma unroll
    for (int q = 0; q < 5; q++) out[q] = v[q];
}

// powm! iterations (linalg.jl:86-96) in FP64 over the stored values, from the
// vector px (loaded whole into every CTA): stops after an iteration whose
// residual is at most tol or rtol * theta, after iteration maxiter + 1 or after
// max_here iterations of this call.  it0 iterations ran before, the last with
// theta_prev.
// A chain of two products, two exchanges and the sums for theta and the scale
// bounds it.  So A'Ax is sent unscaled and the sums overlap its exchange and the
// next product with A, whose result takes the scale instead (a single CTA
// exchanges nothing and scales x first); three warps that
// (mostly) have no slices of A finish the sums.  The residual of an iteration
// needs its theta, so its norm is summed with the next iteration's theta: two
// products beyond the last iteration are dropped.  FP64 1,000 x 2,000 on 8 CTAs:
// a solve with 1,725 iterations 14.0 -> 12.8 ms; 128 LPs of up to 600 rows
// 38-42 -> 32-37 ms.
template <class T, int CS, int NT>
__device__ __noinline__ void res_power(const ResGeo& G, int64_t it0, int64_t max_here,
                                       int64_t maxiter, double tol, double rtol, double theta_prev,
                                       ResPower& P, double* sh, int& phase, ResWait& W,
                                       unsigned& parity_io) {
    constexpr int NW = NT / 32;
    static_assert(NW >= 3, "three warps finish the sums");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = G.rank;
    const int LA = G.LA, LAt = G.LAt, n = G.R.n;
    const T *valA = &sm_at<T>(G.o.valA) + lane, *valAt = &sm_at<T>(G.o.valAt) + lane;
    const uint16_t *idxA = &sm_at<uint16_t>(G.o.idxA) + lane, *idxAt = &sm_at<uint16_t>(G.o.idxAt) + lane;
    const uint32_t *offA = &sm_at<uint32_t>(G.o.offA), *offAt = &sm_at<uint32_t>(G.o.offAt);
    const uint8_t *lenA = &sm_at<uint8_t>(G.o.lenA) + lane, *lenAt = &sm_at<uint8_t>(G.o.lenAt) + lane;
    const double *px = &sm_at<double>(G.px), *ps = &sm_at<double>(G.ps);
    double *pxown = &sm_at<double>(G.px) + G.baseAt + lane, *psown = &sm_at<double>(G.ps) + G.baseA + lane;
    double* pax = &sm_at<double>(G.pax) + lane;  // own x, scaled
    unsigned parity = parity_io;
    double theta = theta_prev, residual = INFINITY, inv = 1.0;
    int64_t it = it0;
    bool stop = false;
    double r2 = 0.0;               // own part of the last iteration's residual^2
    const double* slot = nullptr;  // sums on their way
    bool pending = false;          // they hold an iteration's residual
    const int wa = (w + NW - LAt % NW) % NW;  // slices of A start after those of A'
    const int wq = NW - 1 - w;                // the last three warps finish the sums
    auto product = [&] {
#pragma unroll 1
        for (int l = wa; l < LA; l += NW) {
            const uint32_t o = offA[l];
            psown[l * 32] = slice_sum(idxA + (o >> 8) * 32, valA + (o >> 8) * 32, (int)(o & 255u),
                                      lenA[l * 32], px);
        }
    };
    auto rescale = [&] {
        r2 = 0.0;
#pragma unroll 1
        for (int l = w; l < LAt; l += NW) {
            const double ax = pxown[l * 32];
            if ((l * CS + rank) * 32 + lane < n) {
                const double rr = __fma_rn(-theta, pax[l * 32], ax);
                r2 = __fma_rn(rr, rr, r2);
            }
            pax[l * 32] = mul_rn(ax, inv);
        }
    };
    auto keep = [&] {
#pragma unroll 1
        for (int l = w; l < LAt; l += NW) pxown[l * 32] = pax[l * 32];
    };
#pragma unroll 1
    for (int l = w; l < LAt; l += NW) pax[l * 32] = pxown[l * 32];
    for (;;) {
        // theta, 1 / |A'Ax| and the residual of the iteration before (negative
        // when it ends the iteration)
        if (slot && wq < 3) {
            __syncwarp();
            if constexpr (CS > 1) res_wait<CS>();
            const double s = res_total<CS, NW>(slot, wq);
            double f = s;
            if (wq == 1) f = rsqrt(s);
            if (wq == 2) {
                const double res = sqrt(s);
                f = res <= tol || (rtol > 0 && res <= rtol * theta) ? -1.0 - res : res;
                if (s == -INFINITY) f = s;  // a wait ran out: all CTAs leave here
            }
            if (lane == 0) sh[wq] = f;
            __syncwarp();
        }
        if constexpr (CS > 1) {
            product();
            __syncwarp();
            if (slot && wq >= 3) res_wait<CS>();
        }
        __syncthreads();
        if (pending) {
            residual = sh[2];
            it++;
            stop = it > maxiter || __double_as_longlong(residual) < 0;
            if (stop || it - it0 >= max_here) break;
        }
        if (slot) {
            theta = sh[0];
            inv = sh[1];
        }
        if constexpr (CS > 1) {
#pragma unroll 1
            for (int l = wa; l < LA; l += NW) {
                psown[l * 32] = mul_rn(psown[l * 32], inv);
                res_send<CS>(psown + l * 32 - lane, &W.bar[0], rank);
            }
            if (slot) rescale();
        } else {
            if (slot) {
                rescale();
                keep();
                __syncthreads();
            }
            product();
        }
        pending = slot != nullptr;
        res_receive<CS>(W, 0, G.remA * 8u, parity);
        // (a sum of squares is never -inf; where it is no number already, the next
        // sums tell the group)
        double v[3] = {0.0, 0.0, CS > 1 && (parity & RES_GAVE_UP) ? -INFINITY : r2};
#pragma unroll 1
        for (int l = w; l < LAt; l += NW) {
            const uint32_t o = offAt[l];
            const double s = slice_sum(idxAt + (o >> 8) * 32, valAt + (o >> 8) * 32,
                                       (int)(o & 255u), lenAt[l * 32], ps);
            pxown[l * 32] = s;
            res_send<CS>(pxown + l * 32 - lane, &W.bar[1], rank);
            if ((l * CS + rank) * 32 + lane < n) {
                v[0] = __fma_rn(pax[l * 32], s, v[0]);
                v[1] = __fma_rn(s, s, v[1]);
            }
        }
        __syncwarp();
        double* put = res_slot<CS, NW>(sh, phase);
        res_partial<3, CS, NW>(v, put, w < LAt);
        slot = put;
        if constexpr (CS > 1) res_arrive<CS>();
        res_receive<CS>(W, 1, G.remAt * 8u, parity);
    }
    keep();
    if (CS > 1 && threadIdx.x == 0 && residual == -INFINITY) W.failed = 1;
    if (__double_as_longlong(residual) < 0) residual = -1.0 - residual;
    P.theta = theta;
    P.residual = residual;
    P.it = it;
    P.stop = stop;
    parity_io = parity;
    res_sync<CS>();
}

}  // namespace cpdlp
