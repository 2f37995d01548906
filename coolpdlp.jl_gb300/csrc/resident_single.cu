// resident_single.cu -- one small LP on the resident kernels: a launch runs a
// whole block of steps and the KKT evaluation of its four iterates, where the
// tile engine has two kernels a step (8 us a step for 10,000 nonzeros in FP64,
// against 3.5 us here), and a launch runs the power method, seven kernels an
// iteration there (23 us).  Restart and termination stay on the host.
#include "resident.cuh"

namespace cpdlp {

namespace {

constexpr int RS_NT = 512;

template <class T>
struct BlockArgs {
    ResView<T> v;
    ResLP lp;
    ResBlock<T> b;
    const T *c, *lv, *uv, *lc, *uc, *invD1, *invD2;
};

template <class T, int CS>
__global__ void __launch_bounds__(RS_NT) k_res_block(const __grid_constant__ BlockArgs<T> g) {
    __shared__ double sh[res_sh<CS, RS_NT / 32>()];
    __shared__ ResCoefs<T> tab;
    __shared__ ResGeo G;
    __shared__ ResWait W;
    unsigned parity = 0;
    int phase = 0;
    if (threadIdx.x == 0) {
        res_wait_init(W);
        tab.es = g.b.eta_sum;
    }
    res_load<T, CS, RS_NT>(G, g.lp, g.v);
    res_bounds<T, CS, RS_NT>(G, g.c, g.lv, g.uv, g.lc, g.uc);
    res_load_iterate<T, CS, RS_NT>(G, g.b.x, g.b.avg ? g.b.xa : nullptr, g.b.y,
                                   g.b.avg ? g.b.ya : nullptr);
    res_sync<CS>();  // every CTA has read the buffers that the last step overwrites
    const ResDump<T> d{g.b.to.x, g.b.to.xl, g.b.to.xa, g.b.to.xal, g.b.to.y, g.b.to.yl, g.b.to.ya, g.b.to.yal};
    res_steps<T, CS, RS_NT>(G, g.b.eta, g.b.omega, g.b.steps, g.b.avg != 0, tab, d, W, parity);
    for (int p = 0; p < g.b.nv; p++) {
        double v[5];
        res_kkt_sums<T, CS, RS_NT>(G, p == 0 ? d.x : p == 1 ? d.xa : p == 2 ? d.xl : d.xal,
                                   p == 0 ? d.y : p == 1 ? d.ya : p == 2 ? d.yl : d.yal, g.invD1,
                                   g.invD2, v, sh, phase, W);
        if (G.rank == 0 && threadIdx.x == 0)
            for (int q = 0; q < 5; q++) g.b.out[5 * p + q] = v[q];
    }
    if (threadIdx.x == 0 && (G.rank == 0 || W.failed)) {
        if (W.failed) g.b.out[20] = 1.0;
        __threadfence_system();
    }
    res_sync<CS>();  // no CTA exits while another may write its shared memory
}

template <class T>
struct PowerArgs1 {
    ResView<T> v;
    ResLP lp;
    double *x, *out;
    int64_t it0, max_here, maxiter;
    double tol, rtol, theta_prev;
};
template <class T, int CS>
__global__ void __launch_bounds__(RS_NT) k_res_power(const __grid_constant__ PowerArgs1<T> g) {
    __shared__ double sh[res_sh<CS, RS_NT / 32>()];
    __shared__ ResGeo G;
    __shared__ ResWait W;
    unsigned parity = 0;
    int phase = 0;
    if (threadIdx.x == 0) res_wait_init(W);
    res_load<T, CS, RS_NT>(G, g.lp, g.v);
    double* px = &sm_at<double>(G.px);
    for (int j = threadIdx.x; j < G.R.n; j += RS_NT) px[G.invAt[j]] = __ldcg(g.x + j);
    res_sync<CS>();
    ResPower P;
    res_power<T, CS, RS_NT>(G, g.it0, g.max_here, g.maxiter, g.tol, g.rtol, g.theta_prev, P, sh, phase,
                            W, parity);
    res_rows<CS, RS_NT>(G.LAt, G.rank, G.R.n, [&](int k, int r) { g.x[G.ordAt[r]] = px[G.baseAt + k]; });
    if (threadIdx.x == 0 && (G.rank == 0 || W.failed)) {
        if (G.rank == 0) {
            g.out[0] = P.theta;
            g.out[1] = P.residual;
            g.out[2] = (double)P.it;
            g.out[3] = P.stop ? 1.0 : 0.0;
        }
        if (W.failed) g.out[4] = 1.0;
        __threadfence_system();
    }
    res_sync<CS>();
}

template <class K, class A>
void launch_group(K kern, int cs, uint32_t smem, const A& args, cudaStream_t s) {
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RES_MAX_SMEM));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cs);
    cfg.blockDim = dim3(RS_NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = cs > 1 ? 1 : 0;
    CK(cudaLaunchKernelEx(&cfg, kern, args));
}

}  // namespace

template <class T>
void res_single_build(ProblemT<T>& P, const std::vector<int32_t>& hpA,
                      const std::vector<int32_t>& hpAt, cudaStream_t s) {
    std::vector<int32_t> mA, mAt;
    ResLP r{};
    if (res_plan(hpA.data(), hpAt.data(), P.m, P.n, P.nnz, (int)sizeof(T), true, r, mA, mAt) == 0) return;
    const size_t eA = 32 * (size_t)mA[(size_t)r.cs], eAt = 32 * (size_t)mAt[(size_t)r.cs];
    ResStore<T>& st = P.res;
    st.idxA.alloc(eA);
    st.idxAt.alloc(eAt);
    st.valA.alloc(eA);
    st.valAt.alloc(eAt);
    st.metaA.alloc(mA.size());
    st.metaAt.alloc(mAt.size());
    st.ordA.alloc((size_t)P.m);
    st.ordAt.alloc((size_t)P.n);
    st.invA.alloc((size_t)P.m);
    st.invAt.alloc((size_t)P.n);
    st.lenA.alloc((size_t)P.m);
    st.lenAt.alloc((size_t)P.n);
    DBuf<ResLP> d(1);
    CK(cudaMemcpyAsync(st.metaA.p, mA.data(), sizeof(int32_t) * mA.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(st.metaAt.p, mAt.data(), sizeof(int32_t) * mAt.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(d.p, &r, sizeof(ResLP), cudaMemcpyHostToDevice, s));
    res_build<T>(st, d.p, 1, P.a_ptr.p, P.a_idx.p, P.a_val.p, P.at_ptr.p, P.at_idx.p, P.at_val.p,
                 std::max(P.m, P.n), s);
    P.rlp = r;
}

template <class T>
void res_single_block(const ProblemT<T>& P, const ResBlock<T>& b, cudaStream_t s) {
    const BlockArgs<T> a{res_view(P.res), P.rlp, b, P.c.p, P.lv.p, P.uv.p, P.lc.p, P.uc.p,
                         P.invD1_T(), P.invD2_T()};
    const uint32_t smem = res_layout<T>(P.rlp).total;
    switch (P.rlp.cs) {
        case 1: launch_group(k_res_block<T, 1>, 1, smem, a, s); break;
        case 2: launch_group(k_res_block<T, 2>, 2, smem, a, s); break;
        case 4: launch_group(k_res_block<T, 4>, 4, smem, a, s); break;
        default: launch_group(k_res_block<T, 8>, 8, smem, a, s); break;
    }
}

template <class T>
void res_single_power(const ProblemT<T>& P, double* x, int64_t it0, int64_t max_here,
                      int64_t maxiter, double tol, double rtol, double theta_prev, double* out,
                      cudaStream_t s) {
    const PowerArgs1<T> a{res_view(P.res), P.rlp, x, out, it0, max_here, maxiter, tol, rtol, theta_prev};
    const uint32_t smem = res_layout<T>(P.rlp).total;
    switch (P.rlp.cs) {
        case 1: launch_group(k_res_power<T, 1>, 1, smem, a, s); break;
        case 2: launch_group(k_res_power<T, 2>, 2, smem, a, s); break;
        case 4: launch_group(k_res_power<T, 4>, 4, smem, a, s); break;
        default: launch_group(k_res_power<T, 8>, 8, smem, a, s); break;
    }
}

template void res_single_build<float>(ProblemT<float>&, const std::vector<int32_t>&,
                                      const std::vector<int32_t>&, cudaStream_t);
template void res_single_build<double>(ProblemT<double>&, const std::vector<int32_t>&,
                                       const std::vector<int32_t>&, cudaStream_t);
template void res_single_block<float>(const ProblemT<float>&, const ResBlock<float>&, cudaStream_t);
template void res_single_block<double>(const ProblemT<double>&, const ResBlock<double>&, cudaStream_t);
template void res_single_power<float>(const ProblemT<float>&, double*, int64_t, int64_t, int64_t,
                                      double, double, double, double*, cudaStream_t);
template void res_single_power<double>(const ProblemT<double>&, double*, int64_t, int64_t, int64_t,
                                       double, double, double, double*, cudaStream_t);

}  // namespace cpdlp
