// Device pieces shared by the launch-per-phase Krylov solvers (krylov.cu, separable.cu):
// the operators, the deterministic fused reduction and the status rule.
#pragma once
#include "operators.cuh"
#include "solver.h"

namespace cuibm {

// ---- operators seen by the solver -------------------------------------------
struct Op1 {
    Lhs1Coef c;
    Grid g;
    const double *w;  // symmetrisation weights or nullptr
    template <class X>
    __device__ __forceinline__ double row(int i, const X &x) const
    {
        double y = lhs1_row_f(c, g, i, x);
        return w ? w[i] * y : y;
    }
};
struct Op2 {
    Lhs2Coef c;
    Grid g;
    const double *w;
    template <class X>
    __device__ __forceinline__ double row(int i, const X &x) const
    {
        double y = lhs2_row_f(c, g, i, x);
        return w ? w[i] * y : y;
    }
};

struct ScaledAccess {
    const double *__restrict__ p, *__restrict__ d;
    __device__ __forceinline__ double operator()(int j) const { return p[j] * d[j]; }
};

// ---- deterministic fused reduction --------------------------------------------
template <int NV>
__device__ __forceinline__ bool reduce_arrive(double (&v)[NV], double *partials, unsigned int *arrive,
                                              double (&tot)[NV])
{
    __shared__ double sh[NV][32];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double a = v[k];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sh[k][wid] = a;
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double a = lane < nw ? sh[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
            if (lane == 0) partials[blockIdx.x * 4 + k] = a;
        }
    }
    __threadfence();
    if (threadIdx.x == 0) is_last = (atomicAdd(arrive, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    // fixed-order sum of the per-block partials
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double a = 0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) a += __ldcg(partials + b * 4 + k);
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sh[k][wid] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double a = 0;
        for (int q = 0; q < nw; ++q) a += sh[k][q];
        tot[k] = a;
    }
    if (threadIdx.x == 0) *arrive = 0;
    return true;
}

__device__ __forceinline__ void set_cond(cudaGraphConditionalHandle h, int use, unsigned int v)
{
    if (use) cudaGraphSetConditional(h, v);
}

__device__ __forceinline__ void finish_status(KrylovScalars *ks, int *err_word, int which)
{
    if (ks->status == KS_RUNNING) {
        // a non-finite residual or right-hand side (an overflowed field passes
        // ||r|| <= tol ||b|| as inf <= inf) is reported, not taken as convergence
        if (!isfinite(ks->rnorm) || !isfinite(ks->tol)) ks->status = KS_NAN;
        else if (ks->rnorm <= ks->tol) ks->status = KS_CONVERGED;
        else if (ks->it >= ks->maxit) ks->status = KS_MAXIT;
    }
    if ((ks->status == KS_MAXIT || ks->status == KS_NAN) && err_word && *err_word == 0)
        *err_word = which * 16 + ks->status;
}

// ---- kernels of both launchers ---------------------------------------------------
static __global__ void __launch_bounds__(256) k_bicg_5(int n, double *p, const double *__restrict__ r,
                                                const double *__restrict__ AMp, const KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = r[i] + ks->beta * (p[i] - ks->omega * AMp[i]);
}

// ---- CG on the symmetrised system -------------------------------------------------
template <class Op, int PC>
__global__ void __launch_bounds__(256) k_cg_init(Op A, int n, const double *__restrict__ b,
                                                 const double *__restrict__ w, const double *x, double *r,
                                                 double *z, double *p, const double *__restrict__ dinv,
                                                 double *partials, KrylovScalars *ks, int *err, int which,
                                                 cudaGraphConditionalHandle h, int use_cond)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[3] = {0, 0, 0};
    if (i < n) {
        double bi = b[i], ri = w[i] * bi - A.row(i, PtrAccess{x});
        r[i] = ri;
        double ro = ri / w[i];
        v[0] = ro * ro;
        v[1] = bi * bi;
        if (PC != 2) {
            double zi = PC == 1 ? ri * dinv[i] : ri;
            z[i] = zi;
            p[i] = zi;
            v[2] = ri * zi;
        }
    }
    double t[3];
    if (reduce_arrive<3>(v, partials, &ks->arrive, t) && threadIdx.x == 0) {
        ks->rnorm = sqrt(t[0]);
        ks->bnorm = sqrt(t[1]);
        ks->rho = t[2];
        ks->tol = ks->rtol * ks->bnorm;
        ks->it = 0;
        ks->body_runs = 0;
        ks->status = KS_RUNNING;
        finish_status(ks, err, which);
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

template <class Op>
__global__ void __launch_bounds__(256) k_cg_1(Op A, int n, const double *p, double *q, double *partials,
                                              KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[1] = {0};
    if (i < n) {
        double qi = A.row(i, PtrAccess{p});
        q[i] = qi;
        v[0] = p[i] * qi;
    }
    double t[1];
    if (reduce_arrive<1>(v, partials, &ks->arrive, t) && threadIdx.x == 0) {
        ks->alpha = ks->rho / t[0];
        ks->body_runs += 1;
    }
}

// x += alpha p; r -= alpha q; (PC<2) z = M r and r.z; residual norm of the original system
template <int PC>
__global__ void __launch_bounds__(256) k_cg_2(int n, double *x, double *r, double *z, const double *__restrict__ p,
                                              const double *__restrict__ q, const double *__restrict__ w,
                                              const double *__restrict__ dinv, double *partials,
                                              KrylovScalars *ks, int *err, int which,
                                              cudaGraphConditionalHandle h, int use_cond)
{
    if (ks->status != KS_RUNNING) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double alpha = ks->alpha;
    double v[2] = {0, 0};
    if (i < n) {
        x[i] += alpha * p[i];
        double ri = r[i] - alpha * q[i];
        r[i] = ri;
        double ro = ri / w[i];
        v[0] = ro * ro;
        if (PC != 2) {
            double zi = PC == 1 ? ri * dinv[i] : ri;
            z[i] = zi;
            v[1] = ri * zi;
        }
    }
    double t[2];
    if (reduce_arrive<2>(v, partials, &ks->arrive, t) && threadIdx.x == 0) {
        ks->it += 1;
        ks->rnorm = sqrt(t[0]);
        if (PC != 2) {
            ks->beta = t[1] / ks->rho;
            ks->rho = t[1];
        }
        finish_status(ks, err, which);
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

// external preconditioner: rho_new = r.z, beta (first=1: p = z, rho = r.z)
static __global__ void __launch_bounds__(256) k_cg_rz(int n, const double *__restrict__ r, const double *__restrict__ z,
                                               double *partials, KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[1] = {0};
    if (i < n) v[0] = r[i] * z[i];
    double t[1];
    if (reduce_arrive<1>(v, partials, &ks->arrive, t) && threadIdx.x == 0) {
        ks->beta = ks->it == 0 ? 0.0 : t[0] / ks->rho;
        ks->rho = t[0];
    }
}

static __global__ void __launch_bounds__(256) k_cg_3(int n, double *p, const double *__restrict__ z,
                                              const KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = ks->it == 0 ? z[i] : z[i] + ks->beta * p[i];
}

// ---- host side ------------------------------------------------------------------
inline Op1 op1(Context &c, const double *w) { return Op1{c.l1, c.g, w}; }
inline Op2 op2(Context &c, const double *w) { return Op2{c.l2, c.g, w}; }

// A conditional node after what c.stream has captured so far; its handle's value is 0 at
// each launch of the graph.  make() creates the handle before the kernels that set it.
struct CondNode {
    Context &c;
    cudaGraphConditionalHandle h{};

    explicit CondNode(Context &c_) : c(c_)
    {
        cudaStreamCaptureStatus st;
        cudaGraph_t graph;
        CUIBM_TRY(cudaStreamGetCaptureInfo(c.stream, &st, nullptr, &graph, nullptr, nullptr, nullptr));
        CUIBM_TRY(cudaGraphConditionalHandleCreate(&h, graph, 0, cudaGraphCondAssignDefault));
    }
    template <class F>
    int add(cudaGraphConditionalNodeType type, const F &body)
    {
        cudaStreamCaptureStatus st;
        cudaGraph_t graph;
        const cudaGraphNode_t *deps = nullptr;
        size_t ndeps = 0;
        CUIBM_TRY(cudaStreamGetCaptureInfo(c.stream, &st, nullptr, &graph, &deps, nullptr, &ndeps));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = type;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        CUIBM_TRY(cudaGraphAddNode(&node, graph, deps, nullptr, ndeps, &cp));
        cudaStream_t main = c.stream, side = c.side_stream;
        CUIBM_TRY(cudaStreamBeginCaptureToGraph(side, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                cudaStreamCaptureModeRelaxed));
        c.stream = side;
        try {
            body();
        } catch (...) {
            c.stream = main;
            cudaGraph_t dummy;
            cudaStreamEndCapture(side, &dummy);
            throw;
        }
        c.stream = main;
        cudaGraph_t got;
        CUIBM_TRY(cudaStreamEndCapture(side, &got));
        CUIBM_TRY(cudaStreamUpdateCaptureDependencies(c.stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
        return count_kernel_nodes(got);
    }
};

}  // namespace cuibm
