// sgipc_pcg.cu — symmetric block SpMV and MAS-preconditioned conjugate gradients.
//
// Algorithm of PCGSolver::pcg (StiffGIPC/linear_system/solver/pcg_solver.cu:174-267):
//   r = b, z = M r, p = z, rz0 = rz = r.z
//   for k = 1 .. max_iter-1:
//     Ap = A p; alpha = rz / p.Ap; x += alpha p; r -= alpha Ap
//     if |rz| <= tol * rz0: break          (tested on the rz from before the update)
//     z = M r; rz_new = r.z; p = z + (rz_new / rz) p; rz = rz_new
// The reference does each dot with a two-pass reduction and a blocking cudaMemcpy (two
// host round trips per iteration).  Here every scalar stays in device memory, each
// reduction finishes in the kernel's last CTA, and the whole loop is one CUDA graph whose
// while-node condition is set on the device — one launch per solve.
//
// One iteration is four kernels (T = vector type, M = MAS type, NR = right-hand sides):
//   K1 spmv_dot   p = z + beta p_old formed on the fly (ping-pong buffers), Ap = A p over
//                 the full symmetric static CSR plus the unique contact blocks, p.Ap;
//                 last CTA: rz, alpha, the r.z stop test
//   K2 update     x += alpha p, r -= alpha Ap, restriction of r to MAS levels 0 and 1
//                 (bank-local, no atomics); last CTA: ||r||^2, the true-residual stop test
//   K3 domains    CTA 0 restricts r to the coarse levels and solves their domains, the
//                 other CTAs solve the level-0/1 domains Z_d = A_d^-1 R_d
//   K4 prolong    z = sum_l Z (gather), r.z; its first thread decides whether the graph
//                 runs another body (stop state, iteration cap, body bound) and sets the
//                 while-node condition; later bodies return at once once `halt` is set.
#include <cstdlib>
#include <cub/cub.cuh>
#include <vector>

#include "sgipc_internal.cuh"
#include "sgipc_mas_dev.cuh"
#include "sgipc_pcg_dev.cuh"

using namespace sgipc;

namespace sgipc {

// Publishes this CTA's partial sums; returns true in every thread of the last CTA to
// arrive, after which out[r] holds the deterministic (CTA-order) total.  Every CTA of the
// grid must call it (the early returns before it are grid-uniform).
template <int NR>
__device__ __forceinline__ bool grid_sum(double (&v)[NR], double* partial, unsigned int* ticket, double* out,
                                         double* smem) {
    block_sum<NR>(v, smem);
    __shared__ bool last;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) partial[r * gridDim.x + blockIdx.x] = v[r];
        __threadfence();
        unsigned int t = atomicAdd(ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        acc[r] = 0;
        for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x)
            acc[r] += ((volatile double*)partial)[r * gridDim.x + k];
    }
    block_sum<NR>(acc, smem);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) out[r] = acc[r];
        *ticket = 0;
    }
    __syncthreads();
    return true;
}

template <class T>
__global__ void k_spmv(Topo tp, MatView<T> A, const T* __restrict__ x, T* __restrict__ y) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t / kSpG, g = t % kSpG;
    Operand<T, 1> op;
    op.a = x;
    op.b = nullptr;
    op.beta[0] = 0;
    T acc[1][3];
    row_mv<T, 1>(tp, A, op, i, g, acc);
    if (i < tp.n && g == 0) {
        y[3 * i] = acc[0][0];
        y[3 * i + 1] = acc[0][1];
        y[3 * i + 2] = acc[0][2];
    }
}

// ---- PCG kernels ----------------------------------------------------------------------------
template <class T, int NR>
struct PcgPtrs {
    T* x;
    T* r;
    T* z;
    T* p[2];
    T* Ap;
    PcgScalars* sc;
    double* partial;
    unsigned int* ticket;
};

// K1
template <class T, int NR>
__global__ void __launch_bounds__(256) k_pcg_spmv_dot(Topo tp, MatView<T> A, PcgPtrs<T, NR> P) {
    __shared__ double smem[NR * 32];
    __shared__ int run[NR];
    __shared__ double beta[NR];
    __shared__ int halt, nb;
    if (threadIdx.x < NR) {
        const PcgScalars& s = P.sc[threadIdx.x];
        run[threadIdx.x] = s.state == 0;
        beta[threadIdx.x] = s.first ? 0.0 : s.rz_next / s.rz;
    }
    if (threadIdx.x == 0) {
        halt = P.sc[0].halt;
        // this iteration's direction buffer: the running right-hand sides have all done the
        // same number of iterations
        nb = 0;
        for (int r = NR - 1; r >= 0; r--)
            if (P.sc[r].state == 0) nb = P.sc[r].iter & 1;
    }
    __syncthreads();
    bool any = false;
#pragma unroll
    for (int r = 0; r < NR; r++) any |= run[r] != 0;
    // grid-uniform: these words change only in this kernel's last CTA, after every CTA has
    // read them, or in later kernels
    if (!any || halt) return;
    // rows of finished right-hand sides are computed too (cheaper than masking) and ignored
    Operand<T, NR> op;
    op.a = P.z;
    op.b = nb ? P.p[0] : P.p[1];
#pragma unroll
    for (int r = 0; r < NR; r++) op.beta[r] = (T)beta[r];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t / kSpG, g = t % kSpG;
    double part[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) part[r] = 0.0;
    T acc[NR][3];
    row_mv<T, NR>(tp, A, op, i, g, acc);
    if (i < tp.n && g == 0) {
        T* pw = nb ? P.p[1] : P.p[0];
        T pi[NR][3];
        op.load(i, pi);
#pragma unroll
        for (int r = 0; r < NR; r++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const size_t k = (size_t)(3 * i + q) * NR + r;
                if (run[r]) {
                    pw[k] = pi[r][q];
                    P.Ap[k] = acc[r][q];
                }
                part[r] += (double)pi[r][q] * (double)acc[r][q];
            }
    }
    double tot[NR];
    if (grid_sum<NR>(part, P.partial, P.ticket, tot, smem) && threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            PcgScalars& s = P.sc[r];
            if (!run[r]) continue;
            s.rz = s.rz_next;
            s.pAp = tot[r];
            s.pcur = nb;
            s.first = 0;
            s.iter += 1;
            if (!(tot[r] > 0.0) || !isfinite(tot[r]) || !isfinite(s.rz)) {
                s.state = 2;
                s.status = SGIPC_BREAKDOWN;
                continue;
            }
            s.alpha = s.rz / tot[r];
            if (s.crit == SGIPC_CRIT_RZ && fabs(s.rz) <= s.tol * s.rz0) s.state = 1;
        }
    }
}

// K2: one thread per MAS position (16-lane banks), so that the restriction of the updated
// residual to levels 0 and 1 is a bank-local reduction with plain stores
template <class T, class M, int NR>
__global__ void __launch_bounds__(256) k_pcg_update(PcgPtrs<T, NR> P, MasView mv, M* __restrict__ R) {
    __shared__ double smem[NR * 32];
    __shared__ int st[NR];
    __shared__ int pc[NR];
    __shared__ double alpha[NR];
    __shared__ int halt;
    if (threadIdx.x < NR) {
        st[threadIdx.x] = P.sc[threadIdx.x].state;
        alpha[threadIdx.x] = P.sc[threadIdx.x].alpha;
        pc[threadIdx.x] = P.sc[threadIdx.x].pcur;
    }
    if (threadIdx.x == 0) halt = P.sc[0].halt;
    __syncthreads();
    bool any = false;
#pragma unroll
    for (int r = 0; r < NR; r++) any |= st[r] < 2;
    if (!any || halt) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = p < mv.npos ? mv.part_map[p] : -1;
    double part[NR];
    M val[NR * 3];
#pragma unroll
    for (int r = 0; r < NR; r++) part[r] = 0.0;
#pragma unroll
    for (int k = 0; k < NR * 3; k++) val[k] = 0;
    if (v >= 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if (st[r] == 2) continue;
            const T a = (T)alpha[r];
            const T* pr = pc[r] ? P.p[1] : P.p[0];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const size_t k = (size_t)(3 * v + q) * NR + r;
                P.x[k] += a * pr[k];
                T rv = P.r[k] - a * P.Ap[k];
                P.r[k] = rv;
                part[r] += (double)rv * (double)rv;
                if (st[r] == 0) val[r * 3 + q] = (M)rv;
            }
        }
    }
    if (p < mv.npos)
#pragma unroll
        for (int q = 0; q < 3; q++)
#pragma unroll
            for (int r = 0; r < NR; r++) R[(size_t)(3 * p + q) * NR + r] = val[r * 3 + q];
    bank_reduce_store<M, NR>(v >= 0 ? mv.up[p] : -1, val, R);
    double tot[NR];
    if (grid_sum<NR>(part, P.partial + NR * gridDim.x, P.ticket + 1, tot, smem) && threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            PcgScalars& s = P.sc[r];
            if (st[r] == 2) continue;
            s.rr = tot[r];
            if (st[r] == 1) s.state = 2;  // the final update of an r.z-converged solve is applied
            else if (s.crit == SGIPC_CRIT_TRUE && tot[r] <= s.tol * s.tol * s.bnorm2) s.state = 2;
        }
    }
}

// K3: CTA 0 restricts to levels 2.. and solves the coarse domains; CTAs >= 1 take four
// level-0/1 domains each (48 threads per domain, Z_d = A_d^-1 R_d read once for NR columns)
template <class M, int NR>
__device__ __forceinline__ void domain_solve(const M* __restrict__ inv, const M* __restrict__ R, M* __restrict__ Z,
                                             int d, int i, M (*sR)[48 * NR]) {
    const M* Ad = inv + (size_t)d * 2304;
    M acc[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) acc[r] = 0;
#pragma unroll 4
    for (int j = 0; j < 48; j++) {
        M a = Ad[j * 48 + i];
#pragma unroll
        for (int r = 0; r < NR; r++) acc[r] += a * (*sR)[j * NR + r];
    }
#pragma unroll
    for (int r = 0; r < NR; r++) Z[(48 * (size_t)d + i) * NR + r] = acc[r];
}

template <class M, int NR>
__global__ void __launch_bounds__(192) k_pcg_domains(MasView mv, const PcgScalars* __restrict__ sc,
                                                     const M* __restrict__ inv, M* __restrict__ R, M* __restrict__ Z) {
    __shared__ M sR[4][48 * NR];
    __shared__ int go;
    if (threadIdx.x == 0) {
        int a = 0;
        for (int r = 0; r < NR; r++) a |= sc[r].state == 0;
        go = a && !sc[0].halt;
    }
    __syncthreads();
    if (!go) return;
    const int ld = threadIdx.x / 48, i = threadIdx.x % 48;
    const int ndom = mv.info[16] >> 4;
    const int nd01 = mv.L > 2 ? (mv.info[2] >> 4) : ndom;  // domains of levels 0 and 1
    if (blockIdx.x == 0) {
        restrict_coarse_cta<M, NR>(mv.info, mv.up, mv.L, R);
        for (int d0 = nd01; d0 < ndom; d0 += 4) {
            const int d = d0 + ld;
            if (d < ndom)
#pragma unroll
                for (int r = 0; r < NR; r++) sR[ld][i * NR + r] = R[(48 * (size_t)d + i) * NR + r];
            __syncthreads();
            if (d < ndom) domain_solve<M, NR>(inv, R, Z, d, i, &sR[ld]);
            __syncthreads();
        }
        return;
    }
    const int d = (blockIdx.x - 1) * 4 + ld;
    if (d < nd01)
#pragma unroll
        for (int r = 0; r < NR; r++) sR[ld][i * NR + r] = R[(48 * (size_t)d + i) * NR + r];
    __syncthreads();
    if (d < nd01) domain_solve<M, NR>(inv, R, Z, d, i, &sR[ld]);
}

// K4
template <class T, class M, int NR>
__global__ void __launch_bounds__(256) k_pcg_prolong_dot(int nv, PcgPtrs<T, NR> P, MasView mv,
                                                         const M* __restrict__ Z, cudaGraphConditionalHandle h,
                                                         int decide, int use_cond) {
    __shared__ double smem[NR * 32];
    __shared__ int run[NR];
    if (threadIdx.x < NR) run[threadIdx.x] = P.sc[threadIdx.x].state == 0;
    if (decide && blockIdx.x == 0 && threadIdx.x == 0) {
        // continuation of the iteration loop; reads only words final for this body
        PcgScalars& s0 = P.sc[0];
        int cont = 0;
        for (int r = 0; r < NR; r++) {
            const PcgScalars& s = P.sc[r];
            if (s.state == 0 && s.iter + 1 < s.max_iter) cont = 1;
        }
        s0.bodies += 1;
        if (s0.bodies >= s0.max_iter + 2) cont = 0;
        if (!cont) s0.halt = 1;
        if (use_cond) cudaGraphSetConditional(h, cont);
    }
    __syncthreads();
    bool any = false;
#pragma unroll
    for (int r = 0; r < NR; r++) any |= run[r] != 0;
    if (!any) return;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    double part[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) part[r] = 0.0;
    if (v < nv) {
        const int* tv = mv.table + (size_t)v * mv.L;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if (!run[r]) continue;
            M a0 = 0, a1 = 0, a2 = 0;
            for (int l = 0; l < mv.L; l++) {
                int g = tv[l];
                a0 += Z[(size_t)(3 * g) * NR + r];
                a1 += Z[(size_t)(3 * g + 1) * NR + r];
                a2 += Z[(size_t)(3 * g + 2) * NR + r];
            }
            T zz[3] = {(T)a0, (T)a1, (T)a2};
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const size_t k = (size_t)(3 * v + q) * NR + r;
                P.z[k] = zz[q];
                part[r] += (double)P.r[k] * (double)zz[q];
            }
        }
    }
    double tot[NR];
    if (grid_sum<NR>(part, P.partial + 2 * NR * gridDim.x, P.ticket + 2, tot, smem) && threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (run[r]) P.sc[r].rz_next = tot[r];
    }
}

// ---- solve set-up kernels -------------------------------------------------------------------
template <class T, class M, int NR>
__global__ void k_pcg_init(const double* __restrict__ b, PcgPtrs<T, NR> P, MasView mv, M* __restrict__ R, double tol,
                           int max_iter, int crit) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < NR) {
        PcgScalars& s = P.sc[p];
        s.state = 0;
        s.status = SGIPC_OK;
        s.iter = 0;
        s.bodies = 0;
        s.first = 1;
        s.pcur = 0;
        s.halt = 0;
        s.tol = tol;
        s.max_iter = max_iter;
        s.crit = crit;
    }
    const int v = p < mv.npos ? mv.part_map[p] : -1;
    M val[NR * 3];
#pragma unroll
    for (int k = 0; k < NR * 3; k++) val[k] = 0;
    if (v >= 0) {
#pragma unroll
        for (int r = 0; r < NR; r++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const size_t k = (size_t)(3 * v + q) * NR + r;
                T rv = (T)b[k];
                P.r[k] = rv;
                P.x[k] = 0;
                P.p[0][k] = 0;
                P.p[1][k] = 0;
                val[r * 3 + q] = (M)rv;
            }
    }
    if (p < mv.npos)
#pragma unroll
        for (int q = 0; q < 3; q++)
#pragma unroll
            for (int r = 0; r < NR; r++) R[(size_t)(3 * p + q) * NR + r] = val[r * 3 + q];
    bank_reduce_store<M, NR>(v >= 0 ? mv.up[p] : -1, val, R);
}

template <class T, int NR>
__global__ void k_pcg_init_finish(int n3, const double* __restrict__ b, PcgPtrs<T, NR> P) {
    __shared__ double smem[NR * 32];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double part[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        part[r] = 0.0;
        if (k < n3) {
            const size_t e = (size_t)k * NR + r;
            part[r] = b[e] * b[e];
        }
    }
    double tot[NR];
    if (grid_sum<NR>(part, P.partial + 3 * NR * gridDim.x, P.ticket + 3, tot, smem) && threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
            PcgScalars& s = P.sc[r];
            s.rz0 = s.rz = s.rz_next;
            s.bnorm2 = tot[r];
            s.rr = tot[r];
            if (!(s.rz0 > 0.0) || !isfinite(s.rz0)) {
                // b = 0 (or an indefinite preconditioner): nothing to iterate
                s.state = 2;
                if (!isfinite(s.rz0) || s.rz0 < 0.0) s.status = SGIPC_BREAKDOWN;
            }
        }
    }
}

// ---- dot products and vector helpers --------------------------------------------------------
__global__ void k_dot(int n, const double* __restrict__ a, const double* __restrict__ b, double* partial,
                      unsigned int* ticket, double* out) {
    __shared__ double smem[32];
    double v[1] = {0.0};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) v[0] += a[k] * b[k];
    double tot[1];
    if (grid_sum<1>(v, partial, ticket, tot, smem) && threadIdx.x == 0) out[0] = tot[0];
}

__global__ void k_axpby_res(int n, const double* __restrict__ b, const double* __restrict__ Ax, double* __restrict__ r) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) r[k] = b[k] - Ax[k];
}

// x += d, or x = d (assign: the first refinement, x not read)
__global__ void k_add_f32(int n, const float* __restrict__ d, double* __restrict__ x, int assign) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) x[k] = (assign ? 0.0 : x[k]) + (double)d[k];
}

// rhs-major [nrhs][n3] <-> interleaved [n3][nrhs]
template <class A, class B>
__global__ void k_interleave(int n3, int nrhs, const A* __restrict__ src, B* __restrict__ dst, int to_interleaved) {
    long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (long long)n3 * nrhs) return;
    int r = (int)(k / n3), i = (int)(k % n3);
    if (to_interleaved)
        dst[(size_t)i * nrhs + r] = (B)src[k];
    else
        dst[k] = (B)src[(size_t)i * nrhs + r];
}

}  // namespace sgipc

// --------------------------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------------------------
namespace {

template <class T, int NR>
PcgPtrs<T, NR> ptrs_of(PcgWork& w) {
    PcgPtrs<T, NR> P;
    P.x = (T*)w.x;
    P.r = (T*)w.r;
    P.z = (T*)w.z;
    P.p[0] = (T*)w.p;
    P.p[1] = (T*)w.p2;
    P.Ap = (T*)w.Ap;
    P.sc = w.sc;
    P.partial = w.partial;
    P.ticket = w.ticket;
    return P;
}

// grid of K3: one coarse CTA + the level-0/1 domains, four per CTA
int domain_grid(SgipcCtx* c) {
    const int* h = c->mas.h_info;
    const int ndom = h[16] / 16;
    const int nd01 = c->mas.levelnum > 2 ? h[2] / 16 : ndom;
    return 1 + (nd01 + 3) / 4;
}

template <class T, class M, int NR>
void enqueue_body(SgipcCtx* c, PcgWork& w, const M* inv, M* R, M* Z, cudaGraphConditionalHandle h, int use_cond,
                  int k3grid, cudaStream_t s) {
    const int n = c->n, nv = c->nv;
    PcgPtrs<T, NR> P = ptrs_of<T, NR>(w);
    MasView mv = mas_view(c);
    k_pcg_spmv_dot<T, NR><<<spmv_grid(n), 256, 0, s>>>(topo_of(c), mat_view<T>(c), P);
    k_pcg_update<T, M, NR><<<nblk(mv.npos), 256, 0, s>>>(P, mv, R);
    k_pcg_domains<M, NR><<<k3grid, 192, 0, s>>>(mv, w.sc, inv, R, Z);
    k_pcg_prolong_dot<T, M, NR><<<nblk(nv), 256, 0, s>>>(nv, P, mv, Z, h, 1, use_cond);
}

// Build (or reuse) the executable graph of the iteration loop for this workspace.
template <class T, class M, int NR>
SgipcStatus get_loop_graph(SgipcCtx* c, PcgWork& w, const M* inv, M* R, M* Z, int k3grid, int tag) {
    const long long key = (long long)tag * 100000000LL + k3grid;
    if (w.exec && w.captured_key == key) return SGIPC_OK;
    if (w.exec) {
        cudaGraphExecDestroy(w.exec);
        w.exec = nullptr;
    }
    cudaGraph_t g = nullptr;
    SG_CHECK(c, cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h = 0;
    // SGIPC_NO_COND_GRAPH=1 selects the relaunched fixed-length graph (profilers that do
    // not descend into conditional bodies then see every iteration kernel)
    const char* nc = getenv("SGIPC_NO_COND_GRAPH");
    cudaError_t e = (nc && nc[0] == '1') ? cudaErrorNotSupported
                                         : cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
    bool ok = e == cudaSuccess;
    cudaGraphNode_t node;
    cudaGraph_t body = nullptr;
    if (ok) {
        cudaGraphNodeParams prm = {};
        prm.type = cudaGraphNodeTypeConditional;
        prm.conditional.handle = h;
        prm.conditional.type = cudaGraphCondTypeWhile;
        prm.conditional.size = 1;
        e = cudaGraphAddNode(&node, g, nullptr, 0, &prm);
        ok = e == cudaSuccess;
        if (ok) body = prm.conditional.phGraph_out[0];
    }
    if (ok) {
        e = cudaStreamBeginCaptureToGraph(c->cap_stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        ok = e == cudaSuccess;
        if (ok) {
            enqueue_body<T, M, NR>(c, w, inv, R, Z, h, 1, k3grid, c->cap_stream);
            cudaGraph_t out = nullptr;
            e = cudaStreamEndCapture(c->cap_stream, &out);
            ok = e == cudaSuccess;
        }
    }
    if (ok) {
        e = cudaGraphInstantiate(&w.exec, g, 0);
        ok = e == cudaSuccess;
    }
    cudaGraphDestroy(g);
    cudaGetLastError();
    if (ok) {
        w.cond_graph = true;
        w.captured_key = key;
        return SGIPC_OK;
    }
    // fallback: a graph of 8 iteration bodies, relaunched until the halt word is set
    w.cond_graph = false;
    w.exec = nullptr;
    SG_CHECK(c, cudaStreamBeginCapture(c->cap_stream, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < 8; k++) enqueue_body<T, M, NR>(c, w, inv, R, Z, h, 0, k3grid, c->cap_stream);
    cudaGraph_t cg = nullptr;
    SG_CHECK(c, cudaStreamEndCapture(c->cap_stream, &cg));
    e = cudaGraphInstantiate(&w.exec, cg, 0);
    cudaGraphDestroy(cg);
    SG_CHECK(c, e);
    w.captured_key = key;
    return SGIPC_OK;
}

// One PCG solve of A x = b (b, x: interleaved [3n][NR], b FP64, x in T) with MAS type M.
template <class T, class M, int NR>
SgipcStatus run_pcg(SgipcCtx* c, PcgWork& w, int fp32_mas, const double* b, double tol, int max_iter, int crit,
                    cudaStream_t s, int tag, RefineArgs* ref = nullptr) {
    MasWork& m = c->mas;
    const M* inv = fp32_mas ? (const M*)m.dom32 : (const M*)m.dom64;
    M* R = fp32_mas ? (M*)m.R32 : (M*)m.R64;
    M* Z = fp32_mas ? (M*)m.Z32 : (M*)m.Z64;
    // one persistent kernel for the whole solve where the device co-schedules it
    bool coop = false;
    if (ref) ref->done = false;
    SgipcStatus st = run_pcg_coop<T, M, NR>(c, w, fp32_mas, b, tol, max_iter, crit, s, &coop, ref);
    w.last_coop = coop;
    if (st != SGIPC_OK || coop) return st;
    const int k3grid = domain_grid(c);
    st = get_loop_graph<T, M, NR>(c, w, inv, R, Z, k3grid, tag);
    if (st != SGIPC_OK) return st;
    const int nv = c->nv, n = c->n;
    PcgPtrs<T, NR> P = ptrs_of<T, NR>(w);
    MasView mv = mas_view(c);
    SG_COUNT(c, 4);
    k_pcg_init<T, M, NR><<<nblk(mv.npos), 256, 0, s>>>(b, P, mv, R, tol, max_iter, crit);
    k_pcg_domains<M, NR><<<k3grid, 192, 0, s>>>(mv, w.sc, inv, R, Z);
    k_pcg_prolong_dot<T, M, NR><<<nblk(nv), 256, 0, s>>>(nv, P, mv, Z, 0, 0, 0);
    k_pcg_init_finish<T, NR><<<nblk(3LL * n), 256, 0, s>>>(3 * n, b, P);
    SG_LAUNCH_CHECK(c, "pcg init");
    if (w.cond_graph) {
        SG_CHECK(c, cudaGraphLaunch(w.exec, s));
    } else {
        for (int guard = 0; guard < 2 + max_iter / 8; guard++) {
            SG_CHECK(c, cudaGraphLaunch(w.exec, s));
            PcgScalars hs[NR];
            SG_CHECK(c, cudaMemcpyAsync(hs, w.sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
            SG_CHECK(c, cudaStreamSynchronize(s));
            if (hs[0].halt) break;
        }
    }
    return SGIPC_OK;
}

// status of a finished solve: still running (state 0) means the iteration cap was hit
int final_status(SgipcCtx* c, const PcgScalars& s) {
    if (s.status == SGIPC_CUDA_ERROR)
        snprintf(c->err, sizeof(c->err), "pcg: a grid barrier of the persistent solve exceeded its wait limit");
    if (s.state == 0) return SGIPC_NOT_CONVERGED;
    return s.status;
}

SgipcStatus alloc_work(SgipcCtx* c, PcgWork& w, size_t elem, int nrhs) {
    const size_t n3 = 3 * (size_t)c->n * nrhs;
    void** vs[] = {&w.x, &w.r, &w.r2, &w.z, &w.p, &w.p2, &w.Ap, &w.Ap2, &w.w};
    for (void** v : vs) SG_CHECK(c, cudaMalloc(v, elem * n3));
    SG_CHECK(c, cudaMalloc((void**)&w.sc, sizeof(PcgScalars) * nrhs));
    SG_CHECK(c, cudaMalloc((void**)&w.partial, sizeof(double) * 4 * nrhs * c->max_blocks));
    SG_CHECK(c, cudaMalloc((void**)&w.ticket, sizeof(unsigned int) * 8));
    SG_CHECK(c, cudaMemset(w.ticket, 0, sizeof(unsigned int) * 8));
    SG_CHECK(c, cudaMemset(w.sc, 0, sizeof(PcgScalars) * nrhs));
    w.coop_cap = coop_max_grid(c->device);
    if (w.coop_cap < 1) w.coop_cap = 1;
    // grid-reduction partials: two parity halves of up to three values per right-hand side
    // and CTA (the fused solve's phase-A reduction)
    SG_CHECK(c, cudaMalloc((void**)&w.coop, sizeof(double) * 2 * 3 * nrhs * (size_t)w.coop_cap));
    return SGIPC_OK;
}

void free_work(PcgWork& w) {
    void* ps[] = {w.x, w.r, w.r2, w.z, w.p, w.p2, w.Ap, w.Ap2, w.w, w.sc, w.partial, w.ticket, w.coop};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (w.exec) cudaGraphExecDestroy(w.exec);
}

}  // namespace

namespace sgipc {

SgipcStatus pcg_create(SgipcCtx* c) {
    int maxn = c->n > c->nv ? c->n : c->nv;
    c->max_blocks = nblk((long long)kSpG * maxn, 256) + 8;
    SgipcStatus st;
    if ((st = alloc_work(c, c->pcg64, sizeof(double), c->max_rhs)) != SGIPC_OK) return st;
    if ((st = alloc_work(c, c->pcg32, sizeof(float), c->max_rhs)) != SGIPC_OK) return st;
    SG_CHECK(c, cudaMalloc((void**)&c->tmp64, sizeof(double) * 3 * (size_t)c->n * c->max_rhs));
    SG_CHECK(c, cudaMalloc((void**)&c->tmp64b, sizeof(double) * 3 * (size_t)c->n * c->max_rhs));
    SG_CHECK(c, cudaMalloc((void**)&c->dot_partial, sizeof(double) * 2048));
    SG_CHECK(c, cudaMalloc((void**)&c->dot_ticket, sizeof(unsigned int) * 4));
    SG_CHECK(c, cudaMemset(c->dot_ticket, 0, sizeof(unsigned int) * 4));
    SG_CHECK(c, cudaMalloc((void**)&c->dot_out, sizeof(double) * 16));
    SG_CHECK(c, cudaMallocHost((void**)&c->h_pinned, sizeof(double) * 64));
    SG_CHECK(c, cudaMallocHost((void**)&c->h_scalars, sizeof(PcgScalars) * 4));
    SG_CHECK(c, cudaStreamCreateWithFlags(&c->cap_stream, cudaStreamNonBlocking));
    // the contact merge is a chain of small dependent kernels on the assembly's critical path:
    // its stream gets the highest priority, so that its blocks go ahead of the element and MAS
    // kernels running beside it
    int prio_least = 0, prio_greatest = 0;
    SG_CHECK(c, cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest));
    SG_CHECK(c, cudaStreamCreateWithPriority(&c->asm_stream, cudaStreamNonBlocking, prio_greatest));
    for (cudaEvent_t& e : c->ev_asm) SG_CHECK(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return SGIPC_OK;
}

void pcg_destroy(SgipcCtx* c) {
    free_work(c->pcg64);
    free_work(c->pcg32);
    void* ps[] = {c->tmp64, c->tmp64b, c->dot_partial, c->dot_ticket, c->dot_out};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (c->h_pinned) cudaFreeHost(c->h_pinned);
    if (c->h_scalars) cudaFreeHost(c->h_scalars);
    if (c->cap_stream) cudaStreamDestroy(c->cap_stream);
    if (c->asm_stream) {
        cudaStreamSynchronize(c->asm_stream);
        cudaStreamDestroy(c->asm_stream);
    }
    for (cudaEvent_t e : c->ev_asm)
        if (e) cudaEventDestroy(e);
}

template <class T>
SgipcStatus spmv_t(SgipcCtx* c, const T* x, T* y, cudaStream_t s) {
    SG_COUNT(c, 1);
    k_spmv<T><<<spmv_grid(c->n), 256, 0, s>>>(topo_of(c), mat_view<T>(c), x, y);
    SG_LAUNCH_CHECK(c, "spmv");
    return SGIPC_OK;
}
template SgipcStatus spmv_t<double>(SgipcCtx*, const double*, double*, cudaStream_t);
template SgipcStatus spmv_t<float>(SgipcCtx*, const float*, float*, cudaStream_t);

SgipcStatus dot64(SgipcCtx* c, const double* a, const double* b, int n, double* out_dev, cudaStream_t s) {
    int g = nblk(n, 256);
    if (g > 1024) g = 1024;
    SG_COUNT(c, 1);
    k_dot<<<g, 256, 0, s>>>(n, a, b, c->dot_partial, c->dot_ticket, out_dev);
    SG_LAUNCH_CHECK(c, "dot");
    return SGIPC_OK;
}

}  // namespace sgipc

// --------------------------------------------------------------------------------------------
// C ABI
// --------------------------------------------------------------------------------------------
extern "C" SgipcStatus sgipc_spmv(SgipcCtx* c, const double* x, double* y, void* stream) {
    if (!c || !x || !y) return SGIPC_BAD_INPUT;
    if (!c->assembled) return SGIPC_NOT_READY;
    SG_DEVICE(c);
    return spmv_t<double>(c, x, y, (cudaStream_t)stream);
}

// ||b - A x||^2 and ||b||^2 of right-hand sides blockIdx.y = 0 .. (b, x rhs-major) in one launch: rows by groups
// of kSpG lanes, per-CTA partials, the last CTA of a right-hand side adds them in order
constexpr int kResidualCtas = 256;  // per right-hand side: dot_partial holds two sums of four
__global__ void __launch_bounds__(256) k_true_residual(Topo tp, MatView<double> A, const double* __restrict__ b,
                                                       const double* __restrict__ x, double* __restrict__ partial,
                                                       unsigned int* __restrict__ ticket, double* __restrict__ out) {
    __shared__ double smem[2 * 32];
    const size_t first = 3 * (size_t)tp.n * blockIdx.y;
    Operand<double, 1> op;
    op.a = x + first;
    op.b = nullptr;
    op.beta[0] = 0;
    constexpr int rows = 256 / kSpG;
    double v[2] = {0.0, 0.0};
    for (int i0 = blockIdx.x * rows; i0 < tp.n; i0 += gridDim.x * rows) {  // CTA-uniform
        const int i = i0 + (int)threadIdx.x / kSpG, g = threadIdx.x % kSpG;
        double acc[1][3];
        row_mv<double, 1>(tp, A, op, i, g, acc);
        if (i < tp.n && g == 0)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const double bi = b[first + 3 * (size_t)i + q], r = bi - acc[0][q];
                v[0] += r * r;
                v[1] += bi * bi;
            }
    }
    double tot[2];
    if (grid_sum<2>(v, partial + blockIdx.y * 2 * kResidualCtas, ticket + blockIdx.y, tot, smem) && threadIdx.x == 0) {
        out[2 * blockIdx.y] = tot[0];
        out[2 * blockIdx.y + 1] = tot[1];
    }
}

// enqueue ||b - A x||^2 and ||b||^2 of nrhs <= 4 right-hand sides, on their way to h_pinned[0 ..]
static SgipcStatus enqueue_residuals(SgipcCtx* c, const double* b, const double* x, int nrhs, cudaStream_t s) {
    SG_COUNT(c, 1);
    const int grid = spmv_grid(c->n) < kResidualCtas ? spmv_grid(c->n) : kResidualCtas;
    k_true_residual<<<dim3(grid, nrhs), 256, 0, s>>>(topo_of(c), mat_view<double>(c), b, x, c->dot_partial,
                                                     c->dot_ticket, c->dot_out);
    SG_LAUNCH_CHECK(c, "true residual");
    SG_CHECK(c, cudaMemcpyAsync(c->h_pinned, c->dot_out, 2 * nrhs * sizeof(double), cudaMemcpyDeviceToHost, s));
    return SGIPC_OK;
}

// pinned host word for the device input-error flag, read with a solve's final copies
static int* input_flag(SgipcCtx* c) { return reinterpret_cast<int*>(c->h_pinned + 32); }

// pinned landing area of a solve's scalars (four right-hand sides at most)
static PcgScalars* pinned_scalars(SgipcCtx* c) { return c->h_scalars; }

static SgipcStatus input_error(SgipcCtx* c, cudaStream_t s) {
    *input_flag(c) = 0;
    SG_CHECK(c, cudaMemsetAsync(c->dflag, 0, sizeof(int), s));
    snprintf(c->err, sizeof(c->err), "a contact pair names a vertex outside [0, vertex_num); it was skipped");
    return SGIPC_BAD_INPUT;
}

static SgipcStatus solve_one(SgipcCtx* c, SgipcPrecision prec, SgipcCriterion crit, double tol, int max_iter,
                             const double* b, double* x, SgipcSolveStats* stats, cudaStream_t s) {
    const int n3 = 3 * c->n;
    if (max_iter <= 0) max_iter = (int)(0.3 * n3);
    if (max_iter < 2) max_iter = 2;
    SgipcSolveStats out = {};
    SgipcStatus st;
    if (prec == SGIPC_FP64 || prec == SGIPC_REF) {
        const int f32 = prec == SGIPC_REF ? 1 : 0;
        if (f32)
            st = run_pcg<double, float, 1>(c, c->pcg64, 1, b, tol, max_iter, (int)crit, s, 11);
        else
            st = run_pcg<double, double, 1>(c, c->pcg64, 0, b, tol, max_iter, (int)crit, s, 10);
        if (st != SGIPC_OK) return st;
        SG_CHECK(c, cudaMemcpyAsync(x, c->pcg64.x, sizeof(double) * n3, cudaMemcpyDeviceToDevice, s));
        // the solve's scalars, its input flag and the true residual come back together
        PcgScalars& hs = *pinned_scalars(c);
        SG_CHECK(c, cudaMemcpyAsync(&hs, c->pcg64.sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
        if ((st = enqueue_residuals(c, b, x, 1, s)) != SGIPC_OK) return st;
        // the persistent solve copies the bad-input flag into its scalars: one read-back
        if (!c->pcg64.last_coop)
            SG_CHECK(c, cudaMemcpyAsync(input_flag(c), c->dflag, sizeof(int), cudaMemcpyDeviceToHost, s));
        SG_CHECK(c, cudaStreamSynchronize(s));
        if (c->pcg64.last_coop) *input_flag(c) = hs.input_flag;
        if (*input_flag(c)) return input_error(c, s);
        SG_COUNT(c, 4LL * hs.bodies);
        out.iterations = hs.iter;
        out.refinements = 0;
        out.rz0 = hs.rz0;
        out.rz = hs.rz_next;
        out.rel_residual = c->h_pinned[1] > 0.0 ? sqrt(c->h_pinned[0] / c->h_pinned[1]) : 0.0;
        out.status = final_status(c, hs);
    } else {
        // mixed: FP32 MAS-PCG inner solves on the FP32 matrix copy, FP64 residual refinement
        // the first inner solve takes b itself and sets x = its correction (nothing to zero or
        // copy first); later ones take the FP64 residual r64 and add to x
        double* r64 = c->tmp64;
        double rz0 = -1.0, rz = 0.0, bn2 = 0.0, rr = 0.0;
        int total_it = 0, ref = 0, status = SGIPC_OK;
        for (ref = 0; ref < 8; ref++) {
            // the reduction the inner solve still has to make, on its own right-hand side (the
            // FP64 residual): r.z by rz0 / rz; on the true residual, ||r|| to tol ||b||, aimed
            // at half of it, so that the FP32 inner residual's drift from the FP64 one rarely
            // costs another refinement
            double inner_tol = tol;
            if (rz0 > 0 && rz > 0) inner_tol = fmin(1.0, fmax(tol * rz0 / rz, 1e-10));
            if (crit == SGIPC_CRIT_TRUE)
                inner_tol = bn2 > 0 && rr > 0 ? fmin(1.0, fmax(0.5 * tol * sqrt(bn2 / rr), 1e-10)) : 0.5 * tol;
            // the persistent solve refines itself where it can (x += x32, FP64 residual, its
            // r.z and r.r); otherwise the same steps follow here
            RefineArgs rf{x, b, r64, false, ref == 0};
            st = run_pcg<float, float, 1>(c, c->pcg32, 1, ref == 0 ? b : r64, inner_tol, max_iter, (int)crit, s, 20,
                                          &rf);
            if (st != SGIPC_OK) return st;
            PcgScalars& hs = *pinned_scalars(c);
            if (!rf.done) {
                SG_COUNT(c, 2);
                k_add_f32<<<nblk(n3), 256, 0, s>>>(n3, (const float*)c->pcg32.x, x, ref == 0 ? 1 : 0);
                // r = b - A x in FP64
                if ((st = spmv_t<double>(c, x, c->tmp64b, s)) != SGIPC_OK) return st;
                k_axpby_res<<<nblk(n3), 256, 0, s>>>(n3, b, c->tmp64b, r64);
                // rz of the refined residual with the same (FP32) preconditioner
                if ((st = mas_apply_t<double>(c, r64, c->tmp64b, 1, s)) != SGIPC_OK) return st;
                if ((st = dot64(c, r64, c->tmp64b, n3, c->dot_out, s)) != SGIPC_OK) return st;
                if ((st = dot64(c, r64, r64, n3, c->dot_out + 1, s)) != SGIPC_OK) return st;
                SG_CHECK(c, cudaMemcpyAsync(c->h_pinned, c->dot_out, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
            }
            SG_CHECK(c, cudaMemcpyAsync(&hs, c->pcg32.sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
            if (!c->pcg32.last_coop)
                SG_CHECK(c, cudaMemcpyAsync(input_flag(c), c->dflag, sizeof(int), cudaMemcpyDeviceToHost, s));
            SG_CHECK(c, cudaStreamSynchronize(s));
            if (c->pcg32.last_coop) *input_flag(c) = hs.input_flag;
            if (*input_flag(c)) return input_error(c, s);
            if (rf.done) {
                c->h_pinned[0] = hs.rz_ref;
                c->h_pinned[1] = hs.rr_ref;
            }
            total_it += hs.iter;
            SG_COUNT(c, 4LL * hs.bodies);
            if (ref == 0) {
                rz0 = hs.rz0;
                bn2 = hs.bnorm2;
            }
            rz = c->h_pinned[0];
            rr = c->h_pinned[1];
            if (hs.status == SGIPC_BREAKDOWN || hs.status == SGIPC_CUDA_ERROR) {
                status = final_status(c, hs);
                break;
            }
            bool done = crit == SGIPC_CRIT_RZ ? fabs(rz) <= tol * rz0 : c->h_pinned[1] <= tol * tol * bn2;
            if (done || total_it >= max_iter) {
                if (!done) status = SGIPC_NOT_CONVERGED;
                break;
            }
        }
        out.iterations = total_it;
        out.refinements = ref + 1;
        out.rz0 = rz0;
        out.rz = rz;
        out.status = status;
        // the last refinement computed r = b - A x in FP64 and ||r||^2 (h_pinned[1]);
        // ||b||^2 is the first inner solve's right-hand side norm
        out.rel_residual = bn2 > 0.0 ? sqrt(c->h_pinned[1] / bn2) : 0.0;
    }
    if (stats) *stats = out;
    return (SgipcStatus)out.status;
}

extern "C" SgipcStatus sgipc_pcg_solve(SgipcCtx* c, SgipcPrecision prec, SgipcCriterion crit, double tol,
                                       int32_t max_iter, const double* b, double* x, SgipcSolveStats* stats,
                                       void* stream) {
    if (!c || !b || !x || !(tol > 0.0)) return SGIPC_BAD_INPUT;
    if (!c->assembled || !c->mas.built) return SGIPC_NOT_READY;
    SG_DEVICE(c);
    // the MAS inverses must exist in the precision the solve reads
    if ((prec == SGIPC_FP64) != (c->mas.built == SGIPC_FP64 + 1)) return SGIPC_NOT_READY;
    // a contact pair with an out-of-range vertex (flagged by the assembly kernels) is
    // reported from the solve's own synchronisation, not from an extra one here
    return solve_one(c, prec, crit, tol, max_iter, b, x, stats, (cudaStream_t)stream);
}

extern "C" SgipcStatus sgipc_solve(SgipcCtx* c, const SgipcContacts* con, SgipcPrecision prec, SgipcCriterion crit,
                                   double tol, int32_t max_iter, double* move_dir, SgipcSolveStats* stats,
                                   void* stream) {
    if (!c || !move_dir) return SGIPC_BAD_INPUT;
    if (!c->assembled) return SGIPC_NOT_READY;
    SG_DEVICE(c);
    SgipcStatus st = sgipc_mas_build(c, con, prec, stream);
    if (st != SGIPC_OK) return st;
    return sgipc_pcg_solve(c, prec, crit, tol, max_iter, c->b, move_dir, stats, stream);
}

extern "C" SgipcStatus sgipc_pcg_solve_batched(SgipcCtx* c, SgipcPrecision prec, SgipcCriterion crit, double tol,
                                               int32_t max_iter, int32_t nrhs, const double* b, double* x,
                                               SgipcSolveStats* stats, void* stream) {
    if (!c || !b || !x || nrhs < 1 || !(tol > 0.0)) return SGIPC_BAD_INPUT;
    if (nrhs > c->max_rhs) return SGIPC_CAPACITY;
    if (!c->assembled || !c->mas.built) return SGIPC_NOT_READY;
    if ((prec == SGIPC_FP64) != (c->mas.built == SGIPC_FP64 + 1)) return SGIPC_NOT_READY;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    const int n3 = 3 * c->n;
    if (max_iter <= 0) max_iter = (int)(0.3 * n3);
    if (max_iter < 2) max_iter = 2;
    if (nrhs != 4) {
        // one right-hand side at a time
        SgipcStatus worst = SGIPC_OK;
        for (int r = 0; r < nrhs; r++) {
            SgipcStatus st = solve_one(c, prec, crit, tol, max_iter, b + (size_t)r * n3, x + (size_t)r * n3,
                                       stats ? stats + r : nullptr, s);
            if (st == SGIPC_CUDA_ERROR || st == SGIPC_BAD_INPUT) return st;
            if (st != SGIPC_OK) worst = st;
        }
        return worst;
    }
    // four right-hand sides interleaved: every matrix / MAS block read serves all four
    double* bi = c->tmp64;
    SG_COUNT(c, 2);
    k_interleave<double, double><<<nblk(4LL * n3), 256, 0, s>>>(n3, 4, b, bi, 1);
    SgipcStatus st;
    PcgWork& w = (prec == SGIPC_MIXED) ? c->pcg32 : c->pcg64;
    if (prec == SGIPC_FP64)
        st = run_pcg<double, double, 4>(c, w, 0, bi, tol, max_iter, (int)crit, s, 40);
    else if (prec == SGIPC_REF)
        st = run_pcg<double, float, 4>(c, w, 1, bi, tol, max_iter, (int)crit, s, 41);
    else
        st = run_pcg<float, float, 4>(c, w, 1, bi, tol, max_iter, (int)crit, s, 42);
    if (st != SGIPC_OK) return st;
    if (prec == SGIPC_MIXED)
        k_interleave<float, double><<<nblk(4LL * n3), 256, 0, s>>>(n3, 4, (const float*)w.x, x, 0);
    else
        k_interleave<double, double><<<nblk(4LL * n3), 256, 0, s>>>(n3, 4, (const double*)w.x, x, 0);
    PcgScalars* hs = pinned_scalars(c);
    SG_CHECK(c, cudaMemcpyAsync(hs, w.sc, 4 * sizeof(PcgScalars), cudaMemcpyDeviceToHost, s));
    if (stats && (st = enqueue_residuals(c, b, x, 4, s)) != SGIPC_OK) return st;
    SG_CHECK(c, cudaStreamSynchronize(s));
    SgipcStatus worst = SGIPC_OK;
    SG_COUNT(c, 4LL * hs[0].bodies);
    for (int r = 0; r < 4; r++) {
        const int fs = final_status(c, hs[r]);
        if (stats) {
            stats[r] = SgipcSolveStats{};
            stats[r].iterations = hs[r].iter;
            stats[r].rz0 = hs[r].rz0;
            stats[r].rz = hs[r].rz_next;
            stats[r].status = fs;
            stats[r].rel_residual = c->h_pinned[2 * r + 1] > 0.0 ? sqrt(c->h_pinned[2 * r] / c->h_pinned[2 * r + 1]) : 0.0;
        }
        if (fs != SGIPC_OK) worst = (SgipcStatus)fs;
    }
    return worst;
}

namespace sgipc {
// "pcg32" / "pcg64": one PCG solve of the last right-hand side to the 1e-4 r.z criterion
// (FP32 vectors + FP32 MAS, the inner solve of the mixed mode / FP64 throughout), i.e. one
// launch of the persistent solve.  Algorithmic bytes: iterations x (SpMV + 2 dots + 2
// axpys + MAS apply), each compulsory array read or written once:
//   SpMV nb (sb + 4) + (n + 1) 4 + 2 (3n) sv;  dots 2 x 2 (3n) sv;  axpys 6 (3n) sv + 3 (3n) sv;
//   MAS (3n) sv + 12 Nc + (Nc / 16) 136 sb + 12 Nc + 4 L Nc + (3n) sv
// with sv / sb the vector / 3x3-block bytes, nb the stored upper blocks, Nc the clusters.
static SgipcStatus pcg_solve_hook(SgipcCtx* c, bool f64, cudaStream_t s, double* bytes) {
    if (!c->mas.built || (c->mas.built == SGIPC_FP64 + 1) != f64) {
        snprintf(c->err, sizeof(c->err), "time_kernel pcg%s: the MAS was built in the other precision",
                 f64 ? "64" : "32");
        return SGIPC_BAD_INPUT;
    }
    const int n3 = 3 * c->n;
    const int max_iter = n3 * 3 / 10 > 2 ? n3 * 3 / 10 : 2;
    SgipcStatus st = f64 ? run_pcg<double, double, 1>(c, c->pcg64, 0, c->b, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 10)
                         : run_pcg<float, float, 1>(c, c->pcg32, 1, c->b, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 20);
    if (st != SGIPC_OK) return st;
    if (*bytes == 0.0) {  // untimed first launch: read the iteration count and block count
        PcgScalars hs;
        int nuc = 0;
        SG_CHECK(c, cudaMemcpyAsync(&hs, (f64 ? c->pcg64 : c->pcg32).sc, sizeof(hs), cudaMemcpyDeviceToHost, s));
        SG_CHECK(c, cudaMemcpyAsync(&nuc, c->nuc, sizeof(int), cudaMemcpyDeviceToHost, s));
        SG_CHECK(c, cudaStreamSynchronize(s));
        const double sv = f64 ? 8 : 4, sb = f64 ? 72 : 36, Nc = c->mas.h_info[16], L = c->mas.levelnum;
        const double nb = (double)c->nnz + nuc;
        const double spmv = nb * (sb + 4) + (c->n + 1.0) * 4 + 2.0 * n3 * sv;
        const double dots = 2 * 2.0 * n3 * sv, axpy = 9.0 * n3 * sv;
        const double mas = 2.0 * n3 * sv + 24 * Nc + Nc / 16 * 136 * sb + 4 * L * Nc;
        *bytes = hs.iter * (spmv + dots + axpy + mas);
    }
    return SGIPC_OK;
}

SgipcStatus pcg_time_hook(SgipcCtx* c, const char* name, cudaStream_t s, double* bytes) {
    if (!strcmp(name, "pcg32") || !strcmp(name, "pcg64")) return pcg_solve_hook(c, name[3] == '6', s, bytes);
    const bool f64 = !strcmp(name, "spmv64"), f32 = !strcmp(name, "spmv32");
    if (!f64 && !f32) return SGIPC_NOT_READY;
    // the contact block count is read once, on the untimed first launch (*bytes still 0),
    // so that the timed launches carry no host synchronisation
    if (*bytes == 0.0) {
        int nuc = 0;
        SG_CHECK(c, cudaMemcpyAsync(&nuc, c->nuc, sizeof(int), cudaMemcpyDeviceToHost, s));
        SG_CHECK(c, cudaStreamSynchronize(s));
        const double sb = f64 ? 72 : 36, sv = f64 ? 8 : 4;
        // algorithmic: nb (sb + 4) + (n + 1) 4 + 2 * 3n * sv, nb = upper static + unique contact blocks
        *bytes = ((double)c->nnz + nuc) * (sb + 4) + (c->n + 1.0) * 4 + 2.0 * 3 * c->n * sv;
    }
    SG_COUNT(c, 1);
    if (f64)
        k_spmv<double><<<spmv_grid(c->n), 256, 0, s>>>(topo_of(c), mat_view<double>(c), c->tmp64, c->tmp64b);
    else
        k_spmv<float><<<spmv_grid(c->n), 256, 0, s>>>(topo_of(c), mat_view<float>(c), (const float*)c->tmp64,
                                                      (float*)c->tmp64b);
    SG_LAUNCH_CHECK(c, name);
    return SGIPC_OK;
}
}  // namespace sgipc

extern "C" SgipcStatus sgipc_launch_count(SgipcCtx* c, int64_t* launches) {
    if (!c || !launches) return SGIPC_BAD_INPUT;
    SG_DEVICE(c);
    SG_CHECK(c, cudaDeviceSynchronize());
    *launches = c->launches;
    return SGIPC_OK;
}

namespace {
// four copies of b interleaved ([3n][4]) for the 4-right-hand-side phase profile
__global__ void k_replicate4(int n3, const double* __restrict__ b, double* __restrict__ bi) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n3) {
        const double v = b[k];
        reinterpret_cast<double2*>(bi)[2 * k] = make_double2(v, v);
        reinterpret_cast<double2*>(bi)[2 * k + 1] = make_double2(v, v);
    }
}
}  // namespace

extern "C" SgipcStatus sgipc_profile_pcg(SgipcCtx* c, const char* name, int32_t max_epochs, uint64_t* stamps,
                                         int32_t* grid, int32_t* epochs, void* stream) {
    if (!c || !name || max_epochs < 2 || !stamps || !grid || !epochs) return SGIPC_BAD_INPUT;
    if (!c->assembled || !c->mas.built) return SGIPC_NOT_READY;
    const bool x4 = !strcmp(name, "pcg32x4") || !strcmp(name, "pcg64x4");
    const bool f64 = !strcmp(name, "pcg64") || !strcmp(name, "pcg64x4");
    if (!x4 && strcmp(name, "pcg32") && strcmp(name, "pcg64")) return SGIPC_BAD_INPUT;
    if ((c->mas.built == SGIPC_FP64 + 1) != f64) {
        snprintf(c->err, sizeof(c->err), "profile_pcg %s: the MAS was built in the other precision", name);
        return SGIPC_BAD_INPUT;
    }
    if (x4 && c->max_rhs < 4) return SGIPC_CAPACITY;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    const int cap = c->pcg64.coop_cap > c->pcg32.coop_cap ? c->pcg64.coop_cap : c->pcg32.coop_cap;
    const size_t words = (size_t)cap * max_epochs * 2 + max_epochs;  // stamps, then the phase tags
    unsigned long long* d = nullptr;
    SG_CHECK(c, cudaMalloc((void**)&d, words * sizeof(unsigned long long)));
    SgipcStatus st = SGIPC_OK;
    cudaError_t e = cudaMemsetAsync(d, 0, words * sizeof(unsigned long long), s);
    const int n3 = 3 * c->n;
    const int max_iter = n3 * 3 / 10 > 2 ? n3 * 3 / 10 : 2;
    if (e == cudaSuccess) {
        c->stamps = d;
        c->stamp_epochs = max_epochs;
        if (!x4) {
            st = f64 ? run_pcg<double, double, 1>(c, c->pcg64, 0, c->b, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 10)
                     : run_pcg<float, float, 1>(c, c->pcg32, 1, c->b, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 20);
        } else {
            SG_COUNT(c, 1);
            k_replicate4<<<nblk(n3), 256, 0, s>>>(n3, c->b, c->tmp64);
            st = f64 ? run_pcg<double, double, 4>(c, c->pcg64, 0, c->tmp64, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 40)
                     : run_pcg<float, float, 4>(c, c->pcg32, 1, c->tmp64, 1e-4, max_iter, SGIPC_CRIT_RZ, s, 42);
        }
        c->stamps = nullptr;
        c->stamp_epochs = 0;
        e = cudaStreamSynchronize(s);
    }
    // the grid the solve ran with: the CTAs that stamped epoch 0
    if (st == SGIPC_OK && e == cudaSuccess)
        e = cudaMemcpy(stamps, d, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (st != SGIPC_OK) return st;
    if (e != cudaSuccess) return cuda_fail(c, e, "profile_pcg");
    int g = 0, ep = 0;
    while (g < cap && stamps[(size_t)g * max_epochs * 2] != 0) g++;
    if (g == 0) {
        snprintf(c->err, sizeof(c->err), "profile_pcg: the solve ran as the graph of per-phase kernels");
        return SGIPC_NOT_READY;
    }
    while (ep < max_epochs && stamps[(size_t)ep * 2 + 1] != 0) ep++;
    // the launch wrote its phase tags after its own grid's stamps: move them behind the
    // capacity's, where the caller finds them
    if (g < cap)
        memmove(stamps + (size_t)cap * max_epochs * 2, stamps + (size_t)g * max_epochs * 2,
                sizeof(uint64_t) * max_epochs);
    *grid = g;
    *epochs = ep;
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_time_kernel(SgipcCtx* c, const char* name, int32_t reps, void* stream, float* avg_ms,
                                         double* bytes_per_launch) {
    if (!c || !name || reps < 1 || !avg_ms) return SGIPC_BAD_INPUT;
    if (!c->assembled) return SGIPC_NOT_READY;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    // spmv reads tmp64: give it a defined vector
    SG_CHECK(c, cudaMemsetAsync(c->tmp64, 0, sizeof(double) * 3 * c->n, s));
    SgipcStatus (*hooks[3])(SgipcCtx*, const char*, cudaStream_t, double*) = {assemble_time_hook, mas_time_hook,
                                                                              pcg_time_hook};
    double bytes = 0;
    int owner = -1;
    for (int h = 0; h < 3 && owner < 0; h++) {
        SgipcStatus st = hooks[h](c, name, s, &bytes);  // warm-up launch
        if (st == SGIPC_OK) owner = h;
        else if (st != SGIPC_NOT_READY) return st;
    }
    if (owner < 0) return SGIPC_BAD_INPUT;
    cudaEvent_t e0, e1;
    SG_CHECK(c, cudaEventCreate(&e0));
    SG_CHECK(c, cudaEventCreate(&e1));
    SG_CHECK(c, cudaEventRecord(e0, s));
    for (int r = 0; r < reps; r++) {
        SgipcStatus st = hooks[owner](c, name, s, &bytes);
        if (st != SGIPC_OK) return st;
    }
    SG_CHECK(c, cudaEventRecord(e1, s));
    SG_CHECK(c, cudaEventSynchronize(e1));
    float ms = 0;
    SG_CHECK(c, cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *avg_ms = ms / reps;
    if (bytes_per_launch) *bytes_per_launch = bytes;
    // the MAS kernels overwrite the domain matrices: rebuild them as they were
    if (owner == 1 && c->mas.built) {
        SgipcPrecision prec = (SgipcPrecision)(c->mas.built - 1);
        SgipcStatus st = mas_build(c, c->mas_has_con ? &c->mas_con : nullptr, prec, s);
        if (st != SGIPC_OK) return st;
    }
    SG_CHECK(c, cudaStreamSynchronize(s));
    return SGIPC_OK;
}
