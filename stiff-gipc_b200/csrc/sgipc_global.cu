// sgipc_global.cu — the global FEM + ABD linear system: one PCG over [ABD | FEM] DOFs.
//
// Semantics of StiffGIPC's GlobalLinearSystem with its two subsystems (gipc/gipc.cu:42-70):
// the ABD subsystem comes first (12 DOFs = 4 block rows per body), the FEM subsystem after
// it (3 DOFs per vertex), offsets by an exclusive scan of the subsystem sizes
// (global_linear_system.cu:8-74).  The matrix is the symmetric upper BCOO of both
// (global_linear_system.cu:182-199, spmv.cu): here the FEM context's assembled matrix on
// the FEM rows and the ABD context's merged body-space blocks (body rows, and body x FEM
// coupling in FEM columns) used with their transposes.  The preconditioner is the identity
// overwritten by each local preconditioner on its own range (apply_preconditioner,
// global_linear_system.cu:152-166): ABDPreconditioner (12x12 block Jacobi) on the body
// rows, MAS_Preconditioner on the FEM rows.  PCGSolver::pcg (pcg_solver.cu:174-267) with
// its stop rule.  distribute_solution (global_linear_system.cu:76-87) hands the FEM part
// back as the FEM move direction and maps every body's dq to its points:
// dx = J(x_bar) dq (ABDLinearSubsystem::retrieve_solution, abd_linear_subsystem.cu:33-56,
// cal_x_from_q.cu:34-66 forms J q - J (q - dq), the same quantity).
//
// B200 layout: one kernel multiplies: FEM rows as the FEM context's SpMV (four lanes a row,
// contact lists included) with their transposed coupling blocks, body rows by one warp each over
// the row-sorted merged blocks and a column-sorted index of their transposes, so every output is
// summed in a fixed order (no atomics).  It forms p = z + beta p_old where it reads it and p.Ap
// with it; the kernel that prolongs the MAS and applies the bodies' block Jacobi also takes r.z.
// The last CTA of each adds the partial sums in order and writes the loop's scalars (alpha,
// beta, the stop tests), which live on the device.  The host enqueues one iteration ahead and
// then waits for the state of the one before: the kernels of an iteration after the stop return
// at once, so that the read-back costs no idle time and the last iteration a few empty launches.
// (Sixteen launches an iteration and a wait after each: 2.17 ms for 500 boxes over a bed; the
// body rows with one thread each took 28 us, the coupling 13 us.)
#include <cub/cub.cuh>

#include "sgipc_abd_ctx.cuh"
#include "sgipc_pcg_dev.cuh"

using namespace sgipc;

namespace {

__device__ __forceinline__ int lower_bound_i(const int* a, int n, int v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int lower_bound_k(const unsigned long long* a, int n, unsigned long long v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// rptr[r] = first merged block of body row r (blocks are sorted by (row, col))
__global__ void k_g_rowptr(int nrows, const int* __restrict__ nu, const int* __restrict__ u_row, int* __restrict__ rptr) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r <= nrows) rptr[r] = lower_bound_i(u_row, nu[0], r);
}

// transposed index: the off-diagonal blocks keyed by (col, row), the row in `bits` bits; diagonal
// blocks, unused slots and columns beyond the FEM rows sort past every column
__global__ void k_g_tkeys(int m, int bits, int ncols, const int* __restrict__ nu, const int* __restrict__ u_row,
                          const int* __restrict__ u_col, unsigned long long* __restrict__ key, int* __restrict__ idx) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const bool off = k < nu[0] && u_row[k] != u_col[k] && (unsigned)u_col[k] < (unsigned)ncols;
    key[k] = off ? (((unsigned long long)(unsigned)u_col[k] << bits) | (unsigned)u_row[k]) : ~0ull;
    idx[k] = k;
}

__global__ void k_g_colptr(int ncols, int m, int bits, const unsigned long long* __restrict__ key_s,
                           int* __restrict__ cptr) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= ncols) cptr[c] = lower_bound_k(key_s, m, (unsigned long long)(unsigned)c << bits);
}

__device__ __forceinline__ void block_mv(const double* V, const double (&x)[3], double (&y)[3]) {
    y[0] += V[0] * x[0] + V[1] * x[1] + V[2] * x[2];
    y[1] += V[3] * x[0] + V[4] * x[1] + V[5] * x[2];
    y[2] += V[6] * x[0] + V[7] * x[1] + V[8] * x[2];
}

__device__ __forceinline__ void block_mtv(const double* V, const double (&x)[3], double (&y)[3]) {
    y[0] += V[0] * x[0] + V[3] * x[1] + V[6] * x[2];
    y[1] += V[1] * x[0] + V[4] * x[1] + V[7] * x[2];
    y[2] += V[2] * x[0] + V[5] * x[1] + V[8] * x[2];
}

// Device state of the loop (PCGSolver::pcg's scalars).  stop: 0 running, 1 converged or broken
// down, 2 at the iteration cap; an iteration that finds it set does nothing.
struct GState {
    double rz0, rz, bn2, alpha, beta, res2;
    int iters, halt, status, stop;  // halt: alpha is not usable, the update of this iteration is skipped
};
constexpr int kGThreads = 256;
constexpr int kGBodyRows = kGThreads / 32;        // body rows per CTA of the SpMV
constexpr int kGFemRows = kGThreads / kSpG;       // FEM rows per CTA

// Adds v over the grid: per-CTA partials, and the last CTA to arrive adds them (each thread its
// strided share in order, then fixed trees).  True in the last CTA's thread 0, with the total.
__device__ bool grid_total(double v, double* part, unsigned int* ticket, double& total) {
    __shared__ double smem[32];
    __shared__ bool s_last;
    double a[1] = {v};
    block_sum<1>(a, smem);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = a[0];
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    a[0] = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) a[0] += __ldcg(part + k);
    block_sum<1>(a, smem);
    if (threadIdx.x != 0) return false;
    *ticket = 0u;
    total = a[0];
    return true;
}

struct GMat {
    Topo tp;
    MatView<double> A;
    int nb, nfem;  // body block rows, FEM block rows
    const int* rptr;
    const int* cptr;
    const int* tidx;
    const int* u_row;
    const int* u_col;
    const double* u_val;
};

// kResidual = false: p = z + beta p_old (p = z in the first iteration), y = A p, alpha = r.z / p.Ap and
// the stop tests of iteration k.  kResidual = true: y = b - A z, y.y into st->res2.
template <bool kResidual>
__global__ void __launch_bounds__(kGThreads) k_g_spmv(GMat g, GState* st, const double* __restrict__ z,
                                                      const double* __restrict__ p_old, double* __restrict__ p,
                                                      double* __restrict__ y, const double* __restrict__ b, int k,
                                                      int crit, double tol, int max_iter, double* part,
                                                      unsigned int* ticket) {
    if (!kResidual && (st->stop || st->halt)) return;
    const int lane = threadIdx.x & 31;
    const int body_ctas = (g.nb + kGBodyRows - 1) / kGBodyRows;
    Operand<double, 1> op;
    op.a = z;
    op.b = p_old;
    op.beta[0] = kResidual ? 0.0 : st->beta;
    double dot = 0.0;
    int row = -1;            // the global block row this thread finishes
    double acc[1][3] = {{0.0, 0.0, 0.0}};
    if ((int)blockIdx.x < body_ctas) {
        const int r = blockIdx.x * kGBodyRows + (int)(threadIdx.x >> 5);
        if (r < g.nb) {
            const int k0 = g.rptr[r], n0 = g.rptr[r + 1] - k0, j0 = g.cptr[r], n = n0 + g.cptr[r + 1] - j0;
            for (int e = lane; e < n; e += 32) {
                const bool up = e < n0;
                const int u = up ? k0 + e : g.tidx[j0 + e - n0];
                double xj[1][3];
                op.load(up ? g.u_col[u] : g.u_row[u], xj);
                if (up) block_mv(g.u_val + 9 * (size_t)u, xj[0], acc[0]);
                else block_mtv(g.u_val + 9 * (size_t)u, xj[0], acc[0]);
            }
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[0][q] += __shfl_xor_sync(0xffffffffu, acc[0][q], o);
            if (lane == 0) row = r;
        }
    } else {
        const int t = (blockIdx.x - body_ctas) * kGThreads + threadIdx.x;
        const int i = t / kSpG, l = t % kSpG;
        Operand<double, 1> fo = op;  // FEM columns are counted from the FEM vector's start
        fo.a = z + 3 * (size_t)g.nb;
        fo.b = p_old ? p_old + 3 * (size_t)g.nb : nullptr;
        row_mv<double, 1>(g.tp, g.A, fo, i, l, acc);
        int j0 = 0, j1 = 0;
        if (i < g.nfem) j0 = g.cptr[g.nb + i], j1 = g.cptr[g.nb + i + 1];
        if (__any_sync(0xffffffffu, j0 < j1)) {
            double c3[3] = {0.0, 0.0, 0.0};
            for (int j = j0 + l; j < j1; j += kSpG) {
                const int u = g.tidx[j];
                double xj[1][3];
                op.load(g.u_row[u], xj);
                block_mtv(g.u_val + 9 * (size_t)u, xj[0], c3);
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
#pragma unroll
                for (int o = 1; o < kSpG; o <<= 1) c3[q] += __shfl_xor_sync(0xffffffffu, c3[q], o, kSpG);
                acc[0][q] += c3[q];
            }
        }
        if (i < g.nfem && l == 0) row = g.nb + i;
    }
    if (row >= 0) {
        double x3[1][3];
        if (!kResidual) op.load(row, x3);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const size_t e = 3 * (size_t)row + q;
            if (kResidual) {
                const double r = b[e] - acc[0][q];
                y[e] = r;
                dot += r * r;
            } else {
                p[e] = x3[0][q];
                y[e] = acc[0][q];
                dot += x3[0][q] * acc[0][q];
            }
        }
    }
    double total;
    if (!grid_total(dot, part, ticket, total)) return;
    if (kResidual) {
        st->res2 = total;
        return;
    }
    // alpha = r.z / p.Ap; the r.z test is that of the current iterate (the reference stops after
    // this iteration's update), then the iteration cap
    st->iters = k;
    if (!(total > 0.0) || !isfinite(total)) {
        st->status = SGIPC_BREAKDOWN;
        st->halt = 1;
        return;
    }
    st->alpha = st->rz / total;
    if (crit == SGIPC_CRIT_RZ && fabs(st->rz) <= tol * st->rz0) st->stop = 1;
    else if (crit == SGIPC_CRIT_RZ && k + 1 >= max_iter) st->stop = 2;
}

// x += alpha p, r -= alpha Ap of iteration k; with the true-residual test also r.r and the stop.
// (The stop that the SpMV of this iteration set does not skip its update: st->iters tells.)
__global__ void __launch_bounds__(kGThreads) k_g_update(long long n, GState* st, const double* __restrict__ p,
                                                        const double* __restrict__ Ap, double* __restrict__ x,
                                                        double* __restrict__ r, int k, int crit, double tol,
                                                        int max_iter, double* part, unsigned int* ticket) {
    if (st->halt || st->iters != k) return;
    const long long i = (long long)blockIdx.x * kGThreads + threadIdx.x;
    double dot = 0.0;
    if (i < n) {
        const double alpha = st->alpha;
        x[i] += alpha * p[i];
        const double v = r[i] - alpha * Ap[i];
        r[i] = v;
        dot = v * v;
    }
    if (crit != SGIPC_CRIT_TRUE) return;
    double total;
    if (!grid_total(dot, part, ticket, total)) return;
    if (total <= tol * tol * st->bn2) st->stop = 1;
    else if (k + 1 >= max_iter) st->stop = 2;
}

// x = 0, r = b, b.b
__global__ void __launch_bounds__(kGThreads) k_g_init(long long n, GState* st, const double* __restrict__ b,
                                                      double* __restrict__ x, double* __restrict__ r, double* part,
                                                      unsigned int* ticket) {
    const long long i = (long long)blockIdx.x * kGThreads + threadIdx.x;
    double v = 0.0;
    if (i < n) {
        v = b[i];
        x[i] = 0.0;
        r[i] = v;
    }
    double total;
    if (!grid_total(v * v, part, ticket, total)) return;
    *st = GState{};
    st->bn2 = total;
}

// z = M^-1 r: the bodies' block Jacobi (12 x 12 inverses), the sum of the MAS levels on the FEM rows;
// r.z, and from it beta (or, at the start, r0.z0).  One thread per block row.
template <class M>
__global__ void __launch_bounds__(kGThreads) k_g_precond(int nb, int nfem, GState* st, const double* __restrict__ pinv,
                                                         const int* __restrict__ table, int L,
                                                         const M* __restrict__ Z, const double* __restrict__ r,
                                                         double* __restrict__ z, int start, double* part,
                                                         unsigned int* ticket) {
    if (!start && (st->stop || st->halt)) return;
    const int t = blockIdx.x * kGThreads + threadIdx.x;
    double zz[3] = {0.0, 0.0, 0.0}, dot = 0.0;
    if (t < nb) {
        const double* P = pinv + 144 * (size_t)(t / 4) + 36 * (t % 4);
        const double* rb = r + 12 * (size_t)(t / 4);
#pragma unroll
        for (int j = 0; j < 12; j++) {
            const double v = rb[j];
#pragma unroll
            for (int q = 0; q < 3; q++) zz[q] += P[12 * q + j] * v;
        }
    } else if (t < nb + nfem) {
        const int* tv = table + (size_t)(t - nb) * L;
        M s[3] = {0, 0, 0};
        for (int l = 0; l < L; l++) {
            const int c = tv[l];
#pragma unroll
            for (int q = 0; q < 3; q++) s[q] += Z[3 * (size_t)c + q];
        }
#pragma unroll
        for (int q = 0; q < 3; q++) zz[q] = (double)s[q];
    }
    if (t < nb + nfem)
#pragma unroll
        for (int q = 0; q < 3; q++) {
            z[3 * (size_t)t + q] = zz[q];
            dot += r[3 * (size_t)t + q] * zz[q];
        }
    double total;
    if (!grid_total(dot, part, ticket, total)) return;
    if (start) {
        const bool run = total > 0.0 && isfinite(total);
        st->rz0 = st->rz = total;
        st->halt = run ? 0 : 1;
        st->status = (!run && (!isfinite(total) || total < 0.0)) ? SGIPC_BREAKDOWN : SGIPC_OK;
    } else {
        st->beta = total / st->rz;
        st->rz = total;
    }
}

// dx of every ABD point: J(x_bar) dq of its body (translation + x_bar . da_r per row)
__global__ void k_g_point_dx(int P, const int* __restrict__ point_body, const double* __restrict__ x_bar,
                             const double* __restrict__ dq, double* __restrict__ dx) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const double* q = dq + 12 * (size_t)point_body[p];
    const double* xb = x_bar + 3 * (size_t)p;
    for (int r = 0; r < 3; r++)
        dx[3 * (size_t)p + r] = q[r] + xb[0] * q[3 + 3 * r] + xb[1] * q[4 + 3 * r] + xb[2] * q[5 + 3 * r];
}

template <class T>
SgipcStatus grow(SgipcCtx* f, T** p, size_t n) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    SG_CHECK(f, cudaMalloc((void**)p, sizeof(T) * (n > 0 ? n : 1)));
    return SGIPC_OK;
}

struct Global {
    SgipcCtx* f;
    SgipcAbdCtx* a;
    int nb;     // body block rows 4B
    int nfem;   // FEM block rows
    long long N;
    cudaStream_t s;
    int fp32_mas;
    GMat mat;
    GState* st;
    double* part;
    unsigned int* ticket;
};

int g_spmv_grid(int nb, int nfem) { return nblk(nb, kGBodyRows) + nblk(nfem, kGFemRows); }

// z = M^-1 r and the scalars that follow from r.z
SgipcStatus g_precond(const Global& g, const double* r, double* z, bool start) {
    const MasWork& m = g.f->mas;
    SgipcStatus st = mas_domains(g.f, r + 3 * (size_t)g.nb, g.fp32_mas, start ? nullptr : &g.st->stop, g.s);
    if (st != SGIPC_OK) return st;
    SG_COUNT(g.f, 1);
    const int grid = nblk((long long)g.nb + g.nfem, kGThreads);
    if (g.fp32_mas)
        k_g_precond<float><<<grid, kGThreads, 0, g.s>>>(g.nb, g.nfem, g.st, g.a->pinv, m.table, m.levelnum, m.Z32, r, z,
                                                        start, g.part, g.ticket);
    else
        k_g_precond<double><<<grid, kGThreads, 0, g.s>>>(g.nb, g.nfem, g.st, g.a->pinv, m.table, m.levelnum, m.Z64, r,
                                                         z, start, g.part, g.ticket);
    SG_LAUNCH_CHECK(g.f, "global preconditioner");
    return SGIPC_OK;
}

}  // namespace

extern "C" SgipcStatus sgipc_global_pcg_solve(SgipcCtx* f, SgipcAbdCtx* a, SgipcCriterion crit, double tol,
                                              int32_t max_iter, const double* b, double* x, double* abd_point_dx,
                                              SgipcSolveStats* stats, void* stream) {
    if (!f || !a || !b || !x || !(tol >= 0.0)) return SGIPC_BAD_INPUT;
    if (crit != SGIPC_CRIT_RZ && crit != SGIPC_CRIT_TRUE) return SGIPC_BAD_INPUT;
    if (a->device != f->device) {
        snprintf(f->err, sizeof(f->err), "global solve: the FEM and ABD contexts live on different devices");
        return SGIPC_BAD_INPUT;
    }
    if (!f->assembled || !f->mas.built || !a->assembled || !a->pbuilt) {
        snprintf(f->err, sizeof(f->err), "global solve: assemble both systems and build both preconditioners first");
        return SGIPC_NOT_READY;
    }
    SG_DEVICE(f);
    Global g{f, a, 4 * a->B, f->n, 3LL * (4LL * a->B + f->n), (cudaStream_t)stream,
             f->mas.built == SGIPC_FP64 + 1 ? 0 : 1, {}, nullptr, nullptr, nullptr};
    if (g.N > 0x7fffffffLL) return SGIPC_CAPACITY;
    if (max_iter <= 0) max_iter = (int)(0.3 * (double)g.N);
    if (max_iter < 2) max_iter = 2;
    // ---- buffers (grown on demand) and the merged blocks' row / column index
    SgipcStatus st;
    const int ncols = g.nb + g.nfem, m = a->m_last;  // m: emitted slots, at least the unique blocks
    if (a->g_cap_blk < a->cap) {
        if ((st = grow(f, &a->g_tkey, a->cap)) || (st = grow(f, &a->g_tkey_s, a->cap)) ||
            (st = grow(f, &a->g_tidx, a->cap)) || (st = grow(f, &a->g_tidx_s, a->cap)))
            return st;
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, a->g_tkey, a->g_tkey_s, a->g_tidx, a->g_tidx_s, a->cap);
        if ((st = grow(f, (char**)&a->g_cub, tb))) return st;
        a->g_cub_bytes = tb;
        a->g_cap_blk = a->cap;
    }
    if (a->g_cap_ptr < ncols + 1) {
        if ((st = grow(f, &a->g_rptr, g.nb + 1)) || (st = grow(f, &a->g_cptr, ncols + 1))) return st;
        a->g_cap_ptr = ncols + 1;
    }
    if (a->g_cap_vec < (size_t)g.N) {
        const int parts = std::max(g_spmv_grid(g.nb, g.nfem), nblk(g.N, kGThreads));
        a->g_cap_vec = 0;
        if ((st = grow(f, &a->g_vec, 5 * (size_t)g.N)) || (st = grow(f, &a->g_part, parts)) ||
            (st = grow(f, &a->g_dot, 32)))
            return st;
        a->g_cap_vec = (size_t)g.N;
    }
    for (cudaEvent_t& e : a->g_ev)
        if (!e) SG_CHECK(f, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    int row_bits = 1, col_bits = 1;
    while ((1LL << row_bits) < g.nb) row_bits++;
    while ((1LL << col_bits) <= ncols) col_bits++;  // all ones stays above every column
    SG_COUNT(f, 3);
    k_g_rowptr<<<nblk(g.nb + 1), SGIPC_BLOCK, 0, g.s>>>(g.nb, a->nu, a->u_row, a->g_rptr);
    k_g_tkeys<<<nblk(m), SGIPC_BLOCK, 0, g.s>>>(m, row_bits, ncols, a->nu, a->u_row, a->u_col, a->g_tkey, a->g_tidx);
    size_t tb = a->g_cub_bytes;
    SG_CHECK(f, cub::DeviceRadixSort::SortPairs(a->g_cub, tb, a->g_tkey, a->g_tkey_s, a->g_tidx, a->g_tidx_s, m, 0,
                                                row_bits + col_bits, g.s));
    k_g_colptr<<<nblk(ncols + 1), SGIPC_BLOCK, 0, g.s>>>(ncols, m, row_bits, a->g_tkey_s, a->g_cptr);
    SG_LAUNCH_CHECK(f, "global index");

    // ---- PCG (PCGSolver::pcg semantics, as the persistent FEM solve)
    double* r = a->g_vec;
    double* z = r + g.N;
    double* p[2] = {z + g.N, z + 2 * g.N};
    double* Ap = z + 3 * g.N;
    const int gb = nblk(g.N, kGThreads), gs = g_spmv_grid(g.nb, g.nfem);
    g.st = reinterpret_cast<GState*>(a->g_dot);
    g.ticket = reinterpret_cast<unsigned int*>(a->g_dot + 24);
    g.part = a->g_part;
    g.mat = GMat{topo_of(f), mat_view<double>(f), g.nb, g.nfem, a->g_rptr, a->g_cptr, a->g_tidx_s, a->u_row, a->u_col,
                 a->u_val};
    GState* hs = reinterpret_cast<GState*>(f->h_pinned + 40);  // [2], pinned
    static_assert(2 * sizeof(GState) <= 24 * sizeof(double) && sizeof(GState) <= 24 * sizeof(double), "state slots");
    // state and ticket, in the caller's stream order (a plain cudaMemset runs on the default stream,
    // which a side stream does not wait for), and for every solve: one that left early on an error
    // leaves no ticket behind
    SG_CHECK(f, cudaMemsetAsync(a->g_dot, 0, sizeof(double) * 32, g.s));
    SG_COUNT(f, 1);
    k_g_init<<<gb, kGThreads, 0, g.s>>>(g.N, g.st, b, x, r, g.part, g.ticket);
    if ((st = g_precond(g, r, z, true))) return st;
    auto iterate = [&](int k) -> SgipcStatus {
        double* pn = p[k & 1];
        const double* po = k == 1 ? nullptr : p[(k + 1) & 1];
        SG_COUNT(f, 2);
        k_g_spmv<false><<<gs, kGThreads, 0, g.s>>>(g.mat, g.st, z, po, pn, Ap, nullptr, k, (int)crit, tol, max_iter,
                                                   g.part, g.ticket);
        k_g_update<<<gb, kGThreads, 0, g.s>>>(g.N, g.st, pn, Ap, x, r, k, (int)crit, tol, max_iter, g.part, g.ticket);
        SG_LAUNCH_CHECK(f, "global pcg");
        SG_CHECK(f, cudaMemcpyAsync(hs + (k & 1), g.st, sizeof(GState), cudaMemcpyDeviceToHost, g.s));
        SG_CHECK(f, cudaEventRecord(a->g_ev[k & 1], g.s));
        return g_precond(g, r, z, false);
    };
    // iteration k + 1 is enqueued before iteration k's state is awaited
    int k = 1;
    if ((st = iterate(1))) return st;
    for (;; k++) {
        const bool more = k + 1 < max_iter;
        if (more && (st = iterate(k + 1))) return st;
        SG_CHECK(f, cudaEventSynchronize(a->g_ev[k & 1]));
        if (hs[k & 1].halt || hs[k & 1].stop || !more) break;
    }
    const GState fin = hs[k & 1];
    int status = fin.status;
    // still running at the cap: not converged
    if (status == SGIPC_OK && !fin.halt && fin.stop != 1) status = SGIPC_NOT_CONVERGED;
    // ---- true residual, distribute_solution
    SG_COUNT(f, 1);
    k_g_spmv<true><<<gs, kGThreads, 0, g.s>>>(g.mat, g.st, x, nullptr, nullptr, Ap, b, 0, 0, 0.0, 0, g.part, g.ticket);
    SG_CHECK(f, cudaMemcpyAsync(hs, g.st, sizeof(GState), cudaMemcpyDeviceToHost, g.s));
    if (abd_point_dx && a->P > 0) {
        SG_COUNT(f, 1);
        k_g_point_dx<<<nblk(a->P), SGIPC_BLOCK, 0, g.s>>>(a->P, a->point_body, a->x_bar, x, abd_point_dx);
    }
    SG_LAUNCH_CHECK(f, "global residual, abd point dx");
    SG_CHECK(f, cudaStreamSynchronize(g.s));
    const double res2 = hs->res2, bn2 = fin.bn2;
    const double rel = bn2 > 0 ? std::sqrt(res2 / bn2) : std::sqrt(res2);
    const double rz0 = fin.rz0, rz = fin.rz;
    const int iters = fin.iters;
    if (stats) {
        *stats = SgipcSolveStats{};
        stats->iterations = iters;
        stats->rz0 = rz0;
        stats->rz = rz;
        stats->rel_residual = rel;
        stats->status = status;
    }
    return (SgipcStatus)status;
}
