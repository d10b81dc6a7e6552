// sgipc_assemble.cu — gradient and Hessian assembly of one Newton iteration.
//
// Follows GIPC::computeGradientAndHessian (StiffGIPC/GIPC.cu:10110-10344):
//   kinetic gradient M(x - x~)                          GIPC.cu:6339
//   IPC barrier, RANK 2, Gauss-Newton Hessian            GIPC.cu:3106-4945
//   lagged smoothed friction (pairs and ground)          GIPC.cu:1357-1800, 5047-5270
//   ground barrier, soft constraints                     GIPC.cu:6363-6514
//   stable Neo-Hookean tets with the analytic projection femEnergy.cu:1593-1857
//   Dirichlet zeroing, mass diagonal                     GIPC.cu:10295-10336
//   b = fb + shape_grads, Dirichlet rows zeroed          fem_linear_subsystem.cu:56-84
//
// Layout on the GPU (all FP64):
//   * static part: element kernels write oriented 3x3 blocks into per-element slots
//     (eblk) and per-vertex gradient rows (egrad); gather kernels sum them into the BSR
//     values and shape_grads through CSR lists built at context creation;
//   * dynamic part: a contact pair's blocks are products of a few vectors, so each pair stores
//     those (its factors, 128 B) instead of ten 3x3 blocks (840 B with their keys), and its
//     vertices are sorted once, one 32-bit key each.  A warp (or a CTA, for long lists) then
//     walks the pairs of one vertex in order, forms the blocks of that row and adds them up in
//     shared memory: the unique blocks row-sorted, the transposed lists that the SpMV reads
//     without atomics, and the contact gradient, all in a fixed order.  (Sorting the blocks
//     themselves under 64-bit keys and summing the runs moved 4 GB for the million pairs of a
//     256^2 rolled cloth: 3.3 ms of kernels.)
#include <algorithm>
#include <cmath>

#include <cub/cub.cuh>

#include "sgipc_internal.cuh"

using namespace sgipc;

namespace {

// ------------------------------------------------------------------------------------------
// kinetic gradient, reset of the contact gradient
// ------------------------------------------------------------------------------------------
__global__ void k_kinetic(int nv, const double* __restrict__ x, const double* __restrict__ xt,
                          const double* __restrict__ m, double* __restrict__ shape_grads, double* __restrict__ fb) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * nv) return;
    shape_grads[i] = m[i / 3] * (x[i] - xt[i]);
    fb[i] = 0.0;
}

// ------------------------------------------------------------------------------------------
// stable Neo-Hookean tet (USE_SNK1): PK1 femEnergy.cu:432-459, eigensystem 1593-1717
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_snk(int nt, const uint32_t* __restrict__ tets, const double* __restrict__ x,
                                             const double* __restrict__ dminv, const double* __restrict__ vol,
                                             const double* __restrict__ lr, const double* __restrict__ vr, double dt2,
                                             double* __restrict__ eblk, double* __restrict__ egrad) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    uint4 tv = reinterpret_cast<const uint4*>(tets)[t];
    const uint32_t vid[4] = {tv.x, tv.y, tv.z, tv.w};
    d3 X0 = ld3(x, tv.x), X1 = ld3(x, tv.y), X2 = ld3(x, tv.z), X3 = ld3(x, tv.w);
    double Di[3][3];
#pragma unroll
    for (int k = 0; k < 9; k++) Di[k / 3][k % 3] = dminv[9 * (size_t)t + k];
    const double mu = lr[t], lam = vr[t], sc = dt2 * vol[t];
    d3 e1 = X1 - X0, e2 = X2 - X0, e3 = X3 - X0;
    double F[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        double a = comp(e1, i), b = comp(e2, i), c = comp(e3, i);
#pragma unroll
        for (int j = 0; j < 3; j++) F[i][j] = a * Di[0][j] + b * Di[1][j] + c * Di[2][j];
    }
    d3 f0 = mk(F[0][0], F[1][0], F[2][0]), f1 = mk(F[0][1], F[1][1], F[2][1]), f2 = mk(F[0][2], F[1][2], F[2][2]);
    d3 g0 = cross(f1, f2), g1 = cross(f2, f0), g2 = cross(f0, f1);
    const double J = dot(f0, g0);
    const double ev = lam * (J - 1.0) - mu;  // evScale of the twist/flip pairs
    // P = mu F + (lam (J - 1) - mu) cof(F); gradient rows G = P Dm^-T
    d3 P0 = mu * f0 + ev * g0, P1 = mu * f1 + ev * g1, P2 = mu * f2 + ev * g2;
    d3 gr[4];
#pragma unroll
    for (int k = 0; k < 3; k++) gr[k + 1] = sc * (Di[k][0] * P0 + Di[k][1] * P1 + Di[k][2] * P2);
    gr[0] = -(gr[1] + gr[2] + gr[3]);
#pragma unroll
    for (int a = 0; a < 4; a++) {
        double* o = egrad + 3 * (4 * (size_t)t + a);
        o[0] = gr[a].x;
        o[1] = gr[a].y;
        o[2] = gr[a].z;
    }
    // analytic eigensystem of d2Psi/dF2 (Smith et al., "Analytic eigensystems for isotropic
    // distortion energies"): twist/flip pairs per axis plus a 3x3 scaling block
    double U[3][3], S[3], V[3][3];
    svd3_rv(F, U, S, V);
    double c1[3], c2[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        double lt = fmax(mu + ev * S[k], 0.0), lf = fmax(mu - ev * S[k], 0.0);
        c1[k] = 0.5 * (lt + lf);
        c2[k] = 0.5 * (lf - lt);
    }
    double A[3][3], Q[3][3];
    const double es = lam * (2.0 * J - 1.0) - mu;
    A[0][0] = mu + lam * S[1] * S[1] * S[2] * S[2];
    A[1][1] = mu + lam * S[0] * S[0] * S[2] * S[2];
    A[2][2] = mu + lam * S[0] * S[0] * S[1] * S[1];
    A[0][1] = A[1][0] = es * S[2];
    A[0][2] = A[2][0] = es * S[1];
    A[1][2] = A[2][1] = es * S[0];
    sym_eig3(A, Q);
    double Sp[3][3];
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = 0; q < 3; q++) {
            double s = 0;
#pragma unroll
            for (int m = 0; m < 3; m++) s += fmax(A[m][m], 0.0) * Q[p][m] * Q[q][m];
            Sp[p][q] = s;
        }
    // d_a = V^T D(a,:)^T with D the rows of dF/dx
    double d[4][3];
#pragma unroll
    for (int p = 0; p < 3; p++) {
        double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double v = V[j][p];
            s1 += v * Di[0][j];
            s2 += v * Di[1][j];
            s3 += v * Di[2][j];
        }
        s0 = -(s1 + s2 + s3);
        d[0][p] = s0;
        d[1][p] = s1;
        d[2][p] = s2;
        d[3][p] = s3;
    }
    const int pa[10] = {0, 0, 0, 0, 1, 1, 1, 2, 2, 3};
    const int pb[10] = {0, 1, 2, 3, 1, 2, 3, 2, 3, 3};
    const int ax_i[3] = {1, 0, 0}, ax_j[3] = {2, 2, 1};
    // (unrolled: the vertex pair of each block is then a compile-time index into d, which a
    // rolled loop kept in local memory; 168 registers, measured 4 % faster than rolled)
#pragma unroll
    for (int k = 0; k < 10; k++) {
        const int a = pa[k], b = pb[k];
        double K[3][3];
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) K[p][q] = Sp[p][q] * d[a][p] * d[b][q];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const int i = ax_i[m], j = ax_j[m];
            K[j][j] += c1[m] * d[a][i] * d[b][i];
            K[i][i] += c1[m] * d[a][j] * d[b][j];
            K[j][i] += c2[m] * d[a][i] * d[b][j];
            K[i][j] += c2[m] * d[a][j] * d[b][i];
        }
        // H = sc * U K U^T, written transposed when the element's vertex order is reversed
        double UK[3][3];
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) UK[p][q] = U[p][0] * K[0][q] + U[p][1] * K[1][q] + U[p][2] * K[2][q];
        const bool tr = vid[a] > vid[b];
        double* o = eblk + 9 * (10 * (size_t)t + k);
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                double h = sc * (UK[p][0] * U[q][0] + UK[p][1] * U[q][1] + UK[p][2] * U[q][2]);
                o[tr ? (3 * q + p) : (3 * p + q)] = h;
            }
    }
}

// ------------------------------------------------------------------------------------------
// cloth membrane: Baraff-Witkin stretch + shear (femEnergy.cu:351-403 stress, 535-707 the
// two projected Hessians, 2146-2215 the element kernel).  F = Ds Dm^-1 (3x2), columns
// f0, f1.  Energy density k_st (S(|f0|) + S(|f1|)) + k_sh (f0.f1)^2 with
// S(t) = (t-1)^2 + [t > 1] s (t-1)^3, times area*thickness*dt^2.  The reference projects
// the stretch and the shear Hessian separately and sums them; both projections have closed
// forms used here:
//   stretch, per column (n = f/t):  [t > 1] S'(t)/t (I - n n^T) + c n n^T, with
//     c = S''(t) for t > 1 and 2 otherwise (the negative transverse part clamped);
//   shear, E = I6^2 with I6 = f0.f1, g = [f1; f0], a = [f0; f1], swap S = [[0,I],[I,0]]:
//     the exact Hessian 2(g g^T + I6 S) has, in span{a, g}, the eigenpair
//     2 lambda0 with q ~ I6 a + lambda0 g, lambda0 = (I2 + sqrt(I2^2 + 12 I6^2)) / 2, and in
//     the complement +-2|I6| on the eigenspaces of S; the projection keeps
//     2 lambda0 q q^T + |I6| [[Pw, sg Pw], [sg Pw, Pw]], sg = sign(I6) (+1 at 0),
//     Pw = I - w w^T / |w|^2, w = f0 + sg f1 (the part of the sg-eigenspace outside span{a,g}).
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_tri_bw(int nf, const uint32_t* __restrict__ tris, const double* __restrict__ x,
                                                const double* __restrict__ dminv, const double* __restrict__ area,
                                                double kst, double ksh, double srate, double dt2, int eoff, int goff,
                                                double* __restrict__ eblk, double* __restrict__ egrad) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    int vid[3];
#pragma unroll
    for (int a = 0; a < 3; a++) vid[a] = (int)tris[3 * f + a];
    const d3 x0 = ld3(x, vid[0]), e1 = ld3(x, vid[1]) - x0, e2 = ld3(x, vid[2]) - x0;
    const double* Di = dminv + 4 * (size_t)f;  // row-major 2x2
    const d3 col[2] = {Di[0] * e1 + Di[2] * e2, Di[1] * e1 + Di[3] * e2};
    // dF(:,j)/dx_a = D[a][j] I
    const double D[3][2] = {{-(Di[0] + Di[2]), -(Di[1] + Di[3])}, {Di[0], Di[1]}, {Di[2], Di[3]}};
    const double scale = area[f] * dt2;

    // stress P (columns) and the 6x6 projected Hessian as 3x3 blocks Hq[j][k]
    d3 P[2];
    double Hq[2][2][3][3];
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
                for (int q = 0; q < 3; q++) Hq[j][k][p][q] = 0.0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const d3 fj = col[j];
        const double t = sqrt(sq(fj));
        const double u = t - 1.0;
        const double dS = 2.0 * u + (t > 1.0 ? 3.0 * srate * u * u : 0.0);
        P[j] = (kst * dS / t) * fj;
        const double ct = t > 1.0 ? dS / t : 0.0;                    // transverse (clamped)
        const double cn = t > 1.0 ? 2.0 + 6.0 * srate * u : 2.0;     // along n
        const double n[3] = {fj.x / t, fj.y / t, fj.z / t};
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++)
                Hq[j][j][p][q] += kst * ((p == q ? ct : 0.0) + (cn - ct) * n[p] * n[q]);
    }
    {
        const d3 f0 = col[0], f1 = col[1];
        const double I6 = dot(f0, f1), I2 = sq(f0) + sq(f1);
        P[0] = P[0] + (2.0 * ksh * I6) * f1;
        P[1] = P[1] + (2.0 * ksh * I6) * f0;
        const double lam0 = 0.5 * (I2 + sqrt(I2 * I2 + 12.0 * I6 * I6));
        const d3 qa = I6 * f0 + lam0 * f1, qb = I6 * f1 + lam0 * f0;  // q = [qa; qb] unnormalised
        const double qn = sq(qa) + sq(qb);
        const double iq = qn > 0.0 ? 1.0 / qn : 0.0;
        const double sg = I6 >= 0.0 ? 1.0 : -1.0;
        const d3 w = f0 + sg * f1;
        const double ww = sq(w);
        const double iw = ww > 0.0 ? 1.0 / ww : 0.0;
        const double q0[2][3] = {{qa.x, qa.y, qa.z}, {qb.x, qb.y, qb.z}};
        const double wv[3] = {w.x, w.y, w.z};
        const double aI6 = fabs(I6);
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double s = j == k ? 1.0 : sg;
#pragma unroll
                for (int p = 0; p < 3; p++)
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        const double Pw = (p == q ? 1.0 : 0.0) - wv[p] * wv[q] * iw;
                        Hq[j][k][p][q] += ksh * (2.0 * lam0 * q0[j][p] * q0[k][q] * iq + aI6 * s * Pw);
                    }
            }
    }
    // gradient rows and the 6 oriented upper blocks
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const d3 g = scale * (D[a][0] * P[0] + D[a][1] * P[1]);
        double* o = egrad + 3 * ((size_t)goff + 3 * (size_t)f + a);
        o[0] = g.x;
        o[1] = g.y;
        o[2] = g.z;
    }
    const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const int a = pa[k], b = pb[k];
        const bool tr = vid[a] > vid[b];
        double* o = eblk + 9 * ((size_t)eoff + 6 * (size_t)f + k);
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                double h = 0.0;
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int l = 0; l < 2; l++) h += D[a][j] * D[b][l] * Hq[j][l][p][q];
                o[tr ? (3 * q + p) : (3 * p + q)] = scale * h;
            }
    }
}

// ------------------------------------------------------------------------------------------
// quadratic bending (femEnergy.cu:2623-2753; Q from the rest shape, :2492-2618): per
// interior edge with vertices [e0, e1, opposite of triangle 1, opposite of triangle 2],
// E = 1/2 c x^T (Q (x) I3) x, c = |rest e0 - rest e1| * bendStiff * dt^2: gradient c Q x,
// constant Hessian c Q (x) I3.  Boundary edges (no second triangle) contribute nothing.  A block
// c Q(a,b) I3 is stored as its one number (hblk, 10 per hinge; k_gather_blocks puts it on the
// diagonal): as 3x3 blocks the 195 000 hinges of a 256^2 cloth were 140 MB to write and read.
// ------------------------------------------------------------------------------------------
__global__ void k_hinge_quad(int nh, const uint32_t* __restrict__ edges, const int32_t* __restrict__ adj,
                             const double* __restrict__ x, const double* __restrict__ rest,
                             const double* __restrict__ Qcm, double kb_dt2, int goff,
                             double* __restrict__ hblk, double* __restrict__ egrad) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nh) return;
    const int v[4] = {(int)edges[2 * h], (int)edges[2 * h + 1], adj[2 * h], adj[2 * h + 1]};
    const bool boundary = v[2] < 0 || v[3] < 0;
    double Q[4][4];
    double c = 0.0;
    if (!boundary) {
        c = sqrt(sq(ld3(rest, v[0]) - ld3(rest, v[1]))) * kb_dt2;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) Q[i][j] = Qcm[16 * (size_t)h + 4 * j + i];  // column-major
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) Q[i][j] = 0.0;
    }
    d3 xv[4];
#pragma unroll
    for (int a = 0; a < 4; a++) xv[a] = boundary ? mk(0, 0, 0) : ld3(x, v[a]);
#pragma unroll
    for (int a = 0; a < 4; a++) {
        d3 g = mk(0, 0, 0);
#pragma unroll
        for (int b = 0; b < 4; b++) g = g + (c * Q[a][b]) * xv[b];
        double* o = egrad + 3 * ((size_t)goff + 4 * (size_t)h + a);
        o[0] = g.x;
        o[1] = g.y;
        o[2] = g.z;
    }
    const int pa[10] = {0, 0, 0, 0, 1, 1, 1, 2, 2, 3}, pb[10] = {0, 1, 2, 3, 1, 2, 3, 2, 3, 3};
    double d[10];
#pragma unroll
    for (int k = 0; k < 10; k++) {
        // block (a, b) is that of (min, max): from Q(b,a) when the element's order is reversed
        const bool tr = v[pa[k]] > v[pb[k]];
        d[k] = c * (tr ? Q[pb[k]][pa[k]] : Q[pa[k]][pb[k]]);
    }
    double2* o = reinterpret_cast<double2*>(hblk + 10 * (size_t)h);
#pragma unroll
    for (int k = 0; k < 5; k++) o[k] = make_double2(d[2 * k], d[2 * k + 1]);
}

// ------------------------------------------------------------------------------------------
// static gathers
// ------------------------------------------------------------------------------------------
struct StaticOut {
    double* v64;       // upper slots (the MAS scatter and the BCOO export read these)
    const int* fup;    // full-pattern index of each upper slot
    const int* flo;    // full-pattern index of its transpose (-1 on the diagonal)
    double* f64;       // full symmetric copy
    float* f32;
};

// kHinges: contributions from hfirst on are hinges (without any, their test cost the tets' gather 15 %)
template <bool kHinges>
__global__ void k_gather_blocks(int nnz, const int* __restrict__ cptr, const int* __restrict__ contrib,
                                const double* __restrict__ eblk, const double* __restrict__ hblk, int hfirst,
                                const int* __restrict__ slot_row, const int* __restrict__ col, const int32_t* __restrict__ btype,
                                const double* __restrict__ mass, StaticOut o) {
    long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= 9LL * nnz) return;
    int s = (int)(tid / 9), q = (int)(tid % 9);
    int r = slot_row[s], c = col[s];
    const int k0 = cptr[s], k1 = cptr[s + 1];
    // the contributions four at a time, their index and value loads issued together (one by
    // one, each waited out two L2 round trips), added in list order as before; the boundary
    // test is applied after the loads
    const bool diag = q % 4 == 0;  // a hinge's block is a multiple of the identity
    auto entry = [&](int i) -> double {
        if (!kHinges || i < hfirst) return eblk[9 * (size_t)i + q];
        return diag ? hblk[i - hfirst] : 0.0;
    };
    double acc = 0.0;
    int k = k0;
    for (; k + 4 <= k1; k += 4) {
        int ix[4];
#pragma unroll
        for (int u = 0; u < 4; u++) ix[u] = contrib[k + u];
        double e[4];
#pragma unroll
        for (int u = 0; u < 4; u++) e[u] = entry(ix[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) acc += e[u];
    }
    for (; k < k1; k++) acc += entry(contrib[k]);
    if (btype[r] != 0 || btype[c] != 0) acc = 0.0;
    if (r == c && (q == 0 || q == 4 || q == 8)) acc += mass[r];
    o.v64[tid] = acc;
    const size_t fu = 9 * (size_t)o.fup[s] + q;
    o.f64[fu] = acc;
    o.f32[fu] = (float)acc;
    const int fl = o.flo[s];
    if (fl >= 0) {
        const size_t ft = 9 * (size_t)fl + 3 * (q % 3) + q / 3;
        o.f64[ft] = acc;
        o.f32[ft] = (float)acc;
    }
}

static StaticOut static_out(SgipcCtx* c) {
    StaticOut o;
    o.v64 = c->val64;
    o.fup = c->fup;
    o.flo = c->flo;
    o.f64 = c->fval64;
    o.f32 = c->fval32;
    return o;
}

__global__ void k_gather_grad(int nv, const int* __restrict__ vptr, const int* __restrict__ vinc,
                              const double* __restrict__ egrad, double* __restrict__ shape_grads) {
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= 3 * nv) return;
    int v = tid / 3, q = tid % 3;
    const int k0 = vptr[v], k1 = vptr[v + 1];
    double acc = 0.0;
    int k = k0;
    for (; k + 4 <= k1; k += 4) {  // four incident elements in flight, added in list order
        int ix[4];
#pragma unroll
        for (int u = 0; u < 4; u++) ix[u] = vinc[k + u];
        double e[4];
#pragma unroll
        for (int u = 0; u < 4; u++) e[u] = egrad[3 * (size_t)ix[u] + q];
#pragma unroll
        for (int u = 0; u < 4; u++) acc += e[u];
    }
    for (; k < k1; k++) acc += egrad[3 * (size_t)vinc[k] + q];
    shape_grads[tid] += acc;
}

__global__ void k_rhs(int nv, const double* __restrict__ fb, const double* __restrict__ sg,
                      const int32_t* __restrict__ btype, double* __restrict__ b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * nv) return;
    b[i] = btype[i / 3] != 0 ? 0.0 : fb[i] + sg[i];
}

// ------------------------------------------------------------------------------------------
// contact blocks
// ------------------------------------------------------------------------------------------
// A pair's factors, kFac doubles (one 128-byte line):
//   barrier   [0] lam, [1..12] g (four vertices), [13] s:   block (a, b) = lam g_a g_b^T, gradient s g_a
//   friction  [0..8] W, [9..12] c, [13..15] t:              block (a, b) = c_a c_b W,     gradient c_a t
//   mollified [0] M11, [1..12] gf, [13] df, [14] M01, and a second line [0] M00, [1..12] gc, [13] dc:
//             block (a, b) = M00 gc_a gc_b^T + M01 (gc_a gf_b^T + gf_a gc_b^T) + M11 gf_a gf_b^T,
//             gradient dc gc_a + df gf_a
// (a before b in the pair's order; the block of a vertex pair in the other order is its
// transpose).  Ground contacts and soft constraints ("singles") store their 3x3 block.
constexpr int kFac = 16;
constexpr int kMollBit = 1 << 30;  // in vertex 0 of a mollified pair's ids
constexpr int kTwiceBit = 1 << 29;  // ... of a pair that names a vertex twice (a mesh has far fewer vertices)
constexpr int kIdMask = ~(kMollBit | kTwiceBit);
struct ContactStore {
    int4* ids;         // [pairs] vertices, -1 where a pair has fewer (all -1: no blocks)
    double* fac;       // [kFac * pairs]
    double* fac2;      // [kFac * barrier pairs] second line of the mollified ones
    int* sid;          // [singles] vertex, -1: none
    double* sval;      // [9 * singles]
    uint32_t* key;     // [4 * pairs + singles] vertex of each incidence 4 pair + a, or 4 pairs + single; n: none
    uint32_t* val;     // the incidence itself
    int pairs, barrier_pairs, n;
    int nv;
    int* flag;         // set to 1 when a pair names a vertex outside [0, nv)
};

__device__ __forceinline__ bool ids_ok(const ContactStore& cs, const int* v, int n) {
    for (int a = 0; a < n; a++)
        if (v[a] < 0 || v[a] >= cs.nv) {
            atomicOr(cs.flag, 1);
            return false;
        }
    return true;
}

// vertices and incidence keys of pair `item` (nvp of them in use; 0: no blocks)
__device__ __forceinline__ void store_ids(const ContactStore& cs, int item, int nvp, const int* v, bool moll) {
    int id[4];
    uint32_t k[4];
#pragma unroll
    for (int a = 0; a < 4; a++) {
        id[a] = a < nvp ? v[a] : -1;
        k[a] = a < nvp ? (uint32_t)v[a] : (uint32_t)cs.n;
    }
    bool twice = false;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = a + 1; b < 4; b++) twice |= b < nvp && v[a] == v[b];
    if (moll && nvp > 0) id[0] |= kMollBit;
    if (twice) id[0] |= kTwiceBit;
    cs.ids[item] = make_int4(id[0], id[1], id[2], id[3]);
    reinterpret_cast<uint4*>(cs.key)[item] = make_uint4(k[0], k[1], k[2], k[3]);
    const uint32_t o = 4u * (uint32_t)item;
    reinterpret_cast<uint4*>(cs.val)[item] = make_uint4(o, o + 1, o + 2, o + 3);
}

__device__ __forceinline__ void store_single(const ContactStore& cs, int j, int v, const double (&H)[3][3]) {
    const int o = 4 * cs.pairs + j;
    cs.sid[j] = v;
    cs.key[o] = v >= 0 ? (uint32_t)v : (uint32_t)cs.n;
    cs.val[o] = (uint32_t)o;
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = 0; q < 3; q++) cs.sval[9 * (size_t)j + 3 * p + q] = H[p][q];
}

// Entry (p, q) of a pair's block at (row vertex a, column vertex b): the product is formed with
// the pair's earlier vertex first, so that the blocks (a, b) and (b, a) are exact transposes.
// f: the pair's factors, f2: the second line (mollified pairs).
// kPairApart: added to the type of the rare pairs that the row sums take one after another.
enum PairType { kPairBarrier = 0, kPairFriction = 1, kPairMollified = 2, kPairSingle = 3, kPairApart = 4 };
__device__ __forceinline__ double pair_entry(int type, const double* f, const double* f2, int a, int b, int p, int q) {
    if (a > b) {
        const int t = a, u = p;
        a = b, b = t;
        p = q, q = u;
    }
    if (type == kPairBarrier) return f[0] * (f[1 + 3 * a + p] * f[1 + 3 * b + q]);
    if (type == kPairFriction) return f[9 + a] * f[9 + b] * f[3 * p + q];
    const double *gf = f + 1, *gc = f2 + 1;
    return f2[0] * gc[3 * a + p] * gc[3 * b + q] +
           f[14] * (gc[3 * a + p] * gf[3 * b + q] + gf[3 * a + p] * gc[3 * b + q]) +
           f[0] * gf[3 * a + p] * gf[3 * b + q];
}
__device__ __forceinline__ double pair_grad(int type, const double* f, const double* f2, int a, int q) {
    if (type == kPairBarrier) return f[13] * f[1 + 3 * a + q];
    if (type == kPairFriction) return f[9 + a] * f[13 + q];
    return f2[13] * f2[1 + 3 * a + q] + f[13] * f[1 + 3 * a + q];
}

// Decoded barrier pair: kind 0 PP, 1 PE, 2 PT, 3 EE, 4 mollified EE, 5 mollified PE,
// 6 mollified PP (encoding of StiffGIPC/mlbvh.cu:560-1059, decoded as GIPC.cu:3131-4945)
__device__ __forceinline__ int decode_pair(int4 e, int* v, int& nvp) {
    if (e.x >= 0) {
        v[0] = e.x; v[1] = e.y; v[2] = e.z;
        if (e.w >= 0) { v[3] = e.w; nvp = 4; return 3; }
        v[3] = -e.w - 1; nvp = 4; return 4;
    }
    v[0] = -e.x - 1;
    if (e.z < 0) {
        if (e.y < 0) { v[1] = -e.y - 1; v[2] = -e.z - 1; v[3] = -e.w - 1; nvp = 4; return 6; }
        v[1] = e.y; v[2] = v[3] = 0; nvp = 2; return 0;
    }
    if (e.w < 0) {
        if (e.y < 0) { v[1] = -e.y - 1; v[2] = e.z; v[3] = -e.w - 1; nvp = 4; return 5; }
        v[1] = e.y; v[2] = e.z; v[3] = 0; nvp = 3; return 1;
    }
    v[1] = e.y; v[2] = e.z; v[3] = e.w; nvp = 4; return 2;
}

// squared distance and its gradient (hand-derived, see the derivation in each branch)
__device__ __forceinline__ double dist2_grad(int kind, const d3* X, d3* g) {
    if (kind == 0 || kind == 6) {  // |a - b|^2
        d3 d = X[0] - X[1];
        g[0] = 2.0 * d;
        g[1] = -2.0 * d;
        g[2] = g[3] = mk(0, 0, 0);
        return sq(d);
    }
    if (kind == 1 || kind == 5) {  // |(e0-p) x (e1-p)|^2 / |e1-e0|^2
        d3 p = X[0], e0 = X[1], e1 = X[2];
        d3 c = cross(e0 - p, e1 - p), e = e1 - e0;
        double L = sq(e), C = sq(c);
        d3 gp = 2.0 * cross(c, e), ge0 = 2.0 * cross(e1 - p, c), ge1 = 2.0 * cross(c, e0 - p);
        double iL = 1.0 / L, r = C * iL * iL;
        g[0] = iL * gp;
        g[1] = iL * ge0 + (2.0 * r) * e;
        g[2] = iL * ge1 - (2.0 * r) * e;
        g[3] = mk(0, 0, 0);
        return C * iL;
    }
    if (kind == 2) {  // s^2 / |n|^2, n = (t1-t0) x (t2-t0), s = (p - t0).n
        d3 p = X[0], t0 = X[1], t1 = X[2], t2 = X[3];
        d3 e1 = t1 - t0, e2 = t2 - t0, w = p - t0;
        d3 n = cross(e1, e2);
        double s = dot(w, n), N = sq(n), iN = 1.0 / N;
        d3 sp = n, s0 = cross(e1 - e2, w) - n, s1 = cross(e2, w), s2 = cross(w, e1);
        d3 N0 = 2.0 * cross(e1 - e2, n), N1 = 2.0 * cross(e2, n), N2 = 2.0 * cross(n, e1);
        double a = 2.0 * s * iN, b = s * s * iN * iN;
        g[0] = a * sp;
        g[1] = a * s0 - b * N0;
        g[2] = a * s1 - b * N1;
        g[3] = a * s2 - b * N2;
        return s * s * iN;
    }
    // EE: s^2/|n|^2, n = (a1-a0) x (b1-b0), s = (b0 - a0).n
    d3 a0 = X[0], a1 = X[1], b0 = X[2], b1 = X[3];
    d3 u = a1 - a0, v = b1 - b0, w = b0 - a0;
    d3 n = cross(u, v);
    double s = dot(w, n), N = sq(n), iN = 1.0 / N;
    d3 vw = cross(v, w), wu = cross(w, u), vn = cross(v, n), nu = cross(n, u);
    double a = 2.0 * s * iN, b = s * s * iN * iN;
    g[0] = a * (-1.0 * n - vw) + (2.0 * b) * vn;
    g[1] = a * vw - (2.0 * b) * vn;
    g[2] = a * (n - wu) + (2.0 * b) * nu;
    g[3] = a * wu - (2.0 * b) * nu;
    return s * s * iN;
}

// B(I) = c (I-1)^2 ln(I)^2 and its first two derivatives in I
__device__ __forceinline__ void barrier_s(double I, double c, double& B, double& dB, double& d2B) {
    double L = log(I), t = I - 1.0;
    B = c * t * t * L * L;
    dB = c * (2.0 * t * L * L + 2.0 * t * t * L / I);
    d2B = c * (2.0 * L * L + 8.0 * t * L / I + 2.0 * t * t * (1.0 - L) / (I * I));
}

__device__ __forceinline__ void set3(double* f, d3 v) { f[0] = v.x, f[1] = v.y, f[2] = v.z; }

// item p's factors into f (the CTA's staging line); false: it has no blocks
__device__ __forceinline__ bool barrier_one(int p, const int4* __restrict__ pairs, const double* __restrict__ x,
                                            const double* __restrict__ rest, double dhat, double kappa,
                                            const ContactStore& cs, int item, double* f) {
    int v[4], nvp;
    int kind = decode_pair(pairs[p], v, nvp);
    if (!ids_ok(cs, v, nvp)) {
        store_ids(cs, item, 0, v, false);
        return false;
    }
    d3 X[4];
#pragma unroll
    for (int a = 0; a < 4; a++) X[a] = a < nvp ? ld3(x, v[a]) : mk(0, 0, 0);
    d3 gd2[4];
    double d2 = dist2_grad(kind, X, gd2);
    const double sdh = sqrt(dhat), dist = sqrt(d2);
    const double I = d2 / dhat, fr = sqrt(I);
    d3 gf[4];
#pragma unroll
    for (int a = 0; a < 4; a++) gf[a] = (1.0 / (2.0 * dist * sdh)) * gd2[a];
    if (kind <= 3) {
        double B, dB, d2B;
        barrier_s(I, kappa * dhat * dhat, B, dB, d2B);
        double dBdf = 2.0 * fr * dB;
        double Ic = d2 < 1e-6 * dhat ? 1e-6 : I;  // gassThreshold clamp (GIPC.cu:3258-3272)
        double Bc, dBc, d2Bc;
        barrier_s(Ic, kappa * dhat * dhat, Bc, dBc, d2Bc);
        double lam0 = 4.0 * Ic * d2Bc + 2.0 * dBc;
        store_ids(cs, item, nvp, v, false);
        f[0] = lam0;
#pragma unroll
        for (int a = 0; a < 4; a++) set3(f + 1 + 3 * a, gf[a]);
        f[13] = dBdf;
        f[14] = f[15] = 0.0;
        return true;
    }
    // mollified pairs: b = kappa e(c^2) Bt(I), c = |edge0 x edge1|
    int ea0, ea1, eb0, eb1;
    if (kind == 4) { ea0 = 0; ea1 = 1; eb0 = 2; eb1 = 3; }
    else if (kind == 6) { ea0 = 0; ea1 = 2; eb0 = 1; eb1 = 3; }
    else { ea0 = 0; ea1 = 3; eb0 = 1; eb1 = 2; }
    d3 u = X[ea1] - X[ea0], w = X[eb1] - X[eb0];
    d3 n = cross(u, w);
    double I1 = sq(n);
    if (I1 == 0.0) {
        store_ids(cs, item, 0, v, false);
        return false;
    }
    double c = sqrt(I1);
    d3 gc[4];
    {
        d3 wn = cross(w, n), nu = cross(n, u);
        double k = 1.0 / (2.0 * c);
        gc[ea0] = (-2.0 * k) * wn;
        gc[ea1] = (2.0 * k) * wn;
        gc[eb0] = (-2.0 * k) * nu;
        gc[eb1] = (2.0 * k) * nu;
    }
    d3 r0 = ld3(rest, v[ea0]), r1 = ld3(rest, v[ea1]), r2 = ld3(rest, v[eb0]), r3 = ld3(rest, v[eb1]);
    double ex = 1e-3 * sq(r0 - r1) * sq(r2 - r3);  // _compute_epx, mlbvh.cu:264
    double em = -I1 * I1 / (ex * ex) + 2.0 * I1 / ex;
    double dem = -2.0 * I1 / (ex * ex) + 2.0 / ex;
    double B, dB, d2B;
    barrier_s(I, dhat * dhat, B, dB, d2B);
    double dbdc = kappa * dem * 2.0 * c * B, dbdf = kappa * em * dB * 2.0 * fr;
    double M00 = kappa * B * (-4.0 * (3.0 * I1 - ex) / (ex * ex));
    double M11 = kappa * em * (4.0 * I * d2B + 2.0 * dB);
    double M01 = kappa * dem * 2.0 * c * dB * 2.0 * fr;
    make_pd2(M00, M01, M11);
    store_ids(cs, item, 4, v, true);
    f[0] = M11;
    f[13] = dbdf;
    f[14] = M01;
    f[15] = 0.0;
    double* f2 = cs.fac2 + kFac * (size_t)item;  // rare: straight to memory
    f2[0] = M00;
    f2[13] = dbdc;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        set3(f + 1 + 3 * a, gf[a]);
        set3(f2 + 1 + 3 * a, gc[a]);
    }
    return true;
}

// friction pairs (FrictionUtils.cuh, GIPC.cu:1439-1800 and 5087-5270), C1 static clamping
__device__ __forceinline__ bool friction_one(int p, const int4* __restrict__ pairs, const double* __restrict__ x,
                                             const double* __restrict__ x0, const double* __restrict__ lam,
                                             const double* __restrict__ coord, const double* __restrict__ basis,
                                             double mu, double eps2, const ContactStore& cs, int item, double* f) {
    int4 e = pairs[p];
    int v[4] = {0, 0, 0, 0}, nvp = 0;
    double cf[4] = {0, 0, 0, 0};
    double g1 = coord[2 * p], g2 = coord[2 * p + 1];
    if (e.x >= 0) {
        if (e.w >= 0) {
            v[0] = e.x; v[1] = e.y; v[2] = e.z; v[3] = e.w; nvp = 4;
            cf[0] = 1.0 - g1; cf[1] = g1; cf[2] = g2 - 1.0; cf[3] = -g2;
        }
    } else if (e.y >= 0) {
        v[0] = -e.x - 1;
        if (e.z < 0) { v[1] = e.y; nvp = 2; cf[0] = 1.0; cf[1] = -1.0; }
        else if (e.w < 0) { v[1] = e.y; v[2] = e.z; nvp = 3; cf[0] = 1.0; cf[1] = g1 - 1.0; cf[2] = -g1; }
        else { v[1] = e.y; v[2] = e.z; v[3] = e.w; nvp = 4; cf[0] = 1.0; cf[1] = -1.0 + g1 + g2; cf[2] = -g1; cf[3] = -g2; }
    }
    if (nvp == 0 || !ids_ok(cs, v, nvp)) {
        store_ids(cs, item, 0, v, false);
        return false;
    }
    const double* Tb = basis + 6 * (size_t)p;  // 3x2 row-major
    d3 t0 = mk(Tb[0], Tb[2], Tb[4]), t1 = mk(Tb[1], Tb[3], Tb[5]);
    d3 rel = mk(0, 0, 0);
    for (int a = 0; a < nvp; a++) rel = rel + cf[a] * (ld3(x, v[a]) - ld3(x0, v[a]));
    double u0 = dot(t0, rel), u1 = dot(t1, rel);
    double un2 = u0 * u0 + u1 * u1, un = sqrt(un2), eps = sqrt(eps2);
    double f1d, M00, M01, M11;
    if (un2 > eps2) {
        f1d = 1.0 / un;
        double k = 1.0 / (un2 * un);
        M00 = f1d - k * u0 * u0; M01 = -k * u0 * u1; M11 = f1d - k * u1 * u1;
    } else {
        f1d = (-un + 2.0 * eps) / (eps * eps);
        double f2 = 2.0 * (eps - un) / (eps * eps);
        if (f2 != f1d && un2 != 0.0) {
            double k = (f1d - f2) / un2;
            M00 = f1d - k * u0 * u0; M01 = -k * u0 * u1; M11 = f1d - k * u1 * u1;
        } else {
            M00 = M11 = f1d; M01 = 0.0;
        }
    }
    make_pd2(M00, M01, M11);
    const double s = mu * lam[p];
    d3 gt = (s * f1d) * (u0 * t0 + u1 * t1);
    store_ids(cs, item, nvp, v, false);
    // W = basis M basis^T
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (j < i) continue;
            double ti0 = comp(t0, i), ti1 = comp(t1, i), tj0 = comp(t0, j), tj1 = comp(t1, j);
            f[3 * i + j] = f[3 * j + i] = s * (ti0 * (M00 * tj0 + M01 * tj1) + ti1 * (M01 * tj0 + M11 * tj1));
        }
#pragma unroll
    for (int a = 0; a < 4; a++) f[9 + a] = cf[a];
    set3(f + 13, gt);
    return true;
}

// ground barrier (GIPC.cu:6463-6514), plane y = offset
__device__ __forceinline__ void ground_one(int p, const uint32_t* __restrict__ gp, const double* __restrict__ x,
                                           double offset, double dhat, double kappa, double* __restrict__ fb,
                                           const ContactStore& cs, int single) {
    int v = gp[p];
    double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    if (!ids_ok(cs, &v, 1)) {
        store_single(cs, single, -1, H);
        return;
    }
    double dist = x[3 * v + 1] - offset, d2 = dist * dist, t = d2 - dhat;
    double gb = t * log(d2 / dhat) * -2.0 - (t * t) / d2;
    double hb = (log(d2 / dhat) * -2.0 - t * 4.0 / d2) + 1.0 / (d2 * d2) * (t * t);
    atomicAdd(fb + 3 * v + 1, kappa * gb * 2.0 * dist);
    H[1][1] = kappa * (4.0 * hb * d2 + 2.0 * gb);
    store_single(cs, single, v, H);
}


// ground friction (GIPC.cu:1357-1437, 5047-5085), normal +y
__device__ __forceinline__ void fric_ground_one(int p, const uint32_t* __restrict__ gp, const double* __restrict__ x,
                                                const double* __restrict__ x0, const double* __restrict__ lam,
                                                double mu, double eps2, double* __restrict__ fb,
                                                const ContactStore& cs, int single) {
    int v = gp[p];
    double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    if (!ids_ok(cs, &v, 1)) {
        store_single(cs, single, -1, H);
        return;
    }
    double vx = x[3 * v] - x0[3 * v], vz = x[3 * v + 2] - x0[3 * v + 2];
    double m2 = vx * vx + vz * vz, s = mu * lam[p], eps = sqrt(eps2);
    if (m2 > eps2) {
        double m = sqrt(m2), k = s / (m2 * m);
        atomicAdd(fb + 3 * v, s * vx / m);
        atomicAdd(fb + 3 * v + 2, s * vz / m);
        double a = s / m - k * vx * vx, b = -k * vx * vz, c = s / m - k * vz * vz;
        make_pd2(a, b, c);
        H[0][0] = a; H[0][2] = b; H[2][0] = b; H[2][2] = c;
    } else {
        atomicAdd(fb + 3 * v, s * vx / eps);
        atomicAdd(fb + 3 * v + 2, s * vz / eps);
        H[0][0] = s / eps;
        H[2][2] = s / eps;
    }
    store_single(cs, single, v, H);
}


// All contact terms of a call in one launch: the CTAs take the barrier pairs, then the
// friction pairs, then the ground and the ground-friction vertices (128 threads each), so the
// four kinds run side by side instead of one after another.  The factors of a CTA's pairs are
// staged in shared memory and leave it as whole lines.  kGrad: the pairs' gradients are added
// into fb here, by atomics (callers that do not build the matrix); else k_row_sums adds them.
struct ContactLaunch {
    int np, nf, ng, ngf;           // items of each kind (0: none)
    int cb, cf, cg;                // first CTA of friction, ground, ground friction
    const int4* pairs;
    const int4* fpairs;
    const uint32_t* gpairs;
    const uint32_t* gfpairs;
    const double* x;
    const double* x0;
    const double* rest;
    const double* flam;
    const double* fcoord;
    const double* fbasis;
    const double* gflam;
    double dhat, kappa, mu, gmu, eps2, offset;
};

constexpr int kConThreads = 128;
template <bool kGrad>
__global__ void __launch_bounds__(kConThreads) k_contacts(ContactLaunch L, double* __restrict__ fb, ContactStore cs) {
    __shared__ double stage[kConThreads][kFac + 1];
    const int b = blockIdx.x, t = threadIdx.x;
    if (b >= L.cf) {  // CTA-uniform
        if (b < L.cg) {
            const int p = (b - L.cf) * kConThreads + t;
            if (p < L.ng) ground_one(p, L.gpairs, L.x, L.offset, L.dhat, L.kappa, fb, cs, p);
        } else {
            const int p = (b - L.cg) * kConThreads + t;
            if (p < L.ngf) fric_ground_one(p, L.gfpairs, L.x, L.x0, L.gflam, L.gmu, L.eps2, fb, cs, L.ng + p);
        }
        return;
    }
    const bool fric = b >= L.cb;
    const int p0 = (fric ? b - L.cb : b) * kConThreads, p = p0 + t, n = fric ? L.nf : L.np;
    const int item0 = (fric ? L.np : 0) + p0;
    bool on = false;
    if (p < n)
        on = fric ? friction_one(p, L.fpairs, L.x, L.x0, L.flam, L.fcoord, L.fbasis, L.mu, L.eps2, cs, item0 + t, stage[t])
                  : barrier_one(p, L.pairs, L.x, L.rest, L.dhat, L.kappa, cs, item0 + t, stage[t]);
    if (kGrad && on) {
        const int4 id = cs.ids[item0 + t];
        const int v[4] = {id.x & kIdMask, id.y, id.z, id.w};
        const int type = fric ? kPairFriction : ((id.x & kMollBit) ? kPairMollified : kPairBarrier);
        const double* f2 = type == kPairMollified ? cs.fac2 + kFac * (size_t)(item0 + t) : nullptr;
        for (int a = 0; a < 4; a++)
            if (v[a] >= 0)
                for (int q = 0; q < 3; q++) atomicAdd(fb + 3 * (size_t)v[a] + q, pair_grad(type, stage[t], f2, a, q));
    }
    if (!on)
#pragma unroll
        for (int k = 0; k < kFac; k++) stage[t][k] = 0.0;
    __syncthreads();
    const int words = kFac * min(kConThreads, n - p0);
    double* out = cs.fac + kFac * (size_t)item0;
    for (int k = t; k < words; k += kConThreads) out[k] = stage[k / kFac][k % kFac];
}

// soft constraints (GIPC.cu:6363-6407)
__global__ void k_soft(int ns, const uint32_t* __restrict__ idx, const double* __restrict__ x,
                       const double* __restrict__ target, double k, double* __restrict__ sg, ContactStore cs, int first) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ns) return;
    int v = idx[p];
    for (int q = 0; q < 3; q++) atomicAdd(sg + 3 * v + q, k * (x[3 * v + q] - target[3 * p + q]));
    double H[3][3] = {{k, 0, 0}, {0, k, 0}, {0, 0, k}};
    store_single(cs, first + p, v, H);
}

// ---- contact rows ---------------------------------------------------------------------------
// After the incidences are sorted by vertex (stable: each vertex's list is in pair order), row v
// of the contact matrix is made from v's list alone: every pair in it gives the blocks (v, w) of
// its vertices w >= v, and the columns w < v, whose blocks are copied from row w.  One warp takes a
// row of up to kRowLong incidences, a CTA a longer one.  The distinct columns go into a small hash
// table in shared memory and are ranked; the blocks are added up in shared memory, pair by pair in
// the list's order (each half-warp its share, the shares' sums in order): the same result on every
// run.  A row of more columns than the table holds (a corner of a large triangle under a fine
// cloth) is split into windows of kRowCols columns, each with the list of the pairs that have one
// there, and the windows are summed as rows are: the work stays in proportion to the list.
constexpr int kRowWarps = 4;
// incidences above which a CTA takes the row.  Newton step of rolled cloths with 244, 548 and 978 thousand
// pairs: 1125, 2304 and 3294 us with 64, 1073, 2190 and 3075 with 128, 1064, 2142 and 2961 with 256,
// 1070, 2137 and 2946 with 512; two 21^3 cubes, whose longest rows are these: k_row_counts 7.0, 7.6, 11.5
// and 11.4 us, k_row_sums 36.6, 41.4, 42.1 and 44.6.
constexpr int kRowLong = 128;
constexpr int kRowHash = 256;
constexpr int kRowCols = 40;   // columns of a window (each of 32 * kRowWarps lanes may add one more)
constexpr int kRowCtas = 4;    // CTAs of k_row_sums per SM (128 registers, 55 KB)
static_assert(kRowCols + 32 * kRowWarps < kRowHash, "the hash table never fills up");

// row pointers of the sorted incidences, the lists of rows to make, zeroed block counts
__global__ void k_inc_rows(int n, int m, const uint32_t* __restrict__ ks, int* __restrict__ ptr,
                           int* __restrict__ list, int* __restrict__ cnt, unsigned long long* __restrict__ ucnt) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    auto first = [&](int v) {  // first incidence with key >= v: an 8-way search, seven probes in flight
        int lo = 0, hi = m;
        while (lo < hi) {
            const int step = (hi - lo + 7) >> 3;
            int below = 0;
#pragma unroll
            for (int j = 1; j < 8; j++) {
                const int p = lo + j * step - 1;
                below += (p < hi && (int)__ldg(ks + p) < v) ? 1 : 0;
            }
            // the answer lies in [lo + below * step, lo + (below + 1) * step - 1], or up to hi
            if (below < 7) hi = min(hi, lo + (below + 1) * step - 1);
            lo += below * step;
        }
        return lo;
    };
    const int p0 = t <= n ? first(t) : 0;
    if (t <= n) {
        ptr[t] = p0;
        ucnt[t] = 0ull;
    }
    int p1 = __shfl_down_sync(0xffffffffu, p0, 1);
    if (lane == 31 && t < n) p1 = first(t + 1);
    const int len = t < n ? p1 - p0 : 0;
#pragma unroll
    for (int c = 0; c < 2; c++) {  // short lists, long lists
        const bool on = c == 0 ? len > 0 && len <= kRowLong : len > kRowLong;
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (!b) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(cnt + c, __popc(b));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (on) list[(size_t)c * n + base + __popc(b & ((1u << lane) - 1u))] = t;
    }
}

// numbers of: rows with short and with long lists, rows to split; places of the split's scratch in
// use; windows with short and with long lists; next short list to be summed
enum RowCount { kRowsShort = 0, kRowsLong = 1, kRowsSplit = 2, kSplitCols = 3, kSplitList = 4, kWinShort = 5,
                kWinLong = 6, kRowNext = 7, kRowCounts = 8 };

// a window of a split row: kRowCols columns of it from the diagonal on, and their pairs
struct RowWindow {
    int v;
    int i0, len;    // list: of the whole row (first = 0) or in RowArgs::wlist
    int c0, cols;   // columns, in RowArgs::wcol
    int first;      // their first one's place among the row's upper blocks
};

struct RowArgs {
    ContactStore cs;
    const uint32_t* inc;   // sorted incidences
    const int* ptr;
    int* list;             // [3n] rows with short lists, with long ones (~v: split), rows to split
    int* cnt;              // [kRowCounts]
    int n;
    int* wcol;             // [4 * incidences] sorted columns of the split rows
    uint32_t* wlist;       // [3 * incidences] lists of their windows
    RowWindow* win;        // [win_cap] windows: short lists from the front, long ones from the back
    int win_cap;
};

// the vertices of incidence i's pair (a single's vertex alone); returns its type
__device__ __forceinline__ int inc_pair(const RowArgs& a, uint32_t i, int (&v)[4], int& item, int& local) {
    if (i >= 4u * (uint32_t)a.cs.pairs) {
        item = (int)(i - 4u * (uint32_t)a.cs.pairs);
        local = 0;
        v[0] = a.cs.sid[item];
        v[1] = v[2] = v[3] = -1;
        return kPairSingle;
    }
    item = (int)(i >> 2);
    local = (int)(i & 3u);
    const int4 id = __ldg(a.cs.ids + item);
    v[0] = id.x & kIdMask, v[1] = id.y, v[2] = id.z, v[3] = id.w;
    const int type = item >= a.cs.barrier_pairs ? kPairFriction : ((id.x & kMollBit) ? kPairMollified : kPairBarrier);
    return (id.x & (kMollBit | kTwiceBit)) ? type | kPairApart : type;
}

// shared state of one row: a warp's, or (long rows) the CTA's, kept in the first warp's
struct RowTable {
    int hash[kRowHash];             // column, -1: free
    unsigned char rank[kRowHash];   // its place among the window's sorted columns
    unsigned short slot[kRowCols + 32 * kRowWarps];  // table slots in use, in order of arrival
    int found[kRowCols + 32 * kRowWarps];            // and their columns
    int col[kRowCols];              // sorted columns
    int used, over;
};

template <bool kCta>
__device__ __forceinline__ void row_sync() {
    if (kCta) __syncthreads();
    else __syncwarp();
}

// The distinct columns of the row into the table; false: more than kRowCols of them.
// t: this thread's index among the nt of its row.
template <bool kCta>
__device__ __forceinline__ bool row_columns(const RowArgs& a, RowTable& T, int i0, int i1, int t, int nt) {
    for (int k = t; k < kRowHash; k += nt) T.hash[k] = -1;
    if (t == 0) T.used = T.over = 0;
    row_sync<kCta>();
    constexpr int kU = 4;  // pairs in flight
    for (int k0 = i0 + t; k0 < i1 && !*(volatile int*)&T.over; k0 += kU * nt) {
        uint32_t inc[kU];
        int v[kU][4];
#pragma unroll
        for (int u = 0; u < kU; u++) inc[u] = k0 + u * nt < i1 ? __ldg(a.inc + k0 + u * nt) : ~0u;
#pragma unroll
        for (int u = 0; u < kU; u++) {
            int item, local;
            if (inc[u] != ~0u) inc_pair(a, inc[u], v[u], item, local);
            else v[u][0] = v[u][1] = v[u][2] = v[u][3] = -1;
        }
#pragma unroll
        for (int e = 0; e < 4 * kU; e++) {
            const int c = v[e / 4][e % 4];
            if (c < 0) continue;
            unsigned h = ((unsigned)c * 2654435761u) >> 24;
            for (;;) {
                const int seen = *(volatile int*)&T.hash[h];
                if (seen == c) break;
                if (seen < 0) {
                    if (*(volatile int*)&T.used > kRowCols) {  // full
                        T.over = 1;
                        break;
                    }
                    const int old = atomicCAS(&T.hash[h], -1, c);
                    if (old == c) break;
                    if (old < 0) {
                        const int k = atomicAdd(&T.used, 1);
                        T.slot[k] = (unsigned short)h;
                        T.found[k] = c;
                        break;
                    }
                }
                h = (h + 1) & (kRowHash - 1);
            }
        }
    }
    row_sync<kCta>();
    const bool ok = !T.over && T.used <= kRowCols;
    row_sync<kCta>();
    return ok;
}

// ranks the table's columns; U of them
template <bool kCta>
__device__ __forceinline__ void row_ranks(RowTable& T, int t, int nt) {
    const int U = T.used;
    for (int k = t; k < U; k += nt) {
        const int c = T.found[k];
        int r = 0;
#pragma unroll 4
        for (int j = 0; j < U; j++) r += T.found[j] < c;
        T.rank[T.slot[k]] = (unsigned char)r;
        T.col[r] = c;
    }
    row_sync<kCta>();
}

// the table of a window: its columns are known and sorted
template <bool kCta>
__device__ __forceinline__ void window_table(const RowArgs& a, RowTable& T, int c0, int cols, int t, int nt) {
    for (int k = t; k < kRowHash; k += nt) T.hash[k] = -1;
    if (t == 0) T.used = cols;
    row_sync<kCta>();
    for (int k = t; k < cols; k += nt) {
        const int c = a.wcol[c0 + k];
        unsigned h = ((unsigned)c * 2654435761u) >> 24;
        while (atomicCAS(&T.hash[h], -1, c) != -1) h = (h + 1) & (kRowHash - 1);
        T.rank[h] = (unsigned char)k;
        T.col[k] = c;
    }
    row_sync<kCta>();
}

// unique blocks of every row: upper ones (column >= row) and transposed ones (<< 32); rows that the
// table does not hold are listed for k_row_split
__global__ void __launch_bounds__(32 * kRowWarps) k_row_counts(RowArgs a, unsigned long long* __restrict__ ucnt) {
    __shared__ RowTable tables[kRowWarps];
    auto count = [&](auto cta, int* entry, RowTable& T, int t, int nt) {
        const int v = *entry;
        if (!row_columns<decltype(cta)::value>(a, T, a.ptr[v], a.ptr[v + 1], t, nt)) {
            if (t == 0) {
                *entry = ~v;
                a.list[2 * (size_t)a.n + atomicAdd(a.cnt + kRowsSplit, 1)] = v;
            }
            return;
        }
        unsigned up = 0, low = 0;  // of this thread's share of the columns
        for (int k = t; k < T.used; k += nt) {
            if (T.found[k] >= v) up++;
            else low++;
        }
        up = __reduce_add_sync(0xffffffffu, up);
        low = __reduce_add_sync(0xffffffffu, low);
        if ((threadIdx.x & 31) == 0 && (up | low)) atomicAdd(ucnt + v, (unsigned long long)up | ((unsigned long long)low << 32));
        row_sync<decltype(cta)::value>();
    };
    const int n_short = a.cnt[kRowsShort], n_long = a.cnt[kRowsLong];
    for (int k = blockIdx.x; k < n_long; k += gridDim.x)
        count(std::true_type{}, a.list + (size_t)a.n + k, tables[0], threadIdx.x, 32 * kRowWarps);
    __syncthreads();
    // (counted from the last CTA: the first ones may have taken a long row more)
    for (int k = (gridDim.x - 1 - blockIdx.x) * kRowWarps + (threadIdx.x >> 5); k < n_short; k += gridDim.x * kRowWarps)
        count(std::false_type{}, a.list + k, tables[threadIdx.x >> 5], threadIdx.x & 31, 32);
}

// Rows of more than kRowCols columns, a CTA each: their sorted distinct columns by a bitmap of the
// vertices, their block counts, and windows of kRowCols upper columns with the lists of the pairs that
// have a column there.  The first window starts at the diagonal, which every pair has: its list is the
// row's.  The others' lists are a stable split of it: each warp counts, and then places, its own part
// of the list in order.  Three passes over the list whatever its columns, bound by the latency of its
// gathers: 24 us for a row of 1000 pairs and columns, 110 us for 5000, 340 us for 20 000, with 45, 147
// and 470 us of k_row_sums; the whole assembly of a 31^3 cube with such a row 270, 495 and 1087 us, and
// 317, 506 and 1139 us when the pairs' blocks were sorted.  (Windows found by halving from all columns, each
// attempt and each sum reading the whole list, made it 3.0, 136 and 3491 ms.)
constexpr int kSplitWarps = 8;
constexpr int kSplitSpan = 1 << 18;  // columns of the bitmap (32 KB); a larger mesh takes several
constexpr int kSplitWin = 896;       // windows listed at a time: kSplitWarps counts each and their first columns
static_assert((kSplitWarps + 1) * kSplitWin <= kSplitSpan / 32 && kSplitWin <= 4 * 32 * kSplitWarps, "shared memory");

__global__ void __launch_bounds__(32 * kSplitWarps) k_row_split(RowArgs a, unsigned long long* __restrict__ ucnt) {
    __shared__ unsigned s_mem[kSplitSpan / 32];  // bitmap, then the windows' first columns and counts
    __shared__ int s_sum[kSplitWarps];
    __shared__ int s_base, s_low, s_list;
    const int t = threadIdx.x, nt = 32 * kSplitWarps, w = t >> 5, lane = t & 31;
    // exclusive sum over the CTA in thread order, and the total
    auto scan = [&](int x, int& total) -> int {
        int in = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, in, o);
            if (lane >= o) in += y;
        }
        __syncthreads();  // s_sum is free
        if (lane == 31) s_sum[w] = in;
        __syncthreads();
        int before = 0;
        total = 0;
#pragma unroll
        for (int k = 0; k < kSplitWarps; k++) {
            if (k < w) before += s_sum[k];
            total += s_sum[k];
        }
        return before + in - x;
    };
    auto put = [&](const RowWindow& x) {
        if (x.len > kRowLong) a.win[a.win_cap - 1 - atomicAdd(a.cnt + kWinLong, 1)] = x;
        else a.win[atomicAdd(a.cnt + kWinShort, 1)] = x;
    };
    const int rows = a.cnt[kRowsSplit];
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {  // CTA-uniform
        const int v = a.list[2 * (size_t)a.n + row], i0 = a.ptr[v], i1 = a.ptr[v + 1], len = i1 - i0;
        if (t == 0) s_base = atomicAdd(a.cnt + kSplitCols, 3 * len + 1);  // a pair has three other vertices
        int cols = 0;
        for (int s0 = 0; s0 < a.n; s0 += kSplitSpan) {
            const int span = min(kSplitSpan, a.n - s0), words = (span + 31) >> 5;
            __syncthreads();
            for (int k = t; k < words; k += nt) s_mem[k] = 0u;
            __syncthreads();
            for (int k0 = i0 + t; k0 < i1; k0 += 4 * nt) {
                uint32_t inc[4];
                int id[4][4];
#pragma unroll
                for (int u = 0; u < 4; u++) inc[u] = k0 + u * nt < i1 ? __ldg(a.inc + k0 + u * nt) : ~0u;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    int item, local;
                    if (inc[u] != ~0u) inc_pair(a, inc[u], id[u], item, local);
                    else id[u][0] = id[u][1] = id[u][2] = id[u][3] = -1;
                }
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    const int c = id[e / 4][e % 4] - s0;
                    if (c < 0 || c >= span) continue;  // (-1 too)
                    const unsigned bit = 1u << (c & 31);
                    if (!(*(volatile unsigned*)&s_mem[c >> 5] & bit)) atomicOr(&s_mem[c >> 5], bit);
                }
            }
            __syncthreads();
            for (int k0 = 0; k0 < words; k0 += nt) {  // CTA-uniform
                unsigned m = k0 + t < words ? s_mem[k0 + t] : 0u;
                int total, at = cols + scan(__popc(m), total);
                for (; m; m &= m - 1, at++) {
                    const int c = s0 + 32 * (k0 + t) + __ffs(m) - 1;
                    a.wcol[s_base + at] = c;
                    if (c == v) s_low = at;
                }
                cols += total;
            }
        }
        __syncthreads();
        const int low = s_low, up = cols - low, c0 = s_base + low, nwin = (up + kRowCols - 1) / kRowCols;
        if (t == 0) {
            ucnt[v] = (unsigned long long)(unsigned)up | ((unsigned long long)(unsigned)low << 32);
            put({v, i0, len, c0, min(kRowCols, up), 0});
        }
        int* first = reinterpret_cast<int*>(s_mem);  // a window's first column
        int* count = first + kSplitWin;              // [kSplitWarps][kSplitWin]
        const int part = ((len + kSplitWarps - 1) / kSplitWarps + 31) & ~31;
        const int b0 = i0 + w * part, b1 = min(i1, b0 + part);
        for (int w0 = 1; w0 < nwin; w0 += kSplitWin) {  // CTA-uniform
            const int nw = min(kSplitWin, nwin - w0);
            __syncthreads();
            for (int k = t; k < nw; k += nt) first[k] = a.wcol[c0 + kRowCols * (w0 + k)];
            for (int k = t; k < kSplitWarps * kSplitWin; k += nt) count[k] = 0;
            const int end = w0 + nw < nwin ? a.wcol[c0 + kRowCols * (w0 + nw)] : a.n;
            __syncthreads();
            // the windows (of these nw) of incidence i's pair, each once, -1: none
            auto windows = [&](uint32_t i, int (&id)[4]) {
                int item, local;
                if (i != ~0u) inc_pair(a, i, id, item, local);
                else id[0] = id[1] = id[2] = id[3] = -1;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int c = id[k];
                    int lo = -1;
                    if (c >= first[0] && c < end) {
                        lo = 0;  // last window whose first column is not above c
                        for (int hi = nw; hi - lo > 1;) {
                            const int mid = (lo + hi) >> 1;
                            if (first[mid] <= c) lo = mid;
                            else hi = mid;
                        }
                    }
                    id[k] = lo;
                }
#pragma unroll
                for (int k = 1; k < 4; k++)
#pragma unroll
                    for (int j = 0; j < k; j++)
                        if (id[k] == id[j]) id[k] = -1;
            };
            for (int i = b0 + lane; i < b1; i += 32) {
                int id[4];
                windows(__ldg(a.inc + i), id);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (id[k] >= 0) atomicAdd(count + w * kSplitWin + id[k], 1);
            }
            __syncthreads();
            // places: window by window, warp by warp; a thread's four windows are neighbours
            int sum = 0, total;
            for (int k = 4 * t; k < min(4 * t + 4, nw); k++)
                for (int j = 0; j < kSplitWarps; j++) sum += count[j * kSplitWin + k];
            int at = scan(sum, total);
            if (t == 0) s_list = atomicAdd(a.cnt + kSplitList, total);
            __syncthreads();
            for (int k = 4 * t; k < min(4 * t + 4, nw); k++) {
                const int start = at;
                for (int j = 0; j < kSplitWarps; j++) {
                    const int c = count[j * kSplitWin + k];
                    count[j * kSplitWin + k] = at;
                    at += c;
                }
                const int f = kRowCols * (w0 + k);
                put({v, s_list + start, at - start, c0 + f, min(kRowCols, up - f), f});
            }
            __syncthreads();
            uint32_t* out = a.wlist + s_list;
            for (int i = b0; i < b1; i += 32) {  // warp-uniform
                const uint32_t inc = i + lane < b1 ? __ldg(a.inc + i + lane) : ~0u;
                int id[4];
                windows(inc, id);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned same = __match_any_sync(0xffffffffu, id[k]);
                    int* c = count + w * kSplitWin + id[k];
                    if (id[k] >= 0) out[*c + __popc(same & ((1u << lane) - 1u))] = inc;
                    __syncwarp();
                    if (id[k] >= 0 && lane == __ffs(same) - 1) *c += __popc(same);
                    __syncwarp();
                }
            }
        }
        __syncthreads();
    }
}

struct RowOut {
    const unsigned long long* uoff;
    const int32_t* btype;
    int* nuc;
    int* cu_ptr;
    int* cl_ptr;
    int* uc_row;
    int* uc_col;
    double* u64;
    float* u32;
    int* cl_col;
    double* grad;
};

// A half-warp adds up its share of a row's list (every second pair of a warp's, every eighth of a
// CTA's): a lane stages one pair, scaled for this row, and then lanes 0..11 take column q of the
// block of vertex b (three entries each) and lanes 12..14 the gradient's component q, four
// shared-memory reads and three products for a pair whatever its kind; the next pairs' lines are
// on their way meanwhile.  1062 us for the rolled cloth's eight million incidences, 46 warp
// instructions each; the shared-memory pipe is busy 59 % of it, mostly with the sums.  (One lane
// per entry, each kind its own code: 1557 us; two lanes a pair staging, in place: 1516, pipelined:
// 1187.)
// A staged line: barrier [0..2] g_v, [3..14] g, friction [0..8] W, [9..12] c_v c, single [0..8] its
// block, [9..12] 1; [15..17] the pair's gradient at v, [18] 1, [19] lam or 1.
constexpr int kLine = 21;  // odd: the two halves' lines start in different banks
struct RowWarp {
    double acc[2][kRowCols * 9];
    double line[32][kLine];
    signed char col[32][4];   // window column of each of the pair's vertices, -1: none
    signed char wide[32];     // 1: the block is c_b times nine numbers
};
constexpr size_t kRowShared = sizeof(RowTable) * kRowWarps + sizeof(RowWarp) * kRowWarps;

// half-warp hw of nh over list[i0, i1): its acc (zeroed) of the columns in [lo, hi), and g, the gradient
// (first: in the window of the diagonal, whose list is the whole row's)
__device__ __forceinline__ void row_accumulate(const RowArgs& a, const uint32_t* __restrict__ list, const RowTable& T,
                                               RowWarp& W, int v, int U, int i0, int i1, int hw, int nh, int lo,
                                               int hi, bool first, double& g) {
    const int lane = threadIdx.x & 31, h = lane >> 4, hl = lane & 15;
    const bool grad = hl >= 12;
    const int b = grad ? 0 : hl / 3, q = hl % 3;
    double* acc = W.acc[h];
    for (int k = lane; k < 9 * U; k += 32) W.acc[0][k] = W.acc[1][k] = 0.0;
    W.line[lane][18] = 1.0;
    // (lane 15 of a half reads with the others and keeps nothing)
    const int s_thin = grad ? 18 : 3 + 3 * b + q, s_wide = grad ? 18 : 9 + b;
    const int r_thin = grad ? 15 + (hl < 15 ? q : 0) : 0, r_wide = grad ? r_thin : q;
    const int d_thin = grad ? 0 : 1, d_wide = grad ? 0 : 3, s_lam = grad ? 18 : 19;
    const int turns = (i1 - i0 + 16 * nh - 1) / (16 * nh);  // the same for all of the row's half-warps
    auto incidence = [&](int t) -> uint32_t {
        const int i = i0 + nh * (16 * t + hl) + hw;
        return i < i1 ? __ldg(list + i) : ~0u;
    };
    // a turn's pair is read while the sums of the turn before run
    double2 f[8];
    int vert[4], pair = 0, local = 0, type = -1;
    auto fetch = [&](uint32_t inc) {
        type = -1;
        if (inc == ~0u) return;
        type = inc_pair(a, inc, vert, pair, local);
        if (type == kPairSingle || (type & kPairApart)) return;
        const double2* src = reinterpret_cast<const double2*>(a.cs.fac + kFac * (size_t)pair);
#pragma unroll
        for (int k = 0; k < 8; k++) f[k] = __ldg(src + k);
    };
    bool apart = false;
    fetch(incidence(0));
    uint32_t inc_next = incidence(1);
    for (int t = 0; t < turns; t++) {
        __syncwarp();
        double* L = W.line[lane];
        int u[4] = {-1, -1, -1, -1};
        double gr[3] = {0.0, 0.0, 0.0};
        if (type == kPairBarrier) {
            double w[16];
#pragma unroll
            for (int k = 0; k < 8; k++) w[2 * k] = f[k].x, w[2 * k + 1] = f[k].y;
            double gv[3];
#pragma unroll
            for (int p = 0; p < 3; p++)
                gv[p] = local == 0 ? w[1 + p] : (local == 1 ? w[4 + p] : (local == 2 ? w[7 + p] : w[10 + p]));
#pragma unroll
            for (int p = 0; p < 3; p++) {
                L[p] = gv[p];
                gr[p] = w[13] * gv[p];
            }
#pragma unroll
            for (int k = 0; k < 12; k++) L[3 + k] = w[1 + k];
            L[19] = w[0];
        } else if (type == kPairFriction) {
            double w[16];
#pragma unroll
            for (int k = 0; k < 8; k++) w[2 * k] = f[k].x, w[2 * k + 1] = f[k].y;
            const double cv = local == 0 ? w[9] : (local == 1 ? w[10] : (local == 2 ? w[11] : w[12]));
#pragma unroll
            for (int k = 0; k < 9; k++) L[k] = w[k];
#pragma unroll
            for (int k = 0; k < 4; k++) L[9 + k] = cv * w[9 + k];
            L[19] = 1.0;
#pragma unroll
            for (int p = 0; p < 3; p++) gr[p] = cv * w[13 + p];
        } else if (type == kPairSingle) {
#pragma unroll
            for (int k = 0; k < 9; k++) L[k] = a.cs.sval[9 * (size_t)pair + k];
#pragma unroll
            for (int k = 0; k < 4; k++) L[9 + k] = 1.0;
            L[19] = 1.0;
        }
#pragma unroll
        for (int p = 0; p < 3; p++) L[15 + p] = first ? gr[p] : 0.0;
        if (type >= 0 && (type & kPairApart)) apart = true;  // below
        else if (type >= 0)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int c = vert[k];
                if (c < lo || c >= hi) continue;
                unsigned x = ((unsigned)c * 2654435761u) >> 24;
                while (T.hash[x] != c) x = (x + 1) & (kRowHash - 1);
                u[k] = T.rank[x];
            }
        *reinterpret_cast<char4*>(W.col[lane]) = make_char4(u[0], u[1], u[2], u[3]);
        W.wide[lane] = type == kPairBarrier ? 0 : 1;
        fetch(inc_next);
        inc_next = incidence(t + 2);
        __syncwarp();
        const int kmax = min(16, (i1 - i0 - 16 * nh * t + nh - 1) / nh);  // warp-uniform
        for (int k0 = 0; k0 < kmax; k0 += 4) {
            double x[4][3];
            int d[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int j = 16 * h + k0 + k;
                const double* m = W.line[j];
                const bool wide = W.wide[j] != 0;
                const double sc = m[wide ? s_wide : s_thin];
                const double* r = m + (wide ? r_wide : r_thin);
                const int dr = wide ? d_wide : d_thin;
                const double lam = m[s_lam];
                x[k][0] = lam * (sc * r[0]);
                x[k][1] = lam * (sc * r[dr]);
                x[k][2] = lam * (sc * r[2 * dr]);
                d[k] = grad ? -1 : W.col[j][b];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (grad) {
                    g += x[k][0];
                } else if (d[k] >= 0) {
                    double* o = acc + 9 * d[k] + q;
                    const double o0 = o[0], o1 = o[3], o2 = o[6];
                    o[0] = o0 + x[k][0];
                    o[3] = o1 + x[k][1];
                    o[6] = o2 + x[k][2];
                }
                __syncwarp();
            }
        }
    }
    // Mollified pairs and pairs that name a vertex twice (none come from the pair search), one
    // after another.  Two equal vertices of a pair have one column, so the blocks of a row are added
    // vertex by vertex; the row of such a vertex meets the pair once for each of its places, which
    // gives all four of the vertex's blocks.
    if (__any_sync(0xffffffffu, apart)) {
        for (int i = i0 + hw; i - hw < i1; i += nh) {  // the same turns in both halves
            int w[4], item = 0, la = 0, ty = -1, d = -1;
            double x[3] = {0.0, 0.0, 0.0};
            if (i < i1) ty = inc_pair(a, __ldg(list + i), w, item, la);
            if (ty >= 0 && (ty & kPairApart) && hl < 15) {
                const int base = ty & ~kPairApart;
                const double *m = a.cs.fac + kFac * (size_t)item, *m2 = a.cs.fac2 + kFac * (size_t)item;
                const int c = w[b];
                if (grad) {
                    if (first) g += pair_grad(base, m, m2, la, q);
                } else if (c >= lo && c < hi) {
                    unsigned s = ((unsigned)c * 2654435761u) >> 24;
                    while (T.hash[s] != c) s = (s + 1) & (kRowHash - 1);
                    d = 9 * T.rank[s] + q;
#pragma unroll
                    for (int p = 0; p < 3; p++) x[p] = pair_entry(base, m, m2, la, b, p, q);
                }
            }
            for (int turn = 0; turn < 4; turn++) {
                if (d >= 0 && b == turn)
#pragma unroll
                    for (int p = 0; p < 3; p++) acc[d + 3 * p] += x[p];
                __syncwarp();
            }
        }
    }
    __syncwarp();
}

// stores the upper blocks of the table's columns nlow .. U - 1 (threads t of nt) from place `up` on, acc
// summed over the row's warps in order
template <bool kCta>
__device__ __forceinline__ void row_store(const RowOut& o, const RowTable& T, const RowWarp* W, int v, int nlow, int U,
                                          int t, int nt, size_t up) {
    const bool fixed_row = o.btype && o.btype[v] != 0;
    for (int e = 9 * nlow + t; e < 9 * U; e += nt) {
        const int u = e / 9, q = e % 9, c = T.col[u];
        double s = W[0].acc[0][e] + W[0].acc[1][e];
        if (kCta)
#pragma unroll
            for (int w = 1; w < kRowWarps; w++) s = s + W[w].acc[0][e] + W[w].acc[1][e];
        if (fixed_row || (o.btype && o.btype[c] != 0)) s = 0.0;
        const size_t k = up + (u - nlow);
        o.u64[9 * k + q] = s;
        o.u32[9 * k + q] = (float)s;
        if (q == 0) {
            o.uc_row[k] = v;
            o.uc_col[k] = c;
        }
    }
}

__global__ void __launch_bounds__(32 * kRowWarps, kRowCtas) k_row_sums(RowArgs a, RowOut o) {
    extern __shared__ __align__(16) unsigned char row_smem[];
    __shared__ double s_grad[2 * kRowWarps][3];
    RowWarp* warps = reinterpret_cast<RowWarp*>(row_smem);
    RowTable* tables = reinterpret_cast<RowTable*>(row_smem + sizeof(RowWarp) * kRowWarps);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
    // row pointers of the two block lists
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= a.n; i += gridDim.x * blockDim.x) {
        const unsigned long long f = o.uoff[i];
        o.cu_ptr[i] = (int)(f & 0xffffffffull);
        o.cl_ptr[i] = (int)(f >> 32);
        if (i == a.n) o.nuc[0] = (int)(f & 0xffffffffull);
    }
    // a row, or a window of a split one (win), by nt threads: its blocks, the columns of its transposed
    // list and its gradient
    auto make = [&](auto cta, RowTable& T, RowWarp* W, int t, int nt, int v, const RowWindow* win) {
        constexpr bool kCta = decltype(cta)::value;
        int i0, i1, lo, hi, nlow = 0;
        size_t up = (size_t)(o.uoff[v] & 0xffffffffull);
        const int low = (int)(o.uoff[v] >> 32);
        const uint32_t* list = a.inc;
        bool first = true;
        if (win) {
            first = win->first == 0;
            if (!first) list = a.wlist;
            i0 = win->i0;
            i1 = i0 + win->len;
            window_table<kCta>(a, T, win->c0, win->cols, t, nt);
            lo = T.col[0];
            hi = T.col[T.used - 1] + 1;
            up += win->first;
            if (first) {
                const int n = (int)(o.uoff[v + 1] >> 32) - low;
                for (int k = t; k < n; k += nt) o.cl_col[low + k] = a.wcol[win->c0 - n + k];
            }
        } else {
            i0 = a.ptr[v];
            i1 = a.ptr[v + 1];
            row_columns<kCta>(a, T, i0, i1, t, nt);
            row_ranks<kCta>(T, t, nt);
            lo = v;  // upper blocks only
            hi = a.n;
            nlow = (int)(o.uoff[v + 1] >> 32) - low;
            for (int k = t; k < nlow; k += nt) o.cl_col[low + k] = T.col[k];
        }
        double g = 0.0;
        row_accumulate(a, list, T, W[kCta ? w : 0], v, T.used, i0, i1, kCta ? hw : (hw & 1), kCta ? 2 * kRowWarps : 2, lo,
                       hi, first, g);
        row_sync<kCta>();
        row_store<kCta>(o, T, W, v, nlow, T.used, t, nt, up);
        if (kCta) {
            if (hl >= 12 && hl < 15) s_grad[hw][hl - 12] = g;
            __syncthreads();
            if (first && threadIdx.x < 3) {
                double s = s_grad[0][lane];
#pragma unroll
                for (int k = 1; k < 2 * kRowWarps; k++) s += s_grad[k][lane];
                o.grad[3 * (size_t)v + lane] += s;
            }
        } else {
            g += __shfl_down_sync(0xffffffffu, g, 16);  // the halves in list order
            if (first && lane >= 12 && lane < 15) o.grad[3 * (size_t)v + lane - 12] += g;
        }
        row_sync<kCta>();
    };
    const int n_short = a.cnt[kRowsShort], n_long = a.cnt[kRowsLong];
    const int w_short = a.cnt[kWinShort], w_long = a.cnt[kWinLong];
    for (int k = blockIdx.x; k < w_long + n_long; k += gridDim.x) {
        const RowWindow* win = k < w_long ? a.win + (a.win_cap - 1 - k) : nullptr;
        const int v = win ? win->v : a.list[(size_t)a.n + k - w_long];
        if (v >= 0) make(std::true_type{}, tables[0], warps, threadIdx.x, 32 * kRowWarps, v, win);
    }
    __syncthreads();
    // Short lists go to whichever warp is free, the next one fetched ahead: the kernel runs beside the static
    // scatter, and CTAs that find their place late had held up a fixed share of the rows (rolled
    // cloth: from 950 to 1500 us).
    auto next = [&]() { return lane == 0 ? atomicAdd(a.cnt + kRowNext, 1) : 0; };
    for (int k = __shfl_sync(0xffffffffu, next(), 0); k < n_short + w_short;) {
        const int ahead = next();
        const RowWindow* win = k < n_short ? nullptr : a.win + (k - n_short);
        const int v = win ? win->v : a.list[k];
        if (v >= 0) make(std::false_type{}, tables[w], warps + w, lane, 32, v, win);
        k = __shfl_sync(0xffffffffu, ahead, 0);
    }
}

// The transposed copies: block u = (r, c), r < c, goes to the place of column r in c's list.  A copy,
// not a second sum over c's list, whose pairs are shared out differently: the matrix stays exactly
// symmetric (the solve's p.Ap recurrence takes it so), in FP64 and in FP32.  A warp finds the places
// of 32 blocks, one a lane, and then moves their 288 entries with whole lines on the reading side.
__global__ void __launch_bounds__(SGIPC_BLOCK) k_row_transposes(const int* __restrict__ nuc,
                                                                const int* __restrict__ uc_row,
                                                                const int* __restrict__ uc_col,
                                                                const double* __restrict__ u64,
                                                                const float* __restrict__ u32,
                                                                const int* __restrict__ cl_ptr,
                                                                const int* __restrict__ cl_col,
                                                                double* __restrict__ l64, float* __restrict__ l32) {
    const int nu = nuc[0], lane = threadIdx.x & 31;
    const int step = (gridDim.x * blockDim.x) & ~31;
    for (int u0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; u0 < nu; u0 += step) {  // warp-uniform
        int k = -1;
        if (u0 + lane < nu) {
            const int r = uc_row[u0 + lane], c = uc_col[u0 + lane];
            if (r < c) {
                k = cl_ptr[c];
                int hi = cl_ptr[c + 1];
                while (k < hi) {  // first place whose column is not below r: r is in the list
                    const int mid = (k + hi) >> 1;
                    if (__ldg(cl_col + mid) < r) k = mid + 1;
                    else hi = mid;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const int e = 32 * t + lane, q = e % 9;
            const int at = __shfl_sync(0xffffffffu, k, e / 9);
            if (at < 0) continue;
            const size_t to = 9 * (size_t)at + 3 * (q % 3) + q / 3;
            l64[to] = u64[9 * (size_t)u0 + e];
            l32[to] = u32[9 * (size_t)u0 + e];
        }
    }
}

// ------------------------------------------------------------------------------------------
// line-search energy (GIPC::computeEnergy, GIPC.cu:10520-10580; per-term reductions
// Energy_Add_Reduction_Algorithm, GIPC.cu:10347-10518).  Each kernel writes one partial sum
// per CTA; every sum runs in a fixed order, so the energy is the same bit for bit on every
// run.  The scalings of computeEnergy (dt^2 on the elastic terms, kappa, the friction rates)
// are applied per element, as in the gradient kernels above.
// ------------------------------------------------------------------------------------------
// fixed-order CTA sum of one value per thread into part[blockIdx.x]; every thread calls it
__device__ __forceinline__ void cta_energy(double e, double* __restrict__ part) {
    __shared__ double sw[SGIPC_BLOCK / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sw[w];
        part[blockIdx.x] = t;
    }
}

// kinetic 1/2 m |x - x_tilde|^2 (_getKineticEnergy_Reduction_3D)
__device__ __forceinline__ double en_kinetic(int gi, int nv, const double* __restrict__ x, const double* __restrict__ xt,
                             const double* __restrict__ m) {
    const int i = gi;
    double e = 0.0;
    if (i < nv) {
        const d3 d = ld3(x, i) - ld3(xt, i);
        e = 0.5 * m[i] * sq(d);
    }
    return e;
}

// stable Neo-Hookean: dt^2 vol 1/2 (mu (|F|^2 - 3) + lam (J - 1 - mu/lam)^2)
// (_getFEMEnergy_Reduction_3D; femEnergy.cu:1042-1050)
__device__ __forceinline__ double en_snk(int gi, int nt, const uint32_t* __restrict__ tets, const double* __restrict__ x,
                         const double* __restrict__ dminv, const double* __restrict__ vol,
                         const double* __restrict__ lr, const double* __restrict__ vr, double dt2) {
    const int t = gi;
    double e = 0.0;
    if (t < nt) {
        const uint4 tv = reinterpret_cast<const uint4*>(tets)[t];
        const d3 X0 = ld3(x, tv.x), e1 = ld3(x, tv.y) - X0, e2 = ld3(x, tv.z) - X0, e3 = ld3(x, tv.w) - X0;
        const double* Di = dminv + 9 * (size_t)t;
        double F[3][3];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) F[i][j] = comp(e1, i) * Di[j] + comp(e2, i) * Di[3 + j] + comp(e3, i) * Di[6 + j];
        double I2 = 0.0;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) I2 += F[i][j] * F[i][j];
        const double J = F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) -
                         F[0][1] * (F[1][0] * F[2][2] - F[1][2] * F[2][0]) +
                         F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]);
        const double mu = lr[t], lam = vr[t], Jm = J - 1.0 - mu / lam;
        e = 0.5 * (mu * (I2 - 3.0) + lam * Jm * Jm) * vol[t] * dt2;
    }
    return e;
}

// cloth membrane: dt^2 area (kst sum_j S(|f_j|) + ksh (f_0 . f_1)^2), S(t) = (t-1)^2 (+ srate
// (t-1)^3 when stretched) (_getFEMEnergy_Reduction_3D_triangle, femEnergy.cu:351-403)
__device__ __forceinline__ double en_tri(int gi, int nf, const uint32_t* __restrict__ tris, const double* __restrict__ x,
                         const double* __restrict__ dminv, const double* __restrict__ area, double kst, double ksh,
                         double srate, double dt2) {
    const int f = gi;
    double e = 0.0;
    if (f < nf) {
        const d3 x0 = ld3(x, tris[3 * f]), e1 = ld3(x, tris[3 * f + 1]) - x0, e2 = ld3(x, tris[3 * f + 2]) - x0;
        const double* Di = dminv + 4 * (size_t)f;
        const d3 col[2] = {Di[0] * e1 + Di[2] * e2, Di[1] * e1 + Di[3] * e2};
        double E = 0.0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const double t = sqrt(sq(col[j])), u = t - 1.0;
            E += kst * (u * u + (t > 1.0 ? srate * u * u * u : 0.0));
        }
        const double I6 = dot(col[0], col[1]);
        E += ksh * I6 * I6;
        e = E * area[f] * dt2;
    }
    return e;
}

// quadratic bending: 1/2 c sum_ab Q_ab x_a . x_b, c = |rest e| bendStiff dt^2; boundary
// edges (a missing wing) carry none (femEnergy.cu:2623-2753)
__device__ __forceinline__ double en_hinge(int gi, int nh, const uint32_t* __restrict__ edges, const int32_t* __restrict__ adj,
                           const double* __restrict__ x, const double* __restrict__ rest,
                           const double* __restrict__ Qcm, double kb_dt2) {
    const int h = gi;
    double e = 0.0;
    if (h < nh && adj[2 * h] >= 0 && adj[2 * h + 1] >= 0) {
        const int v[4] = {(int)edges[2 * h], (int)edges[2 * h + 1], adj[2 * h], adj[2 * h + 1]};
        const double c = sqrt(sq(ld3(rest, v[0]) - ld3(rest, v[1]))) * kb_dt2;
        d3 xv[4];
#pragma unroll
        for (int a = 0; a < 4; a++) xv[a] = ld3(x, v[a]);
        double E = 0.0;
#pragma unroll
        for (int a = 0; a < 4; a++) {
            d3 g = mk(0, 0, 0);
#pragma unroll
            for (int b = 0; b < 4; b++) g = g + Qcm[16 * (size_t)h + 4 * b + a] * xv[b];
            E += 0.5 * c * dot(xv[a], g);
        }
        e = E;
    }
    return e;
}

// soft constraints 1/2 k |x - target|^2, k = motionRate softRate^2 (GIPC.cu:6363-6407)
__device__ __forceinline__ double en_soft(int gi, int ns, const uint32_t* __restrict__ idx, const double* __restrict__ x,
                          const double* __restrict__ target, double k) {
    const int p = gi;
    double e = 0.0;
    if (p < ns) e = 0.5 * k * sq(ld3(x, idx[p]) - ld3(target, p));
    return e;
}

// barrier pairs: kappa dhat^2 (I-1)^2 ln^2 I, I = d^2/dhat; mollified EE / PE / PP pairs
// times e(c^2) (_getBarrierEnergy_Reduction_3D, GIPC.cu:701-958)
__device__ __forceinline__ double en_barrier(int gi, int np, int nv, const int4* __restrict__ pairs, const double* __restrict__ x,
                             const double* __restrict__ rest, double dhat, double kappa) {
    const int p = gi;
    double e = 0.0;
    if (p < np) {
        int v[4], nvp;
        const int kind = decode_pair(pairs[p], v, nvp);
        bool ok = true;
        for (int a = 0; a < nvp; a++) ok = ok && v[a] >= 0 && v[a] < nv;
        if (ok) {
            d3 X[4], gd2[4];
#pragma unroll
            for (int a = 0; a < 4; a++) X[a] = a < nvp ? ld3(x, v[a]) : mk(0, 0, 0);
            const double I = dist2_grad(kind, X, gd2) / dhat;
            double B, dB, d2B;
            if (kind <= 3) {
                barrier_s(I, kappa * dhat * dhat, B, dB, d2B);
                e = B;
            } else {
                int ea0, ea1, eb0, eb1;
                if (kind == 4) { ea0 = 0; ea1 = 1; eb0 = 2; eb1 = 3; }
                else if (kind == 6) { ea0 = 0; ea1 = 2; eb0 = 1; eb1 = 3; }
                else { ea0 = 0; ea1 = 3; eb0 = 1; eb1 = 2; }
                const double I1 = sq(cross(X[ea1] - X[ea0], X[eb1] - X[eb0]));
                if (I1 != 0.0) {
                    const double ex = 1e-3 * sq(ld3(rest, v[ea0]) - ld3(rest, v[ea1])) *
                                      sq(ld3(rest, v[eb0]) - ld3(rest, v[eb1]));
                    const double em = -I1 * I1 / (ex * ex) + 2.0 * I1 / ex;
                    barrier_s(I, dhat * dhat, B, dB, d2B);
                    e = kappa * em * B;
                }
            }
        }
    }
    return e;
}

// ground barrier -kappa (d^2 - dhat)^2 ln(d^2/dhat), d = y - offset (GIPC.cu:6463-6514)
__device__ __forceinline__ double en_ground(int gi, int ng, int nv, const uint32_t* __restrict__ gp, const double* __restrict__ x,
                            double offset, double dhat, double kappa) {
    const int p = gi;
    double e = 0.0;
    if (p < ng && (int)gp[p] < nv) {
        const double dist = x[3 * gp[p] + 1] - offset, d2 = dist * dist, t = d2 - dhat;
        e = -kappa * t * t * log(d2 / dhat);
    }
    return e;
}

// pair friction mu lambda f0(|u|): f0 = |u| beyond eps, else |u|^2 (eps - |u|/3) / eps^2 +
// eps/3 (_getFrictionEnergy_Reduction_3D, GIPC.cu:1252-1356)
__device__ __forceinline__ double en_friction(int gi, int np, int nv, const int4* __restrict__ pairs, const double* __restrict__ x,
                              const double* __restrict__ x0, const double* __restrict__ lam,
                              const double* __restrict__ coord, const double* __restrict__ basis, double mu,
                              double eps2) {
    const int p = gi;
    double e = 0.0;
    if (p < np) {
        const int4 q = pairs[p];
        int v[4] = {0, 0, 0, 0}, nvp = 0;
        double cf[4] = {0, 0, 0, 0};
        const double g1 = coord[2 * p], g2 = coord[2 * p + 1];
        if (q.x >= 0) {
            if (q.w >= 0) {
                v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; nvp = 4;
                cf[0] = 1.0 - g1; cf[1] = g1; cf[2] = g2 - 1.0; cf[3] = -g2;
            }
        } else if (q.y >= 0) {
            v[0] = -q.x - 1;
            if (q.z < 0) { v[1] = q.y; nvp = 2; cf[0] = 1.0; cf[1] = -1.0; }
            else if (q.w < 0) { v[1] = q.y; v[2] = q.z; nvp = 3; cf[0] = 1.0; cf[1] = g1 - 1.0; cf[2] = -g1; }
            else { v[1] = q.y; v[2] = q.z; v[3] = q.w; nvp = 4; cf[0] = 1.0; cf[1] = -1.0 + g1 + g2; cf[2] = -g1; cf[3] = -g2; }
        }
        bool ok = nvp > 0;
        for (int a = 0; a < nvp; a++) ok = ok && v[a] >= 0 && v[a] < nv;
        if (ok) {
            const double* Tb = basis + 6 * (size_t)p;
            const d3 t0 = mk(Tb[0], Tb[2], Tb[4]), t1 = mk(Tb[1], Tb[3], Tb[5]);
            d3 rel = mk(0, 0, 0);
            for (int a = 0; a < nvp; a++) rel = rel + cf[a] * (ld3(x, v[a]) - ld3(x0, v[a]));
            const double u0 = dot(t0, rel), u1 = dot(t1, rel);
            const double un2 = u0 * u0 + u1 * u1, un = sqrt(un2), eps = sqrt(eps2);
            const double f0 = un2 > eps2 ? un : un2 * (-un / 3.0 + eps) / (eps * eps) + eps / 3.0;
            e = mu * lam[p] * f0;
        }
    }
    return e;
}

// ground friction mu lambda (|v| - eps/2) beyond eps, else mu lambda |v|^2 / (2 eps), v the
// tangential (x, z) step (_getFrictionEnergy_gd_Reduction_3D, GIPC.cu:1357-1437)
__device__ __forceinline__ double en_fric_ground(int gi, int ng, int nv, const uint32_t* __restrict__ gp, const double* __restrict__ x,
                                 const double* __restrict__ x0, const double* __restrict__ lam, double mu,
                                 double eps2) {
    const int p = gi;
    double e = 0.0;
    if (p < ng && (int)gp[p] < nv) {
        const int v = gp[p];
        const double vx = x[3 * v] - x0[3 * v], vz = x[3 * v + 2] - x0[3 * v + 2];
        const double m2 = vx * vx + vz * vz, s = mu * lam[p], eps = sqrt(eps2);
        e = m2 > eps2 ? s * (sqrt(m2) - eps * 0.5) : s * m2 / eps * 0.5;
    }
    return e;
}

// Everything in one launch: CTA b evaluates term t where off[t] <= b < off[t + 1] (its
// elements (b - off[t]) * blockDim + threadIdx), stores its partial, and the last CTA to
// finish (a ticket counter, reset by that CTA) sums each term's partials in order into
// terms[t] and their total into terms[9].
struct EnergyOffsets {
    int off[10];
};
struct EnergyArgs {
    int nv, nt, nf, nh, ns, npair, nground, nfric, nfg;
    const double *x, *xt, *m, *x0, *rest;
    const uint32_t *tets, *tris, *hinges, *soft_idx, *gp, *fgp;
    const int32_t* adj;
    const int4 *pairs, *fpairs;
    const double *dminv, *vol, *lr, *vr, *tdminv, *area, *Q, *target, *flam, *coord, *basis, *fglam;
    double dt2, kst, ksh, srate, kb_dt2, ksoft, dhat, kappa, offset, mu, mu_gd, eps2;
};
__global__ void __launch_bounds__(SGIPC_BLOCK) k_energy(EnergyArgs a, EnergyOffsets o, double* __restrict__ part,
                                                        double* __restrict__ terms, unsigned int* __restrict__ ticket) {
    int t = 0;
    while (t < 8 && (int)blockIdx.x >= o.off[t + 1]) t++;
    const int gi = ((int)blockIdx.x - o.off[t]) * blockDim.x + threadIdx.x;
    double e = 0.0;
    switch (t) {
        case 0: e = en_kinetic(gi, a.nv, a.x, a.xt, a.m); break;
        case 1: e = en_snk(gi, a.nt, a.tets, a.x, a.dminv, a.vol, a.lr, a.vr, a.dt2); break;
        case 2: e = en_tri(gi, a.nf, a.tris, a.x, a.tdminv, a.area, a.kst, a.ksh, a.srate, a.dt2); break;
        case 3: e = en_hinge(gi, a.nh, a.hinges, a.adj, a.x, a.rest, a.Q, a.kb_dt2); break;
        case 4: e = en_soft(gi, a.ns, a.soft_idx, a.x, a.target, a.ksoft); break;
        case 5: e = en_barrier(gi, a.npair, a.nv, a.pairs, a.x, a.rest, a.dhat, a.kappa); break;
        case 6: e = en_ground(gi, a.nground, a.nv, a.gp, a.x, a.offset, a.dhat, a.kappa); break;
        case 7: e = en_friction(gi, a.nfric, a.nv, a.fpairs, a.x, a.x0, a.flam, a.coord, a.basis, a.mu, a.eps2); break;
        default: e = en_fric_ground(gi, a.nfg, a.nv, a.fgp, a.x, a.x0, a.fglam, a.mu_gd, a.eps2); break;
    }
    cta_energy(e, part);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the terms' partials side by side: warp w adds terms w and w + 8 (lane l takes partials
    // l, l + 32, ... of a term, four loads in flight, then a fixed xor tree); thread 0 adds
    // the terms in order
    __shared__ double st[9];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = w; q < 9; q += (int)(blockDim.x >> 5)) {
        double sum = 0.0;
#pragma unroll 4
        for (int i = o.off[q] + lane; i < o.off[q + 1]; i += 32) sum += __ldcg(part + i);
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
        if (lane == 0) st[q] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0.0;
        for (int q = 0; q < 9; q++) {
            terms[q] = st[q];
            total += st[q];
        }
        terms[9] = total;
        *ticket = 0u;
    }
}

}  // namespace

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
static SgipcStatus energy_launch(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k, const SgipcParams* p,
                                 cudaStream_t s, double* bytes);
static SgipcStatus check_inputs(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k, const SgipcParams* p) {
    if (!c || !f || !p) return SGIPC_BAD_INPUT;
    if (!f->vertexes || !f->xTilta || !f->masses || !f->BoundaryType) return SGIPC_BAD_INPUT;
    if (c->nt && (!f->DmInverses || !f->volum || !f->lengthRate || !f->volumeRate)) return SGIPC_BAD_INPUT;
    if (c->nf && (!f->triDmInverses || !f->area)) return SGIPC_BAD_INPUT;
    if (c->nh && (!f->quad_bending_Q || !f->rest_vertexes)) return SGIPC_BAD_INPUT;
    if (c->nsoft && !f->targetVert) return SGIPC_BAD_INPUT;
    if (!(p->dt > 0.0) || !(p->dHat > 0.0) || !(p->kappa >= 0.0)) return SGIPC_BAD_INPUT;
    if (k) {
        if (k->pair_num < 0 || k->ground_num < 0 || k->fric_num < 0 || k->fric_gd_num < 0) return SGIPC_BAD_INPUT;
        if (k->pair_num > c->max_pairs || k->ground_num > c->max_ground || k->fric_num > c->max_fric ||
            k->fric_gd_num > c->max_fric_gd) {
            snprintf(c->err, sizeof(c->err), "contact counts exceed the context capacity");
            return SGIPC_CAPACITY;
        }
        if ((k->pair_num && (!k->pairs || !f->rest_vertexes)) || (k->ground_num && !k->ground_pairs) ||
            (k->fric_num && (!k->fric_pairs || !k->fric_lambda || !k->fric_coord || !k->fric_basis || !f->o_vertexes)) ||
            (k->fric_gd_num && (!k->fric_gd_pairs || !k->fric_gd_lambda || !f->o_vertexes)))
            return SGIPC_BAD_INPUT;
    }
    return SGIPC_OK;
}

// contact items of a call: barrier and friction pairs, ground and ground-friction vertices
struct ContactCounts {
    int np = 0, nf = 0, ng = 0, ngf = 0;
    int pairs() const { return np + nf; }
    int singles() const { return ng + ngf; }
};
static ContactCounts contact_counts(const SgipcContacts* k, const SgipcParams* p) {
    ContactCounts c;
    if (!k) return c;
    c.np = k->pair_num > 0 ? k->pair_num : 0;
    c.nf = k->fric_num > 0 && p->frictionRate > 0.0 ? k->fric_num : 0;
    c.ng = k->ground_num > 0 ? k->ground_num : 0;
    c.ngf = k->fric_gd_num > 0 && p->gd_frictionRate > 0.0 ? k->fric_gd_num : 0;
    return c;
}

static ContactStore contact_store(SgipcCtx* c, const ContactCounts& cc) {
    return {c->con_ids, c->con_fac, c->con_fac2, c->con_sid, c->con_sval, c->con_key, c->con_val,
            cc.pairs(), cc.np, c->n, c->nv, c->dflag};
}

// launch the contact kernel: factors, incidences and, into grad, the singles' gradient (kGrad:
// the pairs' too)
template <bool kGrad>
static void launch_contacts(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k, const SgipcParams* p,
                            double* grad, cudaStream_t s) {
    const ContactCounts cc = contact_counts(k, p);
    if (cc.pairs() + cc.singles() == 0) return;
    ContactLaunch L{};
    L.np = cc.np;
    L.nf = cc.nf;
    L.ng = cc.ng;
    L.ngf = cc.ngf;
    L.cb = nblk(L.np, kConThreads);
    L.cf = L.cb + nblk(L.nf, kConThreads);
    L.cg = L.cf + nblk(L.ng, kConThreads);
    const int grid = L.cg + nblk(L.ngf, kConThreads);
    L.pairs = (const int4*)k->pairs;
    L.fpairs = (const int4*)k->fric_pairs;
    L.gpairs = k->ground_pairs;
    L.gfpairs = k->fric_gd_pairs;
    L.x = f->vertexes;
    L.x0 = f->o_vertexes;
    L.rest = f->rest_vertexes;
    L.flam = k->fric_lambda;
    L.fcoord = k->fric_coord;
    L.fbasis = k->fric_basis;
    L.gflam = k->fric_gd_lambda;
    L.dhat = p->dHat;
    L.kappa = p->kappa;
    L.mu = p->frictionRate;
    L.gmu = p->gd_frictionRate;
    L.eps2 = p->fDhat * p->dt * p->dt;
    L.offset = p->ground_offset;
    SG_COUNT(c, 1);
    k_contacts<kGrad><<<grid, kConThreads, 0, s>>>(L, grad, contact_store(c, cc));
}

// The contact rows (unique upper blocks, transposed lists, the pairs' gradient added into grad)
// from the stored factors of cc's pairs and `singles` singles.
static SgipcStatus merge_contacts(SgipcCtx* c, const ContactCounts& cc, int singles, const int32_t* btype,
                                  double* grad, cudaStream_t s) {
    const int m = 4 * cc.pairs() + singles, n = c->n;
    if (m == 0) {
        SG_CHECK(c, cudaMemsetAsync(c->nuc, 0, sizeof(int), s));
        SG_CHECK(c, cudaMemsetAsync(c->cu_ptr, 0, sizeof(int) * (n + 1), s));
        SG_CHECK(c, cudaMemsetAsync(c->cl_ptr, 0, sizeof(int) * (n + 1), s));
        return SGIPC_OK;
    }
    SG_COUNT(c, 5);
    SG_CHECK(c, cudaMemsetAsync(c->row_cnt, 0, kRowCounts * sizeof(int), s));
    size_t tb = c->cub_tmp_bytes;
    SG_CHECK(c, cub::DeviceRadixSort::SortPairs(c->cub_tmp, tb, c->con_key, c->con_key_s, c->con_val, c->con_val_s, m,
                                                0, c->key_bits, s));
    k_inc_rows<<<nblk(n + 1), SGIPC_BLOCK, 0, s>>>(n, m, c->con_key_s, c->inc_ptr, c->row_list, c->row_cnt, c->ucnt);
    // The split's scratch lies in the transposed blocks' values, which are written last: 72 bytes for each
    // of a pair's ten block slots, against 32 for each of its four incidences.  (A split row has at least
    // 14 incidences and no more than 3 len / 40 + 1 windows: a sixth of its incidences bounds them.)
    int* wcol = reinterpret_cast<int*>(c->cl64);
    uint32_t* wlist = reinterpret_cast<uint32_t*>(wcol + 4 * (size_t)m);
    RowWindow* win = reinterpret_cast<RowWindow*>(wlist + 3 * (size_t)m);
    static_assert(sizeof(RowWindow) == 24 && 7 * 4 + 24 / 6 <= 32, "the scratch fits");
    const RowArgs a{contact_store(c, cc), c->con_val_s, c->inc_ptr, c->row_list, c->row_cnt, n, wcol, wlist, win,
                    m / 6 + 1};
    // (the grids cover the chip once)
    const int most = nblk(m, 8);  // no more CTAs than a small call has work for
    k_row_counts<<<std::min(most, 148 * 8), 32 * kRowWarps, 0, s>>>(a, c->ucnt);
    k_row_split<<<std::min(most, 148 * 4), 32 * kSplitWarps, 0, s>>>(a, c->ucnt);
    tb = c->cub_tmp_bytes;
    SG_CHECK(c, cub::DeviceScan::ExclusiveSum(c->cub_tmp, tb, c->ucnt, c->uoff, n + 1, s));
    const RowOut o{c->uoff, btype, c->nuc, c->cu_ptr, c->cl_ptr, c->uc_row, c->uc_col, c->uc64, c->uc32, c->cl_col,
                   grad};
    SG_CHECK(c, cudaFuncSetAttribute(k_row_sums, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowShared));
    k_row_sums<<<std::min(std::max(most, 148), 148 * kRowCtas), 32 * kRowWarps, kRowShared, s>>>(a, o);
    // (no pair has more than six blocks off the diagonal)
    k_row_transposes<<<std::min(nblk(6LL * cc.pairs() + 1), 148 * 8), SGIPC_BLOCK, 0, s>>>(
        c->nuc, c->uc_row, c->uc_col, c->uc64, c->uc32, c->cl_ptr, c->cl_col, c->cl64, c->cl32);
    SG_LAUNCH_CHECK(c, "contact rows");
    return SGIPC_OK;
}

static SgipcStatus launch_fem(SgipcCtx* c, const SgipcFemData* f, const SgipcParams* p, cudaStream_t s) {
    const double dt2 = p->dt * p->dt;
    if (c->nt > 0) {
        SG_COUNT(c, 1);
        k_snk<<<nblk(c->nt, 128), 128, 0, s>>>(c->nt, c->tets, f->vertexes, f->DmInverses, f->volum, f->lengthRate,
                                               f->volumeRate, dt2, c->eblk, c->egrad);
    }
    // element block / gradient row offsets: tets (10 / 4 each), triangles (6 / 3), hinges (10 / 4)
    if (c->nf > 0) {
        SG_COUNT(c, 1);
        k_tri_bw<<<nblk(c->nf, 128), 128, 0, s>>>(c->nf, c->tris, f->vertexes, f->triDmInverses, f->area,
                                                  p->stretchStiff, p->shearStiff, p->strainRate, dt2, 10 * c->nt,
                                                  4 * c->nt, c->eblk, c->egrad);
    }
    if (c->nh > 0) {
        SG_COUNT(c, 1);
        k_hinge_quad<<<nblk(c->nh), SGIPC_BLOCK, 0, s>>>(c->nh, c->hinges, c->hinge_adj, f->vertexes, f->rest_vertexes,
                                                         f->quad_bending_Q, p->bendStiff * dt2, 4 * c->nt + 3 * c->nf,
                                                         c->hblk, c->egrad);
    }
    SG_LAUNCH_CHECK(c, "fem element kernels");
    return SGIPC_OK;
}

static void launch_gather_blocks(SgipcCtx* c, const SgipcFemData* f, cudaStream_t s) {
    auto* kernel = c->nh > 0 ? k_gather_blocks<true> : k_gather_blocks<false>;
    kernel<<<nblk(9LL * c->nnz), SGIPC_BLOCK, 0, s>>>(c->nnz, c->contrib_ptr, c->contrib, c->eblk, c->hblk,
                                                      10 * c->nt + 6 * c->nf, c->slot_row, c->col, f->BoundaryType,
                                                      f->masses, static_out(c));
}

static SgipcStatus gather_static(SgipcCtx* c, const SgipcFemData* f, cudaStream_t s) {
    c->mas.pre_scattered = 0;  // a scatter of the previous static matrix is stale
    SG_COUNT(c, 1 + (c->n_egrad > 0));
    launch_gather_blocks(c, f, s);
    if (c->n_egrad > 0)
        k_gather_grad<<<nblk(3LL * c->nv), SGIPC_BLOCK, 0, s>>>(c->nv, c->vinc_ptr, c->vinc, c->egrad, c->shape_grads);
    SG_LAUNCH_CHECK(c, "static gather");
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_assemble(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                      const SgipcParams* p, void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    // the MAS hierarchy of these contacts on its own stream, first (it needs the contact
    // graph only; started before the assembly kernels, it runs beside them and
    // sgipc_mas_build reuses it)
    if ((st = mas_mark_start(c, s)) != SGIPC_OK) return st;
    if ((st = mas_prebuild(c, k, s)) != SGIPC_OK) return st;
    c->btype = f->BoundaryType;
    c->last_fem = *f;
    c->last_prm = *p;
    c->last_has_con = k != nullptr;
    if (k) c->last_con = *k;
    SG_COUNT(c, 2 + (c->nsoft > 0));
    k_kinetic<<<nblk(3LL * c->nv), SGIPC_BLOCK, 0, s>>>(c->nv, f->vertexes, f->xTilta, f->masses, c->shape_grads, c->fb);
    // contacts (fb, contact block slots) on asm_stream, elements (element blocks, static
    // matrix, shape_grads) on s; the merge needs the soft-constraint slots from s, the
    // right-hand side both
    // (the soft constraints go first on s: the merge needs their block slots, and they add
    // to shape_grads before the element gradients do)
    cudaStream_t sc = c->asm_stream;
    const ContactCounts cc = contact_counts(k, p);
    if (c->nsoft > 0)
        k_soft<<<nblk(c->nsoft), SGIPC_BLOCK, 0, s>>>(c->nsoft, c->soft_idx, f->vertexes, f->targetVert,
                                                      p->motionRate * p->softRate * p->softRate, c->shape_grads,
                                                      contact_store(c, cc), cc.singles());
    SG_CHECK(c, cudaEventRecord(c->ev_asm[0], s));
    SG_CHECK(c, cudaStreamWaitEvent(sc, c->ev_asm[0], 0));
    launch_contacts<false>(c, f, k, p, c->fb, sc);
    SG_LAUNCH_CHECK(c, "contact kernels");
    if ((st = merge_contacts(c, cc, cc.singles() + c->nsoft, f->BoundaryType, c->fb, sc)) != SGIPC_OK) return st;
    if ((st = launch_fem(c, f, p, s)) != SGIPC_OK) return st;
    if ((st = gather_static(c, f, s)) != SGIPC_OK) return st;
    // the static blocks into the prebuilt hierarchy's domains, on the MAS stream beside the merge
    if ((st = mas_prescatter(c, s)) != SGIPC_OK) return st;
    SG_CHECK(c, cudaEventRecord(c->ev_asm[2], sc));
    SG_CHECK(c, cudaStreamWaitEvent(s, c->ev_asm[2], 0));
    k_rhs<<<nblk(3LL * c->nv), SGIPC_BLOCK, 0, s>>>(c->nv, c->fb, c->shape_grads, f->BoundaryType, c->b);
    SG_LAUNCH_CHECK(c, "rhs");
    c->assembled = 1;
    c->mas.built = 0;
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_barrier_grad_hess(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                               const SgipcParams* p, double* grad, void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    if (!grad || !k) return SGIPC_BAD_INPUT;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    SgipcContacts only = *k;
    only.fric_num = 0;
    only.ground_num = 0;
    only.fric_gd_num = 0;
    launch_contacts<false>(c, f, &only, p, grad, s);
    SG_LAUNCH_CHECK(c, "barrier");
    const ContactCounts cc = contact_counts(&only, p);
    return merge_contacts(c, cc, cc.singles(), f->BoundaryType, grad, s);
}

extern "C" SgipcStatus sgipc_friction_grad_hess(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                                const SgipcParams* p, double* grad, void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    if (!grad || !k) return SGIPC_BAD_INPUT;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    SgipcContacts only = *k;
    only.pair_num = 0;
    only.ground_num = 0;
    launch_contacts<false>(c, f, &only, p, grad, s);
    SG_LAUNCH_CHECK(c, "friction");
    const ContactCounts cc = contact_counts(&only, p);
    return merge_contacts(c, cc, cc.singles(), f->BoundaryType, grad, s);
}

extern "C" SgipcStatus sgipc_fem_grad_hess(SgipcCtx* c, const SgipcFemData* f, const SgipcParams* p, double* grad,
                                           void* stream) {
    SgipcStatus st = check_inputs(c, f, nullptr, p);
    if (st != SGIPC_OK) return st;
    if (!grad) return SGIPC_BAD_INPUT;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    if ((st = launch_fem(c, f, p, s)) != SGIPC_OK) return st;
    if ((st = gather_static(c, f, s)) != SGIPC_OK) return st;
    // gather_static added the element gradient into shape_grads; hand it to the caller
    if (c->n_egrad > 0)
        k_gather_grad<<<nblk(3LL * c->nv), SGIPC_BLOCK, 0, s>>>(c->nv, c->vinc_ptr, c->vinc, c->egrad, grad);
    SG_LAUNCH_CHECK(c, "fem gradient");
    return SGIPC_OK;
}

// ------------------------------------------------------------------------------------------
// timing hook
// ------------------------------------------------------------------------------------------
namespace sgipc {
// ---- class partition of the contact terms (affine-body points) ------------------------------
// Upper block `slot` of the contact terms: 10 per pair ((a, b) with a <= b in the pair's order),
// then one per single.  False: unused.  (r, c): its row and column, r <= c; a, b the local vertices
// with a at r.
__device__ __forceinline__ bool part_slot(const ContactStore& cs, int singles, int slot, int& r, int& c, int& item,
                                          int& a, int& b) {
    if (slot >= 10 * cs.pairs) {
        item = slot - 10 * cs.pairs;
        r = c = item < singles ? cs.sid[item] : -1;
        a = b = 0;
        return r >= 0;
    }
    item = slot / 10;
    const int k = slot % 10;
    a = k < 4 ? 0 : (k < 7 ? 1 : (k < 9 ? 2 : 3));
    b = k < 4 ? k : (k < 7 ? k - 3 : (k < 9 ? k - 5 : 3));
    const int4 id = cs.ids[item];
    const int v[4] = {id.x < 0 ? -1 : id.x & kIdMask, id.y, id.z, id.w};
    r = v[a], c = v[b];
    if (r < 0 || c < 0) return false;
    if (r > c) {
        const int t = r, u = a;
        r = c, c = t;
        a = b, b = u;
    }
    return true;
}
// its entry (p, q)
__device__ __forceinline__ double part_entry(const ContactStore& cs, int slot, int item, int a, int b, int p, int q) {
    if (slot >= 10 * cs.pairs) return cs.sval[9 * (size_t)item + 3 * p + q];
    const int type = item >= cs.barrier_pairs ? kPairFriction
                                              : ((cs.ids[item].x & kMollBit) ? kPairMollified : kPairBarrier);
    return pair_entry(type, cs.fac + kFac * (size_t)item, cs.fac2 + kFac * (size_t)item, a, b, p, q);
}

// slot s of the contact blocks: fa[s] = 1 for an ABD-ABD block, ff[s] = 1 for an ABD-FEM block
// (upper blocks: r <= c, so an ABD-FEM block has r < af <= c)
__global__ void k_part_flags(int m, int singles, ContactStore cs, int af, int* __restrict__ fa, int* __restrict__ ff) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s > m) return;
    int r, c, item, a, b;
    const bool on = s < m && part_slot(cs, singles, s, r, c, item, a, b);
    fa[s] = on && r >= af;
    ff[s] = on && r < af && c >= af;
}

// emit the flagged blocks at their scanned positions (slot order): ABD-ABD as (point, point)
// with point ids counted from af, ABD-FEM as (point, FEM vertex) with the block transposed to
// that orientation
__global__ void k_part_emit(int m, int singles, ContactStore cs, int af, const int* __restrict__ oa,
                            const int* __restrict__ of, int cap, int32_t* __restrict__ arow,
                            int32_t* __restrict__ acol, double* __restrict__ aval, int32_t* __restrict__ frow,
                            int32_t* __restrict__ fcol, double* __restrict__ fval) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    int r, c, item, a, b;
    if (s >= m || !part_slot(cs, singles, s, r, c, item, a, b) || c < af) return;
    const int i = r >= af ? oa[s] : of[s];
    if (i >= cap) return;
    if (r >= af) {
        arow[i] = r - af;
        acol[i] = c - af;
    } else {
        frow[i] = c - af;
        fcol[i] = r;
    }
    for (int p = 0; p < 3; p++)
        for (int q = 0; q < 3; q++) {
            const double v = part_entry(cs, s, item, a, b, p, q);
            if (r >= af) aval[9 * (size_t)i + 3 * p + q] = v;
            else fval[9 * (size_t)i + 3 * q + p] = v;
        }
}

__global__ void k_part_grad(int npt, int af, const double* __restrict__ g, double* __restrict__ pg) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < 3 * npt) pg[k] = g[3 * (size_t)af + k];
}

extern "C" SgipcStatus sgipc_contact_partition(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                               const SgipcParams* p, int32_t abd_first, int32_t cap,
                                               int32_t* abd_rows, int32_t* abd_cols, double* abd_vals,
                                               int32_t* abd_count, int32_t* fem_rows, int32_t* fem_cols,
                                               double* fem_vals, int32_t* fem_count, double* point_grad,
                                               void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    if (abd_first < 0 || abd_first > c->nv || cap < 0 || !abd_count || !fem_count) {
        snprintf(c->err, sizeof(c->err), "contact_partition: abd_first %d outside [0, %d] or a missing count",
                 abd_first, c->nv);
        return SGIPC_BAD_INPUT;
    }
    if (cap > 0 && (!abd_rows || !abd_cols || !abd_vals || !fem_rows || !fem_cols || !fem_vals)) return SGIPC_BAD_INPUT;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    const int npt = c->nv - abd_first;
    SG_CHECK(c, cudaMemsetAsync(c->tmp64, 0, sizeof(double) * 3 * (size_t)c->nv, s));
    launch_contacts<true>(c, f, k, p, c->tmp64, s);
    SG_LAUNCH_CHECK(c, "contact kernels (partition)");
    const ContactCounts cc = contact_counts(k, p);
    const ContactStore cs = contact_store(c, cc);
    const int m = 10 * cc.pairs() + cc.singles();
    int* fa = c->part_a;
    int* ff = c->part_f;
    SG_COUNT(c, 2 + (npt > 0 && point_grad ? 1 : 0));
    k_part_flags<<<nblk(m + 1), SGIPC_BLOCK, 0, s>>>(m, cc.singles(), cs, abd_first, fa, ff);
    size_t tb = c->cub_tmp_bytes;
    SG_CHECK(c, cub::DeviceScan::ExclusiveSum(c->cub_tmp, tb, fa, fa, m + 1, s));
    tb = c->cub_tmp_bytes;
    SG_CHECK(c, cub::DeviceScan::ExclusiveSum(c->cub_tmp, tb, ff, ff, m + 1, s));
    if (m > 0)
        k_part_emit<<<nblk(m), SGIPC_BLOCK, 0, s>>>(m, cc.singles(), cs, abd_first, fa, ff, cap, abd_rows, abd_cols,
                                                    abd_vals, fem_rows, fem_cols, fem_vals);
    if (npt > 0 && point_grad) k_part_grad<<<nblk(3LL * npt), SGIPC_BLOCK, 0, s>>>(npt, abd_first, c->tmp64, point_grad);
    SG_LAUNCH_CHECK(c, "contact partition");
    int cnt[2];
    SG_CHECK(c, cudaMemcpyAsync(&cnt[0], fa + m, sizeof(int), cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaMemcpyAsync(&cnt[1], ff + m, sizeof(int), cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaStreamSynchronize(s));
    *abd_count = cnt[0];
    *fem_count = cnt[1];
    if (cnt[0] > cap || cnt[1] > cap) {
        snprintf(c->err, sizeof(c->err), "contact_partition: %d ABD-ABD and %d ABD-FEM blocks beyond the capacity %d",
                 cnt[0], cnt[1], cap);
        return SGIPC_CAPACITY;
    }
    return SGIPC_OK;
}

// ---- barrier stiffness adaptation (GIPC::initKappa / suggestKappa / upperBoundKappa,
// GIPC.cu:9850-9929; the close-constraint checks of GIPC::postLineSearch, GIPC.cu:10777-10806)
// shape_grads += the tet rows (the first 4 * nt element gradient rows) of each vertex
__global__ void k_gather_grad_tets(int nv, int limit, const int* __restrict__ vptr, const int* __restrict__ vinc,
                                   const double* __restrict__ egrad, double* __restrict__ out) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= 3 * nv) return;
    const int v = tid / 3, q = tid % 3;
    double acc = 0.0;
    for (int k = vptr[v]; k < vptr[v + 1]; k++) {
        const int e = vinc[k];
        if (e < limit) acc += egrad[3 * (size_t)e + q];
    }
    out[tid] += acc;
}

// compute_H_b (GIPC.cu, used by suggestKappa / upperBoundKappa): the barrier's second
// derivative scale at d = 1e-16 bbox^2
static double kappa_hb(double bbox_diag2, double dhat) {
    const double d = 1.0e-16 * bbox_diag2, t = d - dhat;
    return (std::log(d / dhat) * -2.0 - t * 4.0 / d) + 1.0 / (d * d) * (t * t);
}

extern "C" SgipcStatus sgipc_init_kappa(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                        const SgipcParams* p, double mean_mass, double bbox_diag2,
                                        double min_kappa_coef, double* kappa, void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    if (!kappa || !(bbox_diag2 > 0.0)) return SGIPC_BAD_INPUT;
    if (!k || k->pair_num <= 0) return SGIPC_OK;  // the reference adapts only with contact pairs
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    const int nv = c->nv;
    double* GE = c->tmp64;   // kinetic + tet elastic + soft-constraint gradient
    double* gc = c->tmp64b;  // barrier + ground gradient at kappa = 1
    SG_COUNT(c, 2 + (c->nsoft > 0));
    k_kinetic<<<nblk(3LL * nv), SGIPC_BLOCK, 0, s>>>(nv, f->vertexes, f->xTilta, f->masses, GE, gc);
    if ((st = launch_fem(c, f, p, s)) != SGIPC_OK) return st;
    k_gather_grad_tets<<<nblk(3LL * nv), SGIPC_BLOCK, 0, s>>>(nv, 4 * c->nt, c->vinc_ptr, c->vinc, c->egrad, GE);
    if (c->nsoft > 0)
        k_soft<<<nblk(c->nsoft), SGIPC_BLOCK, 0, s>>>(c->nsoft, c->soft_idx, f->vertexes, f->targetVert,
                                                      p->motionRate * p->softRate * p->softRate, GE,
                                                      contact_store(c, ContactCounts{}), 0);
    SgipcContacts only = *k;
    only.fric_num = 0;
    only.fric_gd_num = 0;
    SgipcParams p1 = *p;
    p1.kappa = 1.0;
    p1.frictionRate = 0.0;
    p1.gd_frictionRate = 0.0;
    launch_contacts<true>(c, f, &only, &p1, gc, s);
    SG_LAUNCH_CHECK(c, "init kappa gradients");
    if ((st = dot64(c, gc, GE, 3 * nv, c->dot_out, s)) != SGIPC_OK) return st;
    if ((st = dot64(c, gc, gc, 3 * nv, c->dot_out + 1, s)) != SGIPC_OK) return st;
    double h[2];
    SG_CHECK(c, cudaMemcpyAsync(h, c->dot_out, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaStreamSynchronize(s));
    double K = *kappa;
    double minK = -h[0] / h[1];
    if (minK > 0.0) K = minK;
    const double hb = kappa_hb(bbox_diag2, p->dHat);
    // suggestKappa overwrites minKappa with its suggestion, which then bounds Kappa below
    minK = mean_mass == 0.0 ? min_kappa_coef / (4.0e-16 * bbox_diag2 * hb)
                            : min_kappa_coef * mean_mass / (4.0e-16 * bbox_diag2 * hb);
    if (K < minK) K = minK;
    double kmax = 100 * min_kappa_coef * mean_mass / (4.0e-16 * bbox_diag2 * hb);
    if (mean_mass == 0.0) kmax = 100 * min_kappa_coef / (4.0e-16 * bbox_diag2 * hb);
    if (K > kmax) K = kmax;
    *kappa = K;
    return SGIPC_OK;
}

// close constraints: ground vertices and pairs closer than dTol (squared), with their value
__global__ void k_close_ground_record(int ng, const uint32_t* __restrict__ gp, const double* __restrict__ x,
                                      double offset, double dtol, uint32_t* __restrict__ id,
                                      double* __restrict__ val, unsigned int* __restrict__ cnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ng) return;
    const uint32_t v = gp[p];
    const double d = x[3 * (size_t)v + 1] - offset, d2 = d * d;
    if (d2 < dtol) {
        const unsigned int i = atomicAdd(cnt, 1u);
        id[i] = v;
        val[i] = d2;
    }
}

__global__ void k_close_pair_record(int np, const int4* __restrict__ pairs, const double* __restrict__ x,
                                    double dtol, int4* __restrict__ id, double* __restrict__ val,
                                    unsigned int* __restrict__ cnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    int v[4], nvp;
    const int kind = decode_pair(pairs[p], v, nvp);
    d3 X[4], g[4];
#pragma unroll
    for (int a = 0; a < 4; a++) X[a] = a < nvp ? ld3(x, v[a]) : mk(0, 0, 0);
    const double d2 = dist2_grad(kind, X, g);
    if (d2 < dtol) {
        const unsigned int i = atomicAdd(cnt + 1, 1u);
        id[i] = pairs[p];
        val[i] = d2;
    }
}

// flag[0] = 1 when a recorded ground vertex or pair is closer now than when recorded
__global__ void k_close_check(int ng, int np, const uint32_t* __restrict__ gid, const double* __restrict__ gval,
                              const int4* __restrict__ pid, const double* __restrict__ pval,
                              const double* __restrict__ x, double offset, int* __restrict__ flag) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ng) {
        const double d = x[3 * (size_t)gid[t] + 1] - offset;
        if (d * d < gval[t]) *flag = 1;
    } else if (t < ng + np) {
        int v[4], nvp;
        const int kind = decode_pair(pid[t - ng], v, nvp);
        d3 X[4], g[4];
#pragma unroll
        for (int a = 0; a < 4; a++) X[a] = a < nvp ? ld3(x, v[a]) : mk(0, 0, 0);
        if (dist2_grad(kind, X, g) < pval[t - ng]) *flag = 1;
    }
}

extern "C" SgipcStatus sgipc_close_record(SgipcCtx* c, const double* x, const SgipcContacts* k, double dtol,
                                          double ground_offset, int32_t* counts, void* stream) {
    if (!c || !x || !k || (k->pair_num > 0 && !k->pairs) || (k->ground_num > 0 && !k->ground_pairs))
        return SGIPC_BAD_INPUT;
    if (k->pair_num > c->max_pairs || k->ground_num > c->max_ground) return SGIPC_CAPACITY;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    if (!c->close_cnt) {
        SG_CHECK(c, cudaMalloc((void**)&c->close_gid, sizeof(uint32_t) * (size_t)std::max(c->max_ground, 1)));
        SG_CHECK(c, cudaMalloc((void**)&c->close_gval, sizeof(double) * (size_t)std::max(c->max_ground, 1)));
        SG_CHECK(c, cudaMalloc((void**)&c->close_pid, sizeof(int4) * (size_t)std::max(c->max_pairs, 1)));
        SG_CHECK(c, cudaMalloc((void**)&c->close_pval, sizeof(double) * (size_t)std::max(c->max_pairs, 1)));
        SG_CHECK(c, cudaMalloc((void**)&c->close_cnt, sizeof(unsigned int) * 4));
    }
    SG_CHECK(c, cudaMemsetAsync(c->close_cnt, 0, sizeof(unsigned int) * 4, s));
    SG_COUNT(c, (k->ground_num > 0) + (k->pair_num > 0));
    if (k->ground_num > 0)
        k_close_ground_record<<<nblk(k->ground_num), SGIPC_BLOCK, 0, s>>>(
            k->ground_num, k->ground_pairs, x, ground_offset, dtol, c->close_gid, c->close_gval, c->close_cnt);
    if (k->pair_num > 0)
        k_close_pair_record<<<nblk(k->pair_num), SGIPC_BLOCK, 0, s>>>(
            k->pair_num, (const int4*)k->pairs, x, dtol, (int4*)c->close_pid, c->close_pval, c->close_cnt);
    SG_LAUNCH_CHECK(c, "close constraints");
    unsigned int h[2];
    SG_CHECK(c, cudaMemcpyAsync(h, c->close_cnt, 2 * sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaStreamSynchronize(s));
    c->close_num[0] = (int)h[0];
    c->close_num[1] = (int)h[1];
    if (counts) {
        counts[0] = (int32_t)h[0];
        counts[1] = (int32_t)h[1];
    }
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_close_check(SgipcCtx* c, const double* x, double ground_offset, int32_t* changed,
                                         void* stream) {
    if (!c || !x || !changed) return SGIPC_BAD_INPUT;
    *changed = 0;
    const int ng = c->close_cnt ? c->close_num[0] : 0, np = c->close_cnt ? c->close_num[1] : 0;
    if (ng + np == 0) return SGIPC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    SG_CHECK(c, cudaMemsetAsync(c->close_cnt + 2, 0, sizeof(unsigned int), s));
    SG_COUNT(c, 1);
    k_close_check<<<nblk(ng + np), SGIPC_BLOCK, 0, s>>>(ng, np, c->close_gid, c->close_gval, (const int4*)c->close_pid,
                                                        c->close_pval, x, ground_offset,
                                                        reinterpret_cast<int*>(c->close_cnt + 2));
    SG_LAUNCH_CHECK(c, "close check");
    unsigned int h = 0;
    SG_CHECK(c, cudaMemcpyAsync(&h, c->close_cnt + 2, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaStreamSynchronize(s));
    *changed = h != 0;
    return SGIPC_OK;
}

SgipcStatus assemble_time_hook(SgipcCtx* c, const char* name, cudaStream_t s, double* bytes) {
    const SgipcFemData* f = &c->last_fem;
    const SgipcParams* p = &c->last_prm;
    const SgipcContacts* k = c->last_has_con ? &c->last_con : nullptr;
    double* scratch = c->tmp64b;  // gradient sink that keeps fb untouched
    if (!strcmp(name, "energy")) return energy_launch(c, f, k, p, s, bytes);
    if (!strcmp(name, "snk")) {
        if (c->nt <= 0) return SGIPC_BAD_INPUT;
        SG_COUNT(c, 1);
        k_snk<<<nblk(c->nt, 128), 128, 0, s>>>(c->nt, c->tets, f->vertexes, f->DmInverses, f->volum, f->lengthRate,
                                               f->volumeRate, p->dt * p->dt, c->eblk, c->egrad);
        // positions, DmInv, volume, (mu, lambda), indices in; 10 FP64 blocks and 4 gradient rows out
        *bytes = (double)c->nt * (4 * 24 + 72 + 8 + 16 + 16 + 10 * 72 + 12 * 8);
    } else if (!strcmp(name, "gather_blocks")) {
        SG_COUNT(c, 1);
        launch_gather_blocks(c, f, s);
        // element blocks and their indices in; per upper slot its indices, flags and the FP64
        // upper value out, the full-pattern FP64 + FP32 copy, and the transposed copy off the
        // diagonal
        *bytes = (double)(10LL * c->nt + 6LL * c->nf) * 72 + 80.0 * c->nh + 4.0 * c->n_eblk +
                 (double)c->nnz * (28 + 72 + 108) + (double)(c->nnz - c->n) * 108;
    } else if (!strcmp(name, "barrier") || !strcmp(name, "friction")) {
        // one kind's launch, into the places of the first pairs (the factors and keys are scratch: every
        // assembly writes them anew before it reads them)
        if (!k) return SGIPC_BAD_INPUT;
        const bool fric = name[0] == 'f';
        SgipcContacts only = *k;
        only.ground_num = only.fric_gd_num = 0;
        if (fric) only.pair_num = 0;
        else only.fric_num = 0;
        const ContactCounts cc = contact_counts(&only, p);
        if (cc.pairs() <= 0) return SGIPC_BAD_INPUT;
        launch_contacts<false>(c, f, &only, p, scratch, s);
        // pair, 4 positions and 4 rest (or start-of-step) positions in, the friction data; ids,
        // incidence keys and values, and the factors out
        *bytes = (double)cc.pairs() * (16 + 8 * 24 + (fric ? 8 + 16 + 48 : 0) + 16 + 4 * 8 + 8 * kFac);
    } else {
        return SGIPC_NOT_READY;
    }
    SG_LAUNCH_CHECK(c, name);
    return SGIPC_OK;
}
}  // namespace sgipc

// ------------------------------------------------------------------------------------------
// line-search energy: host side
// ------------------------------------------------------------------------------------------
// Launch the energy kernels and the final sum on s (no synchronisation); the last CTA writes the
// terms straight into pinned host memory (c->h_en).
// Terms: 0 kinetic, 1 tets, 2 triangles, 3 hinges, 4 soft, 5 barrier, 6 ground, 7 friction,
// 8 ground friction; 9 the total.  *bytes: algorithmic bytes of the launch sequence.
static SgipcStatus energy_launch(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k, const SgipcParams* p,
                                 cudaStream_t s, double* bytes) {
    const double dt2 = p->dt * p->dt, eps2 = p->fDhat * dt2;
    const int npair = k ? k->pair_num : 0, nground = k ? k->ground_num : 0;
    const int nfric = k && p->frictionRate > 0.0 ? k->fric_num : 0;
    const int nfg = k && p->gd_frictionRate > 0.0 ? k->fric_gd_num : 0;
    const int cnt[9] = {c->nv, c->nt, c->nf, c->nh, c->nsoft, npair, nground, nfric, nfg};
    EnergyOffsets o;
    o.off[0] = 0;
    for (int t = 0; t < 9; t++) o.off[t + 1] = o.off[t] + nblk(cnt[t]);
    if (o.off[9] > c->en_cap) {
        snprintf(c->err, sizeof(c->err), "energy: %d partial sums exceed the context's %d", o.off[9], c->en_cap);
        return SGIPC_CAPACITY;
    }
    EnergyArgs a;
    a.nv = c->nv; a.nt = c->nt; a.nf = c->nf; a.nh = c->nh; a.ns = c->nsoft;
    a.npair = npair; a.nground = nground; a.nfric = nfric; a.nfg = nfg;
    a.x = f->vertexes; a.xt = f->xTilta; a.m = f->masses; a.x0 = f->o_vertexes; a.rest = f->rest_vertexes;
    a.tets = c->tets; a.tris = c->tris; a.hinges = c->hinges; a.soft_idx = c->soft_idx;
    a.gp = k ? k->ground_pairs : nullptr; a.fgp = k ? k->fric_gd_pairs : nullptr; a.adj = c->hinge_adj;
    a.pairs = k ? (const int4*)k->pairs : nullptr; a.fpairs = k ? (const int4*)k->fric_pairs : nullptr;
    a.dminv = f->DmInverses; a.vol = f->volum; a.lr = f->lengthRate; a.vr = f->volumeRate;
    a.tdminv = f->triDmInverses; a.area = f->area; a.Q = f->quad_bending_Q; a.target = f->targetVert;
    a.flam = k ? k->fric_lambda : nullptr; a.coord = k ? k->fric_coord : nullptr; a.basis = k ? k->fric_basis : nullptr;
    a.fglam = k ? k->fric_gd_lambda : nullptr;
    a.dt2 = dt2; a.kst = p->stretchStiff; a.ksh = p->shearStiff; a.srate = p->strainRate; a.kb_dt2 = p->bendStiff * dt2;
    a.ksoft = p->motionRate * p->softRate * p->softRate; a.dhat = p->dHat; a.kappa = p->kappa;
    a.offset = p->ground_offset; a.mu = p->frictionRate; a.mu_gd = p->gd_frictionRate; a.eps2 = eps2;
    k_energy<<<o.off[9], SGIPC_BLOCK, 0, s>>>(a, o, c->en_part, c->h_en, c->en_ticket);
    SG_COUNT(c, 1);
    SG_LAUNCH_CHECK(c, "energy");
    if (bytes)  // positions (and the per-element inputs) in, one partial per CTA out and back
        *bytes = (double)c->nv * (24 + 24 + 8) + (double)c->nt * (16 + 4 * 24 + 72 + 8 + 16) +
                 (double)c->nf * (12 + 3 * 24 + 32 + 8) + (double)c->nh * (16 + 4 * 24 + 2 * 24 + 128) +
                 (double)c->nsoft * (4 + 24 + 24) + (double)npair * (16 + 4 * 24 + 4 * 24) + (double)nground * (4 + 8) +
                 (double)nfric * (16 + 8 + 16 + 48 + 8 * 24) + (double)nfg * (4 + 8 + 48) + 2.0 * 8 * o.off[9];
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_compute_energy(SgipcCtx* c, const SgipcFemData* f, const SgipcContacts* k,
                                            const SgipcParams* p, double* energy, double* terms, void* stream) {
    SgipcStatus st = check_inputs(c, f, k, p);
    if (st != SGIPC_OK) return st;
    if (!energy) return SGIPC_BAD_INPUT;
    cudaStream_t s = (cudaStream_t)stream;
    SG_DEVICE(c);
    if ((st = energy_launch(c, f, k, p, s, nullptr)) != SGIPC_OK) return st;
    SG_CHECK(c, cudaStreamSynchronize(s));
    *energy = c->h_en[9];
    if (terms)
        for (int t = 0; t < 9; t++) terms[t] = c->h_en[t];
    return SGIPC_OK;
}
