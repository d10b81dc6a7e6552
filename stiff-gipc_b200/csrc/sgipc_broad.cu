// sgipc_broad.cu — the contact pairs of a Newton iterate and the lagged friction set-up on the GPU.
//
// GIPC::buildCP (StiffGIPC/GIPC.cu:9065-9083) finds, through two LBVHs (mlbvh.cu), every
// surface point closer than d-hat to a surface triangle and every pair of surface edges closer
// than d-hat, and encodes each as the int4 the barrier kernels read (_checkPTintersection /
// _checkEEintersection, mlbvh.cu:534-1059), with its CCD candidate, its MatIndex (the pair's rank
// among the pairs of its Hessian size) and the counters _cpNum[5] (total, -, two-, three- and
// four-vertex pairs); _GroundCollisionDetect (GIPC.cu:6433) lists the surface points near the
// ground.  The reference appends with atomics, so its order changes from run to run.
//
// Here two packed trees of fan-out 32 replace them.  The triangles, the edges and the surface
// points are sorted together by the Morton code of their box centres (one radix sort); 32
// consecutive primitives form a leaf group, 32 groups a node, and a box is stored for every
// primitive, group and node: there is no tree to build, only the boxes to reduce.  A warp takes
// 32 neighbouring queries (points against triangles, edges against the edges behind them in
// the sorted order) and walks the nodes and groups whose box meets the union of its queries'
// boxes, one child per lane; the pairs of groups are then shared out evenly, one per warp: the
// primitives that meet a query's own box are queued, and every 32 queued candidates are tested
// exactly, one per lane.  Boxes are FP32, rounded outwards, so
// that they only ever let more candidates through; every decision is made in FP64.  (The
// search was a uniform grid before, its cell as wide as the scene's largest primitive, with
// one thread per query and two passes: with small primitives beside large ones a cell held
// hundreds of candidates, and the exact test ran in whichever lane had found one.)
//
// The records found are 64-bit keys (kind, query, primitive) and sorted once, which gives a
// deterministic order: point-triangle pairs by surface point, then by triangle; edge-edge pairs
// by (edge, other edge); then the ground points.  The pairs are encoded from the sorted keys,
// and MatIndex is the rank in that order.  The pair tests restate the reference's
// closest-feature classification and squared distances term for term; this file is compiled
// without contracting multiply-adds (-fmad=false), so a pair at the edge of d-hat, or of a
// feature region, is decided as the reference's own arithmetic decides it.
//
// The lagged friction set-up (_calFrictionLastH_DistAndTan / _calFrictionLastH_gd,
// GIPC.cu:8362-8499, run once per frame in GIPC.cu:8660-8696) maps every non-mollified pair to
// its normal force, closest-point coordinates and tangent basis (FrictionUtils.cuh:52-399);
// the outputs keep the input order.
#include <cub/cub.cuh>

#include "sgipc_geom.cuh"
#include "sgipc_internal.cuh"

namespace sgipc {

// per-context buffers of the pair search (grown when a call needs more)
struct BroadWork {
    int cap_prim = 0, cap_leaf = 0, cap_item = 0, cap_rec = 0, cap_q = 0;
    unsigned* key = nullptr;               // [primitives] kind and Morton code
    unsigned* key_s = nullptr;
    int* val = nullptr;                    // [primitives] index within its kind
    int* val_s = nullptr;
    float4* leaf = nullptr;                // [2 * leaves] boxes in sorted order: (lo, index), (hi, -)
    float4* group = nullptr;               // [2 * leaves / 32]
    float4* node = nullptr;                // [2 * leaves / 1024]
    int2* item = nullptr;                  // [2 * items] query group and leaf group that meet
    unsigned long long* bounds = nullptr;  // [8] ordered min xyz, max xyz, largest box extent, bad index
    int* gflag = nullptr;                  // [pairs + 1] friction set-up: takes part, and its place
    int* goff = nullptr;
    unsigned long long* reckey = nullptr;  // [records] kind, query, primitive
    unsigned long long* reckey_s = nullptr;
    unsigned long long* gscan = nullptr;   // [records] packed ranks per Hessian size
    unsigned int* d_counts = nullptr;      // [16] see Count
    unsigned int* h_counts = nullptr;      // pinned copy
    void* cub = nullptr;
    size_t cub_bytes = 0;
};

}  // namespace sgipc

using namespace sgipc;

namespace {

constexpr int kSpanBits = 21;  // a scene's extent over its largest primitive's, at most
constexpr int kGroupBits = 21;  // packed rank fields: three 21-bit counters in one 64-bit word
constexpr int kQueryWarps = 4;
constexpr int kQueryCtas = 4;  // per SM (128 registers a thread)
constexpr int kNodeLeaves = 1024;  // primitives below a node: 32 groups of 32
// d_counts: records, ground points, scene error, pairs per Hessian size, edge and point items
enum Count { kCntRec = 0, kCntGround = 2, kCntBad = 3, kCntSize = 4, kCntItem = 8, kCntNum = 16 };
constexpr int kItemsPerGroup = 64;  // items of one kind the lists hold per query group, on average

// order-preserving map of doubles to unsigned integers (min / max by integer atomics)
__device__ __forceinline__ unsigned long long ord(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double unord(unsigned long long u) {
    return __longlong_as_double((long long)((u >> 63) ? (u & 0x7fffffffffffffffull) : ~u));
}

__device__ __forceinline__ d3 ldp(const double* x, unsigned v) { return {x[3 * v], x[3 * v + 1], x[3 * v + 2]}; }

constexpr int kBoundsWarps = 8;

// scene bounds of the surface points and the largest extent of a triangle or edge box;
// bounds[7] != 0 when an index names no vertex (nothing is loaded from such an index)
__global__ void k_bounds(const double* __restrict__ x, int nv, const unsigned* __restrict__ sv, int nsv,
                         const unsigned* __restrict__ faces, int nf, const unsigned* __restrict__ edges, int ne,
                         unsigned long long* bounds) {
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, ext = 0.0;
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nsv + nf + ne; i += stride) {
        if (i < nsv) {
            if (sv[i] >= (unsigned)nv) {
                atomicOr(bounds + 7, 1ull);
                continue;
            }
            const d3 p = ldp(x, sv[i]);
            lo[0] = fmin(lo[0], p.x), lo[1] = fmin(lo[1], p.y), lo[2] = fmin(lo[2], p.z);
            hi[0] = fmax(hi[0], p.x), hi[1] = fmax(hi[1], p.y), hi[2] = fmax(hi[2], p.z);
        } else {
            const bool tri = i < nsv + nf;
            const int k = tri ? i - nsv : i - nsv - nf;
            const unsigned* v = tri ? faces + 3 * k : edges + 2 * k;
            if (v[0] >= (unsigned)nv || v[1] >= (unsigned)nv || (tri && v[2] >= (unsigned)nv)) {
                atomicOr(bounds + 7, 1ull);
                continue;
            }
            const d3 a = ldp(x, v[0]), b = ldp(x, v[1]), c = tri ? ldp(x, v[2]) : a;
            ext = fmax(ext, fmax(fmax(a.x, b.x), c.x) - fmin(fmin(a.x, b.x), c.x));
            ext = fmax(ext, fmax(fmax(a.y, b.y), c.y) - fmin(fmin(a.y, b.y), c.y));
            ext = fmax(ext, fmax(fmax(a.z, b.z), c.z) - fmin(fmin(a.z, b.z), c.z));
        }
    }
    // one atomic per value and CTA
    __shared__ double s_red[kBoundsWarps][7];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v[7] = {lo[0], lo[1], lo[2], -hi[0], -hi[1], -hi[2], -ext};  // all minima
#pragma unroll
    for (int q = 0; q < 7; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] = fmin(v[q], __shfl_xor_sync(0xffffffffu, v[q], o));
        if (lane == 0) s_red[w][q] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double m = s_red[0][threadIdx.x];
        for (int k = 1; k < kBoundsWarps; k++) m = fmin(m, s_red[k][threadIdx.x]);
        if (threadIdx.x < 3) atomicMin(bounds + threadIdx.x, ord(m));
        else atomicMax(bounds + threadIdx.x, ord(-m));
    }
}

// 1 when the scene spans more than 2^21 times its largest primitive along an axis (or is not
// finite), 2 when an index names no vertex (every later kernel then returns at once)
__device__ int scene_error(const unsigned long long* bounds, double gap) {
    const double ext = unord(bounds[6]);
    const double h = (ext + 2.0 * gap) * 1.001 + 1e-12;
    int bad = 0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const double lo = unord(bounds[q]), hi = unord(bounds[3 + q]);
        if (!(hi >= lo) || (hi - (lo - gap - h)) / h + 2.0 >= (double)(1 << kSpanBits)) bad = 1;
    }
    return bounds[7] ? 2 : bad;
}

// grown box of a triangle (grow = gap) or an edge (grow = gap / 2)
struct Box {
    d3 lo, hi;
};
__device__ __forceinline__ Box grown_box(const double* x, const unsigned* v, int nvert, double grow) {
    d3 a = ldp(x, v[0]), lo = a, hi = a;
    for (int k = 1; k < nvert; k++) {
        const d3 b = ldp(x, v[k]);
        lo = {fmin(lo.x, b.x), fmin(lo.y, b.y), fmin(lo.z, b.z)};
        hi = {fmax(hi.x, b.x), fmax(hi.y, b.y), fmax(hi.z, b.z)};
    }
    return {{lo.x - grow, lo.y - grow, lo.z - grow}, {hi.x + grow, hi.y + grow, hi.z + grow}};
}

// ten bits, spread to every third
__device__ __forceinline__ unsigned spread3(unsigned v) {
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}

// Sort keys: kind (0 triangle, 1 edge, 2 surface point) above the 30-bit Morton code of the
// box centre in the scene's bounds.  Ten bits an axis: finer codes sort no better (primitives of
// one code stay in mesh order, which is local) and cost a radix pass each.
__global__ void k_keys(const double* __restrict__ x, const unsigned* __restrict__ faces, int nf,
                       const unsigned* __restrict__ edges, int ne, const unsigned* __restrict__ sv, int nsv,
                       const unsigned long long* __restrict__ bounds, double gap, unsigned* __restrict__ key,
                       int* __restrict__ val, unsigned* __restrict__ counts) {
    __shared__ int s_bad;
    __shared__ double s_lo[3], s_scale[3];
    if (threadIdx.x == 0) {
        s_bad = scene_error(bounds, gap);
        if (blockIdx.x == 0) counts[kCntBad] = (unsigned)s_bad;
    }
    if (threadIdx.x < 3) {
        const double lo = unord(bounds[threadIdx.x]), hi = unord(bounds[3 + threadIdx.x]);
        s_lo[threadIdx.x] = lo;
        s_scale[threadIdx.x] = hi > lo ? 1024.0 / (hi - lo) : 0.0;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nf + ne + nsv || s_bad) return;
    const int kind = i < nf ? 0 : (i < nf + ne ? 1 : 2);
    const int p = i - (kind > 0 ? nf : 0) - (kind > 1 ? ne : 0);
    const unsigned* v = kind == 0 ? faces + 3 * (size_t)p : (kind == 1 ? edges + 2 * (size_t)p : sv + p);
    const Box b = grown_box(x, v, 3 - kind, 0.0);
    const double c[3] = {0.5 * (b.lo.x + b.hi.x), 0.5 * (b.lo.y + b.hi.y), 0.5 * (b.lo.z + b.hi.z)};
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < 3; q++)
        m |= spread3((unsigned)fmin(fmax((c[q] - s_lo[q]) * s_scale[q], 0.0), 1023.0)) << q;
    key[i] = ((unsigned)kind << 30) | m;
    val[i] = p;
}

// FP32 boxes that enclose FP64 ones
struct BoxF {
    float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ BoxF outward(const Box& b) {
    return {__double2float_rd(b.lo.x), __double2float_rd(b.lo.y), __double2float_rd(b.lo.z),
            __double2float_ru(b.hi.x), __double2float_ru(b.hi.y), __double2float_ru(b.hi.z)};
}
__device__ __forceinline__ BoxF empty_box() { return {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY}; }
__device__ __forceinline__ bool meet(const BoxF& a, const BoxF& b) {
    return !(a.lx > b.hx || b.lx > a.hx || a.ly > b.hy || b.ly > a.hy || a.lz > b.hz || b.lz > a.hz);
}
__device__ __forceinline__ BoxF warp_union(BoxF b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        b.lx = fminf(b.lx, __shfl_xor_sync(0xffffffffu, b.lx, o));
        b.ly = fminf(b.ly, __shfl_xor_sync(0xffffffffu, b.ly, o));
        b.lz = fminf(b.lz, __shfl_xor_sync(0xffffffffu, b.lz, o));
        b.hx = fmaxf(b.hx, __shfl_xor_sync(0xffffffffu, b.hx, o));
        b.hy = fmaxf(b.hy, __shfl_xor_sync(0xffffffffu, b.hy, o));
        b.hz = fmaxf(b.hz, __shfl_xor_sync(0xffffffffu, b.hz, o));
    }
    return b;
}
__device__ __forceinline__ BoxF shfl_box(const BoxF& b, int j) {
    return {__shfl_sync(0xffffffffu, b.lx, j), __shfl_sync(0xffffffffu, b.ly, j), __shfl_sync(0xffffffffu, b.lz, j),
            __shfl_sync(0xffffffffu, b.hx, j), __shfl_sync(0xffffffffu, b.hy, j), __shfl_sync(0xffffffffu, b.hz, j)};
}
__device__ __forceinline__ void store_box(float4* at, int i, const BoxF& b, int id) {
    at[2 * (size_t)i] = make_float4(b.lx, b.ly, b.lz, __int_as_float(id));
    at[2 * (size_t)i + 1] = make_float4(b.hx, b.hy, b.hz, 0.f);
}
__device__ __forceinline__ BoxF load_box(const float4* at, int i, int& id) {
    const float4 l = __ldg(at + 2 * (size_t)i), h = __ldg(at + 2 * (size_t)i + 1);
    id = __float_as_int(l.w);
    return {l.x, l.y, l.z, h.x, h.y, h.z};
}

// Boxes of the sorted triangles (grown by the gap) and edges (by half of it), of their groups of
// 32 and of their nodes of 1024, one node per CTA; the first tri_nodes CTAs take the triangles.
// Places beyond the last primitive get empty boxes and index -1.
__global__ void __launch_bounds__(kNodeLeaves) k_boxes(const double* __restrict__ x,
                                                       const unsigned* __restrict__ faces, int nf,
                                                       const unsigned* __restrict__ edges, int ne, int tri_nodes,
                                                       const int* __restrict__ val, double gap,
                                                       const unsigned* __restrict__ counts, float4* leaf,
                                                       float4* group, float4* node) {
    __shared__ BoxF s_group[32];
    if (counts[kCntBad]) return;
    const bool tri = (int)blockIdx.x < tri_nodes;
    const int k = ((int)blockIdx.x - (tri ? 0 : tri_nodes)) * kNodeLeaves + threadIdx.x;
    BoxF b = empty_box();
    int p = -1;
    if (k < (tri ? nf : ne)) {
        p = val[tri ? k : nf + k];
        b = tri ? outward(grown_box(x, faces + 3 * (size_t)p, 3, gap)) : outward(grown_box(x, edges + 2 * (size_t)p, 2, 0.5 * gap));
    }
    const int i = blockIdx.x * kNodeLeaves + threadIdx.x, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    store_box(leaf, i, b, p);
    b = warp_union(b);
    if (lane == 0) {
        s_group[w] = b;
        store_box(group, i >> 5, b, 0);
    }
    __syncthreads();
    if (w == 0) {
        b = warp_union(s_group[lane]);
        if (lane == 0) store_box(node, blockIdx.x, b, 0);
    }
}

struct PairOut {
    int4 pair, ccd;
    int group;  // 0: two vertices (6 x 6), 1: three (9 x 9), 2: four (12 x 12)
};

// _checkPTintersection (mlbvh.cu:534-645): point p against triangle (a, b, c)
__device__ __forceinline__ bool check_pt(const double* x, unsigned p, unsigned a, unsigned b, unsigned c, double dhat,
                                         PairOut& o) {
    const d3 v0 = ldp(x, p), v1 = ldp(x, a), v2 = ldp(x, b), v3 = ldp(x, c);
    const int t = pt_type(v0, v1, v2, v3);
    double d;
    switch (t) {
        case 0: d = pp_d2(v0, v1); break;
        case 1: d = pp_d2(v0, v2); break;
        case 2: d = pp_d2(v0, v3); break;
        case 3: d = pe_d2(v0, v1, v2); break;
        case 4: d = pe_d2(v0, v2, v3); break;
        case 5: d = pe_d2(v0, v3, v1); break;
        default: d = pplane_d2(v0, v1, v2, v3); break;
    }
    if (!(d < dhat)) return false;
    const int q = -(int)p - 1;
    o.ccd = make_int4(q, (int)a, (int)b, (int)c);
    switch (t) {
        case 0: o.pair = make_int4(q, (int)a, -1, -1), o.group = 0; break;
        case 1: o.pair = make_int4(q, (int)b, -1, -1), o.group = 0; break;
        case 2: o.pair = make_int4(q, (int)c, -1, -1), o.group = 0; break;
        case 3: o.pair = make_int4(q, (int)a, (int)b, -1), o.group = 1; break;
        case 4: o.pair = make_int4(q, (int)b, (int)c, -1), o.group = 1; break;
        case 5: o.pair = make_int4(q, (int)c, (int)a, -1), o.group = 1; break;
        default: o.pair = make_int4(q, (int)a, (int)b, (int)c), o.group = 2; break;
    }
    return true;
}

// _checkEEintersection (mlbvh.cu:685-1059): edge (i0, i1) against the other edge (i2, i3) of
// index other; nearly parallel edges mark their point-point / point-edge pair with
// w = -other - 2 (the mollified encodings are off in the reference, smooth = false)
__device__ __forceinline__ bool check_ee(const double* x, const double* rest, unsigned i0, unsigned i1, unsigned i2,
                                         unsigned i3, int other, double dhat, PairOut& o) {
    const d3 v0 = ldp(x, i0), v1 = ldp(x, i1), v2 = ldp(x, i2), v3 = ldp(x, i3);
    const int t = ee_type(v0, v1, v2, v3);
    double d;
    switch (t) {
        case 0: d = pp_d2(v0, v2); break;
        case 1: d = pp_d2(v0, v3); break;
        case 2: d = pe_d2(v0, v2, v3); break;
        case 3: d = pp_d2(v1, v2); break;
        case 4: d = pp_d2(v1, v3); break;
        case 5: d = pe_d2(v1, v2, v3); break;
        case 6: d = pe_d2(v2, v0, v1); break;
        case 7: d = pe_d2(v3, v0, v1); break;
        default: d = ll_d2(v0, v1, v2, v3); break;
    }
    if (!(d < dhat)) return false;
    const d3 r0 = ldp(rest, i0), r1 = ldp(rest, i1), r2 = ldp(rest, i2), r3 = ldp(rest, i3);
    const double cr = sq(cross(v0 - v1, v2 - v3));
    const double eps = 1e-3 * sq(r0 - r1) * sq(r2 - r3);
    const int add_e = cr < eps ? -other - 2 : -1;
    const int a = (int)i0, b = (int)i1, c = (int)i2, e = (int)i3;
    o.ccd = make_int4(a, b, c, e);
    switch (t) {
        case 0: o.pair = make_int4(-a - 1, c, -1, add_e), o.group = 0; break;
        case 1: o.pair = make_int4(-a - 1, e, -1, add_e), o.group = 0; break;
        case 2: o.pair = make_int4(-a - 1, c, e, add_e), o.group = 1; break;
        case 3: o.pair = make_int4(-b - 1, c, -1, add_e), o.group = 0; break;
        case 4: o.pair = make_int4(-b - 1, e, -1, add_e), o.group = 0; break;
        case 5: o.pair = make_int4(-b - 1, c, e, add_e), o.group = 1; break;
        case 6: o.pair = make_int4(-c - 1, a, b, add_e), o.group = 1; break;
        case 7: o.pair = make_int4(-e - 1, a, b, add_e), o.group = 1; break;
        default: o.pair = make_int4(a, b, c, e), o.group = 2; break;
    }
    return true;
}

struct QueryArgs {
    const double* x;
    const double* rest;
    const unsigned* sv;
    const unsigned* faces;
    const unsigned* edges;
    const int* body;
    const int* btype;
    int nsv, nf, ne;
    double dhat, gap, ground_offset;
    const int* val;  // the sorted order: triangles, edges, surface points
    const float4* leaf;
    const float4* group;
    const float4* node;
    int tri_nodes, edge_nodes, edge_groups, point_groups;
    int2* item;  // [item_cap] of the edges, then [item_cap] of the points
    unsigned item_cap;
    unsigned* counts;
    unsigned long long* rec;
    unsigned rec_cap;
    int qshift, kshift;  // key = kind << kshift | query << qshift | primitive
};

__device__ __forceinline__ bool all_fixed(const int* bt, unsigned a, unsigned b, unsigned c, unsigned d) {
    return bt && bt[a] >= 2 && bt[b] >= 2 && bt[c] >= 2 && bt[d] >= 2;
}

// surface point q against triangle f, with _selfQuery_vf's filters (mlbvh.cu:1350-1362)
__device__ __forceinline__ bool test_pt(const QueryArgs& a, int q, int f, PairOut& o) {
    const unsigned p = a.sv[q];
    const unsigned t0 = a.faces[3 * (size_t)f], t1 = a.faces[3 * (size_t)f + 1], t2 = a.faces[3 * (size_t)f + 2];
    if (!(a.body[p] != a.body[t0] || a.body[p] == -1)) return false;
    if (p == t0 || p == t1 || p == t2) return false;
    if (all_fixed(a.btype, p, t0, t1, t2)) return false;
    return check_pt(a.x, p, t0, t1, t2, a.dhat, o);
}

// edge s against the edge `other` > s, with _selfQuery_ee's filters (mlbvh.cu:1550-1566); the two
// boxes, each grown by half the gap, have to overlap
__device__ __forceinline__ bool test_ee(const QueryArgs& a, int s, int other, PairOut& o) {
    const unsigned e0 = a.edges[2 * (size_t)s], e1 = a.edges[2 * (size_t)s + 1];
    const unsigned f0 = a.edges[2 * (size_t)other], f1 = a.edges[2 * (size_t)other + 1];
    if (!(a.body[e0] != a.body[f0] || a.body[e0] == -1)) return false;
    if (e0 == f0 || e0 == f1 || e1 == f0 || e1 == f1) return false;
    if (all_fixed(a.btype, e0, e1, f0, f1)) return false;
    const Box bs = grown_box(a.x, a.edges + 2 * (size_t)s, 2, 0.5 * a.gap);
    const Box bo = grown_box(a.x, a.edges + 2 * (size_t)other, 2, 0.5 * a.gap);
    if (bo.lo.x > bs.hi.x || bs.lo.x > bo.hi.x || bo.lo.y > bs.hi.y || bs.lo.y > bo.hi.y || bo.lo.z > bs.hi.z ||
        bs.lo.z > bo.hi.z)
        return false;
    return check_ee(a.x, a.rest, e0, e1, f0, f1, other, a.dhat, o);
}

// appends the lanes' keys (one atomic per warp); a record past the capacity is counted only
__device__ __forceinline__ void append(const QueryArgs& a, bool on, unsigned long long key) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(a.counts + kCntRec, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
    if (on && base < a.rec_cap) a.rec[base] = key;
}

// A warp's 32 queries of one kind (group g of the sorted edges or surface points) and their
// candidates so far
struct QueryGroup {
    int q;     // the lane's query (-1: none)
    BoxF box;  // and its box
};
template <bool kEdge>
__device__ __forceinline__ QueryGroup query_group(const QueryArgs& a, int g) {
    const int lane = threadIdx.x & 31;
    QueryGroup r{-1, empty_box()};
    if (kEdge) {
        r.box = load_box(a.leaf, a.tri_nodes * kNodeLeaves + 32 * g + lane, r.q);
    } else if (32 * g + lane < a.nsv) {
        r.q = __ldg(a.val + a.nf + a.ne + 32 * g + lane);
        r.box = outward(grown_box(a.x, a.sv + r.q, 1, 0.0));
    }
    return r;
}

// tests the last `count` (<= 32) queued candidates exactly, one per lane
template <bool kEdge>
__device__ __forceinline__ void drain(const QueryArgs& a, const int2* queue, int& queued, int count,
                                      unsigned (&by_size)[3]) {
    const int lane = threadIdx.x & 31;
    bool found = false;
    PairOut o;
    unsigned long long key = 0;
    if (lane < count) {
        const int2 c = queue[queued - count + lane];
        int s = c.x, t = c.y;
        if (kEdge && t < s) s = c.y, t = c.x;  // each pair as (edge, larger edge) (mlbvh.cu:1550-1560)
        found = kEdge ? test_ee(a, s, t, o) : test_pt(a, s, t, o);
        key = ((kEdge ? 1ull : 0ull) << a.kshift) | ((unsigned long long)(unsigned)s << a.qshift) | (unsigned)t;
    }
    queued -= count;
    __syncwarp();
    if (found)
#pragma unroll
        for (int k = 0; k < 3; k++) by_size[k] += o.group == k;
    append(a, found, key);
}

// the queries of group g against the primitives of leaf group c: those that meet a query's box
// are queued, and tested 32 at a time
template <bool kEdge>
__device__ __forceinline__ void query_leaves(const QueryArgs& a, int g, int c, const QueryGroup& qg, const BoxF& ub,
                                             int2* queue, int& queued, unsigned (&by_size)[3]) {
    const int lane = threadIdx.x & 31;
    int prim;
    const BoxF cb = load_box(a.leaf, (kEdge ? a.tri_nodes * kNodeLeaves : 0) + 32 * c + lane, prim);
    for (unsigned m = __ballot_sync(0xffffffffu, prim >= 0 && meet(cb, ub)); m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const BoxF jb = shfl_box(cb, j);
        const int jp = __shfl_sync(0xffffffffu, prim, j);
        // edges: only those behind the query in the sorted order (each unordered pair once)
        const bool hit = qg.q >= 0 && meet(qg.box, jb) && (!kEdge || c > g || j > lane);
        const unsigned h = __ballot_sync(0xffffffffu, hit);
        if (!h) continue;
        if (hit) queue[queued + __popc(h & ((1u << lane) - 1u))] = make_int2(qg.q, jp);
        queued += __popc(h);
        __syncwarp();
        if (queued >= 32) drain<kEdge>(a, queue, queued, 32, by_size);
    }
}

__device__ __forceinline__ void add_sizes(const QueryArgs& a, const unsigned (&by_size)[3]) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const unsigned t = __reduce_add_sync(0xffffffffu, by_size[k]);
        if ((threadIdx.x & 31) == 0 && t) atomicAdd(a.counts + kCntSize + k, t);
    }
}

// One warp per query group and 32 nodes: the leaf groups whose box meets the queries', as items
// for k_query.  A group that the list has no room for is searched here and now.
template <bool kEdge>
__device__ __forceinline__ void group_items(const QueryArgs& a, int g, int n0, int2* queue) {
    const int lane = threadIdx.x & 31;
    const int node0 = kEdge ? a.tri_nodes : 0, nnode = kEdge ? a.edge_nodes : a.tri_nodes;
    if (kEdge && n0 + 31 < (g >> 5)) return;  // edges: the leaf groups from the queries' own on
    const QueryGroup qg = query_group<kEdge>(a, g);
    const BoxF ub = warp_union(qg.box);
    int2* list = a.item + (kEdge ? 0 : a.item_cap);
    unsigned* count = a.counts + kCntItem + (kEdge ? 0 : 1);
    unsigned by_size[3] = {0, 0, 0};
    int queued = 0, id;
    const bool on2 = n0 + lane < nnode && meet(load_box(a.node, node0 + n0 + lane, id), ub);
    for (unsigned m2 = __ballot_sync(0xffffffffu, on2); m2; m2 &= m2 - 1) {
        const int c = 32 * (n0 + __ffs(m2) - 1) + lane;  // the lane's leaf group
        const bool on = (!kEdge || c >= g) && meet(load_box(a.group, 32 * node0 + c, id), ub);
        const unsigned m1 = __ballot_sync(0xffffffffu, on);
        if (!m1) continue;
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(count, (unsigned)__popc(m1));
        base = __shfl_sync(0xffffffffu, base, 0) + __popc(m1 & ((1u << lane) - 1u));
        const bool room = base < a.item_cap;
        if (on && room) list[base] = make_int2(g, c);
        for (unsigned m = __ballot_sync(0xffffffffu, on && !room); m; m &= m - 1)
            query_leaves<kEdge>(a, g, __shfl_sync(0xffffffffu, c, __ffs(m) - 1), qg, ub, queue, queued, by_size);
    }
    if (queued > 0) drain<kEdge>(a, queue, queued, queued, by_size);
    add_sizes(a, by_size);
}

// Warps: edge groups x chunks of 32 edge nodes, then point groups x chunks of 32 triangle nodes;
// the first chunk's also test the points against the ground plane (_GroundCollisionDetect,
// GIPC.cu:6433-6450: (n.x - offset)^2 <= dHat with the normal +y).
__global__ void __launch_bounds__(32 * kQueryWarps) k_items(QueryArgs a) {
    __shared__ int2 s_queue[kQueryWarps][64];
    if (a.counts[kCntBad]) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long i = (long long)blockIdx.x * kQueryWarps + w;  // warp-uniform, as all that follows
    const long long edge_warps = (long long)a.edge_groups * ((a.edge_nodes + 31) / 32);
    if (i < edge_warps) {
        group_items<true>(a, (int)(i % a.edge_groups), (int)(i / a.edge_groups) * 32, s_queue[w]);
        return;
    }
    const long long j = i - edge_warps;
    const int chunk = a.point_groups > 0 ? (int)(j / a.point_groups) : 1, g = (int)(j - (long long)chunk * a.point_groups);
    if (chunk > 0 && 32 * chunk >= a.tri_nodes) return;
    if (chunk == 0) {
        bool low = false;
        int q = 0;
        if (32 * g + lane < a.nsv) {
            q = a.val[a.nf + a.ne + 32 * g + lane];
            const double dist = a.x[3 * (size_t)a.sv[q] + 1] - a.ground_offset;
            low = !(dist * dist > a.dhat);
        }
        append(a, low, (2ull << a.kshift) | ((unsigned long long)(unsigned)q << a.qshift));
        const unsigned m = __ballot_sync(0xffffffffu, low);
        if (lane == 0 && m) atomicAdd(a.counts + kCntGround, (unsigned)__popc(m));
    }
    if (32 * chunk < a.tri_nodes) group_items<false>(a, g, 32 * chunk, s_queue[w]);
}

template <bool kEdge>
__device__ __forceinline__ void query_items(const QueryArgs& a, int w0, int nw, int2* queue) {
    const int n = (int)min(a.counts[kCntItem + (kEdge ? 0 : 1)], a.item_cap);
    const int2* list = a.item + (kEdge ? 0 : a.item_cap);
    unsigned by_size[3] = {0, 0, 0};
    int queued = 0;
    for (int i = w0; i < n; i += nw) {  // warp-uniform
        const int2 it = list[i];
        const QueryGroup qg = query_group<kEdge>(a, it.x);
        query_leaves<kEdge>(a, it.x, it.y, qg, warp_union(qg.box), queue, queued, by_size);
    }
    if (queued > 0) drain<kEdge>(a, queue, queued, queued, by_size);
    add_sizes(a, by_size);
}

// The items, one per warp and turn; every warp takes its share of both kinds.  (With one warp
// walking all of a query group's leaf groups, the few groups of large primitives beside small
// ones ran for milliseconds after the others had ended: 5.8 ms for the 256^2 cloth over a sphere,
// SMs busy 11 % of it.)
__global__ void __launch_bounds__(32 * kQueryWarps) k_query(QueryArgs a) {
    __shared__ int2 s_queue[kQueryWarps][64];
    if (a.counts[kCntBad]) return;
    const int nw = gridDim.x * kQueryWarps, w0 = blockIdx.x * kQueryWarps + (threadIdx.x >> 5);
    int2* queue = s_queue[threadIdx.x >> 5];
    query_items<true>(a, w0, nw, queue);
    query_items<false>(a, nw - 1 - w0, nw, queue);
}

// The sorted records as pairs with their CCD candidates and Hessian sizes (flags of the rank
// scan; mat_index holds the size codes until k_mat_index), then the ground points.
__global__ void k_emit(QueryArgs a, int total, int ng, const unsigned long long* __restrict__ rec, int4* pairs,
                       int4* ccd, int* mat_index, unsigned long long* flags, unsigned* ground, unsigned* gp_num) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *gp_num = (unsigned)ng;
    if (k >= total + ng) return;
    const unsigned long long key = rec[k];
    const int kind = (int)(key >> a.kshift);
    const int q = (int)((key >> a.qshift) & ((1ull << (a.kshift - a.qshift)) - 1));
    const int p = (int)(key & ((1ull << a.qshift) - 1));
    if (kind == 2) {
        ground[k - total] = a.sv[q];
        return;
    }
    PairOut o;
    o.group = 0;
    if (kind == 0) test_pt(a, q, p, o);
    else test_ee(a, q, p, o);
    pairs[k] = o.pair;
    ccd[k] = o.ccd;
    mat_index[k] = o.group;
    flags[k] = 1ull << (kGroupBits * o.group);
}

// MatIndex = rank among the pairs of the same group; cp_num = total, 0, per-group counts
__global__ void k_mat_index(int n, int* mat_index, const unsigned long long* __restrict__ flags,
                            const unsigned long long* __restrict__ scan, unsigned* cp_num) {
    // mat_index holds the group codes on entry; each thread rewrites only its own entry
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long m = (1ull << kGroupBits) - 1;
    if (k < n) mat_index[k] = (int)((scan[k] >> (kGroupBits * mat_index[k])) & m);
    if (k == 0) {
        const unsigned long long last = n > 0 ? scan[n - 1] + flags[n - 1] : 0ull;
        cp_num[0] = (unsigned)n;
        cp_num[1] = 0;
        for (int g = 0; g < 3; g++) cp_num[2 + g] = (unsigned)((last >> (kGroupBits * g)) & m);
    }
}

// ------------------------------------------------------------------------------------------
// lagged friction set-up
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ d3 normalized(d3 v) {
    const double inv = 1.0 / sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
    return {v.x * inv, v.y * inv, v.z * inv};
}

// 2 x 2 inverse by Gauss-Jordan elimination with the reference's pivot rule (an entry below
// 1e-15 in magnitude is replaced by adding a later row; __Inverse2x2, gpu_eigen_libs.cu:1342-1411);
// a singular matrix gives zeros
__device__ inline void inverse2x2(const double A[2][2], double R[2][2]) {
    double m[2][4] = {{A[0][0], A[0][1], 1.0, 0.0}, {A[1][0], A[1][1], 0.0, 1.0}};
    R[0][0] = R[0][1] = R[1][0] = R[1][1] = 0.0;
    for (int i = 0; i < 2; i++) {
        if (fabs(m[i][i]) < 1e-15) {
            int j = i + 1;
            for (; j < 2; j++)
                if (fabs(m[j][i]) > 1e-15) break;
            if (j == 2) return;
            for (int r = i; r < 4; r++) m[i][r] += m[j][r];
        }
        const double ep = m[i][i];
        for (int r = i; r < 4; r++) m[i][r] /= ep;
        for (int j = i + 1; j < 2; j++) {
            const double e = -1 * (m[j][i] / m[i][i]);
            for (int r = i; r < 4; r++) m[j][r] += e * m[i][r];
        }
    }
    for (int i = 1; i >= 0; i--)
        for (int j = i - 1; j >= 0; j--) {
            const double e = -1 * (m[j][i] / m[i][i]);
            for (int r = i; r < 4; r++) m[j][r] += e * m[i][r];
        }
    for (int i = 0; i < 2; i++) R[i][0] = m[i][2], R[i][1] = m[i][3];
}

// (first tangent, second tangent) stored as the columns of a row-major 3 x 2 basis
__device__ __forceinline__ void store_basis(double* B, d3 c0, d3 c1) {
    B[0] = c0.x, B[1] = c1.x, B[2] = c0.y, B[3] = c1.y, B[4] = c0.z, B[5] = c1.z;
}

__device__ __forceinline__ bool in_mesh(int v, int nv) { return v >= 0 && v < nv; }

// flags: 1 when pair k takes part in friction (not mollified); a pair naming a vertex
// outside the mesh is left out and raises bad[0]
__global__ void k_fric_flags(const int4* __restrict__ pairs, int n, int nv, int* flag, unsigned* bad) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int4 p = pairs[k];
    int f;
    bool ok;
    if (p.x >= 0) {
        f = p.w >= 0;
        ok = !f || (in_mesh(p.x, nv) && in_mesh(p.y, nv) && in_mesh(p.z, nv) && in_mesh(p.w, nv));
    } else if (p.z < 0) {
        f = p.y >= 0;
        ok = !f || (in_mesh(-p.x - 1, nv) && in_mesh(p.y, nv));
    } else if (p.w < 0) {
        f = p.y >= 0;
        ok = !f || (in_mesh(-p.x - 1, nv) && in_mesh(p.y, nv) && in_mesh(p.z, nv));
    } else {
        f = 1;
        ok = in_mesh(-p.x - 1, nv) && in_mesh(p.y, nv) && in_mesh(p.z, nv) && in_mesh(p.w, nv);
    }
    if (!ok) {
        f = 0;
        atomicOr(bad, 1u);
    }
    flag[k] = f;
}

// _calFrictionLastH_DistAndTan (GIPC.cu:8388-8499) with the closest points and tangent bases
// of FrictionUtils.cuh:52-399; the lagged normal force is that of the RANK-2 barrier
__global__ void k_fric_setup(const double* __restrict__ x, const int4* __restrict__ pairs, int n,
                             const int* __restrict__ flag, const int* __restrict__ off, double dhat, double kappa,
                             int4* out_pairs, double* lambda, double* coord, double* basis, unsigned* cp_num_last) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = k < n && flag[k];
    const int4 p = on ? pairs[k] : make_int4(-1, 0, -1, -1);
    // integer counts (the same totals in any order), one atomic per size and CTA: with one per
    // pair the counters' address bounded the kernel (395 us for a million pairs)
    __shared__ unsigned s_size[3];
    if (threadIdx.x < 3) s_size[threadIdx.x] = 0;
    __syncthreads();
    const int size = p.x >= 0 ? 2 : (p.z < 0 ? 0 : (p.w < 0 ? 1 : 2));
    for (int q = 0; q < 3; q++) {
        const unsigned m = __ballot_sync(0xffffffffu, on && size == q);
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(s_size + q, (unsigned)__popc(m));
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_size[threadIdx.x]) {
        atomicAdd(cp_num_last, s_size[threadIdx.x]);
        atomicAdd(cp_num_last + 2 + threadIdx.x, s_size[threadIdx.x]);
    }
    if (!on) return;
    const int o = off[k];
    double dis, c0 = 0.0, c1 = 0.0;
    double* B = basis + 6 * (size_t)o;
    if (p.x >= 0) {  // edge-edge
        const d3 v0 = ldp(x, p.x), v1 = ldp(x, p.y), v2 = ldp(x, p.z), v3 = ldp(x, p.w);
        dis = ll_d2(v0, v1, v2, v3);
        const d3 e20 = v0 - v2, e01 = v1 - v0, e23 = v3 - v2;
        const double A[2][2] = {{sq(e01), -dot(e23, e01)}, {-dot(e23, e01), sq(e23)}};
        double R[2][2];
        inverse2x2(A, R);
        const double r0 = -dot(e20, e01), r1 = dot(e20, e23);
        c0 = R[0][0] * r0 + R[0][1] * r1;
        c1 = R[1][0] * r0 + R[1][1] * r1;
        store_basis(B, normalized(e01), normalized(cross(cross(e01, e23), e01)));
    } else {
        const unsigned v = (unsigned)(-p.x - 1);
        const d3 v0 = ldp(x, v), v1 = ldp(x, p.y);
        if (p.z < 0) {  // point-point
            dis = pp_d2(v0, v1);
            const d3 v01 = v1 - v0;
            const d3 xc = {0.0, -v01.z, v01.y}, yc = {v01.z, 0.0, -v01.x};
            const d3 t0 = sq(xc) > sq(yc) ? xc : yc;
            store_basis(B, normalized(t0), normalized(cross(v01, t0)));
        } else if (p.w < 0) {  // point-edge
            const d3 v2 = ldp(x, p.z);
            dis = pe_d2(v0, v1, v2);
            const d3 e12 = v2 - v1;
            c0 = dot(v0 - v1, e12) / sq(e12);
            store_basis(B, normalized(e12), normalized(cross(e12, v0 - v1)));
        } else {  // point-triangle
            const d3 v2 = ldp(x, p.z), v3 = ldp(x, p.w);
            dis = pplane_d2(v0, v1, v2, v3);
            const d3 v12 = v2 - v1, v13 = v3 - v1, v10 = v0 - v1;
            const double A[2][2] = {{v12.x * v12.x + v12.y * v12.y + v12.z * v12.z, v12.x * v13.x + v12.y * v13.y + v12.z * v13.z},
                                    {v13.x * v12.x + v13.y * v12.y + v13.z * v12.z, v13.x * v13.x + v13.y * v13.y + v13.z * v13.z}};
            double R[2][2];
            inverse2x2(A, R);
            const double b0 = v12.x * v10.x + v12.y * v10.y + v12.z * v10.z;
            const double b1 = v13.x * v10.x + v13.y * v10.y + v13.z * v10.z;
            c0 = R[0][0] * b0 + R[0][1] * b1;
            c1 = R[1][0] * b0 + R[1][1] * b1;
            store_basis(B, normalized(v12), normalized(cross(cross(v12, v13), v12)));
        }
    }
    const double l = log(dis / dhat);
    lambda[o] = -kappa * 2.0 * sqrt(dis) * (l * l * (2 * dis - 2 * dhat) + (2 * l * (dis - dhat) * (dis - dhat)) / dis);
    coord[2 * (size_t)o] = c0;
    coord[2 * (size_t)o + 1] = c1;
    out_pairs[o] = p;
}

// _calFrictionLastH_gd (GIPC.cu:8362-8386): the ground pairs' normal forces (the RANK-1 form
// of the ground barrier, as the reference writes it)
__global__ void k_fric_ground(const double* __restrict__ x, int nv, const unsigned* __restrict__ gp, int n,
                              double offset, double dhat, double kappa, double* lambda, unsigned* out, unsigned* bad) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const unsigned g = gp[k];
    if (g >= (unsigned)nv) {
        atomicOr(bad, 1u);
        lambda[k] = 0.0;
        out[k] = g;
        return;
    }
    const double dist = x[3 * g + 1] - offset;
    const double dist2 = dist * dist;
    const double t = dist2 - dhat;
    const double g_b = t * log(dist2 / dhat) * -2.0 - (t * t) / dist2;
    lambda[k] = -kappa * 2.0 * sqrt(dist2) * g_b;
    out[k] = g;
}

template <class T>
SgipcStatus regrow(SgipcCtx* c, T** p, size_t n) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    SG_CHECK(c, cudaMalloc((void**)p, sizeof(T) * (n > 0 ? n : 1)));
    return SGIPC_OK;
}

// buffers for np primitives, nl leaf places (whole nodes), ni items of each kind, nrec records
// and nfr friction pairs
SgipcStatus broad_reserve(SgipcCtx* c, int np, int nl, int ni, int nrec, int nfr) {
    if (!c->broad) c->broad = new BroadWork();
    BroadWork& w = *c->broad;
    if (!w.bounds) SG_CHECK(c, cudaMalloc((void**)&w.bounds, sizeof(unsigned long long) * 8));
    if (!w.d_counts) SG_CHECK(c, cudaMalloc((void**)&w.d_counts, sizeof(unsigned) * kCntNum));
    if (!w.h_counts) SG_CHECK(c, cudaMallocHost((void**)&w.h_counts, sizeof(unsigned) * kCntNum));
    SgipcStatus st;
    bool cub_again = !w.cub;
    // a capacity is raised only after all of its buffers exist
    if (np > w.cap_prim) {
        w.cap_prim = 0;
        if ((st = regrow(c, &w.key, np)) || (st = regrow(c, &w.key_s, np)) || (st = regrow(c, &w.val, np)) ||
            (st = regrow(c, &w.val_s, np)))
            return st;
        w.cap_prim = np;
        cub_again = true;
    }
    if (nl > w.cap_leaf) {
        w.cap_leaf = 0;
        if ((st = regrow(c, &w.leaf, 2 * (size_t)nl)) || (st = regrow(c, &w.group, 2 * (size_t)nl / 32)) ||
            (st = regrow(c, &w.node, 2 * (size_t)nl / kNodeLeaves)))
            return st;
        w.cap_leaf = nl;
    }
    if (ni > w.cap_item) {
        w.cap_item = 0;
        if ((st = regrow(c, &w.item, 2 * (size_t)ni))) return st;
        w.cap_item = ni;
    }
    if (nrec > w.cap_rec) {
        w.cap_rec = 0;
        if ((st = regrow(c, &w.reckey, nrec)) || (st = regrow(c, &w.reckey_s, nrec)) || (st = regrow(c, &w.gscan, nrec)))
            return st;
        w.cap_rec = nrec;
        cub_again = true;
    }
    if (nfr + 1 > w.cap_q) {
        w.cap_q = 0;
        if ((st = regrow(c, &w.gflag, (size_t)nfr + 1)) || (st = regrow(c, &w.goff, (size_t)nfr + 1))) return st;
        w.cap_q = nfr + 1;
        cub_again = true;
    }
    if (cub_again) {
        size_t b = 0, t = 0;
        SG_CHECK(c, cub::DeviceRadixSort::SortPairs(nullptr, t, w.key, w.key_s, w.val, w.val_s, w.cap_prim));
        b = t > b ? t : b;
        SG_CHECK(c, cub::DeviceRadixSort::SortKeys(nullptr, t, w.reckey, w.reckey_s, w.cap_rec));
        b = t > b ? t : b;
        SG_CHECK(c, cub::DeviceScan::ExclusiveSum(nullptr, t, w.gflag, w.goff, w.cap_q));
        b = t > b ? t : b;
        SG_CHECK(c, cub::DeviceScan::ExclusiveSum(nullptr, t, w.gscan, w.reckey, w.cap_rec));
        b = t > b ? t : b;
        if (b > w.cub_bytes || !w.cub) {
            w.cub_bytes = 0;
            if ((st = regrow(c, (char**)&w.cub, b))) return st;
            w.cub_bytes = b;
        }
    }
    return SGIPC_OK;
}

// bits that hold 0 .. n - 1
int index_bits(int n) {
    int b = 1;
    while (b < 31 && (1LL << b) < (long long)n) b++;
    return b;
}

}  // namespace

namespace sgipc {
void broad_destroy(SgipcCtx* c) {
    if (!c->broad) return;
    BroadWork& w = *c->broad;
    void* ps[] = {w.key, w.key_s, w.val, w.val_s, w.leaf, w.group, w.node, w.item, w.bounds, w.d_counts, w.gflag, w.goff,
                  w.reckey, w.reckey_s, w.gscan, w.cub};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (w.h_counts) cudaFreeHost(w.h_counts);
    delete c->broad;
    c->broad = nullptr;
}
}  // namespace sgipc

extern "C" SgipcStatus sgipc_build_cp(SgipcCtx* c, const double* x, const double* rest, const SgipcSurface* surf,
                                      const int32_t* body_id, const int32_t* boundary_type, double dHat,
                                      double ground_offset, int32_t cap, int32_t* pairs, int32_t* ccd_pairs,
                                      int32_t* mat_index, uint32_t* cp_num, int32_t ground_cap, uint32_t* ground_pairs,
                                      uint32_t* gp_num, uint32_t* h_cp_num, uint32_t* h_gp_num, void* stream) {
    if (!c || !x || !rest || !surf || !body_id || !pairs || !ccd_pairs || !mat_index || !cp_num || !ground_pairs ||
        !gp_num || !h_cp_num || !h_gp_num || cap < 0 || ground_cap < 0 || !(dHat > 0.0))
        return SGIPC_BAD_INPUT;
    const int nsv = surf->surf_vert_num, nf = surf->face_num, ne = surf->edge_num;
    if (nsv < 0 || nf < 0 || ne < 0 || (nsv && !surf->surf_verts) || (nf && !surf->faces) || (ne && !surf->edges))
        return SGIPC_BAD_INPUT;
    if (cap >= (1 << kGroupBits)) {
        snprintf(c->err, sizeof(c->err), "build_cp: capacity %d beyond the %d pairs one call ranks", cap,
                 (1 << kGroupBits) - 1);
        return SGIPC_BAD_INPUT;
    }
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    const int tri_nodes = nblk(nf, kNodeLeaves), edge_nodes = nblk(ne, kNodeLeaves);
    const int np = nf + ne + nsv;
    const int edge_groups = nblk(ne, 32), point_groups = nblk(nsv, 32);
    const int items = kItemsPerGroup * (edge_groups > point_groups ? edge_groups : point_groups) + 1024;
    SgipcStatus st = broad_reserve(c, np, (tri_nodes + edge_nodes) * kNodeLeaves, items, cap + nsv, 0);
    if (st != SGIPC_OK) return st;
    BroadWork& w = *c->broad;
    const double gap = sqrt(dHat);
    // bounds: min entries start at the largest key, max entries at 0
    SG_CHECK(c, cudaMemsetAsync(w.bounds, 0xff, sizeof(unsigned long long) * 3, s));
    SG_CHECK(c, cudaMemsetAsync(w.bounds + 3, 0, sizeof(unsigned long long) * 5, s));  // and the index flag
    SG_CHECK(c, cudaMemsetAsync(w.d_counts, 0, sizeof(unsigned) * kCntNum, s));
    SG_COUNT(c, 2);
    k_bounds<<<148, 32 * kBoundsWarps, 0, s>>>(x, c->nv, surf->surf_verts, nsv, surf->faces, nf, surf->edges, ne,
                                               w.bounds);
    k_keys<<<nblk(np > 0 ? np : 1), SGIPC_BLOCK, 0, s>>>(x, surf->faces, nf, surf->edges, ne, surf->surf_verts, nsv,
                                                         w.bounds, gap, w.key, w.val, w.d_counts);
    QueryArgs qa{x, rest, surf->surf_verts, surf->faces, surf->edges, body_id, boundary_type, nsv, nf, ne, dHat, gap,
                 ground_offset, w.val_s, w.leaf, w.group, w.node, tri_nodes, edge_nodes, edge_groups, point_groups,
                 w.item, (unsigned)items, w.d_counts, w.reckey, (unsigned)(cap + nsv), 0, 0};
    qa.qshift = index_bits(nf > ne ? nf : ne);
    qa.kshift = qa.qshift + index_bits(nsv > ne ? nsv : ne);
    if (np > 0) {
        size_t t = w.cub_bytes;
        SG_CHECK(c, cub::DeviceRadixSort::SortPairs(w.cub, t, w.key, w.key_s, w.val, w.val_s, np, 0, 32, s));
        if (tri_nodes + edge_nodes > 0) {
            SG_COUNT(c, 1);
            k_boxes<<<tri_nodes + edge_nodes, kNodeLeaves, 0, s>>>(x, surf->faces, nf, surf->edges, ne, tri_nodes,
                                                                   w.val_s, gap, w.d_counts, w.leaf, w.group, w.node);
        }
        const int tri_chunks = nblk(tri_nodes, 32);
        const long long warps = (long long)edge_groups * nblk(edge_nodes, 32) +
                                (long long)point_groups * (tri_chunks > 1 ? tri_chunks : 1);
        if (warps > 0) {  // (none with triangles alone: no points, no edges, nothing to search with)
            SG_COUNT(c, 2);
            k_items<<<nblk(warps, kQueryWarps), 32 * kQueryWarps, 0, s>>>(qa);
            k_query<<<148 * kQueryCtas, 32 * kQueryWarps, 0, s>>>(qa);
        }
    }
    SG_CHECK(c, cudaMemcpyAsync(w.h_counts, w.d_counts, sizeof(unsigned) * kCntNum, cudaMemcpyDeviceToHost, s));
    SG_CHECK(c, cudaStreamSynchronize(s));
    const unsigned* h = w.h_counts;
    const int ng = (int)h[kCntGround], total = (int)(h[kCntRec] - h[kCntGround]);
    for (int k = 0; k < 5; k++) h_cp_num[k] = 0;
    h_cp_num[0] = (unsigned)total;
    *h_gp_num = (unsigned)ng;
    if (h[kCntBad] == 2) {
        snprintf(c->err, sizeof(c->err), "build_cp: a surface point, triangle or edge names a vertex outside the mesh");
        return SGIPC_BAD_INPUT;
    }
    if (h[kCntBad]) {
        snprintf(c->err, sizeof(c->err),
                 "build_cp: the surface points' bounds are empty, not finite or more than 2^%d times the largest primitive",
                 kSpanBits);
        return SGIPC_BAD_INPUT;
    }
    if (total > cap || ng > ground_cap) {
        snprintf(c->err, sizeof(c->err), "build_cp: %d pairs for capacity %d, %d ground pairs for capacity %d",
                 total, cap, ng, ground_cap);
        return SGIPC_CAPACITY;
    }
    for (int k = 0; k < 3; k++) h_cp_num[2 + k] = h[kCntSize + k];
    if (total + ng > 0) {
        size_t t = w.cub_bytes;
        SG_CHECK(c, cub::DeviceRadixSort::SortKeys(w.cub, t, w.reckey, w.reckey_s, total + ng, 0, qa.kshift + 2, s));
    }
    SG_COUNT(c, 2);
    k_emit<<<nblk(total + ng > 0 ? total + ng : 1, 128), 128, 0, s>>>(
        qa, total, ng, w.reckey_s, reinterpret_cast<int4*>(pairs), reinterpret_cast<int4*>(ccd_pairs), mat_index,
        w.gscan, ground_pairs, gp_num);
    // ranks per Hessian size (the unsorted records are no longer needed: their buffer takes the scan)
    if (total > 0) {
        size_t t = w.cub_bytes;
        SG_CHECK(c, cub::DeviceScan::ExclusiveSum(w.cub, t, w.gscan, w.reckey, total, s));
    }
    k_mat_index<<<nblk(total > 0 ? total : 1), SGIPC_BLOCK, 0, s>>>(total, mat_index, w.gscan, w.reckey, cp_num);
    SG_LAUNCH_CHECK(c, "build_cp");
    SG_CHECK(c, cudaStreamSynchronize(s));
    return SGIPC_OK;
}

extern "C" SgipcStatus sgipc_friction_setup(SgipcCtx* c, const double* x, const int32_t* pairs, int32_t pair_num,
                                            const uint32_t* ground_pairs, int32_t ground_num, double dHat,
                                            double kappa, double ground_offset, int32_t* fric_pairs,
                                            double* fric_lambda, double* fric_coord, double* fric_basis,
                                            uint32_t* cp_num_last, uint32_t* fric_gd_pairs, double* fric_gd_lambda,
                                            uint32_t* h_cp_num_last, void* stream) {
    if (!c || !x || pair_num < 0 || ground_num < 0 || !(dHat > 0.0) || !cp_num_last)
        return SGIPC_BAD_INPUT;
    if (pair_num > 0 && (!pairs || !fric_pairs || !fric_lambda || !fric_coord || !fric_basis)) return SGIPC_BAD_INPUT;
    if (ground_num > 0 && (!ground_pairs || !fric_gd_pairs || !fric_gd_lambda)) return SGIPC_BAD_INPUT;
    SG_DEVICE(c);
    cudaStream_t s = (cudaStream_t)stream;
    SgipcStatus st = broad_reserve(c, 0, 0, 0, 0, pair_num);  // flags / offsets over the pairs
    if (st != SGIPC_OK) return st;
    BroadWork& w = *c->broad;
    SG_CHECK(c, cudaMemsetAsync(cp_num_last, 0, sizeof(unsigned) * 5, s));
    if (pair_num > 0) {
        const int4* P = reinterpret_cast<const int4*>(pairs);
        SG_COUNT(c, 2);
        k_fric_flags<<<nblk(pair_num), SGIPC_BLOCK, 0, s>>>(P, pair_num, c->nv, w.gflag, cp_num_last + 1);
        size_t t = w.cub_bytes;
        SG_CHECK(c, cub::DeviceScan::ExclusiveSum(w.cub, t, w.gflag, w.goff, pair_num, s));
        k_fric_setup<<<nblk(pair_num), SGIPC_BLOCK, 0, s>>>(x, P, pair_num, w.gflag, w.goff, dHat, kappa,
                                                            reinterpret_cast<int4*>(fric_pairs), fric_lambda,
                                                            fric_coord, fric_basis, cp_num_last);
    }
    if (ground_num > 0) {
        SG_COUNT(c, 1);
        k_fric_ground<<<nblk(ground_num), SGIPC_BLOCK, 0, s>>>(x, c->nv, ground_pairs, ground_num, ground_offset, dHat,
                                                               kappa, fric_gd_lambda, fric_gd_pairs, cp_num_last + 1);
    }
    SG_LAUNCH_CHECK(c, "friction_setup");
    if (h_cp_num_last) {
        SG_CHECK(c, cudaMemcpyAsync(h_cp_num_last, cp_num_last, sizeof(unsigned) * 5, cudaMemcpyDeviceToHost, s));
        SG_CHECK(c, cudaStreamSynchronize(s));
        if (h_cp_num_last[1]) {
            snprintf(c->err, sizeof(c->err), "friction_setup: a pair or ground pair names a vertex outside the mesh");
            return SGIPC_BAD_INPUT;
        }
    }
    return SGIPC_OK;
}
