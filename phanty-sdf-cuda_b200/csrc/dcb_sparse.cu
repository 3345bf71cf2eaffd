// dcb_sparse.cu — the reference's sparse (brick) dual contouring and its multi-vertex variant
// (CudaSparseDualContouringBackend / CudaSparseMvdcDualContouringBackend,
// src/cuda/dc_cuda_sparse.cu:271-1415). Compiled with --fmad=false: every float operation is
// rounded as written, so the results are the reference's arithmetic without contraction.
//
// Semantics (reference line numbers in dc_cuda_sparse.cu):
//   bricks    brick_size^3 cells; active iff its points [b*s, b*s + s] (clipped) hold a value
//             < 0 and a value > 0 (:271-308)
//   cells     a cell of an active brick is active iff it has corners of both strict signs
//             or a corner with |v| <= 0.45*vx (:321-377); vertices in ascending linear order
//   samples   crossing edges (fa*fb <= 0 in float) and thin edges (same sign, both within
//             0.45*vx of zero, end gradients with dot < -0.3: two samples) (:310-319, :676-752)
//   vertices  one QEF per cell; the multi-vertex variant splits the samples in two when the
//             most opposed normal pair has dot < -0.3 and both halves hold two samples
//             (:445-620, :753-826); max-pivot Jacobi (15 rotations), pinv above 0.01,
//             centroid fallback, clamp into the cell (:181-269, :380-443)
//   faces     each active cell's min-corner X, Y, Z edges with a strict crossing or a thin
//             edge whose four cells have vertices; a thin edge adds the reversed quad; winding
//             by the sum of the end gradients (:829-1102); order: active cell, then X, Y, Z.
//
// B200 layout: the grid is read once by a warp-ballot pass into neg / pos / near-zero bit
// words per point row; bricks and cells are decided on those bits; the active cells get the
// dense path's bitmap layout, so its scan and rank expansion give the ascending active list
// and O(1) cell -> vertex lookups (no cell-sized index map as in the reference).
#include "dcb_kernels.cuh"

namespace dcb {

namespace {

__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 add3(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 sub3(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 mul3(float s, float3 b) { return f3(s * b.x, s * b.y, s * b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
    return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ bool finite3(float3 v) {
    return !(isnan(v.x) || isnan(v.y) || isnan(v.z) || isinf(v.x) || isinf(v.y) || isinf(v.z));
}
// bits [lo, hi) of a word, 0 <= lo <= hi <= 32
__device__ __forceinline__ uint32_t range_bits(int lo, int hi) {
    const uint32_t h = hi >= 32 ? 0xffffffffu : ((1u << hi) - 1u);
    return h & ~((1u << lo) - 1u);
}

__device__ __forceinline__ float sval(const GridDesc& g, int i, int j, int k) { return __ldg(g.v + pidx(g, i, j, k)); }

// Central differences with clamped neighbours (:155-179).
__device__ float3 sgrad(const GridDesc& g, int i, int j, int k) {
    const int im = i > 0 ? i - 1 : 0, ip = i < g.nx - 1 ? i + 1 : g.nx - 1;
    const int jm = j > 0 ? j - 1 : 0, jp = j < g.ny - 1 ? j + 1 : g.ny - 1;
    const int km = k > 0 ? k - 1 : 0, kp = k < g.nz - 1 ? k + 1 : g.nz - 1;
    float3 o = f3(0.f, 0.f, 0.f);
    const float dx = (float)(ip - im) * g.vx, dy = (float)(jp - jm) * g.vy, dz = (float)(kp - km) * g.vz;
    if (dx > 1e-12f) o.x = (sval(g, ip, j, k) - sval(g, im, j, k)) / dx;
    if (dy > 1e-12f) o.y = (sval(g, i, jp, k) - sval(g, i, jm, k)) / dy;
    if (dz > 1e-12f) o.z = (sval(g, i, j, kp) - sval(g, i, j, km)) / dz;
    return o;
}

// Whether the edge between points with values fa, fb may be thin (:310-319): same sign, both
// close to zero. It is if the end gradients' dot product is below -0.3.
__device__ __forceinline__ bool thin_candidate(const SparseParams& P, float fa, float fb) {
    return !(fa * fb <= 0.0f) && !(fabsf(fa) > P.close || fabsf(fb) > P.close);
}

// Float positions of a cell's two planes along each axis.
struct CellBox { float3 lo, hi; };
__device__ __forceinline__ CellBox cell_box(const GridDesc& g, int i, int j, int k) {
    CellBox B;
    B.lo = f3(g.ox + (float)i * g.vx, g.oy + (float)j * g.vy, g.oz + (float)k * g.vz);
    B.hi = f3(g.ox + (float)(i + 1) * g.vx, g.oy + (float)(j + 1) * g.vy, g.oz + (float)(k + 1) * g.vz);
    return B;
}
// Trilinear gradient of the cell at p (:91-153).
__device__ float3 tri_gradient(const float s[8], const CellBox& B, float3 p) {
    const float3 c0 = B.lo;
    const float dx = B.hi.x - c0.x, dy = B.hi.y - c0.y, dz = B.hi.z - c0.z;
    float u = 0.5f, v = 0.5f, w = 0.5f;
    if (fabsf(dx) > 1e-12f) u = (p.x - c0.x) / dx;
    if (fabsf(dy) > 1e-12f) v = (p.y - c0.y) / dy;
    if (fabsf(dz) > 1e-12f) w = (p.z - c0.z) / dz;
    u = fmaxf(0.0f, fminf(1.0f, u));
    v = fmaxf(0.0f, fminf(1.0f, v));
    w = fmaxf(0.0f, fminf(1.0f, w));
    const float omu = 1.0f - u, omv = 1.0f - v, omw = 1.0f - w;
    const float S000 = s[0], S100 = s[1], S110 = s[2], S010 = s[3];
    const float S001 = s[4], S101 = s[5], S111 = s[6], S011 = s[7];
    const float du = (S100 - S000) * omv * omw + (S110 - S010) * v * omw + (S101 - S001) * omv * w + (S111 - S011) * v * w;
    const float dv = (S010 - S000) * omu * omw + (S110 - S100) * u * omw + (S011 - S001) * omu * w + (S111 - S101) * u * w;
    const float dw = (S001 - S000) * omu * omv + (S101 - S100) * u * omv + (S011 - S010) * omu * v + (S111 - S110) * u * v;
    float3 gr = f3(0.f, 0.f, 0.f);
    if (fabsf(dx) > 1e-12f) gr.x = du / dx;
    if (fabsf(dy) > 1e-12f) gr.y = dv / dy;
    if (fabsf(dz) > 1e-12f) gr.z = dw / dz;
    return gr;
}

// Max-pivot Jacobi with at most 15 rotations and the pinv of the diagonal above 0.01
// (:181-269): y = V S^+ V^T d. The symmetric matrix as its six entries; the pivot's entries are
// selected, not indexed, so that everything stays in registers.
struct Sym3 { float xx, xy, xz, yy, yz, zz; };

__device__ void pivot_jacobi_solve(Sym3 A, const float d[3], float y[3], bool& singular) {
    float V[3][3] = {{1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}};
#pragma unroll 1
    for (int it = 0; it < 15; ++it) {
        // the largest off-diagonal entry (p, q); o is the third index
        int pivot = 0;                            // 0: (x,y), 1: (x,z), 2: (y,z)
        float mv = fabsf(A.xy);
        if (fabsf(A.xz) > mv) { pivot = 1; mv = fabsf(A.xz); }
        if (fabsf(A.yz) > mv) { pivot = 2; mv = fabsf(A.yz); }
        if (mv < 1e-7f) break;
        const float ap = pivot == 2 ? A.yy : A.xx, aq = pivot == 0 ? A.yy : A.zz;
        const float apq = pivot == 0 ? A.xy : pivot == 1 ? A.xz : A.yz;
        const float aop = pivot == 0 ? A.xz : A.xy, aoq = pivot == 2 ? A.xz : A.yz;
        const float phi = 0.5f * (aq - ap) / apq;
        float t = 1.0f / (fabsf(phi) + sqrtf(phi * phi + 1.0f));
        if (phi < 0.0f) t = -t;
        const float c = 1.0f / sqrtf(t * t + 1.0f), s = t * c;
        const float nop = c * aop - s * aoq, noq = s * aop + c * aoq;
        const float np = ap - t * apq, nq = aq + t * apq;
        if (pivot == 0)      { A.xz = nop; A.yz = noq; A.xx = np; A.yy = nq; A.xy = 0.0f; }
        else if (pivot == 1) { A.xy = nop; A.yz = noq; A.xx = np; A.zz = nq; A.xz = 0.0f; }
        else                 { A.xy = nop; A.xz = noq; A.yy = np; A.zz = nq; A.yz = 0.0f; }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float vip = pivot == 2 ? V[i][1] : V[i][0], viq = pivot == 0 ? V[i][1] : V[i][2];
            const float wp = c * vip - s * viq, wq = s * vip + c * viq;
            if (pivot == 2) V[i][1] = wp; else V[i][0] = wp;
            if (pivot == 0) V[i][1] = wq; else V[i][2] = wq;
        }
    }
    const float S[3] = {A.xx, A.yy, A.zz};
    float Si[3];
    int ok = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        Si[i] = 0.0f;
        if (S[i] > 0.01f) { Si[i] = 1.0f / S[i]; ++ok; }
    }
    singular = ok == 0;
    float t0 = V[0][0] * d[0] + V[1][0] * d[1] + V[2][0] * d[2];
    float t1 = V[0][1] * d[0] + V[1][1] * d[1] + V[2][1] * d[2];
    float t2 = V[0][2] * d[0] + V[1][2] * d[1] + V[2][2] * d[2];
    t0 *= Si[0]; t1 *= Si[1]; t2 *= Si[2];
    y[0] = V[0][0] * t0 + V[0][1] * t1 + V[0][2] * t2;
    y[1] = V[1][0] * t0 + V[1][1] * t1 + V[1][2] * t2;
    y[2] = V[2][0] * t0 + V[2][1] * t1 + V[2][2] * t2;
}

// Corner offsets and edge ends as bit sets and arithmetic, for edges that differ by lane.
__device__ __forceinline__ int cdx(int c) { return (0x66 >> c) & 1; }
__device__ __forceinline__ int cdy(int c) { return (0xcc >> c) & 1; }
__device__ __forceinline__ int cdz(int c) { return (0xf0 >> c) & 1; }
__device__ __forceinline__ int ea(int e) { return e < 8 ? e : e - 8; }
__device__ __forceinline__ int eb(int e) { return e < 4 ? (e + 1) & 3 : e < 8 ? 4 + ((e + 1) & 3) : e - 4; }
__device__ __forceinline__ float3 corner_of(const CellBox& B, int c) {
    return f3(cdx(c) ? B.hi.x : B.lo.x, cdy(c) ? B.hi.y : B.lo.y, cdz(c) ? B.hi.z : B.lo.z);
}
__device__ __forceinline__ float3 edge_point(const CellBox& B, int e, float t) {
    return add3(mul3(1.0f - t, corner_of(B, ea(e))), mul3(t, corner_of(B, eb(e))));
}

// The samples of a warp's 32 cells, a column per cell: normal and lerp parameter, local edge.
constexpr int kSparseWarps = 4;
struct SparseWarp {
    float corner[8][32];
    float4 sample[12][32];
    uint8_t edge[12][32];
    uint16_t item[12 * 32];        // cell | edge << 5
    uint32_t thin[32];             // thin edges of each cell
};

// The vertex of a cell's samples selected by `sel` (bit q = sample q), in sample order (:380-443).
__device__ float3 cluster_vertex(const SparseWarp& W, int lane, int m, uint32_t sel, const CellBox& B, float3 half,
                                 unsigned int* cnt) {
    const int k = __popc(sel & ((1u << m) - 1u));
    if (k == 0) return add3(B.lo, half);
    float3 c = f3(0.f, 0.f, 0.f);
    for (int q = 0; q < m; ++q)
        if (sel >> q & 1u) c = add3(c, edge_point(B, W.edge[q][lane], W.sample[q][lane].w));
    c = mul3(1.0f / (float)k, c);
    Sym3 A = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float d[3] = {0.f, 0.f, 0.f};
    for (int q = 0; q < m; ++q) {
        if (!(sel >> q & 1u)) continue;
        const float4 n = W.sample[q][lane];
        const float dv = dot3(f3(n.x, n.y, n.z), sub3(edge_point(B, W.edge[q][lane], n.w), c));
        A.xx += n.x * n.x; A.xy += n.x * n.y; A.xz += n.x * n.z;
        A.yy += n.y * n.y; A.yz += n.y * n.z; A.zz += n.z * n.z;
        d[0] += n.x * dv; d[1] += n.y * dv; d[2] += n.z * dv;
    }
    float y[3];
    bool singular;
    pivot_jacobi_solve(A, d, y, singular);
    float3 v = add3(c, f3(y[0], y[1], y[2]));
    if (singular || !finite3(v)) { atomicAdd(cnt + kScFallback, 1u); v = c; }
    if (!finite3(v)) { atomicAdd(cnt + kScInvalid, 1u); v = add3(B.lo, half); }
    if (v.x < B.lo.x || v.x > B.hi.x || v.y < B.lo.y || v.y > B.hi.y || v.z < B.lo.z || v.z > B.hi.z) {
        atomicAdd(cnt + kScClamp, 1u);
        v.x = fmaxf(B.lo.x, fminf(B.hi.x, v.x));
        v.y = fmaxf(B.lo.y, fminf(B.hi.y, v.y));
        v.z = fmaxf(B.lo.z, fminf(B.hi.z, v.z));
    }
    return v;
}

// How many samples a cell holds before edge `e` (12 at most: an edge's one goes in below 12, a
// thin edge's two below 11), e = 12: in all.
__device__ __forceinline__ int samples_before(uint32_t cross, uint32_t thin, int e) {
    if (__popc(cross) + 2 * __popc(thin) <= 12) {
        const uint32_t below = (1u << e) - 1u;
        return __popc(cross & below) + 2 * __popc(thin & below);
    }
    int m = 0;
    for (int x = 0; x < e; ++x) {
        if (cross >> x & 1u) { if (m < 12) ++m; }
        else if (thin >> x & 1u) { if (m < 11) m += 2; }
    }
    return m;
}

// Lists the set bits of the lanes' masks as (lane | bit << 5), lane by lane; their number.
__device__ __forceinline__ int deal(uint16_t* item, uint32_t mask, int lane) {
    const int cnt = __popc(mask);
    int off = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, off, o);
        if (lane >= o) off += v;
    }
    const int total = __shfl_sync(0xffffffffu, off, 31);
    off -= cnt;
    __syncwarp();
    for (uint32_t m = mask; m; m &= m - 1) item[off++] = (uint16_t)(lane | (__ffs(m) - 1) << 5);
    __syncwarp();
    return total;
}

__device__ __forceinline__ float3 unit_or(float3 a, float3 fb) {
    const float l = sqrtf(dot3(a, a));
    return l > 1e-6f ? mul3(1.0f / l, a) : fb;
}

__device__ __forceinline__ long long live_cells(const SparseParams& P) {
    return !P.live ? P.nactive : (long long)*P.live > P.nactive ? 0 : (long long)*P.live;
}

// Active-cell bit of cell (i,j,k) and its rank.
__device__ __forceinline__ bool cell_active(const SparseParams& P, int i, int j, int k) {
    const uint32_t w = __ldg(P.bits + ((int64_t)j + (int64_t)P.g.cy * k) * P.g.W + (i >> 5));
    return (w >> (i & 31)) & 1u;
}

// Vertex of the active face cell of rank r for the gradient sum gn, or -1 (:829-851).
__device__ int face_vertex(const SparseParams& P, uint32_t r, float3 gn) {
    if (!P.mvdc) return (int)r;
    const int st = (int)__ldg(P.vstart + r);
    if (__ldg(P.vcount + r) == 1u) return st;
    const float3 n0 = f3(__ldg(P.N + 3 * (size_t)st), __ldg(P.N + 3 * (size_t)st + 1), __ldg(P.N + 3 * (size_t)st + 2));
    const float3 n1 = f3(__ldg(P.N + 3 * (size_t)st + 3), __ldg(P.N + 3 * (size_t)st + 4), __ldg(P.N + 3 * (size_t)st + 5));
    const float d0 = dot3(gn, n0), d1 = dot3(gn, n1);
    const int best = d0 >= d1 ? st : st + 1;
    return fmaxf(d0, d1) < -0.5f ? -1 : best;
}

}  // namespace

// ---- marking ----------------------------------------------------------------------------

// Negative / positive / near-zero bit words of every point row (32 points a word), a warp
// per 32 consecutive words of a row: a coalesced load and three ballots per word, eight loads in
// flight; lane u keeps word u. (Four points a lane with the words put together by shuffles took
// half as many instructions again: 210 us for 512^3.)
__global__ void __launch_bounds__(256) k_sparse_points(const __grid_constant__ SparseParams P) {
    const GridDesc& g = P.g;
    const int lane = threadIdx.x & 31;
    const uint32_t cpr = (P.Wp + 31) / 32, nchunks = (uint32_t)g.ny * g.nz * cpr;      // grids here are below 2^31 points
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nchunks; c += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t row = cpr == 1 ? c : c / cpr;
        const int w0 = (int)(c - row * cpr) * 32;
        const float* src = g.v + (size_t)row * g.nx;
        const int nw = min(32, P.Wp - w0);
        uint32_t mn = 0, mp = 0, mc = 0;
        for (int u0 = 0; u0 < nw; u0 += 8) {
            float v[8];
            const int x0 = (w0 + u0) * 32 + lane;
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = x0 + 32 * u < g.nx ? __ldg(src + x0 + 32 * u) : __int_as_float(0x7fc00000);
#pragma unroll
            for (int u = 0; u < 8; ++u) {                        // beyond the row: NaN, in no word
                const uint32_t bn = __ballot_sync(0xffffffffu, v[u] < 0.f);
                const uint32_t bp = __ballot_sync(0xffffffffu, v[u] > 0.f);
                const uint32_t bc = __ballot_sync(0xffffffffu, fabsf(v[u]) <= P.close);
                if (lane == u0 + u) { mn = bn; mp = bp; mc = bc; }
            }
        }
        if (lane < nw) {
            const size_t o = (size_t)row * P.Wp + w0 + lane;
            P.pn[o] = mn; P.pp[o] = mp; P.pc[o] = mc;
        }
    }
}

// Brick flags from the point words (:271-308): a block per row of bricks (by, bz). Its threads
// OR the point words of the brick row's (s+1)^2 point rows into shared memory, a word each
// (coalesced) and, where the rows are short, several threads a word with every so many rows (512
// points: 16 words, 8 threads each); then a thread per brick tests its x-range of points.
constexpr int kBrickThreads = 128;
constexpr int kMaxPointWords = 2048;           // nx <= 65536

__global__ void __launch_bounds__(kBrickThreads) k_sparse_bricks(const __grid_constant__ SparseParams P) {
    const GridDesc& g = P.g;
    __shared__ uint32_t s_n[kMaxPointWords], s_p[kMaxPointWords];
    __shared__ unsigned int s_active;
    if (threadIdx.x == 0) s_active = 0;
    const long long nrow = (long long)P.nby * P.nbz;
    for (long long br = blockIdx.x; br < nrow; br += gridDim.x) {
        const int by = (int)(br % P.nby), bz = (int)(br / P.nby);
        const int j0 = by * P.bs, k0 = bz * P.bs;
        const int j1 = min(j0 + P.bs + 1, g.ny), k1 = min(k0 + P.bs + 1, g.nz);
        __syncthreads();
        for (int w = threadIdx.x; w < P.Wp; w += blockDim.x) s_n[w] = s_p[w] = 0;
        __syncthreads();
        const int parts = max(1, (int)blockDim.x / P.Wp), sj = j1 - j0, rows = sj * (k1 - k0);
        const int part = (int)threadIdx.x / P.Wp;
        if (part < parts) {
            for (int w = (int)threadIdx.x - part * P.Wp; w < P.Wp; w += blockDim.x) {
                uint32_t n = 0, p = 0;
                for (int q = part; q < rows; q += parts) {
                    const size_t o = ((size_t)(j0 + q % sj) + (size_t)g.ny * (k0 + q / sj)) * P.Wp + w;
                    n |= __ldg(P.pn + o);
                    p |= __ldg(P.pp + o);
                }
                if (n) atomicOr(&s_n[w], n);
                if (p) atomicOr(&s_p[w], p);
            }
        }
        __syncthreads();
        for (int bx = threadIdx.x; bx < P.nbx; bx += blockDim.x) {
            const int i0 = bx * P.bs, i1 = min(i0 + P.bs + 1, g.nx);
            bool neg = false, pos = false;
            for (int w = i0 >> 5; w <= (i1 - 1) >> 5; ++w) {
                const uint32_t m = range_bits(max(i0 - 32 * w, 0), min(i1 - 32 * w, 32));
                neg |= (s_n[w] & m) != 0u;
                pos |= (s_p[w] & m) != 0u;
            }
            const bool act = neg && pos;
            P.brick[bx + (long long)P.nbx * br] = act ? 1 : 0;
            if (act) atomicAdd(&s_active, 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_active) atomicAdd(P.counters + kScActiveBricks, (unsigned long long)s_active);
}

// Active-cell words (:321-377) in the dense path's layout: a lane builds a cell word from the
// point words of the four point rows around it. A warp takes 32 words of a cell row or, where
// rows have at most 8 or 16 words, four or two rows.
__global__ void __launch_bounds__(256) k_sparse_cells(const __grid_constant__ SparseParams P) {
    const GridDesc& g = P.g;
    const int lane = threadIdx.x & 31;
    const uint32_t nseg = (uint32_t)g.cy * g.cz * P.nxt;
    const int lanes = g.W <= 8 ? 8 : g.W <= 16 ? 16 : 32, wl = lane & (lanes - 1);
    const uint32_t per = 32 / lanes;
    for (uint32_t s0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per; s0 < nseg;
         s0 += ((gridDim.x * blockDim.x) >> 5) * per) {                // warp-uniform
        const uint32_t sg = s0 + lane / lanes;
        const uint32_t row = P.nxt == 1 ? sg : sg / P.nxt;
        const int xt = (int)(sg - row * P.nxt);
        const int k = (int)(row / g.cy), j = (int)(row - (uint32_t)k * g.cy);
        const int w = sg < nseg ? xt * 32 + wl : g.W;
        uint32_t act = 0;
        if (w < g.W && 32 * w < g.cx) {
            const size_t r00 = ((size_t)j + (size_t)g.ny * k) * P.Wp;
            const size_t r10 = r00 + P.Wp, r01 = r00 + (size_t)g.ny * P.Wp, r11 = r01 + P.Wp;
            const bool nxw = w + 1 < P.Wp;
            // some corner of the cells in a word of points
            auto corners = [&](const uint32_t* a) {
                const uint32_t lo = __ldg(a + r00 + w) | __ldg(a + r10 + w) | __ldg(a + r01 + w) | __ldg(a + r11 + w);
                const uint32_t hi = nxw ? (__ldg(a + r00 + w + 1) | __ldg(a + r10 + w + 1) | __ldg(a + r01 + w + 1) |
                                           __ldg(a + r11 + w + 1)) : 0u;
                return lo | (lo >> 1) | (hi << 31);
            };
            // most words have no negative or no near-zero point: nothing more to load or to mask
            const uint32_t neg = corners(P.pn), near = corners(P.pc);
            act = near;
            if (neg) act |= neg & corners(P.pp);
            const int c0 = 32 * w, c1 = min(32 * w + 32, g.cx);
            act &= range_bits(0, c1 - c0);
            if (act) {
                const int by = j / P.bs, bz = k / P.bs;
                uint32_t bm = 0;
                for (int bx = c0 / P.bs; bx * P.bs < c1; ++bx)
                    if (__ldg(P.brick + bx + (long long)P.nbx * (by + (long long)P.nby * bz)))
                        bm |= range_bits(max(bx * P.bs, c0) - c0, min(bx * P.bs + P.bs, c1) - c0);
                act &= bm;
            }
        }
        if (w < g.W) P.bits[(size_t)row * g.W + w] = act;
        uint32_t cnt = __popc(act);
        for (int o = lanes >> 1; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (wl == 0 && sg < nseg) P.seg_count[sg] = cnt;
    }
}

// ---- vertices -----------------------------------------------------------------------------

// A warp takes 32 active cells (:445-826). Their thin candidates, then their sampled edges, are
// dealt to the lanes one (cell, edge) each, the samples go to shared memory in edge order; then a
// lane per cell sums its samples and solves. Cells hold 0 to 12 samples and up to 12 candidates
// (two 6-point gradients each): with a thread per cell 9.5 of 32 lanes were active (512^3 CSG,
// 2.4M cells: 831 us, 64.8% issue).
// The single-vertex variant writes V[rank] directly; the multi-vertex one writes both slots of
// the cell into Vtmp / Ntmp and its count, placed after the scan by k_sparse_place.
template <bool MVDC>
__global__ void __launch_bounds__(32 * kSparseWarps) k_sparse_vertices(const __grid_constant__ SparseParams P) {
    __shared__ unsigned int s_cnt[kScCount];
    __shared__ SparseWarp s_warp[kSparseWarps];
    if (threadIdx.x < kScCount) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const long long nact = live_cells(P);
    const GridDesc& g = P.g;
    const float3 half = mul3(0.5f, f3(g.vx, g.vy, g.vz));
    const int lane = threadIdx.x & 31;
    SparseWarp& W = s_warp[threadIdx.x >> 5];
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < nact;
         base += (long long)gridDim.x * blockDim.x) {                 // warp-uniform
        const long long r = base + lane;
        const bool mine = r < nact;
        int i = 0, j = 0, k = 0;
        uint32_t cross = 0, cand = 0;
        __syncwarp();
        if (mine) {
            unpack_cell(P.list[r], i, j, k);
            float s[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                s[c] = sval(g, i + corner_dx(c), j + corner_dy(c), k + corner_dz(c));
                W.corner[c][lane] = s[c];
            }
#pragma unroll
            for (int e = 0; e < 12; ++e) {
                const float fa = s[edge_a(e)], fb = s[edge_b(e)];
                if (fa * fb <= 0.0f) cross |= 1u << e;
                else if (thin_candidate(P, fa, fb)) cand |= 1u << e;
            }
        }
        W.thin[lane] = 0;
        const int ncand = deal(W.item, cand, lane);
        for (int t0 = 0; t0 < ncand; t0 += 32) {
            const int it = W.item[min(t0 + lane, ncand - 1)], src = it & 31, e = it >> 5;
            const int ci = __shfl_sync(0xffffffffu, i, src), cj = __shfl_sync(0xffffffffu, j, src), ck = __shfl_sync(0xffffffffu, k, src);
            if (t0 + lane < ncand) {
                const int a = ea(e), b = eb(e);
                const float3 ga = sgrad(g, ci + cdx(a), cj + cdy(a), ck + cdz(a));
                const float3 gb = sgrad(g, ci + cdx(b), cj + cdy(b), ck + cdz(b));
                if (dot3(ga, gb) < -0.3f) atomicOr(&W.thin[src], 1u << e);
            }
        }
        __syncwarp();
        const uint32_t thin = W.thin[lane];
        const int nitem = deal(W.item, cross | thin, lane);
        for (int t0 = 0; t0 < nitem; t0 += 32) {
            const int it = W.item[min(t0 + lane, nitem - 1)], src = it & 31, e = it >> 5;
            const int ci = __shfl_sync(0xffffffffu, i, src), cj = __shfl_sync(0xffffffffu, j, src), ck = __shfl_sync(0xffffffffu, k, src);
            const uint32_t cr = __shfl_sync(0xffffffffu, cross, src), th = __shfl_sync(0xffffffffu, thin, src);
            if (t0 + lane >= nitem) continue;
            const int a = ea(e), b = eb(e);
            const float fa = W.corner[a][src], fb = W.corner[b][src];
            const bool crossing = cr >> e & 1u;
            const int m = samples_before(cr, th, e);
            float t = crossing ? fa / (fa - fb + 1e-12f) : fabsf(fa) / (fabsf(fa) + fabsf(fb) + 1e-12f);
            t = fmaxf(0.0f, fminf(1.0f, t));
            if (!crossing || P.normal_mode == 1) {
                float3 ga = sgrad(g, ci + cdx(a), cj + cdy(a), ck + cdz(a));
                float3 gb = sgrad(g, ci + cdx(b), cj + cdy(b), ck + cdz(b));
                if (crossing) {
                    float3 n = add3(mul3(1.0f - t, ga), mul3(t, gb));
                    const float ln = sqrtf(dot3(n, n));
                    if (ln > 1e-6f) n = mul3(1.0f / ln, n);
                    if (m < 12) { W.sample[m][src] = make_float4(n.x, n.y, n.z, t); W.edge[m][src] = (uint8_t)e; }
                } else if (m < 11) {
                    const float la = sqrtf(dot3(ga, ga)), lb = sqrtf(dot3(gb, gb));
                    if (la > 1e-6f) ga = mul3(1.0f / la, ga);
                    if (lb > 1e-6f) gb = mul3(1.0f / lb, gb);
                    W.sample[m][src] = make_float4(ga.x, ga.y, ga.z, t);
                    W.sample[m + 1][src] = make_float4(gb.x, gb.y, gb.z, t);
                    W.edge[m][src] = W.edge[m + 1][src] = (uint8_t)e;
                }
            } else {
                float s[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) s[c] = W.corner[c][src];
                const CellBox B = cell_box(g, ci, cj, ck);
                float3 n = tri_gradient(s, B, edge_point(B, e, t));
                const float ln = sqrtf(dot3(n, n));
                if (ln > 1e-6f) n = mul3(1.0f / ln, n);
                if (m < 12) { W.sample[m][src] = make_float4(n.x, n.y, n.z, t); W.edge[m][src] = (uint8_t)e; }
            }
        }
        __syncwarp();
        if (!mine) continue;
        const int m = samples_before(cross, thin, 12);
        const CellBox B = cell_box(g, i, j, k);
        const uint32_t all = (1u << m) - 1u;
        if (!MVDC) {
            const float3 v = cluster_vertex(W, lane, m, all, B, half, s_cnt);
            P.V[3 * r] = v.x; P.V[3 * r + 1] = v.y; P.V[3 * r + 2] = v.z;
            continue;
        }
        auto normal = [&](int q) { const float4 n = W.sample[q][lane]; return f3(n.x, n.y, n.z); };
        // the most opposed normal pair (first minimum in (i, j > i) order)
        int pa = -1, pb = -1;
        float mind = 1.0f;
        for (int q = 0; q < m; ++q) {
            const float3 nq = normal(q);
            for (int u = q + 1; u < m; ++u) {
                const float dt = dot3(nq, normal(u));
                if (dt < mind) { mind = dt; pa = q; pb = u; }
            }
        }
        uint32_t selA = 0;
        int count = 1;
        if (m >= 2 && pa >= 0 && mind < -0.3f) {
            const float3 nA = normal(pa), nB = normal(pb);
            for (int q = 0; q < m; ++q) if (dot3(normal(q), nA) >= dot3(normal(q), nB)) selA |= 1u << q;
            const int ca = __popc(selA);
            if (ca < 2 || m - ca < 2) atomicAdd(&s_cnt[kScSplitReject], 1u);
            else count = 2;
        }
        float* const vt = P.vtmp + 6 * r;
        float* const nt = P.ntmp + 6 * r;
#pragma unroll 1
        for (int h = 0; h < count; ++h) {
            const uint32_t sel = count == 1 ? all : h == 0 ? selA : all & ~selA;
            const float3 v = cluster_vertex(W, lane, m, sel, B, half, s_cnt);
            float3 sum = f3(0.f, 0.f, 0.f);
            for (int q = 0; q < m; ++q) if (sel >> q & 1u) sum = add3(sum, normal(q));
            const float3 n = unit_or(sum, count == 1 ? f3(0.f, 1.f, 0.f) : normal(h == 0 ? pa : pb));
            vt[3 * h] = v.x; vt[3 * h + 1] = v.y; vt[3 * h + 2] = v.z;
            nt[3 * h] = n.x; nt[3 * h + 1] = n.y; nt[3 * h + 2] = n.z;
        }
        P.vcount[r] = (uint32_t)count;
        if (count == 1) {
            atomicAdd(&s_cnt[kScOne], 1u);
        } else {
            atomicAdd(&s_cnt[kScAmbiguous], 1u);
            atomicAdd(&s_cnt[kScMulti], 1u);
            atomicAdd(&s_cnt[kScTwo], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < kScCount && s_cnt[threadIdx.x])
        atomicAdd(P.counters + threadIdx.x, (unsigned long long)s_cnt[threadIdx.x]);
}

// Multi-vertex variant: each cell's vertices (and normals, and the cell of each vertex) at
// their scanned positions.
__global__ void __launch_bounds__(256) k_sparse_place(const __grid_constant__ SparseParams P) {
    const long long nact = live_cells(P);
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < nact;
         r += (long long)gridDim.x * blockDim.x) {
        const uint32_t st = P.vstart[r], c = P.vcount[r];
        const uint64_t cell = P.list[r];
        for (uint32_t q = 0; q < c; ++q) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                P.V[3 * (size_t)(st + q) + d] = P.vtmp[6 * r + 3 * q + d];
                P.N[3 * (size_t)(st + q) + d] = P.ntmp[6 * r + 3 * q + d];
            }
            P.vcell[st + q] = cell;
        }
    }
}

// ---- faces ----------------------------------------------------------------------------------

// A warp takes 32 active cells (:853-1102): their min-corner edges with a crossing or a thin
// candidate are dealt to the lanes, each of which decides one edge and writes its face (and
// a thin edge's reversed one) to the cell's staging slots 2 * axis and 2 * axis + 1;
// k_sparse_compact moves the faces to their scanned positions. A cell without faces adds nothing
// to the skipped-face counter (the reference's emit pass returns for it, :954). With a thread per
// cell 7.7 of 32 lanes were active (512^3 CSG: 302 us).
__global__ void __launch_bounds__(32 * kSparseWarps) k_sparse_faces(const __grid_constant__ SparseParams P) {
    __shared__ unsigned int s_skipped;
    __shared__ uint16_t s_item[kSparseWarps][3 * 32];
    __shared__ uint32_t s_slots[kSparseWarps][32], s_missing[kSparseWarps][32];
    if (threadIdx.x == 0) s_skipped = 0;
    __syncthreads();
    const long long nact = live_cells(P);
    const GridDesc& g = P.g;
    const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < nact;
         base += (long long)gridDim.x * blockDim.x) {                 // warp-uniform
        const long long r = base + lane;
        int i = 0, j = 0, k = 0;
        float s0 = 0.f;
        uint32_t edges = 0, sure = 0;
        if (r < nact) {
            unpack_cell(P.list[r], i, j, k);
            s0 = sval(g, i, j, k);
#pragma unroll
            for (int axis = 0; axis < 3; ++axis) {
                if (axis == 0 && !(j >= 1 && k >= 1)) continue;
                if (axis == 1 && !(i >= 1 && k >= 1 && j < g.ny - 1)) continue;
                if (axis == 2 && !(i >= 1 && j >= 1 && k < g.nz - 1)) continue;
                const float s1 = sval(g, i + (axis == 0), j + (axis == 1), k + (axis == 2));
                if (s0 * s1 < 0.0f) { edges |= 1u << axis; sure |= 1u << axis; }
                else if (thin_candidate(P, s0, s1)) edges |= 1u << axis;
            }
        }
        s_slots[wb][lane] = 0;
        s_missing[wb][lane] = 0;
        const int nitem = deal(s_item[wb], edges, lane);
        for (int t0 = 0; t0 < nitem; t0 += 32) {
            const int it = s_item[wb][min(t0 + lane, nitem - 1)], src = it & 31, axis = it >> 5;
            const int ci = __shfl_sync(0xffffffffu, i, src), cj = __shfl_sync(0xffffffffu, j, src), ck = __shfl_sync(0xffffffffu, k, src);
            const uint32_t crossed = __shfl_sync(0xffffffffu, sure, src) >> axis & 1u;
            if (t0 + lane >= nitem) continue;
            const uint32_t cr = (uint32_t)(base + src);
            const float3 g0 = sgrad(g, ci, cj, ck), g1 = sgrad(g, ci + (axis == 0), cj + (axis == 1), ck + (axis == 2));
            if (!crossed && !(dot3(g0, g1) < -0.3f)) continue;
            const float3 gn = add3(g0, g1);
            // ranks of the cells c0, c1, c3 around the edge (c2 is this cell); where two of them are
            // neighbours along x and active, the lower one's rank is the other's less one
            const int a1 = axis == 2 ? 1 : 2, a0 = axis == 0 ? 1 : 0;
            const bool act1 = cell_active(P, ci, cj - (a1 == 1), ck - (a1 == 2));                             // c1
            const bool act3 = cell_active(P, ci - (a0 == 0), cj - (a0 == 1), ck);                             // c3
            const bool act0 = cell_active(P, ci - (a0 == 0), cj - (a0 == 1) - (a1 == 1), ck - (a1 == 2));     // c0
            int v0 = -1, v1 = -1, v2 = -1, v3 = -1;
            if (act0 && act1 && act3) {
                const uint32_t r1 = cell_rank(P.bits, P.super, g, ci, cj - (a1 == 1), ck - (a1 == 2));
                const uint32_t r3 = axis == 0 ? cell_rank(P.bits, P.super, g, ci, cj - 1, ck) : cr - 1u;
                const uint32_t r0 = axis == 0 ? cell_rank(P.bits, P.super, g, ci, cj - 1, ck - 1) : r1 - 1u;
                v0 = face_vertex(P, r0, gn);
                v1 = face_vertex(P, r1, gn);
                v2 = face_vertex(P, cr, gn);
                v3 = face_vertex(P, r3, gn);
            }
            if (v0 < 0 || v1 < 0 || v2 < 0 || v3 < 0) {
                if (P.mvdc) atomicAdd(&s_missing[wb][src], 1u);
                continue;
            }
            auto vtx = [&](int v) {
                return f3(__ldg(P.V + 3 * (size_t)v), __ldg(P.V + 3 * (size_t)v + 1), __ldg(P.V + 3 * (size_t)v + 2));
            };
            const float3 pa = vtx(v0), pb = vtx(v1), pc = vtx(v2), pd = vtx(v3);
            float3 qn = cross3(sub3(pb, pa), sub3(pd, pa));
            if (dot3(qn, qn) < 1e-12f) qn = cross3(sub3(pc, pa), sub3(pd, pa));
            if (dot3(gn, gn) > 0.0f && dot3(qn, qn) > 0.0f && dot3(qn, gn) < 0.0f) { const int t = v1; v1 = v3; v3 = t; }
            int4* const out = P.stage + 6 * (size_t)cr + 2 * axis;
            out[0] = make_int4(v0, v1, v2, v3);
            if (!crossed) out[1] = make_int4(v0, v3, v2, v1);
            atomicOr(&s_slots[wb][src], (crossed ? 1u : 3u) << (2 * axis));
        }
        __syncwarp();
        if (r < nact) {
            const uint32_t slots = s_slots[wb][lane], missing = s_missing[wb][lane];
            P.fslots[r] = (uint8_t)slots;
            P.fcount[r] = __popc(slots);
            if (slots && missing) atomicAdd(&s_skipped, missing);
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_skipped) atomicAdd(P.counters + kScSkipped, (unsigned long long)s_skipped);
}

// Each cell's staged faces, in slot order, to their scanned positions.
__global__ void __launch_bounds__(256) k_sparse_compact(const __grid_constant__ SparseParams P) {
    const long long nact = live_cells(P);
    if ((long long)P.counters[kScFaces] > P.faces_cap) return;        // the host places them once it has room
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < nact;
         r += (long long)gridDim.x * blockDim.x) {
        uint32_t at = P.fstart[r];
        for (uint32_t m = P.fslots[r]; m; m &= m - 1) P.faces[at++] = P.stage[6 * r + __ffs(m) - 1];
    }
}

// ---- launchers --------------------------------------------------------------------------------

namespace {
unsigned blocks_for(long long items, int threads, int num_sms, int per_sm) {
    long long b = (items + threads - 1) / threads;
    const long long cap = (long long)num_sms * per_sm;
    if (b > cap) b = cap;
    return (unsigned)(b < 1 ? 1 : b);
}
}  // namespace

cudaError_t launch_sparse_mark(const SparseParams& P, int num_sms, cudaStream_t s) {
    const long long chunks = (long long)P.g.ny * P.g.nz * ((P.Wp + 31) / 32);
    k_sparse_points<<<blocks_for(chunks * 32, 256, num_sms, 16), 256, 0, s>>>(P);
    const long long nrow = (long long)P.nby * P.nbz;
    k_sparse_bricks<<<(unsigned)std::min<long long>(nrow, (long long)num_sms * 16), kBrickThreads, 0, s>>>(P);
    const long long nseg = (long long)P.g.cy * P.g.cz * P.nxt;
    const int lanes = P.g.W <= 8 ? 8 : P.g.W <= 16 ? 16 : 32;
    k_sparse_cells<<<blocks_for(nseg * lanes, 256, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sparse_vertices(const SparseParams& P, int num_sms, cudaStream_t s) {
    if (P.nactive <= 0) return cudaSuccess;
    const unsigned blocks = blocks_for(P.nactive, 32 * kSparseWarps, num_sms, 16);
    if (P.mvdc) k_sparse_vertices<true><<<blocks, 32 * kSparseWarps, 0, s>>>(P);
    else        k_sparse_vertices<false><<<blocks, 32 * kSparseWarps, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sparse_place(const SparseParams& P, int num_sms, cudaStream_t s) {
    if (P.nactive <= 0) return cudaSuccess;
    k_sparse_place<<<blocks_for(P.nactive, 256, num_sms, 8), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sparse_faces(const SparseParams& P, int num_sms, cudaStream_t s) {
    if (P.nactive <= 0) return cudaSuccess;
    k_sparse_faces<<<blocks_for(P.nactive, 32 * kSparseWarps, num_sms, 16), 32 * kSparseWarps, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sparse_compact(const SparseParams& P, int num_sms, cudaStream_t s) {
    if (P.nactive <= 0) return cudaSuccess;
    k_sparse_compact<<<blocks_for(P.nactive, 256, num_sms, 8), 256, 0, s>>>(P);
    return cudaGetLastError();
}

}  // namespace dcb
