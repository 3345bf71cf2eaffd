// dcb_ours.cu — the outer/inner vertex refinement ("Ours", contouring.cpp:1255-1328) on the GPU.
//
// Starting from a dual-contouring extraction (cells, vertices, quads), every outer iteration:
//   1. winds the quads with the current vertices and triangulates them (triangulate_v1 with
//      orient_triangles_for_quad, contouring.cpp:40-113),
//   2. builds a BVH over those triangles (Morton-sorted leaves, radix tree after Karras 2012,
//      boxes bottom-up) and finds for every selected grid point — all points with
//      |S| < 3 * cell diagonal, filled up to batch_size with seeded random others
//      (assign_spheres_to_cells, contouring.cpp:807-933) — its closest point on the mesh; a
//      sphere (centre = grid point, radius |S|) goes to the active cell holding that point
//      unless it floats more than a cell diagonal off the mesh; each cell's spheres are
//      ordered by radius,
//   3. intersects every cell's segments to its six face neighbours' vertices with the shared
//      faces and blends them into the cell's face points (compute_face_cell_intersections,
//      contouring.cpp:1081-1183),
//   4. from the second iteration on, fits a plane (PCA) to the four vertices around every
//      averaged Hermite edge and blends its normal and its crossing with the edge into the
//      four cells' Hermite data (update_hermite_points_and_normals, hermite_update.cpp:441-607),
//   5. runs each cell's inner loop: the local fan of triangles (vertex, Hermite point, face
//      point), every sphere's closest point on it and its barycentric coordinates
//      (vertex_refinement.cpp:110-280), and the regularised QEF with Hermite, sphere and
//      proximal rows (Cell::minimize_qef, Cell.cpp:364-473), until the vertex moves less
//      than 1e-6 (contouring.cpp:1288-1309).
// Everything is FP64 and compiled with --fmad=false, like the CPU restatement it is checked
// against. One thread per cell (steps 3, 4), per quad (1), per grid point (2; a warp for the
// points with long searches), a lane per (cell, sphere), (cell, sum) and cell (5).
#include <cfloat>
#include "dcb_f64.cuh"
#include "dcb_sort.cuh"

namespace dcb {

namespace {

// The four edges around each face, faces 0:+X 1:-X 2:+Y 3:-Y 4:+Z 5:-Z (between consecutive
// corners of vertex_refinement.cpp:12-19).
__constant__ int kFaceEdges[6][4] = {{9, 5, 10, 1}, {3, 11, 7, 8}, {10, 6, 11, 2}, {8, 4, 9, 0}, {7, 6, 5, 4}, {0, 1, 2, 3}};

__device__ __forceinline__ double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ double norm3(const double* a) { return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); }
__device__ __forceinline__ void cross3(const double* a, const double* b, double* o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ bool active_bit(const OursParams& P, int i, int j, int k) {
    const uint32_t w = __ldg(P.bits + ((long long)j + (long long)P.g.cy * k) * P.g.W + (i >> 5));
    return (w >> (i & 31)) & 1u;
}

__device__ __forceinline__ double gpos(const GridDesc& g, int axis, int i) {
    return axis == 0 ? (double)pos_axis(g.ox, g.vx, i) : axis == 1 ? (double)pos_axis(g.oy, g.vy, i)
                                                                   : (double)pos_axis(g.oz, g.vz, i);
}

__device__ __forceinline__ void point_of(const GridDesc& g, long long gidx, double c[3]) {
    const int i = (int)(gidx % g.nx);
    const int j = (int)((gidx / g.nx) % g.ny);
    const int k = (int)(gidx / ((long long)g.nx * g.ny));
    c[0] = gpos(g, 0, i); c[1] = gpos(g, 1, j); c[2] = gpos(g, 2, k);
}

// Closest point of triangle (a,b,c) to p (Ericson, Real-Time Collision Detection §5.1.5);
// degenerate triangles fall back to the closest of their three edges.
__device__ void seg_closest(const double* p, const double* a, const double* b, double* out) {
    double ab[3], ap[3];
    for (int d = 0; d < 3; ++d) { ab[d] = b[d] - a[d]; ap[d] = p[d] - a[d]; }
    const double l2 = dot3(ab, ab);
    double t = l2 > 0.0 ? dot3(ap, ab) / l2 : 0.0;
    t = fmin(1.0, fmax(0.0, t));
    for (int d = 0; d < 3; ++d) out[d] = a[d] + t * ab[d];
}

__device__ __noinline__ void tri_closest_degenerate(const double* p, const double* a, const double* b, const double* c, double* out) {
    double q[3], best = DBL_MAX;
    const double* E[3][2] = {{a, b}, {b, c}, {c, a}};
    for (int s = 0; s < 3; ++s) {
        seg_closest(p, E[s][0], E[s][1], q);
        double dd[3] = {q[0] - p[0], q[1] - p[1], q[2] - p[2]};
        const double d2q = dot3(dd, dd);
        if (d2q < best) { best = d2q; out[0] = q[0]; out[1] = q[1]; out[2] = q[2]; }
    }
}

// The regions (vertex a, b, edge ab, vertex c, edges ac, bc, interior, tested in that order)
// select what one division and one sum are made of, so that lanes in different regions run
// the same instructions; every lane's operations are its region's own.
__device__ __forceinline__ void tri_closest(const double* p, const double* a, const double* b, const double* c, double* out) {
    double ab[3], ac[3], ap[3], bp[3], cp[3];
    for (int d = 0; d < 3; ++d) {
        ab[d] = b[d] - a[d]; ac[d] = c[d] - a[d];
        ap[d] = p[d] - a[d]; bp[d] = p[d] - b[d]; cp[d] = p[d] - c[d];
    }
    const double d1 = dot3(ab, ap), d2 = dot3(ac, ap), d3 = dot3(ab, bp), d4 = dot3(ac, bp), d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    const double vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    const bool at_a = d1 <= 0.0 && d2 <= 0.0;
    const bool at_b = !at_a && d3 >= 0.0 && d4 <= d3;
    bool rest = !at_a && !at_b;
    const bool on_ab = rest && vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0;
    rest = rest && !on_ab;
    const bool at_c = rest && d6 >= 0.0 && d5 <= d6;
    rest = rest && !at_c;
    const bool on_ac = rest && vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0;
    rest = rest && !on_ac;
    const double e = d4 - d3, f = d5 - d6;
    const bool on_bc = rest && va <= 0.0 && e >= 0.0 && f >= 0.0;
    rest = rest && !on_bc;
    const double sum = va + vb + vc;
    double num = 1.0, den = 1.0;
    if (on_ab) { num = d1; den = d1 - d3; }
    if (on_ac) { num = d2; den = d2 - d6; }
    if (on_bc) { num = e; den = e + f; }
    if (rest) den = sum;
    const double ratio = num / den;
    const double first = rest ? vb * ratio : ratio, second = vc * ratio;
    const bool corner = at_a || at_b || at_c;
    for (int d = 0; d < 3; ++d) {
        const double from = at_b || on_bc ? b[d] : at_c ? c[d] : a[d];
        const double along = on_ac ? ac[d] : on_bc ? c[d] - b[d] : ab[d];
        double x = from;
        if (!corner) x = from + first * along;
        if (rest) x = x + ac[d] * second;
        out[d] = x;
    }
    if (rest && !(sum != 0.0 && isfinite(sum) && isfinite(out[0]) && isfinite(out[1]) && isfinite(out[2])))
        tri_closest_degenerate(p, a, b, c, out);
}

// compute_barycentric_coords (vertex_refinement.cpp:36-66).
__device__ void barycentric(const double* P, const double* V0, const double* V1, const double* V2, double out[3]) {
    double e1[3], e2[3], ep[3];
    for (int d = 0; d < 3; ++d) { e1[d] = V1[d] - V0[d]; e2[d] = V2[d] - V0[d]; ep[d] = P[d] - V0[d]; }
    const double d11 = dot3(e1, e1), d12 = dot3(e1, e2), d22 = dot3(e2, e2);
    const double dP1 = dot3(ep, e1), dP2 = dot3(ep, e2);
    const double denom = d11 * d22 - d12 * d12;
    if (fabs(denom) < 1e-12) { out[0] = 1.0; out[1] = 0.0; out[2] = 0.0; return; }
    const double beta = (d22 * dP1 - d12 * dP2) / denom;
    const double gamma = (d11 * dP2 - d12 * dP1) / denom;
    out[0] = 1.0 - beta - gamma; out[1] = beta; out[2] = gamma;
}

// Hermite sample of edge e with the 4-cell average, and whether the edge was averaged.
__device__ bool edge_sample_avg(const GridDesc& g, const f64::Cell64& C, int i, int j, int k, int e, double p[3],
                                double n[3], bool& avg) {
    avg = false;
    if (!f64::hermite(C, e, p, n)) return false;
    int cc[4][3], ex[4];
    const int a = edge_a(e), b = edge_b(e);
    const int Pa[3] = {i + corner_dx(a), j + corner_dy(a), k + corner_dz(a)};
    const int Pb[3] = {i + corner_dx(b), j + corner_dy(b), k + corner_dz(b)};
    int Pm[3], PM[3];
    for (int d = 0; d < 3; ++d) { Pm[d] = min(Pa[d], Pb[d]); PM[d] = max(Pa[d], Pb[d]); }
    const bool in0 = Pm[0] > 0 && Pm[0] < g.nx - 1 && Pm[1] > 0 && Pm[1] < g.ny - 1 && Pm[2] > 0 && Pm[2] < g.nz - 1;
    const bool in1 = PM[0] > 0 && PM[0] < g.nx - 1 && PM[1] > 0 && PM[1] < g.ny - 1 && PM[2] > 0 && PM[2] < g.nz - 1;
    if (!in0 && !in1) return true;
    const int axis = Pa[0] != Pb[0] ? 0 : (Pa[1] != Pb[1] ? 1 : 2);
    const int d1 = axis == 0 ? 1 : 0, d2 = axis == 2 ? 1 : 2;
    double nq[4][3];
    for (int q = 0; q < 4; ++q) {
        cc[q][0] = Pm[0]; cc[q][1] = Pm[1]; cc[q][2] = Pm[2];
        if (q & 1) cc[q][d1] -= 1;
        if (q & 2) cc[q][d2] -= 1;
        if (cc[q][0] == i && cc[q][1] == j && cc[q][2] == k) { for (int d = 0; d < 3; ++d) nq[q][d] = n[d]; continue; }
        f64::Cell64 X;
        f64::load_cell(g, cc[q][0], cc[q][1], cc[q][2], X);
        if (!f64::active(X)) return true;
        ex[q] = f64::local_edge(axis, Pm[d1] - cc[q][d1], Pm[d2] - cc[q][d2]);
        double px[3];
        if (!f64::hermite(X, ex[q], px, nq[q])) return true;
    }
    double acc[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < 4; ++q)
        if (sqrt(f64::sq3(nq[q])) > 0) { acc[0] += nq[q][0]; acc[1] += nq[q][1]; acc[2] += nq[q][2]; }
    f64::normalize3(acc);
    for (int d = 0; d < 3; ++d) n[d] = acc[d];
    avg = true;
    return true;
}

__device__ __forceinline__ unsigned long long expand_bits10(unsigned long long v) {
    v = (v * 0x00010001ull) & 0xFF0000FFull;
    v = (v * 0x00000101ull) & 0x0F00F00Full;
    v = (v * 0x00000011ull) & 0xC30C30C3ull;
    v = (v * 0x00000005ull) & 0x49249249ull;
    return v;
}

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

}  // namespace

// Cells of the inner loop by their number of spheres (below kTeamSpheres[i]): few, some tens (both
// packed into a block's rows, the larger ones first), a block per cell.
constexpr unsigned int kTeamSpheres[2] = {16, 128};

// ---- setup -------------------------------------------------------------------------------

// Per cell: Hermite points and normals as the refinement starts (after Cell::update and the
// second average_hermite_normals, contouring.cpp:1233-1241), vertex = Hermite centroid
// (contouring.cpp:1258-1263), and the extraction's FP64 vertex for the first mesh.
__global__ void __launch_bounds__(128) k_ours_init(OursParams P) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < P.nv; r += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        unpack_cell(P.list[r], i, j, k);
        f64::Cell64 C;
        f64::load_cell(P.g, i, j, k, C);
        OursCell& S = P.cells[r];
        int hmask = 0, m = 0;
        double c[3] = {0.0, 0.0, 0.0};
        for (int e = 0; e < 12; ++e) {
            double p[3], n[3];
            bool avg;
            if (!edge_sample_avg(P.g, C, i, j, k, e, p, n, avg)) continue;
            if (avg) {
                // the second averaging sums the four (identical) averaged normals again
                double acc[3];
                for (int d = 0; d < 3; ++d) acc[d] = ((n[d] + n[d]) + n[d]) + n[d];
                if (sqrt(f64::sq3(n)) > 0) f64::normalize3(acc);
                else acc[0] = acc[1] = acc[2] = 0.0;
                for (int d = 0; d < 3; ++d) n[d] = acc[d];
            }
            for (int d = 0; d < 3; ++d) { S.hp[e][d] = p[d]; S.hn[e][d] = n[d]; c[d] += p[d]; }
            hmask |= 1 << e;
            ++m;
        }
        for (int d = 0; d < 3; ++d) S.v[d] = m ? c[d] / double(m) : 0.0;
        S.hmask = hmask;
        S.fmask = 0;
        double x[3];
        f64::cell_vertex_thread(P.g, i, j, k, 0.01, x);        // Cell::update's threshold (Cell.cpp:314)
        for (int d = 0; d < 3; ++d) P.Vm[3 * r + d] = x[d];
    }
}

// Per extracted quad: the canonical cell order of its grid edge (contouring.cpp:607-729; the
// extraction may have swapped c1 and c3) and the edge's gradient sum gradientAt(p0)+gradientAt(p1).
__global__ void __launch_bounds__(128) k_ours_quads(OursParams P) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < P.nq; q += (long long)gridDim.x * blockDim.x) {
        const int4 f = P.dc_faces[q];
        int a0, a1, a2, c0, c1, c2, b0, b1, b2;
        unpack_cell(P.list[f.x], a0, a1, a2);
        unpack_cell(P.list[f.z], c0, c1, c2);
        unpack_cell(P.list[f.y], b0, b1, b2);
        const int axis = a0 == c0 ? 0 : (a1 == c1 ? 1 : 2);
        // canonical c1 = c2 - e_z for x and y edges, c2 - e_y for z edges
        int w0 = c0, w1 = c1, w2 = c2;
        if (axis == 2) w1 -= 1; else w2 -= 1;
        const bool canon = b0 == w0 && b1 == w1 && b2 == w2;
        P.quads[q] = canon ? f : make_int4(f.x, f.w, f.z, f.y);
        double g0[3], g1[3];
        f64::grid_gradient(P.g, c0, c1, c2, g0);
        f64::grid_gradient(P.g, c0 + (axis == 0), c1 + (axis == 1), c2 + (axis == 2), g1);
        for (int d = 0; d < 3; ++d) P.gsum[3 * q + d] = g0[d] + g1[d];
    }
}

// Grid points with |S| < 3 * cell diagonal (the sphere batch) and the others (the random fill).
__global__ void __launch_bounds__(256) k_ours_select(OursParams P, long long npts, uint32_t* band, uint32_t* rest,
                                                     unsigned int* counts) {
    const int lane = threadIdx.x & 31;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < npts;
         base += (long long)gridDim.x * blockDim.x) {
        const long long t = base + lane;
        bool in = false, ok = t < npts;
        if (ok) in = fabs((double)__ldg(P.g.v + t)) < 3.0 * P.cell_diag;
        for (int w = 0; w < 2; ++w) {
            const uint32_t m = __ballot_sync(0xffffffffu, ok && (w == 0 ? in : !in));
            if (!m) continue;
            unsigned int first = 0;
            if (lane == __ffs(m) - 1) first = atomicAdd(counts + w, (unsigned int)__popc(m));
            first = __shfl_sync(0xffffffffu, first, __ffs(m) - 1);
            if (ok && (w == 0 ? in : !in)) (w == 0 ? band : rest)[first + __popc(m & ((1u << lane) - 1u))] = (uint32_t)t;
        }
    }
}

__device__ __forceinline__ unsigned long long spread21(unsigned long long v) {
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Morton keys of the selected grid points: the queries of a warp then cover a compact block.
__global__ void k_ours_point_keys(OursParams P, const uint32_t* sel, long long n, unsigned long long* keys) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const long long g = sel[t];
        const unsigned long long i = g % P.g.nx, j = (g / P.g.nx) % P.g.ny, k = g / ((long long)P.g.nx * P.g.ny);
        keys[t] = spread21(i) | (spread21(j) << 1) | (spread21(k) << 2);
    }
}

// The random fill of one outer iteration (seeded): the `take` candidates with the smallest random
// keys. The keys of one iteration differ (two bijections of the point), so the set is unique;
// its order does not matter. A histogram of the keys' first 12 bits gives the bin that the last
// one lies in; keys below it are taken, those in it listed, and one block selects among them.
// Instead of a 64-bit sort of all candidates: 0.41 ms of an outer iteration at 128^3 (two
// million candidates), now 0.04. Sorted by Morton code afterwards only beyond kFillUnsorted points:
// below, the sort costs more than the nearness of a warp's queries saves. An outer iteration of
// 128^3 with a fill of 8,000, 16,000, 32,000, 64,000, 128,000 points, sorted: 1.79, 2.08, 2.35, 3.15,
// 4.41 ms; unsorted: 1.73, 1.96, 2.24, 3.07, 4.43. At 80^3 and 192^3 the lines cross between the same
// two sizes.
constexpr long long kFillUnsorted = 98304;
constexpr int kFillBins = 4096, kFillThreads = 256, kFillDigit = 11;

__device__ __forceinline__ unsigned long long fill_key(unsigned long long seed, int it, uint32_t point) {
    return splitmix64(seed ^ splitmix64(((unsigned long long)it << 40) ^ (unsigned long long)point));
}

__global__ void __launch_bounds__(kFillThreads) k_ours_fill_hist(const uint32_t* rest, long long n, unsigned long long seed,
                                                                 int it, unsigned int* hist) {
    __shared__ unsigned int s_hist[kFillBins];
    for (int b = threadIdx.x; b < kFillBins; b += kFillThreads) s_hist[b] = 0;
    __syncthreads();
    for (long long t = (long long)blockIdx.x * kFillThreads + threadIdx.x; t < n; t += (long long)gridDim.x * kFillThreads)
        atomicAdd(s_hist + (fill_key(seed, it, rest[t]) >> 52), 1u);
    __syncthreads();
    for (int b = threadIdx.x; b < kFillBins; b += kFillThreads)
        if (s_hist[b]) atomicAdd(hist + b, s_hist[b]);
}

// The bin of the take-th smallest of the entries counted in hist[0..n) and how many lie in the
// bins before it. By a whole block of THREADS (n a multiple of it); s: THREADS words.
template <int THREADS>
__device__ void bin_of(const unsigned int* hist, int n, unsigned int take, unsigned int* s, int& bin, unsigned int& below) {
    __shared__ int s_bin;
    __shared__ unsigned int s_below;
    const int per = n / THREADS, tid = threadIdx.x;
    unsigned int sum = 0;
    for (int b = tid * per; b < (tid + 1) * per; ++b) sum += hist[b];
    s[tid] = sum;
    __syncthreads();
    for (int o = 1; o < THREADS; o <<= 1) {
        const unsigned int t = tid >= o ? s[tid - o] : 0u;
        __syncthreads();
        s[tid] += t;
        __syncthreads();
    }
    unsigned int at = s[tid] - sum;
    if (at < take && take <= s[tid]) {
        int b = tid * per;
        while (at + hist[b] < take) at += hist[b++];
        s_bin = b;
        s_below = at;
    }
    __syncthreads();
    bin = s_bin;
    below = s_below;
    __syncthreads();
}

// counts: [0] taken, [1] listed.
__global__ void __launch_bounds__(kFillThreads) k_ours_fill_take(const uint32_t* rest, long long n, unsigned long long seed,
                                                                 int it, unsigned int take, const unsigned int* hist,
                                                                 uint32_t* out, unsigned long long* keys, uint32_t* points,
                                                                 unsigned int* counts) {
    __shared__ unsigned int s[kFillThreads];
    int bin;
    unsigned int below;
    bin_of<kFillThreads>(hist, kFillBins, take, s, bin, below);
    for (long long t = (long long)blockIdx.x * kFillThreads + threadIdx.x; t < n; t += (long long)gridDim.x * kFillThreads) {
        const uint32_t point = rest[t];
        const unsigned long long key = fill_key(seed, it, point);
        const int b = (int)(key >> 52);
        if (b < bin) out[atomicAdd(counts, 1u)] = point;
        else if (b == bin) {
            const unsigned int at = atomicAdd(counts + 1, 1u);
            keys[at] = key;
            points[at] = point;
        }
    }
}

// Of the listed points those with the smallest keys until `take` are taken: their last key by
// digits (the first 12 bits are equal), then one pass.
__global__ void __launch_bounds__(1024) k_ours_fill_last(unsigned int take, const unsigned long long* keys,
                                                         const uint32_t* points, uint32_t* out, unsigned int* counts) {
    constexpr int kBins = 1 << kFillDigit;
    __shared__ unsigned int hist[kBins], s[1024];
    const unsigned int n = counts[1];
    const unsigned int need0 = take - counts[0];
    __syncthreads();
    unsigned int need = need0;
    unsigned long long prefix = keys[0] >> 52;
    for (int low = 52; low > 0;) {
        const int bits = low < kFillDigit ? low : kFillDigit;
        for (int b = threadIdx.x; b < kBins; b += 1024) hist[b] = 0;
        __syncthreads();
        for (unsigned int t = threadIdx.x; t < n; t += 1024)
            if (keys[t] >> low == prefix) atomicAdd(hist + ((keys[t] >> (low - bits)) & ((1u << bits) - 1u)), 1u);
        __syncthreads();
        int bin;
        unsigned int below;
        bin_of<1024>(hist, kBins, need, s, bin, below);
        need -= below;
        low -= bits;
        prefix = prefix << bits | (unsigned int)bin;
    }
    for (unsigned int t = threadIdx.x; t < n; t += 1024)
        if (keys[t] <= prefix) out[atomicAdd(counts, 1u)] = points[t];
}

// ---- the mesh's BVH ----------------------------------------------------------------------

// The quad of canonical cells wound by its grid edge's gradient (contouring.cpp:624-641).
__device__ __forceinline__ int4 wound_quad(const OursParams& P, long long q) {
    int4 f = P.quads[q];
    const double* pa = P.Vm + 3 * (long long)f.x;
    const double* pb = P.Vm + 3 * (long long)f.y;
    const double* pc = P.Vm + 3 * (long long)f.z;
    const double* pd = P.Vm + 3 * (long long)f.w;
    double u[3], w[3], n[3];
    for (int d = 0; d < 3; ++d) { u[d] = pb[d] - pa[d]; w[d] = pd[d] - pa[d]; }
    cross3(u, w, n);
    if (dot3(n, n) < 1e-24) { for (int d = 0; d < 3; ++d) u[d] = pc[d] - pa[d]; cross3(u, w, n); }
    const double* gs = P.gsum + 3 * q;
    if (dot3(gs, gs) > 0 && dot3(n, n) > 0 && dot3(n, gs) < 0.0) { const int t = f.y; f.y = f.w; f.w = t; }
    return f;
}

// triangulate_v1 + orient_triangles_for_quad (contouring.cpp:40-113) of a wound quad.
__device__ __forceinline__ void quad_triangles(const OursParams& P, int4 f, int t0[3], int t1[3]) {
    const double* qa = P.Vm + 3 * (long long)f.x;
    const double* qb = P.Vm + 3 * (long long)f.y;
    const double* qc = P.Vm + 3 * (long long)f.z;
    const double* qd = P.Vm + 3 * (long long)f.w;
    double u[3], w[3], qn[3];
    for (int d = 0; d < 3; ++d) { u[d] = qb[d] - qa[d]; w[d] = qd[d] - qa[d]; }
    cross3(u, w, qn);
    if (dot3(qn, qn) < 1e-24) { for (int d = 0; d < 3; ++d) u[d] = qc[d] - qa[d]; cross3(u, w, qn); }
    t0[0] = f.x; t0[1] = f.y; t0[2] = f.z;
    t1[0] = f.x; t1[1] = f.z; t1[2] = f.w;
    if (dot3(qn, qn) < 1e-24) return;                 // degenerate quad: left as it is
    int* tt[2] = {t0, t1};
    for (int h = 0; h < 2; ++h) {
        const double* p1 = P.Vm + 3 * (long long)tt[h][0];
        const double* p2 = P.Vm + 3 * (long long)tt[h][1];
        const double* p3 = P.Vm + 3 * (long long)tt[h][2];
        double x[3], y[3], tn[3];
        for (int d = 0; d < 3; ++d) { x[d] = p2[d] - p1[d]; y[d] = p3[d] - p1[d]; }
        cross3(x, y, tn);
        if (dot3(tn, qn) < 0.0) { const int s = tt[h][1]; tt[h][1] = tt[h][2]; tt[h][2] = s; }
    }
}

// The current mesh's triangles (the quads wound with the current vertices, then
// triangulate_v1) with their Morton keys (key << 32 | triangle).
__global__ void __launch_bounds__(128) k_ours_tris(OursParams P) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < P.nq; q += (long long)gridDim.x * blockDim.x) {
        int id[2][3];
        quad_triangles(P, wound_quad(P, q), id[0], id[1]);
        for (int h = 0; h < 2; ++h) {
            const long long t = 2 * q + h;
            double cen[3] = {0.0, 0.0, 0.0};
            for (int v = 0; v < 3; ++v)
                for (int d = 0; d < 3; ++d) {
                    const double x = P.Vm[3 * (long long)id[h][v] + d];
                    P.tri9[9 * t + 3 * v + d] = x;
                    cen[d] += x;
                }
            unsigned long long code = 0;
            for (int d = 0; d < 3; ++d) {
                double u = (cen[d] / 3.0 - P.lo[d]) / (P.hi[d] - P.lo[d]);
                u = fmin(1.0, fmax(0.0, u));
                const unsigned long long b = (unsigned long long)fmin(1023.0, u * 1024.0);
                code |= expand_bits10(b) << (2 - d);
            }
            P.tcode[t] = (uint32_t)code;
            P.tidx[t] = (uint32_t)t;
        }
    }
}

// Unique sorted keys (Morton code << 32 | triangle): the pairs were sorted stably by code, so
// equal codes keep ascending triangle order.
__global__ void k_bvh_keys(OursParams P) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < P.nt; i += (long long)gridDim.x * blockDim.x)
        P.mkeys_sorted[i] = ((unsigned long long)P.tcode_sorted[i] << 32) | P.tidx_sorted[i];
}

// Radix tree over the sorted keys (Karras, "Maximizing parallelism in the construction of
// BVHs, octrees, and k-d trees", HPG 2012).
__device__ __forceinline__ int key_delta(const unsigned long long* k, long long n, long long a, long long b) {
    if (b < 0 || b >= n) return -1;
    return __clzll(k[a] ^ k[b]);
}

__global__ void __launch_bounds__(128) k_bvh_tree(OursParams P) {
    const long long n = P.nt;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long* K = P.mkeys_sorted;
        const int d = (key_delta(K, n, i, i + 1) - key_delta(K, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = key_delta(K, n, i, i - d);
        long long lmax = 2;
        while (key_delta(K, n, i, i + lmax * d) > dmin) lmax *= 2;
        long long l = 0;
        for (long long t = lmax / 2; t >= 1; t /= 2)
            if (key_delta(K, n, i, i + (l + t) * d) > dmin) l += t;
        const long long j = i + l * d;
        const int dnode = key_delta(K, n, i, j);
        long long s = 0;
        for (long long div = 2;; div *= 2) {
            const long long t = (l + div - 1) / div;
            if (key_delta(K, n, i, i + (s + t) * d) > dnode) s += t;
            if (t <= 1) break;
        }
        const long long gamma = i + s * d + (d < 0 ? -1 : 0);
        const long long lo = i < j ? i : j, hi = i < j ? j : i;
        const bool leaf_l = lo == gamma, leaf_r = hi == gamma + 1;
        P.nodes[i].child[0] = leaf_l ? ~(int)(K[gamma] & 0xffffffffull) : (int)gamma;
        P.nodes[i].child[1] = leaf_r ? ~(int)(K[gamma + 1] & 0xffffffffull) : (int)(gamma + 1);
        P.parent[leaf_l ? n - 1 + gamma : gamma] = (int)i << 1;
        P.parent[leaf_r ? n + gamma : gamma + 1] = (int)i << 1 | 1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) P.parent[0] = -1;
}

// Boxes bottom-up: leaf boxes rounded outward to float, every box stored at its parent; the
// second child to arrive at a node carries the union on.
__global__ void __launch_bounds__(128) k_bvh_boxes(OursParams P) {
    const long long n = P.nt;
    for (long long L = (long long)blockIdx.x * blockDim.x + threadIdx.x; L < n; L += (long long)gridDim.x * blockDim.x) {
        const long long t = (long long)(P.mkeys_sorted[L] & 0xffffffffull);
        float box[6];
        for (int d = 0; d < 3; ++d) {
            double a = P.tri9[9 * t + d], b = P.tri9[9 * t + 3 + d], c = P.tri9[9 * t + 6 + d];
            box[d] = __double2float_rd(fmin(a, fmin(b, c)));
            box[3 + d] = __double2float_ru(fmax(a, fmax(b, c)));
        }
        int up = P.parent[n - 1 + L];
        while (up >= 0) {
            const int node = up >> 1;
            float2* const dst = reinterpret_cast<float2*>(P.nodes[node].box[up & 1]);
            for (int d = 0; d < 3; ++d) dst[d] = make_float2(box[2 * d], box[2 * d + 1]);
            __threadfence();
            if (atomicAdd(P.flags + node, 1u) == 0) break;       // the other child is not done yet
            __threadfence();
            const float2* const other = reinterpret_cast<const float2*>(P.nodes[node].box[1 - (up & 1)]);
            float2 o[3];
            for (int d = 0; d < 3; ++d) o[d] = __ldcg(other + d);
            const float ob[6] = {o[0].x, o[0].y, o[1].x, o[1].y, o[2].x, o[2].y};
            for (int d = 0; d < 3; ++d) { box[d] = fminf(box[d], ob[d]); box[3 + d] = fmaxf(box[3 + d], ob[3 + d]); }
            up = P.parent[node];
        }
    }
}

// A query point in double and, rounded both ways, in float.
struct QueryPoint {
    double p[3];
    float lo[3], hi[3];
};

// Lower bound of the squared distance to a box, every operation rounded down: searches skip
// only what is provably farther than the best so far, so the answer is that of exact bounds.
__device__ __forceinline__ float box_below(const QueryPoint& q, const float* box) {
    float e[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) e[d] = fmaxf(fmaxf(__fsub_rd(box[d], q.hi[d]), __fsub_rd(q.lo[d], box[3 + d])), 0.f);
    return __fmaf_rd(e[0], e[0], __fmaf_rd(e[1], e[1], __fmul_rd(e[2], e[2])));
}

// Closest point of the mesh to a query (point_mesh_squared_distance, contouring.cpp:869): among
// equally close triangles the one of smallest index, so the answer does not depend on the
// traversal order (nodes as close as the best so far are still visited).
struct Closest {
    double d2 = DBL_MAX;
    int t = 0x7fffffff;
    float above = FLT_MAX;              // d2 rounded up
    double c[3] = {0.0, 0.0, 0.0};
};

// One copy of the distance for all callers (instruction cache).
__device__ __noinline__ double tri_distance(const double* p, const double* T, double* c) {
    tri_closest(p, T, T + 3, T + 6, c);
    double dd[3] = {c[0] - p[0], c[1] - p[1], c[2] - p[2]};
    return dot3(dd, dd);
}

__device__ __forceinline__ void closest_test(const OursParams& P, const QueryPoint& q, int t, Closest& best) {
    double c[3];
    const double d2 = tri_distance(q.p, P.tri9 + 9 * (size_t)t, c);
    if (d2 < best.d2 || (d2 == best.d2 && t < best.t)) {
        best.d2 = d2;
        best.t = t;
        best.above = __double2float_ru(d2);
        best.c[0] = c[0]; best.c[1] = c[1]; best.c[2] = c[2];
    }
}

__device__ __forceinline__ void load_node(const OursParams& P, int node, float (&box)[2][6], int (&child)[2]) {
    const float4* const src = reinterpret_cast<const float4*>(P.nodes + node);
    const float4 a = __ldg(src), b = __ldg(src + 1), c = __ldg(src + 2), d = __ldg(src + 3);
    box[0][0] = a.x; box[0][1] = a.y; box[0][2] = a.z; box[0][3] = a.w; box[0][4] = b.x; box[0][5] = b.y;
    box[1][0] = b.z; box[1][1] = b.w; box[1][2] = c.x; box[1][3] = c.y; box[1][4] = c.z; box[1][5] = c.w;
    child[0] = __float_as_int(d.x);
    child[1] = __float_as_int(d.y);
}

// ---- sphere assignment ---------------------------------------------------------------------

// The query of selected point s, without its answer.
__device__ __forceinline__ QueryPoint query_point(const OursParams& P, long long s) {
    QueryPoint q;
    point_of(P.g, P.sel[s], q.p);
    for (int d = 0; d < 3; ++d) { q.lo[d] = __double2float_rd(q.p[d]); q.hi[d] = __double2float_ru(q.p[d]); }
    return q;
}

// The sphere about selected point s to the active cell that holds its closest mesh point.
__device__ __forceinline__ void assign_sphere(const OursParams& P, long long s, const Closest& best) {
    const long long gidx = P.sel[s];
    P.prev_tri[gidx] = best.t;
    const double radius = fabs((double)__ldg(P.g.v + gidx));
    int rank = -1;
    if (best.d2 < DBL_MAX && sqrt(best.d2) - radius < P.cell_diag) {
        int ci[3];
        const int cmax[3] = {P.g.nx - 2, P.g.ny - 2, P.g.nz - 2};
        for (int d = 0; d < 3; ++d) {
            const double f = floor((best.c[d] - P.gmin[d]) / P.gd[d]);
            int v = f < -1e9 ? -1000000000 : (f > 1e9 ? 1000000000 : (int)f);
            ci[d] = max(0, min(v, cmax[d]));
        }
        if (active_bit(P, ci[0], ci[1], ci[2])) {
            rank = (int)cell_rank(P.bits, P.super, P.g, ci[0], ci[1], ci[2]);
            atomicAdd(P.cell_count + rank, 1u);
        }
    }
    P.sel_cell[s] = rank;
}

// A thread per query, depth first, the near child first; the search starts with the point's
// answer of the previous outer iteration. A search of more than kQueryBudget nodes is left to
// k_ours_query_long (with the best triangle so far): the mean is 80 nodes, but a point far
// from the mesh visits thousands, and one such thread kept the launch (128^3 perturbed sphere,
// 200,000 points: 6.9 ms at 4.5% issue, 1.1 with both kernels; with a budget of 96 nodes 1.2,
// of 320 1.4, of 640 1.9).
constexpr int kQueryBudget = 160;
__global__ void __launch_bounds__(128) k_ours_query(OursParams P) {
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < P.nsel; s += (long long)gridDim.x * blockDim.x) {
        const QueryPoint q = query_point(P, s);
        const int seed = P.prev_tri[P.sel[s]];
        Closest best;
        if (seed >= 0 && seed < P.nt) closest_test(P, q, seed, best);
        int stack[96], sp = 0;                   // a tree over unique 62-bit keys is at most 62 deep
        float bound[96];
        if (P.nt == 1) closest_test(P, q, 0, best);
        else { stack[sp] = 0; bound[sp++] = 0.f; }
        for (int visits = 0; sp > 0 && visits < kQueryBudget;) {
            --sp;
            if (bound[sp] > best.above) continue;
            ++visits;
            float box[2][6];
            int child[2];
            load_node(P, stack[sp], box, child);
            const float d0 = box_below(q, box[0]), d1 = box_below(q, box[1]);
            const bool swap = d1 < d0;
            const int near = swap ? child[1] : child[0], far = swap ? child[0] : child[1];
            const float dn = swap ? d1 : d0, df = swap ? d0 : d1;
            // leaves now, internal nodes onto the stack (the nearer one on top)
            for (int w = 0; w < 2; ++w) {
                const int c = w == 0 ? near : far;
                if (c < 0 && (w == 0 ? dn : df) <= best.above) closest_test(P, q, ~c, best);
            }
            if (far >= 0 && df <= best.above) { stack[sp] = far; bound[sp++] = df; }
            if (near >= 0 && dn <= best.above) { stack[sp] = near; bound[sp++] = dn; }
            if (sp > 94) { set_error(P.err, kErrOverflow); sp = 0; }
        }
        if (sp > 0) {
            P.prev_tri[P.sel[s]] = best.t < P.nt ? best.t : -1;
            P.long_query[atomicAdd(P.long_count, 1u)] = (uint32_t)s;
        } else {
            assign_sphere(P, s, best);
        }
    }
}

// The long searches, a warp each: the lanes take the top nodes of one stack. 32 at a time push
// at most 64; near the stack's end one node at a time (depth first) adds at most the tree's
// depth.
constexpr int kLongStack = 768, kLongWarps = 4;
__global__ void __launch_bounds__(32 * kLongWarps) k_ours_query_long(OursParams P) {
    __shared__ int s_node[kLongWarps][kLongStack];
    __shared__ float s_bound[kLongWarps][kLongStack];
    const int lane = threadIdx.x & 31;
    int* const node = s_node[threadIdx.x >> 5];
    float* const bound = s_bound[threadIdx.x >> 5];
    const unsigned int n = *P.long_count;
    for (unsigned int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += (gridDim.x * blockDim.x) >> 5) {
        const long long s = P.long_query[w];
        const QueryPoint q = query_point(P, s);
        const int seed = P.prev_tri[P.sel[s]];
        Closest best;
        if (seed >= 0) closest_test(P, q, seed, best);
        __syncwarp();
        if (lane == 0) { node[0] = 0; bound[0] = 0.f; }
        int sp = 1;
        while (sp > 0) {
            __syncwarp();
            const int take = kLongStack - sp >= 192 ? min(sp, 32) : 1;
            const int at = sp - 1 - lane;
            const bool mine = lane < take && bound[at] <= best.above;
            int child[2] = {-1, -1};
            float d[2] = {0.f, 0.f};
            bool push[2] = {false, false};
            const double had = best.d2;
            const int had_t = best.t;
            if (mine) {
                float box[2][6];
                load_node(P, node[at], box, child);
                d[0] = box_below(q, box[0]);
                d[1] = box_below(q, box[1]);
                for (int c = 0; c < 2; ++c) {
                    if (child[c] >= 0) push[c] = true;
                    else if (d[c] <= best.above) closest_test(P, q, ~child[c], best);
                }
            }
            __syncwarp();
            // the lanes' best (ties: smallest index)
            if (__any_sync(0xffffffffu, best.d2 < had || best.t != had_t)) {
                for (int o = 16; o > 0; o >>= 1) {
                    const double od = __shfl_xor_sync(0xffffffffu, best.d2, o);
                    const int ot = __shfl_xor_sync(0xffffffffu, best.t, o);
                    if (od < best.d2 || (od == best.d2 && ot < best.t)) { best.d2 = od; best.t = ot; }
                }
                best.above = best.d2 < DBL_MAX ? __double2float_ru(best.d2) : FLT_MAX;
            }
            sp -= take;
            for (int c = 0; c < 2; ++c) {
                const bool on = push[c] && d[c] <= best.above;
                const unsigned int votes = __ballot_sync(0xffffffffu, on);
                if (on) {
                    const int to = sp + __popc(votes & ((1u << lane) - 1u));
                    node[to] = child[c];
                    bound[to] = d[c];
                }
                sp += __popc(votes);
            }
        }
        if (lane == 0) {
            if (best.t < P.nt) tri_distance(q.p, P.tri9 + 9 * (size_t)best.t, best.c);
            assign_sphere(P, s, best);
        }
    }
}

__global__ void __launch_bounds__(128) k_ours_scatter(OursParams P) {
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < P.nsel; s += (long long)gridDim.x * blockDim.x) {
        const int rank = P.sel_cell[s];
        if (rank < 0) continue;
        const unsigned int at = P.cell_start[rank] + atomicAdd(P.cell_fill + rank, 1u);
        P.cell_spheres[at] = P.sel[s];
    }
}

// Each cell's spheres by radius (then grid index, for a deterministic order among equal radii),
// and their centres (float grid positions) with the values there.
__global__ void __launch_bounds__(128) k_ours_sort(OursParams P) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < P.nv; r += (long long)gridDim.x * blockDim.x) {
        const unsigned int n = P.cell_count[r];
        if (n) {
            const int team = n < kTeamSpheres[0] ? 0 : n < kTeamSpheres[1] ? 1 : 2;
            P.team_list[team][atomicAdd(P.team_count + team, 1u)] = (uint32_t)r;
        }
        uint32_t* a = P.cell_spheres + P.cell_start[r];
        auto less = [&](uint32_t x, uint32_t y) {
            const float rx = fabsf(__ldg(P.g.v + x)), ry = fabsf(__ldg(P.g.v + y));
            return rx < ry || (rx == ry && x < y);
        };
        // Shell sort (Ciura gaps)
        const unsigned int gaps[8] = {701, 301, 132, 57, 23, 10, 4, 1};
        for (int gi = 0; gi < 8; ++gi) {
            const unsigned int gap = gaps[gi];
            for (unsigned int x = gap; x < n; ++x) {
                const uint32_t t = a[x];
                unsigned int y = x;
                while (y >= gap && less(t, a[y - gap])) { a[y] = a[y - gap]; y -= gap; }
                a[y] = t;
            }
        }
        for (unsigned int x = 0; x < n; ++x) {
            double c[3];
            point_of(P.g, a[x], c);
            P.cell_centres[P.cell_start[r] + x] = make_float4((float)c[0], (float)c[1], (float)c[2], __ldg(P.g.v + a[x]));
        }
    }
}

// ---- per-cell steps --------------------------------------------------------------------------

// compute_face_cell_intersections (contouring.cpp:1081-1183).
__global__ void __launch_bounds__(128) k_ours_faces(OursParams P) {
    const int dirs[6][3] = {{1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < P.nv; r += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        unpack_cell(P.list[r], i, j, k);
        OursCell& S = P.cells[r];
        const double v[3] = {S.v[0], S.v[1], S.v[2]};
        const double mn[3] = {gpos(P.g, 0, i), gpos(P.g, 1, j), gpos(P.g, 2, k)};
        const double mx[3] = {gpos(P.g, 0, i + 1), gpos(P.g, 1, j + 1), gpos(P.g, 2, k + 1)};
        int fmask = S.fmask;
        for (int d = 0; d < 6; ++d) {
            const int ni = i + dirs[d][0], nj = j + dirs[d][1], nk = k + dirs[d][2];
            if (ni < 0 || ni >= P.g.cx || nj < 0 || nj >= P.g.cy || nk < 0 || nk >= P.g.cz) continue;
            if (!active_bit(P, ni, nj, nk)) continue;
            const OursCell& N = P.cells[cell_rank(P.bits, P.super, P.g, ni, nj, nk)];
            double seg[3];
            for (int a = 0; a < 3; ++a) seg[a] = N.v[a] - v[a];
            const int ax = d >> 1;
            const double plane = (d & 1) ? mn[ax] : mx[ax];
            const double num = plane - v[ax], den = seg[ax];
            if (fabs(den) < 1e-9) continue;
            const double t = num / den;
            if (t >= -1e-6 && t <= 1.0 + 1e-6) {
                double x[3];
                for (int a = 0; a < 3; ++a) x[a] = v[a] + t * seg[a];
                if (!(fmask & (1 << d))) {
                    for (int a = 0; a < 3; ++a) S.fi[d][a] = x[a];
                    fmask |= 1 << d;
                } else {
                    for (int a = 0; a < 3; ++a) S.fi[d][a] = x[a] * P.wface + S.fi[d][a] * (1.0 - P.wface);
                }
            }
        }
        S.fmask = fmask;
    }
}

// update_hermite_points_and_normals (hermite_update.cpp:441-607): one thread per (cell, edge);
// the cell at the edge's minimum endpoint handles an edge whose four cells have vertices.
__global__ void __launch_bounds__(128) k_ours_hermite(OursParams P) {
    const long long nrow = 12 * P.nv;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nrow; t += (long long)gridDim.x * blockDim.x) {
        const long long r = t / 12;
        const int e = (int)(t - 12 * r);
        if (e != 0 && e != 3 && e != 8) continue;          // edges leaving corner 0: the owner's
        int i, j, k;
        unpack_cell(P.list[r], i, j, k);
        const OursCell& S0 = P.cells[r];
        if (!(S0.hmask & (1 << e))) continue;
        int cc[4][3], ex[4];
        if (!f64::edge_cells(P.g, i, j, k, e, cc, ex)) continue;
        long long rk[4];
        bool all = true;
        for (int q = 0; q < 4 && all; ++q) {
            if (q == 0) { rk[0] = r; continue; }
            all = active_bit(P, cc[q][0], cc[q][1], cc[q][2]);
            if (all) rk[q] = cell_rank(P.bits, P.super, P.g, cc[q][0], cc[q][1], cc[q][2]);
        }
        if (!all) continue;
        ex[0] = e;
        // PCA of the four vertices: the normal is the direction of least variance
        double V[4][3], cen[3] = {0.0, 0.0, 0.0};
        for (int q = 0; q < 4; ++q)
            for (int d = 0; d < 3; ++d) { V[q][d] = P.cells[rk[q]].v[d]; cen[d] += V[q][d]; }
        for (int d = 0; d < 3; ++d) cen[d] /= 4.0;
        double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, U[3][3];
        for (int q = 0; q < 4; ++q) {
            double x[3];
            for (int d = 0; d < 3; ++d) x[d] = V[q][d] - cen[d];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) M[a][b] += x[a] * x[b];
        }
        f64::jacobi3(M, U);
        int qmin = 0;
        for (int q = 1; q < 3; ++q) if (M[q][q] <= M[qmin][qmin]) qmin = q;
        double nrm[3] = {U[0][qmin], U[1][qmin], U[2][qmin]};
        f64::normalize3(nrm);
        // orientation against the edge of the owner cell (EDGE_PAIRS order)
        const int ca = edge_a(e), cb = edge_b(e);
        const double pA[3] = {gpos(P.g, 0, i + corner_dx(ca)), gpos(P.g, 1, j + corner_dy(ca)), gpos(P.g, 2, k + corner_dz(ca))};
        const double pB[3] = {gpos(P.g, 0, i + corner_dx(cb)), gpos(P.g, 1, j + corner_dy(cb)), gpos(P.g, 2, k + corner_dz(cb))};
        const double sA = (double)__ldg(P.g.v + pidx(P.g, i + corner_dx(ca), j + corner_dy(ca), k + corner_dz(ca)));
        double dir[3];
        for (int d = 0; d < 3; ++d) dir[d] = pB[d] - pA[d];
        const double len = norm3(dir);
        if (len > 0.0) for (int d = 0; d < 3; ++d) dir[d] /= len;
        double out[3];
        for (int d = 0; d < 3; ++d) out[d] = dir[d] * (sA < 0 ? -1.0 : 1.0);
        if (dot3(nrm, out) > 0) for (int d = 0; d < 3; ++d) nrm[d] = -nrm[d];
        const bool has_n = norm3(nrm) > 0;
        for (int q = 0; q < 4; ++q) {
            OursCell& C = P.cells[rk[q]];
            if (!has_n) continue;
            double u[3];
            for (int d = 0; d < 3; ++d) u[d] = (1.0 - P.wnormal) * C.hn[ex[q]][d] + P.wnormal * nrm[d];
            f64::normalize3(u);
            for (int d = 0; d < 3; ++d) C.hn[ex[q]][d] = u[d];
        }
        const double denom = dot3(nrm, dir);
        if (fabs(denom) > 1e-6) {
            double w[3];
            for (int d = 0; d < 3; ++d) w[d] = cen[d] - pA[d];
            double tt = dot3(nrm, w) / denom;
            if (tt < 0 || tt > len) continue;
            tt = fmax(0.0, fmin(tt, len));
            double x[3];
            for (int d = 0; d < 3; ++d) x[d] = pA[d] + tt * dir[d];
            for (int q = 0; q < 4; ++q) {
                OursCell& C = P.cells[rk[q]];
                for (int d = 0; d < 3; ++d) C.hp[ex[q]][d] = (1.0 - P.wpos) * C.hp[ex[q]][d] + P.wpos * x[d];
            }
        }
    }
}

// What the team of one cell works on.
struct TeamCell {
    double hp[12][3], fi[6][3];
    double prev[3];                  // the vertex this iteration starts from
    double h0[9], cen[3], sums[9];
    unsigned char fan[24];           // edge | face << 4
};

// One sphere's row of Cell::minimize_qef (Cell.cpp:400-446) for a cell whose vertex is prev:
// its closest point on the local fan (first minimum in fan order), the point on the sphere,
// the barycentric blend of (vertex, Hermite point, face point). False if the row is skipped.
// row: three entries and the right-hand side. One copy for all callers (instruction cache).
__device__ __noinline__ bool sphere_row(const TeamCell& C, int nfan, const float4* sphere, double ssw, double* row) {
    const double prev[3] = {C.prev[0], C.prev[1], C.prev[2]};
    const float4 centre = __ldg(sphere);
    const double c[3] = {(double)centre.x, (double)centre.y, (double)centre.z};
    const double sval = (double)centre.w;
    const double rs = fabs(sval);
    double best = DBL_MAX, tm[3] = {0, 0, 0};
    int bf = 0;
    for (int f = 0; f < nfan; ++f) {
        const int e = C.fan[f] & 15, d = C.fan[f] >> 4;
        double q[3];
        tri_closest(c, prev, C.hp[e], C.fi[d], q);
        double dd[3] = {q[0] - c[0], q[1] - c[1], q[2] - c[2]};
        const double d2 = dot3(dd, dd);
        if (d2 < best) { best = d2; bf = f; tm[0] = q[0]; tm[1] = q[1]; tm[2] = q[2]; }
    }
    const int e = C.fan[bf] & 15, d = C.fan[bf] >> 4;
    const double* Hp = C.hp[e];
    const double* Fp = C.fi[d];
    double ct[3];
    for (int a = 0; a < 3; ++a) ct[a] = tm[a] - c[a];
    const double rho0 = norm3(ct);
    double qs[3];
    if (rho0 < 1e-9) for (int a = 0; a < 3; ++a) qs[a] = c[a];
    else for (int a = 0; a < 3; ++a) qs[a] = c[a] + (ct[a] / rho0) * rs;
    double bc[3];
    barycentric(tm, prev, Hp, Fp, bc);
    double alpha = bc[0], beta = bc[1], gamma = bc[2];
    if (fabs(alpha) < 1e-6) { alpha = 1.0; beta = 0.0; gamma = 0.0; }
    double tt[3], ctt[3];
    for (int a = 0; a < 3; ++a) { tt[a] = alpha * prev[a] + beta * Hp[a] + gamma * Fp[a]; ctt[a] = tt[a] - c[a]; }
    const double rho = norm3(ctt);
    double qc[3];
    for (int a = 0; a < 3; ++a) qc[a] = qs[a] - c[a];
    const double radius = norm3(qc);
    if (rho > radius && sval < 0.0) return false;          // sign -1 (Cell.cpp:419-426)
    double q[3];
    if (rho < 1e-9) for (int a = 0; a < 3; ++a) q[a] = c[a];
    else for (int a = 0; a < 3; ++a) q[a] = c[a] + (ctt[a] / rho) * radius;
    double dv[3];
    for (int a = 0; a < 3; ++a) dv[a] = q[a] - c[a];
    for (int a = 0; a < 3; ++a) row[a] = alpha * ssw * dv[a];
    row[3] = ssw * ((dot3(q, dv) - beta * dot3(Hp, dv)) - gamma * dot3(Fp, dv));
    return true;
}

// The Hermite rows dc_weight * n_e in edge order and the Hermite centroid.
__device__ void hermite_rows(const OursParams& P, const OursCell& S, double* H0, double* cen) {
    for (int q = 0; q < 9; ++q) H0[q] = 0.0;
    cen[0] = cen[1] = cen[2] = 0.0;
    int m = 0;
    for (int e = 0; e < 12; ++e) {
        if (!(S.hmask & (1 << e))) continue;
        double sn[3];
        for (int d = 0; d < 3; ++d) sn[d] = P.dc_weight * S.hn[e][d];
        const double b = dot3(sn, S.hp[e]);
        H0[0] += sn[0] * sn[0]; H0[1] += sn[0] * sn[1]; H0[2] += sn[0] * sn[2];
        H0[3] += sn[1] * sn[1]; H0[4] += sn[1] * sn[2]; H0[5] += sn[2] * sn[2];
        H0[6] += sn[0] * b; H0[7] += sn[1] * b; H0[8] += sn[2] * b;
        for (int d = 0; d < 3; ++d) cen[d] += S.hp[e][d];
        ++m;
    }
    for (int d = 0; d < 3; ++d) cen[d] /= double(m);
}

// solve_quadratic_system (Cell.cpp:324-361) with the proximal rows sqrt(mu) * I added.
__device__ void inner_solve(const OursParams& P, const double Acc[9], const double* prev, const double cen[3],
                            double smu, double x[3]) {
    double A[3][3] = {{Acc[0], Acc[1], Acc[2]}, {Acc[1], Acc[3], Acc[4]}, {Acc[2], Acc[4], Acc[5]}};
    double b[3] = {Acc[6], Acc[7], Acc[8]};
    for (int a = 0; a < 3; ++a) { A[a][a] += smu * smu; b[a] += smu * (smu * prev[a]); }
    double E[3][3], U[3][3];
    for (int a = 0; a < 3; ++a) for (int c = 0; c < 3; ++c) E[a][c] = A[a][c];
    f64::jacobi3(E, U);
    double rhs[3];
    for (int a = 0; a < 3; ++a) rhs[a] = b[a] - (A[a][0] * cen[0] + A[a][1] * cen[1] + A[a][2] * cen[2]);
    x[0] = cen[0]; x[1] = cen[1]; x[2] = cen[2];
    for (int q = 0; q < 3; ++q) {
        const double sv = fabs(E[q][q]);
        if (sv > P.thr) {
            const double coef = (U[0][q] * rhs[0] + U[1][q] * rhs[1] + U[2][q] * rhs[2]) / sv;
            for (int a = 0; a < 3; ++a) x[a] += U[a][q] * coef;
        }
    }
}

// The inner loop of the cells (contouring.cpp:1288-1309): refine_vertex_from_face_intersections
// (vertex_refinement.cpp:201-280) + Cell::minimize_qef (Cell.cpp:364-473) until the vertex
// moves less than 1e-6. A sphere's row is skipped or adds to the 6 entries of the symmetric
// A^T A (00 01 02 11 12 22) and the 3 of A^T b; rows are summed in 32 chunks of consecutive
// spheres, each from zero, added in chunk order: the same sums however the rows are dealt.
//
// A block holds up to kSlots cells, of at most kRows spheres together, and takes more from a
// counter as cells finish. An iteration of all of them: a lane per (cell, sphere) forms the rows
// (the distances to the local fan, most of the work), a lane per (cell, sum) adds them up,
// one warp solves, a lane per cell.
//
// What bounds it: FP64 instructions at their latency (43% of the issue slots of busy SMs), then cells
// of 100 iterations, a chain each. An outer iteration of a 128^3 perturbed sphere takes 2.7 ms
// (72^3, with cells of up to 1,600 spheres: 5.3; a 128^3 sphere 0.6). A team of 8 lanes per cell,
// each lane solving, took 4.7 (6.8): half the instructions were the same solves again, and 10 of
// 32 lanes were active (now 20). 28 slots as measured (32: 2.8; 24 with five blocks an SM: 2.8);
// 8 or 16 cells to a warp without block synchronisations: 5.0 (a warp's chain is too long); four
// lanes a sphere: 3.0-3.4. The cells are dealt by columns so that no block gets the large ones
// (taken in list order: 3.0).
constexpr int kInnerThreads = 128;
constexpr int kSlots = 28;                 // a lane of the solving warp each
constexpr unsigned int kRows = 512;
constexpr unsigned int kRefill = 4;        // free slots that are worth a fill
static_assert(kSlots <= 32 && kTeamSpheres[1] - 1 <= kRows && kRows >= kInnerThreads, "");
struct InnerShared {
    TeamCell cell[kSlots];
    double row[4][kRows];                  // entries 0..2 and the right-hand side
    double part[32][9];
    unsigned int first[kSlots + 1];        // each slot's first row; at the end their number
    unsigned int sphere[kSlots], source[kSlots];
    int nfan[kSlots];
    unsigned int fresh, next;
    bool done;
};

// The local fan of a cell: (vertex, Hermite point on edge e, face point d) for each face d with a
// point and each of its four edges with a Hermite point, in face then edge order. Its length;
// 0: nothing to do.
__device__ __forceinline__ int local_fan(int hmask, int fmask, unsigned char* fan) {
    int nfan = 0;
    for (int x = 0; x < 24; ++x) {
        const int d = x >> 2, e = kFaceEdges[d][x & 3];
        if ((fmask & (1 << d)) && (hmask & (1 << e))) fan[nfan++] = (unsigned char)(e | d << 4);
    }
    return nfan;
}

// Factors of the nine sums: row entries 0..2, 3 the right-hand side.
__device__ __forceinline__ int sum_left(int q) { return q < 3 ? 0 : q < 5 ? 1 : q == 5 ? 2 : q - 6; }
__device__ __forceinline__ int sum_right(int q) { return q < 3 ? q : q < 5 ? q - 2 : q == 5 ? 2 : 3; }

// Row `at` of the block from one sphere; a skipped row is zero (a sum that starts from zero is
// unchanged by +0).
__device__ __forceinline__ void put_row(InnerShared& S, unsigned int at, const TeamCell& C, int nfan, const float4* sphere,
                                        double ssw) {
    double row[4];
    const bool ok = sphere_row(C, nfan, sphere, ssw, row);
    for (int q = 0; q < 4; ++q) S.row[q][at] = ok ? row[q] : 0.0;
}

__device__ void inner_packed(const OursParams& P, InnerShared& S) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the warp that solves: another one in each of the blocks that share an SM (they share its schedulers)
    const bool solver = warp == (int)(blockIdx.x / ((gridDim.x + 3) / 4)) % (kInnerThreads / 32);
    const unsigned int big = P.team_count[1], ncells = big + P.team_count[0], share = min((ncells + gridDim.x - 1) / gridDim.x, (unsigned int)kSlots);
    // every take of `share` cells has one of each size class: the list, in pieces of share * blocks, by columns
    const unsigned int piece = share * gridDim.x;
    const double ssw = sqrt(P.sphere_weight), smu = sqrt(P.mu);
    TeamCell& C = S.cell[lane % kSlots];
    bool have = false, runs = false, more = ncells > 0;      // this lane's slot holds a cell; takes part; cells are left
    unsigned int r = 0, n = 0;
    int it = 0;
    for (;;) {
        if (solver) {
            const unsigned int held = __ballot_sync(0xffffffffu, have), waiting = __ballot_sync(0xffffffffu, have && !runs);
            const unsigned int rows = __reduce_add_sync(0xffffffffu, runs ? n : 0u);
            const unsigned int room = kSlots - __popc(held);
            bool fresh = false;
            if (more && !waiting && (room >= kRefill || !held)) {
                const unsigned int want = min(min(room, share), max((kRows - rows) / 8, held ? 0u : 1u));
                if (want) {
                    unsigned int w = 0;
                    if (lane == 0) w = atomicAdd(P.team_count + 3, want);
                    w = __shfl_sync(0xffffffffu, w, 0);
                    const unsigned int k = __popc(~held & ((1u << lane) - 1u));
                    const unsigned int at = (w + k) % piece, x = w + k - at + at % share * gridDim.x + at / share;
                    if (lane < kSlots && !have && k < want && x < ncells) {
                        r = x < big ? P.team_list[1][x] : P.team_list[0][x - big];
                        const OursCell& cell = P.cells[r];
                        const int nfan = local_fan(cell.hmask, cell.fmask, C.fan);
                        fresh = have = nfan > 0;
                        if (have) {
                            n = P.cell_count[r];
                            it = 0;
                            S.sphere[lane] = P.cell_start[r];
                            S.source[lane] = r;
                            S.nfan[lane] = nfan;
                            for (int a = 0; a < 3; ++a) C.prev[a] = cell.v[a];
                            hermite_rows(P, cell, C.h0, C.cen);
                        }
                    }
                    more = w + want < (ncells + piece - 1) / piece * piece;
                }
            }
            // cells wait until their rows have room
            unsigned int before = have && !runs ? n : 0u;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int t = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += t;
            }
            runs = have && (runs || rows + before <= kRows);
            unsigned int end = runs ? n : 0u;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int t = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += t;
            }
            if (lane < kSlots) S.first[lane + 1] = end;
            const unsigned int loads = __ballot_sync(0xffffffffu, fresh), left = __ballot_sync(0xffffffffu, have);
            if (lane == 0) { S.first[0] = 0; S.fresh = loads; S.done = !more && !left; }
        }
        __syncthreads();
        if (S.done) break;
        if (S.fresh) {
            for (int t = warp; t < kSlots; t += kInnerThreads / 32) {
                if (!(S.fresh >> t & 1)) continue;
                const OursCell& cell = P.cells[S.source[t]];
                for (int x = lane; x < 36; x += 32) (&S.cell[t].hp[0][0])[x] = (&cell.hp[0][0])[x];
                if (lane < 18) (&S.cell[t].fi[0][0])[lane] = (&cell.fi[0][0])[lane];
            }
            __syncthreads();
        }
        const unsigned int total = S.first[kSlots];
        for (unsigned int x = threadIdx.x; x < total; x += kInnerThreads) {
            int t = 0;                                  // the last slot that begins at or before x
            for (int st = 16; st; st >>= 1) if (t + st < kSlots && S.first[t + st] <= x) t += st;
            put_row(S, x, S.cell[t], S.nfan[t], P.cell_centres + S.sphere[t] + (x - S.first[t]), ssw);
        }
        __syncthreads();
        for (int x = threadIdx.x; x < 9 * kSlots; x += kInnerThreads) {
            const int t = x / 9, q = x % 9;
            const unsigned int b = S.first[t], m = S.first[t + 1] - b;
            if (!m) continue;
            const double* const l = S.row[sum_left(q)] + b;
            const double* const g = S.row[sum_right(q)] + b;
            double sum = S.cell[t].h0[q];
            if (m <= 32) {                              // a row a chunk
#pragma unroll 8
                for (unsigned int j = 0; j < m; ++j) sum += l[j] * g[j];
            } else {
                const unsigned int cs = (m + 31) / 32;
                for (unsigned int j = 0; j < m;) {
                    const unsigned int e = min(m, j + cs);
                    double part = 0.0;
                    for (; j < e; ++j) part += l[j] * g[j];
                    sum += part;
                }
            }
            S.cell[t].sums[q] = sum;
        }
        __syncthreads();
        if (solver && runs) {
            const double prev[3] = {C.prev[0], C.prev[1], C.prev[2]};
            double v[3];
            inner_solve(P, C.sums, prev, C.cen, smu, v);
            const double dm[3] = {v[0] - prev[0], v[1] - prev[1], v[2] - prev[2]};
            for (int a = 0; a < 3; ++a) C.prev[a] = v[a];
            if (norm3(dm) < 1e-6 || ++it >= P.inner_iters) {
                have = runs = false;
                for (int a = 0; a < 3; ++a) P.cells[r].v[a] = v[a];
            }
        }
    }
}

// The same for one cell with a whole block: 4 lanes a chunk.
__device__ void inner_block(const OursParams& P, InnerShared& S) {
    constexpr int T = kInnerThreads, kLanes = T / 32;
    TeamCell& C = S.cell[0];
    const int tid = threadIdx.x, chunk = tid / kLanes, sub = tid % kLanes;
    const unsigned int ncells = P.team_count[2];
    const double ssw = sqrt(P.sphere_weight), smu = sqrt(P.mu);
    for (;;) {
        __syncthreads();
        if (tid == 0) S.next = atomicAdd(P.team_count + 4, 1u);
        __syncthreads();
        if (S.next >= ncells) break;
        const long long r = P.team_list[2][S.next];
        const OursCell& cell = P.cells[r];
        if (tid == 0) {
            S.nfan[0] = local_fan(cell.hmask, cell.fmask, C.fan);
            hermite_rows(P, cell, C.h0, C.cen);
        }
        for (int x = tid; x < 36; x += T) (&C.hp[0][0])[x] = (&cell.hp[0][0])[x];
        for (int x = tid; x < 18; x += T) (&C.fi[0][0])[x] = (&cell.fi[0][0])[x];
        const unsigned int nsph = P.cell_count[r], cs = (nsph + 31) / 32, nchunks = (nsph + cs - 1) / cs;
        const float4* const sph = P.cell_centres + P.cell_start[r];
        if (tid < 3) C.prev[tid] = cell.v[tid];
        __syncthreads();
        const int nfan = S.nfan[0];
        if (!nfan) continue;
        for (int it = 0; it < P.inner_iters; ++it) {
            for (int x = tid; x < 32 * 9; x += T) (&S.part[0][0])[x] = 0.0;
            for (unsigned int k = 0; k < cs; k += kLanes) {
                const unsigned int s = chunk * cs + k + sub;
                if (k + sub < cs && s < nsph) put_row(S, tid, C, nfan, sph + s, ssw);
                else for (int q = 0; q < 4; ++q) S.row[q][tid] = 0.0;
                __syncthreads();
                for (int x = tid; x < 32 * 9; x += T) {
                    const int l = x / 9, e = x % 9;
                    double part = S.part[l][e];
                    for (int j = l * kLanes; j < (l + 1) * kLanes; ++j)
                        part += S.row[sum_left(e)][j] * S.row[sum_right(e)][j];
                    S.part[l][e] = part;
                }
                __syncthreads();
            }
            if (tid < 9) {
                double sum = C.h0[tid];
                for (unsigned int l = 0; l < nchunks; ++l) sum += S.part[l][tid];
                C.sums[tid] = sum;
            }
            __syncthreads();
            bool done = false;
            if (tid < 32) {
                const double prev[3] = {C.prev[0], C.prev[1], C.prev[2]};
                double v[3];
                inner_solve(P, C.sums, prev, C.cen, smu, v);
                const double dm[3] = {v[0] - prev[0], v[1] - prev[1], v[2] - prev[2]};
                done = norm3(dm) < 1e-6;
                __syncwarp();
                if (tid < 3) C.prev[tid] = tid == 0 ? v[0] : tid == 1 ? v[1] : v[2];
            }
            if (__syncthreads_or(done)) break;
        }
        if (tid < 3) P.cells[r].v[tid] = C.prev[tid];
    }
}

// Longest cells first; every block that fits on the GPU takes cells from the counters, so a block
// with a long cell keeps only itself.
constexpr int kInnerBlocks = 4;            // per SM
__global__ void __launch_bounds__(kInnerThreads, kInnerBlocks) k_ours_inner(const __grid_constant__ OursParams P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    InnerShared& S = *reinterpret_cast<InnerShared*>(s_raw);
    inner_block(P, S);
    __syncthreads();
    inner_packed(P, S);
}

__global__ void k_ours_mesh(OursParams P) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < P.nv; r += (long long)gridDim.x * blockDim.x)
        for (int d = 0; d < 3; ++d) P.Vm[3 * r + d] = P.cells[r].v[d];
}

// The output: vertices as float; quads wound by the edge's gradient (contouring.cpp:624-641),
// or their triangles oriented like the quad (triangulate_v1 + orient_triangles_for_quad,
// contouring.cpp:40-113).
__global__ void __launch_bounds__(128) k_ours_output(OursParams P, int triangles) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < P.nv; r += stride)
        for (int d = 0; d < 3; ++d) P.out_V[3 * r + d] = (float)P.Vm[3 * r + d];
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < P.nq; q += stride) {
        const int4 f = wound_quad(P, q);
        if (!triangles) { P.out_faces[q] = f; continue; }
        int t0[3], t1[3];
        quad_triangles(P, f, t0, t1);
        int* out = reinterpret_cast<int*>(P.out_faces) + 6 * q;
        out[0] = t0[0]; out[1] = t0[1]; out[2] = t0[2];
        out[3] = t1[0]; out[4] = t1[1]; out[5] = t1[2];
    }
}

// ---- host --------------------------------------------------------------------------------

namespace {
inline unsigned grid_for(long long n, int threads, int num_sms) {
    long long b = (n + threads - 1) / threads;
    const long long cap = (long long)num_sms * 32;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}
inline size_t al(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

size_t ours_workspace_bytes(long long nv, long long nq, long long npts, size_t* sort_bytes) {
    const long long nt = 2 * nq;
    // radix sorts: triangle codes (32-bit keys) and point keys (64-bit keys), 32-bit values
    *sort_bytes = std::max(radix_sort_temp_bytes(std::max(1LL, nt), 4, true),
                          radix_sort_temp_bytes(std::max(1LL, npts), 8, true));
    size_t b = 0;
    b += al(sizeof(OursCell) * nv) + al(sizeof(double) * 3 * nv);            // cells, Vm
    b += al(sizeof(int4) * nq) + al(sizeof(double) * 3 * nq);               // quads, gsum
    b += 3 * al(sizeof(uint32_t) * npts) + al(sizeof(int) * npts);           // sel, band/rest, sel_cell
    b += al(sizeof(unsigned long long) * 2 * npts) + al(sizeof(uint32_t) * npts);  // fill keys/values; sphere centres, long searches
    b += 3 * al(sizeof(unsigned int) * (nv + 1)) + al(sizeof(uint32_t) * npts);    // count/start/fill, spheres
    b += 3 * al(sizeof(uint32_t) * (nv + 1));                                // cells by number of spheres
    b += al(sizeof(uint32_t) * npts);                                        // selected points, sorted
    b += al(sizeof(int) * npts);                                             // last closest triangle per point
    b += al(sizeof(unsigned long long) * nt) + al(sizeof(BvhNode) * nt) + al(sizeof(int) * 2 * nt);
    b += 4 * al(sizeof(uint32_t) * nt);                                      // triangle codes / indices
    b += al(sizeof(unsigned int) * nt) + al(sizeof(double) * 9 * nt);
    b += al(sizeof(uint32_t) * (scan_partials_len(nv + 1) + 1)) + al(64);    // scan partials, counters
    b += al(sizeof(unsigned int) * (kFillBins + 2));                         // random fill
    b += al(*sort_bytes);
    return b + 4096;
}

cudaError_t ours_run(OursRun& R, cudaStream_t s) {
    OursParams& P = R.P;
    const long long nv = P.nv, nq = P.nq, nt = 2 * nq, npts = (long long)P.g.nx * P.g.ny * P.g.nz;
    char* base = reinterpret_cast<char*>(R.workspace);
    size_t at = 0;
    auto take = [&](size_t bytes) { void* p = base + at; at += al(bytes); return p; };
    P.cells = (OursCell*)take(sizeof(OursCell) * nv);
    P.Vm = (double*)take(sizeof(double) * 3 * nv);
    P.quads = (int4*)take(sizeof(int4) * nq);
    P.gsum = (double*)take(sizeof(double) * 3 * nq);
    uint32_t* sel = (uint32_t*)take(sizeof(uint32_t) * npts);
    uint32_t* band = (uint32_t*)take(sizeof(uint32_t) * npts);
    uint32_t* rest = (uint32_t*)take(sizeof(uint32_t) * npts);
    P.sel_cell = (int*)take(sizeof(int) * npts);
    // the keys and values of the selection are done with when the queries begin; the spheres'
    // centres and the list of long searches then take their place
    unsigned long long* fk = (unsigned long long*)take(sizeof(unsigned long long) * 2 * npts);
    unsigned long long* fk2 = fk + npts;
    uint32_t* fv2 = (uint32_t*)take(sizeof(uint32_t) * npts);
    P.cell_centres = (float4*)fk;
    P.long_query = fv2;
    static_assert(sizeof(float4) == 2 * sizeof(unsigned long long), "");
    P.cell_count = (unsigned int*)take(sizeof(unsigned int) * (nv + 1));
    P.cell_start = (unsigned int*)take(sizeof(unsigned int) * (nv + 1));
    P.cell_fill = (unsigned int*)take(sizeof(unsigned int) * (nv + 1));
    P.cell_spheres = (uint32_t*)take(sizeof(uint32_t) * npts);
    for (int q = 0; q < 3; ++q) P.team_list[q] = (uint32_t*)take(sizeof(uint32_t) * (nv + 1));
    P.mkeys_sorted = (unsigned long long*)take(sizeof(unsigned long long) * nt);
    P.tcode = (uint32_t*)take(sizeof(uint32_t) * nt);
    P.tidx = (uint32_t*)take(sizeof(uint32_t) * nt);
    P.tcode_sorted = (uint32_t*)take(sizeof(uint32_t) * nt);
    P.tidx_sorted = (uint32_t*)take(sizeof(uint32_t) * nt);
    P.nodes = (BvhNode*)take(sizeof(BvhNode) * nt);
    P.parent = (int*)take(sizeof(int) * 2 * nt);
    P.flags = (unsigned int*)take(sizeof(unsigned int) * nt);
    P.tri9 = (double*)take(sizeof(double) * 9 * nt);
    uint32_t* partials = (uint32_t*)take(sizeof(uint32_t) * (scan_partials_len(nv + 1) + 1));
    unsigned int* counters = (unsigned int*)take(64);
    void* sort_temp = take(R.sort_bytes);
    uint32_t* sel_sorted = (uint32_t*)take(sizeof(uint32_t) * npts);
    P.prev_tri = (int*)take(sizeof(int) * npts);
    unsigned int* fill_hist = (unsigned int*)take(sizeof(unsigned int) * (kFillBins + 2));
    P.team_count = counters + 8;
    P.long_count = counters + 14;
    P.sel = sel_sorted;
    P.nt = nt;
    const int sms = R.num_sms;
    cudaError_t e;
#define OURS_TRY(x) do { e = (x); if (e != cudaSuccess) return e; } while (0)
    OURS_TRY(cudaMemsetAsync(counters, 0, 64, s));
    OURS_TRY(cudaMemsetAsync(P.prev_tri, 0xff, sizeof(int) * npts, s));
    k_ours_init<<<grid_for(nv, 128, sms), 128, 0, s>>>(P);
    k_ours_quads<<<grid_for(nq, 128, sms), 128, 0, s>>>(P);
    k_ours_select<<<grid_for(npts, 256, sms), 256, 0, s>>>(P, npts, band, rest, counters);
    OURS_TRY(cudaGetLastError());
    unsigned int hc[2] = {0, 0};
    OURS_TRY(cudaMemcpyAsync(hc, counters, sizeof(hc), cudaMemcpyDeviceToHost, s));
    OURS_TRY(cudaStreamSynchronize(s));
    const long long nband = hc[0], nrest = hc[1];
    const long long bounded = std::min<long long>(R.batch_size, npts);
    const long long nfill = nband < bounded ? std::min(bounded - nband, nrest) : 0;
    P.nsel = nband + nfill;
    // the near-surface points never change: Morton-ordered once (a warp's queries then cover
    // a compact block of the grid); a random fill is ordered again every outer iteration
    if (nband > 0) {
        k_ours_point_keys<<<grid_for(nband, 256, sms), 256, 0, s>>>(P, band, nband, fk);
        OURS_TRY(radix_sort_pairs(sort_temp, R.sort_bytes, fk, fk2, band, sel_sorted, nband, 0, 63, s));
    }
    OURS_TRY(cudaFuncSetAttribute(k_ours_inner, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(InnerShared)));
    for (int it = 0; it < R.outer_iters; ++it) {
        if (nq > 0) {
            k_ours_tris<<<grid_for(nq, 128, sms), 128, 0, s>>>(P);
            OURS_TRY(radix_sort_pairs(sort_temp, R.sort_bytes, P.tcode, P.tcode_sorted, P.tidx, P.tidx_sorted, nt, 0, 30, s));
            k_bvh_keys<<<grid_for(nt, 256, sms), 256, 0, s>>>(P);
            OURS_TRY(cudaMemsetAsync(P.flags, 0, sizeof(unsigned int) * nt, s));
            if (nt > 1) k_bvh_tree<<<grid_for(nt - 1, 128, sms), 128, 0, s>>>(P);
            else OURS_TRY(cudaMemsetAsync(P.parent, 0xff, sizeof(int) * 2, s));
            k_bvh_boxes<<<grid_for(nt, 128, sms), 128, 0, s>>>(P);
            if (nfill > 0) {
                const unsigned int take = (unsigned int)nfill, blocks = grid_for(nrest, 4 * kFillThreads, sms / 4);
                uint32_t* const out = nfill > kFillUnsorted ? sel : sel_sorted + nband;
                OURS_TRY(cudaMemsetAsync(fill_hist, 0, sizeof(unsigned int) * (kFillBins + 2), s));
                k_ours_fill_hist<<<blocks, kFillThreads, 0, s>>>(rest, nrest, R.seed, it, fill_hist);
                k_ours_fill_take<<<blocks, kFillThreads, 0, s>>>(rest, nrest, R.seed, it, take, fill_hist, out, fk, fv2,
                                                                 fill_hist + kFillBins);
                k_ours_fill_last<<<1, 1024, 0, s>>>(take, fk, fv2, out, fill_hist + kFillBins);
                if (out == sel) {
                    k_ours_point_keys<<<grid_for(nfill, 256, sms), 256, 0, s>>>(P, sel, nfill, fk);
                    OURS_TRY(radix_sort_pairs(sort_temp, R.sort_bytes, fk, fk2, sel, sel_sorted + nband, nfill, 0, 63, s));
                }
            }
            OURS_TRY(cudaMemsetAsync(P.cell_count, 0, sizeof(unsigned int) * (nv + 1), s));
            OURS_TRY(cudaMemsetAsync(P.cell_fill, 0, sizeof(unsigned int) * (nv + 1), s));
            OURS_TRY(cudaMemsetAsync(P.team_count, 0, sizeof(unsigned int) * 7, s));
            k_ours_query<<<grid_for(P.nsel, 128, sms), 128, 0, s>>>(P);
            k_ours_query_long<<<(unsigned)sms * 8, 32 * kLongWarps, 0, s>>>(P);
            OURS_TRY(launch_scan(P.cell_count, nv, partials, P.cell_start,
                                 reinterpret_cast<unsigned long long*>(counters + 4), s));
            k_ours_scatter<<<grid_for(P.nsel, 128, sms), 128, 0, s>>>(P);
            k_ours_sort<<<grid_for(nv, 128, sms), 128, 0, s>>>(P);
        } else {
            OURS_TRY(cudaMemsetAsync(P.cell_count, 0, sizeof(unsigned int) * (nv + 1), s));
            OURS_TRY(cudaMemsetAsync(P.team_count, 0, sizeof(unsigned int) * 7, s));
        }
        k_ours_faces<<<grid_for(nv, 128, sms), 128, 0, s>>>(P);
        if (R.hermite_update && it > 0) k_ours_hermite<<<grid_for(12 * nv, 128, sms), 128, 0, s>>>(P);
        if (P.inner_iters > 0) k_ours_inner<<<(unsigned)sms * kInnerBlocks, kInnerThreads, sizeof(InnerShared), s>>>(P);
        k_ours_mesh<<<grid_for(nv, 128, sms), 128, 0, s>>>(P);
        OURS_TRY(cudaGetLastError());
    }
    if (R.outer_iters == 0) k_ours_mesh<<<grid_for(nv, 128, sms), 128, 0, s>>>(P);
    k_ours_output<<<grid_for(std::max(nv, nq), 128, sms), 128, 0, s>>>(P, R.triangles);
    OURS_TRY(cudaGetLastError());
#undef OURS_TRY
    return cudaSuccess;
}

}  // namespace dcb
