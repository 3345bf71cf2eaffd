// dcb_mesh_sdf.cu — triangle mesh -> dense signed distance grid.
//
// Semantics: compute_mesh_sdf_device_cuda without voxelisation
// (src/cuda/mesh_to_sdf_cuda.cu:740-1009, branch :862-951):
//   bins         g = max(1, n/8) per axis, bin size (n*v)/g, every triangle listed in each bin
//                its bounding box grown by 2*max(v) overlaps (:99-190)
//   active bins  some bin of the 3x3x3 block around it is non-empty (:192-224)
//   band         per grid point: closest point over the triangles of its bin, then of the 26
//                neighbours (z, y, x order), ties within 1e-5 relative sum area- (or, at a
//                vertex, angle-) weighted normals; sign from the summed normal; |d| beyond 2.5
//                bins -> far (:226-360)
//   sign fill    far points reached from the border or from a positive point through far
//                points are +10, the other far points -10 (:362-428)
//   relaxation   4 Jacobi passes of |v| <- min(|v|, |neighbour| + h) beyond 1.5 h (:430-456)
// Determinism (the reference fills bins with atomics and floods with racing in-place
// passes): bins list their triangles in ascending index, and the flood runs to its fixpoint.
// The file is compiled with --fmad=false: every float expression is rounded as written, like
// the CPU restatement it is checked against.
//
// B200 layout of the work:
//   k_tri_prep      triangle records (bounding sphere, vertices, unit normal, doubled area)
//                   + per-bin counts (atomics)
//   k_tri_bins      scatter into bins (atomics), then k_bin_order ranks each bin's entries
//                   by triangle index (CTA per bin, shared-memory tiles), so the order is the
//                   ascending one whatever the atomics did
//   k_bin_active    the active bins as a list of work items; k_axis_starts the
//                   first grid point of every bin per axis; k_fill_far sets every value far
//   k_band          persistent CTAs take work items (a bin or a part of a long one) from a
//                   counter; the distinct triangles that may be nearest to the item's points are
//                   staged once in shared memory, a warp takes 32 points at a time (a brick of up
//                   to 4x4x2), finds each point's minimum and the triangles that tie with it,
//                   and decides value and sign on those (the reference's walk over every listed
//                   triangle, without the ones that cannot change its result)
//   k_sdf_masks     far / positive bit words (ballots over x rows)
//   k_flood         exterior flood on bit words: 4x16x16-word tiles iterate to local
//                   convergence in shared memory; the host repeats until nothing changes
//   k_sdf_relax     far -> +-10 and the 4 relaxation passes in one sweep
#include <algorithm>
#include <cfloat>
#include "dcb_kernels.cuh"

namespace dcb {

namespace {

constexpr float kFar = FLT_MAX;

// Triangle record, 6 x 16 bytes. Behind the records: every triangle's unit normal (within them it would
// take 2 to 4% of the band's time at 100^3: records of 112 or 128 bytes).
struct Tri {
    float4 s;       // bounding sphere: centroid xyz, radius grown by a rounding allowance
    float a2;       // doubled area (0: skipped, as the reference skips area <= 1e-12)
    uint32_t r[3];  // bins it is listed in, per axis: first | last << 16 (kPackedBins axes and below)
    float v[9];     // vertices
    float n[3];     // unit normal; 0 where it bounds no distance (a thin triangle's) or its weight may
                    // leave a sum of normals without a side (a corner angle of 0, an area whose
                    // square overflows)
    float w[4];     // tie weights of its vertices: the angles there
};
constexpr int kTriF4 = 6;
constexpr int kTriList = 5;             // of them the distances need
constexpr int kTriAngles = 5;
constexpr int kPackedBins = 65536;
static_assert(sizeof(Tri) == kTriF4 * sizeof(float4), "record = kTriF4 float4s");

__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 add(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 sub(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 scl(float s, float3 a) { return f3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
    return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

__device__ __forceinline__ int bin_coord(float x, float o, float bd, int g) {
    return max(0, min(g - 1, (int)floorf((x - o) / bd)));
}

// Closest point on triangle abc to p and its squared distance (Ericson, Real-Time Collision
// Detection 5.1.5; the case analysis of mesh_to_sdf_cuda.cu:40-97).
__device__ float point_triangle(float3 p, float3 a, float3 b, float3 c, float3& out) {
    const float3 ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
    const float d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0.0f && d2 <= 0.0f) { out = a; return dot(ap, ap); }
    const float3 bp = sub(p, b);
    const float d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= 0.0f && d4 <= d3) { out = b; return dot(bp, bp); }
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        const float v = d1 / (d1 - d3);
        out = add(a, scl(v, ab));
        const float3 e = sub(p, out);
        return dot(e, e);
    }
    const float3 cp = sub(p, c);
    const float d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0.0f && d5 <= d6) { out = c; return dot(cp, cp); }
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        const float w = d2 / (d2 - d6);
        out = add(a, scl(w, ac));
        const float3 e = sub(p, out);
        return dot(e, e);
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        out = add(b, scl(w, sub(c, b)));
        const float3 e = sub(p, out);
        return dot(e, e);
    }
    const float denom = 1.0f / (va + vb + vc);
    const float v = vb * denom, w = vc * denom;
    out = add(add(a, scl(v, ab)), scl(w, ac));
    const float3 e = sub(p, out);
    return dot(e, e);
}

__device__ __forceinline__ float angle_at(float3 e1, float3 e2, float fallback) {
    const float l1 = sqrtf(dot(e1, e1)), l2 = sqrtf(dot(e2, e2));
    if (l1 > 1e-6f && l2 > 1e-6f) {
        const float c = fmaxf(-1.0f, fminf(1.0f, dot(e1, e2) / (l1 * l2)));
        return (float)acos((double)c);
    }
    return fallback;
}

__device__ __forceinline__ void tri_bin_range(const SdfParams& P, float3 a, float3 b, float3 c, int* r) {
    const float mnx = fminf(a.x, fminf(b.x, c.x)) - P.margin;
    const float mny = fminf(a.y, fminf(b.y, c.y)) - P.margin;
    const float mnz = fminf(a.z, fminf(b.z, c.z)) - P.margin;
    const float mxx = fmaxf(a.x, fmaxf(b.x, c.x)) + P.margin;
    const float mxy = fmaxf(a.y, fmaxf(b.y, c.y)) + P.margin;
    const float mxz = fmaxf(a.z, fmaxf(b.z, c.z)) + P.margin;
    r[0] = bin_coord(mnx, P.ox, P.bdx, P.gx); r[1] = bin_coord(mxx, P.ox, P.bdx, P.gx);
    r[2] = bin_coord(mny, P.oy, P.bdy, P.gy); r[3] = bin_coord(mxy, P.oy, P.bdy, P.gy);
    r[4] = bin_coord(mnz, P.oz, P.bdz, P.gz); r[5] = bin_coord(mxz, P.oz, P.bdz, P.gz);
}

__device__ __forceinline__ bool load_tri(const SdfParams& P, long long f, float3& a, float3& b, float3& c) {
    const int i0 = P.faces[3 * f], i1 = P.faces[3 * f + 1], i2 = P.faces[3 * f + 2];
    if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= P.nv || i1 >= P.nv || i2 >= P.nv) {
        set_error(P.err, kErrInvalid);
        return false;
    }
    a = f3(P.verts[3 * (size_t)i0], P.verts[3 * (size_t)i0 + 1], P.verts[3 * (size_t)i0 + 2]);
    b = f3(P.verts[3 * (size_t)i1], P.verts[3 * (size_t)i1 + 1], P.verts[3 * (size_t)i1 + 2]);
    c = f3(P.verts[3 * (size_t)i2], P.verts[3 * (size_t)i2 + 1], P.verts[3 * (size_t)i2 + 2]);
    return true;
}

__global__ void __launch_bounds__(256) k_tri_prep(SdfParams P) {
    unsigned long long entries = 0;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < P.nf; f += (long long)gridDim.x * blockDim.x) {
        float3 a, b, c;
        if (!load_tri(P, f, a, b, c)) continue;
        float3 n = cross(sub(b, a), sub(c, a));
        const float a2 = sqrtf(dot(n, n));
        const bool ok = a2 > 1e-12f;
        if (ok) n = f3(n.x / a2, n.y / a2, n.z / a2);
        // Bounding sphere about the centroid; the radius is grown by 1e-5 of the coordinate
        // magnitudes so that it bounds the float closest points as well.
        const float3 cc = f3((a.x + b.x + c.x) / 3.f, (a.y + b.y + c.y) / 3.f, (a.z + b.z + c.z) / 3.f);
        const float3 da = sub(a, cc), db = sub(b, cc), dcv = sub(c, cc);
        const float R = sqrtf(fmaxf(dot(da, da), fmaxf(dot(db, db), dot(dcv, dcv))));
        const float mag = fmaxf(fmaxf(fabsf(cc.x), fabsf(cc.y)), fabsf(cc.z)) + R;
        int r[6];
        tri_bin_range(P, a, b, c, r);
        float4* t = reinterpret_cast<float4*>(P.tris) + kTriF4 * (size_t)f;
        t[0] = make_float4(cc.x, cc.y, cc.z, R * 1.0001f + 1e-5f * mag);
        t[1] = make_float4(ok ? a2 : 0.f, __uint_as_float((uint32_t)r[0] | (uint32_t)r[1] << 16),
                           __uint_as_float((uint32_t)r[2] | (uint32_t)r[3] << 16),
                           __uint_as_float((uint32_t)r[4] | (uint32_t)r[5] << 16));
        t[2] = make_float4(a.x, a.y, a.z, b.x);
        t[3] = make_float4(b.y, b.z, c.x, c.y);
        const float3 w = f3(angle_at(sub(b, a), sub(c, a), a2), angle_at(sub(a, b), sub(c, b), a2),
                            angle_at(sub(a, c), sub(b, c), a2));
        // The float normal is off by up to 3 sqrt(3) ulps (2^-24) of the longest edge's square over
        // the doubled area, the edge being two radii at most: the triangle leaves the plane by that
        // angle's part of R. Half of the allowance of `beyond` without its pm may go there.
        const bool thin = !(1.25e-6f * R * R * R <= 1e-5f * a2 * (R + fabsf(cc.x) + fabsf(cc.y) + fabsf(cc.z)));
        // (kBandTies areas, each added by up to 27 bins, have a square below FLT_MAX)
        const bool plain = !thin && w.x > 0.f && w.y > 0.f && w.z > 0.f && a2 < 5e16f;
        t[4] = plain ? make_float4(c.z, n.x, n.y, n.z) : make_float4(c.z, 0.f, 0.f, 0.f);
        t[kTriAngles] = make_float4(w.x, w.y, w.z, 0.f);
        reinterpret_cast<float4*>(P.tris)[kTriF4 * (size_t)P.nf + f] = make_float4(n.x, n.y, n.z, 0.f);
        entries += (unsigned long long)(r[1] - r[0] + 1) * (unsigned)(r[3] - r[2] + 1) * (unsigned)(r[5] - r[4] + 1);
        for (int bz = r[4]; bz <= r[5]; ++bz)
            for (int by = r[2]; by <= r[3]; ++by)
                for (int bx = r[0]; bx <= r[1]; ++bx)
                    atomicAdd(&P.bin_count[bx + (long long)P.gx * (by + (long long)P.gy * bz)], 1u);
    }
    // their number in 64 bits (the bins' starts have 32: the host refuses more)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) entries += __shfl_xor_sync(0xffffffffu, entries, o);
    if ((threadIdx.x & 31) == 0 && entries) atomicAdd(P.entries, entries);
}

__global__ void __launch_bounds__(256) k_tri_bins(SdfParams P) {
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < P.nf; f += (long long)gridDim.x * blockDim.x) {
        float3 a, b, c;
        if (!load_tri(P, f, a, b, c)) continue;
        int r[6];
        tri_bin_range(P, a, b, c, r);
        for (int bz = r[4]; bz <= r[5]; ++bz)
            for (int by = r[2]; by <= r[3]; ++by)
                for (int bx = r[0]; bx <= r[1]; ++bx) {
                    const long long bin = bx + (long long)P.gx * (by + (long long)P.gy * bz);
                    const uint32_t slot = P.bin_start[bin] + atomicAdd(&P.bin_fill[bin], 1u);
                    P.bin_scratch[slot] = (uint32_t)f;
                }
    }
}

// CTA per bin: entry e goes to position (number of entries with a smaller triangle index);
// triangle indices are unique within a bin.
constexpr int kOrderThreads = 128;
constexpr int kOrderTile = 1024;
__global__ void __launch_bounds__(kOrderThreads) k_bin_order(SdfParams P) {
    __shared__ uint32_t s_key[kOrderTile];
    for (long long bin = blockIdx.x; bin < P.nbins; bin += gridDim.x) {
        const uint32_t start = P.bin_start[bin], n = P.bin_count[bin];
        if (n == 0) continue;
        const uint32_t* in = P.bin_scratch + start;
        for (uint32_t i0 = 0; i0 < n; i0 += kOrderThreads * 8) {
            uint32_t key[8], rank[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t i = i0 + threadIdx.x + q * kOrderThreads;
                key[q] = i < n ? in[i] : 0xffffffffu;
                rank[q] = 0;
            }
            for (uint32_t j0 = 0; j0 < n; j0 += kOrderTile) {
                const uint32_t m = min((uint32_t)kOrderTile, n - j0);
                __syncthreads();
                for (uint32_t j = threadIdx.x; j < m; j += kOrderThreads) s_key[j] = in[j0 + j];
                __syncthreads();
                for (uint32_t j = 0; j < m; ++j) {
                    const uint32_t kj = s_key[j];
#pragma unroll
                    for (int q = 0; q < 8; ++q) rank[q] += kj < key[q] ? 1u : 0u;
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t i = i0 + threadIdx.x + q * kOrderThreads;
                if (i < n) P.bin_tris[start + rank[q]] = key[q];
            }
        }
        __syncthreads();
    }
}

// Work items of the band kernel: at most 1 + entries / kPartEntries a bin. Parts repeat the
// staging of their bin's triangles (512^3, 163,840 triangles: 13.5 ms with parts of 256 entries,
// 11.3 with 1024) but spread the few long bins of a dense mesh (100^3, 10,240 triangles: 2.0 ms
// whole, 1.2 with either).
constexpr uint32_t kPartEntries = 1024;
__global__ void __launch_bounds__(256) k_bin_active(SdfParams P) {
    for (long long bin = (long long)blockIdx.x * blockDim.x + threadIdx.x; bin < P.nbins; bin += (long long)gridDim.x * blockDim.x) {
        const int bx = (int)(bin % P.gx), by = (int)((bin / P.gx) % P.gy), bz = (int)(bin / ((long long)P.gx * P.gy));
        uint32_t entries = 0;
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    const int x = bx + dx, y = by + dy, z = bz + dz;
                    if (x < 0 || x >= P.gx || y < 0 || y >= P.gy || z < 0 || z >= P.gz) continue;
                    entries += P.bin_count[x + (long long)P.gx * (y + (long long)P.gy * z)];
                }
        if (!entries) continue;
        // a bin with many entries is worked on in parts by several CTAs (its order in the list is
        // irrelevant: parts from the front, whole bins from the end)
        const uint32_t parts = entries <= kPartEntries ? 1u : entries <= 4 * kPartEntries ? 2u : entries <= 8 * kPartEntries ? 4u : 8u;
        const uint32_t at = atomicAdd(P.item_counts + (parts > 1 ? 0 : 1), parts);
        for (uint32_t q = 0; q < parts; ++q)
            P.items[parts > 1 ? at + q : P.items_cap - 1 - at] = make_uint2((uint32_t)bin, q | parts << 8);
    }
}

// First grid point along an axis whose bin coordinate is >= b: bisection, since bins are monotone in
// the point index. (Not a search from near the nominal b*n/g: where the spacing is small against the
// origin, positions round together and a bin can begin any number of points earlier.)
__device__ int first_point_of_bin(int b, int n, int g, float o, float v, float bd) {
    if (b <= 0) return 0;
    if (b >= g) return n;
    int lo = 0, hi = n;                          // the first one is in [lo, hi]
    while (lo < hi) {
        const int x = lo + (hi - lo) / 2;
        if (bin_coord(o + (float)x * v, o, bd, g) < b) lo = x + 1;
        else hi = x;
    }
    return lo;
}

// axis_start = [x: gx+1][y: gy+1][z: gz+1] first points of the bins along each axis.
__global__ void k_axis_starts(SdfParams P) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t <= P.gx) P.axis_start[t] = first_point_of_bin(t, P.nx, P.gx, P.ox, P.vx, P.bdx);
    else if (t <= P.gx + 1 + P.gy) P.axis_start[t] = first_point_of_bin(t - (P.gx + 1), P.ny, P.gy, P.oy, P.vy, P.bdy);
    else if (t <= P.gx + P.gy + P.gz + 2) P.axis_start[t] = first_point_of_bin(t - (P.gx + P.gy + 2), P.nz, P.gz, P.oz, P.vz, P.bdz);
}

// Every value starts far; the band kernel overwrites the points of the active bins. (Scalar
// stores: the caller's array need not be 16-byte aligned.)
__global__ void __launch_bounds__(256) k_fill_far(SdfParams P) {
    const long long n = (long long)P.nx * P.ny * P.nz;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        P.out[q] = kFar;
}

constexpr int kBandThreads = 128;
constexpr int kBandWarps = kBandThreads / 32;
constexpr int kBandCtasPerSm = 6;
// Triangle records a CTA holds at a time: what leaves room for six CTAs on an SM (a list of 224
// sends more bins through several lists: 11.8 ms against 11.3 at 512^3).
constexpr int kBandList = 336;
constexpr int kBandTies = 7;       // triangles within the tie window of a point's minimum
// Bricks that need the full walk have a bit each, by their number modulo kBandBits. Evenly spaced
// bins have at most 15 points an axis (125 bricks, most bins 16); where the spacing is small
// against the origin, positions round together and a bin can hold any number of points. So an item
// is worked on in pieces of kBandPiece bricks, whose groups of kBandWarps fall on different bits.
constexpr int kBandBits = 128, kBandPiece = kBandBits - kBandWarps;
static_assert(kBandBits % 32 == 0 && 32 % kBandWarps == 0, "a group of bricks lies in one word");

// Running closest-triangle state of one grid point: squared distance, closest point, summed normals.
struct BandPoint {
    float best;
    float3 bp, bn;
};

__device__ __forceinline__ float tie_tol(float best) { return 1e-5f * (best + 1e-8f); }
constexpr float kWindow = 12.f;
__device__ __forceinline__ float window_top(float best) { return best + kWindow * tie_tol(best); }

// Beyond this distance from a point whose largest coordinate is pm, a triangle's float distance
// is above best and its tie tolerance.
__device__ __forceinline__ float reach_of(float best, float pm) {
    if (best == kFar) return kFar;
    return sqrtf(best + tie_tol(best)) * 1.00001f + 1e-5f * pm;
}

__device__ __forceinline__ float3 rec_v0(const float4* rec) { return f3(rec[2].x, rec[2].y, rec[2].z); }
__device__ __forceinline__ float3 rec_v1(const float4* rec) { return f3(rec[2].w, rec[3].x, rec[3].y); }
__device__ __forceinline__ float3 rec_v2(const float4* rec) { return f3(rec[3].z, rec[3].w, rec[4].x); }
// The record's normal (0 for some); the triangle's.
__device__ __forceinline__ float3 rec_normal(const float4* rec) { return f3(rec[4].y, rec[4].z, rec[4].w); }
__device__ __forceinline__ float3 tri_normal(const SdfParams& P, const float4* rec, uint32_t f) {
    const float3 n = rec_normal(rec);
    if (n.x != 0.f || n.y != 0.f || n.z != 0.f) return n;
    const float4 u = reinterpret_cast<const float4*>(P.tris)[kTriF4 * (size_t)P.nf + f];
    return f3(u.x, u.y, u.z);
}

// The closest point of a record's triangle to p (xyz) and its squared distance (w). One copy for
// all callers: inlined, the band kernel no longer fits the instruction cache (14 of 28 stall
// cycles an instruction were fetches).
__device__ __noinline__ float4 closest(float3 p, const float4* rec) {
    float3 cp;
    const float d = point_triangle(p, rec_v0(rec), rec_v1(rec), rec_v2(rec), cp);
    return make_float4(cp.x, cp.y, cp.z, d);
}

// A square root from the hardware's approximation, a little below the true one.
__device__ __forceinline__ float sqrt_below(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return __fmul_rn(r, 0.999999f);
}

// Whether the triangle's float distance from p provably exceeds what `reach` was made from:
// by its bounding sphere, then by its plane distance h and the lateral distance beyond the
// sphere (d^2 >= h^2 + (l - R)^2; a normal of 0 leaves the sphere's bound).
__device__ __forceinline__ bool beyond(const float4* rec, float3 p, float pm, float reach) {
    const float4 ts = rec[0];
    const float dx = p.x - ts.x, dy = p.y - ts.y, dz = p.z - ts.z;
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
    const float lim = reach + ts.w;
    if (d2 > __fmul_rn(__fmul_rn(lim, lim), 1.00002f)) return true;
    const float3 n = rec_normal(rec);
    const float reach2 = __fmul_rn(__fmul_rn(reach, reach), 1.00002f);
    const float allow = 2e-5f * (pm + fabsf(ts.x) + fabsf(ts.y) + fabsf(ts.z) + ts.w);
    const float h = __fmaf_rn(dx, n.x, __fmaf_rn(dy, n.y, __fmul_rn(dz, n.z)));
    const float hh = fmaxf(0.f, fabsf(h) - allow);
    const float lat = sqrt_below(fmaxf(0.f, d2 - h * h));
    const float ll = fmaxf(0.f, lat - ts.w - allow);
    return __fmaf_rn(hh, hh, __fmul_rn(ll, ll)) > reach2;
}

// The tie weight of triangle f whose closest point is cp: the doubled area, or the angle at a
// vertex the closest point sits on (from the record).
__device__ __forceinline__ float tie_weight(const SdfParams& P, uint32_t f, const float4* rec, float3 cp, float veps) {
    const float3 c0v = sub(cp, rec_v0(rec)), c1v = sub(cp, rec_v1(rec)), c2v = sub(cp, rec_v2(rec));
    const float* angle = P.tris + 4 * (kTriF4 * (size_t)f + kTriAngles);
    if (dot(c0v, c0v) < veps) return angle[0];
    if (dot(c1v, c1v) < veps) return angle[1];
    if (dot(c2v, c2v) < veps) return angle[2];
    return rec[1].x;
}

// One visit of a triangle at squared distance d: replaces the running minimum, ties with it
// or is ignored, exactly as evaluate_sdf_grid_kernel's loop body. False: ignored.
__device__ __forceinline__ bool visit(BandPoint& q, float d, float w, float3 tn) {
    const float tol = tie_tol(q.best);
    if (d < q.best - tol) {
        q.best = d;
        q.bn = f3(w * tn.x, w * tn.y, w * tn.z);
        return true;
    }
    if (fabsf(d - q.best) <= tol) q.bn = f3(q.bn.x + w * tn.x, q.bn.y + w * tn.y, q.bn.z + w * tn.z);
    return false;
}

// Signed distance of a point from its closest-triangle state; kFar without one and beyond 2.5 bins.
__device__ __forceinline__ float band_value(const SdfParams& P, float3 p, const BandPoint& q) {
    if (q.best == kFar) return kFar;
    float dist = sqrtf(q.best);
    float3 bn = q.bn;
    const float nl = sqrtf(dot(bn, bn));
    if (nl > 1e-12f) bn = f3(bn.x / nl, bn.y / nl, bn.z / nl);
    if (dot(sub(p, q.bp), bn) < 0.0f) dist = -dist;
    return dist > 2.5f * P.min_box || dist < -2.5f * P.min_box ? kFar : dist;
}

// Visiting order of the 27 bins around a bin: the centre, then the shell in z, y, x order.
// Bit t of the result: the t-th of them lies in the triangle's bin range (packed, rec[1].yzw).
__device__ __forceinline__ uint32_t slot_mask(float4 q, int bx, int by, int bz) {
    auto three = [](float packed, int b) {
        const uint32_t u = __float_as_uint(packed);
        const int lo = (int)(u & 0xffffu), hi = (int)(u >> 16);
        return (lo <= b - 1 && b - 1 <= hi ? 1u : 0u) | (lo <= b && b <= hi ? 2u : 0u) | (lo <= b + 1 && b + 1 <= hi ? 4u : 0u);
    };
    const uint32_t mx = three(q.y, bx), my = three(q.z, by), mz = three(q.w, bz);
    const uint32_t plane = (my & 1u ? mx : 0u) | (my & 2u ? mx << 3 : 0u) | (my & 4u ? mx << 6 : 0u);
    const uint32_t m = (mz & 1u ? plane : 0u) | (mz & 2u ? plane << 9 : 0u) | (mz & 4u ? plane << 18 : 0u);
    return ((m >> 13) & 1u) | ((m & 0x1fffu) << 1) | (m & ~0x3fffu);
}

struct BandShared {
    float4 tri[kBandList][kTriList];
    uint32_t idx[kBandList];
    // triangles in the window of the lanes' minima: place in the list (with several lists the
    // triangle) and distance
    uint32_t tie_e[kBandWarps][kBandTies][32];
    float tie_d[kBandWarps][kBandTies][32];
    uint32_t live[kBandWarps][(kBandList + 31) / 32];
    int seq_bin[27];
    uint32_t seq_start[28];
    uint32_t next, n, reach, votes[kBandWarps], brick_next;
    int piece;                     // of the item
    uint32_t redo[kBandBits / 32]; // bricks of the piece for the full walk
    int brick[3];
};

// Entry sq of the bin's visiting sequence: its slot and triangle.
__device__ __forceinline__ uint32_t seq_entry(const SdfParams& P, const BandShared& S, uint32_t sq, int& slot) {
    int b = 0;                                   // last slot with start <= sq
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (b + step < 27 && S.seq_start[b + step] <= sq) b += step;
    slot = b;
    return P.bin_tris[P.bin_start[S.seq_bin[b]] + (sq - S.seq_start[b])];
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Whether a bounding sphere lies farther than `reach` from the box [lo, hi].
__device__ __forceinline__ bool sphere_beyond_box(float4 ts, float3 lo, float3 hi, float reach) {
    const float ex = fmaxf(fmaxf(lo.x - ts.x, ts.x - hi.x), 0.f);
    const float ey = fmaxf(fmaxf(lo.y - ts.y, ts.y - hi.y), 0.f);
    const float ez = fmaxf(fmaxf(lo.z - ts.z, ts.z - hi.z), 0.f);
    const float dd = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
    const float lim = reach + ts.w;
    return dd > __fmul_rn(__fmul_rn(lim, lim), 1.00002f);
}

// Signed distances of the active bins' points.
//
// What the reference computes per point is a walk over the triangles of 27 bins, a triangle
// once per bin that lists it (about five times), with a running minimum and a tie rule. The
// walk's result depends only on the triangles within a few tolerances of the minimum d*: for a
// g >= d* with no distance in (g, g + 1.15 tol], the first triangle at or below g replaces
// whatever the walk holds (it is more than tol below everything visited before), and nothing
// above the gap can tie with or replace what follows. So a warp takes the distinct triangles in
// any order, keeps those within kWindow tolerances of each point's minimum, finds the gap
// and decides on the kept ones alone: the magnitude is the distance of the one visited first (they
// tie), the sign that of its normal's side where all the kept normals agree clearly; else the
// walk is repeated on the kept ones (their slots among the 27 bins, from the record's bin
// range, in visiting order, ascending triangle index inside a slot). Points without a gap
// in the window or with more than kBandTies triangles in it take the full walk (band_serial);
// so does a grid with over 65536 bins an axis.
//
// Bound: instructions (float distances without contraction; 54% issue at 256^3). At 512^3 points
// and 163,840 triangles the full walk for every point took 46.1 ms, this takes 11.3 ms; 256^3
// with the same mesh 19.9 and 6.4 ms, 100^3 with 10,240 triangles 4.2 and 1.2 ms.
__device__ __noinline__ float band_serial(const SdfParams& P, BandShared& S, float3 pt, float pm, bool mine, float3 wlo,
                                          float3 whi, bool wanted, float veps) {
    const uint32_t L = S.seq_start[27];
    const int lane = threadIdx.x & 31;
    BandPoint q;
    q.best = kFar;
    q.bp = f3(0.f, 0.f, 0.f);
    q.bn = f3(0.f, 1.f, 0.f);
    float reach = kFar;
    for (uint32_t c0 = 0; c0 < L; c0 += kBandThreads) {
        const uint32_t m = min((uint32_t)kBandThreads, L - c0);
        __syncthreads();
        if (threadIdx.x < m) {
            int slot;
            const uint32_t f = seq_entry(P, S, c0 + threadIdx.x, slot);
            const float4* rec = reinterpret_cast<const float4*>(P.tris) + kTriF4 * (size_t)f;
#pragma unroll
            for (int part = 0; part < kTriList; ++part) S.tri[threadIdx.x][part] = rec[part];
            S.idx[threadIdx.x] = f;
        }
        __syncthreads();
        if (!wanted) continue;
        for (uint32_t base = 0; base < m; base += 32) {
            const float wr = warp_max(mine ? reach : 0.f);
            const uint32_t e = base + lane;
            const bool cand = e < m && S.tri[e][1].x > 0.f && (wr == kFar || !sphere_beyond_box(S.tri[e][0], wlo, whi, wr));
            uint32_t live = __ballot_sync(0xffffffffu, cand);
            while (live) {
                const uint32_t c = base + __ffs(live) - 1;
                live &= live - 1;
                const float4* rec = S.tri[c];
                if (mine && (reach == kFar || !beyond(rec, pt, pm, reach))) {
                    const float4 r = closest(pt, rec);
                    const float3 cp = f3(r.x, r.y, r.z);
                    if (visit(q, r.w, tie_weight(P, S.idx[c], rec, cp, veps), tri_normal(P, rec, S.idx[c]))) {
                        q.bp = cp;
                        reach = reach_of(r.w, pm);
                    }
                }
                __syncwarp();
            }
        }
    }
    return band_value(P, pt, q);
}

// A kept triangle's record and index (tie_e is a place in the list, or with several lists the
// triangle).
__device__ __forceinline__ const float4* tie_record(const SdfParams& P, const BandShared& S, bool single, uint32_t e) {
    return single ? S.tri[e] : reinterpret_cast<const float4*>(P.tris) + kTriF4 * (size_t)e;
}
__device__ __forceinline__ uint32_t tie_triangle(const BandShared& S, bool single, uint32_t e) { return single ? S.idx[e] : e; }

// The walk on a lane's k kept triangles.
__device__ __noinline__ float band_walk(const SdfParams& P, BandShared& S, bool single, int k, float3 p, int bx, int by, int bz,
                                        float veps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 tn[kBandTies];                                    // ascending triangle: weighted normal, slots
    uint32_t slots = 0;
    for (int t = 0; t < k; ++t) {
        const uint32_t e = S.tie_e[warp][t][lane];
        const float dt = S.tie_d[warp][t][lane];
        const float4* rec = tie_record(P, S, single, e);
        const float4 r = closest(p, rec);
        const uint32_t f = tie_triangle(S, single, e), mask = slot_mask(rec[1], bx, by, bz);
        const float w = tie_weight(P, f, rec, f3(r.x, r.y, r.z), veps);
        const float3 n = tri_normal(P, rec, f);
        slots |= mask;
        int to = t;
        while (to > 0 && tie_triangle(S, single, S.tie_e[warp][to - 1][lane]) > f) {
            S.tie_e[warp][to][lane] = S.tie_e[warp][to - 1][lane];
            S.tie_d[warp][to][lane] = S.tie_d[warp][to - 1][lane];
            tn[to] = tn[to - 1];
            --to;
        }
        S.tie_e[warp][to][lane] = e;
        S.tie_d[warp][to][lane] = dt;
        tn[to] = make_float4(w * n.x, w * n.y, w * n.z, __uint_as_float(mask));
    }
    BandPoint q;
    q.best = kFar;
    q.bn = f3(0.f, 1.f, 0.f);
    int setter = 0;
    while (slots) {
        const uint32_t bit = slots & (0u - slots);
        slots ^= bit;
        for (int t = 0; t < k; ++t)
            if ((__float_as_uint(tn[t].w) & bit) && visit(q, S.tie_d[warp][t][lane], 1.f, f3(tn[t].x, tn[t].y, tn[t].z)))
                setter = t;
    }
    const float4 r = closest(p, tie_record(P, S, single, S.tie_e[warp][setter][lane]));
    q.bp = f3(r.x, r.y, r.z);
    return band_value(P, p, q);
}

// Fills the shared list with the next distinct triangles of the bin's sequence (from entry e0)
// that may lie within `reach` of the box [lo, hi]; returns the entry it stopped at (S.n: how
// many it holds). CTA-wide.
__device__ uint32_t band_fill(const SdfParams& P, BandShared& S, uint32_t e0, int bx, int by, int bz, float3 lo, float3 hi,
                              float reach) {
    const uint32_t L = S.seq_start[27];
    const int lane = threadIdx.x & 31;
    __syncthreads();
    uint32_t have = 0;
    while (e0 < L) {
        const uint32_t sq = e0 + threadIdx.x;
        bool keep = false;
        uint32_t f = 0, mask = 0;
        float4 ts = make_float4(0.f, 0.f, 0.f, 0.f), tq = ts;
        const float4* rec = nullptr;
        if (sq < L) {
            int slot;
            f = seq_entry(P, S, sq, slot);
            rec = reinterpret_cast<const float4*>(P.tris) + kTriF4 * (size_t)f;
            ts = rec[0];
            tq = rec[1];
            mask = slot_mask(tq, bx, by, bz);
            keep = tq.x > 0.f && slot == __ffs(mask) - 1 && !sphere_beyond_box(ts, lo, hi, reach);
        }
        const uint32_t votes = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) S.votes[threadIdx.x >> 5] = __popc(votes);
        __syncthreads();
        uint32_t at = have + __popc(votes & ((1u << lane) - 1u)), all = 0;
#pragma unroll
        for (int w = 0; w < kBandWarps; ++w) {
            if (w < (int)(threadIdx.x >> 5)) at += S.votes[w];
            all += S.votes[w];
        }
        if (have + all > (uint32_t)kBandList) break;     // this stretch starts the next list
        if (keep) {
            S.tri[at][0] = ts;
            S.tri[at][1] = tq;
#pragma unroll
            for (int part = 2; part < kTriList; ++part) S.tri[at][part] = rec[part];
            S.idx[at] = f;
        }
        have += all;
        e0 += kBandThreads;
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x == 0) S.n = have;
    __syncthreads();
    return e0;
}

__global__ void __launch_bounds__(kBandThreads, kBandCtasPerSm) k_band(SdfParams P) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    BandShared& S = *reinterpret_cast<BandShared*>(s_raw);
    const uint32_t nlong = P.item_counts[0], nitems = nlong + P.item_counts[1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float veps = 1e-6f * P.min_box * P.min_box;
    // squared distances beyond far2 make a point far, whatever its ties
    const float far1 = (2.5f * P.min_box) * (2.5f * P.min_box);
    const float far2 = far1 > FLT_MIN && far1 < 1e37f ? far1 * 1.001f + 2.f * kWindow * tie_tol(far1) : kFar;
    const bool packed = P.gx <= kPackedBins && P.gy <= kPackedBins && P.gz <= kPackedBins;
    if (threadIdx.x == 0) S.piece = 0;
    for (;;) {
        // next item from the shared work counter (bins differ a lot in cost: the parts of the long
        // ones come first, the others stand at the end of the list)
        __syncthreads();
        if (threadIdx.x == 0 && S.piece == 0) S.next = atomicAdd(P.work_next, 1u);
        __syncthreads();
        const uint32_t ai = S.next;
        const int piece = S.piece;
        if (ai >= nitems) break;
        const uint2 item = P.items[ai < nlong ? ai : P.items_cap - 1 - (ai - nlong)];
        const long long bin = item.x;
        const int part = (int)(item.y & 0xffu), parts = (int)(item.y >> 8);
        const int bx = (int)(bin % P.gx), by = (int)((bin / P.gx) % P.gy), bz = (int)(bin / ((long long)P.gx * P.gy));
        const int* ys_ = P.axis_start + P.gx + 1;
        const int* zs_ = ys_ + P.gy + 1;
        const int x0 = P.axis_start[bx], y0 = ys_[by], z0 = zs_[bz];
        const int sx = P.axis_start[bx + 1] - x0, sy = ys_[by + 1] - y0, sz = zs_[bz + 1] - z0;
        if (sx <= 0 || sy <= 0 || sz <= 0) continue;
        if (threadIdx.x < 32) {
            // visiting sequence: lane t takes the t-th of the 27 slots, a warp scan gives the starts
            const int t = threadIdx.x;
            int nb = -1;
            if (t == 0) {
                nb = (int)bin;
            } else if (t < 27) {
                const int r = t <= 13 ? t - 1 : t;          // shell slots skip the centre (13)
                const int xx = bx + r % 3 - 1, yy = by + (r / 3) % 3 - 1, zz = bz + r / 9 - 1;
                if (xx >= 0 && xx < P.gx && yy >= 0 && yy < P.gy && zz >= 0 && zz < P.gz)
                    nb = (int)(xx + (long long)P.gx * (yy + (long long)P.gy * zz));
            }
            const uint32_t c = nb >= 0 ? P.bin_count[nb] : 0u;
            uint32_t incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (t >= o) incl += v;
            }
            if (t < 27) { S.seq_bin[t] = nb; S.seq_start[t] = incl - c; }
            if (t == 26) S.seq_start[27] = incl;
            // brick of points per warp, a point a lane: sides of 2 to 4 points that cover the bin
            // in the fewest bricks (8 points an axis: 4x4x2; 9: 3x3x3)
            const int kx = (sx + 1 + t % 3) / (2 + t % 3), ky = (sy + 1 + t / 3 % 3) / (2 + t / 3 % 3),
                      kz = (sz + 1 + t / 9) / (2 + t / 9);
            const int wx = (sx + kx - 1) / kx, wy = (sy + ky - 1) / ky, wz = (sz + kz - 1) / kz;
            const long long count = (long long)kx * ky * kz;
            int cost = t < 27 && wx * wy * wz <= 32 ? 32 * (int)min(count, 0x3fffffdLL) + t : 0x7fffffff;
            const int mine_cost = cost;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cost = min(cost, __shfl_xor_sync(0xffffffffu, cost, o));
            if (mine_cost == cost) { S.brick[0] = wx; S.brick[1] = wy; S.brick[2] = wz; }
            if (t == 0) S.reach = __float_as_uint(kFar);
            if (t < kBandBits / 32) S.redo[t] = 0;
        }
        __syncthreads();
        const uint32_t L = S.seq_start[27];
        const int wx = S.brick[0], wy = S.brick[1], wz = S.brick[2];
        const int nbx = (sx + wx - 1) / wx, nby = (sy + wy - 1) / wy, nbz = (sz + wz - 1) / wz;
        const int nbricks = nbx * nby * nbz;
        const int item_hi = (int)((long long)nbricks * (part + 1) / parts);
        const int brick_lo = (int)((long long)nbricks * part / parts) + piece * kBandPiece, brick_hi = min(item_hi, brick_lo + kBandPiece);
        if (brick_lo >= brick_hi) continue;
        if (threadIdx.x == 0) { S.brick_next = brick_lo; S.piece = brick_hi < item_hi ? piece + 1 : 0; }
        const int zlo = z0 + wz * (brick_lo / (nbx * nby)), zhi = min(z0 + sz, z0 + wz * ((brick_hi - 1) / (nbx * nby) + 1)) - 1;
        // the item's points, and a bound of their distances: to the centroid nearest their middle
        const float3 blo = f3(P.ox + (float)x0 * P.vx, P.oy + (float)y0 * P.vy, P.oz + (float)zlo * P.vz);
        const float3 bhi = f3(P.ox + (float)(x0 + sx - 1) * P.vx, P.oy + (float)(y0 + sy - 1) * P.vy,
                              P.oz + (float)zhi * P.vz);
        const float bpm = fmaxf(fmaxf(fmaxf(fabsf(blo.x), fabsf(bhi.x)), fmaxf(fabsf(blo.y), fabsf(bhi.y))),
                                fmaxf(fabsf(blo.z), fabsf(bhi.z)));
        float reach_bin = reach_of(far2, bpm);
        uint32_t stop = 0;
        bool single = false;
        if (packed) {
            // Only triangles whose float distances are good are asked: not slivers (a2 is 2.6 R^2
            // for an equilateral one) nor tiny ones (barycentrics lose (distance / side)^2 ulps);
            // two radii of slack. Nor beyond 1e9, where the barycentrics' products overflow (a side's
            // and a distance's square: such distances come out too long).
            const float3 mid = f3(0.5f * (blo.x + bhi.x), 0.5f * (blo.y + bhi.y), 0.5f * (blo.z + bhi.z));
            const float small = 0.004f * reach_bin;
            float near = kFar;
#pragma unroll 4
            for (uint32_t sq = threadIdx.x; sq < L; sq += kBandThreads) {
                int slot;
                const uint32_t f = seq_entry(P, S, sq, slot);
                const float4* rec = reinterpret_cast<const float4*>(P.tris) + kTriF4 * (size_t)f;
                const float4 ts = rec[0];
                const float3 e = f3(ts.x - mid.x, ts.y - mid.y, ts.z - mid.z);
                const float d = sqrtf(dot(e, e)) + 2.f * ts.w;
                if (ts.w > small && rec[1].x > 0.26f * ts.w * ts.w) near = fminf(near, d);
            }
            near = warp_min(near);
            if (lane == 0) atomicMin(&S.reach, __float_as_uint(near));     // non-negative floats order as integers
            __syncthreads();
            near = __uint_as_float(S.reach);
            if (near < 1e9f) {
                const float3 hd = sub(bhi, mid);
                const float ub = (near + sqrtf(dot(hd, hd))) * 1.0001f + 1e-5f * bpm;
                const float bound = reach_of(ub * ub * 1.001f + 2.f * kWindow * tie_tol(ub * ub), bpm);
                if (ub < 1e9f) reach_bin = fminf(reach_bin, bound);
            }
            stop = band_fill(P, S, 0, bx, by, bz, blo, bhi, reach_bin);
            single = stop >= L;
        }
        float3 pt;
        float pm, val;
        bool mine;
        long long at;
        float3 wlo, whi;                     // box of this warp's points (lanes without a point add nothing)
        auto take = [&](int brick) {
            const int qx = brick % nbx, qy = (brick / nbx) % nby, qz = brick / (nbx * nby);
            const int lx = wx * qx + lane % wx, ly = wy * qy + (lane / wx) % wy, lz = wz * qz + lane / (wx * wy);
            mine = brick < brick_hi && lane < wx * wy * wz && lx < sx && ly < sy && lz < sz;
            const int ix = x0 + (mine ? lx : 0), iy = y0 + (mine ? ly : 0), iz = z0 + (mine ? lz : 0);
            at = ix + (long long)P.nx * (iy + (long long)P.ny * iz);
            pt = f3(P.ox + (float)ix * P.vx, P.oy + (float)iy * P.vy, P.oz + (float)iz * P.vz);
            pm = fmaxf(fabsf(pt.x), fmaxf(fabsf(pt.y), fabsf(pt.z)));
            val = kFar;
            wlo = f3(warp_min(mine ? pt.x : kFar), warp_min(mine ? pt.y : kFar), warp_min(mine ? pt.z : kFar));
            whi = f3(warp_max(mine ? pt.x : -kFar), warp_max(mine ? pt.y : -kFar), warp_max(mine ? pt.z : -kFar));
        };
        // Minimum and kept triangles of the warp's points over the list in shared memory.
        float best = 0.f, reach = 0.f;
        int m = 0;
        bool serial = false;
        auto start = [&]() {
            serial = false;
            best = far2;
            reach = fminf(reach_of(far2, pm), reach_bin);
            m = 0;
        };
        auto gather = [&](uint32_t n) {
            // a first reach: the triangle whose centroid is nearest the brick's middle
            const float3 mid = f3(0.5f * (wlo.x + whi.x), 0.5f * (wlo.y + whi.y), 0.5f * (wlo.z + whi.z));
            float near = kFar;
            uint32_t seed = 0;
            for (uint32_t e = lane; e < n; e += 32) {
                const float4 ts = S.tri[e][0];
                const float3 v = f3(ts.x - mid.x, ts.y - mid.y, ts.z - mid.z);
                const float d2 = dot(v, v);
                if (d2 < near) { near = d2; seed = e; }
            }
            const float all = warp_min(near);
            const uint32_t who = __ballot_sync(0xffffffffu, near == all);
            seed = __shfl_sync(0xffffffffu, seed, __ffs(who) - 1);
            // Three stages through one loop (one copy of its code): 0, the seed; 1, of what is left
            // against the brick's box the triangle with the centroid nearest each point; 2, what may
            // reach each point, 32 triangles at a time, every lane taking its own, so that
            // lanes work on different triangles at a time.
            uint32_t own = seed, bits = mine ? 1u : 0u, base = seed;
            for (int stage = 0;;) {
                while (__ballot_sync(0xffffffffu, bits != 0u)) {
                    if (bits) {
                        const uint32_t e = base + __ffs(bits) - 1;
                        bits &= bits - 1;
                        const float d = closest(pt, S.tri[e]).w;
                        if (d <= window_top(best)) {
                            if (d < best) {
                                const float top = window_top(d);
                                if (best > top) m = 0;               // all kept ones are out of the window
                                best = d;
                                reach = fminf(reach, reach_of(top, pm));
                            }
                            if (m == kBandTies) {
                                const float top = window_top(best);
                                m = 0;
                                for (int t = 0; t < kBandTies; ++t) {
                                    const float dt = S.tie_d[warp][t][lane];
                                    if (dt > top) continue;
                                    S.tie_d[warp][m][lane] = dt;
                                    S.tie_e[warp][m][lane] = S.tie_e[warp][t][lane];
                                    ++m;
                                }
                            }
                            if (m < kBandTies) {
                                S.tie_d[warp][m][lane] = d;
                                S.tie_e[warp][m][lane] = single ? e : S.idx[e];
                                ++m;
                            } else {
                                serial = true;
                            }
                        }
                    }
                    __syncwarp();
                }
                if (stage == 0) {
                    const float wr = warp_max(mine ? reach : 0.f);
                    float cd = kFar;
                    for (uint32_t b0 = 0; b0 < n; b0 += 32) {
                        const uint32_t e = b0 + lane;
                        const bool cand = e < n && e != seed && !sphere_beyond_box(S.tri[e][0], wlo, whi, wr);
                        uint32_t live = __ballot_sync(0xffffffffu, cand);
                        if (lane == 0) S.live[warp][b0 >> 5] = live;
                        while (live) {
                            const uint32_t c = b0 + __ffs(live) - 1;
                            live &= live - 1;
                            const float4 ts = S.tri[c][0];
                            const float dx = pt.x - ts.x, dy = pt.y - ts.y, dz = pt.z - ts.z;
                            const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
                            if (d2 < cd) { cd = d2; own = c; }
                        }
                    }
                    __syncwarp();
                    base = own;
                    bits = mine && own != seed ? 1u : 0u;
                    stage = 1;
                } else {
                    base = stage == 1 ? 0u : base + 32u;
                    stage = 2;
                    if (base >= n) break;
                    bits = 0;
                    uint32_t live = S.live[warp][base >> 5];
                    while (live) {
                        const int b = __ffs(live) - 1;
                        live &= live - 1;
                        if (!beyond(S.tri[base + b], pt, pm, reach)) bits |= 1u << b;
                    }
                    if (!mine) bits = 0;
                    if (own - base < 32u) bits &= ~(1u << (own - base));
                }
            }
            __syncwarp();
        };
        // The value from the kept triangles; sets serial where the window does not decide.
        auto decide = [&]() {
            if (!mine || !(best < far2) || serial) return;
            const float top = window_top(best), gap = 1.15f * tie_tol(top);
            float g = best;
            for (;;) {
                float next = kFar;
                for (int t = 0; t < m; ++t) {
                    const float dt = S.tie_d[warp][t][lane];
                    if (dt > g) next = fminf(next, dt);
                }
                if (next - g > gap) break;
                g = next;
            }
            if (g + gap > top) { serial = true; return; }
            int k = 0;
            for (int t = 0; t < m; ++t) {                      // those at or below g
                const float dt = S.tie_d[warp][t][lane];
                if (dt > g) continue;
                S.tie_d[warp][k][lane] = dt;
                S.tie_e[warp][k][lane] = S.tie_e[warp][t][lane];
                ++k;
            }
            // the first one visited: by slot, then triangle
            int first = 0;
            if (k > 1) {
                uint32_t slot1 = 33, tri1 = 0;
                for (int t = 0; t < k; ++t) {
                    const uint32_t e = S.tie_e[warp][t][lane];
                    const uint32_t slot = __ffs(slot_mask(tie_record(P, S, single, e)[1], bx, by, bz));
                    const uint32_t tri = tie_triangle(S, single, e);
                    if (slot < slot1 || (slot == slot1 && tri < tri1)) { slot1 = slot; tri1 = tri; first = t; }
                }
            }
            BandPoint q;
            q.best = S.tie_d[warp][first][lane];
            const float4 r = closest(pt, tie_record(P, S, single, S.tie_e[warp][first][lane]));
            q.bp = f3(r.x, r.y, r.z);
            // all tie with the first, and all normals on one side by 1e-3 of the distance: every
            // sum of them with positive weights lies on that side (a normal of 0 is on neither)
            const float3 v = sub(pt, q.bp);
            const float vv = dot(v, v), clear = vv > 1e-30f ? 1e-3f * sqrtf(vv) : kFar;
            bool above = true, below = true;
            for (int t = 0; t < k; ++t) {
                const float side = dot(v, rec_normal(tie_record(P, S, single, S.tie_e[warp][t][lane])));
                above = above && side > clear;
                below = below && side < -clear;
            }
            if ((above || below) && g - best <= 0.99f * tie_tol(best)) {
                q.bn = above ? v : f3(-v.x, -v.y, -v.z);
                val = band_value(P, pt, q);
            } else {
                val = band_walk(P, S, single, k, pt, bx, by, bz, veps);
            }
        };
        auto finish = [&](int brick) {
            if (__ballot_sync(0xffffffffu, serial) && lane == 0 && brick < brick_hi)
                atomicOr(&S.redo[(brick & (kBandBits - 1)) >> 5], 1u << (brick & 31));
            if (mine) P.out[at] = val;
        };
        // With one list the warps take bricks as they come; with several they go through the
        // lists together.
        for (int brick = brick_lo + warp;;) {
            if (single) {
                if (lane == 0) brick = (int)atomicAdd(&S.brick_next, 1u);
                brick = __shfl_sync(0xffffffffu, brick, 0);
            }
            if ((single ? brick : brick - warp) >= brick_hi) break;
            take(brick);
            start();
            if (packed) {
                for (uint32_t e0 = single ? stop : 0u;;) {
                    if (!single) e0 = band_fill(P, S, e0, bx, by, bz, blo, bhi, reach_bin);
                    if (brick < brick_hi && S.n) gather(S.n);
                    if (e0 >= L) break;
                }
                __syncwarp();
                decide();
                __syncwarp();
            } else {
                serial = true;
            }
            finish(brick);
            if (!single) brick += kBandWarps;
        }
        __syncthreads();
        if (S.redo[0] | S.redo[1] | S.redo[2] | S.redo[3]) {
            for (int brick0 = brick_lo / kBandWarps * kBandWarps; brick0 < brick_hi; brick0 += kBandWarps) {
                const uint32_t flags = (S.redo[(brick0 & (kBandBits - 1)) >> 5] >> (brick0 & 31)) & ((1u << kBandWarps) - 1u);
                if (!flags) continue;
                const bool want = (flags >> warp) & 1u;
                take(brick0 + warp);
                val = band_serial(P, S, pt, pm, mine, wlo, whi, want, veps);
                if (want && mine) P.out[at] = val;
            }
        }
    }
}

// Far / positive bit words, warp per 32-word stretch of one x row.
__global__ void __launch_bounds__(256) k_sdf_masks(SdfParams P) {
    const int lane = threadIdx.x & 31;
    const long long rows = (long long)P.ny * P.nz;
    const long long per_row = (P.W + 31) / 32;
    const long long groups = rows * per_row;
    for (long long gq = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; gq < groups;
         gq += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long row = gq / per_row;
        const int w0 = (int)(gq % per_row) * 32;
        const int j = (int)(row % P.ny), k = (int)(row / P.ny);
        const bool border_row = j == 0 || j == P.ny - 1 || k == 0 || k == P.nz - 1;
        const float* src = P.out + row * P.nx;
        uint32_t my_far = 0, my_ext = 0;
        for (int q = 0; q < 32 && w0 + q < P.W; ++q) {
            const int x = 32 * (w0 + q) + lane;
            const float v = x < P.nx ? src[x] : 0.f;
            const bool far = x < P.nx && v == kFar;
            const bool pos = x < P.nx && v != kFar && v > 0.0f;
            const bool border = x < P.nx && (border_row || x == 0 || x == P.nx - 1);
            const uint32_t bf = __ballot_sync(0xffffffffu, far);
            const uint32_t be = __ballot_sync(0xffffffffu, pos || (far && border));
            if (lane == q) { my_far = bf; my_ext = be; }
        }
        if (w0 + lane < P.W) {
            P.far[row * P.W + w0 + lane] = my_far;
            P.ext[row * P.W + w0 + lane] = my_ext;
        }
    }
}

// Exterior flood on bit words. Tile = kFX words x kFY rows x kFZ planes; the neighbouring
// tiles' words are read once per launch as fixed sources; the tile iterates to its local
// fixpoint. ext <- ext | (far & (ext shifted by one point along x, y or z)). Bits only ever
// get set, so reading a word another thread is updating in the same sweep is harmless.
constexpr int kFX = 4, kFY = 16, kFZ = 16;
constexpr int kFloodThreads = 256;
constexpr int kFloodLocalCap = 4 * (32 * kFX + kFY + kFZ);   // local sweeps before yielding
__global__ void __launch_bounds__(kFloodThreads) k_flood(SdfParams P, int* changed) {
    __shared__ uint32_t s_ext[kFZ + 2][kFY + 2][kFX + 2];
    __shared__ uint32_t s_far[kFZ][kFY][kFX];
    __shared__ int s_any, s_tile_changed;
    const long long tx = (P.W + kFX - 1) / kFX, ty = (P.ny + kFY - 1) / kFY, tz = (P.nz + kFZ - 1) / kFZ;
    for (long long tile = blockIdx.x; tile < tx * ty * tz; tile += gridDim.x) {
        const int wx0 = (int)(tile % tx) * kFX, y0 = (int)((tile / tx) % ty) * kFY, z0 = (int)(tile / (tx * ty)) * kFZ;
        __syncthreads();
        if (threadIdx.x == 0) { s_any = 0; s_tile_changed = 0; }
        __syncthreads();
        for (int e = threadIdx.x; e < (kFZ + 2) * (kFY + 2) * (kFX + 2); e += kFloodThreads) {
            const int lx = e % (kFX + 2), ly = (e / (kFX + 2)) % (kFY + 2), lz = e / ((kFX + 2) * (kFY + 2));
            const int w = wx0 + lx - 1, y = y0 + ly - 1, z = z0 + lz - 1;
            uint32_t v = 0;
            if (w >= 0 && w < P.W && y >= 0 && y < P.ny && z >= 0 && z < P.nz) v = P.ext[((long long)z * P.ny + y) * P.W + w];
            s_ext[lz][ly][lx] = v;
            if (lx >= 1 && lx <= kFX && ly >= 1 && ly <= kFY && lz >= 1 && lz <= kFZ) {
                const uint32_t f = (w < P.W && y < P.ny && z < P.nz) ? P.far[((long long)z * P.ny + y) * P.W + w] : 0u;
                s_far[lz - 1][ly - 1][lx - 1] = f;
                if (f & ~v) s_any = 1;   // unreached far points here
            }
        }
        __syncthreads();
        if (!s_any) continue;
        for (int it = 0; it < kFloodLocalCap; ++it) {
            int mine = 0;
            for (int e = threadIdx.x; e < kFZ * kFY * kFX; e += kFloodThreads) {
                const int lx = e % kFX + 1, ly = (e / kFX) % kFY + 1, lz = e / (kFX * kFY) + 1;
                const uint32_t cur = s_ext[lz][ly][lx];
                const uint32_t far = s_far[lz - 1][ly - 1][lx - 1];
                const uint32_t nb = (cur << 1) | (cur >> 1) | (s_ext[lz][ly][lx - 1] >> 31) | (s_ext[lz][ly][lx + 1] << 31) |
                                    s_ext[lz][ly - 1][lx] | s_ext[lz][ly + 1][lx] | s_ext[lz - 1][ly][lx] | s_ext[lz + 1][ly][lx];
                // along x the flood runs through the word's far points at once (both ways, doubling
                // steps); y and z take a sweep a point
                uint32_t nxt = cur | (far & nb);
                uint32_t pass = far;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { nxt |= pass & (nxt << o); pass &= pass << o; }
                pass = far;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { nxt |= pass & (nxt >> o); pass &= pass >> o; }
                if (nxt != cur) { s_ext[lz][ly][lx] = nxt; mine = 1; }
            }
            const int any = __syncthreads_or(mine);
            if (!any) break;
            if (threadIdx.x == 0) s_tile_changed = 1;
        }
        __syncthreads();
        if (s_tile_changed) {
            for (int e = threadIdx.x; e < kFZ * kFY * kFX; e += kFloodThreads) {
                const int lx = e % kFX, ly = (e / kFX) % kFY, lz = e / (kFX * kFY);
                const int w = wx0 + lx, y = y0 + ly, z = z0 + lz;
                if (w < P.W && y < P.ny && z < P.nz) P.ext[((long long)z * P.ny + y) * P.W + w] = s_ext[lz + 1][ly + 1][lx + 1];
            }
            if (threadIdx.x == 0) atomicExch(changed, 1);
        }
    }
}

// A block's sum of `v`, added to *total by one atomic (an atomic per thread on one address kept
// the finishing pass at 0.9 ms for 512^3).
__device__ __forceinline__ void add_block_sum(uint32_t v, unsigned long long* total) {
    __shared__ uint32_t s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_sum, v);
    __syncthreads();
    if (threadIdx.x == 0 && s_sum) atomicAdd(total, (unsigned long long)s_sum);
}

// Far points -> +10 (exterior) or -10, then four Jacobi passes of the relaxation
// (eikonal_relaxation_kernel) in one sweep over the grid, from the band's values in `in` to P.out.
//
// 512^3: 1.57 ms; as five passes over the grid these took 3.2 ms (floor: a read and a write of
// the grid, 164 us). Bound: instructions and the step synchronisation.
// A block owns 56 x 24 columns and marches along z:
// a warp holds two rows of 64 points, lane l the points 2l and 2l+1, and every lane the last two
// planes of its points after 0..3 passes. When plane t arrives, pass s is due on plane t - s:
// its z neighbours are the lane's own, x neighbours come by shuffle, y neighbours from shared
// memory, where every pass leaves its plane one step ahead (two buffers, one synchronisation a
// step). The four columns around the owned ones are worked on redundantly (a point fewer is
// right after every pass). Points outside the grid are +infinity throughout: no neighbour.
constexpr int kRelaxPasses = 4;
constexpr int kRelaxThreads = 512, kRelaxRows = 2;
constexpr int kRelaxW = 64, kRelaxH = kRelaxThreads / 32 * kRelaxRows;          // columns a block works on
constexpr int kRelaxOwnW = kRelaxW - 2 * kRelaxPasses, kRelaxOwnH = kRelaxH - 2 * kRelaxPasses;
struct RelaxShared { float2 plane[kRelaxPasses][2][kRelaxH][32]; };

__device__ __forceinline__ float relaxed(float val, float keep, float x0, float x1, float y0, float y1, float z0, float z1,
                                         const SdfParams& P) {
    if (fabsf(val) <= keep) return val;
    float a = fabsf(val);
    a = fminf(a, fminf(fabsf(x0), fabsf(x1)) + P.vx);       // rounding is monotone: one sum per axis
    a = fminf(a, fminf(fabsf(y0), fabsf(y1)) + P.vy);
    a = fminf(a, fminf(fabsf(z0), fabsf(z1)) + P.vz);
    return copysignf(a, val);                               // val is not zero here
}

__global__ void __launch_bounds__(kRelaxThreads, 2)
k_sdf_relax(const __grid_constant__ SdfParams P, const float* __restrict__ in, int depth, unsigned long long* filled) {
    extern __shared__ __align__(16) unsigned char s_relax[];
    RelaxShared& S = *reinterpret_cast<RelaxShared*>(s_relax);
    const float inf = __int_as_float(0x7f800000);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int ntx = (P.nx + kRelaxOwnW - 1) / kRelaxOwnW;          // x tiles fastest, then y
    const int x = (int)(blockIdx.x % ntx) * kRelaxOwnW - kRelaxPasses + 2 * lane;
    const int y0 = (int)(blockIdx.x / ntx) * kRelaxOwnH - kRelaxPasses + warp * kRelaxRows;
    const int zlo = (int)blockIdx.y * depth, zhi = min(P.nz, zlo + depth);
    const float keep = fminf(P.vx, fminf(P.vy, P.vz)) * 1.5f;
    const bool inx[2] = {x >= 0 && x < P.nx, x + 1 >= 0 && x + 1 < P.nx};
    const bool ownx = lane >= kRelaxPasses / 2 && lane < 32 - kRelaxPasses / 2;
    uint32_t cnt = 0;
    auto fetch = [&](int z, float2 (&v)[kRelaxRows]) {
#pragma unroll
        for (int r = 0; r < kRelaxRows; ++r) {
            const int y = y0 + r;
            v[r] = make_float2(inf, inf);
            if (z < 0 || z >= P.nz || y < 0 || y >= P.ny) continue;
            const float* src = in + ((long long)z * P.ny + y) * P.nx + x;
            if (inx[0]) v[r].x = __ldg(src);
            if (inx[1]) v[r].y = __ldg(src + 1);
        }
    };
    float2 two[kRelaxPasses][kRelaxRows], one[kRelaxPasses][kRelaxRows];       // after s passes: the plane before last, the last
#pragma unroll
    for (int s = 0; s < kRelaxPasses; ++s)
#pragma unroll
        for (int r = 0; r < kRelaxRows; ++r) two[s][r] = one[s][r] = make_float2(inf, inf);
    float2 ahead[kRelaxRows];
    fetch(zlo - kRelaxPasses, ahead);
    for (int t = zlo - kRelaxPasses; t < zhi + kRelaxPasses; ++t) {
        float2 cur[kRelaxRows];
#pragma unroll
        for (int r = 0; r < kRelaxRows; ++r) {
            cur[r] = ahead[r];
            float* const c[2] = {&cur[r].x, &cur[r].y};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (*c[u] != kFar) continue;
                const uint32_t e = __ldg(P.ext + ((long long)t * P.ny + y0 + r) * P.W + ((x + u) >> 5));
                const bool ex = (e >> ((x + u) & 31)) & 1u;
                *c[u] = ex ? 10.0f : -10.0f;
                const int ly = warp * kRelaxRows + r;
                if (ex && ownx && ly >= kRelaxPasses && ly < kRelaxH - kRelaxPasses && t >= zlo && t < zhi) ++cnt;
            }
        }
        if (t + 1 < zhi + kRelaxPasses) fetch(t + 1, ahead);
        const int now = t & 1, before = now ^ 1;
#pragma unroll
        for (int s = 0; s < kRelaxPasses; ++s) {
            // cur: plane t - s after s passes; its pass s + 1 is due on the plane before it
            const bool inz = t - s - 1 >= 0 && t - s - 1 < P.nz;
            float2 next[kRelaxRows];
#pragma unroll
            for (int r = 0; r < kRelaxRows; ++r) {
                const int ly = warp * kRelaxRows + r, y = y0 + r;
                const float2 v = one[s][r];
                const float2 up = r > 0 ? one[s][r - 1] : S.plane[s][before][max(ly - 1, 0)][lane];
                const float2 dn = r + 1 < kRelaxRows ? one[s][r + 1] : S.plane[s][before][min(ly + 1, kRelaxH - 1)][lane];
                const float left = __shfl_up_sync(0xffffffffu, v.y, 1), right = __shfl_down_sync(0xffffffffu, v.x, 1);
                const bool iny = inz && y >= 0 && y < P.ny;
                next[r].x = iny && inx[0] ? relaxed(v.x, keep, left, v.y, up.x, dn.x, two[s][r].x, cur[r].x, P) : inf;
                next[r].y = iny && inx[1] ? relaxed(v.y, keep, v.x, right, up.y, dn.y, two[s][r].y, cur[r].y, P) : inf;
            }
#pragma unroll
            for (int r = 0; r < kRelaxRows; ++r) {
                S.plane[s][now][warp * kRelaxRows + r][lane] = cur[r];
                two[s][r] = one[s][r];
                one[s][r] = cur[r];
                cur[r] = next[r];
            }
        }
        const int z = t - kRelaxPasses;
        if (z >= zlo && ownx) {
#pragma unroll
            for (int r = 0; r < kRelaxRows; ++r) {
                const int ly = warp * kRelaxRows + r, y = y0 + r;
                if (ly < kRelaxPasses || ly >= kRelaxH - kRelaxPasses || y >= P.ny) continue;
                float* dst = P.out + ((long long)z * P.ny + y) * P.nx + x;
                if (inx[0]) dst[0] = cur[r].x;
                if (inx[1]) dst[1] = cur[r].y;
            }
        }
        __syncthreads();
    }
    add_block_sum(cnt, filled);
}

// ---- voxelize-first (compute_mesh_sdf_device_cuda with voxelize_first, :764-832) -------------

// A warp per triangle: every voxel corner of the triangle's voxel box whose squared distance
// to the triangle is within (0.866 * largest voxel side)^2 joins the shell (:458-501). (10,240
// triangles on 256^3 voxels: 253 us with a thread per triangle, 320 warps on the whole GPU.)
__global__ void __launch_bounds__(256) k_vox_raster(SdfParams P) {
    const int vr = P.vres, lane = threadIdx.x & 31;
    const float mvd = fmaxf(P.vox_vx, fmaxf(P.vox_vy, P.vox_vz)) * 0.8660254f;
    const float lim = mvd * mvd;
    for (long long f = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; f < P.nf;
         f += ((long long)gridDim.x * blockDim.x) >> 5) {
        float3 a, b, c;
        if (!load_tri(P, f, a, b, c)) continue;
        const float mnx = fminf(a.x, fminf(b.x, c.x)), mny = fminf(a.y, fminf(b.y, c.y)), mnz = fminf(a.z, fminf(b.z, c.z));
        const float mxx = fmaxf(a.x, fmaxf(b.x, c.x)), mxy = fmaxf(a.y, fmaxf(b.y, c.y)), mxz = fmaxf(a.z, fmaxf(b.z, c.z));
        const int bx0 = bin_coord(mnx, P.ox, P.vox_vx, vr), sx = bin_coord(mxx, P.ox, P.vox_vx, vr) - bx0 + 1;
        const int by0 = bin_coord(mny, P.oy, P.vox_vy, vr), sy = bin_coord(mxy, P.oy, P.vox_vy, vr) - by0 + 1;
        const int bz0 = bin_coord(mnz, P.oz, P.vox_vz, vr), sz = bin_coord(mxz, P.oz, P.vox_vz, vr) - bz0 + 1;
        if (sx <= 0 || sy <= 0 || sz <= 0) continue;
        const long long nvox = (long long)sx * sy * sz;
        for (long long w = lane; w < nvox; w += 32) {
            const int row = (int)(w / sx);
            const int bx = bx0 + (int)(w - (long long)row * sx), by = by0 + row % sy, bz = bz0 + row / sy;
            const float3 q = f3(P.ox + (float)bx * P.vox_vx, P.oy + (float)by * P.vox_vy, P.oz + (float)bz * P.vox_vz);
            float3 closest;
            if (point_triangle(q, a, b, c, closest) <= lim)
                atomicOr(P.vshell + ((long long)bz * vr + by) * P.Wv + (bx >> 5), 1u << (bx & 31));
        }
    }
}

// The shell dilated by one voxel (27-neighbourhood, :503-526), then the flood's inputs: the
// voxels outside the dilated shell pass the exterior flood, and those of them on the border
// seed it (init_voxel_exterior_kernel, :561-575). A thread per 32-voxel word.
__global__ void __launch_bounds__(256) k_vox_dilate(SdfParams P) {
    const int vr = P.vres;
    const long long words = (long long)vr * vr * P.Wv;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < words;
         idx += (long long)gridDim.x * blockDim.x) {
        const int w = (int)(idx % P.Wv);
        const long long row = idx / P.Wv;
        const int y = (int)(row % vr), z = (int)(row / vr);
        uint32_t dil = 0;
        for (int zz = max(0, z - 1); zz <= min(vr - 1, z + 1); ++zz)
            for (int yy = max(0, y - 1); yy <= min(vr - 1, y + 1); ++yy) {
                const uint32_t* src = P.vshell + ((long long)zz * vr + yy) * P.Wv;
                const uint32_t cur = src[w];
                const uint32_t prev = w > 0 ? src[w - 1] : 0u, next = w + 1 < P.Wv ? src[w + 1] : 0u;
                dil |= cur | (cur << 1) | (cur >> 1) | (prev >> 31) | (next << 31);
            }
        const int valid_bits = min(32, vr - 32 * w);
        const uint32_t valid = valid_bits >= 32 ? 0xffffffffu : ((1u << valid_bits) - 1u);
        const uint32_t pass = ~dil & valid;
        uint32_t border;
        if (y == 0 || y == vr - 1 || z == 0 || z == vr - 1) {
            border = valid;
        } else {
            border = 0;
            if (w == 0) border |= 1u;
            if ((vr - 1) >> 5 == w) border |= 1u << ((vr - 1) & 31);
        }
        P.vfar[idx] = pass;
        P.vext[idx] = pass & border;
    }
}

// Far grid points -> -10 inside the solid voxels (not exterior), +10 elsewhere
// (apply_solid_voxel_sign_mask_kernel, :660-690); block per x row.
__global__ void __launch_bounds__(256) k_vox_sign(SdfParams P, unsigned long long* filled) {
    const long long rows = (long long)P.ny * P.nz;
    const int vr = P.vres;
    uint32_t cnt = 0;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        const int iy = (int)(row % P.ny), iz = (int)(row / P.ny);
        float* r = P.out + row * P.nx;
        const float py = P.oy + (float)iy * P.vy, pz = P.oz + (float)iz * P.vz;
        const int vby = bin_coord(py, P.oy, P.vox_vy, vr), vbz = bin_coord(pz, P.oz, P.vox_vz, vr);
        const uint32_t* e = P.vext + ((long long)vbz * vr + vby) * P.Wv;
        for (int ix = threadIdx.x; ix < P.nx; ix += blockDim.x) {
            if (r[ix] != kFar) continue;
            const int vbx = bin_coord(P.ox + (float)ix * P.vx, P.ox, P.vox_vx, vr);
            const bool exterior = (e[vbx >> 5] >> (vbx & 31)) & 1u;
            r[ix] = exterior ? 10.0f : -10.0f;
            cnt += exterior ? 1 : 0;
        }
    }
    add_block_sum(cnt, filled);
}

unsigned grid_for(long long items, int per_block, int num_sms, int per_sm) {
    long long b = (items + per_block - 1) / per_block;
    const long long cap = (long long)num_sms * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

}  // namespace

size_t sdf_tri_record_bytes() { return sizeof(Tri) + sizeof(float4); }

// Bound of the band kernel's work items: the bins' 27-bin entry counts sum to at most 27 * entries.
long long sdf_items_capacity(long long nbins, unsigned long long entries) {
    return nbins + (long long)(27 * entries / kPartEntries) + 1;
}

void sdf_bin_geometry(SdfParams& P) {
    P.gx = std::max(1, P.nx / 8);
    P.gy = std::max(1, P.ny / 8);
    P.gz = std::max(1, P.nz / 8);
    P.bdx = ((float)P.nx * P.vx) / (float)P.gx;
    P.bdy = ((float)P.ny * P.vy) / (float)P.gy;
    P.bdz = ((float)P.nz * P.vz) / (float)P.gz;
    P.margin = 2.0f * std::max(P.vx, std::max(P.vy, P.vz));
    P.min_box = std::min(P.bdx, std::min(P.bdy, P.bdz));
    P.nbins = (long long)P.gx * P.gy * P.gz;
    P.W = (P.nx + 31) / 32;
}

cudaError_t launch_sdf_prep(const SdfParams& P, int num_sms, cudaStream_t s) {
    if (P.nf <= 0) return cudaSuccess;
    k_tri_prep<<<grid_for(P.nf, 256, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sdf_bins(const SdfParams& P, int num_sms, cudaStream_t s) {
    const int na = P.gx + P.gy + P.gz + 3;
    k_axis_starts<<<(na + 127) / 128, 128, 0, s>>>(P);
    k_fill_far<<<grid_for((long long)P.nx * P.ny * P.nz, 256, num_sms, 16), 256, 0, s>>>(P);
    if (P.nf > 0) k_tri_bins<<<grid_for(P.nf, 256, num_sms, 16), 256, 0, s>>>(P);
    k_bin_order<<<grid_for(P.nbins, 1, num_sms, 64), kOrderThreads, 0, s>>>(P);
    k_bin_active<<<grid_for(P.nbins, 256, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sdf_band(const SdfParams& P, int num_sms, cudaStream_t s) {
    // persistent: every CTA that fits on the GPU at once takes bins from the work counter
    cudaError_t e = cudaFuncSetAttribute(k_band, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BandShared));
    if (e != cudaSuccess) return e;
    k_band<<<grid_for(P.items_cap, 1, num_sms, kBandCtasPerSm), kBandThreads, sizeof(BandShared), s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sdf_masks(const SdfParams& P, int num_sms, cudaStream_t s) {
    const long long groups = (long long)P.ny * P.nz * ((P.W + 31) / 32);
    k_sdf_masks<<<grid_for(groups * 32, 256, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_sdf_flood(const SdfParams& P, int* changed, int num_sms, cudaStream_t s) {
    const long long tiles = ((P.W + kFX - 1) / kFX) * (long long)((P.ny + kFY - 1) / kFY) * ((P.nz + kFZ - 1) / kFZ);
    k_flood<<<grid_for(tiles, 1, num_sms, 8), kFloodThreads, 0, s>>>(P, changed);
    return cudaGetLastError();
}

cudaError_t launch_sdf_finish(const SdfParams& P, const float* band, unsigned long long* filled, int num_sms, cudaStream_t s) {
    const long long tiles = (long long)((P.nx + kRelaxOwnW - 1) / kRelaxOwnW) * ((P.ny + kRelaxOwnH - 1) / kRelaxOwnH);
    // planes a block owns: its eight extra ones are an eighth of 64; fewer planes where 64 leave
    // the GPU without two blocks an SM
    int depth = tiles * ((P.nz + 63) / 64) >= 2LL * num_sms ? 64 : 16;
    while ((P.nz + depth - 1) / depth > 65535) depth *= 2;
    cudaError_t e = cudaFuncSetAttribute(k_sdf_relax, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RelaxShared));
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)tiles, (unsigned)((P.nz + depth - 1) / depth));     // 65,535 at most in y
    k_sdf_relax<<<grid, kRelaxThreads, sizeof(RelaxShared), s>>>(P, band, depth, filled);
    return cudaGetLastError();
}

cudaError_t launch_vox_raster(const SdfParams& P, int num_sms, cudaStream_t s) {
    if (P.nf <= 0) return cudaSuccess;
    k_vox_raster<<<grid_for(P.nf, 8, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_vox_dilate(const SdfParams& P, int num_sms, cudaStream_t s) {
    k_vox_dilate<<<grid_for((long long)P.vres * P.vres * P.Wv, 256, num_sms, 16), 256, 0, s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_vox_flood(const SdfParams& P, int* changed, int num_sms, cudaStream_t s) {
    SdfParams V = P;
    V.W = P.Wv;
    V.nx = P.vres; V.ny = P.vres; V.nz = P.vres;
    V.far = P.vfar;
    V.ext = P.vext;
    return launch_sdf_flood(V, changed, num_sms, s);
}

cudaError_t launch_vox_sign(const SdfParams& P, unsigned long long* filled, int num_sms, cudaStream_t s) {
    const long long rows = (long long)P.ny * P.nz;
    k_vox_sign<<<grid_for(rows, 1, num_sms, 8), 256, 0, s>>>(P, filled);
    return cudaGetLastError();
}

}  // namespace dcb
