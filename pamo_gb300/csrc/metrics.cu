// Evaluation kernels of the reference's metrics module (simp_cuda/safe_project/src/pamo_safe_project/
// metrics.py:7-107): squared distances from points to a triangle mesh (the closest-point queries behind its
// Chamfer and Hausdorff distances) and the per-face minimum angles behind compute_min_angle and
// compute_bad_tri_ratio. Off the simplification path; inputs are float64 like the metrics' NumPy arrays.
//
// Point-to-mesh distance: two walks per point through the packed stage-2 LBVH over float copies of the vertices. The
// first, all in float, gives an upper bound of the distance; the second collects the triangles that may be as near, and
// those few take the exact float64 point-triangle distance (Ericson, Real-Time Collision Detection, 5.1.5), the lanes
// of a warp together. The nearest triangle and the smallest index of equally near ones are the same as by trying every
// triangle in float64; the margins below hold what float adds.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../include/pamo_gb300.h"
#include "lbvh.cuh"
#include "pamo_common.cuh"
#include "scan.cuh"

namespace {

using namespace pamo;

constexpr int kT = 256;
constexpr int kQT = 64;
constexpr int kStack = 64;
constexpr int kList = 8;  // triangles a lane collects before the warp evaluates them

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 dsub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 dadd(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 dmul(double s, D3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double ddot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 dload(const double* v, int i) { return {v[3 * i], v[3 * i + 1], v[3 * i + 2]}; }

// closest point of triangle abc to p (region tests on the barycentric parameters)
__device__ D3 closest_point_triangle(D3 p, D3 a, D3 b, D3 c) {
    const D3 ab = dsub(b, a), ac = dsub(c, a), ap = dsub(p, a);
    const double d1 = ddot(ab, ap), d2 = ddot(ac, ap);
    if (d1 <= 0.0 && d2 <= 0.0) return a;
    const D3 bp = dsub(p, b);
    const double d3 = ddot(ab, bp), d4 = ddot(ac, bp);
    if (d3 >= 0.0 && d4 <= d3) return b;
    const double vc = d1 * d4 - d3 * d2;
    if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) return dadd(a, dmul(d1 / (d1 - d3), ab));
    const D3 cp = dsub(p, c);
    const double d5 = ddot(ab, cp), d6 = ddot(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) return c;
    const double vb = d5 * d2 - d1 * d6;
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) return dadd(a, dmul(d2 / (d2 - d6), ac));
    const double va = d3 * d6 - d5 * d4;
    if (va <= 0.0 && (d4 - d3) >= 0.0 && (d5 - d6) >= 0.0)
        return dadd(b, dmul((d4 - d3) / ((d4 - d3) + (d5 - d6)), dsub(c, b)));
    const double den = 1.0 / (va + vb + vc);
    return dadd(a, dadd(dmul(vb * den, ab), dmul(vc * den, ac)));
}

__global__ void k_to_float4(const double* __restrict__ v, int n, float4* out) {
    pdl_wait();
    for (int i = gtid(); i < n; i += gstride())
        out[i] = make_float4((float)v[3 * i], (float)v[3 * i + 1], (float)v[3 * i + 2], 0.f);
}

__global__ void k_to_int4(const int* __restrict__ f, int n, int nv, int4* out, int* status) {
    pdl_wait();
    for (int i = gtid(); i < n; i += gstride()) {
        const int a = f[3 * i], b = f[3 * i + 1], c = f[3 * i + 2];
        if (a < 0 || b < 0 || c < 0 || a >= nv || b >= nv || c >= nv) {
            atomicOr(status, kErrBadIndex);
            out[i] = make_int4(0, 0, 0, 0);
        } else {
            out[i] = make_int4(a, b, c, 0);
        }
    }
}

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 fsub(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float fdot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 f3(float4 v) { return {v.x, v.y, v.z}; }

__device__ __forceinline__ float unit(float x) { return fminf(fmaxf(x, 0.f), 1.f); }  // a NaN counts as 0

// Distance in float from p to the triangle, and its scale: the largest of |ab|, |ac| and the distance. The point that it
// is taken to lies in the triangle whatever the rounding did (the parameters are clamped), so the distance is an upper
// bound of the true one up to the rounding of that point. slim: it is no lower bound to rely on. The parameters come from
// differences of products of size (side * scale)^2, rounded to about 1e-6 of that and divided by n2 = |ab x ac|^2, so the
// point is off by up to 1e-6 side^3 scale^2 / n2, within kLower * scale (with a factor of 4) if side^3 scale <= 25 n2.
__device__ __forceinline__ float tri_distance(F3 p, F3 a, F3 b, F3 c, float& scale, bool& slim) {
    const F3 ab = fsub(b, a), ac = fsub(c, a), ap = fsub(p, a);
    const float d1 = fdot(ab, ap), d2 = fdot(ac, ap);
    const float bb = fdot(ab, ab), cc = fdot(ac, ac), bc = fdot(ab, ac);
    float v = 0.f, w = 0.f;
    if (!(d1 <= 0.f && d2 <= 0.f)) {
        const F3 bp = fsub(p, b), cp = fsub(p, c);
        const float d3 = fdot(ab, bp), d4 = fdot(ac, bp), d5 = fdot(ab, cp), d6 = fdot(ac, cp);
        const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
        if (d3 >= 0.f && d4 <= d3) v = 1.f;
        else if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) v = unit(d1 / (d1 - d3));
        else if (d6 >= 0.f && d5 <= d6) w = 1.f;
        else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) w = unit(d2 / (d2 - d6));
        else if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
            w = unit((d4 - d3) / ((d4 - d3) + (d5 - d6)));
            v = 1.f - w;
        } else {
            const float den = 1.f / (va + vb + vc);
            v = unit(vb * den);
            w = fminf(unit(vc * den), 1.f - v);
        }
    }
    const F3 r = {ab.x * v + ac.x * w - ap.x, ab.y * v + ac.y * w - ap.y, ab.z * v + ac.z * w - ap.z};
    const float d = sqrtf(fdot(r, r));
    const float side = sqrtf(fmaxf(bb, cc)), n2 = bb * cc - bc * bc;
    scale = fmaxf(side, d);
    slim = !(n2 > 1e-30f && n2 < 1e30f && side * side * side * scale <= 25.f * n2);
    return d;
}

// The margins. kCoord of the largest coordinate covers the float copies of a vertex and of the point (2^-24 of it for
// each of three coordinates, twice) and kTiny squares that underflow; a distance to a point of a triangle is computed
// within kUpper of the triangle's scale, and the nearest point of a triangle that is not slim is found within kLower of
// it.
constexpr float kCoord = 5e-7f, kTiny = 1e-18f, kUpper = 2e-6f, kLower = 1e-4f;

__device__ __forceinline__ float box_sq(F3 p, float4 lo, float4 hi) {
    const float dx = fmaxf(fmaxf(lo.x - p.x, 0.f), p.x - hi.x), dy = fmaxf(fmaxf(lo.y - p.y, 0.f), p.y - hi.y),
                dz = fmaxf(fmaxf(lo.z - p.z, 0.f), p.z - hi.z);
    return dx * dx + dy * dy + dz * dz;
}
// squared distances above this are above `upper` for certain
__device__ __forceinline__ float above(float upper, float margin) {
    const float u = upper + margin;
    return u * u * 1.00001f;
}

// One walk per point in float64 with a float64 box bound took 1.97 ms for 20,000 points and 327,680 faces: the float64
// pipes (1/64 of the float32 rate) and three dependent loads a node set its time. The whole call, with its copies from and
// to NumPy arrays, went from 2.94 to 1.16 ms.
__global__ void __launch_bounds__(kQT) k_point_mesh(const double* __restrict__ pts, int np, const double* __restrict__ V,
                                                    const float4* __restrict__ pos, const int4* __restrict__ tri,
                                                    const float4* __restrict__ packed, const unsigned* __restrict__ scene,
                                                    const int* __restrict__ leaf_face, const RoundCounters* rc,
                                                    double* out_d2, int* out_face, int* status) {
    pdl_wait();
    __shared__ int s_node[kStack][kQT];
    __shared__ float s_dist[kStack][kQT];
    __shared__ int s_list[kList][kQT];
    const int nl = rc->n_live, me = threadIdx.x;
    float extent = 0.f;
    for (int d = 0; d < 6; ++d) {
        const unsigned u = scene[d];
        extent = fmaxf(extent, fabsf(__uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u)));
    }
    // all lanes of a warp make the same number of rounds (the walks end in warp votes)
    for (int i0 = gtid() & ~31; i0 < np; i0 += gstride()) {
        const int i = i0 + (me & 31);
        const bool on = i < np;
        const D3 pd = on ? dload(pts, i) : D3{0.0, 0.0, 0.0};
        const F3 p = {(float)pd.x, (float)pd.y, (float)pd.z};
        const float margin = kCoord * fmaxf(extent, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z)))) + kTiny;
        float upper = INFINITY;
        double best = INFINITY;
        int bf = -1;
        auto evaluate = [&](int count) {
            for (int k = 0; __any_sync(0xffffffffu, k < count); ++k) {
                if (k >= count) continue;
                const int f = s_list[k][me];
                const int4 t = tri[f];
                const D3 c = closest_point_triangle(pd, dload(V, t.x), dload(V, t.y), dload(V, t.z));
                const D3 d = dsub(c, pd);
                const double d2 = ddot(d, d);
                if (d2 < best || (d2 == best && f < bf)) {
                    best = d2;
                    bf = f;
                }
            }
        };
        if (nl == 1) {
            if (on) s_list[0][me] = leaf_face[0];
            evaluate(on ? 1 : 0);
        }
        if (nl >= 2) {
            // pass 0: the upper bound; pass 1: the triangles that may be nearest
            for (int pass = 0; pass < 2; ++pass) {
                int sp = 0, node = on ? 0 : -1, guard = 0, count = 0;
                float limit = above(upper, margin);
                while (__any_sync(0xffffffffu, node >= 0)) {
                    if (node >= 0 && ++guard > (1 << 22)) {
                        atomicOr(status, kErrIterLimit);
                        node = -1;
                    }
                    if (node >= 0) {
                        const float4* rec = packed + 4 * (size_t)node;
                        const float4 lo0 = __ldg(rec), hi0 = __ldg(rec + 1), lo1 = __ldg(rec + 2), hi1 = __ldg(rec + 3);
                        float b0 = box_sq(p, lo0, hi0), b1 = box_sq(p, lo1, hi1);
                        int c0 = __float_as_int(lo0.w), c1 = __float_as_int(lo1.w);
                        int g0 = __float_as_int(hi0.w), g1 = __float_as_int(hi1.w);
                        if (b1 < b0) {  // the nearer child first
                            const float tb = b0; b0 = b1; b1 = tb;
                            const int tc = c0; c0 = c1; c1 = tc;
                            const int tg = g0; g0 = g1; g1 = tg;
                        }
                        int n0 = -1, n1 = -1;
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            const float bd = side ? b1 : b0;
                            if (bd > limit) continue;
                            const int x = side ? c1 : c0, f = side ? g1 : g0;
                            if (x >= 0) {
                                if (side) n1 = x;
                                else n0 = x;
                                continue;
                            }
                            const int4 t = tri[f];
                            float scale;
                            bool slim;
                            const float d = tri_distance(p, f3(pos[t.x]), f3(pos[t.y]), f3(pos[t.z]), scale, slim);
                            if (pass == 0) {
                                const float u = d + (kUpper * scale + margin);
                                if (u < upper) {
                                    upper = u;
                                    limit = above(upper, margin);
                                }
                            } else if (slim || !(d - (kLower * scale + margin) > upper)) {
                                s_list[count++][me] = f;
                            }
                        }
                        if (n0 >= 0 && n1 >= 0) {
                            if (sp >= kStack) {
                                atomicOr(status, kErrStackOverflow);
                                node = -1;
                                sp = 0;
                            } else {
                                s_node[sp][me] = n1;
                                s_dist[sp++][me] = b1;
                                node = n0;
                            }
                        } else {
                            node = n0 >= 0 ? n0 : n1;
                        }
                        while (node < 0 && sp > 0) {
                            --sp;
                            if (!(s_dist[sp][me] > limit)) node = s_node[sp][me];
                        }
                    }
                    if (__any_sync(0xffffffffu, count > kList - 2)) {
                        evaluate(count);
                        count = 0;
                    }
                }
                evaluate(count);
            }
        }
        if (on) {
            out_d2[i] = best;
            if (out_face) out_face[i] = bf;
        }
    }
}

// Per face: the minimum angle of compute_min_angle_VF (edge vectors e_k = V[f_k] - V[f_(k+1)], the angle at each
// corner from -dot(e_k, e_(k-1)) / (|e_k| |e_(k-1)|) clipped to [-1, 1]) and of igl.internal_angles (law of
// cosines on the squared edge lengths), in radians; NaN for a face with a repeated index.
__global__ void k_face_min_angles(const double* __restrict__ V, const int* __restrict__ F, int nf, double* out_edge,
                                  double* out_igl) {
    pdl_wait();
    for (int f = gtid(); f < nf; f += gstride()) {
        const int i0 = F[3 * f], i1 = F[3 * f + 1], i2 = F[3 * f + 2];
        if (i0 == i1 || i1 == i2 || i2 == i0) {
            if (out_edge) out_edge[f] = NAN;
            if (out_igl) out_igl[f] = NAN;
            continue;
        }
        const D3 p[3] = {dload(V, i0), dload(V, i1), dload(V, i2)};
        D3 e[3];
        double l[3];
        for (int k = 0; k < 3; ++k) {
            e[k] = dsub(p[k], p[(k + 1) % 3]);
            l[k] = sqrt(ddot(e[k], e[k]));
        }
        if (out_edge) {
            double m = INFINITY;
            for (int k = 0; k < 3; ++k) {
                const int km = (k + 2) % 3;
                double c = -ddot(e[k], e[km]) / (l[k] * l[km]);
                c = fmin(fmax(c, -1.0), 1.0);
                m = fmin(m, acos(c));
            }
            out_edge[f] = m;
        }
        if (out_igl) {
            // corner k is opposite the edge (k+1, k+2), whose squared length is |e_(k+1)|^2
            double m = INFINITY;
            for (int k = 0; k < 3; ++k) {
                const double a2 = l[(k + 1) % 3] * l[(k + 1) % 3];
                const double b = l[k], c = l[(k + 2) % 3];
                double x = (b * b + c * c - a2) / (2.0 * b * c);
                x = fmin(fmax(x, -1.0), 1.0);
                m = fmin(m, acos(x));
            }
            out_igl[f] = m;
        }
    }
}

size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

int cuda_status(cudaError_t e) { return e == cudaSuccess ? PAMO_OK : PAMO_ERR_CUDA; }

}  // namespace

extern "C" {

int pamo_point_mesh_workspace(int32_t n_vertices, int32_t n_triangles, int64_t* bytes) {
    if (n_vertices < 1 || n_triangles < 1 || !bytes) return PAMO_ERR_INVALID_ARG;
    *bytes = (int64_t)(256 + up256(sizeof(RoundCounters)) + up256((size_t)n_vertices * sizeof(float4)) +
                       up256(((size_t)n_triangles + 1) * sizeof(int4)) + bvh_bytes(n_triangles));
    return PAMO_OK;
}

int pamo_point_mesh_sqdist_ws(const double* points, int32_t n_points, const double* vertices, int32_t n_vertices,
                              const int32_t* triangles, int32_t n_triangles, double* out_sqdist, int32_t* out_face,
                              void* workspace, int64_t workspace_bytes, pamo_stream stream) {
    if (!points || !vertices || !triangles || !out_sqdist || n_points < 0 || n_vertices < 1 || n_triangles < 1)
        return PAMO_ERR_INVALID_ARG;
    if (n_points == 0) return PAMO_OK;
    int64_t need = 0;
    pamo_point_mesh_workspace(n_vertices, n_triangles, &need);
    if (!workspace || workspace_bytes < need) return PAMO_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    char* at = reinterpret_cast<char*>(up256(reinterpret_cast<uintptr_t>(workspace)));
    auto take = [&](size_t bytes) {
        char* p = at;
        at += up256(bytes);
        return p;
    };
    RoundCounters* rc = reinterpret_cast<RoundCounters*>(take(sizeof(RoundCounters)));
    float4* pos = reinterpret_cast<float4*>(take((size_t)n_vertices * sizeof(float4)));
    int4* tri = reinterpret_cast<int4*>(take(((size_t)n_triangles + 1) * sizeof(int4)));
    BvhBuffers b;
    bvh_carve(b, n_triangles, at, false);
    cudaMemsetAsync(b.scan_scratch, 0, scan_scratch_ints() * sizeof(int), s);
    RoundCounters h{};
    h.n_pts = n_vertices;
    h.n_tris = n_triangles;
    cudaMemcpyAsync(rc, &h, sizeof(h), cudaMemcpyHostToDevice, s);
    pdl(k_to_float4, grid_for(n_vertices, kT), kT, 0, s)(vertices, n_vertices, pos);
    pdl(k_to_int4, grid_for(n_triangles, kT), kT, 0, s)(triangles, n_triangles, n_vertices, tri, &rc->status);
    note_launches(2);
    bvh_build(b, tri, pos, rc, n_triangles, s, false, BvhQuery(), false);
    pdl(k_point_mesh, grid_for(n_points, kQT, 16), kQT, 0, s)(points, n_points, vertices, pos, tri, b.packed, b.scene,
                                                             b.vals[0], rc, out_sqdist, out_face, &rc->status);
    note_launch();
    int st = 0;
    cudaMemcpyAsync(&st, &rc->status, sizeof(int), cudaMemcpyDeviceToHost, s);
    int r = cuda_status(cudaStreamSynchronize(s));
    if (r == PAMO_OK && (st & kErrBadIndex)) r = PAMO_ERR_INVALID_ARG;
    else if (r == PAMO_OK && st) r = PAMO_ERR_ITER_LIMIT;
    return r;
}

int pamo_point_mesh_sqdist(const double* points, int32_t n_points, const double* vertices, int32_t n_vertices,
                           const int32_t* triangles, int32_t n_triangles, double* out_sqdist, int32_t* out_face,
                           pamo_stream stream) {
    if (!points || !vertices || !triangles || !out_sqdist || n_points < 0 || n_vertices < 1 || n_triangles < 1)
        return PAMO_ERR_INVALID_ARG;
    if (n_points == 0) return PAMO_OK;
    int64_t bytes = 0;
    pamo_point_mesh_workspace(n_vertices, n_triangles, &bytes);
    void* workspace = nullptr;
    if (cudaMalloc(&workspace, (size_t)bytes) != cudaSuccess) return PAMO_ERR_OOM;
    const int r = pamo_point_mesh_sqdist_ws(points, n_points, vertices, n_vertices, triangles, n_triangles, out_sqdist,
                                            out_face, workspace, bytes, stream);
    cudaFree(workspace);
    return r;
}

int pamo_face_min_angles(const double* vertices, const int32_t* triangles, int32_t n_triangles, double* out_edge_form,
                         double* out_igl_form, pamo_stream stream) {
    if (!vertices || !triangles || n_triangles < 0 || (!out_edge_form && !out_igl_form)) return PAMO_ERR_INVALID_ARG;
    if (n_triangles == 0) return PAMO_OK;
    cudaStream_t s = (cudaStream_t)stream;
    pdl(k_face_min_angles, grid_for(n_triangles, kT), kT, 0, s)(vertices, triangles, n_triangles, out_edge_form,
                                                               out_igl_form);
    note_launch();
    return cuda_status(cudaStreamSynchronize(s));
}

}  // extern "C"
