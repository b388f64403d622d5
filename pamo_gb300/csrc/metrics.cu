// Evaluation kernels of the reference's metrics module (simp_cuda/safe_project/src/pamo_safe_project/
// metrics.py:7-107): squared distances from points to a triangle mesh (the closest-point queries behind its
// Chamfer and Hausdorff distances) and the per-face minimum angles behind compute_min_angle and
// compute_bad_tri_ratio. Off the simplification path; inputs are float64 like the metrics' NumPy arrays.
//
// Point-to-mesh distance: two walks per point through the packed stage-2 LBVH over float copies of the vertices. The
// first, all in float, gives an upper bound of the distance; the second collects the triangles that may be as near, and
// those few take the exact float64 point-triangle distance (Ericson, Real-Time Collision Detection, 5.1.5), the lanes
// of a warp together. The nearest triangle and the smallest index of equally near ones are the same as by trying every
// triangle in float64; the margins below hold what float adds. Points that float cannot serve (very far away, or with a
// thousand triangles that it cannot tell apart) are left to a walk in float64.
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
// triangles a lane collects before the warp evaluates them: 4, 8 and 16 take the same time near the mesh (0.62 to 0.65 ms), 4
// two per cent more for points away from it
constexpr int kList = 8;

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

__device__ __forceinline__ F3 fabs3(F3 a) { return {fabsf(a.x), fabsf(a.y), fabsf(a.z)}; }

// What the float walks compare. For a point p let c be a float point near it, the nearest of the mesh's box, and w = p - c.
// With y = x - c, |p - x|^2 = |w|^2 + 2 g(x), g(x) = sum over the axes of y (y / 2 - w). |w|^2 is the point's own, so g orders
// the mesh as the distance does, and from far away it is made of small numbers: its rounding is about 1e-6 of |y| in the
// distance, however far the point is, where the distance itself is rounded by 1e-7 of its value. From within the mesh's
// box w is the rounding of p's float copy (which it takes out) and g half the squared distance.
//
// The margins, each of the numbers that it comes from, so that one far vertex or point widens nothing else (u = 2^-24 is
// float's rounding of a value):
//  * a term y (y / 2 - w) with y, w and each operation rounded is off by at most 6 u |y| (|y| + |w|), with the sum of the
//    three terms: kTerm of the sum of |y| (|y| + |w|);
//  * a box's coordinates are those of float copies: no vertex lies farther out than u of the side's own coordinate (x - u |x|
//    grows with x), and each side is moved out by kBox of it;
//  * a point of a triangle is y = (a - c) + v ab + w ac, off by at most u (|a| + 10 side + 2 |y|) in an axis, vertices' copies
//    included, which counts |r| times, r = y - w being the slope of g: kVert of |r| |a|, kSide of |r| side (side: the longer
//    of |ab| and |ac|; its share of the corner test below included), and the square of both where r vanishes;
//  * kTiny: products that underflow.
//  * kTies: a squared distance in float64 is rounded by a few 2^-53 of itself.
constexpr float kTies = 1e-14f;
constexpr float kTerm = 1e-6f, kBox = 2.5e-7f, kVert = 1.5e-7f, kSide = 1.5e-6f, kTiny = 1e-36f;

// g at its least in a box (the exact vertices'), less its margin
__device__ __forceinline__ void box_axis(float c, float w, float lo, float hi, float& g, float& size) {
    const float y = fminf(fmaxf(w, (lo - c) - kBox * fabsf(lo)), (hi - c) + kBox * fabsf(hi)), m = fabsf(y);
    g += y * (0.5f * y - w);
    size += m * (m + fabsf(w));
}
__device__ __forceinline__ float box_g(F3 c, F3 w, float4 lo, float4 hi) {
    float g = 0.f, size = 0.f;
    box_axis(c.x, w.x, lo.x, hi.x, g, size);
    box_axis(c.y, w.y, lo.y, hi.y, g, size);
    box_axis(c.z, w.z, lo.z, hi.z, g, size);
    return g - kTerm * size;
}

// g at the triangle's nearest point as float finds it, and its margin err: g + err is an upper bound of the triangle's
// least g, since the point lies in the triangle whatever the rounding did (the parameters are clamped). With kLow, low is
// a lower bound: g is convex, so over the triangle it is at least its tangent at that point, which is least at a corner.
// (For the true nearest point the corners all lie on the far side; how far the parameters are off shows in it.)
template <bool kLow>
__device__ __forceinline__ float tri_g(F3 c, F3 w, F3 a, F3 b, F3 d, float& err, float& low) {
    const F3 ya = fsub(a, c), ab = fsub(b, a), ac = fsub(d, a), ap = fsub(w, ya);
    const float d1 = fdot(ab, ap), d2 = fdot(ac, ap);
    const float bb = fdot(ab, ab), cc = fdot(ac, ac);
    float s = 0.f, t = 0.f;
    if (!(d1 <= 0.f && d2 <= 0.f)) {
        const F3 bp = fsub(ap, ab), cp = fsub(ap, ac);
        const float d3 = fdot(ab, bp), d4 = fdot(ac, bp), d5 = fdot(ab, cp), d6 = fdot(ac, cp);
        const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
        if (d3 >= 0.f && d4 <= d3) s = 1.f;
        else if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) s = unit(d1 / (d1 - d3));
        else if (d6 >= 0.f && d5 <= d6) t = 1.f;
        else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) t = unit(d2 / (d2 - d6));
        else if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
            t = unit((d4 - d3) / ((d4 - d3) + (d5 - d6)));
            s = 1.f - t;
        } else {
            const float den = 1.f / (va + vb + vc);
            s = unit(vb * den);
            t = fminf(unit(vc * den), 1.f - s);
        }
    }
    const F3 e = {ab.x * s + ac.x * t, ab.y * s + ac.y * t, ab.z * s + ac.z * t};
    const F3 y = {ya.x + e.x, ya.y + e.y, ya.z + e.z}, r = fsub(y, w);
    const F3 ma = fabs3(a), my = fabs3(y), mr = fabs3(r), mw = fabs3(w);
    const float g = y.x * (0.5f * y.x - w.x) + y.y * (0.5f * y.y - w.y) + y.z * (0.5f * y.z - w.z);
    const float side = sqrtf(fmaxf(bb, cc));
    const float still = kVert * fmaxf(ma.x, fmaxf(ma.y, ma.z)) + kSide * side;
    err = kTerm * fdot(my, F3{my.x + mw.x, my.y + mw.y, my.z + mw.z}) + kVert * fdot(mr, ma) +
          kSide * side * (mr.x + mr.y + mr.z) + still * still;
    if (kLow) {
        const F3 eb = fsub(e, ab), ec = fsub(e, ac);
        low = g - fmaxf(fmaxf(fdot(r, e), fdot(r, eb)), fmaxf(fdot(r, ec), 0.f)) - err;
    }
    return g;
}

// A point farther from the mesh's box than kFar of its extents is left to the float64 walk at once, one with more than kMaxNear
// triangles to evaluate, or kMaxNodes nodes in a walk, when it has that many: from there on the float walk no longer tells what it is for (a flat mesh seen
// from very far: thousands of triangles within the rounding of a float). 2,000 points at 500 extents of a star-shaped mesh
// take 16 ms by the float walk and 46 by the other, but 500 to 1,000 extents above a flat mesh 0.78 ms and 0.56, and that
// gap grows. kMaxNear 256, 1,024 and 4,096 gave the same times in every case tried (the centre of a sphere among them).
constexpr float kFar = 100.f;
constexpr int kMaxNear = 1024, kMaxNodes = 1 << 20;

// One walk per point in float64 with a float64 box bound took 1.97 ms for 20,000 points and 327,680 faces: the float64
// pipes (1/64 of the float32 rate) and three dependent loads a node set its time. The whole call, with its copies from and
// to NumPy arrays, went from 2.94 to 1.16 ms, and to 0.62 ms with the caller's workspace.
// With margins of the whole scene's coordinates and of the distance itself, that case kept its time but a vertex at 1e6
// took 1,079 ms (the float64 walk: 32 ms), 2,000 points at 1e5 1,033 ms (72 ms) and 2,000 points 50 to 100 extents above a
// flat mesh of 286k faces 1,053 ms (1.25 ms): nearly every triangle was a candidate. With g and its margins they take 4.7,
// 46 and 0.56 ms, and 2,000 points at 3 to 100 radii of the mesh 11 to 16 ms (20 to 30; 48 to 72).
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
    float ends[6];
    for (int d = 0; d < 6; ++d) {
        const unsigned u = scene[d];
        ends[d] = __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
    }
    const float extent = fmaxf(ends[3] - ends[0], fmaxf(ends[4] - ends[1], ends[5] - ends[2]));
    // all lanes of a warp make the same number of rounds (the walks end in warp votes)
    for (int i0 = gtid() & ~31; i0 < np; i0 += gstride()) {
        const int i = i0 + (me & 31);
        const bool on = i < np;
        const D3 pd = on ? dload(pts, i) : D3{0.0, 0.0, 0.0};
        const F3 c = {fminf(fmaxf((float)pd.x, ends[0]), ends[3]), fminf(fmaxf((float)pd.y, ends[1]), ends[4]),
                      fminf(fmaxf((float)pd.z, ends[2]), ends[5])};
        const D3 wd = {pd.x - c.x, pd.y - c.y, pd.z - c.z};
        const F3 w = {(float)wd.x, (float)wd.y, (float)wd.z};
        // what counts as equally near: also what float64 does not tell apart (g may be the finer from very far)
        const float tie = kTies * fdot(w, w) + kTiny;
        bool left = nl >= 2 && fmaxf(fabsf(w.x), fmaxf(fabsf(w.y), fabsf(w.z))) > kFar * extent;
        int near = 0;
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
                int sp = 0, node = on && !left ? 0 : -1, guard = 0, count = 0;
                while (__any_sync(0xffffffffu, node >= 0)) {
                    if (node >= 0 && ++guard > kMaxNodes) {
                        left = true;
                        node = -1;
                        sp = 0;
                    }
                    if (node >= 0) {
                        const float4* rec = packed + 4 * (size_t)node;
                        const float4 lo0 = __ldg(rec), hi0 = __ldg(rec + 1), lo1 = __ldg(rec + 2), hi1 = __ldg(rec + 3);
                        float b0 = box_g(c, w, lo0, hi0), b1 = box_g(c, w, lo1, hi1);
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
                            if (bd > upper) continue;
                            const int x = side ? c1 : c0, f = side ? g1 : g0;
                            if (x >= 0) {
                                if (side) n1 = x;
                                else n0 = x;
                                continue;
                            }
                            const int4 t = tri[f];
                            float err, low = 0.f;
                            if (pass == 0) {
                                const float u = tri_g<false>(c, w, f3(pos[t.x]), f3(pos[t.y]), f3(pos[t.z]), err, low) + err + tie;
                                if (u < upper) upper = u;
                                continue;
                            }
                            tri_g<true>(c, w, f3(pos[t.x]), f3(pos[t.y]), f3(pos[t.z]), err, low);
                            if (!(low > upper)) {  // also where low is not a number
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
                            if (!(s_dist[sp][me] > upper)) node = s_node[sp][me];
                        }
                    }
                    if (__any_sync(0xffffffffu, count > kList - 2)) {
                        evaluate(count);
                        near += count;
                        count = 0;
                        if (near > kMaxNear) {
                            left = true;
                            node = -1;
                            sp = 0;
                        }
                    }
                }
                evaluate(count);
            }
        }
        if (on && left) {
            // a negative value: the walk in float64 is to find it, from this bound
            const double bound = ddot(wd, wd) + 2.0 * (double)upper;
            out_d2[i] = -(fmin(bound, best) * (1.0 + 1e-12) + 1e-300);
        } else if (on) {
            out_d2[i] = best;
            if (out_face) out_face[i] = bf;
        }
    }
}

// squared distance from p to a box widened by a relative 2^-22 (so that it bounds the float64 geometry the float box was
// rounded from, by 2^-24 of it), as a lower bound for pruning
__device__ __forceinline__ double box_lower_bound(D3 p, float4 lo, float4 hi) {
    const double e = 2.384185791015625e-07;  // 2^-22
    auto axis = [&](double x, float l, float h) {
        const double dl = (double)l - e * fabs((double)l) - 1e-30, dh = (double)h + e * fabs((double)h) + 1e-30;
        return x < dl ? dl - x : (x > dh ? x - dh : 0.0);
    };
    const double dx = axis(p.x, lo.x, hi.x), dy = axis(p.y, lo.y, hi.y), dz = axis(p.z, lo.z, hi.z);
    return dx * dx + dy * dy + dz * dz;
}

// The points that k_point_mesh left, one thread each and all in float64: far away (a float is coarser than the mesh's
// features there) or with very many triangles at nearly the same distance.
__global__ void __launch_bounds__(kQT) k_point_mesh_wide(const double* __restrict__ pts, int np, const double* __restrict__ V,
                                                         const int4* __restrict__ tri, const float4* __restrict__ packed,
                                                         const RoundCounters* rc, double* out_d2, int* out_face,
                                                         int* status) {
    pdl_wait();
    __shared__ int s_node[kStack][kQT];
    __shared__ double s_dist[kStack][kQT];
    if (rc->n_live < 2) return;  // no point is left then
    const int me = threadIdx.x;
    for (int i = gtid(); i < np; i += gstride()) {
        double best = -out_d2[i];
        if (!(best > 0.0)) continue;
        const D3 p = dload(pts, i);
        int bf = -1, sp = 0, node = 0, guard = 0;
        while (node >= 0) {
            if (++guard > (1 << 22)) {
                atomicOr(status, kErrIterLimit);
                break;
            }
            const float4* rec = packed + 4 * (size_t)node;
            const float4 lo[2] = {__ldg(rec), __ldg(rec + 2)}, hi[2] = {__ldg(rec + 1), __ldg(rec + 3)};
            int n[2] = {-1, -1};
            double nd[2];
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                nd[side] = box_lower_bound(p, lo[side], hi[side]);
                if (nd[side] > best * (1.0 + kTies)) continue;  // equally near ones are all visited
                const int x = __float_as_int(lo[side].w);
                if (x >= 0) {
                    n[side] = x;
                    continue;
                }
                const int f = __float_as_int(hi[side].w);
                const int4 t = tri[f];
                const D3 c = closest_point_triangle(p, dload(V, t.x), dload(V, t.y), dload(V, t.z));
                const D3 d = dsub(c, p);
                const double d2 = ddot(d, d);
                if (d2 < best || (d2 == best && f < bf)) {
                    best = d2;
                    bf = f;
                }
            }
            if (n[0] >= 0 && n[1] >= 0) {
                if (sp >= kStack) {
                    atomicOr(status, kErrStackOverflow);
                    break;
                }
                const bool swap = nd[1] < nd[0];
                s_node[sp][me] = swap ? n[0] : n[1];
                s_dist[sp++][me] = swap ? nd[0] : nd[1];
                node = swap ? n[1] : n[0];
            } else {
                node = n[0] >= 0 ? n[0] : n[1];
            }
            while (node < 0 && sp > 0) {
                --sp;
                if (!(s_dist[sp][me] > best * (1.0 + kTies))) node = s_node[sp][me];
            }
        }
        out_d2[i] = bf >= 0 ? best : INFINITY;
        if (out_face) out_face[i] = bf;
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
    pdl(k_point_mesh_wide, grid_for(n_points, kQT, 16), kQT, 0, s)(points, n_points, vertices, tri, b.packed, rc, out_sqdist,
                                                                  out_face, &rc->status);
    note_launches(2);
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
