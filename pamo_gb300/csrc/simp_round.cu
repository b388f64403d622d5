// Kernels of one PaMO stage-2 collapse round on GB300.
//
// Reference round: CUSimp_Free::forward (simp_cuda/src/cusimp_free.cu:891-1048). Differences in form, not in
// result:
//   * vertex->face lists are filled with atomics and then sorted per vertex, so every float sum over a ring
//     runs in ascending face order and the round is deterministic;
//   * the per-face minimum key of propagate_edge_cost_kernel (:587-610) is replaced by a per-vertex minimum (two
//     64-bit atomicMin per edge instead of one per ring face), whose minimum over a face's vertices it is;
//   * winners are listed in ascending edge order through a scan instead of an atomic counter;
//   * the undo check marks intersecting faces in a flag array and tests ring membership in O(ring) instead
//     of scanning the whole intersection list per collapsed edge (:776-827).
#include <cstdint>
#include <type_traits>
#include <algorithm>

#include "scan.cuh"
#include "simp_round.cuh"
#include "round_ops.cuh"

namespace pamo {

namespace {

constexpr int kT = 256;
constexpr float kCostRange = 10.0f;            // cusimp_free.cu:15
constexpr float kU32MaxF = 4294967296.0f;      // (float)UINT32_MAX

// ------------------------------------------------------------------ set-up
__global__ void k_undo_stuck(const int* __restrict__ verts_undo, int n, int* tmp_undo, int* undo_list,
                             const int* __restrict__ pts_map, int map_len) {
    pdl_wait();
    for (int a = gtid(); a < n; a += gstride()) {
        const int x = verts_undo[a];
        tmp_undo[a] = x;
        undo_list[a] = (x >= 0 && x < map_len) ? pts_map[x] : 0;  // rearrange_index_of_undo_vertices, :869-878
    }
}

__global__ void k_invalid_mark(const int* __restrict__ verts_undo, int n, unsigned char* invalid, int len) {
    pdl_wait();
    for (int a = gtid(); a < n; a += gstride()) {
        const int x = verts_undo[a];
        if (x >= 0 && x < len) invalid[x] = 1;  // compute_invalid_vertices_table, :880-889
    }
}

__global__ void k_load_points(const float* __restrict__ pts, int n, float4* pos, float4* orig, int* occ) {
    pdl_wait();
    for (int v = gtid(); v < n; v += gstride()) {
        const float4 p = make_float4(pts[3 * v], pts[3 * v + 1], pts[3 * v + 2], 0.f);
        pos[v] = p;
        orig[v] = p;
        occ[v] = 1;
    }
    if (gtid() == 0) occ[n] = 0;
}

__global__ void k_load_points4(const float4* __restrict__ pts, int n, float4* pos, float4* orig, int* occ) {
    pdl_wait();
    for (int v = gtid(); v < n; v += gstride()) {
        const float4 p = pts[v];
        pos[v] = p;
        orig[v] = p;
        occ[v] = 1;
    }
    if (gtid() == 0) occ[n] = 0;
}

__global__ void k_load_tris(const int* __restrict__ tris, int n, int n_pts, int4* tri, RoundCounters* rc) {
    pdl_wait();
    for (int f = gtid(); f < n; f += gstride()) {
        const int a = tris[3 * f], b = tris[3 * f + 1], c = tris[3 * f + 2];
        const bool dead = (a == -1 && b == -1 && c == -1);
        const bool ok = dead || (a >= 0 && a < n_pts && b >= 0 && b < n_pts && c >= 0 && c < n_pts);
        if (!ok) atomicOr(&rc->status, kErrBadIndex);
        tri[f] = ok ? make_int4(a, b, c, 0) : make_int4(-1, -1, -1, 0);
    }
}

__global__ void k_copy4(const int4* __restrict__ src, int4* dst, int n) {
    pdl_wait();
    for (int f = gtid(); f < n; f += gstride()) dst[f] = src[f];
}

__global__ void k_shuffle_flags(Feistel fb, int* flags) {
    pdl_wait();
    const long long n = (long long)fb.n;
    for (long long i = gtid(); i < n; i += gstride()) flags[i] = feistel(fb, fb.size, (unsigned long long)i) < fb.m ? 1 : 0;
    if (gtid() == 0) flags[n] = 0;
}

__global__ void k_shuffle_gather(Feistel fb, const int* __restrict__ scan, const int4* __restrict__ src, int4* dst) {
    pdl_wait();
    const long long n = (long long)fb.n;
    for (long long i = gtid(); i < n; i += gstride()) {
        const unsigned long long g = feistel(fb, fb.size, (unsigned long long)i);
        if (g < fb.m) dst[scan[i]] = src[g];
    }
}

// ------------------------------------------------------------------ adjacency
// Per-face values that the vertex rings read many times (every face lies in three rings and every ring is
// read once per incident edge), each computed by the same operations as where the reference computes it. One
// aligned 64-byte record per face, fgeo[4f .. 4f + 3]:
//   (l01, l12, l20, L1)        the edge lengths |p_x - p_y|, |p_y - p_z|, |p_z - p_x| (the ring edge-length
//                              terms, :449-484) and the L1 norm of the unnormalised normal;
//   (o.x, o.y, o.z, p_x.x), (p_x.y, p_x.z, p_y.x, p_y.y), (p_y.z, p_z.x, p_z.y, p_z.z)
//                              the unnormalised normal cross(p_y - p_x, p_z - p_x) (the flip test) and the three
//                              corner positions, so that a ring face needs no gather of its vertices;
// then, after all n records (n = the round's face count), the face planes of tri2plane (:337-346), fgeo[4n + f]
// (precision mode: a double-float pair, fgeo[4n + 2f] and fgeo[4n + 2f + 1]), which only the quadrics read.
// The buffer holds 6 float4 per face.
__device__ __forceinline__ void face_plane(const float4* __restrict__ pos, int4 t, float p[4]);

// ---- precision mode: error-free transforms (Knuth's TwoSum; TwoProd with an explicit fused multiply-add, which
// --fmad=false leaves alone) and a compensated float accumulator (Ogita, Rump and Oishi's Sum2/Dot2)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
    p = a * b;
    e = __fmaf_rn(a, b, -p);
}
struct CSum {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        float t, e;
        two_sum(s, x, t, e);
        s = t;
        c += e;
    }
    __device__ __forceinline__ void add_prod(float a, float b) {
        float p, pe;
        two_prod(a, b, p, pe);
        add(p);
        c += pe;
    }
    __device__ __forceinline__ float value() const { return s + c; }
};
// Double-float numbers (hi + lo, |lo| <= ulp(hi) / 2) from FP32 operations only (Dekker; Hida, Li and Bailey's
// double-double algorithms), for the precision mode's face planes: about 44 significant bits without FP64.
struct DF {
    float hi, lo;
};
__device__ __forceinline__ DF df_fast(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
    float s, e;
    two_sum(a.hi, b.hi, s, e);
    e += a.lo + b.lo;
    return df_fast(s, e);
}
__device__ __forceinline__ DF df_neg(DF a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_mul(DF a, DF b) {
    float p, e;
    two_prod(a.hi, b.hi, p, e);
    e += a.hi * b.lo + a.lo * b.hi;
    return df_fast(p, e);
}
__device__ __forceinline__ DF df_diff(float a, float b) {  // a - b exactly
    float s, e;
    two_sum(a, -b, s, e);
    return {s, e};
}
__device__ __forceinline__ DF df_sqrt(DF a) {
    if (!(a.hi > 0.0f)) return {0.0f, 0.0f};
    const float r = sqrtf(a.hi);
    float p, e;
    two_prod(r, r, p, e);
    return df_fast(r, ((a.hi - p) - e + a.lo) / (2.0f * r));
}
__device__ __forceinline__ DF df_div(DF a, DF b) {
    const float q1 = a.hi / b.hi;
    const DF r = df_add(a, df_neg(df_mul(b, DF{q1, 0.0f})));
    return df_fast(q1, r.hi / b.hi);
}

// The face plane of tri2plane (unit normal of cross(p_y - p_x, p_z - p_x), offset -n.p_x) in double-float
__device__ __forceinline__ void face_plane_df(const float4* __restrict__ pos, int4 t, DF p[4]) {
    const float4 a = pos[t.x], b = pos[t.y], c = pos[t.z];
    const DF e1[3] = {df_diff(b.x, a.x), df_diff(b.y, a.y), df_diff(b.z, a.z)};
    const DF e2[3] = {df_diff(c.x, a.x), df_diff(c.y, a.y), df_diff(c.z, a.z)};
    DF n[3];
    n[0] = df_add(df_mul(e1[1], e2[2]), df_neg(df_mul(e1[2], e2[1])));
    n[1] = df_add(df_mul(e1[2], e2[0]), df_neg(df_mul(e1[0], e2[2])));
    n[2] = df_add(df_mul(e1[0], e2[1]), df_neg(df_mul(e1[1], e2[0])));
    const DF len = df_sqrt(df_add(df_add(df_mul(n[0], n[0]), df_mul(n[1], n[1])), df_mul(n[2], n[2])));
    for (int k = 0; k < 3; ++k) p[k] = df_div(n[k], len);
    const DF d = df_add(df_add(df_mul(p[0], DF{a.x, 0.0f}), df_mul(p[1], DF{a.y, 0.0f})), df_mul(p[2], DF{a.z, 0.0f}));
    p[3] = df_neg(d);
}

__device__ __forceinline__ void acc_add(float& a, float x) { a += x; }
__device__ __forceinline__ void acc_add(CSum& a, float x) { a.add(x); }
__device__ __forceinline__ float acc_value(float a) { return a; }
__device__ __forceinline__ float acc_value(const CSum& a) { return a.value(); }

// plane_df (precision mode): the planes as double-float pairs, fgeo[4n + 2f] (hi) and fgeo[4n + 2f + 1] (lo)
__global__ void __launch_bounds__(kT) k_face_counts(const int4* __restrict__ tri, const RoundCounters* rc, int* valence,
                                                    int* ecount, int* vedges, const float4* __restrict__ pos,
                                                    float4* fgeo, int plane_df, int2* rank, UndoBook book) {
    pdl_wait();
    const int n = rc->n_tris;
    if (book.ls) {
        // stuck: the undo list restarts from the carried vertices mapped through the previous map (:869-878);
        // then the carried vertices are marked invalid (:880-889)
        const int m = book.ls->nu;
        const bool stuck = book.ls->is_stuck != 0;
        for (int a = gtid(); a < m; a += gstride()) {
            const int x = book.verts_undo[a];
            if (stuck) {
                book.tmp_undo[a] = x;
                book.undo_list[a] = (x >= 0 && x < book.map_len) ? book.pts_map[x] : 0;
            }
            if (x >= 0 && x < book.invalid_len) book.invalid[x] = 1;
        }
    }
    for (int f = gtid(); f < n; f += gstride()) {
        const int4 t = tri[f];
        if (face_killed(t)) {
            ecount[f] = 0;
            continue;
        }
        if (fgeo) {
            const V3 o0 = v3(pos[t.x]), o1 = v3(pos[t.y]), o2 = v3(pos[t.z]);
            const V3 ou = vcross(vsub(o1, o0), vsub(o2, o0));
            float4* r = fgeo + 4 * (size_t)f;
            r[0] = make_float4(vnorm(vsub(o0, o1)), vnorm(vsub(o1, o2)), vnorm(vsub(o2, o0)),
                               fabsf(ou.x) + fabsf(ou.y) + fabsf(ou.z));
            r[1] = make_float4(ou.x, ou.y, ou.z, o0.x);
            r[2] = make_float4(o0.y, o0.z, o1.x, o1.y);
            r[3] = make_float4(o1.z, o2.x, o2.y, o2.z);
            if (plane_df) {
                DF pd[4];
                face_plane_df(pos, t, pd);
                fgeo[4 * (size_t)n + 2 * (size_t)f] = make_float4(pd[0].hi, pd[1].hi, pd[2].hi, pd[3].hi);
                fgeo[4 * (size_t)n + 2 * (size_t)f + 1] = make_float4(pd[0].lo, pd[1].lo, pd[2].lo, pd[3].lo);
            } else {
                float pl[4];
                face_plane(pos, t, pl);
                fgeo[4 * (size_t)n + f] = make_float4(pl[0], pl[1], pl[2], pl[3]);
            }
        }
        ecount[f] = (t.x > t.y) + (t.y > t.z) + (t.z > t.x);  // count_edge_kernel, :306-316
        // each count's old value is the corner's place in its ring (and the edge's among those of its lower endpoint, for
        // the vertex-grouped processing order), kept for the fill, which then needs no counters of its own
        const int2 r0 = {atomicAdd(&valence[t.x], 1), t.x > t.y ? atomicAdd(&vedges[t.y], 1) : -1};
        const int2 r1 = {atomicAdd(&valence[t.y], 1), t.y > t.z ? atomicAdd(&vedges[t.z], 1) : -1};
        const int2 r2 = {atomicAdd(&valence[t.z], 1), t.z > t.x ? atomicAdd(&vedges[t.x], 1) : -1};
        int2* at = rank + 3 * (size_t)f;
        at[0] = r0;
        at[1] = r1;
        at[2] = r2;
    }
    if (gtid() == 0) ecount[n] = 0;
}

// d_cap (or null): the length of the edge costs as the reference sizes them; rc->pad[0] says whether it grew, and then the
// costs start from zero (k_ring_quadrics)
__global__ void __launch_bounds__(kT) k_fill_adjacency(const int4* __restrict__ tri, RoundCounters* rc,
                                                       const int* __restrict__ nt_off, const int2* __restrict__ rank,
                                                       int* nt, const int* __restrict__ edge_off, int2* edges,
                                                       const int* __restrict__ voff, int* eorder, int* d_cap) {
    pdl_wait();
    const int n = rc->n_tris;
    if (d_cap && gtid() == 0) {
        const int ne = rc->n_edges;
        const int grow = ne > *d_cap;
        if (grow) *d_cap = ne + ne / 5;
        rc->pad[0] = grow;
    }
    for (int f = gtid(); f < n; f += gstride()) {
        const int4 t = tri[f];
        if (face_killed(t)) continue;
        const int2 r0 = rank[3 * (size_t)f], r1 = rank[3 * (size_t)f + 1], r2 = rank[3 * (size_t)f + 2];
        nt[nt_off[t.x] + r0.x] = f;
        nt[nt_off[t.y] + r1.x] = f;
        nt[nt_off[t.z] + r2.x] = f;
        int e = edge_off[f];  // create_edge_kernel, :318-335
        if (t.x > t.y) {
            eorder[voff[t.y] + r0.y] = e;
            edges[e++] = make_int2(t.y, t.x);
        }
        if (t.y > t.z) {
            eorder[voff[t.z] + r1.y] = e;
            edges[e++] = make_int2(t.z, t.y);
        }
        if (t.z > t.x) {
            eorder[voff[t.x] + r2.y] = e;
            edges[e++] = make_int2(t.x, t.z);
        }
    }
}

// ------------------------------------------------------------------ quadrics (compute_vert_Q_kernel, :337-366)
__device__ __forceinline__ void face_plane(const float4* __restrict__ pos, int4 t, float p[4]) {
    const V3 v0 = v3(pos[t.x]), v1 = v3(pos[t.y]), v2 = v3(pos[t.z]);
    V3 n = vcross(vsub(v1, v0), vsub(v2, v0));
    n = vdiv(n, vnorm(n));
    p[0] = n.x;
    p[1] = n.y;
    p[2] = n.z;
    p[3] = -vdot(n, v0);
}

// Sorts r[0 .. N) ascending (N a power of two) by Batcher's odd-even merge exchange, all in registers.
template <int N>
__device__ __forceinline__ void sort_registers(int (&r)[N]) {
#pragma unroll
    for (int p = 1; p < N; p *= 2)
#pragma unroll
        for (int k = p; k >= 1; k /= 2)
#pragma unroll
            for (int j = k % p; j + k < N; j += 2 * k)
#pragma unroll
                for (int i = 0; i < k; ++i)
                    if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
                        const int lo = min(r[i + j], r[i + j + k]), hi = max(r[i + j], r[i + j + k]);
                        r[i + j] = lo;
                        r[i + j + k] = hi;
                    }
}

// The faces nt[a, b) of a ring into ascending order. The rings are filled by atomics, so their order is arbitrary. A ring
// of up to 16 faces (nearly all) is sorted in registers; sorted in place, its loads and stores were a chain of L2
// latencies (22 us of a mean round of 1.29 ms from 5.24M faces, 9.4 us of one of 0.25 ms from 1,280).
template <int N>
__device__ __forceinline__ void sort_ring_small(int* nt, int a, int m) {
    int r[N];
#pragma unroll
    for (int k = 0; k < N; ++k) r[k] = k < m ? nt[a + k] : 0x7fffffff;
    sort_registers<N>(r);
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (k < m) nt[a + k] = r[k];
}
__device__ __forceinline__ void sort_ring(int* nt, int a, int b) {
    const int m = b - a;
    if (m <= 8) {
        sort_ring_small<8>(nt, a, m);
    } else if (m <= 16) {
        sort_ring_small<16>(nt, a, m);
    } else {
        for (int i = a + 1; i < b; ++i) {
            const int x = nt[i];
            int j = i - 1;
            while (j >= a && nt[j] > x) {
                nt[j + 1] = nt[j];
                --j;
            }
            nt[j + 1] = x;
        }
    }
}

// The rings in face order, then the quadrics from the face planes of fgeo; also, per ring slot s of v (face t =
// tri[nt[s]]), nxt[s] = the vertex after v in t (the link condition's per-slot value) and spc[s] = (the vertex before v,
// the corner c of v: the first of t.x, t.y, t.z equal to v), from which the ring passes rebuild t without reading it.
// Four slots at a time, so that their gathers are in flight together; the sums run in slot order.
// kComp (precision mode): every entry summed with compensation (products by TwoProd, sums by TwoSum), rounded once
// cost (or null): zeroed where the edge costs grew (rc->pad[0], k_fill_adjacency)
template <bool kComp>
__global__ void __launch_bounds__(kT) k_ring_quadrics(const RoundCounters* rc, const int* __restrict__ nt_off, int* nt,
                                                      const int4* __restrict__ tri, const float4* __restrict__ fgeo,
                                                      Quadric* q, int* nxt, int2* spc, Quadric* qlo, uint32_t* cost,
                                                      int cost_len) {
    pdl_wait();
    if (cost && rc->pad[0])
        for (int i = gtid(); i < cost_len; i += gstride()) cost[i] = 0u;
    const int n = rc->n_pts;
    const size_t planes = 4 * (size_t)rc->n_tris;
    for (int v = gtid(); v < n; v += gstride()) {
        float m00 = 0.f, m01 = 0.f, m02 = 0.f, m03 = 0.f, m11 = 0.f, m12 = 0.f, m13 = 0.f, m22 = 0.f, m23 = 0.f, m33 = 0.f;
        CSum c[10];
        const int a = nt_off[v], b = nt_off[v + 1];
        sort_ring(nt, a, b);
        for (int s0 = a; s0 < b; s0 += 4) {
            int f4[4];
            int4 t4[4];
            float4 p4[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) f4[k] = s0 + k < b ? nt[s0 + k] : -1;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (f4[k] < 0) continue;
                t4[k] = tri[f4[k]];
                p4[k] = kComp ? fgeo[planes + 2 * (size_t)f4[k]] : fgeo[planes + f4[k]];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (f4[k] < 0) continue;
                const int s = s0 + k;
                const int4 t = t4[k];
                const int corner = t.x == v ? 0 : (t.y == v ? 1 : 2);
                nxt[s] = corner == 0 ? t.y : (corner == 1 ? t.z : t.x);
                spc[s] = make_int2(corner == 0 ? t.z : (corner == 1 ? t.x : t.y), corner);
                if constexpr (kComp) {  // double-float planes (face_plane_df), double-float products and sums
                    const float4 ph = p4[k], pl = fgeo[planes + 2 * (size_t)f4[k] + 1];
                    const DF d[4] = {{ph.x, pl.x}, {ph.y, pl.y}, {ph.z, pl.z}, {ph.w, pl.w}};
                    const int ij[10][2] = {{0, 0}, {0, 1}, {0, 2}, {0, 3}, {1, 1}, {1, 2}, {1, 3}, {2, 2}, {2, 3}, {3, 3}};
#pragma unroll
                    for (int e = 0; e < 10; ++e) {
                        const DF pr = df_mul(d[ij[e][0]], d[ij[e][1]]);
                        c[e].add(pr.hi);
                        c[e].c += pr.lo;
                    }
                } else {
                    const float p[4] = {p4[k].x, p4[k].y, p4[k].z, p4[k].w};
                    m00 += p[0] * p[0]; m01 += p[0] * p[1]; m02 += p[0] * p[2]; m03 += p[0] * p[3];
                    m11 += p[1] * p[1]; m12 += p[1] * p[2]; m13 += p[1] * p[3];
                    m22 += p[2] * p[2]; m23 += p[2] * p[3];
                    m33 += p[3] * p[3];
                }
            }
        }
        if constexpr (kComp) {  // each entry as hi (q) + lo (qlo)
            float l[10];
#pragma unroll
            for (int k = 0; k < 10; ++k) {
                const DF e = df_fast(c[k].s, c[k].c);
                c[k].s = e.hi;
                l[k] = e.lo;
            }
            m00 = c[0].s; m01 = c[1].s; m02 = c[2].s; m03 = c[3].s; m11 = c[4].s;
            m12 = c[5].s; m13 = c[6].s; m22 = c[7].s; m23 = c[8].s; m33 = c[9].s;
            Quadric L;
            L.a = make_float4(l[0], l[1], l[2], l[3]);
            L.b = make_float4(l[4], l[5], l[6], l[7]);
            L.c = make_float4(l[8], l[9], 0.f, 0.f);
            qlo[v] = L;
        }
        Quadric Q;
        Q.a = make_float4(m00, m01, m02, m03);
        Q.b = make_float4(m11, m12, m13, m22);
        Q.c = make_float4(m23, m33, 0.f, 0.f);
        q[v] = Q;
    }
}

// ------------------------------------------------------------------ edge cost (compute_edge_cost_kernel, :382-585)

// The squared lengths of the skinny term: the reference squares with the device's pow(float, int)
// (cusimp_free.cu:533,573, cusimp.cu:423,463), which on the GPU differs from x * x by one ulp for a few floats in
// a million and costs far more; kPow = false squares by multiplication (the oracle's form).
template <bool kPow>
__device__ __forceinline__ float sq_len(float x) {
    if constexpr (kPow) return pow(x, 2);
    else return x * x;
}

// The skinny sum 4*sqrt(3)*A/l01^2 + l12^2 + l20^2 + 1e-7 (only the first square divides: the reference's
// precedence), in float, or in double for the legacy round (cusimp.cu:423,463: `4.0f * sqrt(3)` takes the
// integer overload of sqrt).
template <bool kLegacy>
__device__ __forceinline__ float skinny_sum(float k4s3, float area, float p01, float p12, float p20) {
    if constexpr (kLegacy)
        return (float)((double)4.0f * sqrt(3.0) * (double)area / (double)p01 + (double)p12 + (double)p20 +
                       (double)0.0000001f);
    else
        return k4s3 * area / p01 + p12 + p20 + 0.0000001f;
}

// The term 1 - clamp(sum, 0, 1) with the reference's squares. The sum is first taken with x * x: the device's
// pow(float, int) is within 2 ulp of it (CUDA's documented powf bound) for squares in the normal range, the sum is
// monotone in each square (area >= 0) and rounding is monotone, so a sum of at least 1 + 1e-5 with x * x is at
// least 1 with the device's squares too, and the term is 0 either way. Only other sums (below the margin, tiny
// squares, NaN) are evaluated again with the device's pow.
template <bool kLegacy, bool kPow>
__device__ __forceinline__ float skinny_term(float k4s3, float area, float l01, float l12, float l20) {
    const float q01 = l01 * l01, q12 = l12 * l12, q20 = l20 * l20;
    float e = skinny_sum<kLegacy>(k4s3, area, q01, q12, q20);
    if constexpr (kPow) {
        const bool saturated = e >= 1.00001f && q01 >= 1e-30f && q12 >= 1e-30f && q20 >= 1e-30f;
        if (!saturated) e = skinny_sum<kLegacy>(k4s3, area, sq_len<true>(l01), sq_len<true>(l12), sq_len<true>(l20));
    }
    return 1.0f - rclamp(e, 0.0f, 1.0f);
}

// What one ring slot gives to the two ring sums of the edge (w, other):
// * the edge-length term (:449-484): the lengths g.x, g.y, g.z of the face's edges whose first vertex is the larger (t.x >
//   t.y, t.y > t.z, t.z > t.x: longer's bits 0, 1, 2);
// * the flip test and the skinny term q with w moved to vm, for a face without `other` (counted); ok = false where the
//   face's normal flips (the edge is invalid).
// The face t is rebuilt from w, nxt[s] and spc[s], and its corners come from the face record, so a slot costs two aligned
// 32-byte sectors of the record and contiguous per-slot words.
// The flip test dot(n_old/|n_old|, n_new/|n_new|) < 0 takes its sign from the unnormalised normals when a
// float bound proves it (|dot| > 1e-5 |n_old|_1 |n_new|_1, far above the ~1e-6 relative rounding of the
// normalised form); otherwise the normalised form is evaluated exactly as the reference does.
struct SlotTerms {
    float4 g;
    unsigned longer;
    bool counted, ok;
    float q;
};
template <bool kLegacy, bool kPow>
__device__ __forceinline__ SlotTerms slot_terms(int w, int other, V3 vm, int s, const int* __restrict__ nt,
                                                const int* __restrict__ nxt, const int2* __restrict__ spc,
                                                const float4* __restrict__ fgeo) {
    const float k4s3 = 4.0f * sqrtf(3.0f);
    const float4* r = fgeo + 4 * (size_t)nt[s];
    const int nx = nxt[s];
    const int2 pc = spc[s];
    const int4 t = pc.y == 0 ? make_int4(w, nx, pc.x, 0) : (pc.y == 1 ? make_int4(pc.x, w, nx, 0)
                                                                      : make_int4(nx, pc.x, w, 0));
    SlotTerms T;
    T.g = r[0];
    T.longer = (t.x > t.y ? 1u : 0u) | (t.y > t.z ? 2u : 0u) | (t.z > t.x ? 4u : 0u);
    T.counted = !(t.x == other || t.y == other || t.z == other);
    T.ok = true;
    T.q = 0.0f;
    if (!T.counted) return T;
    T.ok = false;
    const float4 r1 = r[1], r2 = r[2], r3 = r[3];
    const bool wx = t.x == w, wy = t.y == w, wz = t.z == w;
    const V3 n0 = wx ? vm : V3{r1.w, r2.x, r2.y}, n1 = wy ? vm : V3{r2.z, r2.w, r3.x},
             n2 = wz ? vm : V3{r3.y, r3.z, r3.w};
    const V3 ou = {r1.x, r1.y, r1.z};
    const V3 nu = vcross(vsub(n1, n0), vsub(n2, n0));
    const float du = vdot(ou, nu);
    const float bound = 1e-5f * T.g.w * (fabsf(nu.x) + fabsf(nu.y) + fabsf(nu.z));
    if (du < -bound) return T;
    if (!(du > bound)) {
        const V3 on = vdiv(ou, vnorm(ou));
        const V3 nn = vdiv(nu, vnorm(nu));
        if (vdot(on, nn) < 0) return T;
    }
    // an edge without w keeps its length (same operations as the per-face value)
    const float l01 = (wx || wy) ? vnorm(vsub(n0, n1)) : T.g.x;
    const float l12 = (wy || wz) ? vnorm(vsub(n1, n2)) : T.g.y;
    const float l20 = (wz || wx) ? vnorm(vsub(n2, n0)) : T.g.z;
    const float sh = (l01 + l12 + l20) / 2;  // triangle_area (Heron), :368-375
    const float heron = sh * (sh - l01) * (sh - l12) * (sh - l20);
    // A face with area >= l01^2 / (4 sqrt 3) makes the first quotient of the skinny sum at least 1, so the clamped
    // sum is 1 and the term exactly 0. Most faces are that fat; it is proven here from Heron's product against
    // (l01^2 / (4 sqrt 3))^2 with a 1e-4 relative margin (far above the few ulps of rounding on either side, the
    // 2-ulp difference of the device's pow and the double-precision constant of the legacy sum), which skips the
    // square root and the division. A bound that is not a normal positive number, or a NaN, takes the full path.
    const float tb = l01 * l01 * 0.144337567f;  // l01^2 / (4 sqrt 3)
    const float tb2 = tb * tb;
    if (tb2 > 1e-30f && tb2 < 1e30f && heron >= tb2 * 1.0001f) {
        T.q = 0.0f;  // the saturated term
    } else {
        const float area = sqrtf(heron);
        T.q = skinny_term<kLegacy, kPow>(k4s3, area, l01, l12, l20);
    }
    T.ok = true;
    return T;
}

// One pass over the ring of w (slots in face-index order) for both ring sums of the edge (w, other): lengths to len and
// their count to cnt, skinny terms to qa and the faces to ntri; false as soon as a face flips.
// Called for the ring of u, then of v, each sum runs in the order of the two separate loops of the reference.
template <bool kLegacy, bool kPow, class Acc>
__device__ __forceinline__ bool ring_pass(int w, int other, V3 vm, const int* __restrict__ nt_off,
                                          const int* __restrict__ nt, const int* __restrict__ nxt,
                                          const int2* __restrict__ spc, const float4* __restrict__ fgeo, Acc& len,
                                          int& cnt, Acc& qa, int& ntri) {
    const int b = nt_off[w + 1];
    for (int s = nt_off[w]; s < b; ++s) {
        const SlotTerms T = slot_terms<kLegacy, kPow>(w, other, vm, s, nt, nxt, spc, fgeo);
        if (!T.ok) return false;
        if (T.longer & 1u) { acc_add(len, T.g.x); cnt++; }
        if (T.longer & 2u) { acc_add(len, T.g.y); cnt++; }
        if (T.longer & 4u) { acc_add(len, T.g.z); cnt++; }
        if (T.counted) {
            acc_add(qa, T.q);
            ntri++;
        }
    }
    return true;
}

__device__ __forceinline__ uint32_t f2u_sat(float f) {
    return __float2uint_rz(f);  // round toward zero, saturating like the reference's uint32_t(float) on the GPU
}

// Minimiser of v^T Q v over v = (x, y, z, 1) for the quadric Q of an edge (precision mode 2, optimal placement; the
// reference places at the midpoint, cusimp_free.cu:491,687): A x = -b with A the upper 3x3 block and b the last
// column, by the adjugate. A is positive semi-definite, so its largest diagonal entry bounds its entries: a
// determinant above 1e-2 of its cube (a well-conditioned A) is solved in float, one down to 1e-10 of it (near
// singular) in double from the compensated entries (hi + lo), and a singular one (flat or cylindrical rings) keeps
// the midpoint. Returns 0 (midpoint), 1 (float) or 2 (double).
__device__ __forceinline__ int qem_optimum(const float* m, const float* lo, V3 mid, V3& x) {
    const float m00 = m[0], m01 = m[1], m02 = m[2], m03 = m[3], m11 = m[4], m12 = m[5], m13 = m[6], m22 = m[7],
                m23 = m[8];
    const float nrm = fmaxf(fabsf(m00), fmaxf(fabsf(m11), fabsf(m22)));
    const float n3 = nrm * nrm * nrm;
    const float c00 = m11 * m22 - m12 * m12, c01 = m02 * m12 - m01 * m22, c02 = m01 * m12 - m11 * m02;
    const float det = m00 * c00 + m01 * c01 + m02 * c02;
    if (nrm > 0.0f && fabsf(det) > 1e-2f * n3) {
        const float c11 = m00 * m22 - m02 * m02, c12 = m01 * m02 - m00 * m12, c22 = m00 * m11 - m01 * m01;
        x.x = -(c00 * m03 + c01 * m13 + c02 * m23) / det;
        x.y = -(c01 * m03 + c11 * m13 + c12 * m23) / det;
        x.z = -(c02 * m03 + c12 * m13 + c22 * m23) / det;
        return 1;
    }
    double d[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) d[i] = (double)m[i] + (double)lo[i];
    const double e00 = d[4] * d[7] - d[5] * d[5], e01 = d[2] * d[5] - d[1] * d[7], e02 = d[1] * d[5] - d[4] * d[2];
    const double det64 = d[0] * e00 + d[1] * e01 + d[2] * e02;
    if (nrm > 0.0f && fabs(det64) > 1e-10 * (double)n3) {
        const double e11 = d[0] * d[7] - d[2] * d[2], e12 = d[1] * d[2] - d[0] * d[5], e22 = d[0] * d[4] - d[1] * d[1];
        x.x = (float)(-(e00 * d[3] + e01 * d[6] + e02 * d[8]) / det64);
        x.y = (float)(-(e01 * d[3] + e11 * d[6] + e12 * d[8]) / det64);
        x.z = (float)(-(e02 * d[3] + e12 * d[6] + e22 * d[8]) / det64);
        return 2;
    }
    x = mid;
    return 0;
}

// The edge's quadric Q_u + Q_v: in float (mode 0), or as hi + lo by two-sum with the quadrics' own lo parts added
// (precision modes)
template <int kMode>
__device__ __forceinline__ void edge_quadric(int u, int v, const Quadric* __restrict__ q,
                                             const Quadric* __restrict__ qlo, float m[10], float mlo[10]) {
    const Quadric Qu = q[u], Qv = q[v];
    const float qu[10] = {Qu.a.x, Qu.a.y, Qu.a.z, Qu.a.w, Qu.b.x, Qu.b.y, Qu.b.z, Qu.b.w, Qu.c.x, Qu.c.y};
    const float qv[10] = {Qv.a.x, Qv.a.y, Qv.a.z, Qv.a.w, Qv.b.x, Qv.b.y, Qv.b.z, Qv.b.w, Qv.c.x, Qv.c.y};
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        if constexpr (kMode == 0) {
            m[i] = qu[i] + qv[i];
            mlo[i] = 0.0f;
        } else {
            two_sum(qu[i], qv[i], m[i], mlo[i]);
        }
    }
    if constexpr (kMode != 0) {
        const Quadric Lu = qlo[u], Lv = qlo[v];
        const float lu[10] = {Lu.a.x, Lu.a.y, Lu.a.z, Lu.a.w, Lu.b.x, Lu.b.y, Lu.b.z, Lu.b.w, Lu.c.x, Lu.c.y};
        const float lv[10] = {Lv.a.x, Lv.a.y, Lv.a.z, Lv.a.w, Lv.b.x, Lv.b.y, Lv.b.z, Lv.b.w, Lv.c.x, Lv.c.y};
#pragma unroll
        for (int i = 0; i < 10; ++i) mlo[i] += lu[i] + lv[i];
    }
}

// The cost from the two ring sums (cusimp_free.cu:449-585): the mean ring length, the quadric's value at the placement and
// the mean skinny term.
template <bool kLegacy, int kMode>
__device__ __forceinline__ uint32_t cost_of_sums(int u, int v, V3 v0, V3 v1, V3 vm, float len, int cnt, float qa, int ntri,
                                                 const Quadric* __restrict__ q, const Quadric* __restrict__ qlo, float scale,
                                                 float tres, float& raw) {
    len = len / (float)cnt / scale * tres;
    if (kLegacy) len = len + (len + vnorm(vsub(v0, v1)) / scale * tres);
    else len = len + vnorm(vsub(v0, v1)) / scale * tres;
    float m[10], mlo[10];
    edge_quadric<kMode>(u, v, q, qlo, m, mlo);  // after the ring passes: not live across them
    if (!kLegacy) qa = 5.0f * qa;  // SKINNY_TRIANGLE_PENALTY
    const float x = vm.x, y = vm.y, z = vm.z, w = 1.0f;
    float qem;
    if constexpr (kMode == 0) {
        const float m00 = m[0], m01 = m[1], m02 = m[2], m03 = m[3], m11 = m[4], m12 = m[5], m13 = m[6], m22 = m[7],
                    m23 = m[8], m33 = m[9];
        // Mat4x4::vTMv (cusimp_free.h:145-152) on the symmetric matrix
        const float c0 = m00 * x + m01 * y + m02 * z + m03 * w;
        const float c1 = m01 * x + m11 * y + m12 * z + m13 * w;
        const float c2 = m02 * x + m12 * y + m22 * z + m23 * w;
        const float c3 = m03 * x + m13 * y + m23 * z + m33 * w;
        qem = c0 * x + c1 * y + c2 * z + c3 * w;
    } else {
        // the same products with the matrix as hi + lo, each dot compensated
        const int row[4][4] = {{0, 1, 2, 3}, {1, 4, 5, 6}, {2, 5, 7, 8}, {3, 6, 8, 9}};
        const float vv[4] = {x, y, z, w};
        CSum outer;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            CSum inner;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                inner.add_prod(m[row[r][c]], vv[c]);
                inner.add_prod(mlo[row[r][c]], vv[c]);
            }
            outer.add_prod(inner.s, vv[r]);
            outer.add_prod(inner.c, vv[r]);
        }
        qem = outer.value();
    }
    const float cost = qem / (scale * scale);
    float tot;
    if constexpr (kMode == 0) {
        tot = cost + len + qa / (float)ntri * tres;
    } else {
        CSum t;
        t.add(cost);
        t.add(len);
        t.add(qa / (float)ntri * tres);
        tot = t.value();
    }
    raw = tot;
    return f2u_sat(rclamp(tot, 0.0f, kCostRange) / kCostRange * kU32MaxF);
}

// returns false when the reference leaves the stale cost in place. kLegacy: the cost of CUSimp
// (cusimp.cu:270-471): the mean ring length is counted twice (`edge_len += edge_len + |e|`) and the skinny term
// has no penalty factor. kMode (precision mode, not the reference's arithmetic): 0 the reference's float order;
// 1 quadric, ring-length, skinny and cost sums compensated (TwoSum/TwoProd, rounded once); 2 as 1 with the
// placement at the quadric's minimiser (qem_optimum) instead of the midpoint. raw: the cost before its clamp and
// quantisation; place: the placement, left as it is where there is none (no link of two vertices).
template <bool kLegacy, bool kPow, int kMode>
__device__ __forceinline__ bool edge_cost_value(int u, int v, const int* __restrict__ nt_off, const int* __restrict__ nt,
                                                const int4* __restrict__ tri, const float4* __restrict__ pos,
                                                const Quadric* __restrict__ q, const float4* __restrict__ fgeo,
                                                const int* __restrict__ nxt, const int2* __restrict__ spc, float scale,
                                                float tres, uint32_t& out, float& raw, V3& place,
                                                const Quadric* __restrict__ qlo) {
    raw = __int_as_float(0x7fc00000);  // NaN: no finite cost (invalid)
    // link condition
    int dup = 0;
    const int ua = nt_off[u], ub = nt_off[u + 1], va = nt_off[v], vb = nt_off[v + 1];
    for (int a = ua; a < ub; ++a) {
        const int iu = nxt[a];
        for (int b = va; b < vb; ++b) {
            const int iv = nxt[b];
            if (iu == iv) dup++;
            if (dup > 2) {
                out = 0xFFFFFFFFu;
                return true;
            }
        }
    }
    if (dup != 2) return false;
    typedef typename std::conditional<kMode == 0, float, CSum>::type Acc;
    const V3 v0 = v3(pos[u]), v1 = v3(pos[v]);
    float m[10], mlo[10];
    V3 vm = vdiv(vadd(v0, v1), 2.0f);
    if constexpr (kMode == 2) {
        edge_quadric<kMode>(u, v, q, qlo, m, mlo);
        qem_optimum(m, mlo, vm, vm);
    }
    place = vm;
    Acc lacc{}, qacc{};
    int cnt = 0, ntri = 0;
    if (!ring_pass<kLegacy, kPow>(u, v, vm, nt_off, nt, nxt, spc, fgeo, lacc, cnt, qacc, ntri) ||
        !ring_pass<kLegacy, kPow>(v, u, vm, nt_off, nt, nxt, spc, fgeo, lacc, cnt, qacc, ntri)) {
        out = 0xFFFFFFFFu;
        return true;
    }
    out = cost_of_sums<kLegacy, kMode>(u, v, v0, v1, vm, acc_value(lacc), cnt, acc_value(qacc), ntri, q, qlo, scale, tres, raw);
    return true;
}

// The same cost (the reference's arithmetic) by eight lanes an edge, a lane to a ring slot: the slots' terms are made side by
// side, and every lane adds them in slot order, so the bits are the same. For rounds whose edges leave the GPU idle: there a
// thread's chain over a dozen slots, two gathers each, set the time. It costs about 1.4 times the instructions. 1,280 faces
// 4.26 -> 3.84 ms, 20,480 faces 13.95 -> 12.90 ms, a height field of 286k 15.6 -> 14.8 ms.
constexpr int kCostLanes = 8;
// largest edge bound that takes it: against 2^15, 2^16, 2^18 and 2^19 the height field of 286k ran 1.04, 1.01, 1.02 and 1.08 times
// as fast, the others the same or less so
constexpr int kCostLanesEdges = 1 << 17;

template <bool kPow>
__device__ __forceinline__ bool ring_pass_lanes(int w, int other, V3 vm, int l, unsigned group, const int* __restrict__ nt_off,
                                                const int* __restrict__ nt, const int* __restrict__ nxt,
                                                const int2* __restrict__ spc, const float4* __restrict__ fgeo, float& len,
                                                int& cnt, float& qa, int& ntri) {
    const int a = nt_off[w], b = nt_off[w + 1];
    for (int s0 = a; s0 < b; s0 += kCostLanes) {
        SlotTerms T;
        T.g = make_float4(0.f, 0.f, 0.f, 0.f);
        T.longer = 0;
        T.counted = false;
        T.ok = true;
        T.q = 0.f;
        if (s0 + l < b) T = slot_terms<false, kPow>(w, other, vm, s0 + l, nt, nxt, spc, fgeo);
        if (__any_sync(group, !T.ok)) return false;
        const unsigned bits = T.longer | (T.counted ? 8u : 0u);
        const int m = min(kCostLanes, b - s0);
        for (int k = 0; k < m; ++k) {
            const unsigned f = __shfl_sync(group, bits, k, kCostLanes);
            const float x = __shfl_sync(group, T.g.x, k, kCostLanes), y = __shfl_sync(group, T.g.y, k, kCostLanes),
                        z = __shfl_sync(group, T.g.z, k, kCostLanes), q = __shfl_sync(group, T.q, k, kCostLanes);
            if (f & 1u) len += x;
            if (f & 2u) len += y;
            if (f & 4u) len += z;
            cnt += __popc(f & 7u);
            if (f & 8u) {
                qa += q;
                ntri++;
            }
        }
    }
    return true;
}

template <bool kPow>
__device__ __forceinline__ bool edge_cost_lanes(int u, int v, int l, unsigned group, const int* __restrict__ nt_off,
                                                const int* __restrict__ nt, const float4* __restrict__ pos,
                                                const Quadric* __restrict__ q, const float4* __restrict__ fgeo,
                                                const int* __restrict__ nxt, const int2* __restrict__ spc, float scale,
                                                float tres, uint32_t& out) {
    const int ua = nt_off[u], ub = nt_off[u + 1], va = nt_off[v], vb = nt_off[v + 1];
    int dup = 0;
    for (int a = ua + l; a < ub; a += kCostLanes) {
        const int iu = nxt[a];
        for (int b = va; b < vb; ++b) dup += iu == nxt[b];
    }
    for (int o = kCostLanes / 2; o > 0; o >>= 1) dup += __shfl_xor_sync(group, dup, o);
    if (dup > 2) {
        out = 0xFFFFFFFFu;
        return true;
    }
    if (dup != 2) return false;
    const V3 v0 = v3(pos[u]), v1 = v3(pos[v]);
    const V3 vm = vdiv(vadd(v0, v1), 2.0f);
    float len = 0.f, qa = 0.f;
    int cnt = 0, ntri = 0;
    if (!ring_pass_lanes<kPow>(u, v, vm, l, group, nt_off, nt, nxt, spc, fgeo, len, cnt, qa, ntri) ||
        !ring_pass_lanes<kPow>(v, u, vm, l, group, nt_off, nt, nxt, spc, fgeo, len, cnt, qa, ntri)) {
        out = 0xFFFFFFFFu;
        return true;
    }
    float raw;
    out = cost_of_sums<false, 0>(u, v, v0, v1, vm, len, cnt, qa, ntri, q, nullptr, scale, tres, raw);
    return true;
}

template <bool kPow>
__global__ void __launch_bounds__(kT) k_edge_cost_lanes(const RoundCounters* rc, const int* __restrict__ eorder,
                                                        const int2* __restrict__ edges, const int* __restrict__ nt_off,
                                                        const int* __restrict__ nt, const float4* __restrict__ pos,
                                                        const Quadric* __restrict__ q, const float4* __restrict__ fgeo,
                                                        const int* __restrict__ nxt, const int2* __restrict__ spc,
                                                        const unsigned char* __restrict__ invalid, uint32_t* cost,
                                                        unsigned long long* vmin, const float* d_scale, float tres,
                                                        int is_stuck_host, const int* is_stuck_dev) {
    pdl_wait();
    const int is_stuck = is_stuck_dev ? *is_stuck_dev : is_stuck_host;
    const float scale = *d_scale;
    const int n = rc->n_edges, lane = threadIdx.x & 31, l = lane % kCostLanes;
    const unsigned group = ((1u << kCostLanes) - 1u) << (lane - l);
    for (long long i = gtid() / kCostLanes; i < n; i += gstride() / kCostLanes) {
        const int e = eorder[i];
        const int2 ed = edges[e];
        const int u = ed.x, v = ed.y;
        uint32_t c = 0;
        bool write = false;
        if (invalid[u] && invalid[v]) {
            c = 0xFFFFFFFFu;
            write = true;
        } else if (!is_stuck) {
            write = edge_cost_lanes<kPow>(u, v, l, group, nt_off, nt, pos, q, fgeo, nxt, spc, scale, tres, c);
        }
        if (l != 0) continue;
        if (write) cost[e] = c;
        else c = cost[e];  // stale value of an earlier round
        const unsigned long long key = ((unsigned long long)c << 32) | (unsigned)e;
        atomicMin(&vmin[u], key);
        atomicMin(&vmin[v], key);
    }
}

// kBatch: many meshes in one vertex numbering; the scale and is_stuck of an edge's mesh come from per-mesh arrays
// (mesh of the lower vertex from vmesh) instead of d_scale and the single flag. kOut: raw_out / place_out are
// written (probe and precision modes; a compile-time flag so that the default variant keeps its register budget).
template <bool kLegacy, bool kPow, bool kBatch, int kMode = 0, bool kOut = false>
__global__ void __launch_bounds__(kT) k_edge_cost(const RoundCounters* rc, const int* __restrict__ eorder,
                                                  const int2* __restrict__ edges,
                                                  const int* __restrict__ nt_off, const int* __restrict__ nt,
                                                  const int4* __restrict__ tri, const float4* __restrict__ pos,
                                                  const Quadric* __restrict__ q, const float4* __restrict__ fgeo,
                                                  const int* __restrict__ nxt, const int2* __restrict__ spc,
                                                  const unsigned char* __restrict__ invalid,
                                                  uint32_t* cost, unsigned long long* vmin, const float* d_scale,
                                                  float tres, int is_stuck_host, const int* is_stuck_dev,
                                                  const int* __restrict__ vmesh, const int* __restrict__ mesh_stuck,
                                                  float* raw_out, float4* place_out,
                                                  const Quadric* __restrict__ qlo) {
    pdl_wait();
    int is_stuck = 0;
    float scale = 0.0f;
    if constexpr (!kBatch) {
        is_stuck = is_stuck_dev ? *is_stuck_dev : is_stuck_host;
        scale = *d_scale;
    }
    const int n = rc->n_edges;
    for (int i = gtid(); i < n; i += gstride()) {
        const int e = eorder[i];  // edges grouped by their lower vertex: neighbouring threads share rings
        const int2 ed = edges[e];
        const int u = ed.x, v = ed.y;
        if constexpr (kBatch) {
            const int m = vmesh[u];
            scale = d_scale[m];
            is_stuck = mesh_stuck[m];
        }
        uint32_t c = 0;
        bool write;
        V3 place;
        // an edge that may collapse by the stale cost of an earlier round (no link of two, a stuck round) has no placement
        // of its own: the midpoint
        if constexpr (kOut) place = vdiv(vadd(v3(pos[u]), v3(pos[v])), 2.0f);
        if (!kLegacy && invalid[u] && invalid[v]) {
            c = 0xFFFFFFFFu;
            write = true;
        } else if (!kLegacy && is_stuck) {
            write = false;
        } else {
            float raw;
            write = edge_cost_value<kLegacy, kPow, kMode>(u, v, nt_off, nt, tri, pos, q, fgeo, nxt, spc, scale, tres, c,
                                                          raw, place, qlo);
            if constexpr (kOut) {
                if (raw_out) raw_out[e] = write ? raw : __int_as_float(0x7fc00000);
            }
        }
        if constexpr (kOut) {
            if (place_out) place_out[e] = make_float4(place.x, place.y, place.z, 0.f);
        }
        if (write) cost[e] = c;
        else c = cost[e];  // stale value of an earlier round
        const unsigned long long key = ((unsigned long long)c << 32) | (unsigned)e;
        atomicMin(&vmin[u], key);
        atomicMin(&vmin[v], key);
    }
}

// ------------------------------------------------------------------ collapse (collapse_edge_kernel, :639-774)
__device__ __forceinline__ bool is_skinny(V3 p, V3 q, V3 r) {  // :617-637
    const V3 pq = vsub(q, p), pr = vsub(r, p), qr = vsub(r, q);
    const float lpq = sqrtf(vdot(pq, pq)), lpr = sqrtf(vdot(pr, pr)), lqr = sqrtf(vdot(qr, qr));
    const float maxl = fmaxf(lpq, fmaxf(lpr, lqr));
    const V3 c = {pq.y * pr.z - pq.z * pr.y, pq.z * pr.x - pq.x * pr.z, pq.x * pr.y - pq.y * pr.x};
    const float thr = (float)(1e-6 * (double)maxl * (double)maxl);
    const float area = 0.5f * sqrtf(c.x * c.x + c.y * c.y + c.z * c.z);
    return area < thr;
}


// An edge wins when its key is the least over every face that touches it, that is when no vertex of the rings of u and v
// has a smaller one in vmin (the least key of its edges; a face's key is the least of its three vertices', and u and v
// lie in all faces of their rings). vmin[u] and vmin[v] alone reject nearly every edge; the reference's per-face keys
// (:587-610) are not made.
// A warp reads its edges in order and keeps those that pass, and takes them four at a time, eight lanes to an edge and a
// lane to a ring face: the ring's keys, the collapse and the skinny test (kRestore) are chains of two gathers instead of two
// per face of both rings. Taken by one thread each, where the edge was found, they set the kernel's time (129 us of a mean
// round of 1.1 ms from 5.24M faces, 17 us of one of 0.14 ms from 1,280).
// A collapse that leaves a skinny face is undone in the reference; here its faces are not written (the winners' rings
// share no face, and no winner's ring holds another's endpoint, so no other collapse shows in the test).
// kRestore = false: CUSimp's collapse (cusimp.cu:512-585), without the skinny-ring restore
// kOpt (precision mode 2): the collapse places at the edge's precomputed placement instead of the midpoint
constexpr int kCollapseLanes = 8;

// The face t of the ring of u (side 0) or v (side 1) after the collapse of (u, v) onto u: x = -1 when it dies
__device__ __forceinline__ int4 collapsed_face(int4 t, int u, int v, int side) {
    const int other = side ? u : v;
    if (t.x == other || t.y == other || t.z == other) return make_int4(-1, -1, -1, 0);
    if (side) {
        // a face that holds v twice is in the ring twice, and dies at the second visit, which finds u
        if ((t.x == v) + (t.y == v) + (t.z == v) > 1) return make_int4(-1, -1, -1, 0);
        if (t.x == v) t.x = u;
        else if (t.y == v) t.y = u;
        else if (t.z == v) t.z = u;
    }
    return t;
}

template <bool kRestore, bool kOpt>
__device__ __forceinline__ void try_collapse(int e, unsigned long long key, int l, unsigned group,
                                             const int2* __restrict__ edges,
                                             const unsigned long long* __restrict__ vmin, const int* __restrict__ nxt,
                                             const int2* __restrict__ spc, const int* __restrict__ nt_off,
                                             const int* __restrict__ nt, int4* tri, float4* pos, int* occ, int* win,
                                             const float4* __restrict__ place) {
    const int2 ed = edges[e];
    const int u = ed.x, v = ed.y;
    const int a[2] = {nt_off[u], nt_off[v]}, b[2] = {nt_off[u + 1], nt_off[v + 1]};
    bool low = false;
#pragma unroll
    for (int side = 0; side < 2; ++side)
        for (int s = a[side] + l; s < b[side]; s += kCollapseLanes) low |= vmin[nxt[s]] < key || vmin[spc[s].x] < key;
    if (__any_sync(group, low)) return;
    V3 vm = vdiv(vadd(v3(pos[u]), v3(pos[v])), 2.0f);
    if constexpr (kOpt) vm = v3(place[e]);
    if constexpr (kRestore) {
        // positions as after the collapse: u at vm, v at the origin
        auto at = [&](int i) { return i == u ? vm : i == v ? V3{0.f, 0.f, 0.f} : v3(pos[i]); };
        bool skinny = false;
#pragma unroll
        for (int side = 0; side < 2; ++side)
            for (int s = a[side] + l; s < b[side]; s += kCollapseLanes) {
                const int4 t = collapsed_face(tri[nt[s]], u, v, side);
                if (t.x != -1 && is_skinny(at(t.x), at(t.y), at(t.z))) skinny = true;
            }
        skinny = __any_sync(group, skinny);
        if (l == 0) win[e] = 1;
        if (skinny) return;
    } else {
        if (l == 0) win[e] = 1;
    }
    __syncwarp(group);  // every lane has read what the first one writes
    if (l == 0) {
        pos[u] = make_float4(vm.x, vm.y, vm.z, 0.f);
        pos[v] = make_float4(0.f, 0.f, 0.f, 0.f);
        occ[v] = 0;
    }
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        for (int s = a[side] + l; s < b[side]; s += kCollapseLanes) {
            const int f = nt[s];
            const int4 t = tri[f], c = collapsed_face(t, u, v, side);
            if (t.x != -1 && (c.x != t.x || c.y != t.y || c.z != t.z)) tri[f] = c;
        }
        __syncwarp(group);  // the faces of both rings have died before v's ring is read
    }
}

template <bool kRestore, bool kOpt>
__global__ void __launch_bounds__(kT) k_collapse(RoundCounters* rc, const int2* __restrict__ edges,
                                                 const uint32_t* __restrict__ cost, uint32_t collapse_t,
                                                 const unsigned long long* __restrict__ vmin, const int* __restrict__ nxt,
                                                 const int2* __restrict__ spc, const int* __restrict__ nt_off,
                                                 const int* __restrict__ nt, int4* tri, float4* pos, int* occ, int* win,
                                                 const float4* __restrict__ place) {
    pdl_wait();
    constexpr int kGroups = 32 / kCollapseLanes;
    __shared__ unsigned long long queue[kT / 32][32 + kGroups];  // keys (cost << 32 | edge) of the warp's candidates
    const int n = rc->n_edges;
    const int lane = threadIdx.x & 31, l = lane % kCollapseLanes, g = lane / kCollapseLanes;
    const unsigned group = ((1u << kCollapseLanes) - 1u) << (g * kCollapseLanes);
    unsigned long long* q = queue[threadIdx.x >> 5];
    int held = 0;
    if (gtid() == 0) win[n] = 0;
    for (int i0 = gtid() - lane; i0 < n; i0 += gstride()) {
        const int e = i0 + lane;
        bool candidate = false;
        unsigned long long key = 0;
        if (e < n) {
            win[e] = 0;
            const uint32_t c = cost[e];
            if (c <= collapse_t) {
                const int2 ed = edges[e];
                key = ((unsigned long long)c << 32) | (unsigned)e;
                candidate = vmin[ed.x] == key && vmin[ed.y] == key;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, candidate);
        if (candidate) q[held + __popc(m & ((1u << lane) - 1u))] = key;
        held += __popc(m);
        const bool last = i0 + gstride() >= n;
        __syncwarp();
        int done = 0;
        while (held - done >= (last ? 1 : kGroups)) {
            if (done + g < held) {
                const unsigned long long k = q[done + g];
                try_collapse<kRestore, kOpt>((int)(unsigned)k, k, l, group, edges, vmin, nxt, spc, nt_off, nt, tri, pos,
                                             occ, win, place);
            }
            __syncwarp();
            done = min(done + kGroups, held);
        }
        // the rest, fewer than a warp takes at once, to the front
        const unsigned long long rest = done + lane < held ? q[done + lane] : 0ull;
        __syncwarp();
        if (done + lane < held) q[lane] = rest;
        __syncwarp();
        held -= done;
    }
}

// remove_line_edge_collapse (:234-274), applied in edge order by one thread when any coincident edge exists;
// then the collapsed-list bookkeeping of forward() (:1004-1016).
__device__ void line_apply(RoundCounters* rc, const int2* __restrict__ edges, const int* __restrict__ nt_off,
                           const int* __restrict__ nt, int4* tri, float4* pos, int* occ, int* collapsed, int cap) {
    const int h = rc->n_win;
    int k = h;
    if (*(volatile int*)&rc->n_line > 0) {
        const int n = rc->n_edges;
        for (int e = 0; e < n; ++e) {
            const int2 ed = edges[e];
            const float4 p = pos[ed.x], q = pos[ed.y];
            if (!(p.x == q.x && p.y == q.y && p.z == q.z)) continue;
            if (k >= cap) {
                atomicOr(&rc->status, kErrCapacity);
                break;
            }
            collapsed[k++] = e;
            pos[ed.y] = make_float4(0.f, 0.f, 0.f, 0.f);
            occ[ed.y] = 0;
            rewire(ed.x, ed.y, nt_off, nt, tri);
        }
    }
    rc->n_collapsed = k;
    const int roundup = ((h + 511) / 512) * 512;
    rc->n_considered = (h == 0) ? 0 : (k < roundup ? k : roundup);
}

// After the collapses, in one launch: the winners' list in edge order, the faces that became degenerate removed
// (:218-232), the edges with coincident endpoints counted in rc->n_line, and, with kLines, line_apply by the block that
// finishes last (rc->pad[4] counts them; zero at a round's start). The three passes touch different arrays.
template <bool kLines>
__global__ void __launch_bounds__(kT) k_after_collapse(RoundCounters* rc, const int* __restrict__ scan, int* collapsed,
                                                       const int2* __restrict__ edges, const int* __restrict__ nt_off,
                                                       const int* __restrict__ nt, int4* tri, float4* pos, int* occ,
                                                       int line_cap) {
    pdl_wait();
    const int ne = rc->n_edges, nf = rc->n_tris;
    int found = 0;
    for (int e = gtid(); e < ne; e += gstride()) {
        if (scan[e + 1] != scan[e]) collapsed[scan[e]] = e;
        const int2 ed = edges[e];
        const float4 p = pos[ed.x], q = pos[ed.y];
        if (p.x == q.x && p.y == q.y && p.z == q.z) found = 1;
    }
    for (int f = gtid(); f < nf; f += gstride()) {
        const int4 t = tri[f];
        if (face_killed(t)) continue;
        if (t.x == t.y || t.y == t.z || t.z == t.x) tri[f] = make_int4(-1, -1, -1, 0);
    }
    if (__any_sync(0xffffffffu, found) && (threadIdx.x & 31) == 0) atomicAdd(&rc->n_line, 1);
    if constexpr (kLines) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&rc->pad[4], 1) == (int)gridDim.x - 1) {
                __threadfence();
                line_apply(rc, edges, nt_off, nt, tri, pos, occ, collapsed, line_cap);
            }
        }
    }
}

// ------------------------------------------------------------------ rollback
// Eight lanes a collapsed edge, a lane to a slot of each ring: one thread an edge was a chain over a dozen slots (a height
// field of 286k 14.8 -> 14.7 ms, 20,480 faces 12.9 -> 12.8 ms)
constexpr int kRingLanes = 8;

__global__ void k_mark_query(const RoundCounters* rc, const int* __restrict__ collapsed, const int2* __restrict__ edges,
                             const int* __restrict__ nt_off, const int* __restrict__ nt, int* qflag) {
    pdl_wait();
    const int n = rc->n_considered;
    const int l = threadIdx.x % kRingLanes;
    for (long long c = gtid() / kRingLanes; c < n; c += gstride() / kRingLanes) {
        const int2 ed = edges[collapsed[c]];
        for (int s = nt_off[ed.x] + l; s < nt_off[ed.x + 1]; s += kRingLanes) qflag[nt[s]] = 1;
        for (int s = nt_off[ed.y] + l; s < nt_off[ed.y + 1]; s += kRingLanes) qflag[nt[s]] = 1;
    }
}

// with fflags: also the faces that the compaction keeps (k_live_flags)
__global__ void k_undo_check(RoundCounters* rc, const int* __restrict__ collapsed, const int2* __restrict__ edges,
                             const int* __restrict__ nt_off, const int* __restrict__ nt, const unsigned char* __restrict__ hit,
                             int* uflag, const int4* __restrict__ tri, int* fflags) {
    pdl_wait();
    if (fflags) {
        const int nf = rc->n_tris;
        for (int f = gtid(); f < nf; f += gstride()) fflags[f] = (tri[f].x >= 0) ? 1 : 0;
        if (gtid() == 0) fflags[nf] = 0;
    }
    const int n = rc->n_considered;
    if (gtid() == 0) uflag[n] = 0;
    const int l = threadIdx.x % kRingLanes;
    const unsigned group = ((1u << kRingLanes) - 1u) << ((threadIdx.x & 31) - l);
    for (long long c = gtid() / kRingLanes; c < n; c += gstride() / kRingLanes) {
        const int2 ed = edges[collapsed[c]];
        int f = 0;
        for (int s = nt_off[ed.x] + l; s < nt_off[ed.x + 1]; s += kRingLanes) f |= hit[nt[s]];
        for (int s = nt_off[ed.y] + l; s < nt_off[ed.y + 1]; s += kRingLanes) f |= hit[nt[s]];
        f = __any_sync(group, f);
        if (l == 0) uflag[c] = f ? 1 : 0;
    }
}

__device__ __forceinline__ void after_check(RoundCounters* rc) {
    const int nu = rc->n_undo;
    if (rc->passes < 8) rc->undo_per_pass[rc->passes] = nu;
    rc->passes += 1;
    rc->n_vertices_undo += 2 * nu;
}

__global__ void k_after_check(RoundCounters* rc) {
    pdl_wait();
    after_check(rc);
}

// undo_collapse_kernel (:829-867) + rearrange_index_of_undo_vertices (:869-878). The map is the compaction
// map of the previous call, as in the reference.
__global__ void k_undo_apply(RoundCounters* rc, const int* __restrict__ collapsed, const int* __restrict__ uscan,
                             const int2* __restrict__ edges, const int* __restrict__ nt_off, const int* __restrict__ nt,
                             int4* tri, const int4* __restrict__ orig_tri, float4* pos, const float4* __restrict__ orig_pos,
                             int* occ, int* tmp_undo, int* undo_list, const int* __restrict__ pts_map, int map_len,
                             int list_cap) {
    pdl_wait();
    const int n = rc->n_considered;
    const int first = rc->first_undo;
    for (int c = gtid(); c < n; c += gstride()) {
        if (uscan[c + 1] == uscan[c]) continue;
        const int a = uscan[c];
        const int2 ed = edges[collapsed[c]];
        const int u = ed.x, v = ed.y;
        occ[v] = 1;
        pos[u] = orig_pos[u];
        pos[v] = orig_pos[v];
        restore_ring(u, nt_off, nt, tri, orig_tri);
        restore_ring(v, nt_off, nt, tri, orig_tri);
        if (first + 2 * a + 1 < list_cap) {
            tmp_undo[2 * a] = u;
            tmp_undo[2 * a + 1] = v;
            undo_list[first + 2 * a] = (u < map_len) ? pts_map[u] : 0;
            undo_list[first + 2 * a + 1] = (v < map_len) ? pts_map[v] : 0;
        } else {
            atomicOr(&rc->status, kErrCapacity);
        }
    }
}

__global__ void k_after_apply(RoundCounters* rc) { pdl_wait(); rc->first_undo += 2 * rc->n_undo; }

// ------------------------------------------------------------------ outputs
__global__ void k_live_flags(const RoundCounters* rc, const int4* __restrict__ tri, int* flags) {
    pdl_wait();
    const int n = rc->n_tris;
    for (int f = gtid(); f < n; f += gstride()) flags[f] = (tri[f].x >= 0) ? 1 : 0;
    if (gtid() == 0) flags[n] = 0;
}

// check: also the counters after an intersection check (k_after_check). remap: also the carried tree's leaves in the
// next round's face numbering.
__global__ void k_compact_mesh(RoundCounters* rc, const float4* __restrict__ pos, const int* __restrict__ occ,
                               const int* __restrict__ pts_map, const int4* __restrict__ tri, const int* __restrict__ fscan,
                               float4* out_pos, int4* out_tri, int check, BvhRemap remap) {
    pdl_wait();
    if (remap.leaves) {
        const int n = *remap.leaves;
        for (int i = gtid(); i < n; i += gstride()) {
            const int f = remap.leaf_face[i];
            remap.next[i] = (f >= 0 && fscan[f + 1] != fscan[f]) ? fscan[f] : -1;
        }
    }
    const int np = rc->n_pts, nf = rc->n_tris;
    for (int v = gtid(); v < np; v += gstride())
        if (occ[v]) out_pos[pts_map[v]] = pos[v];
    for (int f = gtid(); f < nf; f += gstride()) {
        if (fscan[f + 1] == fscan[f]) continue;
        const int4 t = tri[f];
        out_tri[fscan[f]] = make_int4(pts_map[t.x], pts_map[t.y], pts_map[t.z], 0);
    }
    if (gtid() == 0) {
        rc->n_pts_out = pts_map[np];
        rc->n_tris_out = fscan[nf];
        if (check) after_check(rc);
    }
}

__global__ void k_export_round(int np, int nf, const float4* __restrict__ pos, const int4* __restrict__ tri,
                               const int* __restrict__ occ, const int* __restrict__ pts_map, const int* __restrict__ undo,
                               float* verts, int* tris, int* vocc, int* vmap, int* vundo, int nu) {
    pdl_wait();
    for (int v = gtid(); v < np; v += gstride()) {
        const float4 p = pos[v];
        verts[3 * v] = p.x;
        verts[3 * v + 1] = p.y;
        verts[3 * v + 2] = p.z;
        if (vocc) vocc[v] = occ[v];
        if (vmap) vmap[v] = pts_map[v];
    }
    for (int f = gtid(); f < nf; f += gstride()) {
        const int4 t = tri[f];
        tris[3 * f] = t.x;
        tris[3 * f + 1] = t.y;
        tris[3 * f + 2] = t.z;
    }
    if (vundo)
        for (int a = gtid(); a < nu; a += gstride()) vundo[a] = undo[a];
}

__global__ void k_export_mesh(int np, int nf, const float4* __restrict__ pos, const int4* __restrict__ tri,
                              const float* __restrict__ add, float* verts, int* tris) {
    pdl_wait();
    const float ax = add ? add[0] : 0.f, ay = add ? add[1] : 0.f, az = add ? add[2] : 0.f;
    for (int v = gtid(); v < np; v += gstride()) {
        const float4 p = pos[v];
        verts[3 * v] = p.x + ax;
        verts[3 * v + 1] = p.y + ay;
        verts[3 * v + 2] = p.z + az;
    }
    for (int f = gtid(); f < nf; f += gstride()) {
        const int4 t = tri[f];
        tris[3 * f] = t.x;
        tris[3 * f + 1] = t.y;
        tris[3 * f + 2] = t.z;
    }
}

// ================================================================== device-driven rounds
// The same steps as the host-sized launchers, with every size read from the device (LoopState, RoundCounters),
// so that one captured graph serves every round of a size class.

// The start of a round in one launch. With r.next (device-driven rounds): *ls = *next, the round's counters as forward()
// sets them (a stuck round starts its undo list with the carried-over entries), the invalid table cleared when undo
// vertices are carried into a round that is not stuck (cusimp_free.cu:905-908), and the previous compaction map kept;
// the sizes come from *next, since the counters are written here. Without: the sizes are rc's. Then the round's
// arrays.
__global__ void k_round_prologue_dev(RoundStart r) {
    pdl_wait();
    int nm = 0, np, nf;
    if (r.next) {
        const LoopState L = *r.next;
        nm = np = L.np;
        nf = L.nf;
        if (gtid() == 0) {
            *r.ls = L;
            RoundCounters z = {};
            z.n_pts = L.np;
            z.n_tris = L.nf;
            if (L.is_stuck) {
                z.first_undo = L.nu;
                z.n_vertices_undo = L.nu;
            }
            *r.rc = z;
        }
        if (!L.is_stuck && L.nu != 0)
            for (int i = gtid(); i < r.invalid_len; i += gstride()) r.invalid[i] = 0;
    } else {
        np = r.rc->n_pts;
        nf = r.rc->n_tris;
    }
    const int n = max(np + 1, nf + 1);
    for (int i = gtid(); i < n; i += gstride()) {
        if (i < nm) r.pts_map_prev[i] = r.pts_map[i];
        if (i < np) {
            const float4 p = r.pts_in[i];
            r.pos[i] = p;
            r.orig_pos[i] = p;
            r.occ[i] = 1;
        } else if (i == np) {
            r.occ[np] = 0;
        }
        if (i <= np) {
            r.valence[i] = r.vedges[i] = 0;
            r.vmin[i] = ~0ull;
        }
        if (i < nf) {
            const int4 t = r.tri_in[i];
            r.tri[i] = t;
            r.orig_tri[i] = t;
        }
        if (i <= nf) r.qflag[i] = 0;
    }
}

// After compaction: the next round's state (pamo/__init__.py:131-159: sizes, undo vertices, the no-progress
// count and is_stuck) computed from this round's start state; recomputing it after an undo pass is harmless.
// Also the undo vertices carried to the next round (the host loop's copy of the previous undo list).
__global__ void k_round_end(const RoundCounters* rc, const LoopState* ls, LoopState* next, const int* __restrict__ undo_list,
                            int* undo_in, int undo_cap) {
    pdl_wait();
    const int n = min(rc->n_vertices_undo, undo_cap);
    for (int i = gtid(); i < n; i += gstride()) undo_in[i] = undo_list[i];
    if (gtid() != 0) return;
    LoopState L = *ls;
    const int nf = rc->n_tris_out;
    if (nf == L.nf) {
        L.count += 1;
    } else {
        L.count = 0;
        L.is_stuck = 0;
    }
    if (L.count >= 2) L.is_stuck = 1;
    L.np = rc->n_pts_out;
    L.nf = nf;
    L.nu = rc->n_vertices_undo;
    *next = L;
}

}  // namespace

// ================================================================== host launchers
Feistel make_feistel(unsigned long long m) {
    Feistel fb{};
    fb.size = feistel_size(m);
    unsigned long long x = 1;  // minstd_rand, default seed
    for (int r = 0; r < 24; ++r) {
        x = (x * 48271ull) % 2147483647ull;
        fb.key[r] = (uint32_t)x;
    }
    fb.n = 1ull << (fb.size.lbits + fb.size.rbits);
    fb.m = m;
    return fb;
}

void launch_undo_bookkeeping(const int* verts_undo, int n_verts_undo, int is_stuck, int* tmp_undo, int* undo_list,
                             const int* pts_map, int pts_map_len, unsigned char* invalid, int invalid_len, cudaStream_t s) {
    if (is_stuck) {
        if (n_verts_undo > 0)
            pdl(k_undo_stuck, grid_for(n_verts_undo, kT), kT, 0, s)(verts_undo, n_verts_undo, tmp_undo, undo_list, pts_map,
                                                                   pts_map_len); note_launch();
    } else if (n_verts_undo != 0) {
        cudaMemsetAsync(invalid, 0, invalid_len, s);
    }
    if (n_verts_undo > 0)
        pdl(k_invalid_mark, grid_for(n_verts_undo, kT), kT, 0, s)(verts_undo, n_verts_undo, invalid, invalid_len); note_launch();
}

void launch_load_points(const float* pts, int n, float4* pos, float4* orig_pos, int* occ, cudaStream_t s) {
    pdl(k_load_points, grid_for(n, kT), kT, 0, s)(pts, n, pos, orig_pos, occ); note_launch();
}
void launch_load_points4(const float4* pts, int n, float4* pos, float4* orig_pos, int* occ, cudaStream_t s) {
    pdl(k_load_points4, grid_for(n, kT), kT, 0, s)(pts, n, pos, orig_pos, occ); note_launch();
}
void launch_load_tris(const int* tris, int n, int n_pts, int4* tri, RoundCounters* rc, cudaStream_t s) {
    pdl(k_load_tris, grid_for(n, kT), kT, 0, s)(tris, n, n_pts, tri, rc); note_launch();
}
void launch_load_tris4(const int4* tris, int n, int4* tri, cudaStream_t s) {
    pdl(k_copy4, grid_for(n, kT), kT, 0, s)(tris, tri, n); note_launch();
}
void launch_copy_tris(const int4* src, int4* dst, int n, cudaStream_t s) {
    pdl(k_copy4, grid_for(n, kT), kT, 0, s)(src, dst, n); note_launch();
}
void launch_shuffle_tris(const Feistel& fb, int* flags, int* scan_scratch, int4* src, int4* dst, int n, cudaStream_t s,
                         int* err) {
    (void)n;
    const int g = grid_for((long long)fb.n, kT);
    pdl(k_shuffle_flags, g, kT, 0, s)(fb, flags); note_launch();
    exclusive_scan(flags, flags, nullptr, (int)fb.n + 1, nullptr, scan_scratch, s, err, 0);
    pdl(k_shuffle_gather, g, kT, 0, s)(fb, flags, src, dst); note_launch();
}

void launch_face_counts(const int4* tri, const RoundCounters* rc, int n_tris_bound, int* valence, int* ecount,
                        int* vedges, cudaStream_t s, const float4* pos, float4* fgeo, int2* rank, bool plane_df,
                        const UndoBook& book) {
    pdl(k_face_counts, grid_for(n_tris_bound, kT), kT, 0, s)(tri, rc, valence, ecount, vedges, pos, fgeo,
                                                            plane_df ? 1 : 0, rank, book);
    note_launch();
}
void launch_fill_adjacency(const int4* tri, RoundCounters* rc, int n_tris_bound, const int* nt_off, const int2* rank,
                           int* nt, const int* edge_off, int2* edges, const int* voff, int* eorder, cudaStream_t s,
                           int* d_cap) {
    pdl(k_fill_adjacency, grid_for(n_tris_bound, kT), kT, 0, s)(tri, rc, nt_off, rank, nt, edge_off, edges, voff, eorder,
                                                               d_cap);
    note_launch();
}
void launch_ring_quadrics(const RoundCounters* rc, int n_pts_bound, const int* nt_off, int* nt, const int4* tri,
                          const float4* fgeo, Quadric* q, int* nxt, int2* spc, cudaStream_t s, Quadric* qlo,
                          uint32_t* cost, int cost_len) {
    const int g = grid_for(n_pts_bound, kT);
    if (qlo) pdl(k_ring_quadrics<true>, g, kT, 0, s)(rc, nt_off, nt, tri, fgeo, q, nxt, spc, qlo, cost, cost_len);
    else pdl(k_ring_quadrics<false>, g, kT, 0, s)(rc, nt_off, nt, tri, fgeo, q, nxt, spc, nullptr, cost, cost_len);
    note_launch();
}
void launch_edge_cost(const RoundCounters* rc, int n_edges_bound, const int* eorder, const int2* edges, const int* nt_off,
                      const int* nt, const int4* tri, const float4* pos, const Quadric* q, const float4* fgeo,
                      const int* nxt, const int2* spc, const unsigned char* invalid, uint32_t* cost,
                      unsigned long long* vmin,
                      const float* d_scale, float tres, int is_stuck, cudaStream_t s, const int* is_stuck_dev, bool legacy,
                      bool device_pow, int mode, float* raw, float4* place, const Quadric* qlo) {
    if (!legacy && mode == 0 && !raw && !place && n_edges_bound <= kCostLanesEdges) {
        const int gl = grid_for((long long)kCostLanes * n_edges_bound, kT);
        pdl(device_pow ? k_edge_cost_lanes<true> : k_edge_cost_lanes<false>, gl, kT, 0, s)(
            rc, eorder, edges, nt_off, nt, pos, q, fgeo, nxt, spc, invalid, cost, vmin, d_scale, tres, is_stuck, is_stuck_dev);
        note_launch();
        return;
    }
    const int g = grid_for(n_edges_bound, kT);
#define PAMO_COST_MODE(M, P, O)                                                                                      \
    pdl(k_edge_cost<false, P, false, M, O>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt,       \
                                                        spc, invalid, cost, vmin, d_scale, tres, is_stuck, is_stuck_dev,  \
                                                        nullptr, nullptr, raw, place, qlo)
    if (!legacy && mode == 1) {
        if (raw || place) {
            if (device_pow) PAMO_COST_MODE(1, true, true);
            else PAMO_COST_MODE(1, false, true);
        } else {
            if (device_pow) PAMO_COST_MODE(1, true, false);
            else PAMO_COST_MODE(1, false, false);
        }
        note_launch();
        return;
    }
    if (!legacy && mode == 2) {
        if (device_pow) PAMO_COST_MODE(2, true, true);
        else PAMO_COST_MODE(2, false, true);
        note_launch();
        return;
    }
    if (raw || place) {  // the reference's arithmetic with the probe outputs
        if (device_pow) PAMO_COST_MODE(0, true, true);
        else PAMO_COST_MODE(0, false, true);
        note_launch();
        return;
    }
#undef PAMO_COST_MODE
    if (legacy) {
        if (device_pow)
            pdl(k_edge_cost<true, true, false>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                            cost, vmin, d_scale, tres, 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
        else
            pdl(k_edge_cost<true, false, false>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                             cost, vmin, d_scale, tres, 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
    } else if (device_pow) {
        pdl(k_edge_cost<false, true, false>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                         cost, vmin, d_scale, tres, is_stuck, is_stuck_dev, nullptr,
                                                         nullptr, nullptr, nullptr, nullptr);
    } else {
        pdl(k_edge_cost<false, false, false>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                          cost, vmin, d_scale, tres, is_stuck, is_stuck_dev, nullptr,
                                                          nullptr, nullptr, nullptr, nullptr);
    }
    note_launch();
}
void launch_edge_cost_batch(const RoundCounters* rc, int n_edges_bound, const int* eorder, const int2* edges,
                            const int* nt_off, const int* nt, const int4* tri, const float4* pos, const Quadric* q,
                            const float4* fgeo, const int* nxt, const int2* spc, const unsigned char* invalid,
                            uint32_t* cost,
                            unsigned long long* vmin, const float* mesh_scale, const int* mesh_stuck, const int* vmesh,
                            float tres, cudaStream_t s, bool device_pow) {
    const int g = grid_for(n_edges_bound, kT);
    if (device_pow)
        pdl(k_edge_cost<false, true, true>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                        cost, vmin, mesh_scale, tres, 0, nullptr, vmesh, mesh_stuck, nullptr, nullptr,
                                                        nullptr);
    else
        pdl(k_edge_cost<false, false, true>, g, kT, 0, s)(rc, eorder, edges, nt_off, nt, tri, pos, q, fgeo, nxt, spc, invalid,
                                                         cost, vmin, mesh_scale, tres, 0, nullptr, vmesh, mesh_stuck, nullptr, nullptr,
                                                        nullptr);
    note_launch();
}
void launch_collapse(RoundCounters* rc, int n_edges_bound, const int2* edges, const uint32_t* cost,
                     uint32_t collapse_t, const unsigned long long* vmin, const int* nxt, const int2* spc,
                     const int* nt_off, const int* nt, int4* tri, float4* pos, int* occ, int* win, cudaStream_t s,
                     bool restore, const float4* place) {
    const int g = grid_for(n_edges_bound, kT);
    if (restore && place)
        pdl(k_collapse<true, true>, g, kT, 0, s)(rc, edges, cost, collapse_t, vmin, nxt, spc, nt_off, nt, tri, pos, occ, win,
                                                 place);
    else if (restore)
        pdl(k_collapse<true, false>, g, kT, 0, s)(rc, edges, cost, collapse_t, vmin, nxt, spc, nt_off, nt, tri, pos, occ,
                                                  win, nullptr);
    else
        pdl(k_collapse<false, false>, g, kT, 0, s)(rc, edges, cost, collapse_t, vmin, nxt, spc, nt_off, nt, tri, pos, occ,
                                                   win, nullptr);
    note_launch();
}
void launch_after_collapse(RoundCounters* rc, int n_edges_bound, int n_tris_bound, const int* win_scan, int* collapsed,
                           const int2* edges, const int* nt_off, const int* nt, int4* tri, float4* pos, int* occ,
                           int line_cap, bool lines, cudaStream_t s) {
    const int g = grid_for(std::max(n_edges_bound, n_tris_bound), kT);
    if (lines)
        pdl(k_after_collapse<true>, g, kT, 0, s)(rc, win_scan, collapsed, edges, nt_off, nt, tri, pos, occ, line_cap);
    else
        pdl(k_after_collapse<false>, g, kT, 0, s)(rc, win_scan, collapsed, edges, nt_off, nt, tri, pos, occ, line_cap);
    note_launch();
}
void launch_mark_query(const RoundCounters* rc, int n_edges_bound, const int* collapsed, const int2* edges,
                       const int* nt_off, const int* nt, int* qflag, cudaStream_t s) {
    pdl(k_mark_query, grid_for(n_edges_bound, kT), kT, 0, s)(rc, collapsed, edges, nt_off, nt, qflag); note_launch();
}
void launch_undo_check(RoundCounters* rc, int n_edges_bound, const int* collapsed, const int2* edges, const int* nt_off,
                       const int* nt, const unsigned char* hit, int* uflag, cudaStream_t s, const int4* tri,
                       int* fflags) {
    pdl(k_undo_check, grid_for(n_edges_bound, kT), kT, 0, s)(rc, collapsed, edges, nt_off, nt, hit, uflag, tri, fflags); note_launch();
}
void launch_undo_apply(RoundCounters* rc, int n_edges_bound, const int* collapsed, const int* uscan, const int2* edges,
                       const int* nt_off, const int* nt, int4* tri, const int4* orig_tri, float4* pos,
                       const float4* orig_pos, int* occ, int* tmp_undo, int* undo_list, const int* pts_map,
                       int list_cap, cudaStream_t s) {
    pdl(k_undo_apply, grid_for(n_edges_bound, kT), kT, 0, s)(rc, collapsed, uscan, edges, nt_off, nt, tri, orig_tri, pos,
                                                            orig_pos, occ, tmp_undo, undo_list, pts_map, list_cap, list_cap); note_launch();
    pdl(k_after_apply, 1, 1, 0, s)(rc); note_launch();
}
void launch_after_check(RoundCounters* rc, cudaStream_t s) {
    pdl(k_after_check, 1, 1, 0, s)(rc); note_launch();
}

void launch_live_flags(const RoundCounters* rc, int n_tris_bound, const int4* tri, int* flags, cudaStream_t s) {
    pdl(k_live_flags, grid_for(n_tris_bound, kT), kT, 0, s)(rc, tri, flags); note_launch();
}
void launch_compact_mesh(RoundCounters* rc, int n_pts_bound, int n_tris_bound, const float4* pos, const int* occ,
                         const int* pts_map, const int4* tri, const int* face_scan, float4* out_pos, int4* out_tri,
                         cudaStream_t s, bool check, const BvhRemap& remap) {
    const int n = n_pts_bound > n_tris_bound ? n_pts_bound : n_tris_bound;
    pdl(k_compact_mesh, grid_for(n, kT), kT, 0, s)(rc, pos, occ, pts_map, tri, face_scan, out_pos, out_tri, check ? 1 : 0,
                                           remap); note_launch();
}
void launch_export_round(const RoundCounters* rc, int n_pts, int n_tris, const float4* pos, const int4* tri,
                         const int* occ, const int* pts_map, const int* undo_list, float* verts, int* tris,
                         int* verts_occ, int* verts_map, int* verts_undo, int n_undo, cudaStream_t s) {
    (void)rc;
    const int n = n_pts > n_tris ? n_pts : n_tris;
    pdl(k_export_round, grid_for(n, kT), kT, 0, s)(n_pts, n_tris, pos, tri, occ, pts_map, undo_list, verts, tris, verts_occ,
                                                  verts_map, verts_undo, n_undo); note_launch();
}
void launch_export_mesh(int n_pts, int n_tris, const float4* pos, const int4* tri, const float* add, float* verts,
                        int* tris, cudaStream_t s) {
    const int n = n_pts > n_tris ? n_pts : n_tris;
    pdl(k_export_mesh, grid_for(n, kT), kT, 0, s)(n_pts, n_tris, pos, tri, add, verts, tris); note_launch();
}

// ---- device-driven rounds ----
void launch_round_prologue_dev(const RoundStart& r, int n_pts_bound, int n_tris_bound, cudaStream_t s) {
    const int n = (n_pts_bound > n_tris_bound ? n_pts_bound : n_tris_bound) + 1;
    pdl(k_round_prologue_dev, grid_for(n, kT), kT, 0, s)(r);
    note_launch();
}
void launch_round_end(const RoundCounters* rc, const LoopState* ls, LoopState* next, const int* undo_list, int* undo_in,
                      int undo_cap, int n_undo_bound, cudaStream_t s) {
    pdl(k_round_end, grid_for(n_undo_bound, kT, 1), kT, 0, s)(rc, ls, next, undo_list, undo_in, undo_cap); note_launch();
}

}  // namespace pamo
