// Stage 1 of PaMO.run (simp_cuda/pamo/__init__.py:58-93): the input is normalised into the unit cube
// (preprocess_mesh), a narrow-band distance field of its triangles is sampled on an R^3 grid, shifted by 0.9
// voxel (`d - 0.9 / R`), and its zero set is extracted as a new mesh, mapped back with the reference's formula
// v = ((c + 0.5) / (R + 1) * margin - band) * tris_max + tris_min for a grid coordinate c. The reference calls
// two external libraries for this (torchcumesh2sdf.get_sdf and pdmc.DMC), which are absent; this file builds
// the same stage GB300-first:
//   * the distance field: every triangle lowers the squared distance of the samples in its box widened by the band
//     (an atomic minimum, so the field does not depend on the order); the rest hold the band value;
//   * the sign: outside is the set of voxels farther than the iso value from the surface that a 6-connected
//     flood fill reaches from the grid boundary; everything else is inside, so open and self-intersecting
//     inputs give a closed shell. The fill and the extraction work on rows of 32 samples a word;
//   * the surface: a dual extraction (one vertex per cell whose corners change sign, at the mean of the cell's
//     edge crossings; two triangles per grid edge with a sign change, joining the four cells around it,
//     oriented from inside to outside). Grid sample i lies at normalised coordinate (i + 0.5) / (R + 1).
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/pamo_gb300.h"
#include "pamo_common.cuh"
#include "scan.cuh"

namespace {

using namespace pamo;

constexpr int kT = 256;

__device__ __forceinline__ unsigned ord(float f) {  // order-preserving float -> uint
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord(unsigned u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u); }

// preprocess_mesh in float32: bounds of (p - mean) over the referenced corners, ext[0..2] the minima and ext[3..5] the
// maxima (max((p - mean) - min) = max(p - mean) - min: rounding is monotone)
__global__ void __launch_bounds__(kT) k_corner_bounds(const float* __restrict__ pts, const int* __restrict__ tris, int nf,
                                                      const float* mean, unsigned* ext, int np, int* status) {
    pdl_wait();
    __shared__ float sm[6][kT / 32];
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    const long long n = 3ll * nf;
    for (long long i = gtid(); i < n; i += gstride()) {
        const int v = tris[i];
        if (v < 0 || v >= np) {
            atomicOr(status, kErrBadIndex);
            continue;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float x = pts[3 * (size_t)v + d] - mean[d];
            mn[d] = fminf(mn[d], x);
            mx[d] = fmaxf(mx[d], x);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            sm[d][threadIdx.x >> 5] = mn[d];
            sm[3 + d][threadIdx.x >> 5] = mx[d];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float r = sm[threadIdx.x][0];
        for (int w = 1; w < kT / 32; ++w) r = threadIdx.x < 3 ? fminf(r, sm[threadIdx.x][w]) : fmaxf(r, sm[threadIdx.x][w]);
        if (threadIdx.x < 3) atomicMin(&ext[threadIdx.x], ord(r));
        else atomicMax(&ext[threadIdx.x], ord(r));
    }
}

// the largest extent (tris_max); a coordinate without a number adds nothing
__device__ __forceinline__ float extent_max(const unsigned* ext) {
    float m = -INFINITY;
    for (int d = 0; d < 3; ++d) m = fmaxf(m, unord(ext[3 + d]) - unord(ext[d]));
    return m;
}

// normalised vertices (tris = (tris / tris_max + band) / margin) and faces as int4 (-1: an index out of range, reported
// when the counts are read)
__global__ void k_normalise(const float* __restrict__ pts, int np, const int* __restrict__ tris, int nf,
                            const float* mean, const unsigned* ext, float band, float margin, float4* q, int4* tri) {
    pdl_wait();
    const float t0 = unord(ext[0]), t1 = unord(ext[1]), t2 = unord(ext[2]), tmax = extent_max(ext);
    for (int v = gtid(); v < np; v += gstride()) {
        const float x = ((pts[3 * v] - mean[0]) - t0) / tmax, y = ((pts[3 * v + 1] - mean[1]) - t1) / tmax,
                    z = ((pts[3 * v + 2] - mean[2]) - t2) / tmax;
        q[v] = make_float4((x + band) / margin, (y + band) / margin, (z + band) / margin, 0.f);
    }
    for (int f = gtid(); f < nf; f += gstride()) {
        const int a = tris[3 * f], b = tris[3 * f + 1], c = tris[3 * f + 2];
        const bool ok = a >= 0 && a < np && b >= 0 && b < np && c >= 0 && c < np;
        tri[f] = ok ? make_int4(a, b, c, 0) : make_int4(-1, -1, -1, 0);
    }
}

__device__ __forceinline__ int cell_lo(float x, float band, int R) {  // first sample index >= x - band
    return max(0, (int)ceilf((x - band) * (float)(R + 1) - 0.5f));
}
__device__ __forceinline__ int cell_hi(float x, float band, int R) {  // last sample index <= x + band
    return min(R - 1, (int)floorf((x + band) * (float)(R + 1) - 0.5f));
}

struct P3f {
    float x, y, z;
};
__device__ __forceinline__ P3f psub(P3f a, P3f b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float pdot(P3f a, P3f b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ P3f p3(float4 v) { return {v.x, v.y, v.z}; }

__device__ float point_tri_sq(P3f p, P3f a, P3f b, P3f c) {  // Ericson 5.1.5, squared distance
    const P3f ab = psub(b, a), ac = psub(c, a), ap = psub(p, a);
    const float d1 = pdot(ab, ap), d2 = pdot(ac, ap);
    P3f r;
    if (d1 <= 0.f && d2 <= 0.f) {
        r = a;
    } else {
        const P3f bp = psub(p, b);
        const float d3 = pdot(ab, bp), d4 = pdot(ac, bp);
        const float vc = d1 * d4 - d3 * d2;
        const P3f cp = psub(p, c);
        const float d5 = pdot(ab, cp), d6 = pdot(ac, cp);
        const float vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
        if (d3 >= 0.f && d4 <= d3) r = b;
        else if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
            const float v = d1 / (d1 - d3);
            r = {a.x + v * ab.x, a.y + v * ab.y, a.z + v * ab.z};
        } else if (d6 >= 0.f && d5 <= d6) r = c;
        else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
            const float w = d2 / (d2 - d6);
            r = {a.x + w * ac.x, a.y + w * ac.y, a.z + w * ac.z};
        } else if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
            const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
            r = {b.x + w * (c.x - b.x), b.y + w * (c.y - b.y), b.z + w * (c.z - b.z)};
        } else {
            const float den = 1.f / (va + vb + vc);
            const float v = vb * den, w = vc * den;
            r = {a.x + ab.x * v + ac.x * w, a.y + ab.y * v + ac.y * w, a.z + ab.z * v + ac.z * w};
        }
    }
    const P3f d = psub(r, p);
    return pdot(d, d);
}

__device__ __forceinline__ float box_sq(P3f p, float4 lo, float4 hi) {
    const float dx = fmaxf(fmaxf(lo.x - p.x, 0.f), p.x - hi.x), dy = fmaxf(fmaxf(lo.y - p.y, 0.f), p.y - hi.y),
                dz = fmaxf(fmaxf(lo.z - p.z, 0.f), p.z - hi.z);
    return dx * dx + dy * dy + dz * dz;
}

// ---- the distance field ---------------------------------------------------------------------------------------------
//
// udf2[i] holds the squared distance of sample i, capped at band^2, as a float whose bits order like an unsigned. A
// warp takes one triangle and its lanes the samples of the triangle's box widened by the band: about 7^3 samples for a
// triangle of a voxel's size. A sample whose distance from the box is not below its current value is left alone; what a
// triangle offers is never below that distance (less kBoxSlack, which keeps the triangle's own value where the two
// round differently), so whether a sample was skipped does not show in the result. A triangle with more than
// kSplatMax samples is cut into chunks that warps of a second kernel take from a queue.
//
// A tree walk per sample in the band (256^3, 327,680 faces) read 60-100 nodes of divergent
// walks at a quarter of the lanes: 7.99 ms, with 0.83 ms to mark the band and 0.25 ms for the tree. The splat does
// about 140 M box tests and stays in L2 (the grid's 67 MB). The whole of stage 1, with the bit rows below: 14.8 -> 1.33
// ms at 256^3 (327,680 faces), 2.58 -> 0.41 ms at 128^3 (20,480 faces); with four samples in flight, the fill's early end and
// the spread of the cells over the warps 1.30 and 0.37 ms.
// Measured on a whole call at 128^3, at 256^3 (the meshes above) and for 300 triangles across the whole grid at 256^3:
// kSplatMax 1024, 2048, 4096: 0.38, 0.38, 0.38 / 1.31, 1.31, 1.31 / 8.9, 8.8, 8.6 ms; kSplatAhead 2, 4, 8: 0.37, 0.38, 0.39 / 1.27, 1.31,
// 1.63 / 8.8, 8.8, 8.9 ms; kMaxChunks 256, 1024, 4096: 9.5, 8.8, 8.6 ms of the last, the others alike. Beyond the queue the
// time grows: 1,500 such triangles 128 ms, 1,000 21 ms (918 and 811 ms with a tree walk per sample).
constexpr int kSplatMax = 2048;      // samples of one warp's task
constexpr int kSplatAhead = 4;       // samples of a lane whose values are loaded together
constexpr int kMaxChunks = 1024;     // tasks of one triangle (larger boxes get larger chunks)
constexpr int kSplatQueue = 1 << 20; // tasks queued; a triangle that finds no room is done in place
constexpr float kBoxSlack = 4e-6f;   // of the band: the rounding of a distance computed near coordinate 1

struct SplatBox {
    int x0, y0, z0, nx, ny, nz;
    float4 lo, hi;
    P3f a, b, c;
};

__device__ __forceinline__ bool splat_box(int4 t, const float4* __restrict__ q, int R, float band, SplatBox& s) {
    if (t.x < 0) return false;
    const float4 a = q[t.x], b = q[t.y], c = q[t.z];
    s.a = p3(a);
    s.b = p3(b);
    s.c = p3(c);
    s.lo = make_float4(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)), 0.f);
    s.hi = make_float4(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)), 0.f);
    s.x0 = cell_lo(s.lo.x, band, R);
    s.y0 = cell_lo(s.lo.y, band, R);
    s.z0 = cell_lo(s.lo.z, band, R);
    const int x1 = cell_hi(s.hi.x, band, R), y1 = cell_hi(s.hi.y, band, R), z1 = cell_hi(s.hi.z, band, R);
    if (x1 < s.x0 || y1 < s.y0 || z1 < s.z0) return false;
    s.nx = x1 - s.x0 + 1;
    s.ny = y1 - s.y0 + 1;
    s.nz = z1 - s.z0 + 1;
    return true;
}

__device__ __forceinline__ P3f splat_point(int x, int y, int z, float inv) {
    return {((float)x + 0.5f) * inv, ((float)y + 0.5f) * inv, ((float)z + 0.5f) * inv};
}

// the triangle's offer to the sample at p, whose value was `best` (lowered by others at most)
__device__ __forceinline__ void splat_sample(const SplatBox& s, P3f p, float best, float slack, unsigned* at) {
    const float bound = box_sq(p, s.lo, s.hi) - slack;
    if (bound >= best) return;
    const float d = point_tri_sq(p, s.a, s.b, s.c);
    if (d < best) atomicMin(at, __float_as_uint(fmaxf(d, bound)));  // a NaN distance offers nothing
}

// samples [i0, i1) of the box, x fastest
__device__ __forceinline__ void splat_range(const SplatBox& s, unsigned i0, unsigned i1, int R, float band, unsigned* udf2) {
    const float inv = 1.0f / (float)(R + 1), slack = kBoxSlack * band;
    const unsigned nx = s.nx, nxy = (unsigned)s.nx * (unsigned)s.ny;
    for (unsigned i = i0 + (threadIdx.x & 31); i < i1; i += 32) {
        const unsigned z = i / nxy, r = i - z * nxy, y = r / nx, x = r - y * nx;
        unsigned* at = udf2 + ((size_t)(s.z0 + z) * R + s.y0 + y) * R + s.x0 + x;
        splat_sample(s, splat_point(s.x0 + x, s.y0 + y, s.z0 + z, inv), __uint_as_float(__ldcg(at)), slack, at);
    }
}

__global__ void __launch_bounds__(kT) k_splat(const float4* __restrict__ q, const int4* __restrict__ tri, int nf, int R,
                                              float band, unsigned* udf2, int2* queue, int* queued) {
    pdl_wait();
    const float inv = 1.0f / (float)(R + 1), slack = kBoxSlack * band;
    const int lane = threadIdx.x & 31;
    for (long long f = gtid() >> 5; f < nf; f += gstride() >> 5) {
        SplatBox s;
        if (!splat_box(tri[f], q, R, band, s)) continue;
        const unsigned n = (unsigned)s.nx * (unsigned)s.ny * (unsigned)s.nz;  // at most 1024^3
        if (n > kSplatMax) {
            const unsigned chunk = max((unsigned)kSplatMax, (n + kMaxChunks - 1) / kMaxChunks);
            const int chunks = (int)((n + chunk - 1) / chunk);
            int base = 0;
            // a full queue is not counted up any further: the count stays far below the type's range
            if (lane == 0) base = *(volatile int*)queued < kSplatQueue ? atomicAdd(queued, chunks) : kSplatQueue;
            base = __shfl_sync(0xffffffffu, base, 0);
            const bool room = base + chunks <= kSplatQueue;
            for (int k = lane; k < chunks && base + k < kSplatQueue; k += 32)
                queue[base + k] = room ? make_int2((int)f, k) : make_int2(-1, 0);
            if (!room) splat_range(s, 0, n, R, band, udf2);
            continue;
        }
        // i / d by a multiplication: exact for i * d < 2^32 (i < 2^11, d <= 2^11; d = 1 apart)
        const unsigned nx = s.nx, nxy = (unsigned)s.nx * (unsigned)s.ny;
        const unsigned mx = nx > 1 ? 0xffffffffu / nx + 1u : 0u, mxy = nxy > 1 ? 0xffffffffu / nxy + 1u : 0u;
        for (unsigned i0 = lane; i0 < n; i0 += 32 * kSplatAhead) {
            unsigned* at[kSplatAhead];
            float best[kSplatAhead];
            P3f p[kSplatAhead];
#pragma unroll
            for (int k = 0; k < kSplatAhead; ++k) {
                const unsigned i = i0 + 32 * k, z = nxy > 1 ? __umulhi(i, mxy) : i, r = i - z * nxy,
                               y = nx > 1 ? __umulhi(r, mx) : r, x = r - y * nx;
                p[k] = splat_point(s.x0 + x, s.y0 + y, s.z0 + z, inv);
                at[k] = udf2 + ((size_t)(s.z0 + z) * R + s.y0 + y) * R + s.x0 + x;
                best[k] = i < n ? __uint_as_float(__ldcg(at[k])) : -1.f;  // past the end: no offer is below
            }
#pragma unroll
            for (int k = 0; k < kSplatAhead; ++k) splat_sample(s, p[k], best[k], slack, at[k]);
        }
    }
}

__global__ void __launch_bounds__(kT) k_splat_big(const float4* __restrict__ q, const int4* __restrict__ tri, int R,
                                                  float band, unsigned* udf2, const int2* __restrict__ queue,
                                                  const int* __restrict__ queued) {
    pdl_wait();
    const int n = min(*queued, kSplatQueue);
    for (int k = gtid() >> 5; k < n; k += gstride() >> 5) {
        const int2 e = queue[k];
        SplatBox s;
        if (e.x < 0 || !splat_box(tri[e.x], q, R, band, s)) continue;
        const unsigned m = (unsigned)s.nx * (unsigned)s.ny * (unsigned)s.nz;
        const unsigned chunk = max((unsigned)kSplatMax, (m + kMaxChunks - 1) / kMaxChunks);
        splat_range(s, (unsigned)e.y * chunk, min(m, ((unsigned)e.y + 1u) * chunk), R, band, udf2);
    }
}

__global__ void k_fill_value(unsigned* p, long long n, unsigned v) {
    pdl_wait();
    const long long n4 = n >> 2;
    for (long long i = gtid(); i < n4; i += gstride()) reinterpret_cast<uint4*>(p)[i] = make_uint4(v, v, v, v);
    if (gtid() < (n & 3)) p[4 * n4 + gtid()] = v;
}

__device__ __forceinline__ float distance_of(unsigned d2, float band) { return fminf(sqrtf(__uint_as_float(d2)), band); }

// ---- the sign ---------------------------------------------------------------------------------------------------------
//
// Rows of samples as bits: word (z R + y) W + w, W = ceil(R / 32), bit b of it sample x = 32 w + b (0 past the row's
// end). far: farther than iso; below: nearer than iso; out: the outside set, at first the far samples on the grid's
// boundary. A warp takes 32 words, so that each lane stores one.
__global__ void __launch_bounds__(kT) k_sign_bits(const unsigned* __restrict__ udf2, int R, int W, float band, float iso,
                                                  unsigned* far, unsigned* below, unsigned* out) {
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long words = (long long)R * R * W;
    for (long long w0 = 32ll * (gtid() >> 5); w0 < words; w0 += gstride()) {
        unsigned mf = 0, mb = 0;
        long long row = w0 / W;
        int w = (int)(w0 - row * W);
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const int x = 32 * w + lane;
            const bool in = w0 + k < words && x < R;
            const float d = in ? distance_of(udf2[row * R + x], band) : iso;
            const unsigned f = __ballot_sync(0xffffffffu, d > iso), l = __ballot_sync(0xffffffffu, d < iso);
            if (k == lane) {
                mf = f;
                mb = l;
            }
            if (++w == W) {
                w = 0;
                ++row;
            }
        }
        const long long i = w0 + lane;
        if (i >= words) continue;
        far[i] = mf;
        below[i] = mb;
        const long long r = i / W;
        const int wi = (int)(i - r * W), y = (int)(r % R), z = (int)(r / R);
        const bool border = y == 0 || z == 0 || y == R - 1 || z == R - 1;
        unsigned edge = border ? 0xffffffffu : 0u;
        if (wi == 0) edge |= 1u;
        if (wi == (R - 1) >> 5) edge |= 1u << ((R - 1) & 31);
        out[i] = mf & edge;
    }
}

// Flood fill of one plane's tile, everything in shared memory: rows along x by the carries of an addition (in the sum
// p + s a seed s inside the passable run p carries to the run's end: the carry-in bits are (p + s) ^ p ^ s; the carries
// between the words of a row are those of the warp's ballots), then across the rows by doubling steps both ways, until
// the tile stays as it is. The planes are taken as (x, y), then as (x, z); a pass over both that changes nothing is the
// end, since every 6-neighbour was then looked at. Each word is written by one block and only gains bits, so a
// neighbour tile's row that is read while it grows is at worst caught up with in the next pass.
//
// A star-shaped shell at 256^3 is filled in the first pass, where a sweep over the samples moved one sample along y and
// z a launch: 64 launches of 87 us before.
constexpr int kFillThreads = 512;
constexpr int kFillRows = 256;  // rows of a tile
constexpr int kFillItems = kFillRows * 32 / kFillThreads;
constexpr int kFillLocal = 16;  // passes over a tile before it is left to the next launch

__device__ __forceinline__ unsigned carries(unsigned p, unsigned s, unsigned cin) { return (p + s + cin) ^ p ^ s; }

__global__ void __launch_bounds__(kFillThreads) k_fill(const unsigned* __restrict__ far, unsigned* out, int R, int W,
                                                       long long plane_stride, long long row_stride, int* changed) {
    pdl_wait();
    extern __shared__ unsigned fill_sm[];
    const int tiles = (R + kFillRows - 1) / kFillRows;
    const int plane = blockIdx.x / tiles, r0 = (blockIdx.x % tiles) * kFillRows;
    const int rows = min(kFillRows, R - r0), n = rows * W;
    unsigned* sg = fill_sm;
    unsigned* sp = fill_sm + n;
    const long long base = plane * plane_stride + r0 * row_stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned p[kFillItems], g0[kFillItems];
#pragma unroll
    for (int j = 0; j < kFillItems; ++j) {
        const int i = threadIdx.x + j * kFillThreads;
        p[j] = g0[j] = 0;
        if (i < n) {
            const int r = i / W, w = i - r * W;
            const long long at = base + r * row_stride + w;
            p[j] = far[at];
            g0[j] = __ldcg(&out[at]);
            unsigned g = g0[j];
            if (r == 0 && r0 > 0) g |= __ldcg(&out[at - row_stride]) & p[j];
            if (r == rows - 1 && r0 + rows < R) g |= __ldcg(&out[at + row_stride]) & p[j];
            sg[i] = g;
            sp[i] = p[j];
        }
    }
    __syncthreads();
    const int rpw = 32 / W;  // rows of a warp's pass
    const int lr = lane / W, lw = lane - lr * W;
    for (int it = 0; it < kFillLocal; ++it) {
        int diff = 0;
        for (int r = warp * rpw; r < rows; r += (kFillThreads / 32) * rpw) {
            const bool on = lr < rpw && r + lr < rows;
            const int i = (r + lr) * W + lw;
            const unsigned pp = on ? sp[i] : 0u, s0 = on ? sg[i] : 0u;
            unsigned s = s0;
            {  // towards higher x
                const bool last = lw == W - 1;
                const unsigned G = __ballot_sync(0xffffffffu, !last && (((unsigned long long)pp + s) >> 32) != 0ull);
                const unsigned A = G | __ballot_sync(0xffffffffu, !last && pp == 0xffffffffu);
                s |= pp & carries(pp, s, (carries(A, G, 0u) >> lane) & 1u);
            }
            {  // towards lower x, mirrored
                const unsigned pr = __brev(pp), sr = __brev(s);
                const bool last = lw == 0;
                const unsigned G = __brev(__ballot_sync(0xffffffffu, !last && (((unsigned long long)pr + sr) >> 32) != 0ull));
                const unsigned A = G | __brev(__ballot_sync(0xffffffffu, !last && pp == 0xffffffffu));
                s |= pp & __brev(carries(pr, sr, (__brev(carries(A, G, 0u)) >> lane) & 1u));
            }
            if (on && s != s0) {
                sg[i] = s;
                diff = 1;
            }
        }
        // a tile whose rows stay as they are and have nothing to give to the rows beside them is done: the doubling steps
        // are for those that have (the last passes of a fill change nothing anywhere)
        if (!__syncthreads_or(diff)) {
            int grows = 0;
#pragma unroll
            for (int j = 0; j < kFillItems; ++j) {
                const int i = threadIdx.x + j * kFillThreads;
                if (i >= n) continue;
                const unsigned beside = (i >= W ? sg[i - W] : 0u) | (i + W < n ? sg[i + W] : 0u);
                grows |= (p[j] & beside & ~sg[i]) != 0u;
            }
            if (!__syncthreads_or(grows)) break;
        }
        diff = 0;
        for (int dir = 0; dir < 2; ++dir) {
            for (int k = W; k < n; k *= 2) {
                unsigned g[kFillItems], q[kFillItems];
#pragma unroll
                for (int j = 0; j < kFillItems; ++j) {
                    const int i = threadIdx.x + j * kFillThreads;
                    g[j] = q[j] = 0;
                    if (i < n) {
                        const int o = dir ? i + k : i - k;
                        const bool has = o >= 0 && o < n;
                        q[j] = sp[i];
                        g[j] = sg[i] | (has ? q[j] & sg[o] : 0u);
                        q[j] = has ? q[j] & sp[o] : 0u;
                    }
                }
                __syncthreads();
#pragma unroll
                for (int j = 0; j < kFillItems; ++j) {
                    const int i = threadIdx.x + j * kFillThreads;
                    if (i < n) {
                        if (g[j] != sg[i]) diff = 1;
                        sg[i] = g[j];
                        sp[i] = q[j];
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int j = 0; j < kFillItems; ++j) {
                const int i = threadIdx.x + j * kFillThreads;
                if (i < n) sp[i] = p[j];
            }
            __syncthreads();
        }
        if (!__syncthreads_or(diff)) break;
    }
    int grown = 0;
#pragma unroll
    for (int j = 0; j < kFillItems; ++j) {
        const int i = threadIdx.x + j * kFillThreads;
        if (i < n && sg[i] != g0[j]) {
            const int r = i / W, w = i - r * W;
            out[base + r * row_stride + w] = sg[i];
            grown = 1;
        }
    }
    if (__syncthreads_or(grown) && threadIdx.x == 0) *changed = 1;
}

// ---- the surface --------------------------------------------------------------------------------------------------------
//
// The field at a sample is |udf - iso|, negative inside (not outside) unless it is zero: neg has those samples' bits.
__global__ void k_negative(const unsigned* __restrict__ far, const unsigned* __restrict__ below,
                           const unsigned* __restrict__ out, long long words, unsigned* neg) {
    pdl_wait();
    for (long long i = gtid(); i < words; i += gstride()) neg[i] = below[i] | (far[i] & ~out[i]);
}

// samples x + 1 of word i of a row
__device__ __forceinline__ unsigned next_x(const unsigned* neg, long long i, int w, int W) {
    return (neg[i] >> 1) | (w + 1 < W ? neg[i + 1] << 31 : 0u);
}
// samples with lo <= x <= hi of word w
__device__ __forceinline__ unsigned x_range(int w, int lo, int hi) {
    unsigned m = 0xffffffffu;
    const int a = lo - 32 * w, b = hi - 32 * w;
    if (b < 0 || a > 31) return 0u;
    if (a > 0) m &= 0xffffffffu << a;
    if (b < 31) m &= 0xffffffffu >> (31 - b);
    return m;
}
// grid edges with a sign change, along each axis from the samples of word (z, y, w), whose four cells exist
__device__ __forceinline__ void edge_bits(const unsigned* neg, long long i, int R, int W, int w, int y, int z,
                                          unsigned e[3]) {
    const unsigned a = neg[i];
    const bool yi = y >= 1 && y <= R - 2, zi = z >= 1 && z <= R - 2;
    const unsigned xi = x_range(w, 1, R - 2);
    e[0] = yi && zi ? (a ^ next_x(neg, i, w, W)) & x_range(w, 0, R - 2) : 0u;
    e[1] = zi && y < R - 1 ? (a ^ neg[i + W]) & xi : 0u;
    e[2] = yi && z < R - 1 ? (a ^ neg[i + (long long)R * W]) & xi : 0u;
}

// per word: the cells (named by their lowest sample) whose corners change sign, their number, and the number of quads
__global__ void k_surface_counts(const unsigned* __restrict__ neg, int R, int W, unsigned* cells, int* ccount,
                                 int* qcount) {
    pdl_wait();
    const long long words = (long long)R * R * W;
    for (long long i = gtid(); i < words; i += gstride()) {
        const long long row = i / W;
        const int w = (int)(i - row * W), y = (int)(row % R), z = (int)(row / R);
        unsigned active = 0;
        if (y < R - 1 && z < R - 1) {
            unsigned any = 0, all = 0xffffffffu;
            for (int k = 0; k < 4; ++k) {
                const long long j = i + ((k & 1) ? W : 0) + ((k & 2) ? (long long)R * W : 0);
                const unsigned a = neg[j], b = next_x(neg, j, w, W);
                any |= a | b;
                all &= a & b;
            }
            active = any & ~all & x_range(w, 0, R - 2);
        }
        unsigned e[3];
        edge_bits(neg, i, R, W, w, y, z, e);
        cells[i] = active;
        ccount[i] = __popc(active);
        qcount[i] = __popc(e[0]) + __popc(e[1]) + __popc(e[2]);
    }
    if (gtid() == 0) ccount[words] = qcount[words] = 0;
}

__constant__ int kEdgeCorners[12][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7},
                                        {0, 4}, {1, 5}, {2, 6}, {3, 7}};

// the vertex of each active cell at the mean of its edge crossings, in cell order; a warp looks at 32 words at a time, far
// apart (the words with cells lie together: 32 in a row were up to 32 turns for one warp), and its lanes take the cells of
// each word that has some
__global__ void __launch_bounds__(kT) k_cell_vertices(const unsigned* __restrict__ udf2, const unsigned* __restrict__ neg,
                                                      const unsigned* __restrict__ cells, int R, int W, float iso,
                                                      const int* __restrict__ cscan, float band, float margin,
                                                      const unsigned* ext, float* verts) {
    pdl_wait();
    const float t0 = unord(ext[0]), t1 = unord(ext[1]), t2 = unord(ext[2]), tmax = extent_max(ext);
    const int lane = threadIdx.x & 31;
    const long long words = (long long)R * R * W, RR = (long long)R * R;
    const long long warp = gtid() >> 5, warps = gstride() >> 5;
    for (long long w0 = warp; w0 < words; w0 += 32 * warps) {
        const unsigned mine = w0 + lane * warps < words ? cells[w0 + lane * warps] : 0u;
        for (unsigned todo = __ballot_sync(0xffffffffu, mine != 0u); todo; todo &= todo - 1u) {
            const int k = __ffs(todo) - 1;
            const unsigned act = __shfl_sync(0xffffffffu, mine, k);
            if (!((act >> lane) & 1u)) continue;
            const long long i = w0 + k * warps, row = i / W;
            const int w = (int)(i - row * W), y = (int)(row % R), z = (int)(row / R), x = 32 * w + lane;
            float v[8];
            for (int c = 0; c < 8; ++c) {
                const long long at = row * R + x + ((c & 2) ? R : 0) + ((c & 4) ? RR : 0) + (c & 1);
                const int xc = x + (c & 1);
                const unsigned nb = neg[(row + ((c & 2) ? 1 : 0) + ((c & 4) ? R : 0)) * W + (xc >> 5)];
                const float d = fabsf(distance_of(udf2[at], band) - iso);
                v[c] = ((nb >> (xc & 31)) & 1u) ? -d : d;
            }
            float sx = 0.f, sy = 0.f, sz = 0.f;
            int m = 0;
            for (int e = 0; e < 12; ++e) {
                const int a = kEdgeCorners[e][0], b = kEdgeCorners[e][1];
                if ((v[a] < 0.f) == (v[b] < 0.f)) continue;
                const float t = v[a] / (v[a] - v[b]);
                sx += (float)(a & 1) + t * (float)((b & 1) - (a & 1));
                sy += (float)((a >> 1) & 1) + t * (float)(((b >> 1) & 1) - ((a >> 1) & 1));
                sz += (float)(a >> 2) + t * (float)((b >> 2) - (a >> 2));
                ++m;
            }
            const float cx = (float)x + sx / (float)m, cy = (float)y + sy / (float)m, cz = (float)z + sz / (float)m;
            // the reference's mapping back: ((c + 0.5) / (R + 1) * margin - band) * tris_max + tris_min
            const float s = 1.0f / (float)(R + 1);
            const long long o = 3 * ((long long)cscan[i] + __popc(act & ((1u << lane) - 1u)));
            verts[o] = ((cx + 0.5f) * s * margin - band) * tmax + t0;
            verts[o + 1] = ((cy + 0.5f) * s * margin - band) * tmax + t1;
            verts[o + 2] = ((cz + 0.5f) * s * margin - band) * tmax + t2;
        }
    }
}

// two triangles for each grid edge with a sign change, in the order of the samples and then of the axes
__global__ void __launch_bounds__(kT) k_quads(const unsigned* __restrict__ neg, const unsigned* __restrict__ cells, int R,
                                              int W, const int* __restrict__ qscan, const int* __restrict__ cscan,
                                              int* tris) {
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const unsigned lower = (1u << lane) - 1u;
    const long long words = (long long)R * R * W;
    auto cell = [&](int cx, int cy, int cz) {
        const long long i = ((long long)cz * R + cy) * W + (cx >> 5);
        return cscan[i] + __popc(cells[i] & ((1u << (cx & 31)) - 1u));
    };
    const long long warp = gtid() >> 5, warps = gstride() >> 5;
    for (long long w0 = warp; w0 < words; w0 += 32 * warps) {
        const long long mine = w0 + lane * warps;
        const bool on = mine < words && qscan[mine + 1] != qscan[mine];
        for (unsigned todo = __ballot_sync(0xffffffffu, on); todo; todo &= todo - 1u) {
            const long long i = w0 + (__ffs(todo) - 1) * warps, row = i / W;
            const int w = (int)(i - row * W), y = (int)(row % R), z = (int)(row / R), x = 32 * w + lane;
            unsigned e[3];
            edge_bits(neg, i, R, W, w, y, z, e);
            if (!(((e[0] | e[1] | e[2]) >> lane) & 1u)) continue;
            const bool il = (neg[i] >> lane) & 1u;  // inside at the lower end
            long long o = 6 * ((long long)qscan[i] + __popc(e[0] & lower) + __popc(e[1] & lower) + __popc(e[2] & lower));
            for (int axis = 0; axis < 3; ++axis) {
                if (!((e[axis] >> lane) & 1u)) continue;
                // the four cells around the edge, counter-clockwise about the axis direction
                int c00, c10, c11, c01;
                if (axis == 0) {  // plane (y, z)
                    c00 = cell(x, y - 1, z - 1); c10 = cell(x, y, z - 1); c11 = cell(x, y, z); c01 = cell(x, y - 1, z);
                } else if (axis == 1) {  // plane (z, x)
                    c00 = cell(x - 1, y, z - 1); c10 = cell(x - 1, y, z); c11 = cell(x, y, z); c01 = cell(x, y, z - 1);
                } else {  // plane (x, y)
                    c00 = cell(x - 1, y - 1, z); c10 = cell(x, y - 1, z); c11 = cell(x, y, z); c01 = cell(x - 1, y, z);
                }
                // inside at the lower end: the surface faces the +axis direction, counter-clockwise seen from there
                if (il) {
                    tris[o] = c00; tris[o + 1] = c10; tris[o + 2] = c11;
                    tris[o + 3] = c00; tris[o + 4] = c11; tris[o + 5] = c01;
                } else {
                    tris[o] = c00; tris[o + 1] = c11; tris[o + 2] = c10;
                    tris[o + 3] = c00; tris[o + 4] = c01; tris[o + 5] = c11;
                }
                o += 6;
            }
        }
    }
}

struct DBuf {
    void* p = nullptr;
    size_t n = 0;
    int grow(size_t bytes) {
        if (bytes <= n && p) return PAMO_OK;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        if (cudaMalloc(&p, bytes) != cudaSuccess) return PAMO_ERR_OOM;
        n = bytes;
        return PAMO_OK;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

}  // namespace

struct pamo_remesher {
    int device = 0;
    DBuf q, tri, udf, queue, bits, counts, verts, tris, small, scratch;
    RoundCounters* rc = nullptr;
    int* h_small = nullptr;  // pinned: status, changed, vertex count, triangle count
    int nv = 0, nf = 0;
    void release() {
        for (DBuf* b : {&q, &tri, &udf, &queue, &bits, &counts, &verts, &tris, &small, &scratch}) b->release();
        if (rc) cudaFree(rc);
        if (h_small) cudaFreeHost(h_small);
        rc = nullptr;
        h_small = nullptr;
    }
};

extern "C" {

int pamo_remesher_create(pamo_remesher** out, int32_t device) {
    if (!out) return PAMO_ERR_INVALID_ARG;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return PAMO_ERR_INVALID_ARG;
    pamo_remesher* m = new pamo_remesher();
    m->device = device;
    if (cudaMalloc((void**)&m->rc, sizeof(RoundCounters)) != cudaSuccess ||
        cudaMallocHost((void**)&m->h_small, 16 * sizeof(int)) != cudaSuccess ||
        m->scratch.grow(2 * scan_scratch_ints() * sizeof(int)) != PAMO_OK || scan_scratch_clear((int*)m->scratch.p) ||
        scan_scratch_clear((int*)m->scratch.p + scan_scratch_ints())) {
        m->release();
        delete m;
        return PAMO_ERR_OOM;
    }
    *out = m;
    return PAMO_OK;
}

int pamo_remesher_destroy(pamo_remesher* m) {
    if (!m) return PAMO_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    cudaDeviceSynchronize();
    m->release();
    delete m;
    return PAMO_OK;
}

int pamo_remesh(pamo_remesher* m, const float* points, const int32_t* triangles, int32_t n_points, int32_t n_triangles,
                int32_t resolution, const float* mean3, int32_t* out_n_points, int32_t* out_n_triangles,
                pamo_stream stream) {
    if (!m || !points || !triangles || !mean3 || n_points < 1 || n_triangles < 1 || resolution < 4 ||
        resolution > 1024)
        return PAMO_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    cudaStream_t s = (cudaStream_t)stream;
    const int R = resolution;
    // the reference's Python floats (float64), applied to float32 arrays
    const float band = (float)(3.0 / R), margin = (float)(3.0 / R * 2.0 + 1.0), iso = (float)(0.9 / R);
    const long long NV = (long long)R * R * R;
    if (NV >= (1ll << 31) - 2) return PAMO_ERR_CAPACITY;
    const int W = (R + 31) / 32;
    const long long words = (long long)R * R * W;
    int r;
    if ((r = m->q.grow((size_t)n_points * sizeof(float4))) || (r = m->tri.grow((size_t)n_triangles * sizeof(int4))) ||
        (r = m->udf.grow(NV * sizeof(unsigned))) || (r = m->queue.grow(kSplatQueue * sizeof(int2))) ||
        (r = m->bits.grow(5 * words * sizeof(unsigned))) || (r = m->counts.grow(2 * (words + 8) * sizeof(int))) ||
        (r = m->small.grow(16 * sizeof(int))))
        return r;
    float* d_mean = (float*)m->small.p;           // 3 floats
    unsigned* ext = (unsigned*)m->small.p + 4;    // 6 words
    int* d_changed = (int*)m->small.p + 10;
    int* d_queued = (int*)m->small.p + 11;
    float4* q = (float4*)m->q.p;
    int4* tri = (int4*)m->tri.p;
    unsigned* udf2 = (unsigned*)m->udf.p;
    unsigned* far = (unsigned*)m->bits.p;
    unsigned *below = far + words, *out = far + 2 * words, *neg = far + 3 * words, *cells = far + 4 * words;
    int* ccount = (int*)m->counts.p;
    int* qcount = ccount + ((words + 4) & ~3ll);  // 16-byte aligned for the scan
    int* scratch = (int*)m->scratch.p;

    cudaMemsetAsync(m->rc, 0, sizeof(RoundCounters), s);
    std::memcpy(m->h_small + 4, mean3, 3 * sizeof(float));
    cudaMemcpyAsync(d_mean, m->h_small + 4, 3 * sizeof(float), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(ext, 0xFF, 3 * sizeof(unsigned), s);
    cudaMemsetAsync(ext + 3, 0x00, 5 * sizeof(unsigned), s);  // the maxima, changed, queued
    pdl(k_corner_bounds, grid_for(3ll * n_triangles, kT), kT, 0, s)(points, triangles, n_triangles, d_mean, ext, n_points,
                                                                   &m->rc->status);
    pdl(k_normalise, grid_for(std::max(n_points, n_triangles), kT), kT, 0, s)(points, n_points, triangles, n_triangles,
                                                                           d_mean, ext, band, margin, q, tri);
    const float band2 = band * band;
    unsigned band2_bits;
    std::memcpy(&band2_bits, &band2, sizeof(band2_bits));
    pdl(k_fill_value, grid_for(NV / 4 + 1, kT), kT, 0, s)(udf2, NV, band2_bits);
    pdl(k_splat, grid_for(32ll * n_triangles, kT), kT, 0, s)(q, tri, n_triangles, R, band, udf2, (int2*)m->queue.p, d_queued);
    pdl(k_splat_big, 8 * kNumSM, kT, 0, s)(q, tri, R, band, udf2, (const int2*)m->queue.p, d_queued);
    pdl(k_sign_bits, grid_for(words, kT), kT, 0, s)(udf2, R, W, band, iso, far, below, out);
    note_launches(6);
    // flood fill: two passes over the planes of both orientations, the second of which notes whether it changed
    // anything, and the counts behind them; again until it did not (each repetition adds at least one sample)
    const int tiles = (R + kFillRows - 1) / kFillRows;
    const size_t fill_smem = 2 * sizeof(unsigned) * (size_t)std::min(R, kFillRows) * W;
    if (cudaFuncSetAttribute(k_fill, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * sizeof(unsigned) * kFillRows * 32) != cudaSuccess)
        return PAMO_ERR_CUDA;
    const long long max_batches = NV + 2;
    for (long long batch = 0; batch < max_batches; ++batch) {
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1) cudaMemsetAsync(d_changed, 0, sizeof(int), s);
            pdl(k_fill, R * tiles, kFillThreads, fill_smem, s)(far, out, R, W, (long long)R * W, W, d_changed);
            pdl(k_fill, R * tiles, kFillThreads, fill_smem, s)(far, out, R, W, W, (long long)R * W, d_changed);
        }
        pdl(k_negative, grid_for(words, kT), kT, 0, s)(far, below, out, words, neg);
        pdl(k_surface_counts, grid_for(words, kT), kT, 0, s)(neg, R, W, cells, ccount, qcount);
        note_launches(6);
        const ScanJob jobs[2] = {{ccount, ccount, nullptr, (int)words + 1, &m->rc->n_win, scratch},
                                 {qcount, qcount, nullptr, (int)words + 1, &m->rc->n_query, scratch + scan_scratch_ints()}};
        exclusive_scans(jobs, 2, s, &m->rc->status, 0);
        cudaMemcpyAsync(m->h_small, &m->rc->status, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(m->h_small + 1, d_changed, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(m->h_small + 2, &m->rc->n_win, sizeof(int), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(m->h_small + 3, &m->rc->n_query, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) return PAMO_ERR_CUDA;
        if (m->h_small[0] & kErrBadIndex) return PAMO_ERR_INVALID_ARG;
        if (m->h_small[0] & kErrIterLimit) return PAMO_ERR_ITER_LIMIT;
        if (m->h_small[1] == 0) break;
    }
    m->nv = m->h_small[2];
    m->nf = 2 * m->h_small[3];
    if ((r = m->verts.grow(((size_t)m->nv + 1) * 3 * sizeof(float))) || (r = m->tris.grow(((size_t)m->nf + 1) * 3 * sizeof(int))))
        return r;
    pdl(k_cell_vertices, grid_for(words, kT), kT, 0, s)(udf2, neg, cells, R, W, iso, ccount, band, margin, ext,
                                                       (float*)m->verts.p);
    pdl(k_quads, grid_for(words, kT), kT, 0, s)(neg, cells, R, W, qcount, ccount, (int*)m->tris.p);
    note_launches(2);
    if (cudaStreamSynchronize(s) != cudaSuccess) return PAMO_ERR_CUDA;
    if (out_n_points) *out_n_points = m->nv;
    if (out_n_triangles) *out_n_triangles = m->nf;
    return PAMO_OK;
}

int pamo_remesh_result(pamo_remesher* m, float* verts, int32_t* tris, pamo_stream stream) {
    if (!m || !verts || !tris) return PAMO_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (m->nv) cudaMemcpyAsync(verts, m->verts.p, (size_t)m->nv * 3 * sizeof(float), cudaMemcpyDeviceToDevice, s);
    if (m->nf) cudaMemcpyAsync(tris, m->tris.p, (size_t)m->nf * 3 * sizeof(int), cudaMemcpyDeviceToDevice, s);
    return cudaStreamSynchronize(s) == cudaSuccess ? PAMO_OK : PAMO_ERR_CUDA;
}

}  // extern "C"
