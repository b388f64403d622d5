// Centring of stage 2 (simp_cuda/pamo/__init__.py:60-72, 117, 126) for one mesh or a batch of meshes: the mean of the
// face means with numpy's float32 semantics (per face ((a + b) + c) / 3, then a sequential float32 sum over the faces
// divided by their count), the centred points, and the scale (their largest extent).
//
// The sequential sum s_k = fl(s_(k-1) + x_k) is what bounds this: a dependent chain of one float add per face (about
// 2.4 ns each on one thread). It is made parallel over chunks of kChunk elements, exactly:
//   * while the running sum stays inside one binade [2^e, 2^(e+1)) (float spacing u = 2^(e-23)) and off its end points,
//     s = S u with an integer S and fl(s + x) = (S + round(x / u)) u. The rounded increments are integers that do not
//     depend on S, except half-way ties, which round to the even sum and so depend on S's parity only;
//   * a chunk is therefore described, for a given binade, by its total increment for an even and for an odd start and
//     by the smallest and largest running increment of either (k_center_incs, every chunk at once, for the binade and
//     sign that an ordinary prefix sum of the chunk sums predicts);
//   * one warp per coordinate then walks the chunks 32 at a time (k_center_walk): a warp scan of the increments gives
//     every chunk's start, a chunk whose predicted binade is the running sum's and whose running increments stay inside
//     it is taken as a whole, and the first that is not is added element by element.
// Before, one block per coordinate re-scanned a window of 16,384 elements for every element that left the binade or
// tied (3.5 ms for 5.24M faces, 2.2 ms for 286k noisy faces), and a batch did so for one mesh after the other. A whole
// stage-2 loop takes 121.7 instead of 124.5 ms on the 5.24M-face mesh, 24.5 instead of 25.1 ms on the noisy height field
// (whose sums change binade in most chunks) and 149.6 instead of 172.9 ms on a batch of 64 meshes (3.2M faces), whose
// loading and shuffle became three launches as well.
#include <cstdint>
#include "scan.cuh"
#include "simp_round.cuh"

namespace pamo {

namespace {

constexpr int kChunk = 512;       // elements a chunk describes; a chunk that leaves its binade costs 512 dependent adds
constexpr int kChunkThreads = 128;
constexpr int kPer = kChunk / kChunkThreads;
constexpr int kPredThreads = 1024;
constexpr int kIncMax = 1 << 21;  // larger increments leave the chunk to the walk (and keep its sums in 32 bits)

// The chunk's increments in units of its predicted spacing, for an even (0) and an odd (1) start.
struct ChunkInfo {
    int a[2];        // total increment
    int mn[2], mx[2];  // smallest and largest running increment after an element
    int key;         // predicted sign and exponent bits of the running sum; -1: not described
    int pad;
};

__device__ __forceinline__ int sum_key(float s) {  // sign and exponent bits; -1 where the integer form does not hold
    const unsigned b = __float_as_uint(s);
    const int ex = (int)((b >> 23) & 0xFFu);
    return (ex < 2 || ex > 253) ? -1 : (int)(b >> 23);
}

struct Inc2 {
    int a0, a1;
};
__device__ __forceinline__ Inc2 then(Inc2 x, Inc2 y) {  // x, then y
    return {x.a0 + ((x.a0 & 1) ? y.a1 : y.a0), x.a1 + (((x.a1 + 1) & 1) ? y.a1 : y.a0)};
}

// round(x / u) for u = 2^(e - 23), for an even and an odd running sum (they differ at a half-way tie only)
__device__ __forceinline__ Inc2 increment(float x, int e, bool& bad) {
    const unsigned b = __float_as_uint(x);
    const int bex = (int)((b >> 23) & 0xFFu);
    if ((b & 0x7FFFFFFFu) == 0u) return {0, 0};
    if (bex == 0xFF) {  // inf or nan
        bad = true;
        return {0, 0};
    }
    const int m = bex ? (int)((b & 0x7FFFFFu) | 0x800000u) : (int)(b & 0x7FFFFFu);
    const int k = e - (bex ? bex - 127 : -126);  // x / u = +-m 2^-k
    if (k <= 0) {
        bad = true;  // at least 2^23 spacings
        return {0, 0};
    }
    if (k > 24) return {0, 0};  // below half a spacing
    const int fl = m >> k, rem = m & ((1 << k) - 1), half = 1 << (k - 1);
    if (fl >= kIncMax) {
        bad = true;
        return {0, 0};
    }
    const bool neg = (b >> 31) != 0;
    if (rem == half) {  // between g and g + 1: the even sum
        const int g = neg ? -(fl + 1) : fl;
        return {g + (g & 1), g + ((g + 1) & 1)};
    }
    const int q = fl + (rem > half ? 1 : 0);
    return neg ? Inc2{-q, -q} : Inc2{q, q};
}

__device__ __forceinline__ int chunks_of(int nf) { return (nf + kChunk - 1) / kChunk; }

// face means (per coordinate, so that the chunks read them in order) and each chunk's plain sum
__global__ void __launch_bounds__(kChunkThreads) k_center_means(CenterJobs J, float* fm_all, float* csum) {
    pdl_wait();
    __shared__ float part[3][kChunkThreads / 32];
    for (int j = blockIdx.y; j < J.n; j += gridDim.y) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const int nf = job.n_tris, nch = chunks_of(nf);
        float* fm = fm_all + 3 * (size_t)job.face0;
        auto corner = [&](int i) {  // a removed face's -1 indexes from the end, as numpy does
            if (i < 0) i += job.n_pts;
            return (i >= 0 && i < job.n_pts) ? i : 0;  // an invalid index is refused when the faces are loaded
        };
        for (int c = blockIdx.x; c < nch; c += gridDim.x) {
            float s[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const int f = c * kChunk + i * kChunkThreads + threadIdx.x;
                if (f >= nf) continue;
                const int a = corner(job.tris[3 * (size_t)f]), b = corner(job.tris[3 * (size_t)f + 1]),
                          t = corner(job.tris[3 * (size_t)f + 2]);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float x = ((job.pts[3 * (size_t)a + d] + job.pts[3 * (size_t)b + d]) + job.pts[3 * (size_t)t + d]) / 3.0f;
                    fm[(size_t)d * nf + f] = x;
                    s[d] += x;
                }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                for (int o = 16; o > 0; o >>= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
                if ((threadIdx.x & 31) == 0) part[d][threadIdx.x >> 5] = s[d];
            }
            __syncthreads();
            if (threadIdx.x < 3) {
                float t = 0.f;
                for (int w = 0; w < kChunkThreads / 32; ++w) t += part[threadIdx.x][w];
                csum[(size_t)threadIdx.x * J.n_chunks + job.chunk0 + c] = t;
            }
            __syncthreads();
        }
    }
}

// the running sum that plain prefix sums predict at each chunk's start (block x = coordinate), in place of the chunk
// sums; a wrong prediction only sends a chunk to the walk's element loop. Also clears the extents.
__global__ void __launch_bounds__(kPredThreads) k_center_predict(CenterJobs J, float* csum) {
    pdl_wait();
    __shared__ double wsum[32];
    __shared__ double carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = blockIdx.y; j < J.n; j += gridDim.y) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const int nch = chunks_of(job.n_tris);
        float* cs = csum + (size_t)blockIdx.x * J.n_chunks + job.chunk0;
        if (threadIdx.x == 0) {
            carry = 0.0;
            unsigned* ext = reinterpret_cast<unsigned*>(job.center + 4);
            ext[blockIdx.x] = 0xFFFFFFFFu;
            ext[3 + blockIdx.x] = 0u;
        }
        __syncthreads();
        for (int base = 0; base < nch; base += kPredThreads) {
            const int c = base + threadIdx.x;
            const double v = c < nch ? (double)cs[c] : 0.0;
            double inc = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane == 31) wsum[warp] = inc;
            __syncthreads();
            double before = carry;
            for (int w = 0; w < warp; ++w) before += wsum[w];
            if (c < nch) cs[c] = (float)(before + (inc - v));
            __syncthreads();
            if (threadIdx.x == kPredThreads - 1) carry = before + inc;
            __syncthreads();
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kChunkThreads) k_center_incs(CenterJobs J, const float* __restrict__ fm_all,
                                                               const float* __restrict__ pred, ChunkInfo* info) {
    pdl_wait();
    constexpr int W = kChunkThreads / 32;
    __shared__ Inc2 wtot[W];
    __shared__ int red[4][W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = blockIdx.z;
    for (int j = blockIdx.y; j < J.n; j += gridDim.y) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const int nf = job.n_tris, nch = chunks_of(nf);
        const float* x = fm_all + 3 * (size_t)job.face0 + (size_t)d * nf;
        for (int c = blockIdx.x; c < nch; c += gridDim.x) {
            const size_t at = (size_t)d * J.n_chunks + job.chunk0 + c;
            const int key = sum_key(pred[at]);
            const int e = (key & 0xFF) - 127;
            const int base = c * kChunk + threadIdx.x * kPer;
            Inc2 el[kPer];
            bool bad = key < 0;
            Inc2 t = {0, 0};
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                el[i] = (key >= 0 && base + i < nf) ? increment(x[base + i], e, bad) : Inc2{0, 0};
                t = then(t, el[i]);
            }
            Inc2 inc = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const Inc2 p = {__shfl_up_sync(0xffffffffu, inc.a0, o), __shfl_up_sync(0xffffffffu, inc.a1, o)};
                if (lane >= o) inc = then(p, inc);
            }
            if (lane == 31) wtot[warp] = inc;
            Inc2 ex = {__shfl_up_sync(0xffffffffu, inc.a0, 1), __shfl_up_sync(0xffffffffu, inc.a1, 1)};
            if (lane == 0) ex = {0, 0};
            const bool any_bad = __syncthreads_or(bad);
            Inc2 before = {0, 0};
            for (int w = 0; w < warp; ++w) before = then(before, wtot[w]);
            ex = then(before, ex);
            // running increments of this thread's elements (past the end they repeat the last one)
            int mn[2] = {0x7fffffff, 0x7fffffff}, mx[2] = {-0x7fffffff, -0x7fffffff};
            int r0 = ex.a0, r1 = ex.a1;
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                r0 += (r0 & 1) ? el[i].a1 : el[i].a0;
                r1 += ((r1 + 1) & 1) ? el[i].a1 : el[i].a0;
                mn[0] = min(mn[0], r0);
                mx[0] = max(mx[0], r0);
                mn[1] = min(mn[1], r1);
                mx[1] = max(mx[1], r1);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    mn[p] = min(mn[p], __shfl_xor_sync(0xffffffffu, mn[p], o));
                    mx[p] = max(mx[p], __shfl_xor_sync(0xffffffffu, mx[p], o));
                }
            }
            if (lane == 0) {
                red[0][warp] = mn[0];
                red[1][warp] = mn[1];
                red[2][warp] = mx[0];
                red[3][warp] = mx[1];
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                ChunkInfo I;
                Inc2 all = wtot[0];
                for (int w = 1; w < W; ++w) {
                    all = then(all, wtot[w]);
                    for (int p = 0; p < 2; ++p) {
                        red[p][0] = min(red[p][0], red[p][w]);
                        red[2 + p][0] = max(red[2 + p][0], red[2 + p][w]);
                    }
                }
                I.a[0] = all.a0;
                I.a[1] = all.a1;
                bool wide = false;  // a running increment of a binade's width cannot stay inside it
                for (int p = 0; p < 2; ++p) {
                    I.mn[p] = red[p][0];
                    I.mx[p] = red[2 + p][0];
                    wide |= I.mn[p] < -(1 << 24) || I.mx[p] > (1 << 24);
                }
                I.key = (any_bad || wide) ? -1 : key;
                I.pad = 0;
                info[at] = I;
            }
            __syncthreads();
        }
    }
}

// One warp per coordinate (block x) walks the chunks; all lanes hold the same running sum.
__global__ void __launch_bounds__(32) k_center_walk(CenterJobs J, const float* __restrict__ fm_all,
                                                    const ChunkInfo* __restrict__ info) {
    pdl_wait();
    __shared__ __align__(16) float stage[kChunk];
    const int lane = threadIdx.x, d = blockIdx.x;
    for (int j = blockIdx.y; j < J.n; j += gridDim.y) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const int nf = job.n_tris, nch = chunks_of(nf);
        const float* x = fm_all + 3 * (size_t)job.face0 + (size_t)d * nf;
        const ChunkInfo* I = info + (size_t)d * J.n_chunks + job.chunk0;
        float s = 0.0f;
        int k = 0;
        while (k < nch) {  // every pass takes at least one chunk
            const int key = sum_key(s);
            int take = 0;
            if (key >= 0) {
                const unsigned sb = __float_as_uint(s);
                const int mag = (int)((sb & 0x7FFFFFu) | 0x800000u);
                const int S = (sb >> 31) ? -mag : mag;
                const int lo = S > 0 ? (1 << 23) + 1 : -((1 << 24) - 1), hi = S > 0 ? (1 << 24) - 1 : -((1 << 23) + 1);
                ChunkInfo c;
                c.key = -1;
                if (k + lane < nch) c = I[k + lane];
                bool ok = c.key == key;
                Inc2 inc = ok ? Inc2{c.a[0], c.a[1]} : Inc2{0, 0};
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const Inc2 p = {__shfl_up_sync(0xffffffffu, inc.a0, o), __shfl_up_sync(0xffffffffu, inc.a1, o)};
                    if (lane >= o) inc = then(p, inc);
                }
                const int run = (S & 1) ? inc.a1 : inc.a0;  // increment after this lane's chunk
                int start = __shfl_up_sync(0xffffffffu, run, 1);
                start = S + (lane == 0 ? 0 : start);
                const int p = start & 1;
                ok = ok && start + c.mn[p] >= lo && start + c.mx[p] <= hi;
                const unsigned fail = __ballot_sync(0xffffffffu, !ok);
                take = fail ? __ffs(fail) - 1 : 32;
                if (take > 0) {
                    const int R = S + __shfl_sync(0xffffffffu, run, take - 1);
                    s = __uint_as_float((sb & 0xFF800000u) | ((unsigned)(R < 0 ? -R : R) & 0x7FFFFFu));
                    k += take;
                }
            }
            if (take == 32 || k >= nch) continue;
            // the chunk that left the binade (or starts at zero, or is not finite): in order
            const int n = min(kChunk, nf - k * kChunk);
            __syncwarp();
            for (int i = lane; i < n; i += 32) stage[i] = x[(size_t)k * kChunk + i];
            __syncwarp();
            if (n == kChunk) {
#pragma unroll 8
                for (int i = 0; i < kChunk; i += 4) {
                    const float4 q = *reinterpret_cast<const float4*>(stage + i);
                    s = s + q.x;
                    s = s + q.y;
                    s = s + q.z;
                    s = s + q.w;
                }
            } else {
                for (int i = 0; i < n; ++i) s = s + stage[i];
            }
            ++k;
        }
        if (lane == 0) job.center[d] = s / (float)nf;
    }
}

__device__ __forceinline__ unsigned ord_enc(float f) {
    const unsigned a = __float_as_uint(f);
    return (a & 0x80000000u) ? ~a : (a | 0x80000000u);
}
__device__ __forceinline__ float ord_dec(unsigned u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

constexpr int kPtThreads = 256;

__global__ void __launch_bounds__(kPtThreads) k_center_points(CenterJobs J) {
    pdl_wait();
    __shared__ float red[6][kPtThreads / 32];
    for (int j = blockIdx.y; j < J.n; j += gridDim.y) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const float cx = job.center[0], cy = job.center[1], cz = job.center[2];
        float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
        bool any = false;
        for (int v = blockIdx.x * kPtThreads + threadIdx.x; v < job.n_pts; v += gridDim.x * kPtThreads) {
            any = true;
            const float x = job.pts[3 * (size_t)v] - cx, y = job.pts[3 * (size_t)v + 1] - cy, z = job.pts[3 * (size_t)v + 2] - cz;
            job.pos_out[v] = make_float4(x, y, z, 0.f);
            mn[0] = fminf(mn[0], x); mn[1] = fminf(mn[1], y); mn[2] = fminf(mn[2], z);
            mx[0] = fmaxf(mx[0], x); mx[1] = fmaxf(mx[1], y); mx[2] = fmaxf(mx[2], z);
        }
        const bool block_any = __syncthreads_or(any);
        if (!block_any) continue;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            for (int o = 16; o > 0; o >>= 1) {
                mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
                mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
            }
            if ((threadIdx.x & 31) == 0) {
                red[d][threadIdx.x >> 5] = mn[d];
                red[3 + d][threadIdx.x >> 5] = mx[d];
            }
        }
        __syncthreads();
        if (threadIdx.x < 6) {  // one atomic per block and bound
            unsigned* ext = reinterpret_cast<unsigned*>(job.center + 4);
            float m = red[threadIdx.x][0];
            for (int w = 1; w < kPtThreads / 32; ++w)
                m = threadIdx.x < 3 ? fminf(m, red[threadIdx.x][w]) : fmaxf(m, red[threadIdx.x][w]);
            if (threadIdx.x < 3) atomicMin(&ext[threadIdx.x], ord_enc(m));
            else atomicMax(&ext[threadIdx.x], ord_enc(m));
        }
        __syncthreads();
    }
}

// scale = max(max(ex, ey), ez) of the centred points (pamo/__init__.py:126)
__global__ void k_center_scale(CenterJobs J) {
    pdl_wait();
    for (int j = gtid(); j < J.n; j += gstride()) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        const unsigned* ext = reinterpret_cast<const unsigned*>(job.center + 4);
        const float ex = ord_dec(ext[3]) - ord_dec(ext[0]);
        const float ey = ord_dec(ext[4]) - ord_dec(ext[1]);
        const float ez = ord_dec(ext[5]) - ord_dec(ext[2]);
        const float m = (ey > ex) ? ey : ex;
        *job.scale = (ez > m) ? ez : m;
    }
}

// not centring: zero mean, cleared extents
__global__ void k_center_zero(CenterJobs J) {
    pdl_wait();
    for (int j = gtid(); j < J.n; j += gstride()) {
        const CenterJob job = J.many ? J.many[j] : J.one;
        unsigned* ext = reinterpret_cast<unsigned*>(job.center + 4);
        for (int d = 0; d < 3; ++d) {
            job.center[d] = 0.f;
            ext[d] = 0xFFFFFFFFu;
            ext[3 + d] = 0u;
        }
    }
}

}  // namespace

int center_chunks(int n_tris) { return (n_tris + kChunk - 1) / kChunk; }
size_t center_scratch_bytes(long long chunks) { return (size_t)chunks * 3 * (sizeof(ChunkInfo) + sizeof(float)); }

void launch_center_jobs(const CenterJobs& J, float* face_mean, void* scratch, int max_tris, int max_pts, cudaStream_t s,
                        bool centre) {
    if (J.n < 1) return;
    const int gy = J.n < 32768 ? J.n : 32768;
    const int per_job = gy > 64 ? 64 : 4096 / gy;  // blocks of one job: the chip is full from a few thousand on
    if (centre) {
        ChunkInfo* info = reinterpret_cast<ChunkInfo*>(scratch);
        float* csum = reinterpret_cast<float*>(info + 3 * (size_t)J.n_chunks);
        const int nch = center_chunks(max_tris);
        const int gx = nch < per_job ? (nch < 1 ? 1 : nch) : per_job;
        pdl(k_center_means, dim3(gx, gy), kChunkThreads, 0, s)(J, face_mean, csum); note_launch();
        pdl(k_center_predict, dim3(3, gy), kPredThreads, 0, s)(J, csum); note_launch();
        pdl(k_center_incs, dim3(gx, gy, 3), kChunkThreads, 0, s)(J, face_mean, csum, info); note_launch();
        pdl(k_center_walk, dim3(3, gy), 32, 0, s)(J, face_mean, info); note_launch();
    } else {
        pdl(k_center_zero, grid_for(J.n, 256), 256, 0, s)(J); note_launch();
    }
    const int pt = (max_pts + kPtThreads - 1) / kPtThreads;
    const int px = pt < per_job ? (pt < 1 ? 1 : pt) : (per_job < 8 * kNumSM ? per_job : 8 * kNumSM);
    pdl(k_center_points, dim3(px, gy), kPtThreads, 0, s)(J); note_launch();
    pdl(k_center_scale, grid_for(J.n, 256), 256, 0, s)(J); note_launch();
}

void launch_center(const float* pts, const int* tris, int n_pts, int n_tris, float* face_mean, void* scratch,
                   float* center, float* d_scale, float4* pos_out, cudaStream_t s, bool centre) {
    CenterJobs J{};
    J.one.pts = pts;
    J.one.tris = tris;
    J.one.n_pts = n_pts;
    J.one.n_tris = n_tris;
    J.one.center = center;
    J.one.scale = d_scale;
    J.one.pos_out = pos_out;
    J.n = 1;
    J.n_chunks = center_chunks(n_tris);
    launch_center_jobs(J, face_mean, scratch, n_tris, n_pts, s, centre);
}

}  // namespace pamo
