// LBVH over live faces: AABBs and scene bounds, 30-bit Morton codes of box centroids, an in-house stable
// LSD radix sort (8-bit digits, warp-match ranking), Karras (2012) topology with an index tie-break for
// equal codes, bottom-up boxes, and a per-face query that walks the tree with a stack in shared memory and
// runs the reference's pair test on every overlapping leaf.
//
// The tree only filters candidates: a (query f, hit g) pair is tested iff both faces are live, f != g and
// their closed boxes overlap (simp_cuda/src/bvh/query.cuh:8-133, aabb.cuh:154-162), which is the candidate
// set of the reference's global LBVH query.
#include <cstdint>
#include "lbvh.cuh"
#include "scan.cuh"
#include "tritri.cuh"

namespace pamo {

namespace {

constexpr int kSortTiles = 4 * kNumSM;
constexpr size_t kExactQueue = 1 << 20;  // pairs queued for the float64 pass (the rest are decided in place)
constexpr int kSortThreads = 256;
constexpr int kFusedTiles = 16;   // tiles up to which a sort pass is one launch (k_rs_pass)
constexpr int kSortCtl = 4 * 256 + 4 * (1 + kFusedTiles);  // the digit totals, then each pass's ticket and flags
constexpr int kQueryThreads = 128;
constexpr int kStackDepth = 64;  // enough for any tree (depth <= 62 + 1)
constexpr int kShortStack = 24;  // first walk: deeper queries are handed to the second walk
constexpr int kExactThreads = 64;
constexpr int kPairChunk = 128;  // list slots a warp takes at a time
constexpr int kQueryBit = 1 << 30;  // set on a packed leaf's face id when the face is a query face

__device__ __forceinline__ unsigned f2ord(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ unsigned expand10(unsigned v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// ---------------------------------------------------------------- boxes + scene bounds
// One pass over the faces before a build or a refit, which also prepares the pass that follows: the counters of
// bvh_query, the hit flags (q.hit), the number of query faces on a round's first check (rc->n_query) and, for a refit, the
// arrival counts of the carried tree's nodes (leaves: their number). They were five memsets and kernels of their own.
__global__ void __launch_bounds__(256) k_boxes(const int4* __restrict__ tri, const float4* __restrict__ pos,
                                                RoundCounters* rc, float4* box_lo, float4* box_hi, int* live,
                                                unsigned* scene, int all_faces, BvhQuery q, int* xq_count, int* visit,
                                                const int* leaves, int* sort_ctl) {
    pdl_wait();
    if (!leaves)
        for (int i = gtid(); i < kSortCtl; i += gstride()) sort_ctl[i] = 0;
    if (gtid() == 0) {
        rc->pad[1] = rc->pad[2] = rc->pad[3] = 0;  // pair list length, query count, redo count
        *xq_count = 0;
    }
    if (leaves) {
        const int m = *leaves - 1;
        for (int i = gtid(); i < m; i += gstride()) visit[i] = 0;
    }
    const bool count = q.flags && rc->passes == 0;
    int marked = 0;
    const int n = rc->n_tris;
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int f = gtid(); f < n; f += gstride()) {
        int4 t = tri[f];
        int is_live = (t.x != -1);
        if (!leaves) live[f] = all_faces ? 1 : is_live;
        if (q.hit) q.hit[f] = 0;
        if (count) marked += q.flags[f];
        if (!is_live) {
            if (all_faces) {  // an empty box: overlaps nothing
                box_lo[f] = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
                box_hi[f] = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
            }
            continue;
        }
        float4 a = pos[t.x], b = pos[t.y], c = pos[t.z];
        float4 lo = make_float4(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)), 0.f);
        float4 hi = make_float4(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)), 0.f);
        box_lo[f] = lo;
        box_hi[f] = hi;
        mn[0] = fminf(mn[0], lo.x); mn[1] = fminf(mn[1], lo.y); mn[2] = fminf(mn[2], lo.z);
        mx[0] = fmaxf(mx[0], hi.x); mx[1] = fmaxf(mx[1], hi.y); mx[2] = fmaxf(mx[2], hi.z);
    }
    if (count) {
        for (int o = 16; o > 0; o >>= 1) marked += __shfl_xor_sync(0xffffffffu, marked, o);
        if ((threadIdx.x & 31) == 0 && marked) atomicAdd(&rc->n_query, marked);
    }
    if (leaves) return;  // a refit has no codes to make
    if (gtid() == 0) live[n] = 0;
    // one atomic per block and bound: one per warp (58,000 on six addresses) took most of the kernel's 43 us on
    // 327,680 faces
    __shared__ float sm[6][8];
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
    if (threadIdx.x < 3) {
        float l = sm[threadIdx.x][0], h = sm[3 + threadIdx.x][0];
        for (int w = 1; w < 8; ++w) {
            l = fminf(l, sm[threadIdx.x][w]);
            h = fmaxf(h, sm[3 + threadIdx.x][w]);
        }
        if (l <= h) {
            atomicMin(&scene[threadIdx.x], f2ord(l));
            atomicMax(&scene[3 + threadIdx.x], f2ord(h));
        }
    }
}

// ---------------------------------------------------------------- Morton codes of live faces
// fmesh (many meshes in one numbering): the key's top mesh_bits hold the face's mesh and the rest the top bits of its
// Morton code, so that the sort groups each mesh's faces and every Karras node under a mesh boundary covers one mesh
__global__ void __launch_bounds__(256) k_morton(const RoundCounters* rc, const int* live_scan, const float4* box_lo,
                                                 const float4* box_hi, const unsigned* scene, unsigned* keys, int* vals,
                                                 const int* __restrict__ fmesh, int mesh_bits, int* visit) {
    pdl_wait();
    const int n = rc->n_tris;
    float lo[3], ext[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lo[d] = ord2f(scene[d]);
        float hi = ord2f(scene[3 + d]);
        ext[d] = hi - lo[d];
    }
    for (int f = gtid(); f < n; f += gstride()) {
        int i = live_scan[f];
        if (live_scan[f + 1] == i) continue;
        float4 a = box_lo[f], b = box_hi[f];
        float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
        unsigned q[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float t = ext[d] > 0.f ? (c[d] - lo[d]) / ext[d] : 0.f;
            t = fminf(fmaxf(t * 1024.0f, 0.0f), 1023.0f);
            q[d] = (unsigned)t;
        }
        unsigned key = expand10(q[0]) * 4u + expand10(q[1]) * 2u + expand10(q[2]);
        if (fmesh) {
            const unsigned m = (unsigned)fmesh[f];
            key = mesh_bits <= 2 ? ((m << 30) | key) : ((m << (32 - mesh_bits)) | (key >> (mesh_bits - 2)));
        }
        keys[i] = key;
        vals[i] = f;
        visit[i] = 0;  // the nodes' arrival counts (one node fewer than leaves)
    }
}

// ---------------------------------------------------------------- stable LSD radix sort
__device__ __forceinline__ void sort_chunk(int n, int tile, int tiles, int& lo, int& hi) {
    long long chunk = ((long long)n + tiles - 1) / tiles;
    chunk = (chunk + kSortThreads - 1) / kSortThreads * kSortThreads;
    long long a = chunk * tile, b = a + chunk;
    lo = (int)(a < n ? a : n);
    hi = (int)(b < n ? b : n);
}

__global__ void __launch_bounds__(kSortThreads) k_rs_hist(const unsigned* __restrict__ keys, const int* d_n, int shift,
                                                          int* hist) {
    pdl_wait();
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    int lo, hi;
    sort_chunk(*d_n, blockIdx.x, gridDim.x, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += kSortThreads) atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1);
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Scatters keys [lo, hi) by the digit at `shift`, base[d] being the place of the first one with digit d (shared; it moves on
// with the keys). Each tile of 256 keys is ranked stably: lanes of a warp with the same digit find each other with
// __match_any_sync, warps are ordered through per-warp digit counts in shared memory.
struct SortShared {
    int base[256], wcnt[kSortThreads / 32][256], tot[256];
};
__device__ __forceinline__ void sort_scatter(const unsigned* kin, const int* vin, unsigned* kout, int* vout, int lo, int hi,
                                             int shift, SortShared& S) {
    constexpr int W = kSortThreads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int w = 0; w < W; ++w) S.wcnt[w][threadIdx.x] = 0;
    __syncthreads();
    for (int t0 = lo; t0 < hi; t0 += kSortThreads) {
        const int i = t0 + threadIdx.x;
        const bool valid = i < hi;
        unsigned key = valid ? kin[i] : 0u;
        int val = valid ? vin[i] : 0;
        const int dig = valid ? (int)((key >> shift) & 0xFF) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, dig);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) S.wcnt[warp][dig] = __popc(peers);
        __syncthreads();
        {
            int run = 0;
            for (int w = 0; w < W; ++w) {
                int c = S.wcnt[w][threadIdx.x];
                S.wcnt[w][threadIdx.x] = run;
                run += c;
            }
            S.tot[threadIdx.x] = run;
        }
        __syncthreads();
        if (valid) {
            const int dst = S.base[dig] + S.wcnt[warp][dig] + rank;
            kout[dst] = key;
            vout[dst] = val;
        }
        __syncthreads();
        S.base[threadIdx.x] += S.tot[threadIdx.x];
        for (int w = 0; w < W; ++w) S.wcnt[w][threadIdx.x] = 0;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kSortThreads) k_rs_scatter(const unsigned* __restrict__ kin, const int* __restrict__ vin,
                                                             unsigned* kout, int* vout, const int* d_n, int shift,
                                                             const int* hist) {
    pdl_wait();
    __shared__ SortShared S;
    S.base[threadIdx.x] = hist[threadIdx.x * gridDim.x + blockIdx.x];
    int lo, hi;
    sort_chunk(*d_n, blockIdx.x, gridDim.x, lo, hi);
    sort_scatter(kin, vin, kout, vout, lo, hi, shift, S);
}

// Up to kFusedTiles tiles: one kernel counts the digits of all four passes (ctl's first 1024 words, zeroed by k_boxes), and a
// pass is one launch: a tile publishes its own digit counts, waits for the tiles before it, and adds theirs up. Tiles are
// taken in the order the blocks start, so a tile only waits for blocks that run already; the wait is bounded, and a tile
// whose counts have not come by then is counted again by the one that waits, from the pass's keys, so that no place is
// ever formed from counts that were not published. In place of a count, a scan and a scatter launch a pass; with more
// tiles the sums over them (256 tiles^2 / 2 words) cost more than the scan (one intersection check of 327,680 faces, 160
// tiles: 515 -> 532 us). One tile (up to
// 2048 keys): all passes in one block. Twelve launches to five, to one for one tile: a stage-2 run from 1,280 faces 4.44 ->
// 4.33 ms, from 20,480 faces 14.25 -> 14.02 ms.
__global__ void __launch_bounds__(kSortThreads) k_rs_digits(const unsigned* __restrict__ keys, const int* d_n, int* total) {
    pdl_wait();
    __shared__ int h[4][256];
    for (int k = 0; k < 4; ++k) h[k][threadIdx.x] = 0;
    __syncthreads();
    int lo, hi;
    sort_chunk(*d_n, blockIdx.x, gridDim.x, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += kSortThreads) {
        const unsigned key = keys[i];
#pragma unroll
        for (int k = 0; k < 4; ++k) atomicAdd(&h[k][(key >> (8 * k)) & 0xFF], 1);
    }
    __syncthreads();
    for (int k = 0; k < 4; ++k)
        if (h[k][threadIdx.x]) atomicAdd(&total[256 * k + threadIdx.x], h[k][threadIdx.x]);
}

__global__ void __launch_bounds__(kSortThreads) k_rs_pass(const unsigned* __restrict__ kin, const int* __restrict__ vin,
                                                          unsigned* kout, int* vout, const int* d_n, int shift,
                                                          const int* __restrict__ total, int* ticket, int* ready,
                                                          int* hist, int wait_limit) {
    pdl_wait();
    __shared__ SortShared S;
    __shared__ int h[256], sm[33], s_tile;
    __shared__ unsigned s_late;  // the tiles before this one whose counts have not come
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1);
    h[threadIdx.x] = 0;
    __syncthreads();
    const int tile = s_tile, n = *d_n;
    int lo, hi;
    sort_chunk(n, tile, gridDim.x, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += kSortThreads) atomicAdd(&h[(kin[i] >> shift) & 0xFF], 1);
    __syncthreads();
    __stcg(&hist[256 * tile + threadIdx.x], h[threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("st.release.gpu.global.s32 [%0], 1;" ::"l"(&ready[tile]) : "memory");
    }
    if (threadIdx.x < 32) {  // a lane to an earlier tile (at most kFusedTiles - 1)
        int there = (int)threadIdx.x >= tile;
        for (int spins = 0; !there && spins < wait_limit; ++spins)
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(there) : "l"(&ready[threadIdx.x]) : "memory");
        const unsigned late = __ballot_sync(0xffffffffu, !there);
        if (threadIdx.x == 0) s_late = late;
    }
    int all;
    int at = block_exclusive_scan(total[threadIdx.x], &all, sm);  // its barriers follow the waits
    const unsigned late = s_late;
    if (late == 0u) {
#pragma unroll 8
        for (int k = 0; k < tile; ++k) at += __ldcg(&hist[256 * k + threadIdx.x]);
    } else {
        for (int k = 0; k < tile; ++k) {
            if (!((late >> k) & 1u)) {
                at += __ldcg(&hist[256 * k + threadIdx.x]);
                continue;
            }
            __syncthreads();  // the counts of the tile before are no longer read
            h[threadIdx.x] = 0;
            __syncthreads();
            int klo, khi;
            sort_chunk(n, k, gridDim.x, klo, khi);
            for (int i = klo + threadIdx.x; i < khi; i += kSortThreads) atomicAdd(&h[(kin[i] >> shift) & 0xFF], 1);
            __syncthreads();
            at += h[threadIdx.x];
        }
    }
    S.base[threadIdx.x] = at;
    if (hi > lo) sort_scatter(kin, vin, kout, vout, lo, hi, shift, S);
}

__global__ void __launch_bounds__(kSortThreads) k_rs_one_tile(unsigned* k0, int* v0, unsigned* k1, int* v1, const int* d_n) {
    pdl_wait();
    __shared__ SortShared S;
    __shared__ int h[256], sm[33];
    const int n = *d_n;
    for (int pass = 0; pass < 4; ++pass) {
        const unsigned* kin = pass & 1 ? k1 : k0;
        h[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += kSortThreads) atomicAdd(&h[(kin[i] >> (8 * pass)) & 0xFF], 1);
        __syncthreads();
        int all;
        S.base[threadIdx.x] = block_exclusive_scan(h[threadIdx.x], &all, sm);
        sort_scatter(kin, pass & 1 ? v1 : v0, pass & 1 ? k0 : k1, pass & 1 ? v0 : v1, 0, n, 8 * pass, S);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- Karras topology
__device__ __forceinline__ int delta(const unsigned* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned a = k[i], b = k[j];
    if (a != b) return __clz(a ^ b);
    return 32 + __clz((unsigned)(i ^ j));
}

__global__ void __launch_bounds__(256) k_karras(const RoundCounters* rc, const unsigned* keys, int2* child, int* iparent,
                                                 int* lparent, int2* range) {
    pdl_wait();
    const int n = rc->n_live;
    if (n == 1 && gtid() == 0) lparent[0] = -1;
    for (int i = gtid(); i < n - 1; i += gstride()) {
        const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = delta(keys, n, i, i - d);
        int lmax = 2;
        while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
        int l = 0;
        for (int t = lmax >> 1; t >= 1; t >>= 1)
            if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
        const int j = i + l * d;
        const int dnode = delta(keys, n, i, j);
        int s = 0;
        int t = l;
        do {
            t = (t + 1) >> 1;
            if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        } while (t > 1);
        const int gamma = i + s * d + (d < 0 ? -1 : 0);
        const int lo = min(i, j), hi = max(i, j);
        range[i] = make_int2(lo, hi);
        int left, right;
        if (lo == gamma) {
            left = ~gamma;
            lparent[gamma] = i;
        } else {
            left = gamma;
            iparent[gamma] = i;
        }
        if (hi == gamma + 1) {
            right = ~(gamma + 1);
            lparent[gamma + 1] = i;
        } else {
            right = gamma + 1;
            iparent[gamma + 1] = i;
        }
        child[i] = make_int2(left, right);
        if (i == 0) iparent[0] = -1;
    }
}

// Bottom-up boxes over tiles of kTileLeaves consecutive leaves, one thread per leaf. A Karras node covers a
// contiguous leaf range with its own index at one end, so every node whose range lies inside a tile has its
// index inside the tile too: those nodes count arrivals and keep their boxes in shared memory (the tile's leaf
// boxes are staged there as well). A chain that reaches a node whose range leaves the tile counts its arrival
// there in global memory (visit[], zeroed by the leaf kernels), with its own box in nlo/nhi; the second arrival
// queues the node (upq: count, then nodes) and stops, and k_bottom_up_upper finishes the nodes above the tiles,
// so a block never waits at its next tile for a chain climbing the upper tree. The second arrival at a node
// writes its packed record (kPack) and, with kNodes, its box to nlo/nhi. A node's range, children and parent are
// loaded together before its arrival count.
constexpr int kTileLeaves = 512;
constexpr int kTileThreads = kTileLeaves;

// Arrival counts of the bottom-up pass: a release add (the arriving child's box, stored before, becomes visible
// with the count) and an acquire-release add (the second arrival also sees the first child's box).
__device__ __forceinline__ int arrive_release(int* p) {
    int old;
    asm volatile("atom.release.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}
__device__ __forceinline__ int arrive_acq_rel(int* p) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

// The face id of a packed leaf with its query bit
__device__ __forceinline__ int packed_face(int f, const int* qflag) {
    return qflag && f >= 0 && qflag[f] ? f | kQueryBit : f;
}
// The packed 64-byte record of node p (both children's boxes, child references, leaf face ids fa and fc).
__device__ __forceinline__ void write_packed(int p, int2 c, float4 alo, float4 ahi, float4 clo, float4 chi, int fa,
                                             int fc, float4* packed) {
    float4* rec = packed + 4 * (size_t)p;
    alo.w = __int_as_float(c.x);
    ahi.w = __int_as_float(fa);
    clo.w = __int_as_float(c.y);
    chi.w = __int_as_float(fc);
    rec[0] = alo;
    rec[1] = ahi;
    rec[2] = clo;
    rec[3] = chi;
}

// From node p, both of whose children are done: its box from the children's boxes in global memory (and its
// packed record), then on to the parent as long as this is the parent's second arrival.
template <bool kPack>
__device__ void climb_from(RoundCounters* rc, int p, const int2* child, const int* iparent, const float4* llo,
                           const float4* lhi, float4* nlo, float4* nhi, int* visit, const int* leaf_face,
                           const int* qflag, float4* packed) {
    {
        int guard = 0;
        int2 c = child[p];
        int pp = iparent[p];
        while (p >= 0) {
            if (++guard > 4096) {
                atomicOr(&rc->status, kErrIterLimit);
                break;
            }
            float4 alo, ahi, clo, chi;
            if (c.x < 0) { alo = __ldcg(&llo[~c.x]); ahi = __ldcg(&lhi[~c.x]); }
            else { alo = __ldcg(&nlo[c.x]); ahi = __ldcg(&nhi[c.x]); }
            if (c.y < 0) { clo = __ldcg(&llo[~c.y]); chi = __ldcg(&lhi[~c.y]); }
            else { clo = __ldcg(&nlo[c.y]); chi = __ldcg(&nhi[c.y]); }
            const float4 blo = make_float4(fminf(alo.x, clo.x), fminf(alo.y, clo.y), fminf(alo.z, clo.z), 0.f);
            const float4 bhi = make_float4(fmaxf(ahi.x, chi.x), fmaxf(ahi.y, chi.y), fmaxf(ahi.z, chi.z), 0.f);
            __stcg(&nlo[p], blo);  // the parent's second arrival reads it
            __stcg(&nhi[p], bhi);
            if (kPack)
                write_packed(p, c, alo, ahi, clo, chi, c.x < 0 ? packed_face(__ldcg(&leaf_face[~c.x]), qflag) : -1,
                             c.y < 0 ? packed_face(__ldcg(&leaf_face[~c.y]), qflag) : -1, packed);
            if (pp < 0) break;
            // the parent's topology is fixed: loaded before its arrival count, not after
            const int2 cn = child[pp];
            const int ppn = iparent[pp];
            if (arrive_acq_rel(&visit[pp]) == 0) break;
            p = pp;
            c = cn;
            pp = ppn;
        }
    }
}

// kLeaf: where the leaves' boxes come from. kLeafGiven: llo/lhi; kLeafBuild: the boxes of the leaves' faces (leaf_face);
// kLeafReuse: the same for a carried tree, *meta leaves, with the face ids of new_ids where it is given (they become
// leaf_face); a leaf whose face is gone has an empty box. llo/lhi receive the boxes for the nodes above the tile.
// The tile's topology is loaded into shared memory with its leaves: loaded from global memory node by node, it put a
// dependent load of an L2 latency into every level of the climb.
enum { kLeafGiven = 0, kLeafBuild = 1, kLeafReuse = 2 };

template <bool kPack, bool kNodes, int kLeaf>
__global__ void __launch_bounds__(kTileThreads, 3) k_bottom_up_tiles(RoundCounters* rc, const int2* child,
                                                                  const int* iparent, const int* lparent,
                                                                  const int2* range, float4* llo, float4* lhi, float4* nlo,
                                                                  float4* nhi, int* visit, int* leaf_face,
                                                                  const int* __restrict__ new_ids,
                                                                  const float4* __restrict__ box_lo,
                                                                  const float4* __restrict__ box_hi,
                                                                  const int* __restrict__ qflag, float4* packed, int* meta,
                                                                  const int* active, int* upq, int climb) {
    pdl_wait();
    __shared__ int svisit[kTileLeaves], sface[kTileLeaves], sparent[kTileLeaves];
    __shared__ int2 srange[kTileLeaves], schild[kTileLeaves];
    __shared__ float4 slo[kTileLeaves], shi[kTileLeaves];    // internal nodes a .. b-2
    __shared__ float4 sllo[kTileLeaves], slhi[kTileLeaves];  // leaves a .. b-1
    if (active && *active == 0) return;
    const int n = kLeaf == kLeafReuse ? *meta : rc->n_live;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (kLeaf == kLeafReuse) rc->n_live = n;
        else if (kPack) *meta = n;
    }
    // climb: one tile per block, and a chain leaving its tile climbs on here, nothing waits for it; else several
    // tiles per block, and the nodes above the tiles are queued for k_bottom_up_upper
    // tiles in a block-stride loop: the leaf count is read on the device and may exceed the launch's bound
    for (int a = blockIdx.x * kTileLeaves; a < n; a += gridDim.x * kTileLeaves) {
        const int b = min(a + kTileLeaves, n);  // leaves [a, b)
        const int leaf = a + threadIdx.x;
        __syncthreads();  // the previous tile's shared state is no longer read
        svisit[threadIdx.x] = 0;
        float4 blo = make_float4(0.f, 0.f, 0.f, 0.f), bhi = blo;
        int p = -1;
        if (leaf < b) {
            p = lparent[leaf];
            if (leaf < n - 1) {
                srange[threadIdx.x] = range[leaf];
                schild[threadIdx.x] = child[leaf];
                sparent[threadIdx.x] = iparent[leaf];
            }
            if constexpr (kLeaf == kLeafGiven) {
                blo = __ldcg(&llo[leaf]);
                bhi = __ldcg(&lhi[leaf]);
                if (kPack) sface[threadIdx.x] = packed_face(leaf_face[leaf], qflag);
            } else {
                int f;
                if (kLeaf == kLeafReuse && new_ids) {
                    f = new_ids[leaf];
                    __stcg(&leaf_face[leaf], f);
                } else {
                    f = leaf_face[leaf];
                }
                if (f >= 0) {
                    blo = box_lo[f];
                    bhi = box_hi[f];
                } else {
                    blo = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
                    bhi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
                }
                __stcg(&llo[leaf], blo);
                __stcg(&lhi[leaf], bhi);
                if (kPack) sface[threadIdx.x] = packed_face(f, qflag);
            }
            sllo[threadIdx.x] = blo;
            slhi[threadIdx.x] = bhi;
        }
        __syncthreads();
        // up to the tile's edge, in shared memory alone
        int ref = ~leaf;
        int guard = 0;
        bool leaves_tile = false;
        while (p >= 0) {
            if (++guard > 4096) {
                atomicOr(&rc->status, kErrIterLimit);
                break;
            }
            // a node's index is one end of its range: a node with its index outside the tile leaves the tile
            const int k = p - a;
            if (!(p >= a && p < b && srange[k].x >= a && srange[k].y < b)) {
                leaves_tile = true;
                break;
            }
            __threadfence_block();
            if (atomicAdd(&svisit[k], 1) == 0) break;
            __threadfence_block();
            // both children are in this tile
            const int2 c = schild[k];
            const float4 alo = c.x < 0 ? sllo[~c.x - a] : slo[c.x - a], ahi = c.x < 0 ? slhi[~c.x - a] : shi[c.x - a];
            const float4 clo = c.y < 0 ? sllo[~c.y - a] : slo[c.y - a], chi = c.y < 0 ? slhi[~c.y - a] : shi[c.y - a];
            blo = make_float4(fminf(alo.x, clo.x), fminf(alo.y, clo.y), fminf(alo.z, clo.z), 0.f);
            bhi = make_float4(fmaxf(ahi.x, chi.x), fmaxf(ahi.y, chi.y), fmaxf(ahi.z, chi.z), 0.f);
            slo[k] = blo;
            shi[k] = bhi;
            ref = p;
            p = sparent[k];
        }
        // the chains that leave the tile go on before the tile's records are written, whose stores they need not wait
        // for: this child's box goes to global memory for the other child's chain; with several tiles per block the
        // second arrival queues p for k_bottom_up_upper instead of climbing on, so that no chain through the upper
        // tree holds this block at the next tile's barrier
        if (leaves_tile) {
            if (ref >= 0) {
                __stcg(&nlo[ref], blo);
                __stcg(&nhi[ref], bhi);
            }
            if (!climb) {
                if (arrive_release(&visit[p]) != 0) upq[1 + atomicAdd(upq, 1)] = p;
            } else if (arrive_acq_rel(&visit[p]) != 0) {
                climb_from<kPack>(rc, p, child, iparent, llo, lhi, nlo, nhi, visit, leaf_face, qflag, packed);
            }
        }
        __syncthreads();
        // the tile's own nodes, one per thread: consecutive records
        const int k = threadIdx.x;
        if (leaf < b && leaf < n - 1 && srange[k].x >= a && srange[k].y < b) {
            const int2 c = schild[k];
            if (kNodes) {
                __stcg(&nlo[leaf], slo[k]);
                __stcg(&nhi[leaf], shi[k]);
            }
            if (kPack)
                write_packed(leaf, c, c.x < 0 ? sllo[~c.x - a] : slo[c.x - a], c.x < 0 ? slhi[~c.x - a] : shi[c.x - a],
                             c.y < 0 ? sllo[~c.y - a] : slo[c.y - a], c.y < 0 ? slhi[~c.y - a] : shi[c.y - a],
                             c.x < 0 ? sface[~c.x - a] : -1, c.y < 0 ? sface[~c.y - a] : -1, packed);
        }
    }
}

// The nodes above the tiles (their leaf ranges span two tiles or more): each queued node (both children done)
// takes its box from the children's boxes in global memory, and climbs on as the second arrival at each parent.
template <bool kPack, bool kNodes>
__global__ void __launch_bounds__(256) k_bottom_up_upper(RoundCounters* rc, const int2* child, const int* iparent,
                                                         const float4* llo, const float4* lhi, float4* nlo,
                                                         float4* nhi, int* visit, const int* leaf_face,
                                                         const int* qflag, float4* packed, const int* upq,
                                                         const int* active) {
    pdl_wait();
    if (active && *active == 0) return;
    const int nq = upq[0];
    for (int k = gtid(); k < nq; k += gstride())
        climb_from<kPack>(rc, upq[1 + k], child, iparent, llo, lhi, nlo, nhi, visit, leaf_face, qflag, packed);
}

// blocks for k_bottom_up_tiles: a tile per block (a carried tree has up to 4/3 of the faces), except for a capped bound,
// whose block-stride loop covers any number
inline int tile_grid(int n_bound) {
    if (n_bound >= (1 << 19)) return std::max((n_bound + kTileLeaves - 1) / kTileLeaves, 3 * kNumSM);
    return (n_bound + n_bound / 3 + kTileLeaves) / kTileLeaves;
}

// The whole bottom-up pass: the tiles, then the nodes above them (climbed within the tiles' kernel where each block has
// one tile).
template <bool kPack, bool kNodes, int kLeaf>
void bottom_up(BvhBuffers& b, RoundCounters* rc, int n_bound, const int* new_ids, const int* qflag, const int* active,
               cudaStream_t s) {
    const bool climb = n_bound != (1 << 19);  // where callers cap their bounds
    if (!climb) cudaMemsetAsync(b.upq, 0, sizeof(int), s);
    const int gT = tile_grid(n_bound);
    pdl(k_bottom_up_tiles<kPack, kNodes, kLeaf>, gT, kTileThreads, 0, s)(
        rc, b.child, b.iparent, b.lparent, b.range, b.llo, b.lhi, b.nlo, b.nhi, b.visit, b.vals[0], new_ids, b.box_lo,
        b.box_hi, qflag, b.packed, b.meta, active, b.upq, climb ? 1 : 0);
    note_launch();
    if (climb) return;
    const int gU = std::max(1, std::min(gT, 4 * kNumSM));
    pdl(k_bottom_up_upper<kPack, kNodes>, gU, 256, 0, s)(rc, b.child, b.iparent, b.llo, b.lhi, b.nlo, b.nhi, b.visit,
                                                        b.vals[0], qflag, b.packed, b.upq, active);
    note_launch();
}

// ---------------------------------------------------------------- localized query
// 1. k_query_gather: the query faces in leaf (Morton) order, so that neighbouring lanes walk the same
//    part of the tree and test neighbouring faces.
// 2. k_traverse_list: the lanes of a warp walk the tree for its query faces with short stacks in shared memory, an idle
//    lane taking a subtree of another's walk, and list every overlapping leaf g as a candidate pair (f, g); a pair of two
//    query faces is listed only by the lower face index. Queries that overflow the list or the stack walk again
//    (redo_walks) and decide in place.
// 3. k_pairs: one thread per candidate pair decides it in both orders by float certificates, and queues the orders that
//    they leave open.
// 4. k_pairs_exact: one thread per queued order runs the reference's fp64 decision; then the walks of 2. that are to be
//    done again.
__device__ __forceinline__ bool decide_pair(int f, int g, const int4* __restrict__ tri, const float4* __restrict__ pos,
                                            float eps, unsigned& exact) {
    const int4 qt = tri[f], gt = tri[g];
    // two or three shared vertex indices: no intersection in either order (pair_certainly_disjoint), decided
    // before the positions are loaded (edge-adjacent faces are about a quarter of the candidate pairs)
    const int shared = (qt.x == gt.x) + (qt.x == gt.y) + (qt.x == gt.z) + (qt.y == gt.x) + (qt.y == gt.y) +
                       (qt.y == gt.z) + (qt.z == gt.x) + (qt.z == gt.y) + (qt.z == gt.z);
    if (shared >= 2) return false;
    const float4 q0 = pos[qt.x], q1 = pos[qt.y], q2 = pos[qt.z];
    const float4 g0 = pos[gt.x], g1 = pos[gt.y], g2 = pos[gt.z];
    PairGeom ga, gb;
    pair_geom(g0, g1, g2, gt, q0, q1, q2, qt, ga);  // reference order: the hit is "current"
    pair_geom(q0, q1, q2, qt, g0, g1, g2, gt, gb);  // the order seen from g's own query
    const bool need_a = !pair_certainly_disjoint(ga);
    const bool need_b = !pair_certainly_disjoint(gb);
    if (!need_a && !need_b) return false;
    exact += (unsigned)need_a + (unsigned)need_b;
    return (need_a && pair_decide_exact(g0, g1, g2, gt, q0, q1, q2, qt, eps)) ||
           (need_b && pair_decide_exact(q0, q1, q2, qt, g0, g1, g2, gt, eps));
}

// The query faces in leaf order: a block takes chunks of 1024 leaves and a place for each chunk's queries in one atomic
// (the chunks come in any order, which only sets which walks run side by side). In place of a flag kernel, a scan and a
// gather.
__global__ void __launch_bounds__(256) k_query_gather(RoundCounters* rc, const int* __restrict__ leaf_face,
                                                      const int* __restrict__ qflag, int* qsorted) {
    pdl_wait();
    __shared__ int sm[33];
    __shared__ int s_base;
    const int n = rc->n_live;
    for (int lo = blockIdx.x * 1024; lo < n; lo += gridDim.x * 1024) {
        int f[4], cnt = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = lo + 4 * threadIdx.x + k;
            f[k] = i < n ? leaf_face[i] : -1;  // -1: a leaf whose face is gone
            if (f[k] >= 0 && !qflag[f[k]]) f[k] = -1;
            cnt += f[k] >= 0;
        }
        int tot;
        int at = block_exclusive_scan(cnt, &tot, sm);
        if (threadIdx.x == 0) s_base = tot ? atomicAdd(&rc->pad[2], tot) : 0;
        __syncthreads();
        at += s_base;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (f[k] >= 0) qsorted[at++] = f[k];
        __syncthreads();
    }
}

__device__ __forceinline__ bool box_overlap4(float4 qlo, float4 qhi, float4 lo, float4 hi) {
    return !(qhi.x < lo.x || hi.x < qlo.x || qhi.y < lo.y || hi.y < qlo.y || qhi.z < lo.z || hi.z < qlo.z);
}

// First walk: candidate pairs go to the pair list. The loop is flat: a thread whose query is done takes its
// next query in the same iteration in which the other lanes of its warp take their next node. A lane without work or
// queries of its own takes the bottom entry of the pending stack of a lane that has some (the subtree nearest the root,
// the largest), together with that lane's query face and box: the r-th such lane gives to the r-th idle one through
// shared memory. Where there are fewer queries than lanes, each warp takes few of them (the first `own` lanes) and its other
// lanes live on shares, so that a walk of a hundred dependent loads is the work of several lanes from the start. With a
// lane per query and shares found by searching the votes bit by bit, a launch took 43 us of a round from 1,280 faces and
// 79 us of one from a height field of 286k.
// The pairs of a step go to the warp's chunk of the list, one atomic on its length serving many steps; unused slots of
// its last chunk are set to -1. A walk whose pair does not fit the list, or whose deferred siblings do not fit the short
// stack, stops and marks its query in redo[] (counted in rc->pad[3]) for the second walk.
// With fmesh, a query walks only the subtree of its own mesh (mesh_root; < 0: the mesh has one leaf, no pair).
__device__ __forceinline__ int query_root(int f, const int* __restrict__ fmesh, const int* __restrict__ mesh_root) {
    return fmesh ? mesh_root[fmesh[f]] : 0;
}

__global__ void __launch_bounds__(kQueryThreads) k_traverse_list(const float4* __restrict__ packed,
                                                                  const float4* __restrict__ box_lo,
                                                                  const float4* __restrict__ box_hi,
                                                                  const int* __restrict__ qsorted, int2* pairs_out,
                                                                  int pair_cap, RoundCounters* rc, int* redo,
                                                                  const int* __restrict__ fmesh,
                                                                  const int* __restrict__ mesh_root) {
    pdl_wait();
    __shared__ int stack[kShortStack][kQueryThreads];
    __shared__ int2 share_q[kQueryThreads];  // (query face, query), with the node in share_lo.w and the box
    __shared__ float4 share_lo[kQueryThreads], share_hi[kQueryThreads];
    int* n_list = &rc->pad[1];
    const int nq = rc->pad[2];
    const bool empty = rc->n_live < 2;
    unsigned long long npairs = 0;
    const int lane = threadIdx.x & 31, me = threadIdx.x, w0 = me & ~31;
    const unsigned lower = (1u << lane) - 1u;
    const int warps = gstride() >> 5;
    const int own = max(1, min(32, (nq + warps - 1) / warps));
    int cbase = -1, cused = kPairChunk;  // the warp's chunk
    int qi = (gtid() >> 5) * own + lane - warps * own;  // this lane's query iterator
    int wq = -1;                  // the query of the current walk (the lane's own or a shared one)
    bool supply = lane < own;     // this lane may still get queries of its own
    int f = 0, node = -1, sp = 0, bot = 0, guard = 0;  // pending entries: stack[bot .. sp)
    float4 qlo = make_float4(0.f, 0.f, 0.f, 0.f), qhi = qlo;
    while (true) {
        if (node < 0 && supply) {
            qi += warps * own;
            if (qi >= nq) {
                supply = false;
            } else {
                redo[qi] = 0;
                if (!empty) {
                    f = qsorted[qi];
                    node = query_root(f, fmesh, mesh_root);
                    if (node >= 0) {
                        wq = qi;
                        qlo = box_lo[f];
                        qhi = box_hi[f];
                        sp = bot = 0;
                        guard = 0;
                    }
                }
            }
        }
        // sharing, once lanes are out of queries (every lane takes part in the votes)
        const bool idle = node < 0 && !supply;
        const unsigned I = __ballot_sync(0xffffffffu, idle);
        if (I == 0xffffffffu) break;
        const bool gives = node >= 0 && sp > bot;
        const unsigned D = __ballot_sync(0xffffffffu, gives);
        if (I != 0u && D != 0u) {
            const int r = __popc((idle ? I : D) & lower), shares = min(__popc(I), __popc(D));
            if (gives && r < shares) {
                share_q[w0 + r] = make_int2(f, wq);
                share_lo[w0 + r] = make_float4(qlo.x, qlo.y, qlo.z, __int_as_float(stack[bot++][me]));
                share_hi[w0 + r] = qhi;
            }
            __syncwarp();
            if (idle && r < shares) {
                const int2 q = share_q[w0 + r];
                qlo = share_lo[w0 + r];
                qhi = share_hi[w0 + r];
                node = __float_as_int(qlo.w);
                f = q.x;
                wq = q.y;
                sp = bot = 0;
                guard = 0;
            }
            __syncwarp();
        }
        int hit0 = -1, hit1 = -1;
        bool abandon = false;
        if (node >= 0) {
            if (++guard > (1 << 22)) {
                atomicOr(&rc->status, kErrIterLimit);
                node = -1;
            } else {
                const float4* rec = packed + 4 * (size_t)node;
                const float4 alo = __ldg(rec), ahi = __ldg(rec + 1), blo = __ldg(rec + 2), bhi = __ldg(rec + 3);
                int next[2];
                int nn = 0;
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const float4 lo = side ? blo : alo, hi = side ? bhi : ahi;
                    if (!box_overlap4(qlo, qhi, lo, hi)) continue;
                    const int x = __float_as_int(lo.w);
                    if (x < 0) {
                        const int graw = __float_as_int(hi.w);
                        const int g = graw & ~kQueryBit;
                        if (g == f) continue;
                        if (g < f && (graw & kQueryBit)) continue;  // the lower query face owns the pair
                        if (side) hit1 = g;
                        else hit0 = g;
                    } else {
                        next[nn++] = x;
                    }
                }
                if (nn == 2) {
                    if (sp >= kShortStack && bot > 0) {  // entries given away at the bottom: move the rest down
                        for (int k = bot; k < sp; ++k) stack[k - bot][me] = stack[k][me];
                        sp -= bot;
                        bot = 0;
                    }
                    if (sp >= kShortStack) {
                        abandon = true;
                    } else {
                        stack[sp++][me] = next[1];
                        node = next[0];
                    }
                } else if (nn == 1) {
                    node = next[0];
                } else {
                    node = sp > bot ? stack[--sp][me] : -1;
                }
            }
        }
        const unsigned m0 = __ballot_sync(0xffffffffu, hit0 >= 0), m1 = __ballot_sync(0xffffffffu, hit1 >= 0);
        if ((m0 | m1) != 0u) {
            const int n0 = __popc(m0), n = n0 + __popc(m1);
            int fresh = -1;
            if (cused + n > kPairChunk) {
                if (lane == 0) fresh = atomicAdd(n_list, kPairChunk);
                fresh = __shfl_sync(0xffffffffu, fresh, 0);
            }
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int g = side ? hit1 : hit0;
                if (g < 0) continue;
                const int k = cused + (side ? n0 + __popc(m1 & lower) : __popc(m0 & lower));
                const int at = k < kPairChunk ? cbase + k : fresh + (k - kPairChunk);
                if (at < pair_cap) {
                    pairs_out[at] = make_int2(f, g);
                    ++npairs;
                } else {
                    abandon = true;
                }
            }
            cused += n;
            if (fresh >= 0) {
                cbase = fresh;
                cused -= kPairChunk;
            }
        }
        if (abandon) {
            redo[wq] = 1;
            atomicAdd(&rc->pad[3], 1);
            node = -1;
            sp = bot = 0;
        }
    }
    if (cbase >= 0)
        for (int k = cused + lane; k < kPairChunk && cbase + k < pair_cap; k += 32) pairs_out[cbase + k] = make_int2(-1, -1);
    __syncwarp();
    for (int o = 16; o > 0; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    if (lane == 0 && npairs) atomicAdd(&rc->n_pairs, npairs);
}

// k_pairs decides every listed pair by the float certificates; each order of a pair they cannot decide (the float64
// path, a few pairs in a thousand) is queued in xq, and k_pairs_exact runs those one per thread spread over every SM
// (decided where they were listed, they clustered in a few warps and the float64 pipes of a few SMs set the time).
// An order that finds the queue full is decided in place. Either way it sets the same flags.
// The certificate that settles nearly every pair is the same for both orders and is tried first and once; with the walk
// above, one intersection check of 327,680 faces went from 705 to 566 us; with a looser test before it (surely_one_side,
// and no divisions for the translation) to 543 us.
__global__ void __launch_bounds__(128, 8) k_pairs(const int4* __restrict__ tri, const float4* __restrict__ pos,
                                               const int2* __restrict__ pair_list, int pair_cap, unsigned char* hit,
                                               RoundCounters* rc, float eps, int4* xq, int xq_cap, int* xq_count) {
    pdl_wait();
    const int n = min(rc->pad[1], pair_cap);
    unsigned exact = 0;
    for (int i = gtid(); i < n; i += gstride()) {
        const int2 pr = pair_list[i];
        if (pr.x < 0) continue;  // an unused slot of a chunk
        const int f = pr.x, g = pr.y;
        const int4 qt = tri[f], gt = tri[g];
        // two or three shared vertex indices: no intersection in either order (pair_certainly_disjoint), decided
        // before the positions are loaded (edge-adjacent faces are about a quarter of the candidate pairs)
        const int shared = (qt.x == gt.x) + (qt.x == gt.y) + (qt.x == gt.z) + (qt.y == gt.x) + (qt.y == gt.y) +
                           (qt.y == gt.z) + (qt.z == gt.x) + (qt.z == gt.y) + (qt.z == gt.z);
        if (shared >= 2) continue;
        const float4 q0 = pos[qt.x], q1 = pos[qt.y], q2 = pos[qt.z];
        const float4 g0 = pos[gt.x], g1 = pos[gt.y], g2 = pos[gt.z];
        float m[3], reach;
        if (pair_translation_fast(g0, g1, g2, q0, q1, q2, m, reach)) {
            const Tri9 A = {{{g0.x - m[0], g0.y - m[1], g0.z - m[2]}, {g1.x - m[0], g1.y - m[1], g1.z - m[2]},
                             {g2.x - m[0], g2.y - m[1], g2.z - m[2]}}};
            const Tri9 B = {{{q0.x - m[0], q0.y - m[1], q0.z - m[2]}, {q1.x - m[0], q1.y - m[1], q1.z - m[2]},
                             {q2.x - m[0], q2.y - m[1], q2.z - m[2]}}};
            if (shared == 0) {
                if (surely_one_side(A, B, -1, reach) || surely_one_side(B, A, -1, reach)) continue;
            } else {
                // the shared vertex's corners
                const int sa = gt.x == qt.x || gt.x == qt.y || gt.x == qt.z ? 0 : gt.y == qt.x || gt.y == qt.y || gt.y == qt.z ? 1 : 2;
                const int id = sa == 0 ? gt.x : sa == 1 ? gt.y : gt.z;
                const int sb = qt.x == id ? 0 : qt.y == id ? 1 : 2;
                if (surely_one_side(A, B, sb, reach) && surely_one_side(B, A, sa, reach)) continue;
            }
        }
        PairGeom ga;
        pair_geom(g0, g1, g2, gt, q0, q1, q2, qt, ga);  // reference order: the hit is "current"
        // the order seen from g's own query: the same translated faces with A and B exchanged, unless the translation
        // rounds the other way; then the tests of one side against the other's plane are the same ones
        int mx, my, mz;
        pair_translation(q0, q1, q2, g0, g1, g2, mx, my, mz);
        const bool same = mx == ga.mx && my == ga.my && mz == ga.mz;
        if (same && pair_separated(ga)) continue;
        bool need_a, need_b;
        if (same) {
            need_a = !pair_negligible(ga.A, ga.B, ga.cmax);
            need_b = !pair_negligible(ga.B, ga.A, ga.cmax);
        } else {
            need_a = !pair_certainly_disjoint(ga);
            PairGeom gb;
            pair_geom(q0, q1, q2, qt, g0, g1, g2, gt, gb);
            need_b = !pair_certainly_disjoint(gb);
        }
        if (!need_a && !need_b) continue;
        exact += (unsigned)need_a + (unsigned)need_b;
        // one queue slot per order, taken for the whole warp by one atomic
        const unsigned am = __activemask();
        const int lane = threadIdx.x & 31, leader = __ffs(am) - 1;
        const unsigned ma = __ballot_sync(am, need_a), mb = __ballot_sync(am, need_b);
        int base = 0;
        if (lane == leader) base = atomicAdd(xq_count, __popc(ma) + __popc(mb));
        base = __shfl_sync(am, base, leader);
        const unsigned lower = (1u << lane) - 1u;
        const int at_a = base + __popc(ma & lower), at_b = base + __popc(ma) + __popc(mb & lower);
        bool h = false;
        if (need_a) {
            if (at_a < xq_cap) xq[at_a] = make_int4(f, g, 1, 0);
            else h = pair_decide_exact(g0, g1, g2, gt, q0, q1, q2, qt, eps);
        }
        if (need_b) {
            if (at_b < xq_cap) xq[at_b] = make_int4(f, g, 2, 0);
            else if (!h) h = pair_decide_exact(q0, q1, q2, qt, g0, g1, g2, gt, eps);
        }
        if (h) {
            hit[f] = 1;
            hit[g] = 1;
        }
    }
    for (int o = 16; o > 0; o >>= 1) exact += __shfl_xor_sync(0xffffffffu, exact, o);
    if ((threadIdx.x & 31) == 0 && exact) atomicAdd(&rc->n_exact, (unsigned long long)exact);
}

// Second walk, only when the first marked queries: each marked query walks the whole tree again with a stack
// deep enough for any tree (the Karras split prefix grows by at least one of the 62 key bits per level) and
// decides every pair in place (pairs already listed are decided twice, which sets the same flags).
__device__ void redo_walks(const float4* __restrict__ packed, const float4* __restrict__ box_lo,
                           const float4* __restrict__ box_hi, const int4* __restrict__ tri,
                           const float4* __restrict__ pos, const int* __restrict__ qsorted, unsigned char* hit,
                           RoundCounters* rc, float eps, const int* redo, const int* __restrict__ fmesh,
                           const int* __restrict__ mesh_root) {
    __shared__ int stack[kStackDepth][kExactThreads];
    const int nq = rc->pad[2];
    unsigned exact = 0;
    for (int qi = gtid(); qi < nq; qi += gstride()) {
        if (redo[qi] == 0) continue;
        const int f = qsorted[qi];
        int node = query_root(f, fmesh, mesh_root);
        if (node < 0) continue;
        const float4 qlo = box_lo[f], qhi = box_hi[f];
        int sp = 0;
        int guard = 0;
        while (true) {
            if (++guard > (1 << 22)) {
                atomicOr(&rc->status, kErrIterLimit);
                break;
            }
            const float4* rec = packed + 4 * (size_t)node;
            const float4 alo = __ldg(rec), ahi = __ldg(rec + 1), blo = __ldg(rec + 2), bhi = __ldg(rec + 3);
            int next[2];
            int nn = 0;
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const float4 lo = side ? blo : alo, hi = side ? bhi : ahi;
                if (!box_overlap4(qlo, qhi, lo, hi)) continue;
                const int x = __float_as_int(lo.w);
                if (x < 0) {
                    const int graw = __float_as_int(hi.w);
                    const int g = graw & ~kQueryBit;
                    if (g == f) continue;
                    if (g < f && (graw & kQueryBit)) continue;
                    if (decide_pair(f, g, tri, pos, eps, exact)) {
                        hit[f] = 1;
                        hit[g] = 1;
                    }
                } else {
                    next[nn++] = x;
                }
            }
            if (nn == 2) {
                if (sp >= kStackDepth) {
                    atomicOr(&rc->status, kErrStackOverflow);
                    break;
                }
                stack[sp++][threadIdx.x] = next[1];
                node = next[0];
            } else if (nn == 1) {
                node = next[0];
            } else {
                if (sp == 0) break;
                node = stack[--sp][threadIdx.x];
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) exact += __shfl_xor_sync(0xffffffffu, exact, o);
    if ((threadIdx.x & 31) == 0 && exact) atomicAdd(&rc->n_exact, (unsigned long long)exact);
}

// The queued pairs, one per thread, consecutive pairs on different SMs (block-cyclic: item k goes to block
// k mod blocks).
__global__ void __launch_bounds__(kExactThreads) k_pairs_exact(const int4* __restrict__ tri, const float4* __restrict__ pos,
                                                    const int4* __restrict__ xq, int xq_cap,
                                                    const int* __restrict__ xq_count, unsigned char* hit, float eps,
                                                    const float4* __restrict__ packed, const float4* __restrict__ box_lo,
                                                    const float4* __restrict__ box_hi, const int* __restrict__ qsorted,
                                                    RoundCounters* rc, const int* redo, const int* __restrict__ fmesh,
                                                    const int* __restrict__ mesh_root) {
    pdl_wait();
    const int n = min(*xq_count, xq_cap);
    for (long long k = (long long)threadIdx.x * gridDim.x + blockIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const int4 e = xq[k];
        const int f = e.x, g = e.y;
        const int4 qt = tri[f], gt = tri[g];
        const float4 q0 = pos[qt.x], q1 = pos[qt.y], q2 = pos[qt.z];
        const float4 g0 = pos[gt.x], g1 = pos[gt.y], g2 = pos[gt.z];
        const bool h = e.z == 1 ? pair_decide_exact(g0, g1, g2, gt, q0, q1, q2, qt, eps)
                                : pair_decide_exact(q0, q1, q2, qt, g0, g1, g2, gt, eps);
        if (h) {
            hit[f] = 1;
            hit[g] = 1;
        }
    }
    if (rc->pad[3] != 0) redo_walks(packed, box_lo, box_hi, tri, pos, qsorted, hit, rc, eps, redo, fmesh, mesh_root);
}

// The subtree root of each mesh: its live faces are the leaves [live_scan[f0], live_scan[f0 + nf]) of a tree built
// with mesh keys; a Karras node has one end of its range at its own index, so the node covering exactly that range
// is internal node lo or hi. -1 for a mesh with fewer than two leaves.
__global__ void k_mesh_roots(const RoundCounters* rc, const int* __restrict__ live_scan, const int2* __restrict__ range,
                             const int* __restrict__ mesh_f0, const int* __restrict__ mesh_nf, const int* d_count,
                             int* root) {
    pdl_wait();
    const int n = *d_count;
    const int n_live = rc->n_live;
    for (int m = gtid(); m < n; m += gstride()) {
        const int lo = live_scan[mesh_f0[m]], hi = live_scan[mesh_f0[m] + mesh_nf[m]] - 1;
        int r = -1;
        if (hi > lo && n_live >= 2) {
            const int2 a = range[lo];
            r = (a.x == lo && a.y == hi) ? lo : hi;
        }
        root[m] = r;
    }
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

size_t bvh_bytes(int cap) {
    size_t c = (size_t)cap + 1;
    size_t b = 0;
    b += 2 * align256(16 * c);              // box_lo / hi
    b += align256(4 * (c + 1));             // live_scan
    b += 2 * align256(4 * c);               // keys
    b += 2 * align256(4 * c);               // vals
    b += align256(4 * (256 * (size_t)kSortTiles + 1));
    b += align256(4 * kSortCtl);
    b += align256(8 * c);                   // child
    b += align256(8 * c);                   // range
    b += 2 * align256(4 * c);               // iparent, lparent
    b += 4 * align256(16 * c);              // nlo nhi llo lhi
    b += align256(4 * c);                   // visit
    b += align256(4 * (c + 1));             // upq
    b += align256(16 * std::min<size_t>(c, kExactQueue) + 16);  // xq and its count
    b += align256(4 * 8);                   // scene
    b += align256(4 * scan_scratch_ints());
    b += align256(64 * c);                  // packed internal nodes
    b += align256(16);                      // meta
    return b;
}

void bvh_carve(BvhBuffers& b, int cap, char* base, bool clear_scan_scratch) {
    size_t c = (size_t)cap + 1;
    char* p = base;
    auto take = [&](size_t bytes) {
        char* r = p;
        p += align256(bytes);
        return r;
    };
    b.cap = cap;
    b.box_lo = (float4*)take(16 * c);
    b.box_hi = (float4*)take(16 * c);
    b.live_scan = (int*)take(4 * (c + 1));
    b.keys[0] = (unsigned*)take(4 * c);
    b.keys[1] = (unsigned*)take(4 * c);
    b.vals[0] = (int*)take(4 * c);
    b.vals[1] = (int*)take(4 * c);
    b.hist = (int*)take(4 * (256 * (size_t)kSortTiles + 1));
    b.sort_ctl = (int*)take(4 * kSortCtl);
    b.child = (int2*)take(8 * c);
    b.range = (int2*)take(8 * c);
    b.iparent = (int*)take(4 * c);
    b.lparent = (int*)take(4 * c);
    b.nlo = (float4*)take(16 * c);
    b.nhi = (float4*)take(16 * c);
    b.llo = (float4*)take(16 * c);
    b.lhi = (float4*)take(16 * c);
    b.visit = (int*)take(4 * c);
    b.upq = (int*)take(4 * (c + 1));
    b.xq_cap = (int)std::min<size_t>(c, kExactQueue);
    b.xq = (int4*)take(16 * (size_t)b.xq_cap + 16);
    b.xq_count = reinterpret_cast<int*>(b.xq + b.xq_cap);
    b.scene = (unsigned*)take(4 * 8);
    b.scan_scratch = (int*)take(4 * scan_scratch_ints());
    b.packed = (float4*)take(64 * c);
    b.meta = (int*)take(16);
    if (clear_scan_scratch) scan_scratch_clear(b.scan_scratch);
}

void bvh_build(BvhBuffers& b, const int4* tri, const float4* pos, RoundCounters* rc, int n_tris_bound, cudaStream_t s,
               bool all_faces, const BvhQuery& query, bool nodes, const BvhMeshes* meshes) {
    cudaMemsetAsync(b.scene, 0xFF, 3 * sizeof(unsigned), s);
    cudaMemsetAsync(b.scene + 3, 0x00, 3 * sizeof(unsigned), s);
    const int gF = grid_for(n_tris_bound, 256);
    pdl(k_boxes, gF, 256, 0, s)(tri, pos, rc, b.box_lo, b.box_hi, b.live_scan, b.scene, all_faces ? 1 : 0, query,
                                   b.xq_count, b.visit, nullptr, b.sort_ctl); note_launch();
    exclusive_scan(b.live_scan, b.live_scan, &rc->n_tris, 1, &rc->n_live, b.scan_scratch, s, &rc->status, n_tris_bound);
    pdl(k_morton, gF, 256, 0, s)(rc, b.live_scan, b.box_lo, b.box_hi, b.scene, b.keys[0], b.vals[0],
                                meshes ? meshes->fmesh : nullptr, meshes ? meshes->bits : 0, b.visit); note_launch();
    // sort tiles from the launch's bound (about 2048 keys per tile; all kSortTiles from 2^19 on, where callers
    // cap their bounds); the histogram is
    // digit-major over the tiles, so its scan gives each tile's output offset per digit
    long long st = n_tris_bound >= (1 << 19) ? kSortTiles : ((long long)n_tris_bound + 2047) / 2048;
    const int sort_tiles = (int)(st < 1 ? 1 : (st > kSortTiles ? kSortTiles : st));
    if (sort_tiles == 1) {
        pdl(k_rs_one_tile, 1, kSortThreads, 0, s)(b.keys[0], b.vals[0], b.keys[1], b.vals[1], &rc->n_live); note_launch();
    } else if (sort_tiles <= kFusedTiles) {
        pdl(k_rs_digits, sort_tiles, kSortThreads, 0, s)(b.keys[0], &rc->n_live, b.sort_ctl); note_launch();
        for (int pass = 0; pass < 4; ++pass) {
            const int in = pass & 1, out = in ^ 1;
            int* ticket = b.sort_ctl + 1024 + pass * (1 + kFusedTiles);
            pdl(k_rs_pass, sort_tiles, kSortThreads, 0, s)(b.keys[in], b.vals[in], b.keys[out], b.vals[out], &rc->n_live,
                                                          8 * pass, b.sort_ctl + 256 * pass, ticket, ticket + 1, b.hist,
                                                          b.sort_wait); note_launch();
        }
    } else {
        for (int pass = 0; pass < 4; ++pass) {
            const int in = pass & 1, out = in ^ 1;
            pdl(k_rs_hist, sort_tiles, kSortThreads, 0, s)(b.keys[in], &rc->n_live, 8 * pass, b.hist); note_launch();
            exclusive_scan(b.hist, b.hist, nullptr, 256 * sort_tiles, nullptr, b.scan_scratch, s, &rc->status, 0);
            pdl(k_rs_scatter, sort_tiles, kSortThreads, 0, s)(b.keys[in], b.vals[in], b.keys[out], b.vals[out], &rc->n_live,
                                                             8 * pass, b.hist); note_launch();
        }
    }
    pdl(k_karras, gF, 256, 0, s)(rc, b.keys[0], b.child, b.iparent, b.lparent, b.range); note_launch();
    if (meshes) {
        pdl(k_mesh_roots, grid_for(meshes->count_bound, 256), 256, 0, s)(rc, b.live_scan, b.range, meshes->f0, meshes->nf,
                                                                          meshes->d_count, meshes->root);
        note_launch();
    }
    if (nodes) bottom_up<true, true, kLeafBuild>(b, rc, n_tris_bound, nullptr, query.flags, nullptr, s);
    else bottom_up<true, false, kLeafBuild>(b, rc, n_tris_bound, nullptr, query.flags, nullptr, s);
}

__global__ void __launch_bounds__(256) k_refit_leaves(const RoundCounters* rc, const int4* __restrict__ tri,
                                                      const float4* __restrict__ pos, const int* __restrict__ vals,
                                                      float4* llo, float4* lhi, int* visit, const int* active) {
    pdl_wait();
    if (active && *active == 0) return;
    const int n = rc->n_live;
    for (int i = gtid(); i < n; i += gstride()) {
        const int4 t = tri[vals[i]];
        const float4 a = pos[t.x], b = pos[t.y], c = pos[t.z];
        llo[i] = make_float4(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)), 0.f);
        lhi[i] = make_float4(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)), 0.f);
        if (i < n - 1) visit[i] = 0;
    }
}

void bvh_refit(BvhBuffers& b, const int4* tri, const float4* pos, RoundCounters* rc, int n_tris_bound, cudaStream_t s,
               const int* active) {
    const int gF = grid_for(n_tris_bound, 256);
    pdl(k_refit_leaves, gF, 256, 0, s)(rc, tri, pos, b.vals[0], b.llo, b.lhi, b.visit, active); note_launch();
    bottom_up<false, true, kLeafGiven>(b, rc, n_tris_bound, nullptr, nullptr, active, s);
}

void bvh_refit_faces(BvhBuffers& b, const int4* tri, const float4* pos, RoundCounters* rc, int n_tris_bound,
                     cudaStream_t s, bool next_round, const BvhQuery& query) {
    pdl(k_boxes, grid_for(n_tris_bound, 256), 256, 0, s)(tri, pos, rc, b.box_lo, b.box_hi, b.live_scan, b.scene, 1, query,
                                                       b.xq_count, b.visit, b.meta, nullptr); note_launch();
    bottom_up<true, false, kLeafReuse>(b, rc, n_tris_bound, next_round ? (const int*)b.keys[1] : nullptr, query.flags,
                                       nullptr, s);
}

BvhRemap bvh_remap(const BvhBuffers& b) { return {b.meta, b.vals[0], (int*)b.keys[1]}; }

void bvh_query(const BvhBuffers& b, const int4* tri, const float4* pos, const BvhQuery& query, int2* pair_list,
               int pair_cap, RoundCounters* rc, int n_query_bound, float eps, cudaStream_t s, const int* fmesh,
               const int* mesh_root) {
    // the query faces go to one of the sort's second buffers, free after the build
    pdl(k_query_gather, grid_for((n_query_bound + 3) / 4, 256), 256, 0, s)(rc, b.vals[0], query.flags, b.vals[1]);
    note_launch();
    // b.visit (free between a tree's bottom-up passes) holds the per-query redo marks
    // a function-local static initialiser runs once even when worker threads query concurrently
    static const int blocks_per_sm = [] {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_traverse_list, kQueryThreads, 0) != cudaSuccess || nb < 1)
            nb = 4;
        return nb;
    }();
    // four lanes a query while the GPU has room (k_traverse_list spreads them)
    pdl(k_traverse_list, grid_for(4ll * n_query_bound, kQueryThreads, blocks_per_sm), kQueryThreads, 0, s)(
        b.packed, b.box_lo, b.box_hi, b.vals[1], pair_list, pair_cap, rc, b.visit, fmesh, mesh_root);
    note_launch();
    pdl(k_pairs, grid_for((long long)pair_cap, 128, 16), 128, 0, s)(tri, pos, pair_list, pair_cap, query.hit, rc, eps, b.xq,
                                                                  b.xq_cap, b.xq_count);
    note_launch();
    pdl(k_pairs_exact, 4 * kNumSM, kExactThreads, 0, s)(tri, pos, b.xq, b.xq_cap, b.xq_count, query.hit, eps, b.packed,
                                                       b.box_lo, b.box_hi, b.vals[1], rc, b.visit, fmesh, mesh_root);
    note_launch();
}

}  // namespace pamo
