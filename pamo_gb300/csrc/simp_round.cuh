// Kernels of one stage-2 collapse round (host launchers). Every count is read from RoundCounters in device
// memory; the *_bound arguments only size the grids.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "lbvh.cuh"
#include "pamo_common.cuh"

namespace pamo {

// thrust::shuffle's bijection on [0, 2^bits), 2^bits >= m elements (at least 2^4)
struct FeistelSize {
    uint32_t lbits, rbits, lmask, rmask;
};
__host__ __device__ inline FeistelSize feistel_size(unsigned long long m) {
    uint32_t bits = 4;
    if (m > 16) {
        bits = 0;
        for (unsigned long long t = m - 1; t; t >>= 1) ++bits;
    }
    FeistelSize z;
    z.lbits = bits / 2;
    z.rbits = bits - bits / 2;
    z.lmask = (uint32_t)((1ull << z.lbits) - 1);
    z.rmask = (uint32_t)((1ull << z.rbits) - 1);
    return z;
}
struct Feistel {
    uint32_t key[24];  // the same for every size
    FeistelSize size;
    unsigned long long n;  // 2^bits
    unsigned long long m;
};
Feistel make_feistel(unsigned long long m);
__device__ __forceinline__ unsigned long long feistel(const Feistel& fb, const FeistelSize& z, unsigned long long idx) {
    uint32_t s0 = (uint32_t)(idx >> z.rbits), s1 = (uint32_t)(idx & z.rmask);
#pragma unroll 4
    for (int r = 0; r < 24; ++r) {
        const unsigned long long prod = 0xD2B74407B1CE6E93ull * (unsigned long long)s0;
        const uint32_t hi = (uint32_t)(prod >> 32);
        uint32_t lo = (uint32_t)prod;
        lo = (lo << (z.rbits - z.lbits)) | (s1 >> z.lbits);
        s0 = ((hi ^ fb.key[r]) ^ s1) & z.lmask;
        s1 = lo & z.rmask;
    }
    return ((unsigned long long)s0 << z.rbits) | (unsigned long long)s1;
}

// ---- set-up of a round ----
void launch_undo_bookkeeping(const int* verts_undo, int n_verts_undo, int is_stuck, int* tmp_undo, int* undo_list,
                             const int* pts_map, int pts_map_len, unsigned char* invalid, int invalid_len, cudaStream_t s);
void launch_load_points(const float* pts, int n, float4* pos, float4* orig_pos, int* occ, cudaStream_t s);
void launch_load_points4(const float4* pts, int n, float4* pos, float4* orig_pos, int* occ, cudaStream_t s);
void launch_load_tris(const int* tris, int n, int n_pts, int4* tri, RoundCounters* rc, cudaStream_t s);
void launch_load_tris4(const int4* tris, int n, int4* tri, cudaStream_t s);
void launch_shuffle_tris(const Feistel& fb, int* flags, int* scan_scratch, int4* tmp, int4* tri, int n, cudaStream_t s,
                         int* err = nullptr);
void launch_copy_tris(const int4* src, int4* dst, int n, cudaStream_t s);

// ---- adjacency ----
// The bookkeeping of the undo vertices carried into a device round (cusimp_free.cu:869-889), done beside the face counts:
// invalid marked, and in a stuck round the undo list restarted through the previous map. ls null: none.
struct UndoBook {
    const LoopState* ls = nullptr;
    const int* verts_undo = nullptr;
    int* tmp_undo = nullptr;
    int* undo_list = nullptr;
    const int* pts_map = nullptr;
    int map_len = 0;
    unsigned char* invalid = nullptr;
    int invalid_len = 0;
};
// with fgeo: also the per-face geometry the rings read (from pos; room for six float4 per face): a 64-byte record per
// face (fgeo[4f .. 4f + 3]: edge lengths, normal, corner positions), then the planes after all n faces' records, one
// float4 per face (fgeo[4n + f]) or, with plane_df (precision mode), a double-float pair (fgeo[4n + 2f], +1)
// rank: per face, its place in each corner's ring and its edges' places among those of their lower endpoints (three
// pairs), for launch_fill_adjacency
void launch_face_counts(const int4* tri, const RoundCounters* rc, int n_tris_bound, int* valence, int* ecount,
                        int* vedges, cudaStream_t s, const float4* pos, float4* fgeo, int2* rank, bool plane_df = false,
                        const UndoBook& book = UndoBook());
// d_cap (or null): the length of the edge costs as the reference sizes them, grown to the round's edges
void launch_fill_adjacency(const int4* tri, RoundCounters* rc, int n_tris_bound, const int* nt_off, const int2* rank,
                           int* nt, const int* edge_off, int2* edges, const int* voff, int* eorder, cudaStream_t s,
                           int* d_cap = nullptr);

// ---- cost, selection, collapse ----
// The rings sorted by face, and the quadrics.
// qlo (precision mode; needs the plane_df planes): each quadric as a double-float sum, hi parts to q, lo to qlo
// nxt, spc: per ring slot, the vertex after the ring's vertex in the slot's face and (the vertex before it, its corner)
// cost (or null), cost_len: the edge costs, zeroed when their length grew (launch_fill_adjacency)
void launch_ring_quadrics(const RoundCounters* rc, int n_pts_bound, const int* nt_off, int* nt, const int4* tri,
                          const float4* fgeo, Quadric* q, int* nxt, int2* spc, cudaStream_t s, Quadric* qlo = nullptr,
                          uint32_t* cost = nullptr, int cost_len = 0);
// mode: 0 the reference's arithmetic; precision mode 1 (double-float quadrics q + qlo, compensated sums) or 2 (as 1,
// placement at the quadric's minimiser, written to place[e]). raw (optional): each edge's cost before clamp and quantisation (NaN where
// none is computed); place (optional, required by mode 2): each edge's placement.
void launch_edge_cost(const RoundCounters* rc, int n_edges_bound, const int* eorder, const int2* edges, const int* nt_off,
                      const int* nt, const int4* tri, const float4* pos, const Quadric* q, const float4* fgeo,
                      const int* nxt, const int2* spc, const unsigned char* invalid, uint32_t* cost,
                      unsigned long long* vmin,
                      const float* d_scale, float tres, int is_stuck, cudaStream_t s, const int* is_stuck_dev = nullptr,
                      bool legacy = false, bool device_pow = false, int mode = 0, float* raw = nullptr,
                      float4* place = nullptr, const Quadric* qlo = nullptr);
// The edge cost of many meshes in one vertex numbering: the scale and is_stuck of each edge's mesh (vmesh of its
// lower vertex) come from mesh_scale and mesh_stuck.
void launch_edge_cost_batch(const RoundCounters* rc, int n_edges_bound, const int* eorder, const int2* edges,
                            const int* nt_off, const int* nt, const int4* tri, const float4* pos, const Quadric* q,
                            const float4* fgeo, const int* nxt, const int2* spc, const unsigned char* invalid,
                            uint32_t* cost,
                            unsigned long long* vmin, const float* mesh_scale, const int* mesh_stuck, const int* vmesh,
                            float tres, cudaStream_t s, bool device_pow = false);
// vmin: the least key (cost << 32 | edge) over the edges of each vertex
// tri and pos are the round's as it began (a collapse that would leave a skinny face is not made)
void launch_collapse(RoundCounters* rc, int n_edges_bound, const int2* edges, const uint32_t* cost,
                     uint32_t collapse_t, const unsigned long long* vmin, const int* nxt, const int2* spc,
                     const int* nt_off, const int* nt, int4* tri, float4* pos, int* occ, int* win, cudaStream_t s,
                     bool restore = true, const float4* place = nullptr);
// After the collapses: the winners' list, the degenerate faces removed and the edges with coincident endpoints counted in
// rc->n_line; with lines, also collapsed in edge order and appended to the list (up to line_cap), with rc->n_collapsed
// and rc->n_considered. Needs rc->pad[4] = 0, which a round starts with.
void launch_after_collapse(RoundCounters* rc, int n_edges_bound, int n_tris_bound, const int* win_scan, int* collapsed,
                           const int2* edges, const int* nt_off, const int* nt, int4* tri, float4* pos, int* occ,
                           int line_cap, bool lines, cudaStream_t s);

// ---- self-intersection rollback ----
void launch_mark_query(const RoundCounters* rc, int n_edges_bound, const int* collapsed, const int2* edges,
                       const int* nt_off, const int* nt, int* qflag, cudaStream_t s);
// fflags (or null): also the live faces of tri, as launch_live_flags
void launch_undo_check(RoundCounters* rc, int n_edges_bound, const int* collapsed, const int2* edges, const int* nt_off,
                       const int* nt, const unsigned char* hit, int* uflag, cudaStream_t s,
                       const int4* tri = nullptr, int* fflags = nullptr);
void launch_undo_apply(RoundCounters* rc, int n_edges_bound, const int* collapsed, const int* uscan, const int2* edges,
                       const int* nt_off, const int* nt, int4* tri, const int4* orig_tri, float4* pos,
                       const float4* orig_pos, int* occ, int* tmp_undo, int* undo_list, const int* pts_map,
                       int list_cap, cudaStream_t s);

// ---- outputs ----
void launch_live_flags(const RoundCounters* rc, int n_tris_bound, const int4* tri, int* flags, cudaStream_t s);
// check: also launch_after_check's counters; remap: also the carried tree's leaves in the new numbering
void launch_compact_mesh(RoundCounters* rc, int n_pts_bound, int n_tris_bound, const float4* pos, const int* occ,
                         const int* pts_map, const int4* tri, const int* face_scan, float4* out_pos, int4* out_tri,
                         cudaStream_t s, bool check = false, const BvhRemap& remap = BvhRemap());
void launch_export_round(const RoundCounters* rc, int n_pts, int n_tris, const float4* pos, const int4* tri,
                         const int* occ, const int* pts_map, const int* undo_list, float* verts, int* tris,
                         int* verts_occ, int* verts_map, int* verts_undo, int n_undo, cudaStream_t s);
void launch_export_mesh(int n_pts, int n_tris, const float4* pos, const int4* tri, const float* add, float* verts,
                        int* tris, cudaStream_t s);

// ---- whole-loop helpers ----
// One mesh's centring: center[0..2] = tris_mean (zero when not centring), center[4..9] scratch (order-preserving
// extents), *scale = the largest extent of the centred points, pos_out = the centred points.
struct CenterJob {
    const float* pts;
    const int* tris;
    int n_pts, n_tris;   // at least one each
    long long face0;     // the job's first face in the face means (the sum of the earlier jobs' n_tris)
    int chunk0;          // its first chunk (the sum of the earlier jobs' center_chunks)
    float* center;
    float* scale;
    float4* pos_out;
};
struct CenterJobs {
    CenterJob one;          // the job, where many is null
    const CenterJob* many;  // device array of n jobs
    int n, n_chunks;        // jobs and the sum of their center_chunks
};
int center_chunks(int n_tris);
size_t center_scratch_bytes(long long chunks);
// face_mean: three floats per face; scratch: center_scratch_bytes, 16-byte aligned; max_*: the largest job's sizes
void launch_center_jobs(const CenterJobs& J, float* face_mean, void* scratch, int max_tris, int max_pts, cudaStream_t s,
                        bool centre);
void launch_center(const float* pts, const int* tris, int n_pts, int n_tris, float* face_mean, void* scratch,
                   float* center, float* d_scale, float4* pos_out, cudaStream_t s, bool centre = true);
void launch_after_check(RoundCounters* rc, cudaStream_t s);

// ---- device-driven rounds: sizes from LoopState / RoundCounters, host values only bound the grids ----
// The start of a round in one launch: pos = orig_pos = the round's points, occ = 1 and occ[n_pts] = 0; tri = orig_tri = the
// round's faces; valence, vedges = 0 and vmin = ~0 over n_pts + 1 entries; qflag = 0 over n_tris + 1
// entries. With next (device-driven rounds; null: the sizes are rc's and the rest is not touched) also *ls = *next, rc as
// forward() sets it, the invalid table cleared where undo vertices are carried into a round that is not stuck, and
// pts_map_prev[0, n_pts) = pts_map (the previous round's map, read by this round's undo passes).
struct RoundStart {
    const LoopState* next = nullptr;
    LoopState* ls = nullptr;
    RoundCounters* rc = nullptr;
    unsigned char* invalid = nullptr;
    int invalid_len = 0;
    const int* pts_map = nullptr;
    int* pts_map_prev = nullptr;
    const float4* pts_in = nullptr;
    float4 *pos = nullptr, *orig_pos = nullptr;
    int* occ = nullptr;
    const int4* tri_in = nullptr;
    int4 *tri = nullptr, *orig_tri = nullptr;
    int *valence = nullptr, *vedges = nullptr, *qflag = nullptr;
    unsigned long long* vmin = nullptr;
};
void launch_round_prologue_dev(const RoundStart& r, int n_pts_bound, int n_tris_bound, cudaStream_t s);
void launch_round_end(const RoundCounters* rc, const LoopState* ls, LoopState* next, const int* undo_list, int* undo_in,
                      int undo_cap, int n_undo_bound, cudaStream_t s);

}  // namespace pamo
