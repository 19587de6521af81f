// vbd_self_contact.cu -- cloth self-contact for the VBD step on sm_100a.
//
// Restates the reference's particle self-contact path (SolverVBD with
// particle_enable_self_contact=True):
//   detection         TriMeshCollisionDetector.vertex_triangle_collision_detection /
//                     edge_edge_collision_detection (solvers/vbd/tri_mesh_collision.py:645-730;
//                     kernels geometry/kernels.py:1328-1497, :1499-1640), n-ring topological filter
//                     (tri_mesh_collision.py:123-233), rest-shape exclusion radius
//   forces            accumulate_self_contact_force_and_hessian (particle_vbd_kernels.py:1498-1639)
//   truncation        apply_planar_truncation_parallel_by_collision (:2133-2263) + apply_truncation_ts
//                     (:2266-2286) with max displacement margin * relaxation * 0.5
//                     (solver_vbd.py:2026-2063)
//   orchestration     solver_vbd.py:2065-2100 (detection before the forward step), :2540-2545
//                     (detection interval), :3221-3237 (positions become the displacement base)
//
// B200 design.  The reference refits two BVHs and runs 4 threads per primitive with atomics into
// the per-vertex force.  Here:
//   * a hashed uniform grid (cell = margin + longest rest edge) is rebuilt every detection in
//     four device passes -- count per bucket, exclusive scan (CUB), fill, query -- so no host
//     synchronisation is needed and a step stays graph-capturable.  A triangle / edge of at most
//     half a cell sits in the one bucket of its box centre's cell, a larger (stretched) one in
//     every cell its box overlaps; the count pass keeps each element's box;
//   * a query rejects candidates by box overlap before any filter or exact distance and skips
//     entries of other cells that share its bucket; a queue per warp hands the survivors to the
//     exact tests with every lane busy, and the accepted ones end in sorted per-vertex / per-edge
//     lists (so each pair is reported once);
//   * the detected pairs are laid out once per detection for the passes that every color runs over
//     them (entries per vertex for the forces, a flat pair table for the planes);
//   * forces are gathered per vertex of the current color, one warp per vertex taking its entries
//     round-robin in a fixed order (own vertex-triangle pairs, then the pairs of each incident
//     triangle, then the edge-edge pairs of each incident edge) and reduced with xor shuffles, so
//     results are deterministic (while no buffer overflows: below);
//   * truncation ratios are reduced with an integer atomicMin on the (non-negative) float bits,
//     which is exact and order-independent.
// Buffers are fixed-size (reference defaults: 32 triangles per vertex, 64 edges per edge; plus
// 32 vertices per triangle for the gather); candidates beyond a buffer are dropped and counted.  Which
// ones a full row keeps depends on scheduling, so runs repeat bit for bit only while the count is zero.
#include "vbd_self_contact.h"

#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include "vbd_self_contact_math.cuh"

namespace vbd {

namespace {

struct CellRange {
    int3 lo, hi;
};

__device__ __forceinline__ int cell_coord(float x, float inv) { return static_cast<int>(floorf(x * inv)); }

__device__ __forceinline__ CellRange cell_range(float3 lo, float3 hi, float inv) {
    CellRange r;
    r.lo = make_int3(cell_coord(lo.x, inv), cell_coord(lo.y, inv), cell_coord(lo.z, inv));
    r.hi = make_int3(cell_coord(hi.x, inv), cell_coord(hi.y, inv), cell_coord(hi.z, inv));
    return r;
}

__device__ __forceinline__ long long cell_count(const CellRange& r) {
    return (static_cast<long long>(r.hi.x) - r.lo.x + 1) * (static_cast<long long>(r.hi.y) - r.lo.y + 1) *
           (static_cast<long long>(r.hi.z) - r.lo.z + 1);
}

__device__ __forceinline__ unsigned cell_hash(int x, int y, int z, unsigned mask) {
    return ((static_cast<unsigned>(x) * 73856093u) ^ (static_cast<unsigned>(y) * 19349663u) ^
            (static_cast<unsigned>(z) * 83492791u)) &
           mask;
}

__device__ __forceinline__ float3 fmin3(float3 a, float3 b) { return f3(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z)); }
__device__ __forceinline__ float3 fmax3(float3 a, float3 b) { return f3(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z)); }

struct GridArgs {
    const float4* x;      // positions (internal order)
    const int4* elem;     // triangles or edges
    int n;
    bool tri;
    bool all_cells;       // every element goes into every cell its box overlaps (edge grid)
    float inv_cell;
    unsigned mask;
    int* cnt;
    const int* off;
    int* cur;
    int* items;
    float4* item_box;     // [2 cap] the box of every bucket entry, next to its id (fill pass)
    int cap;
    float4* box;          // [2n] element boxes (lo, hi; lo.w = 1 for a large element), count pass
    unsigned* counters;
};

__device__ __forceinline__ void elem_box(const GridArgs& a, int e, float3& lo, float3& hi) {
    const int4 el = a.elem[e];
    const float3 p0 = xyz(a.x[el.x]), p1 = xyz(a.x[el.y]);
    lo = fmin3(p0, p1);
    hi = fmax3(p0, p1);
    if (a.tri) {
        const float3 p2 = xyz(a.x[el.z]);
        lo = fmin3(lo, p2);
        hi = fmax3(hi, p2);
    }
}

__device__ __forceinline__ int3 center_cell(float4 lo, float4 hi, float inv) {
    return make_int3(cell_coord(0.5f * (lo.x + hi.x), inv), cell_coord(0.5f * (lo.y + hi.y), inv),
                     cell_coord(0.5f * (lo.z + hi.z), inv));
}

// Triangle grid (queried by points): a triangle whose half-extent is at most half a cell goes into
// the one bucket of its box centre's cell; a larger one (stretched) goes into every cell its box
// overlaps, up to kMaxLargeCells, and is flagged (lo.w = 1).  A vertex query then looks margin +
// half a cell around its point, however far the cloth stretches elsewhere.
// Edge grid (queried by edge boxes): every edge goes into every cell its box overlaps (flagged),
// so an edge query only covers its box grown by the margin -- for edges shorter than a cell that
// is fewer bucket entries than centre binning's extra half cell on every side -- and a pair is
// taken only in the first cell the two ranges share.
constexpr int kMaxLargeCells = 4096;

// What a bucket entry says about the cell it was put into, in the w components of its box:
//   lo.w: bit k set when the element's box begins before that cell along axis k (a small element: 0);
//   hi.w: the cell's coordinates modulo 1024 (buckets are shared by colliding cells; cells that
//         many apart hold no overlapping boxes).
__device__ __forceinline__ int cell_key(int x, int y, int z) { return (x & 1023) | ((y & 1023) << 10) | ((z & 1023) << 20); }

// A query takes an entry met in cell (x, y, z) of its range when the entry belongs to that cell and
// the cell is the first that the element shares with the range, so that every pair is met once: along
// each axis either the element or the query range begins there.  mask: query_mask of that cell.
__device__ __forceinline__ int query_mask(const CellRange& q, int x, int y, int z) {
    return (x != q.lo.x ? 1 : 0) | (y != q.lo.y ? 2 : 0) | (z != q.lo.z ? 4 : 0);
}
__device__ __forceinline__ bool takes(float4 blo, float4 bhi, int key, int mask) {
    return __float_as_int(bhi.w) == key && (__float_as_int(blo.w) & mask) == 0;
}

__global__ void grid_count_kernel(GridArgs a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.n) return;
    float3 lo, hi;
    elem_box(a, e, lo, hi);
    const float half = 0.5f * fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z);
    const bool large = a.all_cells || !(half <= 0.5f / a.inv_cell);
    const float4 l4 = make_float4(lo.x, lo.y, lo.z, large ? 1.f : 0.f), h4 = make_float4(hi.x, hi.y, hi.z, 0.f);
    a.box[2 * e] = l4;
    a.box[2 * e + 1] = h4;
    if (!large) {
        const int3 c = center_cell(l4, h4, a.inv_cell);
        atomicAdd(&a.cnt[cell_hash(c.x, c.y, c.z, a.mask)], 1);
        return;
    }
    const CellRange r = cell_range(lo, hi, a.inv_cell);
    if (!(cell_count(r) <= kMaxLargeCells)) {
        atomicAdd(&a.counters[kScGridOverflow], 1u);
        return;
    }
    for (int z = r.lo.z; z <= r.hi.z; ++z)
        for (int y = r.lo.y; y <= r.hi.y; ++y)
            for (int x = r.lo.x; x <= r.hi.x; ++x) atomicAdd(&a.cnt[cell_hash(x, y, z, a.mask)], 1);
}

__device__ __forceinline__ void put_entry(const GridArgs& a, int e, float4 lo, float4 hi, int x, int y, int z,
                                          int begun) {
    const unsigned h = cell_hash(x, y, z, a.mask);
    const int k = a.off[h] + atomicAdd(&a.cur[h], 1);
    if (k >= a.cap) {
        atomicAdd(&a.counters[kScGridOverflow], 1u);
        return;
    }
    a.items[k] = e;
    a.item_box[2 * k] = make_float4(lo.x, lo.y, lo.z, __int_as_float(begun));
    a.item_box[2 * k + 1] = make_float4(hi.x, hi.y, hi.z, __int_as_float(cell_key(x, y, z)));
}

__global__ void grid_fill_kernel(GridArgs a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.n) return;
    const float4 l4 = a.box[2 * e], h4 = a.box[2 * e + 1];
    if (l4.w == 0.f) {
        const int3 c = center_cell(l4, h4, a.inv_cell);
        put_entry(a, e, l4, h4, c.x, c.y, c.z, 0);
        return;
    }
    const CellRange r = cell_range(xyz(l4), xyz(h4), a.inv_cell);
    if (!(cell_count(r) <= kMaxLargeCells)) return;
    for (int z = r.lo.z; z <= r.hi.z; ++z)
        for (int y = r.lo.y; y <= r.hi.y; ++y)
            for (int x = r.lo.x; x <= r.hi.x; ++x)
                put_entry(a, e, l4, h4, x, y, z, (x > r.lo.x ? 1 : 0) | (y > r.lo.y ? 2 : 0) | (z > r.lo.z ? 4 : 0));
}

__device__ __forceinline__ bool boxes_overlap(float3 lo, float3 hi, float4 blo, float4 bhi) {
    return !(blo.x > hi.x || bhi.x < lo.x || blo.y > hi.y || bhi.y < lo.y || blo.z > hi.z || bhi.z < lo.z);
}

__device__ __forceinline__ bool filtered(const int* off, const int* list, int row, int x) {
    if (!off) return false;
    const int* b = list + off[row];
    const int* e = list + off[row + 1];
    while (b < e) {
        const int* mid = b + (e - b) / 2;
        if (*mid < x) b = mid + 1;
        else e = mid;
    }
    return b < list + off[row + 1] && *b == x;
}

// whether the list holds u or v (or w): one pass over it
__device__ __forceinline__ bool list_has(const int* b, const int* e, int u, int v, int w) {
    for (const int* p = b; p < e; ++p) {
        const int x = *p;
        if (x == u || x == v || x == w) return true;
    }
    return false;
}

struct QueryArgs {
    const float4* x;
    const int* vworld;
    const int *vfilt_off, *vfilt, *efilt_off, *efilt;  // external filter lists (NULL: none)
    const float4* rest;
    const int4* tri;
    const int4* edge;
    const int* near_off;
    const int* near;
    const int* vt_order;  // query slot -> vertex
    int V, T, E;
    float margin, inv_cell, par_eps, rest_excl;
    unsigned tri_mask, edge_mask;
    const int *tri_cnt, *tri_off, *tri_items;
    const int *edge_cnt, *edge_off, *edge_items;
    const float4 *tri_item_box, *edge_item_box;
    int tri_cap, edge_cap;
    int vbuf, ebuf;
    int* vt_count;
    int* vt_list;
    int* ee_count;
    int* ee_list;
    unsigned* counters;
};

constexpr int kMaxQueryCells = 512;
constexpr int kWarpUnionCells = 128;  // larger warp unions fall back to one walk per lane
constexpr int kQueryBlock = 128;
constexpr int kQueryWarps = kQueryBlock / 32;
constexpr int kEeLanes = 4;  // lanes per edge-edge query (4 measured best of 2, 4, 8)
constexpr int kVtLanes = 4;  // lanes per vertex-triangle query (one lane: 1.49 against 1.25 ms at 1.05 M
                             // vertices, 135 against 37 us at 4,096, where one lane leaves SMs idle)

// ---- candidates -------------------------------------------------------------------------------
// Both queries run in two halves.  The cheap half -- a staged bucket entry against a lane's query:
// cell ownership, box overlap -- runs with every lane on its own query and passes a few entries in a
// hundred; each passed (query, element) pair goes into a small queue of the warp.  The expensive
// half -- the exact distance, the ring and external filters -- takes 32 queued pairs at a time, one
// per lane (a lane that evaluated its own pairs as it met them left most of the warp idle).  The
// distance comes before the filters: most queued pairs are neighbours in the same layer, farther
// apart than the margin, and the ring filter walks a list.  Accepted partners are appended to their
// rows through atomic slots; sort_rows_kernel then orders every row, so the lists do not depend on
// scheduling, but for a row that met more partners than it holds (counted).  On the folded 1.05 M vertex cloth: edge query 4.59 -> 2.59 ms, vertex query 2.31 -> 1.21 ms.
struct PairQueue {
    int2* slots;  // this warp's 64 entries in shared memory
    int n;        // (warp-uniform)
};

// queue (q, t) of the lanes with `cand`; 32 queued pairs are handed to `accept`, one per lane
template <typename Accept>
__device__ __forceinline__ void queue_push(PairQueue& pq, bool cand, int q, int t, Accept accept) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, cand);
    if (m == 0u) return;
    if (cand) pq.slots[pq.n + __popc(m & ((1u << lane) - 1u))] = make_int2(q, t);
    pq.n += __popc(m);
    if (pq.n >= 32) {
        __syncwarp();
        pq.n -= 32;
        const int2 e = pq.slots[pq.n + lane];
        __syncwarp();
        accept(e.x, e.y);
    }
}

template <typename Accept>
__device__ __forceinline__ void queue_flush(PairQueue& pq, Accept accept) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    if (lane < pq.n) {
        const int2 e = pq.slots[lane];
        accept(e.x, e.y);
    }
    pq.n = 0;
}

// ---- vertex-triangle candidates ------------------------------------------------------------
struct VtQuery {
    int i;
    float3 plo, phi;
    CellRange q;
};

// the exact tests of a queued pair; appends t to vertex i's row
__device__ __forceinline__ void vt_accept(const QueryArgs& a, int i, int t) {
    const int4 tr = a.tri[t];
    if (tr.x == i || tr.y == i || tr.z == i) return;
    const int wv = a.vworld[i];
    if (wv >= 0 && tr.w >= 0 && wv != tr.w) return;
    const float3 p = xyz(a.x[i]);
    float3 bary;
    const float dist = length(triangle_closest_point(xyz(a.x[tr.x]), xyz(a.x[tr.y]), xyz(a.x[tr.z]), p, bary) - p);
    if (!(dist < a.margin)) return;
    if (list_has(a.near + a.near_off[i], a.near + a.near_off[i + 1], tr.x, tr.y, tr.z)) return;
    if (filtered(a.vfilt_off, a.vfilt, i, t)) return;
    if (a.rest_excl > 0.f) {
        const float3 rp = xyz(a.rest[i]);
        const float dr = length(
            triangle_closest_point(xyz(a.rest[tr.x]), xyz(a.rest[tr.y]), xyz(a.rest[tr.z]), rp, bary) - rp);
        if (dr < a.rest_excl) return;
    }
    const int k = atomicAdd(&a.vt_count[i], 1);
    if (k < a.vbuf) a.vt_list[static_cast<size_t>(i) * a.vbuf + k] = t;
}

__device__ __forceinline__ void vt_scan_lane(const QueryArgs& a, const VtQuery& v) {
    for (int z = v.q.lo.z; z <= v.q.hi.z; ++z)
        for (int y = v.q.lo.y; y <= v.q.hi.y; ++y)
            for (int x = v.q.lo.x; x <= v.q.hi.x; ++x) {
                const unsigned h = cell_hash(x, y, z, a.tri_mask);
                const int key = cell_key(x, y, z), mask = query_mask(v.q, x, y, z);
                const int b = a.tri_off[h];
                const int e = min(b + a.tri_cnt[h], a.tri_cap);
                for (int k = b; k < e; ++k) {
                    const float4 blo = a.tri_item_box[2 * k], bhi = a.tri_item_box[2 * k + 1];
                    if (!boxes_overlap(v.plo, v.phi, blo, bhi)) continue;
                    if (!takes(blo, bhi, key, mask)) continue;
                    vt_accept(a, v.i, a.tri_items[k]);
                }
            }
}

__device__ __forceinline__ bool warp_union(bool ok, const CellRange& q, CellRange& u) {
    const unsigned all = 0xffffffffu;
    if (__ballot_sync(all, ok) == 0u) return false;
    u.lo = make_int3(__reduce_min_sync(all, ok ? q.lo.x : INT_MAX), __reduce_min_sync(all, ok ? q.lo.y : INT_MAX),
                     __reduce_min_sync(all, ok ? q.lo.z : INT_MAX));
    u.hi = make_int3(__reduce_max_sync(all, ok ? q.hi.x : INT_MIN), __reduce_max_sync(all, ok ? q.hi.y : INT_MIN),
                     __reduce_max_sync(all, ok ? q.hi.z : INT_MIN));
    return true;
}

__device__ __forceinline__ bool in_range(const CellRange& q, int x, int y, int z) {
    return x >= q.lo.x && x <= q.hi.x && y >= q.lo.y && y <= q.hi.y && z >= q.lo.z && z <= q.hi.z;
}

// kVtLanes lanes serve one vertex, so a warp holds 32 / kVtLanes consecutive (spatially close) ones and
// walks the union of their query ranges once: every bucket entry is staged in shared memory by one
// lane, and each lane tests every kVtLanes-th entry against its own query (a walk per lane diverges:
// its buckets differ in length from its neighbours').
__global__ void __launch_bounds__(kQueryBlock) vt_query_kernel(const __grid_constant__ QueryArgs a) {
    __shared__ int s_id[kQueryWarps][32];
    __shared__ float4 s_box[kQueryWarps][64];
    __shared__ int2 s_queue[kQueryWarps][64];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // consecutive query slots are spatially close vertices (Morton order of the rest shape; the
    // internal vertex order is color-major, so neighbours in it are far apart), which keeps the
    // warp's union of cell ranges small
    const int slot = (blockIdx.x * blockDim.x + threadIdx.x) / kVtLanes;
    const int sub = lane % kVtLanes;
    const int i = slot < a.V ? a.vt_order[slot] : a.V;
    VtQuery v;
    v.i = i;
    bool ok = false;
    if (i < a.V) {
        const float3 p = xyz(a.x[i]);
        const float m = a.margin;
        v.plo = p - f3(m, m, m);
        v.phi = p + f3(m, m, m);
        // a small triangle within the margin has its box centre within margin + half a cell of p;
        // a large one is in every cell its box overlaps
        const float r = m + 0.5f / a.inv_cell;
        v.q = cell_range(p - f3(r, r, r), p + f3(r, r, r), a.inv_cell);
        ok = cell_count(v.q) <= kMaxQueryCells;
        if (!ok && sub == 0) atomicAdd(&a.counters[kScGridOverflow], 1u);
    }
    CellRange u;
    if (!warp_union(ok, v.q, u)) return;
    if (cell_count(u) > kWarpUnionCells) {
        if (ok && sub == 0) vt_scan_lane(a, v);
        return;
    }
    PairQueue pq = {s_queue[w], 0};
    auto accept = [&](int q, int t) { vt_accept(a, q, t); };
    for (int z = u.lo.z; z <= u.hi.z; ++z)
        for (int y = u.lo.y; y <= u.hi.y; ++y)
            for (int x = u.lo.x; x <= u.hi.x; ++x) {
                const bool mine = ok && in_range(v.q, x, y, z);
                if (!__any_sync(0xffffffffu, mine)) continue;
                const unsigned h = cell_hash(x, y, z, a.tri_mask);
                const int key = cell_key(x, y, z), mask = query_mask(v.q, x, y, z);
                const int b = a.tri_off[h];
                const int cnt = min(b + a.tri_cnt[h], a.tri_cap) - b;
                for (int c = 0; c < cnt; c += 32) {
                    if (c + lane < cnt) {
                        const int k = b + c + lane;
                        s_id[w][lane] = a.tri_items[k];
                        s_box[w][2 * lane] = a.tri_item_box[2 * k];
                        s_box[w][2 * lane + 1] = a.tri_item_box[2 * k + 1];
                    }
                    __syncwarp();
                    const int mc = min(32, cnt - c);
                    for (int t0 = 0; t0 < mc; t0 += kVtLanes) {
                        const int t = t0 + sub;
                        bool cand = false;
                        if (mine && t < mc) {
                            const float4 blo = s_box[w][2 * t], bhi = s_box[w][2 * t + 1];
                            cand = takes(blo, bhi, key, mask) && boxes_overlap(v.plo, v.phi, blo, bhi);
                        }
                        queue_push(pq, cand, i, t < mc ? s_id[w][t] : -1, accept);
                    }
                    __syncwarp();
                }
            }
    queue_flush(pq, accept);
}

// ---- edge-edge candidates ------------------------------------------------------------------
// Edge-edge pairs are symmetric: edge e only searches partners g > e and records the pair in both
// lists.  A partner sits in every cell its box overlaps and is taken only in the first cell of the
// query range it occupies (takes).
struct EeQuery {
    int e;
    float3 qlo, qhi;
    CellRange q;
};

__device__ __forceinline__ void ee_accept(const QueryArgs& a, int e, int g) {
    const int4 gd = a.edge[g];
    const int4 ed = a.edge[e];
    if (gd.x == ed.x || gd.x == ed.y || gd.y == ed.x || gd.y == ed.y) return;
    if (ed.z >= 0 && gd.z >= 0 && ed.z != gd.z) return;
    float s, t, dist;
    closest_edge_edge(xyz(a.x[ed.x]), xyz(a.x[ed.y]), xyz(a.x[gd.x]), xyz(a.x[gd.y]), a.par_eps, s, t, dist);
    if (!(dist < a.margin)) return;
    if (list_has(a.near + a.near_off[ed.x], a.near + a.near_off[ed.x + 1], gd.x, gd.y, gd.y) ||
        list_has(a.near + a.near_off[ed.y], a.near + a.near_off[ed.y + 1], gd.x, gd.y, gd.y))
        return;
    if (a.rest_excl > 0.f) {
        float sr, tr, dr;
        closest_edge_edge(xyz(a.rest[ed.x]), xyz(a.rest[ed.y]), xyz(a.rest[gd.x]), xyz(a.rest[gd.y]), a.par_eps, sr,
                          tr, dr);
        if (dr < a.rest_excl) return;
    }
    // the distance of (e, g) and of (g, e) is the same test; record both sides (each side's
    // external filter applies to its own list)
    if (!filtered(a.efilt_off, a.efilt, e, g)) {
        const int ke = atomicAdd(&a.ee_count[e], 1);
        if (ke < a.ebuf) a.ee_list[static_cast<size_t>(e) * a.ebuf + ke] = g;
        else atomicAdd(&a.counters[kScEeOverflow], 1u);
    }
    if (!filtered(a.efilt_off, a.efilt, g, e)) {
        const int kg = atomicAdd(&a.ee_count[g], 1);
        if (kg < a.ebuf) a.ee_list[static_cast<size_t>(g) * a.ebuf + kg] = e;
        else atomicAdd(&a.counters[kScEeOverflow], 1u);
    }
}

__device__ __forceinline__ void ee_scan_lane(const QueryArgs& a, const EeQuery& v) {
    for (int z = v.q.lo.z; z <= v.q.hi.z; ++z)
        for (int y = v.q.lo.y; y <= v.q.hi.y; ++y)
            for (int x = v.q.lo.x; x <= v.q.hi.x; ++x) {
                const unsigned h = cell_hash(x, y, z, a.edge_mask);
                const int key = cell_key(x, y, z), mask = query_mask(v.q, x, y, z);
                const int b = a.edge_off[h];
                const int en = min(b + a.edge_cnt[h], a.edge_cap);
                for (int k = b; k < en; ++k) {
                    const int g = a.edge_items[k];
                    if (g <= v.e) continue;
                    const float4 blo = a.edge_item_box[2 * k], bhi = a.edge_item_box[2 * k + 1];
                    if (!boxes_overlap(v.qlo, v.qhi, blo, bhi)) continue;
                    if (!takes(blo, bhi, key, mask)) continue;
                    ee_accept(a, v.e, g);
                }
            }
}

// kEeLanes lanes serve one edge query, so a warp holds 32 / kEeLanes consecutive (spatially
// adjacent) edges: their union of cell ranges stays close to one query's range, and each lane
// tests every kEeLanes-th staged entry.  Each (edge, partner) test runs on exactly one lane.
__global__ void __launch_bounds__(kQueryBlock) ee_query_kernel(const __grid_constant__ QueryArgs a) {
    __shared__ int s_id[kQueryWarps][32];
    __shared__ float4 s_box[kQueryWarps][64];
    __shared__ int2 s_queue[kQueryWarps][64];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) / kEeLanes;
    const int sub = lane % kEeLanes;
    EeQuery v;
    v.e = e;
    bool ok = false;
    if (e < a.E) {
        const int4 ed = a.edge[e];
        const float3 a0 = xyz(a.x[ed.x]), a1 = xyz(a.x[ed.y]);
        const float m = a.margin;
        v.qlo = fmin3(a0, a1) - f3(m, m, m);
        v.qhi = fmax3(a0, a1) + f3(m, m, m);
        // every partner sits in all the cells its box overlaps: the query's own cells suffice
        v.q = cell_range(v.qlo, v.qhi, a.inv_cell);
        ok = cell_count(v.q) <= kMaxQueryCells;
        if (!ok && sub == 0) atomicAdd(&a.counters[kScGridOverflow], 1u);
    }
    CellRange u;
    if (!warp_union(ok, v.q, u)) return;
    if (cell_count(u) > kWarpUnionCells) {
        if (ok && sub == 0) ee_scan_lane(a, v);
        return;
    }
    // partners with id <= the warp's smallest query id are rejected by every lane (g > e): they
    // are dropped while staging, so the lanes only walk the entries that can pass
    const int e_min = __reduce_min_sync(0xffffffffu, ok ? e : INT_MAX);
    PairQueue pq = {s_queue[w], 0};
    auto accept = [&](int q, int g) { ee_accept(a, q, g); };
    for (int z = u.lo.z; z <= u.hi.z; ++z)
        for (int y = u.lo.y; y <= u.hi.y; ++y)
            for (int x = u.lo.x; x <= u.hi.x; ++x) {
                const bool mine = ok && in_range(v.q, x, y, z);
                if (!__any_sync(0xffffffffu, mine)) continue;
                const unsigned h = cell_hash(x, y, z, a.edge_mask);
                const int key = cell_key(x, y, z), mask = query_mask(v.q, x, y, z);
                const int b = a.edge_off[h];
                const int cnt = min(b + a.edge_cnt[h], a.edge_cap) - b;
                for (int c = 0; c < cnt; c += 32) {
                    int gid = -1;
                    if (c + lane < cnt) gid = a.edge_items[b + c + lane];
                    const bool keep = gid > e_min;
                    const unsigned kept = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const int k = b + c + lane;
                        const int slot = __popc(kept & ((1u << lane) - 1u));
                        s_id[w][slot] = gid;
                        s_box[w][2 * slot] = a.edge_item_box[2 * k];
                        s_box[w][2 * slot + 1] = a.edge_item_box[2 * k + 1];
                    }
                    __syncwarp();
                    const int mc = __popc(kept);
                    for (int t0 = 0; t0 < mc; t0 += kEeLanes) {
                        const int t = t0 + sub;
                        bool cand = false;
                        int g = -1;
                        if (mine && t < mc) {
                            g = s_id[w][t];
                            const float4 blo = s_box[w][2 * t], bhi = s_box[w][2 * t + 1];
                            cand = g > e && takes(blo, bhi, key, mask) && boxes_overlap(v.qlo, v.qhi, blo, bhi);
                        }
                        queue_push(pq, cand, e, g, accept);
                    }
                    __syncwarp();
                }
            }
    queue_flush(pq, accept);
}

// Rows in ascending order without duplicates (an element that two colliding cells put into one
// bucket twice is met twice), kSortLanes lanes per row: every entry's rank is the number of smaller
// ones.  Rows with a duplicate or more than kSortMax entries (larger buffers) are sorted by one lane.
// overflow: counts the rows that met more entries than their buffer holds (NULL: already counted).
// (3.1 M edge rows: 0.67 -> 0.51 ms against an insertion sort by one thread per row.)
constexpr int kSortLanes = 16;
constexpr int kSortMax = 4 * kSortLanes;

__global__ void sort_rows_kernel(int rows, int* count, int* list, int buf, unsigned* overflow) {
    const int r = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / kSortLanes);
    const int sub = threadIdx.x % kSortLanes;
    const unsigned group = ((1u << kSortLanes) - 1u) << ((threadIdx.x & 31) & ~(kSortLanes - 1));
    const int met = r < rows ? count[r] : 0;
    const int n = min(met, buf);
    __syncwarp();  // every lane of the row has read the count
    if (met > buf && sub == 0) {
        count[r] = buf;
        if (overflow) atomicAdd(overflow, 1u);
    }
    if (n < 2) return;  // (uniform over the row's lanes)
    int* row = list + static_cast<size_t>(r) * buf;
    bool serial = n > kSortMax;
    int x[kSortMax / kSortLanes], rank[kSortMax / kSortLanes];
    if (!serial) {
        bool dup = false;
#pragma unroll
        for (int q = 0; q < kSortMax / kSortLanes; ++q) {
            const int k = sub + q * kSortLanes;
            x[q] = k < n ? row[k] : INT_MAX;
            rank[q] = 0;
        }
#pragma unroll
        for (int p = 0; p < kSortMax / kSortLanes; ++p) {
            if (p * kSortLanes >= n) break;
            for (int j = 0; j < kSortLanes; ++j) {
                if (p * kSortLanes + j >= n) break;
                const int y = __shfl_sync(group, x[p], j, kSortLanes);
#pragma unroll
                for (int q = 0; q < kSortMax / kSortLanes; ++q) {
                    rank[q] += y < x[q] ? 1 : 0;
                    dup |= y == x[q] && p * kSortLanes + j < sub + q * kSortLanes && sub + q * kSortLanes < n;
                }
            }
        }
        serial = __any_sync(group, dup);
    }
    if (!serial) {
#pragma unroll
        for (int q = 0; q < kSortMax / kSortLanes; ++q)
            if (sub + q * kSortLanes < n) row[rank[q]] = x[q];
        return;
    }
    if (sub != 0) return;
    int m = 0;
    for (int k = 0; k < n; ++k) {
        const int v = row[k];
        int b = m - 1;
        while (b >= 0 && row[b] > v) --b;
        if (b >= 0 && row[b] == v) continue;
        for (int j = m; j > b + 1; --j) row[j] = row[j - 1];
        row[b + 1] = v;
        ++m;
    }
    count[r] = m;
}

__global__ void tri_reverse_kernel(int V, const int* vt_count, const int* vt_list, int vbuf, int* tv_count,
                                   int* tv_list, int tcap, unsigned* counters) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const int* row = vt_list + static_cast<size_t>(i) * vbuf;
    for (int k = 0; k < vt_count[i]; ++k) {
        const int t = row[k];
        const int j = atomicAdd(&tv_count[t], 1);
        if (j < tcap) tv_list[static_cast<size_t>(t) * tcap + j] = i;
        else atomicAdd(&counters[kScTvOverflow], 1u);
    }
}

__global__ void tri_sort_kernel(int T, int* tv_count, int* tv_list, int tcap) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int n = min(tv_count[t], tcap);
    tv_count[t] = n;
    int* row = tv_list + static_cast<size_t>(t) * tcap;
    for (int a = 1; a < n; ++a) {
        const int x = row[a];
        int b = a - 1;
        while (b >= 0 && row[b] > x) {
            row[b + 1] = row[b];
            --b;
        }
        row[b + 1] = x;
    }
}

// ---- pair tables -----------------------------------------------------------------------------
// Built once per detection, read by every color of the iterations until the next one:
//   * entries: per vertex, the pairs it takes part in (its own vertex-triangle row, then those of its
//     incident triangles, then of its incident edges), 16 bytes each and contiguous, so that the
//     force pass streams them with a full warp instead of walking list -> element -> vertex chains
//     with the few lanes that one short list fills;
//   * pairs: every pair once, with the part of its division plane that depends on the base positions
//     only (they stay put between detections).
// Measured on a 1.05 M vertex cloth with a third of it folded over itself (3.5 M vertex-triangle and
// 9.8 M edge-edge pairs near the margin), per color: forces 1,696 -> 183 us, planes 1,519 -> 123 us,
// for 2 ms of table building per detection.
// Offsets come from scans and every slot from a rank inside a sorted row, so the tables do not
// depend on thread scheduling.  Rows that would end beyond a table's capacity are left out of it
// and evaluated from the detection lists.
// Capacities, per vertex on average (51 and 13 in the case above), where the GPU has the memory: 2,688 bytes.
constexpr long long kEntriesPerVertex = 96;
constexpr long long kPairsPerVertex = 24;
constexpr int kIdMask = 0x3fffffff;           // vertex ids are below 2^30

__device__ __forceinline__ int tag(int id, int bits) {
    return static_cast<int>(static_cast<unsigned>(id) | (static_cast<unsigned>(bits) << 30));
}

// An entry also carries a lower bound of its pair's distance at the base positions, in 1/32 of the
// margin: bits 30 of .y and 30-31 of .z and .w.  With the byte bounds of the displacements
// (SelfContact::reach) the force pass rejects about half of the entries after four byte gathers --
// 32 vertices to a sector, instead of two with positions.
// The bound must hold wherever the vertices move from there, so it is of the true distance of the two
// elements, which changes by no more than they do.  The distance that detection and forces use does not:
// an edge shorter than sqrt(edge_parallel_epsilon) counts as its first endpoint, so that one stretched past
// that length jumps (from 2.4 to 1 mm for two 3.1 mm edges that cross at mid-span).  base_distance
// leaves that threshold out and takes off what FP32 can miss: the closest points of near-parallel edges,
// whose determinant is lost in rounding below an angle of about sqrt(16 eps) = 1e-3, which moves the
// distance by up to that angle times the length (4.5e-4 lengths at most in 12 million random pairs; 7e-5
// for triangles of aspect 1/100), and the positions' own rounding.  A thinner triangle has no bound.
// (On the folded 1.05 M vertex cloth a step takes 30.25 ms with it, 30.11 with the distance itself.)
constexpr int kDistanceSteps = 32;
constexpr float kMissedPerLength = 1e-3f, kMissedPerCoordinate = 1e-6f;
constexpr float kThinTriangle = 1e-4f;  // squared: |ab x ac|^2 over the longest side to the fourth
constexpr float kPointEdge = 1e-18f;    // squared length of an edge that is a point

struct TableArgs {
    int V, E;
    const float4* x;  // base positions
    const int4* tri;
    const int4* edge;
    const int *inc_t_off, *inc_e_off;
    const int2 *inc_t, *inc_e;
    const int *vt_count, *vt_list, *ee_count, *ee_list, *tv_count, *tv_list;
    int vbuf, ebuf, tcap;
    bool filtered;    // external edge filters: a pair may be in one of its two rows only
    long long *ent_cnt, *pair_cnt;
    const long long *ent_off, *pair_off;
    int4* ent;
    int4* pair_ids;
    float4 *pair_n, *pair_h;
    long long ent_cap, pair_cap;
    float inv_margin;
    const int *vcolor, *color_start;
    int *act_v, *act_vcnt;
};

// Whether row e of the edge lists reports the pair (e, g): the row of the smaller id does; the
// other one only when the pair is missing from that row (an external filter, or a full row).
__device__ __forceinline__ bool ee_reports(const TableArgs& a, int e, int g) {
    if (g > e) return true;
    const int n = a.ee_count[g];
    if (!a.filtered && n < a.ebuf) return false;
    const int* row = a.ee_list + static_cast<size_t>(g) * a.ebuf;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (row[mid] < e) lo = mid + 1;
        else hi = mid;
    }
    return !(lo < n && row[lo] == e);
}

__global__ void table_count_kernel(TableArgs a) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    long long n = 0;
    int color = -1;
    if (idx < a.V) {
        n = a.vt_count[idx];
        a.pair_cnt[idx] = n;
        for (int k = a.inc_t_off[idx]; k < a.inc_t_off[idx + 1]; ++k) n += a.tv_count[a.inc_t[k].x];
        for (int k = a.inc_e_off[idx]; k < a.inc_e_off[idx + 1]; ++k) n += a.ee_count[a.inc_e[k].x];
        a.ent_cnt[idx] = n;
        color = n > 0 ? a.vcolor[idx] : -1;
    }
    if (idx < a.E) {
        const int m = a.ee_count[idx];
        const int* row = a.ee_list + static_cast<size_t>(idx) * a.ebuf;
        int kept = 0;
        for (int k = 0; k < m; ++k) kept += ee_reports(a, idx, row[k]) ? 1 : 0;
        a.pair_cnt[a.V + idx] = kept;
    }
    if (idx == 0) {
        a.ent_cnt[a.V] = 0;
        a.pair_cnt[a.V + a.E] = 0;
    }
    // the color's list of contact-touching vertices: one atomic per warp and color (consecutive
    // vertices share a color but for the warps at a color's border)
    const unsigned lanes = __match_any_sync(0xffffffffu, color);
    if (color >= 0) {
        const int lane = threadIdx.x & 31, leader = __ffs(lanes) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(&a.act_vcnt[color], __popc(lanes));
        base = __shfl_sync(lanes, base, leader);
        a.act_v[a.color_start[color] + base + __popc(lanes & ((1u << lane) - 1u))] = idx;
    }
}

constexpr int kTableLanes = 8;  // lanes per row / vertex while the tables are filled

// What a division plane (vt_plane, ee_plane) takes from the base positions, in units of the pair's
// distance h: pair_n = (n / h, reach), pair_h = the four participants' heights over the foot of the
// second element along n, over h.  The plane will lie at a level l in [0.05, 0.95]; the first
// element's participants stand at heights of at least about 1, the second's at most about 0, so no
// displacement crosses it whose component along n / h stays below their distance from those levels
// (`reach`, less a tenth for rounding).
__device__ __forceinline__ void write_plane(const TableArgs& a, long long at, int4 ids, float3 n, float h,
                                            float4 height, int firsts) {
    const float inv = 1.0f / h;
    const float4 hh = make_float4(height.x * inv, height.y * inv, height.z * inv, height.w * inv);
    const float up = firsts == 2 ? fminf(hh.x, hh.y) : hh.x;
    const float low = firsts == 2 ? fmaxf(hh.z, hh.w) : fmaxf(fmaxf(hh.y, hh.z), hh.w);
    const float reach = 0.9f * fmaxf(fminf(up - 0.95f, 0.05f - low), 0.f);
    a.pair_ids[at] = ids;
    a.pair_n[at] = make_float4(n.x * inv, n.y * inv, n.z * inv, reach);
    a.pair_h[at] = hh;
}

__device__ __forceinline__ void vt_plane_base(const TableArgs& a, int i, int4 tr, long long at) {
    const float3 v = xyz(a.x[i]), t1 = xyz(a.x[tr.x]), t2 = xyz(a.x[tr.y]), t3 = xyz(a.x[tr.z]);
    float3 bary;
    const float3 cp = triangle_closest_point(t1, t2, t3, v, bary);
    const float3 nh = v - cp;
    const float h = length(nh);
    const int4 ids = make_int4(i, tr.x, tr.y, tr.z);
    if (h < 1e-12f) {
        // the reference's plane has a zero normal here, which shortens nothing
        a.pair_ids[at] = ids;
        a.pair_n[at] = make_float4(0.f, 0.f, 0.f, 1.f);
        a.pair_h[at] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const float3 n = normalized3(nh);
    write_plane(a, at, ids, n, h, make_float4(dot(n, nh), dot(n, t1 - cp), dot(n, t2 - cp), dot(n, t3 - cp)), 1);
}

__device__ __forceinline__ void ee_plane_base(const TableArgs& a, int4 ed, int4 gd, long long at) {
    const float3 a0 = xyz(a.x[ed.x]), a1 = xyz(a.x[ed.y]), b0 = xyz(a.x[gd.x]), b1 = xyz(a.x[gd.y]);
    float s, t, dist;
    closest_edge_edge(a0, a1, b0, b1, 1e-6f, s, t, dist);
    const float3 c1 = a0 + (a1 - a0) * s, c2 = b0 + (b1 - b0) * t;
    const float3 nh = c1 - c2;
    const float h = length(nh);
    const int4 ids = make_int4(tag(ed.x, 1), ed.y, gd.x, gd.y);
    if (h < 1e-12f) {
        // touching edges: the robust normal, heights over the midpoint, no crossing test (reach < 0)
        const float3 n = robust_edge_pair_normal(a0, a1, b0, b1);
        const float3 d = c1 * 0.5f + c2 * 0.5f;
        a.pair_ids[at] = ids;
        a.pair_n[at] = make_float4(n.x, n.y, n.z, -1.f);
        a.pair_h[at] = make_float4(dot(n, a0 - d), dot(n, a1 - d), dot(n, b0 - d), dot(n, b1 - d));
        return;
    }
    const float3 n = normalized3(nh);
    write_plane(a, at, ids, n, h, make_float4(dot(n, a0 - c2), dot(n, a1 - c2), dot(n, b0 - c2), dot(n, b1 - c2)), 2);
}

__global__ void table_pairs_kernel(TableArgs a) {
    const int row_id = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / kTableLanes);
    const int sub = threadIdx.x % kTableLanes, group = (threadIdx.x & 31) / kTableLanes;
    const bool vt = row_id < a.V, ee = !vt && row_id < a.V + a.E;
    int n = 0;
    long long off = 0;
    if (vt || ee) {
        off = a.pair_off[row_id];
        if (a.pair_off[row_id + 1] > off && a.pair_off[row_id + 1] <= a.pair_cap)
            n = vt ? a.vt_count[row_id] : a.ee_count[row_id - a.V];
    }
    if (vt) {
        const int* row = a.vt_list + static_cast<size_t>(row_id) * a.vbuf;
        for (int k = sub; k < n; k += kTableLanes) vt_plane_base(a, row_id, a.tri[row[k]], off + k);
    }
    // edge rows: ranks of the reported partners inside the row, kTableLanes at a time
    const int m = __reduce_max_sync(0xffffffffu, ee ? n : 0);
    const int e = row_id - a.V;
    int kept = 0;
    for (int base = 0; base < m; base += kTableLanes) {
        const int k = base + sub;
        int g = -1;
        if (ee && k < n) {
            g = a.ee_list[static_cast<size_t>(e) * a.ebuf + k];
            if (!ee_reports(a, e, g)) g = -1;
        }
        const unsigned bits = (__ballot_sync(0xffffffffu, g >= 0) >> (group * kTableLanes)) & ((1u << kTableLanes) - 1u);
        if (g >= 0) ee_plane_base(a, a.edge[e], a.edge[g], off + kept + __popc(bits & ((1u << sub) - 1u)));
        kept += __popc(bits);
    }
}

__device__ __forceinline__ float base_distance(const TableArgs& a, int i0, int i1, int i2, int i3, bool ee) {
    const float3 x0 = xyz(a.x[i0]), x1 = xyz(a.x[i1]), x2 = xyz(a.x[i2]), x3 = xyz(a.x[i3]);
    const float3 d01 = x1 - x0;
    float dist, len2;
    if (ee) {
        float s, t;
        closest_edge_edge(x0, x1, x2, x3, kPointEdge, s, t, dist);
        const float3 d23 = x3 - x2;
        len2 = fmaxf(dot(d01, d01), dot(d23, d23));
    } else {
        float3 bary;
        dist = length(triangle_closest_point(x0, x1, x2, x3, bary) - x3);
        const float3 d02 = x2 - x0, d12 = x2 - x1, n = cross(d01, d02);
        len2 = fmaxf(fmaxf(dot(d01, d01), dot(d02, d02)), dot(d12, d12));
        if (!(dot(n, n) >= kThinTriangle * (len2 * len2))) return 0.f;
    }
    const float3 far = fmax3(fmax3(fmax3(x0, x1), fmax3(x2, x3)), -fmin3(fmin3(x0, x1), fmin3(x2, x3)));
    return dist - kMissedPerLength * sqrtf(len2) - kMissedPerCoordinate * fmaxf(fmaxf(far.x, far.y), far.z);
}

// slot: the vertex's participant index; ee: an edge-edge pair (i0, i1; i2, i3), else the
// vertex-triangle pair (i0, i1, i2; i3)
__device__ __forceinline__ int4 make_entry(const TableArgs& a, int i0, int i1, int i2, int i3, int slot, bool ee) {
    const float steps = base_distance(a, i0, i1, i2, i3, ee) * a.inv_margin * (0.999f * kDistanceSteps);
    const int q = min(max(static_cast<int>(steps), 0), kDistanceSteps - 1);
    return make_int4(tag(i0, slot), tag(i1, (ee ? 2 : 0) | (q & 1)), tag(i2, (q >> 1) & 3), tag(i3, q >> 3));
}

__global__ void table_entries_kernel(const __grid_constant__ TableArgs a) {
    const int i = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / kTableLanes);
    const int sub = threadIdx.x % kTableLanes;
    if (i >= a.V) return;
    const long long off = a.ent_off[i], end = a.ent_off[i + 1];
    if (end == off || end > a.ent_cap) return;
    int4* out = a.ent + off;
    const int nv = a.vt_count[i];
    const int* row = a.vt_list + static_cast<size_t>(i) * a.vbuf;
    for (int k = sub; k < nv; k += kTableLanes) {
        const int4 tr = a.tri[row[k]];
        out[k] = make_entry(a, tr.x, tr.y, tr.z, i, 3, false);
    }
    out += nv;
    for (int k = a.inc_t_off[i]; k < a.inc_t_off[i + 1]; ++k) {
        const int2 ts = a.inc_t[k];
        const int n = a.tv_count[ts.x];
        if (n == 0) continue;
        const int4 tr = a.tri[ts.x];
        const int* vl = a.tv_list + static_cast<size_t>(ts.x) * a.tcap;
        for (int j = sub; j < n; j += kTableLanes) out[j] = make_entry(a, tr.x, tr.y, tr.z, vl[j], ts.y, false);
        out += n;
    }
    for (int k = a.inc_e_off[i]; k < a.inc_e_off[i + 1]; ++k) {
        const int2 es = a.inc_e[k];
        const int n = a.ee_count[es.x];
        if (n == 0) continue;
        const int4 ed = a.edge[es.x];
        const int* gl = a.ee_list + static_cast<size_t>(es.x) * a.ebuf;
        for (int j = sub; j < n; j += kTableLanes) {
            const int4 gd = a.edge[gl[j]];
            out[j] = make_entry(a, ed.x, ed.y, gd.x, gd.y, es.y, true);
        }
        out += n;
    }
}

// base positions of a detection; the displacements from them are reset, or (the step's start) given, or
// not known (disp NULL: the iterate has nothing to do with the detected positions, no bound holds)
__global__ void copy_positions_kernel(int V, const float4* src, float4* cd, float4* disp, bool reset,
                                      unsigned char* reach, float reach_inv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    if (src != cd) cd[i] = src[i];
    if (disp && reset) disp[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    reach[i] = static_cast<unsigned char>(!disp ? kReachUnbounded
                                                : (reset ? 0 : reach_of(length(xyz(disp[i])), reach_inv)));
}

// (a position that is not its base plus its displacement: no bound holds)
__global__ void refresh_reach_kernel(int V, const float4* cd, const float4* pos, const float4* disp,
                                     unsigned char* reach, float reach_inv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const float4 c = cd[i], x = pos[i], d = disp[i];
    const bool moved = x.x == __fadd_rn(c.x, d.x) && x.y == __fadd_rn(c.y, d.y) && x.z == __fadd_rn(c.z, d.z);
    reach[i] = static_cast<unsigned char>(moved ? reach_of(length(xyz(d)), reach_inv) : kReachUnbounded);
}

__global__ void load_positions_kernel(int V, const int* perm, const float* q, float4* cd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const int o = perm[i];
    cd[i] = make_float4(q[3 * o], q[3 * o + 1], q[3 * o + 2], 0.f);
}

struct AccumArgs {
    const float4* x;
    const float4* x0;   // anchor: the step's start positions
    const unsigned char* reach;
    float reach_unit, distance_step;
    const int4* tri;
    const int4* edge;
    const int *inc_t_off, *inc_e_off;
    const int2 *inc_t, *inc_e;
    const int *vt_count, *vt_list, *ee_count, *ee_list, *tv_count, *tv_list;
    int vbuf, ebuf, tcap;
    const long long* ent_off;
    const int4* ent;
    long long ent_cap;
    const int* list;    // the color's contact-touching vertices
    const int* count;   // how many (device)
    float r, ke, kd, mu, eps_u, dt, par_eps;
    float4 *f, *h0, *h1;
};

// L lanes per vertex: the vertex's pairs (own vertex-triangle list, then each incident triangle's
// colliding vertices, then each incident edge's colliding edges) are dealt round-robin to the
// lanes, and the partial sums are combined with xor shuffles -- a fixed order, so deterministic.
constexpr int kAccumLanes = 32;

__device__ __forceinline__ float lane_sum(float v) {
    for (int off = kAccumLanes >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// participant `slot`'s share of the vertex-triangle pair (a, b, c; p), or of the edge pair
__device__ __forceinline__ bool vt_share(const AccumArgs& a, int ia, int ib, int ic, int ip, int slot, float3& f,
                                         Sym3& H) {
    auto start = [&](int k) { return xyz(a.x0[k == 0 ? ia : (k == 1 ? ib : (k == 2 ? ic : ip))]); };
    return vt_contact_slot(xyz(a.x[ia]), xyz(a.x[ib]), xyz(a.x[ic]), xyz(a.x[ip]), start, slot, a.r, a.ke, a.kd, a.mu,
                           a.eps_u, a.dt, f, H);
}
__device__ __forceinline__ bool ee_share(const AccumArgs& a, int e0, int e1, int g0, int g1, int slot, float3& f,
                                         Sym3& H) {
    auto start = [&](int k) { return xyz(a.x0[k == 0 ? e0 : (k == 1 ? e1 : (k == 2 ? g0 : g1))]); };
    return ee_contact_slot(xyz(a.x[e0]), xyz(a.x[e1]), xyz(a.x[g0]), xyz(a.x[g1]), start, slot, a.r, a.ke, a.kd, a.mu,
                           a.eps_u, a.dt, a.par_eps, f, H);
}

// whether an entry's pair is within the radius: the same distance, without the forces
__device__ __forceinline__ bool in_radius(const AccumArgs& a, bool ee, int i0, int i1, int i2, int i3) {
    const float3 x0 = xyz(a.x[i0]), x1 = xyz(a.x[i1]), x2 = xyz(a.x[i2]), x3 = xyz(a.x[i3]);
    float dis;
    if (ee) {
        float s, t;
        closest_edge_edge(x0, x1, x2, x3, a.par_eps, s, t, dis);
    } else {
        float3 bary;
        dis = length(x3 - triangle_closest_point(x0, x1, x2, x3, bary));
    }
    return dis < a.r;
}

// this lane's share of the pairs of a vertex without entries (they did not fit the table), from the
// detection lists
__device__ __noinline__ bool accumulate_lists(const AccumArgs& a, int i, int lane, float3& f, Sym3& H) {
    bool hit = false;
    int idx = 0;  // running pair index of this vertex; the lane takes idx % L == lane
    const int* row = a.vt_list + static_cast<size_t>(i) * a.vbuf;
    const int nv = a.vt_count[i];
    for (int k = lane; k < nv; k += kAccumLanes) {
        const int4 tr = a.tri[row[k]];
        hit |= vt_share(a, tr.x, tr.y, tr.z, i, 3, f, H);
    }
    idx += nv;
    for (int k = a.inc_t_off[i]; k < a.inc_t_off[i + 1]; ++k) {
        const int2 ts = a.inc_t[k];
        const int n = a.tv_count[ts.x];
        const int4 tr = a.tri[ts.x];
        const int* vl = a.tv_list + static_cast<size_t>(ts.x) * a.tcap;
        for (int j = (lane - idx) & (kAccumLanes - 1); j < n; j += kAccumLanes)
            hit |= vt_share(a, tr.x, tr.y, tr.z, vl[j], ts.y, f, H);
        idx += n;
    }
    for (int k = a.inc_e_off[i]; k < a.inc_e_off[i + 1]; ++k) {
        const int2 es = a.inc_e[k];
        const int n = a.ee_count[es.x];
        const int4 ed = a.edge[es.x];
        const int* gl = a.ee_list + static_cast<size_t>(es.x) * a.ebuf;
        for (int j = (lane - idx) & (kAccumLanes - 1); j < n; j += kAccumLanes) {
            const int4 gd = a.edge[gl[j]];
            hit |= ee_share(a, ed.x, ed.y, gd.x, gd.y, es.y, f, H);
        }
        idx += n;
    }
    return hit;
}

// Grid-stride over the color's contact-touching vertices (the others hold zero since the last
// detection), a warp per vertex over its contiguous entries, in two halves: every entry's distance
// first, then the forces of those within the radius, 32 of them at a time from a queue of the warp (the
// forces are several times the work, and most entries near the margin have none).  Lane and order of
// every share follow from the entries' order alone, so the sums are deterministic.  (348 us with forces
// in line and no early rejection, 231 with the rejection, 183 with both.)
constexpr int kAccumBlock = 128, kAccumBlocks = 7;

__global__ void __launch_bounds__(kAccumBlock, kAccumBlocks) accumulate_kernel(const __grid_constant__ AccumArgs a) {
    __shared__ int4 s_hits[kAccumBlock / 32][64];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const int n = *a.count;
    const int lane = threadIdx.x & 31;
    int4* hits = s_hits[threadIdx.x >> 5];
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n; w += warps) {
        const int i = a.list[w];
        const long long off = a.ent_off[i], end = a.ent_off[i + 1];
        float3 f = f3(0.f, 0.f, 0.f);
        Sym3 H = zero_sym();
        bool any = false;
        if (end <= a.ent_cap) {
            int held = 0;
            // the forces of queued entry `at`
            auto share = [&](int at) {
                const int4 en = hits[at];
                const int slot = static_cast<int>(static_cast<unsigned>(en.x) >> 30);
                const int i0 = en.x & kIdMask, i1 = en.y & kIdMask, i2 = en.z & kIdMask, i3 = en.w & kIdMask;
                if (en.y >= 0) vt_share(a, i0, i1, i2, i3, slot, f, H);
                else ee_share(a, i0, i1, i2, i3, slot, f, H);
            };
            const int m = static_cast<int>(end - off);
            for (int base = 0; base < m; base += kAccumLanes) {
                bool hit = false;
                int4 en = make_int4(0, 0, 0, 0);
                if (base + lane < m) {
                    en = __ldg(&a.ent[off + base + lane]);
                    const int i0 = en.x & kIdMask, i1 = en.y & kIdMask, i2 = en.z & kIdMask, i3 = en.w & kIdMask;
                    const bool ee = en.y < 0;
                    // the distance cannot have fallen below the radius: base distance less both
                    // elements' largest displacements (kReachUnbounded: no bound)
                    const int m0 = a.reach[i0], m1 = a.reach[i1], m2 = a.reach[i2], m3 = a.reach[i3];
                    const int first = ee ? max(m0, m1) : m3;
                    const int second = ee ? max(m2, m3) : max(max(m0, m1), m2);
                    const int q = ((en.y >> 30) & 1) | (static_cast<int>(static_cast<unsigned>(en.z) >> 30) << 1) |
                                  (static_cast<int>(static_cast<unsigned>(en.w) >> 30) << 3);
                    if (!(max(first, second) < kReachUnbounded &&
                          q * a.distance_step - (first + second) * a.reach_unit > a.r))
                        hit = in_radius(a, ee, i0, i1, i2, i3);
                }
                const unsigned got = __ballot_sync(0xffffffffu, hit);
                if (got == 0u) continue;
                any = true;
                if (hit) hits[held + __popc(got & ((1u << lane) - 1u))] = en;
                held += __popc(got);
                __syncwarp();
                if (held >= 32) {
                    held -= 32;
                    share(held + lane);
                    __syncwarp();
                }
            }
            if (lane < held) share(lane);
            __syncwarp();
        } else {
            any = __any_sync(0xffffffffu, accumulate_lists(a, i, lane, f, H));
        }
        // most vertices near the margin hold no pair inside the radius: nothing to add up
        if (any) {
            f.x = lane_sum(f.x);
            f.y = lane_sum(f.y);
            f.z = lane_sum(f.z);
            H.xx = lane_sum(H.xx);
            H.xy = lane_sum(H.xy);
            H.xz = lane_sum(H.xz);
            H.yy = lane_sum(H.yy);
            H.yz = lane_sum(H.yz);
            H.zz = lane_sum(H.zz);
        }
        if (lane == 0) {
            a.f[i] = make_float4(f.x, f.y, f.z, 0.f);
            a.h0[i] = make_float4(H.xx, H.xy, H.xz, H.yy);
            a.h1[i] = make_float4(H.yz, H.zz, 0.f, 0.f);
        }
    }
}

struct TruncArgs {
    const float4* cd;
    const float4* disp;
    const int4* tri;
    const int4* edge;
    const int *vt_count, *vt_list, *ee_count, *ee_list;
    const long long* pair_off;  // [V + E + 1]
    const int4* pair_ids;
    const float4 *pair_n, *pair_h;
    long long pair_cap;
    int V, E, vbuf, ebuf;
    float eps, gamma;
    unsigned* ts;
};

__device__ __forceinline__ void ts_min(unsigned* ts, int i, float3 x, float3 dx, float3 n, float3 d, float eps,
                                       float gamma) {
    const float t = planar_truncation_t(x, dx, n, d, eps, gamma);
    atomicMin(&ts[i], __float_as_uint(t));
}

// one row of the detection lists (rows that did not fit the pair table)
__device__ __noinline__ void planar_row(const TruncArgs& a, int w) {
    if (w < a.V) {
        const int i = w;
        const float3 v = xyz(a.cd[i]), dv = xyz(a.disp[i]);
        const int* row = a.vt_list + static_cast<size_t>(i) * a.vbuf;
        for (int k = 0; k < a.vt_count[i]; ++k) {
            const int4 tr = a.tri[row[k]];
            const float3 t1 = xyz(a.cd[tr.x]), t2 = xyz(a.cd[tr.y]), t3 = xyz(a.cd[tr.z]);
            const float3 d1 = xyz(a.disp[tr.x]), d2 = xyz(a.disp[tr.y]), d3 = xyz(a.disp[tr.z]);
            float3 n, d;
            const int dummy = vt_plane(v, dv, t1, d1, t2, d2, t3, d3, n, d);
            if (!(dummy & 1)) ts_min(a.ts, i, v, dv, n, d, a.eps, a.gamma);
            if (!(dummy & 2)) ts_min(a.ts, tr.x, t1, d1, n, d, a.eps, a.gamma);
            if (!(dummy & 4)) ts_min(a.ts, tr.y, t2, d2, n, d, a.eps, a.gamma);
            if (!(dummy & 8)) ts_min(a.ts, tr.z, t3, d3, n, d, a.eps, a.gamma);
        }
        return;
    }
    const int e = w - a.V;
    const int4 ed = a.edge[e];
    const float3 a0 = xyz(a.cd[ed.x]), a1 = xyz(a.cd[ed.y]);
    const float3 da0 = xyz(a.disp[ed.x]), da1 = xyz(a.disp[ed.y]);
    const int* row = a.ee_list + static_cast<size_t>(e) * a.ebuf;
    for (int k = 0; k < a.ee_count[e]; ++k) {
        const int4 gd = a.edge[row[k]];
        const float3 b0 = xyz(a.cd[gd.x]), b1 = xyz(a.cd[gd.y]);
        const float3 db0 = xyz(a.disp[gd.x]), db1 = xyz(a.disp[gd.y]);
        float3 n, d;
        const int dummy = ee_plane(a0, da0, a1, da1, b0, db0, b1, db1, n, d);
        if (!(dummy & 1)) ts_min(a.ts, ed.x, a0, da0, n, d, a.eps, a.gamma);
        if (!(dummy & 2)) ts_min(a.ts, ed.y, a1, da1, n, d, a.eps, a.gamma);
        if (!(dummy & 4)) ts_min(a.ts, gd.x, b0, db0, n, d, a.eps, a.gamma);
        if (!(dummy & 8)) ts_min(a.ts, gd.y, b1, db1, n, d, a.eps, a.gamma);
    }
}

// The plane of pair k of the table against its participants' displacements, whose components along
// n / h are q: shortens those that cross it.  (Not inlined: few pairs get here, and the loop that
// finds them needs its registers for warps in flight.)
__device__ __noinline__ void planar_cut(const TruncArgs& a, long long k, int4 id, float4 nn, float4 qq) {
    const bool ee = (id.x >> 30) != 0, touching = nn.w < 0.f;
    const float q[4] = {qq.x, qq.y, qq.z, qq.w};
    const float first_side = fmaxf(ee ? fmaxf(-q[0], -q[1]) : -q[0], 0.f);
    const float second_side = fmaxf(ee ? fmaxf(q[2], q[3]) : fmaxf(fmaxf(q[1], q[2]), q[3]), 0.f);
    const float both = first_side + second_side;
    if (both == 0.f && !touching) return;
    const float4 hh = __ldg(&a.pair_h[k]);
    float l = second_side / both;
    l = l < 0.05f ? 0.05f : (l > 0.95f ? 0.95f : l);
    if (touching) l = 0.f;
    const float h = rsqrtf(dot(xyz(nn), xyz(nn)));  // back to lengths for the parallel tests
    const float far = ee ? 1e-6f : 1e-8f;
    const float height[4] = {hh.x, hh.y, hh.z, hh.w};
    const int who[4] = {id.x & kIdMask, id.y, id.z, id.w};
    const int firsts = ee ? 2 : 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float t = (l - height[j]) / q[j];
        if (!touching) {
            if ((j < firsts ? first_side : second_side) == 0.f || fabsf(q[j]) * h < 1e-6f) continue;
            if (!(t >= -1e-8f && t <= 1.f + far)) continue;
        }
        if (fabsf(q[j]) * h < a.eps || t < 0.f) continue;  // ratio 1
        atomicMin(&a.ts[who[j]], __float_as_uint(clamp01f(fminf(t * a.gamma, t - 1e-3f))));
    }
}

// One pair per thread, grid-stride: the division planes of vt_plane / ee_plane from the table's
// base-position part (write_plane) and the current displacements.  Most pairs end at the reach test,
// with 32 bytes of table and four displacements read: bound by the latency of those gathers, so the
// kernel is held to the registers at which six blocks fit an SM (two with the cut
// inlined: 215 -> 123 us for 13.3 M pairs).  The ratios are reduced with
// atomicMin, which does not depend on the order.
constexpr int kPlanarBlock = 256, kPlanarBlocks = 6;

__global__ void __launch_bounds__(kPlanarBlock, kPlanarBlocks) planar_kernel(const __grid_constant__ TruncArgs a) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const int rows = a.V + a.E;
    const long long total = a.pair_off[rows];
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    long long fit = total;
    int slow = rows;  // first row that is not in the table
    if (total > a.pair_cap) {
        int lo = 0, hi = rows;
        while (lo < hi) {
            const int mid = lo + ((hi - lo) >> 1);
            if (a.pair_off[mid + 1] <= a.pair_cap) lo = mid + 1;
            else hi = mid;
        }
        slow = lo;
        fit = a.pair_off[lo];
    }
    for (long long k = first; k < fit; k += stride) {
        const int4 id = __ldg(&a.pair_ids[k]);
        const float4 nn = __ldg(&a.pair_n[k]);
        const float3 n = xyz(nn);
        const float4 q = make_float4(dot(n, xyz(a.disp[id.x & kIdMask])), dot(n, xyz(a.disp[id.y])),
                                     dot(n, xyz(a.disp[id.z])), dot(n, xyz(a.disp[id.w])));
        if (fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))) < nn.w) continue;
        planar_cut(a, k, id, nn, q);
    }
    for (long long w = slow + first; w < rows; w += stride) planar_row(a, static_cast<int>(w));
}

// apply_truncation_ts: disp *= t, clamp |disp| to max_disp, pos = cd + disp; t is reset to 1.  Only
// where that changes something: the vertices [b, e) (the color just solved, or all), those with t < 1, and
// those without a bound -- displacements beyond max_disp (a warm start's, or one that its clamp left a last
// place too long; reach_of gives none to either) and positions that are not cd + disp.  The others'
// displacements and positions already are what the same arithmetic would write.
__global__ void apply_truncation_kernel(int V, const float4* cd, float4* disp, float4* pos, unsigned* ts,
                                        unsigned char* reach, float reach_inv, float max_disp, int b, int e) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const float t = __uint_as_float(ts[i]);
    const int bound = reach[i];
    const bool cut = t != 1.0f;
    if (!cut && (i < b || i >= e) && bound != kReachUnbounded) return;
    if (cut) ts[i] = __float_as_uint(1.0f);
    const float4 d4 = disp[i];
    float3 d = f3(d4.x * t, d4.y * t, d4.z * t);
    const float l = length(d);
    if (l > max_disp) d = f3(d.x * max_disp / l, d.y * max_disp / l, d.z * max_disp / l);
    disp[i] = make_float4(d.x, d.y, d.z, 0.f);
    reach[i] = reach_of(length(d), reach_inv);
    const float4 c = cd[i];
    pos[i] = make_float4(c.x + d.x, c.y + d.y, c.z + d.z, 0.f);
}

__global__ void fill_u32_kernel(unsigned* p, unsigned v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

unsigned next_pow2(long long x) {
    unsigned v = 1024;
    while (static_cast<long long>(v) < x && v < (1u << 30)) v <<= 1;
    return v;
}

template <typename T>
int upload_vec(T** dst, const std::vector<T>& src) {
    *dst = nullptr;
    const size_t n = std::max<size_t>(src.size(), 1);
    VBD_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(dst), n * sizeof(T)));
    if (!src.empty()) VBD_CUDA_TRY(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
    return VBD_OK;
}

// spreads the low 10 bits of x to every third bit (Morton interleaving)
uint32_t spread3(uint32_t x) {
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// indices of pts in Z-order of their position quantised to 1024 steps per axis of the bounding
// box (ties by index), so that consecutive indices are spatially close
std::vector<int> morton_order(const std::vector<float3>& pts) {
    const size_t n = pts.size();
    std::vector<int> order(n);
    for (size_t k = 0; k < n; ++k) order[k] = static_cast<int>(k);
    if (n == 0) return order;
    float3 lo = pts[0], hi = pts[0];
    for (const float3& p : pts) {
        lo = make_float3(std::min(lo.x, p.x), std::min(lo.y, p.y), std::min(lo.z, p.z));
        hi = make_float3(std::max(hi.x, p.x), std::max(hi.y, p.y), std::max(hi.z, p.z));
    }
    const float ext = std::max(std::max(hi.x - lo.x, hi.y - lo.y), std::max(hi.z - lo.z, 1e-12f));
    const float s = 1023.0f / ext;
    std::vector<uint32_t> code(n);
    for (size_t k = 0; k < n; ++k) {
        const float3 p = pts[k];
        auto q = [&](float v, float l) {
            const float t = (v - l) * s;
            return static_cast<uint32_t>(std::isfinite(t) ? std::min(std::max(t, 0.0f), 1023.0f) : 0.0f);
        };
        code[k] = (spread3(q(p.x, lo.x)) << 2) | (spread3(q(p.y, lo.y)) << 1) | spread3(q(p.z, lo.z));
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return code[a] < code[b]; });
    return order;
}

}  // namespace

bool self_contact_detect_now(const SelfContact& sc, int it) {
    if (!sc.on) return false;
    if (sc.p.interval == 0) return it == 0;
    if (sc.p.interval >= 1) return it % sc.p.interval == 0;
    return false;
}

void self_contact_free(SelfContact& sc) {
    // (the scratch arrays are parts of the arena)
    void* ptrs[] = {sc.arena, sc.tri,      sc.edge,   sc.inc_t_off, sc.inc_t,     sc.inc_e_off, sc.inc_e, sc.near_off,
                    sc.near,  sc.rest,     sc.vworld, sc.vt_order,  sc.vfilt_off, sc.vfilt,     sc.efilt_off,
                    sc.efilt, sc.color_start, sc.vcolor};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    SelfContact empty;
    sc = empty;
}

int self_contact_create(const VbdModelImpl& m, const SelfContactParams& p, SelfContact& sc) {
    self_contact_free(sc);
    if (!(p.margin >= p.radius))
        return fail(VBD_ERR_INVALID_ARGUMENT,
                    "particle_self_contact_margin is smaller than particle_self_contact_radius, this will result in "
                    "missing contacts and cause instability.\nIt is advisable to make particle_self_contact_margin "
                    "1.5-2 times larger than particle_self_contact_radius.");
    if (!(p.radius > 0.f)) return fail(VBD_ERR_INVALID_ARGUMENT, "self contact: radius must be > 0");
    if (p.vertex_buffer < 1 || p.vertex_buffer > 256 || p.edge_buffer < 1 || p.edge_buffer > 512)
        return fail(VBD_ERR_INVALID_ARGUMENT, "self contact: buffer sizes must be in [1, 256] / [1, 512]");
    if (p.filter_threshold > 4)
        return fail(VBD_ERR_UNSUPPORTED, "self contact: topological filter threshold above 4 is not supported");
    auto bad_csr = [](const std::vector<int>& off, const std::vector<int>& lst, int rows, int maxval) {
        if (off.empty()) return false;
        if (static_cast<int>(off.size()) != rows + 1 || off[0] != 0 || off[rows] != static_cast<int>(lst.size()))
            return true;
        for (int r = 0; r < rows; ++r) {
            if (off[r + 1] < off[r]) return true;
            for (int k = off[r]; k < off[r + 1]; ++k)
                if (lst[k] < 0 || lst[k] >= maxval || (k > off[r] && lst[k] <= lst[k - 1])) return true;
        }
        return false;
    };
    if (bad_csr(p.vertex_filter_off, p.vertex_filter, m.V, m.T) || bad_csr(p.edge_filter_off, p.edge_filter, m.E, m.E))
        return fail(VBD_ERR_INVALID_ARGUMENT,
                    "self contact: external filter lists must be CSR rows of ascending element ids in range");
    if (m.rest_q_h.size() != 3 * static_cast<size_t>(m.V))
        return fail(VBD_ERR_INVALID_ARGUMENT, "self contact needs the model's rest positions (VbdModelDesc.particle_q)");
    const int V = m.V, T = m.T, E = m.E;
    sc.p = p;
    sc.V = V;
    sc.T = T;
    sc.E = E;
    sc.max_disp = static_cast<float>(static_cast<double>(p.margin) * static_cast<double>(p.relaxation) * 0.5);
    sc.reach_unit = std::max(sc.max_disp, 1e-30f) / 254.0f;  // (a displacement beyond max_disp has no bound)
    std::vector<int> inv(V);
    for (int i = 0; i < V; ++i) inv[m.perm_host[i]] = i;
    // topology
    std::vector<int4> tri(T), edge(E);
    for (int t = 0; t < T; ++t) {
        const int* ti = m.tri_raw_h.data() + 3 * t;
        tri[t] = make_int4(inv[ti[0]], inv[ti[1]], inv[ti[2]], m.pworld_h[ti[0]]);
    }
    double max_edge = 0.0;
    for (int e = 0; e < E; ++e) {
        const int* ei = m.edge_raw_h.data() + 4 * e;
        edge[e] = make_int4(inv[ei[2]], inv[ei[3]], m.pworld_h[ei[2]], 0);
        const float* ra = m.rest_q_h.data() + 3 * static_cast<size_t>(inv[ei[2]]);
        const float* rb = m.rest_q_h.data() + 3 * static_cast<size_t>(inv[ei[3]]);
        const double dx = ra[0] - rb[0], dy = ra[1] - rb[1], dz = ra[2] - rb[2];
        max_edge = std::max(max_edge, std::sqrt(dx * dx + dy * dy + dz * dz));
    }
    // cell edge: margin + the longest rest edge (twice the largest rest half-extent), so a query
    // spans about three cells per axis while elements keep their rest size
    sc.cell = static_cast<float>(std::max(static_cast<double>(p.margin) + max_edge, 1e-6));
    // incidence (internal vertex -> triangles with slot, endpoint edges with endpoint)
    std::vector<int> it_off(V + 1, 0), ie_off(V + 1, 0);
    std::vector<int2> it_list, ie_list;
    for (int i = 0; i < V; ++i) {
        const int o = m.perm_host[i];
        for (int k = m.adj_t_off_h[o]; k < m.adj_t_off_h[o + 1]; k += 2)
            it_list.push_back(make_int2(m.adj_t_h[k], m.adj_t_h[k + 1]));
        it_off[i + 1] = static_cast<int>(it_list.size());
        for (int k = m.adj_e_off_h[o]; k < m.adj_e_off_h[o + 1]; k += 2)
            if (m.adj_e_h[k + 1] >= 2) ie_list.push_back(make_int2(m.adj_e_h[k], m.adj_e_h[k + 1] - 2));
        ie_off[i + 1] = static_cast<int>(ie_list.size());
    }
    // n-ring filter sets (internal ids): vertices within threshold - 1 edge rings
    std::vector<int> near_off(V + 1, 0), near_list;
    if (p.filter_threshold >= 2) {
        std::vector<std::vector<int>> ring1(V);
        for (int e = 0; e < E; ++e) {
            ring1[edge[e].x].push_back(edge[e].y);
            ring1[edge[e].y].push_back(edge[e].x);
        }
        for (auto& r : ring1) {
            std::sort(r.begin(), r.end());
            r.erase(std::unique(r.begin(), r.end()), r.end());
        }
        const int depth = p.filter_threshold - 1;
        std::vector<int> seen, frontier, next;
        for (int i = 0; i < V; ++i) {
            seen.assign(1, i);
            frontier.assign(1, i);
            for (int k = 0; k < depth && !frontier.empty(); ++k) {
                next.clear();
                for (int u : frontier)
                    for (int w : ring1[u])
                        if (std::find(seen.begin(), seen.end(), w) == seen.end()) {
                            seen.push_back(w);
                            next.push_back(w);
                        }
                frontier.swap(next);
            }
            std::sort(seen.begin(), seen.end());
            for (int w : seen)
                if (w != i) near_list.push_back(w);
            near_off[i + 1] = static_cast<int>(near_list.size());
        }
    }
    std::vector<int> vworld(V);
    for (int i = 0; i < V; ++i) vworld[i] = m.pworld_h[m.perm_host[i]];
    std::vector<float4> rest(V);
    for (int i = 0; i < V; ++i)
        rest[i] = make_float4(m.rest_q_h[3 * i], m.rest_q_h[3 * i + 1], m.rest_q_h[3 * i + 2], 0.f);
    std::vector<float3> vp(V);
    for (int i = 0; i < V; ++i) vp[i] = make_float3(rest[i].x, rest[i].y, rest[i].z);
    const std::vector<int> vt_order = morton_order(vp);

    int rc = VBD_OK;
    if (!rc) rc = upload_vec(&sc.tri, tri);
    if (!rc) rc = upload_vec(&sc.edge, edge);
    if (!rc) rc = upload_vec(&sc.inc_t_off, it_off);
    if (!rc) rc = upload_vec(&sc.inc_t, it_list);
    if (!rc) rc = upload_vec(&sc.inc_e_off, ie_off);
    if (!rc) rc = upload_vec(&sc.inc_e, ie_list);
    if (!rc) rc = upload_vec(&sc.near_off, near_off);
    if (!rc) rc = upload_vec(&sc.near, near_list);
    if (!rc) rc = upload_vec(&sc.vt_order, vt_order);
    if (!rc) rc = upload_vec(&sc.rest, rest);
    if (!rc) rc = upload_vec(&sc.vworld, vworld);
    sc.C = m.C;
    std::vector<int> vcolor(V, -1);
    for (int c = 0; c < m.C; ++c)
        for (int i = m.color_start[c]; i < m.color_start[c + 1]; ++i) vcolor[i] = c;
    if (!rc) rc = upload_vec(&sc.vcolor, vcolor);
    if (!rc) rc = upload_vec(&sc.color_start, m.color_start);
    if (!rc && !p.vertex_filter_off.empty()) {
        std::vector<int> off(V + 1, 0), lst;
        for (int i = 0; i < V; ++i) {
            const int o = m.perm_host[i];
            lst.insert(lst.end(), p.vertex_filter.begin() + p.vertex_filter_off[o],
                       p.vertex_filter.begin() + p.vertex_filter_off[o + 1]);
            off[i + 1] = static_cast<int>(lst.size());
        }
        rc = upload_vec(&sc.vfilt_off, off);
        if (!rc) rc = upload_vec(&sc.vfilt, lst);
    }
    if (!rc && !p.edge_filter_off.empty()) {
        rc = upload_vec(&sc.efilt_off, p.edge_filter_off);
        if (!rc) rc = upload_vec(&sc.efilt, p.edge_filter);
    }
    const unsigned tn = next_pow2(2LL * std::max(T, 1)), en = next_pow2(2LL * std::max(E, 1));
    sc.tri_mask = tn - 1;
    sc.edge_mask = en - 1;
    sc.tri_items_cap = 2 * std::max(T, 1) + 65536;  // large (stretched) elements take several cells
    sc.edge_items_cap = 8 * std::max(E, 1) + 65536;  // an edge shorter than a cell overlaps at most 8 cells
    // one allocation for all of the scratch, every array 256-byte aligned
    std::vector<std::pair<void**, size_t>> placed;
    size_t total = 0;
    auto az = [&](void** ptr, size_t bytes) {
        placed.emplace_back(ptr, total);
        total += (std::max<size_t>(bytes, 16) + 255) & ~static_cast<size_t>(255);
    };
    // what a detection clears, in one span (cleared_bytes): counts, cursors, and the contact terms of
    // vertices that touch no pair, which stay zero until the next one
    az(reinterpret_cast<void**>(&sc.tri_cnt), tn * sizeof(int));
    az(reinterpret_cast<void**>(&sc.tri_cur), tn * sizeof(int));
    az(reinterpret_cast<void**>(&sc.edge_cnt), en * sizeof(int));
    az(reinterpret_cast<void**>(&sc.edge_cur), en * sizeof(int));
    az(reinterpret_cast<void**>(&sc.tv_count), static_cast<size_t>(T) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.vt_count), static_cast<size_t>(V) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.ee_count), static_cast<size_t>(E) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.act_vcnt), static_cast<size_t>(std::max(m.C, 1)) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.sc_f), static_cast<size_t>(V) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.sc_h0), static_cast<size_t>(V) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.sc_h1), static_cast<size_t>(V) * sizeof(float4));
    sc.cleared_bytes = total;
    az(reinterpret_cast<void**>(&sc.tri_off), tn * sizeof(int));
    az(reinterpret_cast<void**>(&sc.tri_items), static_cast<size_t>(sc.tri_items_cap) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.edge_off), en * sizeof(int));
    az(reinterpret_cast<void**>(&sc.edge_items), static_cast<size_t>(sc.edge_items_cap) * sizeof(int));
    az(reinterpret_cast<void**>(&sc.tri_box), 2 * static_cast<size_t>(std::max(T, 1)) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.edge_box), 2 * static_cast<size_t>(std::max(E, 1)) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.tri_item_box), 2 * static_cast<size_t>(sc.tri_items_cap) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.edge_item_box), 2 * static_cast<size_t>(sc.edge_items_cap) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.act_v), static_cast<size_t>(V) * sizeof(int));
    const size_t rows = static_cast<size_t>(V) + E + 1;
    az(reinterpret_cast<void**>(&sc.ent_cnt), (static_cast<size_t>(V) + 1) * sizeof(long long));
    az(reinterpret_cast<void**>(&sc.ent_off), (static_cast<size_t>(V) + 1) * sizeof(long long));
    az(reinterpret_cast<void**>(&sc.pair_cnt), rows * sizeof(long long));
    az(reinterpret_cast<void**>(&sc.pair_off), rows * sizeof(long long));
    az(reinterpret_cast<void**>(&sc.vt_list), static_cast<size_t>(V) * p.vertex_buffer * sizeof(int));
    az(reinterpret_cast<void**>(&sc.ee_list), static_cast<size_t>(E) * p.edge_buffer * sizeof(int));
    az(reinterpret_cast<void**>(&sc.tv_list), static_cast<size_t>(T) * sc.tcap * sizeof(int));
    az(reinterpret_cast<void**>(&sc.cd), static_cast<size_t>(V) * sizeof(float4));
    az(reinterpret_cast<void**>(&sc.reach), static_cast<size_t>(V));
    az(reinterpret_cast<void**>(&sc.ts), static_cast<size_t>(V) * sizeof(unsigned));
    az(reinterpret_cast<void**>(&sc.counters), kScCounters * sizeof(unsigned));
    if (!rc) {
        size_t b1 = 0, b2 = 0;
        cudaError_t e1 = cub::DeviceScan::ExclusiveSum(nullptr, b1, sc.tri_cnt, sc.tri_off, static_cast<int>(tn));
        cudaError_t e2 = cub::DeviceScan::ExclusiveSum(nullptr, b2, sc.edge_cnt, sc.edge_off, static_cast<int>(en));
        size_t b3 = 0;
        cudaError_t e3 = cub::DeviceScan::ExclusiveSum(nullptr, b3, sc.pair_cnt, sc.pair_off, static_cast<int>(rows));
        if (e1 != cudaSuccess) rc = cuda_fail(e1, "cub::DeviceScan::ExclusiveSum (size query)");
        if (!rc && e2 != cudaSuccess) rc = cuda_fail(e2, "cub::DeviceScan::ExclusiveSum (size query)");
        if (!rc && e3 != cudaSuccess) rc = cuda_fail(e3, "cub::DeviceScan::ExclusiveSum (size query)");
        sc.scan_bytes = std::max(std::max(b1, b2), b3);
        az(&sc.scan_tmp, sc.scan_bytes);
    }
    // the pair tables last: where the GPU has no room for them, a quarter, a sixteenth or none of their
    // capacity (the rows that do not fit are evaluated from the lists)
    const size_t others = placed.size(), others_bytes = total;
    for (long long share = 1; !rc && !sc.arena; share *= 4) {
        placed.resize(others);
        total = others_bytes;
        const bool last = share > 16;
        sc.ent_cap = last ? 0 : kEntriesPerVertex * V / share;
        sc.pair_cap = last ? 0 : kPairsPerVertex * V / share;
        az(reinterpret_cast<void**>(&sc.ent), static_cast<size_t>(sc.ent_cap) * sizeof(int4));
        az(reinterpret_cast<void**>(&sc.pair_ids), static_cast<size_t>(sc.pair_cap) * sizeof(int4));
        az(reinterpret_cast<void**>(&sc.pair_n), static_cast<size_t>(sc.pair_cap) * sizeof(float4));
        az(reinterpret_cast<void**>(&sc.pair_h), static_cast<size_t>(sc.pair_cap) * sizeof(float4));
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&sc.arena), total);
        if (e == cudaErrorMemoryAllocation && !last) {
            cudaGetLastError();  // (not an error of this call)
            sc.arena = nullptr;
            continue;
        }
        if (e == cudaSuccess) e = cudaMemset(sc.arena, 0, total);
        if (e != cudaSuccess) rc = cuda_fail(e, "vbd_solver_create: self-contact scratch");
    }
    if (!rc)
        for (const auto& p : placed) *p.first = sc.arena + p.second;
    if (!rc && V > 0) {
        fill_u32_kernel<<<(V + 255) / 256, 256>>>(sc.ts, 0x3f800000u /* 1.0f */, V);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = cuda_fail(e, "fill_u32_kernel");
        if (!rc) {
            const cudaError_t s = cudaDeviceSynchronize();
            if (s != cudaSuccess) rc = cuda_fail(s, "cudaDeviceSynchronize");
        }
    }
    if (rc) {
        self_contact_free(sc);
        return rc;
    }
    sc.on = true;
    return VBD_OK;
}

int self_contact_load_positions(const VbdModelImpl& m, SelfContact& sc, const float* q, cudaStream_t st) {
    if (m.V == 0) return VBD_OK;
    load_positions_kernel<<<(m.V + 255) / 256, 256, 0, st>>>(m.V, m.perm, q, sc.cd);
    VBD_CUDA_TRY(cudaGetLastError());
    return VBD_OK;
}

int self_contact_refresh_reach(const VbdModelImpl& m, SelfContact& sc, const float4* pos, const float4* disp,
                               cudaStream_t st) {
    if (m.V == 0) return VBD_OK;
    refresh_reach_kernel<<<(m.V + 255) / 256, 256, 0, st>>>(m.V, sc.cd, pos, disp, sc.reach, 1.0f / sc.reach_unit);
    VBD_CUDA_TRY(cudaGetLastError());
    return VBD_OK;
}

int self_contact_detect(const VbdModelImpl& m, SelfContact& sc, const float4* positions, float4* disp,
                        bool reset_disp, cudaStream_t st) {
    const int V = m.V, T = m.T, E = m.E;
    if (V == 0) return VBD_OK;
    copy_positions_kernel<<<(V + 255) / 256, 256, 0, st>>>(V, positions, sc.cd, disp, reset_disp, sc.reach,
                                                           1.0f / sc.reach_unit);
    VBD_CUDA_TRY(cudaGetLastError());
    const unsigned tn = sc.tri_mask + 1, en = sc.edge_mask + 1;
    VBD_CUDA_TRY(cudaMemsetAsync(sc.arena, 0, sc.cleared_bytes, st));
    const float inv_cell = 1.0f / sc.cell;
    GridArgs g;
    g.x = sc.cd;
    g.counters = sc.counters;
    g.inv_cell = inv_cell;
    // triangle grid
    g.elem = sc.tri;
    g.n = T;
    g.tri = true;
    g.all_cells = false;
    g.mask = sc.tri_mask;
    g.cnt = sc.tri_cnt;
    g.off = sc.tri_off;
    g.cur = sc.tri_cur;
    g.items = sc.tri_items;
    g.item_box = sc.tri_item_box;
    g.cap = sc.tri_items_cap;
    g.box = sc.tri_box;

    if (T > 0) {
        grid_count_kernel<<<(T + 255) / 256, 256, 0, st>>>(g);
        VBD_CUDA_TRY(cudaGetLastError());
        size_t bytes = sc.scan_bytes;
        VBD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sc.scan_tmp, bytes, sc.tri_cnt, sc.tri_off, static_cast<int>(tn), st));
        grid_fill_kernel<<<(T + 255) / 256, 256, 0, st>>>(g);
        VBD_CUDA_TRY(cudaGetLastError());
    }
    // edge grid
    g.elem = sc.edge;
    g.n = E;
    g.tri = false;
    g.all_cells = true;
    g.mask = sc.edge_mask;
    g.cnt = sc.edge_cnt;
    g.off = sc.edge_off;
    g.cur = sc.edge_cur;
    g.items = sc.edge_items;
    g.item_box = sc.edge_item_box;
    g.cap = sc.edge_items_cap;
    g.box = sc.edge_box;

    if (E > 0) {
        grid_count_kernel<<<(E + 255) / 256, 256, 0, st>>>(g);
        VBD_CUDA_TRY(cudaGetLastError());
        size_t bytes = sc.scan_bytes;
        VBD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sc.scan_tmp, bytes, sc.edge_cnt, sc.edge_off, static_cast<int>(en), st));
        grid_fill_kernel<<<(E + 255) / 256, 256, 0, st>>>(g);
        VBD_CUDA_TRY(cudaGetLastError());
    }
    QueryArgs q;
    q.x = sc.cd;
    q.vworld = sc.vworld;
    q.vfilt_off = sc.vfilt_off;
    q.vfilt = sc.vfilt;
    q.efilt_off = sc.efilt_off;
    q.efilt = sc.efilt;
    q.rest = sc.rest;
    q.tri = sc.tri;
    q.edge = sc.edge;
    q.near_off = sc.near_off;
    q.vt_order = sc.vt_order;
    q.near = sc.near;
    q.V = V;
    q.T = T;
    q.E = E;
    q.margin = sc.p.margin;
    q.inv_cell = inv_cell;
    q.par_eps = sc.p.edge_parallel_epsilon;
    q.rest_excl = sc.p.rest_exclusion_radius;
    q.tri_mask = sc.tri_mask;
    q.edge_mask = sc.edge_mask;
    q.tri_cnt = sc.tri_cnt;
    q.tri_off = sc.tri_off;
    q.tri_items = sc.tri_items;
    q.edge_cnt = sc.edge_cnt;
    q.edge_off = sc.edge_off;
    q.edge_items = sc.edge_items;
    q.tri_item_box = sc.tri_item_box;
    q.edge_item_box = sc.edge_item_box;
    q.tri_cap = sc.tri_items_cap;
    q.edge_cap = sc.edge_items_cap;
    q.vbuf = sc.p.vertex_buffer;
    q.ebuf = sc.p.edge_buffer;
    q.vt_count = sc.vt_count;
    q.vt_list = sc.vt_list;
    q.ee_count = sc.ee_count;
    q.ee_list = sc.ee_list;
    q.counters = sc.counters;
    auto sort_rows = [&](int rows, int* count, int* list, int buf, unsigned* overflow) {
        const long long threads = static_cast<long long>(rows) * kSortLanes;
        sort_rows_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(rows, count, list, buf, overflow);
    };
    if (T > 0) {
        const long long vt_threads = static_cast<long long>(V) * kVtLanes;
        vt_query_kernel<<<static_cast<unsigned>((vt_threads + kQueryBlock - 1) / kQueryBlock), kQueryBlock, 0, st>>>(q);
        VBD_CUDA_TRY(cudaGetLastError());
        sort_rows(V, sc.vt_count, sc.vt_list, sc.p.vertex_buffer, sc.counters + kScVtOverflow);
        VBD_CUDA_TRY(cudaGetLastError());
        tri_reverse_kernel<<<(V + 255) / 256, 256, 0, st>>>(V, sc.vt_count, sc.vt_list, sc.p.vertex_buffer,
                                                            sc.tv_count, sc.tv_list, sc.tcap, sc.counters);
        VBD_CUDA_TRY(cudaGetLastError());
        tri_sort_kernel<<<(T + 255) / 256, 256, 0, st>>>(T, sc.tv_count, sc.tv_list, sc.tcap);
        VBD_CUDA_TRY(cudaGetLastError());
    }
    if (E > 0) {
        const long long ee_threads = static_cast<long long>(E) * kEeLanes;
        ee_query_kernel<<<static_cast<unsigned>((ee_threads + kQueryBlock - 1) / kQueryBlock), kQueryBlock, 0, st>>>(q);
        VBD_CUDA_TRY(cudaGetLastError());
        sort_rows(E, sc.ee_count, sc.ee_list, sc.p.edge_buffer, nullptr);
        VBD_CUDA_TRY(cudaGetLastError());
    }
    TableArgs t;
    t.V = V;
    t.E = E;
    t.x = sc.cd;
    t.tri = sc.tri;
    t.edge = sc.edge;
    t.inc_t_off = sc.inc_t_off;
    t.inc_e_off = sc.inc_e_off;
    t.inc_t = sc.inc_t;
    t.inc_e = sc.inc_e;
    t.vt_count = sc.vt_count;
    t.vt_list = sc.vt_list;
    t.ee_count = sc.ee_count;
    t.ee_list = sc.ee_list;
    t.tv_count = sc.tv_count;
    t.tv_list = sc.tv_list;
    t.vbuf = sc.p.vertex_buffer;
    t.ebuf = sc.p.edge_buffer;
    t.tcap = sc.tcap;
    t.filtered = sc.efilt_off != nullptr;
    t.ent_cnt = sc.ent_cnt;
    t.pair_cnt = sc.pair_cnt;
    t.ent_off = sc.ent_off;
    t.pair_off = sc.pair_off;
    t.ent = sc.ent;
    t.pair_ids = sc.pair_ids;
    t.pair_n = sc.pair_n;
    t.pair_h = sc.pair_h;
    t.ent_cap = sc.ent_cap;
    t.pair_cap = sc.pair_cap;
    t.inv_margin = 1.0f / sc.p.margin;
    t.vcolor = sc.vcolor;
    t.color_start = sc.color_start;
    t.act_v = sc.act_v;
    t.act_vcnt = sc.act_vcnt;
    const int nm = std::max(V, E);
    table_count_kernel<<<(nm + 255) / 256, 256, 0, st>>>(t);
    VBD_CUDA_TRY(cudaGetLastError());
    size_t bytes = sc.scan_bytes;
    VBD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sc.scan_tmp, bytes, sc.ent_cnt, sc.ent_off, V + 1, st));
    bytes = sc.scan_bytes;
    VBD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sc.scan_tmp, bytes, sc.pair_cnt, sc.pair_off, V + E + 1, st));
    auto blocks = [](long long rows) { return static_cast<unsigned>((rows * kTableLanes + 127) / 128); };
    table_pairs_kernel<<<blocks(static_cast<long long>(V) + E), 128, 0, st>>>(t);
    VBD_CUDA_TRY(cudaGetLastError());
    table_entries_kernel<<<blocks(V), 128, 0, st>>>(t);
    VBD_CUDA_TRY(cudaGetLastError());
    return VBD_OK;
}

// the per-color passes are programmatic dependents of the kernel before them (each waits for it
// with griddepcontrol.wait before its first read), so their launches overlap its tail
template <typename... Args>
static int launch_pass(void (*kernel)(Args...), int grid, int block, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    VBD_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    return VBD_OK;
}

int self_contact_accumulate(const VbdModelImpl& m, SelfContact& sc, const float4* pos, const float4* prev,
                            int color, float dt, float friction_epsilon, cudaStream_t st) {
    if (color < 0) {
        for (int c = 0; c < m.C; ++c) {
            const int rc = self_contact_accumulate(m, sc, pos, prev, c, dt, friction_epsilon, st);
            if (rc) return rc;
        }
        return VBD_OK;
    }
    const int size = m.color_start[color + 1] - m.color_start[color];
    if (size <= 0) return VBD_OK;
    AccumArgs a;
    a.x = pos;
    a.x0 = prev;
    a.tri = sc.tri;
    a.edge = sc.edge;
    a.inc_t_off = sc.inc_t_off;
    a.inc_e_off = sc.inc_e_off;
    a.inc_t = sc.inc_t;
    a.inc_e = sc.inc_e;
    a.vt_count = sc.vt_count;
    a.vt_list = sc.vt_list;
    a.ee_count = sc.ee_count;
    a.ee_list = sc.ee_list;
    a.tv_count = sc.tv_count;
    a.tv_list = sc.tv_list;
    a.vbuf = sc.p.vertex_buffer;
    a.ebuf = sc.p.edge_buffer;
    a.tcap = sc.tcap;
    a.reach = sc.reach;
    a.reach_unit = sc.reach_unit;
    a.distance_step = sc.p.margin / kDistanceSteps;
    a.ent_off = sc.ent_off;
    a.ent = sc.ent;
    a.ent_cap = sc.ent_cap;
    a.list = sc.act_v + m.color_start[color];
    a.count = sc.act_vcnt + color;
    a.r = sc.p.radius;
    a.ke = m.soft_ke;
    a.kd = m.soft_kd;
    a.mu = m.soft_mu;
    a.eps_u = friction_epsilon * dt;
    a.dt = dt;
    a.par_eps = sc.p.edge_parallel_epsilon;
    a.f = sc.sc_f;
    a.h0 = sc.sc_h0;
    a.h1 = sc.sc_h1;
    // enough warps for every vertex of the color in one round, capped: the kernel strides
    const long long threads = static_cast<long long>(size) * kAccumLanes;
    const int grid = static_cast<int>(std::min<long long>((threads + kAccumBlock - 1) / kAccumBlock, 148 * 2 * kAccumBlocks));
    return launch_pass(accumulate_kernel, grid, kAccumBlock, st, a);
}

int self_contact_truncate(const VbdModelImpl& m, SelfContact& sc, float4* pos, float4* disp, int color,
                          cudaStream_t st) {
    const int V = m.V;
    if (V == 0) return VBD_OK;
    TruncArgs a;
    a.cd = sc.cd;
    a.disp = disp;
    a.tri = sc.tri;
    a.edge = sc.edge;
    a.vt_count = sc.vt_count;
    a.vt_list = sc.vt_list;
    a.ee_count = sc.ee_count;
    a.ee_list = sc.ee_list;
    a.pair_off = sc.pair_off;
    a.pair_ids = sc.pair_ids;
    a.pair_n = sc.pair_n;
    a.pair_h = sc.pair_h;
    a.pair_cap = sc.pair_cap;
    a.V = V;
    a.E = m.E;
    a.vbuf = sc.p.vertex_buffer;
    a.ebuf = sc.p.edge_buffer;
    a.eps = sc.p.edge_parallel_epsilon;
    a.gamma = sc.p.relaxation;
    a.ts = sc.ts;
    // the number of pairs is on the device: about 16 per vertex before the grid strides
    const long long n = 16LL * V;
    const int rc = launch_pass(planar_kernel,
                               static_cast<int>(std::min<long long>((n + kPlanarBlock - 1) / kPlanarBlock,
                                                                    148 * kPlanarBlocks)),
                               kPlanarBlock, st, a);
    if (rc) return rc;
    return launch_pass(apply_truncation_kernel, (V + 255) / 256, 256, st, V, const_cast<const float4*>(sc.cd), disp, pos,
                       sc.ts, sc.reach, 1.0f / sc.reach_unit, sc.max_disp, color < 0 ? 0 : m.color_start[color], color < 0 ? V : m.color_start[color + 1]);
}

}  // namespace vbd
