// Contacts between bodies: islands, the candidate pairs of nodes and collision triangles, their narrow phase and the
// contact response in the reference's pair order.
//
// Reference: World::build_islands (world.cpp:636-762), World::rebuild_pairs (world.cpp:1851-2308: node-triangle
// pairs only - no capsules, plate mid points or self collision), World::fast_pairs (world.cpp:2314-2520),
// World::near_pairs (world.cpp:2525-2598), World::pair_detect (world.cpp:2807-2858), World::collide_pairs
// (world.cpp:2964-3023) with contact_force<1,3> and hull_push_out<3> (world.cpp:59-120), the wake requests of sleeping
// bodies (world.cpp:2983-2995, 3333-3337).
//
// Layout. Collision triangles of all bodies back to back: int4 (a, b, c as global node indices; flags: bit 0 two-sided,
// bit 1 torn, bits 8.. the body) and their longest rest edge squared. Each frame k_islands labels every body with the
// first body of its island (the reference numbers islands in that order and keeps each island's bodies in body
// order). An island with two or more bodies has contact pairs: the contacts add to its nodes' forces (fnode: gravity
// and beams, k_force) before k_integrate takes the static contacts and integrates.
//
// The pair search runs on the substeps the reference rebuilds on (the frame's first and every rebuild interval after):
// one CTA per island (k_rebuild) sets up the island's search - margins, cell size, partners, the slow bodies' spatial
// hash, the fast bodies' dense grids - and lists its queries (a triangle against a hash or a grid); the queries of all
// islands are counted, placed and written by the whole GPU (bl_pair_search.cuh), the pairs near_pairs keeps in the
// reference's order. Every substep k_detect finds the contacts of all pairs in parallel and k_collide applies them one
// island per CTA, pair after pair: contact_force cancels the force accumulated so far on both sides, so the order
// within an island is the reference's.
#pragma once

#include "bl_kernels.cuh"

namespace blg {

constexpr int kIslMaxBodies = 256;     // bodies of one island with contact pairs (more: DEVERR_ISLAND)
constexpr int kGridCells = 48 * 48 * 48;
constexpr float kFastSpeed = 8.0f;     // world.cpp:1881
constexpr float kTornStretch2 = 2.5f * 2.5f; // softbody.h:154
enum : uint32_t { TF_TWO_SIDED = 1, TF_TORN = 2 };
enum : uint32_t { DEVERR_PAIRS = 4, DEVERR_ISLAND = 8, DEVERR_CONTACT_UNSUPPORTED = 32 };

struct IslSearch;
struct ContactRec;

struct Contacts {
    int4* tri;                 // a, b, c, flags | body << 8
    const float* tri_rest2;
    int* parent;               // per body: union-find
    float* ibox;               // per body: island box (6)
    int* isl_live;             // per root body: the island has an awake body
    int* isl_cnt;              // per root body: its bodies
    int* isl_nodes;            // per root body: its nodes
    int* isl_idx;              // per root body: its rank among the islands with pairs
    int* isl_noff;             // per root body: first node of its scratch
    int* isl_poff;             // per root body: its pairs in `pairs`
    int* isl_pcnt;
    int* isl_contacts;         // per root body: this frame's contacts (stats)
    int* pair_total;           // pairs of all islands (reset before each rebuild)
    int2* pairs;               // (node, triangle), global indices
    float4* hit_a;             // per pair: bary.xyz, pen
    float4* hit_b;             // per pair: normal.xyz, w = 1 when the pair is in contact
    uint32_t* hbits;           // per 32 pairs: bit j set when pair 32 w + j is in contact
    int* hidx;                 // per island's pair range: its contacts' pair indices, in pair order
    int whole_max;             // contacts an island runs whole at most (bl_gpu_config.contact_whole_max)
    int max_pairs;
    // rebuild scratch
    int* pt_node;              // hashed nodes of an island, in order
    int* pt_body;
    int4* pt_cell;
    int* bk_start;             // buckets (4 n + 65 per island)
    int* bk_fill;
    int* bk_items;             // hashed nodes by bucket
    int* run_end;
    int* g_start;              // fast grids: each fast body's cells' starts (a pool of cell_cap)
    int* g_items;              // fast grids' nodes, each listed once, in the lowest cell of its travel
    float4* g_rec;             // ... in the same order: position, reach of its travel (|v| x travel)
    int* g_hi;                 // ... the highest cell of its travel (x | y << 8 | z << 16)
    int4* sb_cell;             // slow hash items in bucket order: cell, body
    float4* sb_pos;            // ... position, node (bits)
    IslSearch* isl;            // per island with pairs (isl_idx): what its queries read
    int4* q_group;             // query groups: island (isl_idx), kind | k << 1 | ko << 9, triangles, first query
    int2* q_chunk;             // chunks of kQueryChunk queries of one group: group, first triangle of the chunk
    int* q_count;              // per query (a triangle of a group): its pairs, then their running sum over the island
    int* sc;                   // search counters: [0] queries [1] groups [2] chunks [3] grid cells [4] ptmp
    int2* ptmp;                // the count pass's pairs, query by query (ptmp_cap)
    int* q_tmp;                // per query with pairs: its pairs in ptmp (-1: not kept)
    int ptmp_cap;
    int q_cap, grp_cap, chunk_cap, cell_cap;
    int* counters;             // [0] pair searches [1] contacts [2] pairs of the searches
    int interval;              // rebuild interval in substeps (world.cpp:1887)
    float dt;
    float wake_speed;          // WorldSettings::sleep_speed
};

// ------------------------------------------------------------------------------------------ geometry (reference order)
__device__ __forceinline__ v3 cross(v3 a, v3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ float length2(v3 a) { return dot(a, a); }
__device__ __forceinline__ v3 vmin3(v3 a, v3 b) { return {smin(a.x, b.x), smin(a.y, b.y), smin(a.z, b.z)}; }
__device__ __forceinline__ v3 vmax3(v3 a, v3 b) { return {smax(a.x, b.x), smax(a.y, b.y), smax(a.z, b.z)}; }
__device__ __forceinline__ v3 neg(v3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ v3 nd_p(const float4* nd, int i) {
    const float4 p = nd[2 * i];
    return V(p.x, p.y, p.z);
}
__device__ __forceinline__ v3 nd_v(const float4* nd, int i) {
    const float4 v = nd[2 * i + 1];
    return V(v.x, v.y, v.z);
}
__device__ __forceinline__ float max_edge2(v3 a, v3 b, v3 c) { return smax(length2(b - a), smax(length2(c - b), length2(a - c))); }

// world.cpp:23-25 (the int products wrap, as the reference's do)
__device__ __forceinline__ uint32_t cell_hash(int x, int y, int z) {
    return ((uint32_t)x * 73856093u) ^ ((uint32_t)y * 19349663u) ^ ((uint32_t)z * 83492791u);
}

// closest_on_triangle (softbody.h:158-190, Ericson 5.1.5)
__device__ v3 closest_on_triangle(v3 p, v3 a, v3 b, v3 c, v3& bary) {
    const v3 ab = b - a, ac = c - a, ap = p - a;
    const float d1 = dot(ab, ap), d2 = dot(ac, ap);
    if (d1 <= 0 && d2 <= 0) {
        bary = V(1, 0, 0);
        return a;
    }
    const v3 bp = p - b;
    const float d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= 0 && d4 <= d3) {
        bary = V(0, 1, 0);
        return b;
    }
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0 && d1 >= 0 && d3 <= 0) {
        const float v = d1 / (d1 - d3);
        bary = V(1 - v, v, 0);
        return a + ab * v;
    }
    const v3 cp = p - c;
    const float d5 = dot(ab, cp), d6 = dot(ac, cp);
    if (d6 >= 0 && d5 <= d6) {
        bary = V(0, 0, 1);
        return c;
    }
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0 && d2 >= 0 && d6 <= 0) {
        const float w = d2 / (d2 - d6);
        bary = V(1 - w, 0, w);
        return a + ac * w;
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        bary = V(0, 1 - w, w);
        return b + (c - b) * w;
    }
    const float denom = 1.0f / (va + vb + vc);
    const float v = vb * denom, w = vc * denom;
    bary = V(1 - v - w, v, w);
    return a + ab * v + ac * w;
}

// near_triangle (world.cpp:1135-1142)
__device__ __forceinline__ bool near_triangle(v3 p, v3 a, v3 b, v3 c, v3 tu, float r, bool two_sided, float depth) {
    const float s = dot(p - a, tu);
    v3 bary;
    if (two_sided) return fabsf(s) <= r && length2(closest_on_triangle(p, a, b, c, bary) - p) <= r * r;
    if (s > r || s < -r - depth) return false;
    const v3 q = p - tu * s;
    return length2(closest_on_triangle(q, a, b, c, bary) - q) <= r * r;
}

__device__ __forceinline__ bool outside(v3 p, v3 mn, v3 mx) { return p.x < mn.x || p.y < mn.y || p.z < mn.z || p.x > mx.x || p.y > mx.y || p.z > mx.z; }

// ------------------------------------------------------------------------------------------ block helpers
// exclusive scan of one int per thread of the block; *total: the block's sum. Every thread of the block calls it.
__device__ int block_scan_excl(int v, int& total, int* s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < nw ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) s_warp[lane] = t;
    }
    __syncthreads();
    const int before = (w > 0 ? s_warp[w - 1] : 0) + x - v;
    total = s_warp[nw - 1];
    __syncthreads();
    return before;
}

// a[0..n) := its inclusive prefix sums, in place, by the whole block: each thread sums a contiguous run, one block scan
// of the runs' sums, each thread rewrites its run (two block scans' barriers however long the array; the same integers
// as scanning it 1,024 entries at a time)
__device__ void block_scan_incl_inplace(int* a, int n, int* s_warp) {
    const int nt = blockDim.x, per = (n + nt - 1) / nt;
    const int lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
    int sum = 0;
    for (int i = lo; i < hi; i++) sum += a[i];
    int tot;
    int run = block_scan_excl(sum, tot, s_warp);
    for (int i = lo; i < hi; i++) run += a[i], a[i] = run;
}

// ------------------------------------------------------------------------------------------ islands (once a frame)
__device__ __forceinline__ int uf_find(volatile int* parent, int x) {
    while (true) {
        const int p = parent[x];
        if (p == x) return x;
        x = p;
    }
}
__device__ void uf_union(int* parent, int a, int b) {
    while (true) {
        a = uf_find(parent, a), b = uf_find(parent, b);
        if (a == b) return;
        if (a > b) {
            const int t = a;
            a = b, b = t;
        }
        if (atomicCAS(&parent[b], b, a) == b) return; // (the larger root under the smaller: a component's root is its first body)
    }
}

// World::build_islands (world.cpp:636-720) for bodies that can touch: node-triangle contacts only (no capsules or
// collision volumes). One block. Bodies with FEM frames take no contacts here: one that would is flagged
// (DEVERR_CONTACT_UNSUPPORTED) and stays in an island of its own.
__global__ void __launch_bounds__(1024) k_islands(Body* __restrict__ bodies, int nb, float frame_time, int world_sleeping, Contacts C,
                                                  uint32_t* __restrict__ deverr) {
    __shared__ int s_warp[32];
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        Body& B = bodies[i];
        if (!world_sleeping) B.sleeping = 0;
        C.parent[i] = i;
        C.isl_live[i] = 0, C.isl_cnt[i] = 0, C.isl_nodes[i] = 0, C.isl_pcnt[i] = 0, C.isl_contacts[i] = 0;
        const float m = (B.sleeping ? 0.05f : smin(B.max_speed, 200.0f) * frame_time * 2.0f + 0.3f) + (B.hull ? B.hull_depth : 0.0f);
        float* bx = C.ibox + 6 * i;
        bx[0] = B.aabb_mn[0] - m, bx[1] = B.aabb_mn[1] - m, bx[2] = B.aabb_mn[2] - m;
        bx[3] = B.aabb_mx[0] + m, bx[4] = B.aabb_mx[1] + m, bx[5] = B.aabb_mx[2] + m;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        const Body& Bi = bodies[i];
        const float* a = C.ibox + 6 * i;
        for (int j = i + 1; j < nb; j++) {
            const float* b = C.ibox + 6 * j;
            if (!(a[0] <= b[3] && a[3] >= b[0] && a[1] <= b[4] && a[4] >= b[1] && a[2] <= b[5] && a[5] >= b[2])) continue;
            const Body& Bj = bodies[j];
            if (Bi.sleeping && Bj.sleeping) continue;
            if (Bi.group != 0 && Bi.group == Bj.group) continue;
            const bool can = (Bi.contacters && Bj.ntris > 0) || (Bj.contacters && Bi.ntris > 0);
            if (!can) continue;
            if (Bi.is_fem || Bj.is_fem) {
                atomicOr(deverr, DEVERR_CONTACT_UNSUPPORTED);
                continue;
            }
            uf_union(C.parent, i, j);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        const int r = uf_find(C.parent, i);
        C.parent[i] = r;
        atomicAdd(&C.isl_cnt[r], 1);
        atomicAdd(&C.isl_nodes[r], bodies[i].nnodes);
        if (!bodies[i].sleeping) atomicOr(&C.isl_live[r], 1);
    }
    __syncthreads();
    // the islands with pairs: their rank and their first node of scratch (in body order)
    int carry_n = 0, carry_i = 0;
    for (int base = 0; base < nb; base += blockDim.x) {
        const int i = base + threadIdx.x;
        bool pr = false;
        if (i < nb) {
            Body& B = bodies[i];
            const int r = C.parent[i];
            const bool live = C.isl_live[r] != 0;
            B.island = live ? r : -1;
            B.pairs = live && C.isl_cnt[r] > 1 ? 1 : 0;
            B.body_contacts = 0;
            pr = r == i && B.pairs;
        }
        int tn, ti;
        const int on = block_scan_excl(pr ? C.isl_nodes[i] : 0, tn, s_warp);
        const int oi = block_scan_excl(pr ? 1 : 0, ti, s_warp);
        if (pr) C.isl_noff[i] = carry_n + on, C.isl_idx[i] = carry_i + oi;
        carry_n += tn, carry_i += ti;
    }
}

// ------------------------------------------------------------------------------------------ wake requests (each substep)
// simulate_island's substep start (world.cpp:3333-3337): a sleeping body a moving partner touched wakes; its beams step
// again (SoftBody::wake, softbody.h:996).
__global__ void k_wake(Body* bodies, uint32_t* bmeta) {
    pdl_wait();
    Body& B = bodies[blockIdx.x];
    if (!B.wake_request || B.island < 0) return;
    for (int j = threadIdx.x; j < B.nbeams; j += blockDim.x) bmeta[B.beam0 + j] &= ~kBeamAsleep;
    __syncthreads();
    if (threadIdx.x == 0) B.wake_request = 0, B.sleeping = 0, B.sleep_timer = 0.0f;
}

// ------------------------------------------------------------------------------------------ the pair search
} // namespace blg
#include "bl_pair_search.cuh"
namespace blg {

// ------------------------------------------------------------------------------------------ narrow phase (each substep)
// World::pair_detect for node-triangle pairs (world.cpp:2819-2858): hit_a = (bary, pen), hit_b = (normal, 1) when
// the pair is in contact, hit_b.w = 0 when not. All of it before the wait (bl_device.cuh): the nodes and the bodies' sleep
// from L2.
__global__ void __launch_bounds__(256) k_detect(const float4* nd, const int4* __restrict__ info, const Body* bodies, Contacts C) {
    auto at = [nd](int i) {
        const float4 p = __ldcg(nd + i);
        return V(p.x, p.y, p.z);
    };
    const int total = min(*C.pair_total, C.max_pairs);
    // (a warp takes 32 consecutive pairs: its ballot is their word of hit bits)
    for (int i0 = blockIdx.x * blockDim.x; i0 < total; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + (int)threadIdx.x;
        bool hit = false;
        if (i < total) {
            const int2 pr = C.pairs[i];
            const int4 tr = C.tri[pr.y];
            const Body& bn = bodies[info[pr.x].w];
            const Body& bt = bodies[tr.w >> 8];
            float4 ha = make_float4(0, 0, 0, 0), hb = make_float4(0, 0, 0, 0);
            do {
                if (__ldcg(&bn.sleeping) && __ldcg(&bt.sleeping)) break;
                if (tr.w & TF_TORN) break; // (torn since the pairs were found)
                const bool two_sided = (tr.w & TF_TWO_SIDED) != 0;
                const v3 np = at(2 * pr.x);
                const v3 a = at(2 * tr.x), b = at(2 * tr.y), cc = at(2 * tr.z);
                v3 bary;
                const float r = bt.faces_only && !two_sided ? bt.face_skin : bn.crad;
                if (!two_sided) {
                    // a hull triangle: over its face pushed out along the face's normal, from as deep as the hull's depth
                    const v3 fn = normalize(cross(b - a, cc - a));
                    const float s = dot(np - a, fn);
                    if (s >= r || s < -bt.hull_depth) break;
                    const v3 q = np - fn * s;
                    const v3 cq = closest_on_triangle(q, a, b, cc, bary);
                    if (length2(cq - q) <= 1e-6f) {
                        ha = make_float4(bary.x, bary.y, bary.z, r - s), hb = make_float4(fn.x, fn.y, fn.z, 0.0f);
                        hit = true;
                        break;
                    }
                    if (s < 0 || bt.faces_only) break;
                } else {
                    const v3 lo = vmin3(a, vmin3(b, cc)) - V(r, r, r), hi = vmax3(a, vmax3(b, cc)) + V(r, r, r);
                    if (outside(np, lo, hi)) break;
                }
                const v3 cp = closest_on_triangle(np, a, b, cc, bary);
                const v3 d = np - cp;
                const float dist2 = dot(d, d);
                if (dist2 >= r * r) break;
                const float dist = sqrtf(dist2);
                v3 nrm;
                if (dist > 1e-5f) {
                    nrm = divs(d, dist);
                } else {
                    nrm = normalize(cross(b - a, cc - a));
                    const v3 vt = at(2 * tr.x + 1) * bary.x + at(2 * tr.y + 1) * bary.y + at(2 * tr.z + 1) * bary.z;
                    if (dot(at(2 * pr.x + 1) - vt, nrm) > 0) nrm = neg(nrm);
                }
                ha = make_float4(bary.x, bary.y, bary.z, r - dist), hb = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
                hit = true;
            } while (false);
            hb.w = hit ? 1.0f : 0.0f;
            C.hit_a[i] = ha;
            C.hit_b[i] = hb;
        }
        const unsigned bits = __ballot_sync(0xffffffffu, hit);
        if ((threadIdx.x & 31) == 0) C.hbits[i >> 5] = bits;
    }
    pdl_wait(); // (it needs the positions, not the forces: it runs beside the forces' kernel)
}

// ------------------------------------------------------------------------------------------ response (each substep)
// World::collide_pairs for node-triangle pairs (world.cpp:2975-3023): each contact cancels the forces accumulated so far
// on its node and its triangle's corners (earlier contacts' included), so an island's contacts run one after another
// in pair order, as the reference's loop (world.cpp:2999) - but only contacts that share a node depend on each other.
// A CTA an island:
//  1. its contacts (its pairs with a hit bit, in pair order) listed by a block scan; their nodes hashed into
//     shared-memory force slots;
//  2. each contact's level, one above its nodes' earlier contacts' levels, so the contacts of one level touch distinct
//     nodes; the contacts sorted by level. Up to kParMax contacts: each slot's contacts in a list, from it each
//     contact's nearest earlier one at each of its nodes, then one warp goes through the contacts 32 at a time
//     (contact_levels). More: one thread, in pair order;
//  3. each contact's record - its slots, the accumulation weights, relative velocity and normal, and every term of the
//     contact law that does not depend on the forces (the slip direction and speed, the Stribeck exponentials, the
//     restitution and push terms, the soft ground's drag and buoyancy) - formed in level order into shared memory, half a
//     buffer at a time, while
//  4. one warp runs the levels one after another, a level's contacts at once, each contact with only its force-dependent
//     arithmetic (apply_contact) - every contact sees the forces the serial loop gives it;
//  5. the forces written back. Above Contacts::whole_max contacts an island runs kRecChunk at a time (records and levels
//     of each chunk in turn); with more distinct contact nodes than the slots hold it runs the loop on global memory
//     (collide_island_global). Results are the same bits every way.
// Up to kSmall contacts each has a thread, its record is formed while one warp finds the levels, and no half buffers are
// needed (nearly every island: 350 contacts at the peak of two vehicles' crash).
// The chain of levels bounds it, an island's latency whatever the others do; next the fetching of its code (the first
// pass through any part of it costs several times the later ones, most with every SM at it). B200, at an island's 350
// contacts in 41 to 57 levels, in 1,000 cycles: the levels 33 by one thread (95 a contact), 20 so; the chain 68 to 89 with the
// records read from global memory and the law's cases branched on, 34 so; the nodes' forces into the slots 16, 7 so.
// A launch for 128 head-on pairs of vehicles 100 us, 63 so; for two crashing trusses (46 contacts) 10.1 and 6.5 us.
__device__ void collide_island_global(const float4* nd, const int4* __restrict__ info, Body* __restrict__ bodies, Contacts C,
                                      float4* __restrict__ Fs, int root, int off, int cnt);

constexpr int kCollideThreads = 512;
constexpr int kKeyBits = 13, kKeys = 1 << kKeyBits; // the hash of an island's contact nodes
constexpr int kSlots = kKeys / 2;                   // force slots, one a distinct contact node (the hash at most half full)
constexpr int kSlotPad = 8;                         // slot levels past the slots (kSlots: a level that stays 0)
constexpr int kRecChunk = 448;                      // contact records formed at a time where an island does not run whole
constexpr int kStage = 6144;                        // contacts of an island that runs whole
constexpr int kParMax = 2048;                       // ... whose levels are found from lists
constexpr int kSmall = 448;                         // ... a thread each, the records of all at once; the last warps stay free

struct alignas(16) ContactRec {
    int sa, sb[3];        // force slots of the node and the triangle's corners
    float ca, cb[3];      // acc = FA ca - sum FB_q cb_q (the terms the movable sides have)
    float wb[3], m;       // barycentric weights; effective mass
    float nx, ny, nz;     // the normal passed to the law (negated where the node's side is immovable)
    float vx, vy, vz;     // the relative velocity passed to the law
    float pen, fric;
    float Vn, rsub;       // vel . normal; the restitution / push term of R where Vn < 0 (else 0); hull: (target - vr) m / dt
    float sx, sy, sz;     // the slip direction (0 where the slip speed is below 1e-9)
    float sv, stop;       // the slip speed; mass sv / dt
    float e1, gsum;       // 1 - exp(-sv / va); the dynamic friction's g + min(t2 sv, 5)
    float dragf, fb0;     // the soft ground's drag factor and buoyancy (where it is soft under the contact)
    int kind;             // 0 none, 1 contact (node movable), 2 contact (node immovable), 3 hull push-out; | ma << 4 | mb << 5
                          // | soft (drag, buoyancy) << 6 | pen >= soft depth << 7
};

struct alignas(16) ContactRecPad { // (a stride whose rows fall in distinct banks)
    ContactRec r;
    int4 pad;
};
// the work area of k_collide (bytes): a small island's records, then its contacts' nearest earlier ones, levels, order and
// level starts - the lists of the levels in the records' place; otherwise up to kStage contacts' slots and levels, or
// up to kParMax contacts' slots, nearest earlier ones, list entries, levels and the list heads
constexpr int kWorkPred = kSmall * (int)sizeof(ContactRecPad), kWorkLv = kWorkPred + 8 * kSmall, kWorkOrd = kWorkLv + 2 * kSmall + 16,
              kWorkLe = kWorkOrd + 2 * kSmall, kCollideWork = kWorkLe + 4 * kSmall + 16;
constexpr int kWorkParPred = 8 * kParMax, kWorkParNext = 16 * kParMax, kWorkLv16 = 8 * kStage, kWorkParHead = kWorkLv16 + 2 * kParMax + 16;
static_assert(kCollideWork >= 10 * kStage && kCollideWork >= kWorkParHead + 4 * kSlots && kWorkParNext + 8 * kParMax <= kWorkLv16, "the work area's uses");

__device__ __forceinline__ int key_hash(int key) { return (int)(((uint32_t)key * 2654435761u) >> (32 - kKeyBits)); }
__device__ __forceinline__ int key_find(const int* keys, int key) {
    int h = key_hash(key);
    while (keys[h] != key) h = (h + 1) & (kKeys - 1);
    return h;
}

// One contact of the chain on the forces in the slots: only the force-dependent arithmetic, the reference's operations
// in its order (contact_force<1, 3> / hull_push_out<3> and primitive_collision, world.cpp:59-120,
// static_world.cpp:8-51, split at their force-independent parts, which the record holds). The kinds and the stick and
// slip cases are chosen at the end, not branched on: a warp's lanes hold different ones, and the chain waits for each.
__device__ __forceinline__ void apply_contact(const ContactRec& R, float4* F_, const GroundModel& gm) {
    const int kind = R.kind & 15;
    const bool ma = R.kind & 16, mb = R.kind & 32;
    const float4 a4 = F_[R.sa], b40 = F_[R.sb[0]], b41 = F_[R.sb[1]], b42 = F_[R.sb[2]];
    const v3 FA = V(a4.x, a4.y, a4.z), FB[3] = {V(b40.x, b40.y, b40.z), V(b41.x, b41.y, b41.z), V(b42.x, b42.y, b42.z)};
    v3 acc = V(0, 0, 0);
    const v3 acca = acc + FA * R.ca;
    if (ma) acc = acca;
    v3 accb = acc;
#pragma unroll
    for (int q = 0; q < 3; q++) accb = accb - FB[q] * R.cb[q];
    if (mb) acc = accb;
    const v3 nrm = V(R.nx, R.ny, R.nz);
    // kind 3: along the normal
    const float fn = R.rsub - dot(acc, nrm) * R.m;
    // kinds 1 and 2: primitive_collision (static_world.cpp:8-51) with its force-independent terms from the record
    v3 F = acc * R.m;
    if (kind != 1) F = neg(F);
    v3 out = V(0, 0, 0);
    const float Vn = R.Vn, Fn = dot(F, nrm);
    if (R.kind & 64) {
        const v3 vel = V(R.vx, R.vy, R.vz);
        out = out + vel * R.dragf;
        float Fb = R.fb0;
        if (Vn >= 0 && Fn < 0 && Fb > -Fn) Fb = -Fn;
        out = out + nrm * Fb;
    }
    float Rn = -Fn;
    if (Vn < 0) Rn -= R.rsub;
    const v3 slipF = F - nrm * Fn, slip = V(R.sx, R.sy, R.sz), nR = nrm * Rn;
    const float G = Rn * gm.strength * R.fric;
    const bool on = (R.kind & 128) && Rn > 0;
    const v3 slide = nR - slip * smin(R.gsum * G, smax(0.0f, R.stop + dot(slipF, slip)));
    v3 hard = slide;
    if (on && R.sv < gm.va && G > 0 && length(slipF) <= gm.ms * G) hard = nR - slip * smin(gm.ms * G * R.e1, R.stop) - slipF;
    const v3 sum = out + hard;
    if (on) out = sum;
    if (kind == 3) out = nrm * fn;
    const bool toA = kind == 3 ? fn > 0 && ma : kind == 1, toB = kind == 3 ? fn > 0 && mb : kind == 2 || mb;
    if (kind == 2) out = neg(out); // (FB + out w as FB - (-out) w: the same bits)
    if (toA) F_[R.sa] = make_float4(FA.x + out.x, FA.y + out.y, FA.z + out.z, 0.0f);
    if (toB)
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const v3 f = FB[q] - out * R.wb[q];
            F_[R.sb[q]] = make_float4(f.x, f.y, f.z, 0.0f);
        }
}

// What a contact's record is formed from
struct ContactIn {
    int2 pr;
    int4 tr;
    float4 ha, hb, P[4], Vv[4]; // (the node's and its triangle's corners')
    int4 ina;
};
__device__ __forceinline__ void load_contact(ContactIn& I, int i, const float4* nd, const int4* __restrict__ info, const Contacts& C) {
    I.ha = C.hit_a[i], I.hb = C.hit_b[i];
    I.pr = C.pairs[i];
    I.tr = C.tri[I.pr.y];
    I.ina = info[I.pr.x];
    const int at[4] = {I.pr.x, I.tr.x, I.tr.y, I.tr.z};
#pragma unroll
    for (int q = 0; q < 4; q++) I.P[q] = nd[2 * at[q]], I.Vv[q] = nd[2 * at[q] + 1];
}

// One contact's record (kind 0 where the law gives it no force; sl: its slots): the accumulation weights and every
// force-independent term of the law, and the wake requests of its sleeping sides. True when it is a contact (counted).
__device__ __forceinline__ bool form_record(ContactRec& R, const ContactIn& I, const int* sl, Body* __restrict__ bodies, const Contacts& C,
                                            const GroundModel& gm, float dt) {
    R.kind = 0;
    const float4 hb4 = I.hb, ha = I.ha;
    const int4 tr = I.tr;
    Body& bn = bodies[I.ina.w];
    Body& bt = bodies[tr.w >> 8];
    // movable (world.cpp:2983-2993): a sleeping side is immovable and asks to wake when the other moves
    bool ma = true, mb = true;
    if (bn.sleeping) {
        if (sqrtf(bt.acc_v2) > smax(C.wake_speed, bt.sleep_speed) * 1.0f) bn.wake_request = 1;
        ma = false;
    }
    if (bt.sleeping) {
        if (sqrtf(bn.acc_v2) > smax(C.wake_speed, bn.sleep_speed) * 1.0f) bt.wake_request = 1;
        mb = false;
    }
    const float wb[3] = {ha.x, ha.y, ha.z};
    const v3 n = V(hb4.x, hb4.y, hb4.z);
    const float pen = ha.w;
    const v3 Av = V(I.Vv[0].x, I.Vv[0].y, I.Vv[0].z);
    const float Aim = I.P[0].w;
    v3 Bv[3];
    float Bim[3];
#pragma unroll
    for (int q = 0; q < 3; q++) Bv[q] = V(I.Vv[q + 1].x, I.Vv[q + 1].y, I.Vv[q + 1].z), Bim[q] = I.P[q + 1].w;
    R.sa = sl[0];
#pragma unroll
    for (int q = 0; q < 3; q++) R.sb[q] = sl[q + 1], R.wb[q] = wb[q], R.cb[q] = wb[q] * Bim[q];
    const int mv = (ma ? 16 : 0) | (mb ? 32 : 0);
    if (!(tr.w & TF_TWO_SIDED) && pen > bn.crad) {
        // hull_push_out<3> (world.cpp:97-118): behind a hull's face
        float W = ma ? Aim : 0.0f;
        if (mb)
            for (int q = 0; q < 3; q++) W += wb[q] * wb[q] * Bim[q];
        if (W <= 1e-12f) return false;
        v3 vb = V(0, 0, 0);
        for (int q = 0; q < 3; q++) vb = vb + Bv[q] * wb[q];
        const float m = 1.0f / W, vr = dot(Av - vb, n), target = smin(0.2f * pen / dt, 2.0f);
        R.ca = Aim, R.m = m, R.nx = n.x, R.ny = n.y, R.nz = n.z;
        R.rsub = (target - vr) * m / dt;
        R.kind = 3 | mv;
    } else {
        // contact_force<1, 3> (world.cpp:59-92), the node's weight 1; a tyre node grips with its own friction
        // (world.cpp:3013)
        const float fric = ((uint32_t)I.ina.x & NF_TYRE) ? __int_as_float(I.ina.y) : 0.8f * smin(bn.cfric, bt.cfric);
        float W = 0;
        if (ma) W += 1.0f * 1.0f * Aim;
        if (mb)
            for (int q = 0; q < 3; q++) W += wb[q] * wb[q] * Bim[q];
        if (W <= 1e-12f) return false;
        const float m = 1.0f / W;
        v3 va = V(0, 0, 0), vb = V(0, 0, 0);
        va = va + Av * 1.0f;
        for (int q = 0; q < 3; q++) vb = vb + Bv[q] * wb[q];
        const v3 vel = ma ? va - vb : vb - va, nrm = ma ? n : neg(n);
        R.ca = 1.0f * Aim, R.m = m, R.fric = fric, R.pen = pen;
        R.nx = nrm.x, R.ny = nrm.y, R.nz = nrm.z, R.vx = vel.x, R.vy = vel.y, R.vz = vel.z;
        // primitive_collision's force-independent terms (static_world.cpp:8-51; push_max 2, slop 0, no
        // restitution)
        const float Vn = dot(vel, nrm), sgl = gm.soft_depth;
        R.Vn = Vn;
        R.rsub = Vn < 0 ? (0.8f * Vn - smin(0.2f * smax(0.0f, pen - sgl - 0.0f) / dt, 2.0f)) * m / dt : 0.0f;
        v3 slip = vel - nrm * Vn;
        const float sv = length(slip);
        if (sv > 1e-9f) slip = divs(slip, sv);
        else slip = V(0, 0, 0);
        R.sx = slip.x, R.sy = slip.y, R.sz = slip.z, R.sv = sv, R.stop = m * sv / dt;
        R.e1 = 1.0f - bl_expf(-sv / gm.va);
        const float g = gm.mc + (gm.ms - gm.mc) * bl_expf(-bl_powf(sv / gm.vs, gm.alpha));
        R.gsum = g + smin(gm.t2 * sv, 5.0f);
        const bool soft = sgl > 0 && pen >= 0;
        R.dragf = soft ? -gm.fluid_drag * smin(1.0f, pen / sgl + 0.2f) : 0.0f;
        R.fb0 = soft ? gm.fluid_density * smin(pen, sgl) * 9.807f * 0.02f : 0.0f;
        R.kind = (ma ? 1 : 2) | mv | (soft ? 64 : 0) | (pen >= sgl ? 128 : 0);
    }
    atomicAdd(&bn.body_contacts, 1);
    atomicAdd(&bt.body_contacts, 1);
    return true;
}

// One warp: each contact's level from its nearest earlier contacts (pred: at each node, n where there is none; lv[n] 0),
// 32 contacts at a time - those before the 32 have their levels, those among them are passed round until none moves.
// Returns the deepest level.
__device__ __forceinline__ int contact_levels(int n, const ushort4* pred, unsigned short* lv) {
    const int lane = threadIdx.x & 31;
    int deepest = 0;
    if (lane == 0) lv[n] = 0;
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c < n; c += 32) {
        const int j = c + lane;
        const ushort4 e4 = j < n ? pred[j] : make_ushort4((unsigned short)n, (unsigned short)n, (unsigned short)n, (unsigned short)n);
        const int e[4] = {e4.x, e4.y, e4.z, e4.w};
        int l = 0;
        bool here[4], any = false;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            here[q] = e[q] >= c && e[q] < n;
            any |= here[q];
            if (!here[q]) l = max(l, (int)lv[e[q]]);
        }
        l++;
        if (__any_sync(0xffffffffu, any)) {
            int before;
#pragma unroll 1
            do {
                before = l;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int v = __shfl_sync(0xffffffffu, before, e[q] - c) + 1;
                    if (here[q]) l = max(l, v);
                }
            } while (__any_sync(0xffffffffu, l != before));
        }
        if (j < n) lv[j] = (unsigned short)l, deepest = max(deepest, l);
        __syncwarp();
    }
    return __reduce_max_sync(0xffffffffu, deepest);
}
// One warp: the contacts by level in ord (a level's in any order: they share no node); le[L]: level L's start, 1 <= L <=
// depth + 1
__device__ __forceinline__ void sort_by_level(int n, int depth, const unsigned short* lv, int* le, unsigned short* ord) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int l = lane; l < depth + 3; l += 32) le[l] = 0;
    __syncwarp();
#pragma unroll 1
    for (int j = lane; j < n; j += 32) atomicAdd(&le[lv[j]], 1);
    __syncwarp();
    int carry = 0;
#pragma unroll 1
    for (int c = 0; c < depth + 2; c += 32) {
        const int l = c + lane;
        int x = l < depth + 2 ? le[l] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (l < depth + 2) le[l] = carry + x;
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    __syncwarp();
#pragma unroll 1
    for (int j = lane; j < n; j += 32) ord[atomicSub(&le[lv[j]], 1) - 1] = (unsigned short)j;
    __syncwarp();
}
// One warp: the contacts at places p .. end of the order, level after level (L: the first's), a lane a contact; the next
// contacts' records (at(place)) loaded while these run
template <class At>
__device__ __forceinline__ void run_levels(int p, int end, int& L, const int* le, At at, float4* F, const GroundModel& gm) {
    const int lane = threadIdx.x & 31;
    int n = p < end ? min(32, min(le[L + 1], end) - p) : 0, n2;
    auto next = [&]() { // the contacts after these
        const int pn = p + n;
        if (pn == le[L + 1]) L++;
        n2 = pn < end ? min(32, min(le[L + 1], end) - pn) : 0;
        p = pn;
    };
    ContactRec cur, nxt;
    if (lane < n) cur = at(p + lane);
#pragma unroll 1
    while (n > 0) {
        const bool on = lane < n && (cur.kind & 15);
        next();
        if (lane < n2) nxt = at(p + lane);
        if (on) apply_contact(cur, F, gm);
        __syncwarp();
        cur = nxt, n = n2;
    }
}

__global__ void __launch_bounds__(kCollideThreads, 1) k_collide(const float4* nd, const int4* __restrict__ info, Body* __restrict__ bodies,
                                                            int nbodies, Contacts C, float4* __restrict__ Fs) {
    extern __shared__ __align__(16) unsigned char csm[];
    int* keys = reinterpret_cast<int*>(csm);                                   // the hash: a node, or -1
    unsigned short* cid = reinterpret_cast<unsigned short*>(keys + kKeys);     // ... its slot
    float4* F = reinterpret_cast<float4*>(cid + kKeys);                        // per slot: the node's force
    int* unode = reinterpret_cast<int*>(F + kSlots);                           // per slot: the node
    unsigned short* slot_lvl = reinterpret_cast<unsigned short*>(unode + kSlots); // per slot: its latest contact's level
    unsigned char* work = reinterpret_cast<unsigned char*>(slot_lvl + kSlots + kSlotPad);
    __shared__ int used, overflow, ncontacts, s_depth;
    const int root = blockIdx.x, tid = threadIdx.x;
    pdl_wait();
    if (root >= nbodies) return;
    const int cnt = C.isl_pcnt[root];
    if (cnt <= 0 || bodies[root].island != root || !bodies[root].pairs) return;
    const int off = C.isl_poff[root];
    const float dt = C.dt;
    const GroundModel& gm = c_ground[3]; // SURF_CONCRETE
    for (int h = tid; h < kKeys / 4; h += kCollideThreads) reinterpret_cast<int4*>(keys)[h] = make_int4(-1, -1, -1, -1);
    if (tid == 0) used = 0, overflow = 0, ncontacts = 0, s_depth = 0;
    __shared__ int s_scan[32];
    // 0. the island's contacts (its pairs with a hit), in pair order, into hidx[off ...): a run of pairs a thread
    int nh_all;
    {
        // (the range's words of hit bits, a run of words a thread, the bits outside the range masked)
        const int w0 = off >> 5, nw = ((off + cnt - 1) >> 5) - w0 + 1;
        const int per = (nw + kCollideThreads - 1) / kCollideThreads;
        const int lo = min(nw, tid * per), hi = min(nw, lo + per);
        auto word = [&](int w) {
            uint32_t m = C.hbits[w0 + w];
            const int b0 = (w0 + w) << 5;
            if (b0 < off) m &= ~0u << (off - b0);
            if (b0 + 32 > off + cnt) m &= (off + cnt - b0 >= 32) ? ~0u : ((1u << (off + cnt - b0)) - 1u);
            return m;
        };
        int mine = 0;
        for (int w = lo; w < hi; w++) mine += __popc(word(w));
        int at = off + block_scan_excl(mine, nh_all, s_scan);
        for (int w = lo; w < hi; w++)
            for (uint32_t m = word(w); m; m &= m - 1) C.hidx[at++] = ((w0 + w) << 5) + __ffs(m) - 1;
    }
    __syncthreads();
    if (nh_all == 0) return;
    const bool whole = nh_all <= C.whole_max, small = whole && nh_all <= kSmall;
    ushort4* sq = reinterpret_cast<ushort4*>(work); // (whole, not small) per contact: its slots
    // 1. the contacts' nodes into slots
    auto insert = [&](int node) { // (the node's place in the hash)
        int h = key_hash(node);
        for (int probe = 0;; probe++) {
            if (probe >= kKeys / 2 || *(volatile int*)&overflow) {
                overflow = 1;
                break;
            }
            int prev = *(volatile int*)&keys[h];
            if (prev == -1) {
                prev = atomicCAS(&keys[h], -1, node);
                if (prev == -1) {
                    const int at = atomicAdd(&used, 1);
                    if (at >= kSlots) overflow = 1; // (kept at most half full: short probes)
                    else cid[h] = (unsigned short)at, unode[at] = node;
                    break;
                }
            }
            if (prev == node) break;
            h = (h + 1) & (kKeys - 1);
        }
        return h;
    };
    ContactIn own; // (small) the thread's contact
    const bool mine = small && tid < nh_all;
    unsigned long long places = 0; // (its nodes' places, 16 bits each)
    if (mine) {
        load_contact(own, C.hidx[off + tid], nd, info, C);
#pragma unroll 1
        for (int q = 0; q < 4; q++)
            places |= (unsigned long long)insert(q == 0 ? own.pr.x : q == 1 ? own.tr.x : q == 2 ? own.tr.y : own.tr.z) << (16 * q);
    }
    for (int j0 = tid; !small && j0 < nh_all; j0 += 4 * kCollideThreads) { // (four contacts a thread at a time: their loads overlap)
        int nodes4[4][4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int j = j0 + u * kCollideThreads;
            nodes4[u][0] = -1;
            if (j >= nh_all) continue;
            const int2 pr = C.pairs[C.hidx[off + j]];
            const int4 tr = C.tri[pr.y];
            nodes4[u][0] = pr.x, nodes4[u][1] = tr.x, nodes4[u][2] = tr.y, nodes4[u][3] = tr.z;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (nodes4[u][0] < 0) continue;
            const ushort4 h4 = make_ushort4((unsigned short)insert(nodes4[u][0]), (unsigned short)insert(nodes4[u][1]),
                                            (unsigned short)insert(nodes4[u][2]), (unsigned short)insert(nodes4[u][3]));
            if (whole) sq[j0 + u * kCollideThreads] = h4;
        }
    }
    __syncthreads();
    if (overflow) {
        if (tid == 0) collide_island_global(nd, info, bodies, C, Fs, root, off, cnt);
        return;
    }
    const int nused = used;
    for (int u = tid; u < nused; u += kCollideThreads) {
        const float4 f = Fs[unode[u]];
        F[u] = make_float4(f.x, f.y, f.z, 0.0f);
    }
    const bool last = tid >= kCollideThreads - 32; // (the warp of the levels and the chain)
    int L = 1;
    auto slots_of = [&](const ContactIn& I, int* sl) {
        sl[0] = cid[key_find(keys, I.pr.x)], sl[1] = cid[key_find(keys, I.tr.x)], sl[2] = cid[key_find(keys, I.tr.y)], sl[3] = cid[key_find(keys, I.tr.z)];
    };
    // contact j's nearest earlier contacts, from its nodes' lists (the four side by side)
    auto nearest = [&](int j, ushort4 h, const int* head, const unsigned short* next) {
        int e[4] = {head[h.x], head[h.y], head[h.z], head[h.w]}, best[4] = {-1, -1, -1, -1};
        while ((e[0] & e[1] & e[2] & e[3]) != 0xffff)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (e[q] == 0xffff) continue;
                const int o = e[q] >> 2;
                if (o < j && o > best[q]) best[q] = o;
                e[q] = next[e[q]];
            }
        auto at = [&](int q) { return (unsigned short)(best[q] < 0 ? nh_all : best[q]); };
        return make_ushort4(at(0), at(1), at(2), at(3));
    };
    auto list = [&](int j, ushort4 h, int* head, unsigned short* next) {
        next[4 * j] = (unsigned short)atomicExch(&head[h.x], 4 * j), next[4 * j + 1] = (unsigned short)atomicExch(&head[h.y], 4 * j + 1);
        next[4 * j + 2] = (unsigned short)atomicExch(&head[h.z], 4 * j + 2), next[4 * j + 3] = (unsigned short)atomicExch(&head[h.w], 4 * j + 3);
    };
    if (small) {
        int* head = reinterpret_cast<int*>(work);                                                      // per slot: its last-listed entry
        unsigned short* next = reinterpret_cast<unsigned short*>(work + 16 * kSmall);                  // per entry: the one listed before
        ushort4* pred = reinterpret_cast<ushort4*>(work + kWorkPred);
        unsigned short *lv = reinterpret_cast<unsigned short*>(work + kWorkLv), *ord = reinterpret_cast<unsigned short*>(work + kWorkOrd);
        int* le = reinterpret_cast<int*>(work + kWorkLe);
        ContactRecPad* rec = reinterpret_cast<ContactRecPad*>(work);
        for (int u = tid; u < nused; u += kCollideThreads) head[u] = 0xffff;
        const ushort4 h = mine ? make_ushort4(cid[places & 0xffff], cid[(places >> 16) & 0xffff], cid[(places >> 32) & 0xffff], cid[places >> 48])
                               : make_ushort4(0, 0, 0, 0);
        __syncthreads();
        if (mine) list(tid, h, head, next);
        __syncthreads();
        if (mine) pred[tid] = nearest(tid, h, head, next);
        __syncthreads();
        // 2. the levels and the order by the last warp, 3. the records by the others
        if (last) {
            const int depth = contact_levels(nh_all, pred, lv);
            sort_by_level(nh_all, depth, lv, le, ord);
        } else if (mine) {
            ContactRec R;
            const int sl[4] = {h.x, h.y, h.z, h.w};
            if (form_record(R, own, sl, bodies, C, gm, dt)) atomicAdd(&ncontacts, 1);
            rec[tid].r = R;
        }
        __syncthreads();
        // 4. the chain
        if (last) run_levels(0, nh_all, L, le, [&](int p) { return rec[ord[p]].r; }, F, gm);
    } else if (whole) {
        unsigned short* lv16 = reinterpret_cast<unsigned short*>(work + kWorkLv16); // per contact: its level
        for (int j = tid; j < nh_all; j += kCollideThreads) {
            const ushort4 h = sq[j];
            sq[j] = make_ushort4(cid[h.x], cid[h.y], cid[h.z], cid[h.w]);
        }
        // 2. the levels (a pair the law gives no force keeps its place, which only orders more)
        unsigned short* ord = reinterpret_cast<unsigned short*>(work); // (over the slots, done with)
        const int ord_bytes = (2 * nh_all + 15) & ~15;
        int* le = reinterpret_cast<int*>(work + ord_bytes);
        if (nh_all <= kParMax) {
            int* head = reinterpret_cast<int*>(work + kWorkParHead);
            unsigned short* next = reinterpret_cast<unsigned short*>(work + kWorkParNext);
            ushort4* pred = reinterpret_cast<ushort4*>(work + kWorkParPred);
            for (int u = tid; u < nused; u += kCollideThreads) head[u] = 0xffff;
            __syncthreads();
            for (int j = tid; j < nh_all; j += kCollideThreads) list(j, sq[j], head, next);
            __syncthreads();
            for (int j = tid; j < nh_all; j += kCollideThreads) pred[j] = nearest(j, sq[j], head, next);
            __syncthreads();
            if (last) {
                const int depth = contact_levels(nh_all, pred, lv16);
                if ((tid & 31) == 0) s_depth = depth;
            }
        } else {
            for (int u = tid; u < nused; u += kCollideThreads) slot_lvl[u] = 0;
            __syncthreads();
            if (tid == kCollideThreads - 32) {
                int depth = 0;
                ushort4 h = sq[0];
                for (int j = 0; j < nh_all; j++) {
                    const ushort4 hn = sq[min(j + 1, nh_all - 1)]; // (loaded before this contact's levels are stored)
                    const int l = max(max((int)slot_lvl[h.x], (int)slot_lvl[h.y]), max((int)slot_lvl[h.z], (int)slot_lvl[h.w])) + 1;
                    slot_lvl[h.x] = slot_lvl[h.y] = slot_lvl[h.z] = slot_lvl[h.w] = (unsigned short)l;
                    lv16[j] = (unsigned short)l;
                    depth = max(depth, l);
                    h = hn;
                }
                s_depth = depth;
            }
        }
        __syncthreads();
        const int le_bytes = (4 * (s_depth + 3) + 15) & ~15; // (with the order below the lists and levels: 6 bytes a contact and 44)
        if (last) sort_by_level(nh_all, s_depth, lv16, le, ord);
        __syncthreads();
        // 3, 4. the records of half a buffer formed by the other warps while the last runs the half before
        ContactRecPad* buf = reinterpret_cast<ContactRecPad*>(work + ord_bytes + le_bytes);
        const int half = (int)((kCollideWork - ord_bytes - le_bytes) / sizeof(ContactRecPad)) / 2;
        auto form = [&](int p0, int step) {
            ContactRecPad* dst = buf + ((p0 / half) & 1) * half;
            const int n = min(half, nh_all - p0);
            for (int r = tid; r < n; r += step) {
                ContactIn I;
                ContactRec R;
                int sl[4];
                load_contact(I, C.hidx[off + ord[p0 + r]], nd, info, C);
                slots_of(I, sl);
                if (form_record(R, I, sl, bodies, C, gm, dt)) atomicAdd(&ncontacts, 1);
                dst[r].r = R;
            }
        };
        form(0, kCollideThreads);
        __syncthreads();
        for (int p0 = 0; p0 < nh_all; p0 += half) {
            const ContactRecPad* src = buf + ((p0 / half) & 1) * half;
            if (last) run_levels(p0, min(nh_all, p0 + half), L, le, [&](int p) { return src[p - p0].r; }, F, gm);
            else if (p0 + half < nh_all) form(p0 + half, kCollideThreads - 32);
            __syncthreads();
        }
    } else {
        // the island's contacts in pair order, kRecChunk at a time
        ContactRec* rec = reinterpret_cast<ContactRec*>(work);
        for (int h = tid; h < kSlots + kSlotPad; h += kCollideThreads) slot_lvl[h] = 0;
        __shared__ int order[kRecChunk], lend[kRecChunk + 3], lv[kRecChunk];
        __shared__ int4 sl[kRecChunk + 1]; // per record: its slots (kSlots x 4: not a contact)
        for (int c0 = 0; c0 < nh_all; c0 += kRecChunk) {
            const int nh = min(kRecChunk, nh_all - c0);
            __syncthreads();
            // 2. the records of these contacts
            for (int r = tid; r < nh; r += kCollideThreads) {
                const int i = C.hidx[off + c0 + r];
                ContactRec& R = rec[r];
                sl[r] = make_int4(kSlots, kSlots, kSlots, kSlots); // (none: the slot whose level stays 0)
                ContactIn I;
                int s4[4];
                load_contact(I, i, nd, info, C);
                slots_of(I, s4);
                if (form_record(R, I, s4, bodies, C, gm, dt)) {
                    sl[r] = make_int4(R.sa, R.sb[0], R.sb[1], R.sb[2]);
                    atomicAdd(&ncontacts, 1);
                }
            }
            __syncthreads();
            // 3. the chain. A contact reads and writes the forces of its four nodes only, so one that shares no node with
            // the contacts between it and an earlier one commutes with them: each contact's level is one above the
            // latest level among its nodes' earlier contacts (one thread, in pair order), the contacts sorted by level,
            // then one warp runs them level after level, a level's contacts at once - every contact sees the forces the
            // serial loop gives it. Where the levels are nearly as many as the contacts, one thread runs the loop.
            for (int l = tid; l < kRecChunk + 3; l += kCollideThreads) lend[l] = 0;
            if (tid == 0) {
                int depth = 0, nk = 0;
                int4 h = sl[0];
                for (int r = 0; r < nh; r++) {
                    const int4 hn = sl[r + 1]; // (loaded before this record's levels are stored; sl[nh] is not used)
                    const int l = max(max((int)slot_lvl[h.x], (int)slot_lvl[h.y]), max((int)slot_lvl[h.z], (int)slot_lvl[h.w])) + 1;
                    const int lk = h.x == kSlots ? 0 : l;
                    slot_lvl[h.x] = slot_lvl[h.y] = slot_lvl[h.z] = slot_lvl[h.w] = (unsigned short)lk;
                    lv[r] = lk;
                    depth = max(depth, lk), nk += lk != 0;
                    h = hn;
                }
                s_depth = 5 * depth > 4 * nk ? -1 : depth;
            }
            __syncthreads();
            const int depth = s_depth;
            if (depth < 0) {
                if (tid == 0)
                    for (int r = 0; r < nh; r++)
                        if (lv[r]) apply_contact(rec[r], F, gm);
            } else if (depth > 0) {
                // by level: counts, ends (a running sum), places (each level's contacts in any order: they share no node)
                for (int r = tid; r < nh; r += kCollideThreads)
                    if (lv[r]) atomicAdd(&lend[lv[r]], 1);
                __syncthreads();
                block_scan_incl_inplace(lend, depth + 1, s_scan);
                __syncthreads();
                if (tid == 0) lend[depth + 1] = lend[depth];
                __syncthreads();
                for (int r = tid; r < nh; r += kCollideThreads)
                    if (lv[r]) order[atomicSub(&lend[lv[r]], 1) - 1] = r; // (lend[L] becomes level L's start)
                __syncthreads();
                if (tid < 32) {
                    // a lane a contact of the level; the next level's first contacts are looked up before this level runs
                    int s0 = lend[1], e0 = lend[2];
                    int rr = s0 + tid < e0 ? order[s0 + tid] : -1;
                    for (int L = 1; L <= depth; L++) {
                        const int s1 = lend[L + 1], e1 = L < depth ? lend[L + 2] : s1;
                        const int rn = s1 + tid < e1 ? order[s1 + tid] : -1;
                        if (rr >= 0) apply_contact(rec[rr], F, gm);
                        for (int k = s0 + tid + 32; k < e0; k += 32) apply_contact(rec[order[k]], F, gm);
                        __syncwarp();
                        s0 = s1, e0 = e1, rr = rn;
                    }
                }
            }
            __syncthreads();
            for (int r = tid; r < nh; r += kCollideThreads) {
                const int4 h = sl[r];
                slot_lvl[h.x] = slot_lvl[h.y] = slot_lvl[h.z] = slot_lvl[h.w] = 0;
            }
        }
    }
    __syncthreads();
    // 5. the forces back
    for (int u = tid; u < nused; u += kCollideThreads) Fs[unode[u]] = F[u];
    if (tid == 0) {
        C.isl_contacts[root] += ncontacts;
        if (ncontacts) atomicAdd(&C.counters[1], ncontacts);
    }
}
constexpr size_t kCollideSmem = sizeof(int) * kKeys + sizeof(unsigned short) * kKeys + sizeof(float4) * kSlots + sizeof(int) * kSlots +
                                sizeof(unsigned short) * (kSlots + kSlotPad) + kCollideWork;
static_assert(sizeof(ContactRec) * kRecChunk <= kCollideWork && sizeof(ContactRec) == 128, "the work area's uses");

// The serial loop on global memory (the path of an island with more distinct contact nodes than the slots hold)
__device__ void collide_island_global(const float4* nd, const int4* __restrict__ info, Body* __restrict__ bodies, Contacts C,
                                      float4* __restrict__ Fs, int root, int off, int cnt) {
    const float dt = C.dt;
    const GroundModel& gm = c_ground[3]; // SURF_CONCRETE
    int contacts = 0;
    for (int i = off; i < off + cnt; i++) {
        const float4 hb4 = C.hit_b[i];
        if (hb4.w == 0.0f) continue;
        const float4 ha = C.hit_a[i];
        const int2 pr = C.pairs[i];
        const int4 tr = C.tri[pr.y];
        Body& bn = bodies[info[pr.x].w];
        Body& bt = bodies[tr.w >> 8];
        // movable (world.cpp:2983-2993): a sleeping side is immovable and asks to wake when the other moves
        bool ma = true, mb = true;
        if (bn.sleeping) {
            if (sqrtf(bt.acc_v2) > smax(C.wake_speed, bt.sleep_speed) * 1.0f) bn.wake_request = 1;
            ma = false;
        }
        if (bt.sleeping) {
            if (sqrtf(bn.acc_v2) > smax(C.wake_speed, bn.sleep_speed) * 1.0f) bt.wake_request = 1;
            mb = false;
        }
        const int ia = pr.x, ib[3] = {tr.x, tr.y, tr.z};
        const float wb[3] = {ha.x, ha.y, ha.z};
        const v3 n = V(hb4.x, hb4.y, hb4.z);
        const float pen = ha.w;
        const float4 pa = nd[2 * ia], va4 = nd[2 * ia + 1];
        const v3 Av = V(va4.x, va4.y, va4.z);
        const float Aim = pa.w;
        v3 Bv[3];
        float Bim[3];
        for (int q = 0; q < 3; q++) {
            const float4 p = nd[2 * ib[q]], v = nd[2 * ib[q] + 1];
            Bv[q] = V(v.x, v.y, v.z), Bim[q] = p.w;
        }
        const float4 fa4 = Fs[ia];
        v3 FA = V(fa4.x, fa4.y, fa4.z);
        v3 FB[3];
        for (int q = 0; q < 3; q++) {
            const float4 f = Fs[ib[q]];
            FB[q] = V(f.x, f.y, f.z);
        }
        if (!(tr.w & TF_TWO_SIDED) && pen > bn.crad) {
            // hull_push_out<3> (world.cpp:97-118): behind a hull's face
            float W = ma ? Aim : 0.0f;
            if (mb)
                for (int q = 0; q < 3; q++) W += wb[q] * wb[q] * Bim[q];
            if (W <= 1e-12f) continue;
            v3 vb = V(0, 0, 0), acc = V(0, 0, 0);
            if (ma) acc = acc + FA * Aim;
            for (int q = 0; q < 3; q++) {
                vb = vb + Bv[q] * wb[q];
                if (mb) acc = acc - FB[q] * (wb[q] * Bim[q]);
            }
            const float m = 1.0f / W, vr = dot(Av - vb, n), target = smin(0.2f * pen / dt, 2.0f);
            const float fn = (target - vr) * m / dt - dot(acc, n) * m;
            if (fn > 0) {
                const v3 f = n * fn;
                if (ma) FA = FA + f;
                if (mb)
                    for (int q = 0; q < 3; q++) FB[q] = FB[q] - f * wb[q];
            }
        } else {
            // contact_force<1, 3> (world.cpp:59-92), the node's weight 1; a tyre node grips with its own friction
            // (world.cpp:3013)
            const int4 ina = info[ia];
            const float fric = ((uint32_t)ina.x & NF_TYRE) ? __int_as_float(ina.y) : 0.8f * smin(bn.cfric, bt.cfric);
            float W = 0;
            if (ma) W += 1.0f * 1.0f * Aim;
            if (mb)
                for (int q = 0; q < 3; q++) W += wb[q] * wb[q] * Bim[q];
            if (W <= 1e-12f) continue;
            const float m = 1.0f / W;
            v3 va = V(0, 0, 0), vb = V(0, 0, 0), acc = V(0, 0, 0);
            va = va + Av * 1.0f;
            if (ma) acc = acc + FA * (1.0f * Aim);
            for (int q = 0; q < 3; q++) {
                vb = vb + Bv[q] * wb[q];
                if (mb) acc = acc - FB[q] * (wb[q] * Bim[q]);
            }
            const v3 f_rel = acc * m;
            if (!ma) {
                const v3 f = primitive_collision(neg(f_rel), vb - va, m, neg(n), dt, gm, pen, fric, 2.0f, 0.0f, -1.0f);
                for (int q = 0; q < 3; q++) FB[q] = FB[q] + f * wb[q];
            } else {
                const v3 f = primitive_collision(f_rel, va - vb, m, n, dt, gm, pen, fric, 2.0f, 0.0f, -1.0f);
                FA = FA + f * 1.0f;
                if (mb)
                    for (int q = 0; q < 3; q++) FB[q] = FB[q] - f * wb[q];
            }
        }
        Fs[ia] = make_float4(FA.x, FA.y, FA.z, 0.0f);
        for (int q = 0; q < 3; q++) Fs[ib[q]] = make_float4(FB[q].x, FB[q].y, FB[q].z, 0.0f);
        contacts++;
        bn.body_contacts++;
        bt.body_contacts++;
    }
    C.isl_contacts[root] += contacts;
    if (contacts) atomicAdd(&C.counters[1], contacts);
}

} // namespace blg
