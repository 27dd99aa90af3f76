// rules.cuh — the reference's fix rules, separatrix checks and value update.
//
// The fix rules (fix_minimum :2554-2586, fix_saddle :2588-3037, fix_2saddle
// :3039-3983, fix_maximum :3985-4303, fix_as_vpath :5135-5244, fix_ds_vpath
// :5246-5295) are a case analysis over the reference's union-valued pairing
// arrays.  They are restated here branch for branch, including the
// reference's quirks.
//
// Cells are codes: anchor vertex * 32 + the cell's bit of FieldState::crit (0
// the vertex, 1..7 edges, 8..19 triangles, 20..25 tetrahedra), so a cell's
// vertices, its partner and the partner's kind come from the anchor's words
// and small tables in shared memory.  The reference tells the kinds apart by
// comparing ids of one dimension with the counts of another and testing the
// back pointer; for a consistent gradient that test succeeds for the partner's
// own kind only, so asking for the kind is the same.  Where a rule's result depends on an
// id's number (an id read as another dimension's), the number is computed and decoded
// as the reference does (tet_verts and so on, "literal" below).
//
// A chain of dependent loads with little arithmetic: bound by latency.  With
// cells as reference ids, every accessor decoded ids by 64-bit divisions (some
// hundred instructions each, fetched cold in every launch) and the rule context was copied
// to each thread's stack for the accessors that were called: a critical-point
// round took 82 us on average on a noisy 97 x 61 x 75 field and 78 us at 16^3,
// then 20 and 22 us (cold caches); 134 -> 54 us at 256^3.  What was left were the
// branches of a warp's cells one after the other and rescans by one thread: with a
// cell per warp as long as there are warps, and the rescans by the warp, a cell
// takes 4 to 6 k cycles of loads and at most 11 k (36 k before).
//
// A rule "lowers" a vertex: it asks for d_deltaBuffer[v] = get_delta(v).
// get_delta depends only on v's own value and counter, which no rule
// modifies, so the reference's atomic-max / store into the delta buffer is
// the same as set membership: a request bit per vertex (atomicOr) plus a list
// of newly requested vertices.  The value is computed once, when applied.
//
// Any index the reference would read or write outside its allocation is not
// performed; it sets bit 0 of the error word instead.
#pragma once
#include "gradient.cuh"

namespace dmtz {

enum { ERR_OOB = 1, ERR_WALK = 2 };

// code of rarely taken paths and of the wall searches, compiled once and called
#define DMTZ_SHARED_CODE __noinline__

struct RuleCtx {
    Grid g;
    FieldState P;      // original field gradient
    FieldState Q;      // decompressed field gradient
    const double *f;   // original values
    const double *gv;  // decompressed values (read-only during the rules)
    const int *cnt;    // delta_counter
    double bound;
    int edit_type;
    uint32_t *reqbits;  // request bit per vertex
    i64 *reqlist;       // newly requested vertices
    unsigned long long *reqn;
    i64 reqcap;
    int *err;
    unsigned long long *progress;  // set when an update changes a value or an edit counter
    double range;                  // max - min of the original field
};

// --------------------------------------------------------------- literal id arithmetic
// getVertexIDsFromEdgeID (main_3d.cu:1760-1900) for any id; (a > b)
__device__ DMTZ_SHARED_CODE void edge_verts(const Grid &g, i64 e, i64 &a, i64 &b) {
    const i64 W = g.W, H = g.H, D = g.D;
    int k = -1;
    for (int i = 0; i < 7; i++)
        if (e < g.eoff[i + 1]) {
            k = i;
            break;
        }
    if (k < 0) {
        a = b = -1;
        return;
    }
    const i64 r = e - g.eoff[k];
    i64 x = 0, y = 0, z = 0, x1 = 0, y1 = 0, z1 = 0;
    switch (k) {
    case 0: z = r / ((W - 1) * H); y = (r % ((W - 1) * H)) / (W - 1); x = r % (W - 1);
            x1 = x + 1; y1 = y; z1 = z; break;
    case 1: z = r / (W * (H - 1)); x = (r % (W * (H - 1))) / (H - 1); y = r % (H - 1);
            x1 = x; y1 = y + 1; z1 = z; break;
    case 2: y = r / (W * (D - 1)); x = (r % (W * (D - 1))) / (D - 1); z = r % (D - 1);
            x1 = x; y1 = y; z1 = z + 1; break;
    case 3: { i64 z2 = r / ((W - 1) * (H - 1)), y2 = (r % ((W - 1) * (H - 1))) / (W - 1), x2 = r % (W - 1);
              x = x2 + 1; y = y2; z = z2; x1 = x2; y1 = y2 + 1; z1 = z2; } break;
    case 4: { i64 x2 = r / ((H - 1) * (D - 1)), y2 = (r % ((H - 1) * (D - 1))) / (D - 1), z2 = r % (D - 1);
              x = x2; y = y2; z = z2; x1 = x2; y1 = y2 + 1; z1 = z2 + 1; } break;
    case 5: { i64 y2 = r / ((W - 1) * (D - 1)), z2 = (r % ((W - 1) * (D - 1))) / (W - 1), x2 = r % (W - 1);
              x = x2 + 1; y = y2; z = z2; x1 = x2; y1 = y2; z1 = z2 + 1; } break;
    default: { i64 z2 = r / ((W - 1) * (H - 1)), y2 = (r % ((W - 1) * (H - 1))) / (W - 1), x2 = r % (W - 1);
               x = x2 + 1; y = y2; z = z2; x1 = x2; y1 = y2 + 1; z1 = z2 + 1; } break;
    }
    i64 i1 = x + y * W + z * W * H, i2 = x1 + y1 * W + z1 * W * H;
    a = i1 > i2 ? i1 : i2;
    b = i1 > i2 ? i2 : i1;
}

__device__ __forceinline__ void sort_desc3(i64 &a, i64 &b, i64 &c) {
    i64 t;
    if (a < b) { t = a; a = b; b = t; }
    if (a < c) { t = a; a = c; c = t; }
    if (b < c) { t = b; b = c; c = t; }
}

// getVerticesFromTriangleID (main_3d.cu:425-565) for any id, sorted descending
__device__ DMTZ_SHARED_CODE void tri_verts(const Grid &g, i64 t, i64 &a, i64 &b, i64 &c) {
    const i64 W = g.W, H = g.H, D = g.D, WH = W * H;
    i64 v1 = 0, v2 = 0, v3 = 0, base, mx, my, mz;
    if (t < 2 * D * (W - 1) * (H - 1)) {
        base = t / 2; mz = base / ((W - 1) * (H - 1)); my = (base % ((W - 1) * (H - 1))) / (W - 1); mx = base % (W - 1);
        if (t % 2 == 0) { v1 = mx + my * W + mz * WH; v2 = mx + 1 + my * W + mz * WH; v3 = mx + (my + 1) * W + mz * WH; }
        else { v1 = mx + 1 + (my + 1) * W + mz * WH; v2 = mx + 1 + my * W + mz * WH; v3 = mx + (my + 1) * W + mz * WH; }
    } else if ((t -= 2 * D * (W - 1) * (H - 1)) < 2 * W * (H - 1) * (D - 1)) {
        base = t / 2; mx = base / ((H - 1) * (D - 1)); my = (base % ((H - 1) * (D - 1))) / (D - 1); mz = base % (D - 1);
        if (t % 2 == 0) { v1 = mx + my * W + mz * WH; v2 = mx + (my + 1) * W + mz * WH; v3 = mx + (my + 1) * W + (mz + 1) * WH; }
        else { v1 = mx + my * W + mz * WH; v2 = mx + my * W + (mz + 1) * WH; v3 = mx + (my + 1) * W + (mz + 1) * WH; }
    } else if ((t -= 2 * W * (H - 1) * (D - 1)) < 2 * H * (W - 1) * (D - 1)) {
        base = t / 2; my = base / ((W - 1) * (D - 1)); mz = (base % ((W - 1) * (D - 1))) / (W - 1); mx = base % (W - 1);
        if (t % 2 == 0) { v1 = mx + my * W + mz * WH; v2 = mx + 1 + my * W + mz * WH; v3 = mx + my * W + (mz + 1) * WH; }
        else { v1 = mx + 1 + my * W + mz * WH; v2 = mx + my * W + (mz + 1) * WH; v3 = mx + 1 + my * W + (mz + 1) * WH; }
    } else {
        t -= 2 * H * (W - 1) * (D - 1);
        base = t / 6; mz = base / ((W - 1) * (H - 1)); my = (base % ((W - 1) * (H - 1))) / (W - 1); mx = base % (W - 1);
        const i64 o = mx + my * W + mz * WH;
        switch (t % 6) {
        case 0: v1 = o; v2 = o + 1; v3 = o + W + WH; break;
        case 1: v1 = o + 1; v2 = o + W; v3 = o + W + WH; break;
        case 2: v1 = o + 1; v2 = o + 1 + W; v3 = o + W + WH; break;
        case 3: v1 = o + 1; v2 = o + WH; v3 = o + W + WH; break;
        case 4: v1 = o + 1; v2 = o + 1 + WH; v3 = o + W + WH; break;
        case 5: v1 = o + 1; v2 = o + W + WH; v3 = o + 1 + W + WH; break;
        default: break;  // negative remainder: the reference leaves the values untouched
        }
    }
    sort_desc3(v1, v2, v3);
    a = v1; b = v2; c = v3;
}

// getVerticesFromTetrahedraID (main_3d.cu:672-740) for any id, sorted descending
__device__ DMTZ_SHARED_CODE void tet_verts(const Grid &g, i64 t, i64 &a, i64 &b, i64 &c, i64 &d) {
    const i64 W = g.W, H = g.H, WH = W * H;
    const i64 base = t / 6;
    const i64 cz = base / ((W - 1) * (H - 1)), cy = (base % ((W - 1) * (H - 1))) / (W - 1), cx = base % (W - 1);
    const i64 o = cx + cy * W + cz * WH;
    i64 v[4] = {0, 0, 0, 0};
    switch (t % 6) {
    case 0: v[0] = o; v[1] = o + 1; v[2] = o + W; v[3] = o + W + WH; break;
    case 1: v[0] = o; v[1] = o + 1; v[2] = o + WH; v[3] = o + W + WH; break;
    case 2: v[0] = o + 1; v[1] = o + W; v[2] = o + 1 + W; v[3] = o + W + WH; break;
    case 3: v[0] = o + 1; v[1] = o + 1 + W; v[2] = o + W + WH; v[3] = o + 1 + W + WH; break;
    case 4: v[0] = o + 1; v[1] = o + WH; v[2] = o + 1 + WH; v[3] = o + W + WH; break;
    case 5: v[0] = o + 1; v[1] = o + 1 + WH; v[2] = o + W + WH; v[3] = o + 1 + W + WH; break;
    default: break;
    }
    // same compare-exchange network as the reference
    i64 tt;
    if (v[0] < v[1]) { tt = v[0]; v[0] = v[1]; v[1] = tt; }
    if (v[0] < v[2]) { tt = v[0]; v[0] = v[2]; v[2] = tt; }
    if (v[0] < v[3]) { tt = v[0]; v[0] = v[3]; v[3] = tt; }
    if (v[1] < v[2]) { tt = v[1]; v[1] = v[2]; v[2] = tt; }
    if (v[1] < v[3]) { tt = v[1]; v[1] = v[3]; v[3] = tt; }
    if (v[2] < v[3]) { tt = v[2]; v[2] = v[3]; v[3] = tt; }
    a = v[0]; b = v[1]; c = v[2]; d = v[3];
}

// --------------------------------------------------------------- pairing accessors
__device__ __forceinline__ i64 edge_ref_pair(const Grid &g, i64 a, i64 b) {
    // edge id of two adjacent vertices
    int ax, ay, az, bx, by, bz;
    decode_v(g, a, ax, ay, az);
    decode_v(g, b, bx, by, bz);
    const int x = min(ax, bx), y = min(ay, by), z = min(az, bz);
    const int ca = (ax - x) + 2 * (ay - y) + 4 * (az - z), cb = (bx - x) + 2 * (by - y) + 4 * (bz - z);
    int k = 0;
    for (int i = 0; i < 7; i++)
        if ((TOPO_EDGE_V[i][0] == ca && TOPO_EDGE_V[i][1] == cb) || (TOPO_EDGE_V[i][0] == cb && TOPO_EDGE_V[i][1] == ca))
            k = i;
    return edge_ref(g, x, y, z, k);
}

// paired_vertices[v]
__device__ DMTZ_SHARED_CODE i64 pv_ref(const RuleCtx &c, const FieldState &s, i64 v) {
    if (v < 0 || v >= c.g.V) {
        atomicOr(c.err, ERR_OOB);
        return -1;
    }
    const int d = s.pv[v];
    if (d == 15) return -1;
    return edge_ref_pair(c.g, v, v + c.g.doff[d]);
}
// paired_edges[e]
__device__ DMTZ_SHARED_CODE i64 pe_ref(const RuleCtx &c, const FieldState &s, i64 e) {
    if (e < 0 || e >= c.g.E) {
        atomicOr(c.err, ERR_OOB);
        return -1;
    }
    int x, y, z, k;
    edge_unref(c.g, e, x, y, z, k);
    const i64 a = x + (i64)y * c.g.W + (i64)z * c.g.WH;
    const int up = eup_get(s.eup[a], k);
    if (up) {
        const signed char *cf = TOPO_EDGE_COF[k][up - 1];
        return face_ref(c.g, x + cf[0], y + cf[1], z + cf[2], cf[3]);
    }
    const int cp = TOPO_EDGE_V[k][0], cq = TOPO_EDGE_V[k][1];
    const i64 p = a + c.g.coff[cp], q = a + c.g.coff[cq];
    if (s.pv[p] == TOPO_CORNER_DIR[cp][cq]) return p;
    if (s.pv[q] == TOPO_CORNER_DIR[cq][cp]) return q;
    return -1;
}
// paired_faces[t]
__device__ DMTZ_SHARED_CODE i64 pf_ref(const RuleCtx &c, const FieldState &s, i64 t) {
    if (t < 0 || t >= c.g.F) {
        atomicOr(c.err, ERR_OOB);
        return -1;
    }
    int x, y, z, sl;
    face_unref(c.g, t, x, y, z, sl);
    const i64 a = x + (i64)y * c.g.W + (i64)z * c.g.WH;
    const int up = fup_get(s.fup[a], sl);
    if (up) {
        const signed char *tc = TOPO_FACE_COF[sl][up - 1];
        return tet_ref(c.g, x + tc[0], y + tc[1], z + tc[2], tc[3]);
    }
    for (int j = 0; j < 3; j++) {
        const signed char *fe = TOPO_FACE_EDGE[sl][j];
        const i64 ea = a + fe[0] + (i64)fe[1] * c.g.W + (i64)fe[2] * c.g.WH;
        if (eup_get(s.eup[ea], fe[3]) == fe[4] + 1) return edge_ref(c.g, x + fe[0], y + fe[1], z + fe[2], fe[3]);
    }
    return -1;
}
// --------------------------------------------------------------- values, order, requests
__device__ __forceinline__ double fval(const RuleCtx &c, i64 v) {
    if (v < 0 || v >= c.g.V) {
        atomicOr(c.err, ERR_OOB);
        return 0.0;
    }
    return c.f[v];
}
__device__ __forceinline__ double gval(const RuleCtx &c, i64 v) {
    if (v < 0 || v >= c.g.V) {
        atomicOr(c.err, ERR_OOB);
        return 0.0;
    }
    return c.gv[v];
}
// compare_vertices(a, b, 0|1): (value, id) order
__device__ __forceinline__ bool above_f(const RuleCtx &c, i64 a, i64 b) {
    const uint64_t ka = okey(fval(c, a)), kb = okey(fval(c, b));
    return ka > kb || (ka == kb && a > b);
}
__device__ __forceinline__ bool above_g(const RuleCtx &c, i64 a, i64 b) {
    const uint64_t ka = okey(gval(c, a)), kb = okey(gval(c, b));
    return ka > kb || (ka == kb && a > b);
}
// get_delta (main_3d.cu:239-244)
__device__ __forceinline__ double get_delta(const RuleCtx &c, i64 v) {
    if (v < 0 || v >= c.g.V) {
        atomicOr(c.err, ERR_OOB);
        return 0.0;
    }
    if (c.edit_type == 1) return -ldexp(1.0, -c.cnt[v]) * c.bound;
    return __dmul_rn(__dsub_rn(__dsub_rn(c.f[v], c.bound), c.gv[v]), 0.5);  // x / 2, rounded the same
}
// The vertices that a rule lowers, at most four.  They are requested once the warp
// is back together: a rule's branches hold no atomics, and the atomics of several
// vertices do not wait for one another.  `rescan`: the two (edge) or three
// (triangle) vertices are lowered only if rescan_warp finds no neighbour to lower
// in their place.
struct Lowered {
    static constexpr i64 NONE = LLONG_MIN;
    i64 v[4] = {NONE, NONE, NONE, NONE};
    int rescan = 0;
    __device__ __forceinline__ void add(i64 w) {
        v[3] = v[2];
        v[2] = v[1];
        v[1] = v[0];
        v[0] = w;
    }
};
// components of the 14 neighbour directions, plus one, two bits each
__host__ __device__ constexpr uint32_t pack_dirs(int axis) {
    uint32_t w = 0;
    for (int i = 0; i < 14; i++) w |= (uint32_t)(cxt::TOPO_DIRS[i][axis] + 1) << (2 * i);
    return w;
}
// the directions as a set of (dx + 1) + 3 (dy + 1) + 9 (dz + 1)
__host__ __device__ constexpr uint32_t mask_dirs() {
    uint32_t m = 0;
    for (int i = 0; i < 14; i++)
        m |= 1u << ((cxt::TOPO_DIRS[i][0] + 1) + 3 * (cxt::TOPO_DIRS[i][1] + 1) + 9 * (cxt::TOPO_DIRS[i][2] + 1));
    return m;
}
__device__ __forceinline__ bool is_neighbour(int dx, int dy, int dz) {
    constexpr uint32_t M = mask_dirs();
    return (unsigned)(dx + 1) < 3u && (unsigned)(dy + 1) < 3u && (unsigned)(dz + 1) < 3u &&
           (M >> ((dx + 1) + 3 * (dy + 1) + 9 * (dz + 1)) & 1u);
}
// The rescans of a warp's rules.  Edge (v1, v2): argmin over the common neighbours n
// with exactly one of v1, v2 above n in the ORIGINAL field (the rescan of
// fix_saddle, main_3d.cu:2942-3015); triangle: argmin over those below exactly
// two of its vertices (get_smallest_vertex, main_3d.cu:2115-2194).  A neighbour per lane,
// two cells at a time: by one thread, a rescan took 10 k (edge) or 15 k cycles,
// where the rest of a rule takes 4 to 6 k.
__device__ __forceinline__ void rescan_warp(const RuleCtx &c, Lowered &o) {
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
    constexpr uint32_t X = pack_dirs(0), Y = pack_dirs(1), Z = pack_dirs(2);
    unsigned pending = __ballot_sync(full, o.rescan != 0);
    while (pending) {
        const int a = __ffs(pending) - 1;
        pending &= pending - 1;
        const int b = pending ? __ffs(pending) - 1 : a;
        pending &= pending - 1;  // 0 stays 0
        const int src = lane < 16 ? a : b, i = lane & 15;
        const int nv = __shfl_sync(full, o.rescan, src);
        const i64 v1 = __shfl_sync(full, o.v[0], src), v2 = __shfl_sync(full, o.v[1], src), v3 = __shfl_sync(full, o.v[2], src);
        uint64_t bk = ~0ull;
        i64 bid = LLONG_MAX;
        if (i < 14) {
            const int dx = (int)(X >> (2 * i) & 3u) - 1, dy = (int)(Y >> (2 * i) & 3u) - 1, dz = (int)(Z >> (2 * i) & 3u) - 1;
            int x, y, z, x2, y2, z2, x3 = 0, y3 = 0, z3 = 0;
            decode_v(c.g, v1, x, y, z);
            decode_v(c.g, v2, x2, y2, z2);
            if (nv == 3) decode_v(c.g, v3, x3, y3, z3);
            x += dx;
            y += dy;
            z += dz;
            if (inb(c.g, x, y, z) && is_neighbour(x - x2, y - y2, z - z2) &&
                (nv == 2 || is_neighbour(x - x3, y - y3, z - z3))) {
                const i64 n = x + (i64)y * c.g.W + (i64)z * c.g.WH;
                const uint64_t kn = okey(c.f[n]), k1 = okey(c.f[v1]), k2 = okey(c.f[v2]), k3 = nv == 3 ? okey(c.f[v3]) : 0;
                const int above = (k1 > kn || (k1 == kn && v1 > n)) + (k2 > kn || (k2 == kn && v2 > n)) +
                                  (nv == 3 && (k3 > kn || (k3 == kn && v3 > n)));
                // (the reference starts from DBL_MAX and INT_MAX)
                if (above == nv - 1 && (kn < DMTZ_KEY_DBL_MAX || (kn == DMTZ_KEY_DBL_MAX && n < INT_MAX))) {
                    bk = kn;
                    bid = n;
                }
            }
        }
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) {
            const uint64_t ok = __shfl_xor_sync(full, bk, s);
            const i64 oid = __shfl_xor_sync(full, bid, s);
            if (ok < bk || (ok == bk && oid < bid)) {
                bk = ok;
                bid = oid;
            }
        }
        const i64 ma = __shfl_sync(full, bid, 0), mb = __shfl_sync(full, bid, 16);
        const i64 m = (int)lane == a ? ma : mb;
        if (((int)lane == a || (int)lane == b) && m != LLONG_MAX) {
            o.v[0] = m;
            o.v[1] = o.v[2] = Lowered::NONE;
        }
    }
}
// every lane of a warp requests its vertices: one atomic per vertex, one per warp
__device__ __forceinline__ void request_warp(const RuleCtx &c, const Lowered &o) {
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
    bool fresh[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        fresh[k] = false;
        if (o.v[k] == Lowered::NONE) continue;
        if (o.v[k] < 0 || o.v[k] >= c.g.V) {
            atomicOr(c.err, ERR_OOB);
            continue;
        }
        const uint32_t bit = 1u << (o.v[k] & 31);
        fresh[k] = !(atomicOr(&c.reqbits[o.v[k] >> 5], bit) & bit);
    }
    unsigned m[4], total = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        m[k] = __ballot_sync(full, fresh[k]);
        total += __popc(m[k]);
    }
    if (!total) return;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(c.reqn, (unsigned long long)total);
    at = __shfl_sync(full, at, 0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned long long mine = at + __popc(m[k] & ((1u << lane) - 1u));
        if (fresh[k] && (i64)mine < c.reqcap) c.reqlist[mine] = o.v[k];
        at += __popc(m[k]);
    }
}
// "lower v": the reference's swap(v, get_delta(v))
__device__ __forceinline__ void lower(const RuleCtx &c, i64 v) {
    if (v < 0 || v >= c.g.V) {
        atomicOr(c.err, ERR_OOB);
        return;
    }
    const uint32_t bit = 1u << (v & 31);
    const uint32_t old = atomicOr(&c.reqbits[v >> 5], bit);
    if (!(old & bit)) {
        const unsigned long long k = agg_slot(c.reqn);
        if ((i64)k < c.reqcap) c.reqlist[k] = v;
    }
}
__device__ __forceinline__ i64 third_of(i64 a, i64 b, i64 cc, i64 v1, i64 v2) {
    i64 v3 = cc;
    if (a != v1 && a != v2) v3 = a;
    else if (b != v1 && b != v2) v3 = b;
    return v3;
}
__device__ __forceinline__ i64 fourth_of(i64 a, i64 b, i64 cc, i64 d, i64 v1, i64 v2, i64 v3) {
    i64 v4 = d;
    if (a != v1 && a != v2 && a != v3) v4 = a;
    else if (b != v1 && b != v2 && b != v3) v4 = b;
    else if (cc != v1 && cc != v2 && cc != v3) v4 = cc;
    return v4;
}
// --------------------------------------------------------------- cells as codes
// Tables of the code arithmetic.  Offsets are (dx+1) | (dy+1) << 2 | (dz+1) <<
// 4 (six bits), corners dx + 2 dy + 4 dz (three bits).
struct RuleTab {
    uint16_t edge[7];     // corners, higher id first: 3 bits each
    uint16_t face[12];    // three corners
    uint16_t tet[6];      // four corners
    uint16_t ecof[42];    // [family * 6 + i]: coface i: offset | slot << 6
    uint16_t fcof[24];    // [slot * 2 + i]: coface i: offset | slot << 6
    uint16_t fedge[36];   // [slot * 3 + j]: edge opposite corner j: offset | family << 6 | (coface index + 1) << 9
    uint16_t tface[24];   // [slot * 4 + j]: facet opposite corner j: offset | slot << 6
};
constexpr uint16_t tab_off(int x, int y, int z) { return (uint16_t)((x + 1) | ((y + 1) << 2) | ((z + 1) << 4)); }
constexpr RuleTab make_rule_tab() {
    RuleTab t = {};
    for (int k = 0; k < 7; k++) {
        t.edge[k] = (uint16_t)(cxt::TOPO_EDGE_V[k][0] | (cxt::TOPO_EDGE_V[k][1] << 3));
        for (int i = 0; i < cxt::TOPO_EDGE_NCOF[k]; i++) {
            const signed char *f = cxt::TOPO_EDGE_COF[k][i];
            t.ecof[k * 6 + i] = (uint16_t)(tab_off(f[0], f[1], f[2]) | (f[3] << 6));
        }
    }
    for (int s = 0; s < 12; s++) {
        for (int j = 0; j < 3; j++) {
            const signed char *e = cxt::TOPO_FACE_EDGE[s][j];
            t.face[s] |= (uint16_t)(cxt::TOPO_FACE_V[s][j] << (3 * j));
            t.fedge[s * 3 + j] = (uint16_t)(tab_off(e[0], e[1], e[2]) | (e[3] << 6) | ((e[4] + 1) << 9));
        }
        for (int i = 0; i < 2; i++) {
            const signed char *f = cxt::TOPO_FACE_COF[s][i];
            t.fcof[s * 2 + i] = (uint16_t)(tab_off(f[0], f[1], f[2]) | (f[3] << 6));
        }
    }
    for (int q = 0; q < 6; q++)
        for (int j = 0; j < 4; j++) {
            const signed char *f = cxt::TOPO_TET_FACE[q][j];
            t.tet[q] |= (uint16_t)(cxt::TOPO_TET_V[q][j] << (3 * j));
            t.tface[q * 4 + j] = (uint16_t)(tab_off(f[0], f[1], f[2]) | (f[3] << 6));
        }
    return t;
}
static __device__ const RuleTab kRuleTab = make_rule_tab();
// the tables into shared memory (every thread of the block calls this)
__device__ __forceinline__ void load_rule_tab(RuleTab &t) {
    const uint16_t *src = reinterpret_cast<const uint16_t *>(&kRuleTab);
    uint16_t *dst = reinterpret_cast<uint16_t *>(&t);
    for (int i = threadIdx.x; i < (int)(sizeof(RuleTab) / 2); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
}

enum { KIND_VERTEX = 0, KIND_EDGE, KIND_FACE, KIND_TET };
__host__ __device__ __forceinline__ i64 edge_code(i64 anchor, int k) { return anchor * 32 + 1 + k; }
__host__ __device__ __forceinline__ i64 face_code(i64 anchor, int s) { return anchor * 32 + 8 + s; }
__host__ __device__ __forceinline__ i64 tet_code(i64 anchor, int t) { return anchor * 32 + 20 + t; }
__host__ __device__ __forceinline__ int cell_kind(i64 code) {
    const int b = (int)(code & 31);
    return b == 0 ? KIND_VERTEX : b < 8 ? KIND_EDGE : b < 20 ? KIND_FACE : KIND_TET;
}
// reference id of a cell
__device__ __forceinline__ i64 code_ref(const Grid &g, i64 code) {
    const i64 v = code >> 5;
    const int b = (int)(code & 31);
    int x, y, z;
    decode_v(g, v, x, y, z);
    return b == 0 ? v : b < 8 ? edge_ref(g, x, y, z, b - 1) : b < 20 ? face_ref(g, x, y, z, b - 8) : tet_ref(g, x, y, z, b - 20);
}

struct Rules {
    const RuleCtx &c;
    const RuleTab &t;
    __device__ __forceinline__ i64 moved(i64 a, unsigned off) const {
        return a + ((int)(off & 3u) - 1) + ((int)((off >> 2) & 3u) - 1) * (i64)c.g.W + ((int)((off >> 4) & 3u) - 1) * c.g.WH;
    }
    __device__ __forceinline__ i64 corner(i64 a, unsigned c3) const {
        return a + (c3 & 1u) + ((c3 >> 1) & 1u) * (i64)c.g.W + ((c3 >> 2) & 1u) * c.g.WH;
    }
    // vertices, highest id first
    __device__ __forceinline__ void verts(i64 code, i64 &v1, i64 &v2) const {
        const unsigned m = t.edge[(code & 31) - 1];
        v1 = corner(code >> 5, m);
        v2 = corner(code >> 5, m >> 3);
    }
    __device__ __forceinline__ void verts(i64 code, i64 &v1, i64 &v2, i64 &v3) const {
        const unsigned m = t.face[(code & 31) - 8];
        v1 = corner(code >> 5, m);
        v2 = corner(code >> 5, m >> 3);
        v3 = corner(code >> 5, m >> 6);
    }
    __device__ __forceinline__ void verts(i64 code, i64 &v1, i64 &v2, i64 &v3, i64 &v4) const {
        const unsigned m = t.tet[(code & 31) - 20];
        v1 = corner(code >> 5, m);
        v2 = corner(code >> 5, m >> 3);
        v3 = corner(code >> 5, m >> 6);
        v4 = corner(code >> 5, m >> 9);
    }
    __device__ __forceinline__ i64 third(i64 face, i64 v1, i64 v2) const {
        i64 a, b, d;
        verts(face, a, b, d);
        return third_of(a, b, d, v1, v2);
    }
    __device__ __forceinline__ i64 fourth(i64 tet, i64 v1, i64 v2, i64 v3) const {
        i64 a, b, d, e;
        verts(tet, a, b, d, e);
        return fourth_of(a, b, d, e, v1, v2, v3);
    }
    // the other end of vertex v's paired edge, or -1
    __device__ __forceinline__ i64 below(const FieldState &s, i64 v) const {
        const int d = s.pv[v];
        return d == 15 ? -1 : v + c.g.doff[d];
    }
    // partners (code, or -1 for a critical cell)
    __device__ __forceinline__ i64 edge_partner(const FieldState &s, i64 e) const {
        const i64 a = e >> 5;
        const int k = (int)(e & 31) - 1, up = eup_get(s.eup[a], k);
        if (up) {
            const unsigned f = t.ecof[k * 6 + up - 1];
            return face_code(moved(a, f), (int)(f >> 6));
        }
        i64 p, q;
        verts(e, p, q);
        const int dp = s.pv[p], dq = s.pv[q];
        if (dp != 15 && p + c.g.doff[dp] == q) return cell_code(p, 0);
        if (dq != 15 && q + c.g.doff[dq] == p) return cell_code(q, 0);
        return -1;
    }
    __device__ __forceinline__ i64 face_partner(const FieldState &s, i64 f) const {
        const i64 a = f >> 5;
        const int sl = (int)(f & 31) - 8, up = fup_get(s.fup[a], sl);
        if (up) {
            const unsigned q = t.fcof[sl * 2 + up - 1];
            return tet_code(moved(a, q), (int)(q >> 6));
        }
        i64 r = -1;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const unsigned e = t.fedge[sl * 3 + j];
            const i64 ea = moved(a, e);
            const int k = (int)((e >> 6) & 7u);
            if (eup_get(s.eup[ea], k) == (int)(e >> 9)) r = edge_code(ea, k);
        }
        return r;
    }
    __device__ __forceinline__ i64 tet_partner(const FieldState &s, i64 q) const {
        const i64 a = q >> 5;
        const int ts = (int)(q & 31) - 20, j = (int)((s.tcode[a] >> (3 * ts)) & 7u);
        if (j == 7) return -1;
        const unsigned f = t.tface[ts * 4 + j];
        return face_code(moved(a, f), (int)(f >> 6));
    }
};

// --------------------------------------------------------------- A8 fix_minimum
__device__ __forceinline__ void rule_min(const Rules &R, i64 v, Lowered &o) {
    const i64 w = R.below(R.c.P, v >> 5);
    o.add(w >= 0 ? w : v >> 5);
}

// --------------------------------------------------------------- A9 fix_saddle
__device__ __forceinline__ void rule_saddle(const Rules &R, i64 id, Lowered &o) {
    const RuleCtx &c = R.c;
    i64 v1, v2;
    R.verts(id, v1, v2);
    const i64 pe = R.edge_partner(c.P, id);
    if (pe != -1 && cell_kind(pe) == KIND_VERTEX) {
        if (v2 == pe >> 5) v2 = v1;
        v1 = pe >> 5;
        const i64 false_v2 = R.below(c.Q, v1);
        if (false_v2 < 0) return;
        const double a = gval(c, v2), b = gval(c, false_v2);
        if (a > b || (a == b && v2 > false_v2)) o.add(v2);
        return;
    }
    const i64 qe = pe == -1 ? R.edge_partner(c.Q, id) : -1;
    if (pe == -1 && (qe == -1 || cell_kind(qe) == KIND_VERTEX)) {
        if (qe != -1) o.add(qe >> 5);
        return;
    }
    const i64 face = pe != -1 ? pe : qe;
    const i64 v3 = R.third(face, v1, v2);
    const bool g1 = above_g(c, v1, v3), g2 = above_g(c, v2, v3), f1 = above_f(c, v1, v3), f2 = above_f(c, v2, v3);
    if (pe != -1) {  // originally paired with this face
        if ((g1 && g2) || (f1 && f2)) {
            o.add(v3);
            return;
        }
        const i64 qf = R.face_partner(c.Q, face);
        if (qf != -1 && cell_kind(qf) == KIND_EDGE) {
            i64 w1, w2;
            R.verts(qf, w1, w2);
            const i64 false_v = (w1 != v1 && w1 != v2) ? w1 : w2;
            const i64 w3 = R.third(face, w1, w2);
            if (above_f(c, w2, w3) && above_f(c, w1, w3)) {
                const i64 pfe = R.edge_partner(c.P, qf);
                if (pfe != -1 && cell_kind(pfe) == KIND_FACE) {
                    o.add(R.third(pfe, w1, w2));
                    return;
                }
            }
            if (fabs(get_delta(c, false_v)) > 0) o.add(false_v);
        } else if (f1 && !g1) {
            o.add(g1 ? v1 : v3);
        } else {
            o.add(g2 ? v2 : v3);
        }
        return;
    }
    // originally critical, now paired with this face
    if (g1 == g2) {
        if (g2 != f2) o.add(v2);
        if (g1 != f1) o.add(v1);
    } else {
        o.add(v2);
        o.add(v1);
        o.rescan = 2;
    }
}

// --------------------------------------------------------------- A10 fix_2saddle
__device__ __forceinline__ void rule_2saddle(const Rules &R, i64 id, Lowered &o) {
    const RuleCtx &c = R.c;
    const Grid &G = c.g;
    const i64 pf = R.face_partner(c.P, id);
    if (pf != -1 && cell_kind(pf) == KIND_EDGE) {
        i64 v1, v2;
        R.verts(pf, v1, v2);
        const i64 v3 = R.third(id, v1, v2);
        const bool g1 = above_g(c, v2, v3), g2 = above_g(c, v1, v3), f1 = above_f(c, v2, v3), f2 = above_f(c, v1, v3);
        if (g1 && g2) {  // the edge's original face is this one
            o.add(v3);
        } else if (f1 != f2 && g1 != g2) {
            const i64 ff = R.edge_partner(c.Q, pf);
            i64 w = v3;
            if (ff != -1 && cell_kind(ff) == KIND_FACE) {
                const i64 u = R.third(ff, v1, v2);
                const bool h1 = above_f(c, v2, u), h2 = above_f(c, v1, u);
                if (above_g(c, v2, u) && above_g(c, v1, u) && h1 != h2) w = !h1 ? v2 : v1;
            }
            o.add(w);
        } else if (!g1 || !g2) {
            o.add(v3);
        }
        return;
    }
    if (pf != -1) {  // originally paired with a tetrahedron
        i64 v1, v2, v3;
        R.verts(id, v1, v2, v3);
        const i64 v4 = R.fourth(pf, v1, v2, v3);
        if (above_f(c, v3, v4) && above_f(c, v2, v4) && above_f(c, v1, v4)) {
            o.add(v4);
            return;
        }
        const i64 pff = R.tet_partner(c.Q, pf);
        if (pff == -1) {
            o.add(v4);
            return;
        }
        i64 u1, u2, u3;
        R.verts(pff, u1, u2, u3);
        const bool ga = above_g(c, u3, v4) && above_g(c, u2, v4) && above_g(c, u1, v4);
        const bool fa = above_f(c, u3, v4) && above_f(c, u2, v4) && above_f(c, u1, v4);
        if (ga || fa) {
            o.add(u1);
            o.add(u2);
            o.add(u3);
            return;
        }
        const i64 id2 = R.face_partner(c.P, pff);
        if (id2 == -1) return;
        if (cell_kind(id2) == KIND_EDGE) {
            i64 w1, w2;
            R.verts(id2, w1, w2);
            o.add(third_of(u1, u2, u3, w1, w2));
        } else {
            // as the reference has it: the fourth vertex is replaced by one of the
            // face's when an earlier one is not on the face
            i64 t1, t2, t3, t4;
            R.verts(id2, t1, t2, t3, t4);
            if (t1 != u1 && t1 != u2 && t1 != u3) t4 = u1;
            else if (t2 != u1 && t2 != u2 && t2 != u3) t4 = u2;
            else if (t3 != u1 && t3 != u2 && t3 != u3) t4 = u3;
            o.add(t1);
            o.add(t2);
            o.add(t3);
            o.add(t4);
        }
        return;
    }
    const i64 qf = R.face_partner(c.Q, id);
    if (qf == -1) return;
    if (cell_kind(qf) == KIND_EDGE) {
        i64 v1, v2;
        R.verts(qf, v1, v2);
        const i64 tf = R.edge_partner(c.P, qf);
        if (tf == -1) return;
        if (cell_kind(tf) == KIND_FACE) {
            o.add(R.third(tf, v1, v2));
        } else {
            o.add(v1);
            o.add(v2);
        }
        return;
    }
    i64 v1, v2, v3;
    R.verts(id, v1, v2, v3);
    const i64 v4 = R.fourth(qf, v1, v2, v3);
    const bool g1 = above_g(c, v3, v4), g2 = above_g(c, v2, v4), g3 = above_g(c, v1, v4);
    const bool f1 = above_f(c, v3, v4), f2 = above_f(c, v2, v4), f3 = above_f(c, v1, v4);
    if (g1 && g2 && g3) {
        if (!f1) o.add(v3);
        else if (!f2) o.add(v2);
        else if (!f3) o.add(v1);
        return;
    }
    // the reference compares this face id with the number of tetrahedra
    const i64 true_cell = R.tet_partner(c.P, qf);
    o.add(v3);
    o.add(v2);
    o.add(v1);
    if (!(true_cell != -1 && code_ref(G, true_cell) < G.T)) o.rescan = 3;
}

// --------------------------------------------------------------- A11 fix_maximum
// the reference reads an edge id as a tetrahedron's: its vertex that is none of v1, v2, v3
__device__ DMTZ_SHARED_CODE i64 literal_fourth(const Grid &G, i64 id, i64 v1, i64 v2, i64 v3, int *err) {
    if (id < 0 || id >= G.T) atomicOr(err, ERR_OOB);
    i64 p, q, r, w;
    tet_verts(G, id, p, q, r, w);
    return fourth_of(p, q, r, w, v1, v2, v3);
}
__device__ __forceinline__ void rule_max(const Rules &R, i64 id, Lowered &o) {
    const RuleCtx &c = R.c;
    const i64 pt = R.tet_partner(c.P, id);
    const i64 face = pt != -1 ? pt : R.tet_partner(c.Q, id);
    if (face == -1) return;  // critical in both: not listed
    i64 v1, v2, v3;
    R.verts(face, v1, v2, v3);
    const i64 v4 = R.fourth(id, v1, v2, v3);
    const bool f1 = above_f(c, v1, v4), f2 = above_f(c, v2, v4), f3 = above_f(c, v3, v4);
    if (pt != -1) {
        if (f1 && f2 && f3) {
            o.add(v4);
            return;
        }
        const i64 fc = R.face_partner(c.Q, face);
        if (fc == -1) return;
        i64 w = v4;
        if (cell_kind(fc) == KIND_EDGE) {
            i64 e1, e2;
            R.verts(fc, e1, e2);
            w = above_g(c, e1, e2) ? e1 : e2;
        }
        o.add(w);
        return;
    }
    const bool g1 = above_g(c, v1, v4), g2 = above_g(c, v2, v4), g3 = above_g(c, v3, v4);
    if (g1 && g2 && g3) {
        if (!f1) o.add(v1);
        if (!f2) o.add(v2);
        if (!f3) o.add(v3);
        if (f1 && f2 && f3) {
            const i64 it = R.face_partner(c.P, face);
            if (it != -1)
                o.add(cell_kind(it) == KIND_TET ? R.fourth(it, v1, v2, v3)
                                                   : literal_fourth(c.g, code_ref(c.g, it), v1, v2, v3, c.err));
        }
        return;
    }
    const i64 pid = R.face_partner(c.P, face);
    if (pid == -1) {
        if (!f1) o.add(v1);
        if (!f2) o.add(v2);
        if (!f3) o.add(v3);
    } else if (cell_kind(pid) == KIND_EDGE) {
        i64 e1, e2;
        R.verts(pid, e1, e2);
        o.add(e1);
        o.add(e2);
    } else {
        i64 p, q, r, w;
        R.verts(pid, p, q, r, w);
        o.add(p);
        o.add(q);
        o.add(r);
        o.add(w);
    }
}

// --------------------------------------------------------------- A15 fix_as_vpath (type 2)
__device__ __forceinline__ void rule_as_path(const Rules &R, i64 tet, Lowered &o) {
    const RuleCtx &c = R.c;
    const i64 tf = R.tet_partner(c.P, tet), ff = R.tet_partner(c.Q, tet);
    i64 v1, v2, v3, a = -1, b = -1, tv3 = -1;
    if (ff == -1) {  // the reference reads its arrays at -1 here
        atomicOr(c.err, ERR_OOB);
        tri_verts(c.g, -1, a, b, tv3);
    } else {
        R.verts(ff, a, b, tv3);
        const i64 pfe = R.face_partner(c.P, ff);
        if (pfe != -1 && cell_kind(pfe) == KIND_TET) {
            o.add(R.fourth(pfe, a, b, tv3));
            return;
        }
    }
    if (tf == -1) tri_verts(c.g, -1, v1, v2, v3);
    else R.verts(tf, v1, v2, v3);
    o.add(fourth_of(a, b, tv3, tv3, v1, v2, v3));
}
// A14 fix_ds_vpath (type 0)
__device__ DMTZ_SHARED_CODE i64 literal_ds_path(const RuleCtx &c, i64 v) {
    const i64 tpe = pv_ref(c, c.P, v);
    i64 v1, v2;
    edge_verts(c.g, tpe, v1, v2);
    return v == v1 ? v2 : v1;
}
__device__ __forceinline__ void rule_ds_path(const Rules &R, i64 v, Lowered &o) {
    const i64 w = v >= 0 && v < R.c.g.V ? R.below(R.c.P, v) : -1;
    o.add(w >= 0 ? w : literal_ds_path(R.c, v));  // literal: no vertex (-1), or a critical one
}

// fix_ds_wall (main_3d.cu:5297-5413) for the wall record edge e: the edge's
// original and decompressed pairings differ
__device__ inline void rule_ds_wall(const RuleCtx &c, i64 e) {
    const Grid &G = c.g;
    const i64 tf = pe_ref(c, c.P, e), ff = pe_ref(c, c.Q, e);
    if (tf == ff) return;
    i64 v1, v2;
    edge_verts(G, e, v1, v2);
    if (tf >= 0 && ff >= 0 && tf < G.F && pf_ref(c, c.P, tf) == e && ff < G.F && pf_ref(c, c.Q, ff) == e) {
        // both pair the edge with a face: lower the original face's third vertex,
        // or both endpoints when that vertex has no room left
        i64 a, b, v3;
        tri_verts(G, tf, a, b, v3);
        if (a != v1 && a != v2) v3 = a;
        if (b != v1 && b != v2) v3 = b;
        if (fabs(get_delta(c, v3)) > 1e-16 * c.range) {
            lower(c, v3);
        } else {
            lower(c, v1);
            lower(c, v2);
        }
    } else if (tf == -1 || tf >= G.F || (tf >= 0 && pf_ref(c, c.P, tf) != e)) {
        lower(c, v1);
        lower(c, v2);
    } else if (ff == -1 || ff >= G.F || (ff >= 0 && pf_ref(c, c.Q, ff) != e)) {
        i64 a, b, v3;
        tri_verts(G, tf, a, b, v3);
        lower(c, third_of(a, b, v3, v1, v2));
    }
}

}  // namespace dmtz
