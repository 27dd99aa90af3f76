// dmtz.cu — kernels and host driver of libdmtz (see include/dmtz.h).
//
// Data layout in HBM, per field (original f, decompressed g), one entry per
// anchor vertex, structure of arrays:
//   pv u8 | eup u32 | fup u32 | crit u32 | tcode u32
// plus, shared: f, g (float64), delta_counter (int32), request bits (1 bit per
// vertex), the request list and the four mismatch lists (cell ids, int64).
//
// One correction round (main_3d.cu:6789-6921) is: fix rules on the mismatch
// lists -> request bits/list; apply (bounded update of g); the gradient of g
// around the requests; mismatch compaction.  Counters live on the device; the
// host reads four words per round (or none, in the CUDA-graph loop).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <atomic>
#include <mutex>
#include <thread>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/dmtz.h"
#include "alloc_retry.cuh"
#include "cnn.cuh"
#include "dmtz_common.cuh"
#include "gradient.cuh"
#include "record_sort.h"
#include "report_wait.cuh"
#include "rules.cuh"

using namespace dmtz;

namespace dmtz {

static const int kBlock = 256;
static inline unsigned grid_for(i64 n) { return (unsigned)std::max<i64>(1, (n + kBlock - 1) / kBlock); }

// --------------------------------------------------------------- mismatch compaction
// A kernel launched so starts while the one before it on the stream still runs, up
// to its own after_previous(); the one before must let it (let_next).  The
// kernels of a round are short, so their launches show: a host-driven loop over the
// extrema of a 64^3 Gaussian mixture (uniform noise of 1e-3, seed 1) takes 10.3 ms so
// and 10.8 ms without.  Not while a graph is captured: inside a loop graph's conditional
// nodes such an edge costs what it hides (97 x 61 x 75, noise of 1e-2, seed 1: 13.6 ms both).
template <typename... P, typename... A>
static void launch_next(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t st, A &&...args) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &capture);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

// mismatch between the decompressed and the original critical cells
// (get_false_minimum / saddle / 2_saddle / maximum, main_3d.cu:2492-2550):
// a scan of the two criticality masks, compacting mismatched cells' ids
__global__ void __launch_bounds__(kBlock) k_mismatch_scan(Grid g, const uint32_t *crit_d, const uint32_t *crit_o, Lists L,
                                                         int want_saddles) {
    const i64 step = (i64)gridDim.x * blockDim.x;
    for (i64 b = (i64)blockIdx.x * blockDim.x; b < g.V; b += step) {  // the block's warps stay whole
        const i64 v = b + threadIdx.x;
        uint32_t d = v < g.V ? crit_d[v] ^ crit_o[v] : 0u;
        if (!want_saddles) d &= 1u | (0x3Fu << 20);
        push_warp(L, v, d);
    }
}

// Dirty bricks.  A cell's pairing depends on the star of its highest vertex,
// so a changed value reaches the cells whose highest vertex is the changed one
// or a neighbour of it: anchors 2 below to 1 above per axis.  Every brick with
// such an anchor is marked (one byte per brick, four to a word) and listed by
// whoever marks it first; the marks stay until the round's end, where the list
// says which ones to clear.  (A kernel that made the list from the marks took 5 of
// a short round's 45 us.)
constexpr int kReachLow = 2, kReachHigh = 1;
struct BrickMarks {
    uint32_t *flags;  // nullptr: not kept
    uint32_t *list;   // packed brick coordinates
    unsigned long long *n;
    int nbx, nby, shx, shy, shz;
    int lanes;   // per vertex: 8 where the reach spans at most two bricks per axis, else 32 (three)
    i64 sample;  // 0: every updated vertex marks; else about so many of them, blocks of bricks (sampled_marks)
};
// Every lane of a warp takes part: lane j of a vertex's lanes has the j-th brick of
// its reach, so that the marks, and then the list's slots, wait for memory once.
__device__ __forceinline__ void mark_dirty(const Grid &g, const BrickMarks &B, bool on, i64 v, int j) {
    uint32_t entry = 0;
    bool first = false;
    if (on) {
        int x, y, z;
        decode_v(g, v, x, y, z);
        const int span = B.lanes == 8 ? 2 : 3;
        const int bx = (max(x - kReachLow, 0) >> B.shx) + j % span, by = (max(y - kReachLow, 0) >> B.shy) + (j / span) % span,
                  bz = (max(z - kReachLow, 0) >> B.shz) + j / (span * span);
        if (bx <= min(x + kReachHigh, g.W - 1) >> B.shx && by <= min(y + kReachHigh, g.H - 1) >> B.shy &&
            bz <= min(z + kReachHigh, g.D - 1) >> B.shz) {
            const i64 b = bx + (i64)B.nbx * (by + (i64)B.nby * bz);
            const uint32_t bit = 1u << (8 * (int)(b & 3));
            if (!(__ldcg(B.flags + (b >> 2)) & bit)) first = !(atomicOr(B.flags + (b >> 2), bit) & bit);
            entry = (uint32_t)bx | ((uint32_t)by << 11) | ((uint32_t)bz << 22);
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, first), lane = threadIdx.x & 31u;
    if (!m) return;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(B.n, (unsigned long long)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (first) B.list[at + __popc(m & ((1u << lane) - 1u))] = entry;
}
__global__ void __launch_bounds__(kBlock) k_mark_dirty(Grid g, BrickMarks B, const i64 *verts, const unsigned long long *nverts) {
    const i64 n = (i64)*nverts;
    const int lane = threadIdx.x & 31, per = 32 / B.lanes, j = lane % B.lanes;
    const i64 step = (i64)gridDim.x * (kBlock / 32) * per;
    for (i64 b = ((i64)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * per; b < n; b += step) {
        const i64 i = b + lane / B.lanes;
        mark_dirty(g, B, i < n, i < n ? verts[i] : 0, j);
    }
}

// --------------------------------------------------------------- export to the reference layout
__global__ void k_export(Grid g, FieldState s, int32_t *PV, int32_t *PE, int32_t *PF, int32_t *PT) {
    i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= g.V) return;
    int x, y, z;
    decode_v(g, v, x, y, z);
    const int d = s.pv[v];
    PV[v] = d == 15 ? -1 : (int32_t)edge_ref_pair(g, v, v + g.doff[d]);
    const uint32_t eu = s.eup[v];
    for (int k = 0; k < 7; k++) {
        int mx, my, mz;
        edge_extent(k, mx, my, mz);
        if (!cell_ok(g, x, y, z, mx, my, mz)) continue;
        i64 val = -1;
        const int up = eup_get(eu, k);
        if (up) {
            const signed char *cf = TOPO_EDGE_COF[k][up - 1];
            val = face_ref(g, x + cf[0], y + cf[1], z + cf[2], cf[3]);
        } else {
            const int cp = TOPO_EDGE_V[k][0], cq = TOPO_EDGE_V[k][1];
            const i64 p = v + g.coff[cp], q = v + g.coff[cq];
            if (s.pv[p] == TOPO_CORNER_DIR[cp][cq]) val = p;
            else if (s.pv[q] == TOPO_CORNER_DIR[cq][cp]) val = q;
        }
        PE[edge_ref(g, x, y, z, k)] = (int32_t)val;
    }
    const uint32_t fu = s.fup[v];
    for (int sl = 0; sl < 12; sl++) {
        int mx, my, mz;
        face_extent(sl, mx, my, mz);
        if (!cell_ok(g, x, y, z, mx, my, mz)) continue;
        i64 val = -1;
        const int up = fup_get(fu, sl);
        if (up) {
            const signed char *tc = TOPO_FACE_COF[sl][up - 1];
            val = tet_ref(g, x + tc[0], y + tc[1], z + tc[2], tc[3]);
        } else {
            for (int j = 0; j < 3; j++) {
                const signed char *fe = TOPO_FACE_EDGE[sl][j];
                const i64 ea = v + fe[0] + (i64)fe[1] * g.W + (i64)fe[2] * g.WH;
                if (eup_get(s.eup[ea], fe[3]) == fe[4] + 1) val = edge_ref(g, x + fe[0], y + fe[1], z + fe[2], fe[3]);
            }
        }
        PF[face_ref(g, x, y, z, sl)] = (int32_t)val;
    }
    if (cell_ok(g, x, y, z, 1, 1, 1)) {
        for (int ts = 0; ts < 6; ts++) {
            i64 val = -1;
            for (int j = 0; j < 4; j++) {
                const signed char *tf = TOPO_TET_FACE[ts][j];
                const i64 fa = v + tf[0] + (i64)tf[1] * g.W + (i64)tf[2] * g.WH;
                if (fup_get(s.fup[fa], tf[3]) == tf[4] + 1) val = face_ref(g, x + tf[0], y + tf[1], z + tf[2], tf[3]);
            }
            PT[tet_ref(g, x, y, z, ts)] = (int32_t)val;
        }
    }
}

// Reference ids in place of cell codes, in a list for the host.  (Decoded there, a code
// took several 64-bit divisions.)
__global__ void __launch_bounds__(kBlock) k_refs(Grid g, i64 *codes, i64 n) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) codes[i] = code_ref(g, codes[i]);
}

// --------------------------------------------------------------- fix rules
struct CpLists {
    const i64 *l[4];
    const unsigned long long *n;
    i64 cap[4];
};

// Cells per warp for n cells (a power of two).  The cells of a warp take different
// branches of a rule, each a chain of loads, one after the other, so as long as
// there are warps to spare a warp takes few cells.
__device__ __forceinline__ int cells_per_warp(i64 n, i64 warps) {
    int c = 1;
    while (c < 32 && n > c * warps) c *= 2;
    return c;
}
// 256-thread blocks of the rules run three to an SM, and the grid is eight blocks per SM
__device__ __forceinline__ i64 rule_warps() { return (i64)gridDim.x * 3; }

// fix_minimum, [fix_saddle, fix_2saddle], fix_maximum over the current lists
// (the host never runs this on an overflowed list; the clamp only keeps
// every read inside the allocation).  The four lists are taken one behind the
// other, each padded to whole warps, so that a warp runs one rule: short
// lists run side by side in different warps, and in long ones (the first
// rounds of noisy fields: millions of cells) all warps of the GPU are in the
// same rule's code.  The rules only set request bits, so the order does not
// matter.  By `blocks` blocks of which this is number `block`; the table is loaded
// unless it is there (all threads of the block).
__device__ __forceinline__ void fix_cells(const RuleCtx &c, const CpLists &L, int preserve_saddles, RuleTab &tab, bool loaded,
                                          unsigned block, unsigned blocks, i64 spare) {
    const i64 n0 = min((i64)L.n[0], L.cap[0]), n1 = preserve_saddles ? min((i64)L.n[1], L.cap[1]) : 0,
              n2 = preserve_saddles ? min((i64)L.n[2], L.cap[2]) : 0, n3 = min((i64)L.n[3], L.cap[3]);
    const int per = cells_per_warp(n0 + n1 + n2 + n3, spare), lane = threadIdx.x & 31;
    auto warps = [&](i64 n) { return (n + per - 1) / per; };
    const i64 w0 = warps(n0), w1 = w0 + warps(n1), w2 = w1 + warps(n2), w3 = w2 + warps(n3);
    const unsigned NW = blockDim.x / 32;
    if ((i64)block * NW >= w3) return;
    if (!loaded) load_rule_tab(tab);
    const Rules R{c, tab};
    for (i64 w = (i64)block * NW + (threadIdx.x >> 5); w < w3; w += (i64)blocks * NW) {
        Lowered o;
        const int k = w < w0 ? 0 : w < w1 ? 1 : w < w2 ? 2 : 3;
        const i64 i = (w - (k == 0 ? 0 : k == 1 ? w0 : k == 2 ? w1 : w2)) * per + lane;
        if (lane < per && i < (k == 0 ? n0 : k == 1 ? n1 : k == 2 ? n2 : n3)) {
            const i64 code = L.l[k][i];
            if (k == 0) rule_min(R, code, o);
            else if (k == 1) rule_saddle(R, code, o);
            else if (k == 2) rule_2saddle(R, code, o);
            else rule_max(R, code, o);
        }
        __syncwarp();
        rescan_warp(c, o);
        request_warp(c, o);
    }
}
__global__ void __launch_bounds__(kBlock) k_fix_cp(const __grid_constant__ RuleCtx c, const __grid_constant__ CpLists L, int preserve_saddles) {
    __shared__ RuleTab tab;
    let_next();
    fix_cells(c, L, preserve_saddles, tab, false, blockIdx.x, gridDim.x, rule_warps());
}

// separatrix records
struct PathRec {
    i64 *as_tet, *as_cur, *ds_edge, *ds_vert;  // cell codes; ds_vert: the vertex (-1: none)
    unsigned long long *n;  // [0] ascending, [1] descending
    i64 cap_as, cap_ds;     // at most one record per original 2-saddle / 1-saddle
};

// Ascending paths (is_false, main_3d.cu:4437-4497) step from a tetrahedron
// through the facet it is paired with to that facet's other coface
// (get_cell_tetra's other one; none = the path leaves the grid).  That coface
// lies in the same cube or in the one across a face, so a step is one byte per
// (slot, facet): direction (0 none, 1 +x, 2 -x, 3 +y, 4 -y, 5 +z, 6 -z) * 8 +
// new slot.  The reference's back-pointer test on the way is always true for a
// consistent gradient.
struct AscTab {
    uint8_t next[24];  // [slot * 4 + facet]
};
constexpr AscTab make_asc_tab() {
    AscTab t = {};
    for (int s = 0; s < 6; s++)
        for (int j = 0; j < 4; j++) {
            const signed char *f = cxt::TOPO_TET_FACE[s][j], *c = cxt::TOPO_FACE_COF[f[3]][1 - f[4]];
            const int dx = f[0] + c[0], dy = f[1] + c[1], dz = f[2] + c[2];
            const int o = dx ? (dx > 0 ? 1 : 2) : dy ? (dy > 0 ? 3 : 4) : dz ? (dz > 0 ? 5 : 6) : 0;
            t.next[s * 4 + j] = (uint8_t)(o * 8 + c[3]);
        }
    return t;
}
constexpr bool asc_steps_are_axial() {
    for (int s = 0; s < 6; s++)
        for (int j = 0; j < 4; j++) {
            const signed char *f = cxt::TOPO_TET_FACE[s][j], *c = cxt::TOPO_FACE_COF[f[3]][1 - f[4]];
            const int dx = f[0] + c[0], dy = f[1] + c[1], dz = f[2] + c[2];
            if (dx * dx + dy * dy + dz * dz > 1) return false;
        }
    return true;
}
static_assert(asc_steps_are_axial(), "a facet's cofaces lie in one cube or in two that share a face");
static __device__ const AscTab kAscTab = make_asc_tab();
// the table into shared memory (every thread of the block calls this)
__device__ __forceinline__ void load_asc_tab(AscTab &t) {
    if (threadIdx.x < 24) t.next[threadIdx.x] = kAscTab.next[threadIdx.x];
    __syncthreads();
}
// one step from (x, y, z, s) with facet j (0..3); false: the path leaves the grid
__device__ __forceinline__ bool asc_move(const Grid &g, const AscTab &t, int &x, int &y, int &z, int &s, int j) {
    const int e = t.next[s * 4 + j], o = e >> 3;
    x += (o == 1) - (o == 2);
    y += (o == 3) - (o == 4);
    z += (o == 5) - (o == 6);
    s = e & 7;
    return (unsigned)x < (unsigned)(g.W - 1) && (unsigned)y < (unsigned)(g.H - 1) && (unsigned)z < (unsigned)(g.D - 1);
}

// compact list of original critical cells of one dimension: criticality
// bits FIRST .. FIRST+SLOTS-1 of an anchor (SLOTS cells per anchor), entry =
// anchor * SLOTS + slot.  The 2-saddle triangles: <8, 12>; the 1-saddle
// edges: <1, 7>.
template <int FIRST, int SLOTS>
__global__ void k_crit_list(Grid g, const uint32_t *critP, i64 *list, i64 cap, unsigned long long *n) {
    // a block takes kBlock x 8 consecutive anchors per step: each thread
    // counts its 8 anchors' 2-saddles, a block scan places them in anchor
    // order, and one atomic per block step reserves the block's range (one
    // atomic per warp over the whole grid serialised this kernel on the
    // counter)
    __shared__ unsigned wtot[kBlock / 32];
    __shared__ unsigned long long bbase;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, full = 0xffffffffu;
    const i64 per = (i64)kBlock * 8;
    for (i64 b0 = (i64)blockIdx.x * per; b0 < g.V; b0 += (i64)gridDim.x * per) {
        const i64 v0 = b0 + (i64)threadIdx.x * 8;
        uint32_t m[8];
        unsigned mine = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            m[j] = v0 + j < g.V ? (critP[v0 + j] >> FIRST) & ((1u << SLOTS) - 1u) : 0u;
            mine += __popc(m[j]);
        }
        unsigned incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned y = __shfl_up_sync(full, incl, off);
            if (lane >= (unsigned)off) incl += y;
        }
        if (lane == 31) wtot[warp] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t = 0;
            for (int w = 0; w < kBlock / 32; w++) {
                const unsigned c = wtot[w];
                wtot[w] = (unsigned)t;
                t += c;
            }
            bbase = t ? atomicAdd(n, t) : 0ull;
        }
        __syncthreads();
        unsigned long long at = bbase + wtot[warp] + incl - mine;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            uint32_t mm = m[j];
            while (mm) {
                const int sl = __ffs(mm) - 1;
                mm &= mm - 1;
                if ((i64)at < cap) list[at] = (v0 + j) * SLOTS + sl;
                at++;
            }
        }
        __syncthreads();  // wtot and bbase are reused by the next step
    }
}

// numbers of original 1-saddle edges (out[0]) and 2-saddle triangles (out[1])
__global__ void k_count_saddles(i64 V, const uint32_t *critP, unsigned long long *out) {
    unsigned long long a = 0, b = 0;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (i64)gridDim.x * blockDim.x) {
        const uint32_t m = critP[v];
        a += __popc((m >> 1) & 0x7Fu);
        b += __popc((m >> 8) & 0xFFFu);
    }
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(&out[0], a);
        if (b) atomicAdd(&out[1], b);
    }
}

// ------------------------------------------------------------------- walls
// preserve_connectors = 1: get_false_ds_wall (main_3d.cu:5064-5121) restated
// without its races.  Every original 2-saddle face runs its own depth-first
// search over the faces reachable by original V-paths, in the reference's
// order: pop a face; if it was not visited, take its edges (v1 v2), (v1 v3),
// (v2 v3) of its descending vertex triple; skip an originally critical edge;
// the first edge whose original and decompressed pairings differ is the
// record; otherwise push the face the edge is originally paired with (when
// it is a face and not this one).
//
// Visited marks are a direct-mapped cache of face ids.  A face found there was
// visited and is skipped; a visited face that fell out of the cache is
// searched again, which never changes the record: V-paths have no cycles and
// the stack finishes a face's descendants before the entries below it, so
// every face reachable from a visited face was visited before it comes back,
// and a repeat only re-checks edges that passed and pushes visited faces.  The
// cache size bounds only the work.  A search that passes its pop limit or
// outgrows its stack is handed to the next tier (larger stack, cache and pop
// limit in device scratch memory); the record does not depend on the tier.
struct WallRec {
    i64 *sad, *edge;        // record: 2-saddle face, first differing edge of its wall
    unsigned long long *n;
    i64 cap;
};
constexpr int kWallStack1 = 24, kWallCacheBits1 = 6;
constexpr long long kWallPops1 = 1024;

__device__ __forceinline__ unsigned wall_slot(i64 t, int bits) {
    return (unsigned)(((unsigned long long)t * 0x9E3779B97F4A7C15ull) >> (64 - bits));
}
// 0: no differing edge, 1: record in rec, 2: stack or pop limit reached
__device__ int wall_dfs(const RuleCtx &c, i64 sad, i64 *stack, int stack_cap, i64 *cache, int cache_bits,
                        long long pop_cap, i64 &rec) {
    const Grid &G = c.g;
    int top = 0;
    stack[top++] = sad;
    long long pops = 0;
    while (top > 0) {
        const i64 t = stack[--top];
        if (++pops > pop_cap) return 2;
        const unsigned slot = wall_slot(t, cache_bits);
        if (cache[slot] == t) continue;
        cache[slot] = t;
        i64 v1, v2, v3;
        tri_verts(G, t, v1, v2, v3);
        const i64 es[3] = {edge_ref_pair(G, v1, v2), edge_ref_pair(G, v1, v3), edge_ref_pair(G, v2, v3)};
        for (int k = 0; k < 3; k++) {
            const i64 j = es[k];
            const i64 pe = pe_ref(c, c.P, j);
            if (pe == -1) continue;
            if (pe != pe_ref(c, c.Q, j)) {
                rec = j;
                return 1;
            }
            if (pe != t && pe >= 0 && pe < G.F && pf_ref(c, c.P, pe) == j) {
                if (top == stack_cap) return 2;
                stack[top++] = pe;
            }
        }
    }
    return 0;
}
__device__ __forceinline__ void wall_emit(const WallRec &W, i64 s, i64 e) {
    const unsigned long long k = atomicAdd(W.n, 1ull);
    if ((i64)k < W.cap) {
        W.sad[k] = s;
        W.edge[k] = e;
    }
}
__device__ __forceinline__ void wall_defer(i64 *list, unsigned long long *n, i64 cap, i64 s) {
    const unsigned long long k = atomicAdd(n, 1ull);
    if ((i64)k < cap) list[k] = s;
}
// first tier: every original 2-saddle (sad2 codes anchor * 12 + slot), stack
// and cache in per-thread local memory
__global__ void k_wall_t1(const __grid_constant__ RuleCtx c, const i64 *sad2, const unsigned long long *nsad, i64 capsad, WallRec W,
                          i64 *next, unsigned long long *nnext, i64 capnext) {
    const i64 n = min((i64)*nsad, capsad);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const i64 code = sad2[i];
        int x, y, z;
        decode_v(c.g, code / 12, x, y, z);
        const i64 sf = face_ref(c.g, x, y, z, (int)(code % 12));
        i64 stack[kWallStack1], cache[1 << kWallCacheBits1];
#pragma unroll
        for (int k = 0; k < (1 << kWallCacheBits1); k++) cache[k] = -1;
        i64 rec = -1;
        const int r = wall_dfs(c, sf, stack, kWallStack1, cache, kWallCacheBits1, kWallPops1, rec);
        if (r == 1) wall_emit(W, sf, rec);
        else if (r == 2) wall_defer(next, nnext, capnext, sf);
    }
}
// a larger tier for list[first, first + count): one thread per 2-saddle face,
// its stack and cache in scratch (stack_cap + 2^cache_bits entries each)
__global__ void k_wall_tn(const __grid_constant__ RuleCtx c, const i64 *list, i64 first, i64 count, WallRec W, i64 *next,
                          unsigned long long *nnext, i64 capnext, i64 *scratch, int stack_cap, int cache_bits,
                          long long pop_cap) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (i64)gridDim.x * blockDim.x) {
        const i64 sf = list[first + i];
        i64 *stack = scratch + i * ((i64)stack_cap + ((i64)1 << cache_bits));
        i64 *cache = stack + stack_cap;
        for (i64 k = 0; k < ((i64)1 << cache_bits); k++) cache[k] = -1;
        i64 rec = -1;
        const int r = wall_dfs(c, sf, stack, stack_cap, cache, cache_bits, pop_cap, rec);
        if (r == 1) wall_emit(W, sf, rec);
        else if (r == 2) wall_defer(next, nnext, capnext, sf);
    }
}
__global__ void k_fix_wall(const __grid_constant__ RuleCtx c, WallRec W) {
    const i64 n = min((i64)*W.n, W.cap);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        rule_ds_wall(c, W.edge[i]);
}

// ------------------------------------------------- connectivity-mode separatrices
// (preserve_vpath=1, preserve_geometry=0): a separatrix counts as false when
// its end differs, not its geometry.
//
// End of the descending path from vertex v under vertex directions pv: the
// minimum reached (the walks of get_orginal_saddle_min_pairs and
// get_false_ds_vpath_connectivity, main_3d.cu:4613-4687, 4961-5062).  With pvo
// given, trouble (if still -1) becomes the first vertex on the way whose
// direction under pvo differs (the reference's trouble_maker; it compares
// before stepping, never at the end vertex).
__device__ i64 desc_end(const Grid &g, const uint8_t *pv, const uint8_t *pvo, i64 v, i64 &trouble, i64 cap,
                        int *err) {
    for (i64 steps = 0;; steps++) {
        const int d = pv[v];
        if (d == 15) return v;
        if (pvo && trouble < 0 && pvo[v] != d) trouble = v;
        v += g.doff[d];
        if (steps > cap) {
            atomicOr(err, ERR_WALK);
            return v;
        }
    }
}
// End of the ascending path from tetrahedron (x, y, z, s) under tet codes tc:
// the maximum reached (reference id) or -1 when the path leaves the grid
// (get_paired_id, main_3d.cu:4499-4537)
__device__ i64 asc_end(const Grid &g, const AscTab &t, const uint32_t *tc, int x, int y, int z, int s, i64 cap, int *err) {
    for (i64 steps = 0;; steps++) {
        const int j = (tc[x + (i64)y * g.W + (i64)z * g.WH] >> (3 * s)) & 7;
        if (j == 7) return tet_ref(g, x, y, z, s);
        if (!asc_move(g, t, x, y, z, s, j)) return -1;
        if (steps > cap) {
            atomicOr(err, ERR_WALK);
            return -1;
        }
    }
}
// is_false (main_3d.cu:4437-4497): along the original ascending path from the
// tetrahedron, the first one whose decompressed pairing differs (into cur)
__device__ bool first_diff(const Grid &g, const AscTab &t, const uint32_t *tcP, const uint32_t *tcQ, int x, int y, int z,
                           int s, i64 cap, int *err, i64 &cur) {
    for (i64 steps = 0;; steps++) {
        const i64 ci = x + (i64)y * g.W + (i64)z * g.WH;
        const int p = (tcP[ci] >> (3 * s)) & 7;
        if (p == 7) return false;
        if (p != (int)((tcQ[ci] >> (3 * s)) & 7)) {
            cur = tet_code(ci, s);
            return true;
        }
        if (!asc_move(g, t, x, y, z, s, p)) return false;
        if (steps > cap) {
            atomicOr(err, ERR_WALK);
            return false;
        }
    }
}
// get_false_ds_vpath_connectivity (main_3d.cu:4961-5062): for each original
// 1-saddle edge, the decompressed descending paths from its endpoints (v1,
// the higher id, first) against the original ones; the first endpoint whose
// minimum differs records (edge, trouble maker), the trouble maker carried
// over from v1's walk into v2's as in the reference.
__global__ void k_conn_ds(const __grid_constant__ RuleCtx c, PathRec R, i64 cap) {
    const Grid &g = c.g;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        uint32_t m = (c.P.crit[v] >> 1) & 0x7Fu;
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1;
            const i64 ends[2] = {v + g.coff[TOPO_EDGE_V[k][0]], v + g.coff[TOPO_EDGE_V[k][1]]};
            i64 trouble = -1, unused = -1;
            for (int j = 0; j < 2; j++) {
                const i64 eq = desc_end(g, c.Q.pv, c.P.pv, ends[j], trouble, cap, c.err);
                const i64 ep = desc_end(g, c.P.pv, nullptr, ends[j], unused, cap, c.err);
                if (eq != ep) {
                    const unsigned long long at = atomicAdd(&R.n[1], 1ull);
                    if ((i64)at < R.cap_ds) {
                        R.ds_edge[at] = edge_code(v, k);
                        R.ds_vert[at] = trouble;
                    }
                    break;
                }
            }
        }
    }
}
// get_false_as_vpath_connectivity (main_3d.cu:4761-4835) as intended: for each
// decompressed 2-saddle triangle, its cofaces in search order; a coface whose
// decompressed ascending path ends at another maximum than the original one
// (the original end is -1 for triangles that are not original 2-saddles, the
// reference's initial value) is checked with is_false, and the first record
// ends the triangle.  The reference indexes its table of original ends by the
// direction loop's counter instead of the triangle (all triangles share 28
// slots, written concurrently), so its own result depends on scheduling.
__global__ void k_conn_as(Grid g, const uint32_t *critP, const uint32_t *critQ, const uint32_t *tcP,
                          const uint32_t *tcQ, PathRec R, i64 cap, int *err) {
    __shared__ AscTab tab;
    load_asc_tab(tab);
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        uint32_t m = (critQ[v] >> 8) & 0xFFFu;
        if (!m) continue;
        const uint32_t mp = (critP[v] >> 8) & 0xFFFu;
        int x, y, z;
        decode_v(g, v, x, y, z);
        while (m) {
            const int sl = __ffs(m) - 1;
            m &= m - 1;
            for (int j = 0; j < TOPO_FACE_NCOF[sl]; j++) {
                const signed char *tc = TOPO_FACE_COF[sl][j];
                const int cx = x + tc[0], cy = y + tc[1], cz = z + tc[2], cs = tc[3];
                if (!cell_ok(g, cx, cy, cz, 1, 1, 1)) continue;
                const i64 eq = asc_end(g, tab, tcQ, cx, cy, cz, cs, cap, err);
                const i64 ep = ((mp >> sl) & 1u) ? asc_end(g, tab, tcP, cx, cy, cz, cs, cap, err) : -1;
                if (eq == ep) continue;
                i64 cur;
                if (first_diff(g, tab, tcP, tcQ, cx, cy, cz, cs, cap, err, cur)) {
                    const unsigned long long at = atomicAdd(&R.n[0], 1ull);
                    if ((i64)at < R.cap_as) {
                        R.as_tet[at] = tet_code(cx + (i64)cy * g.W + (i64)cz * g.WH, cs);
                        R.as_cur[at] = cur;
                    }
                    break;
                }
            }
        }
    }
}

// start tetrahedron (anchor offset, slot) of coface j of a triangle of slot
// sl, from four immediates (9 bits per (sl, j): dx+1, dy+1, dz+1, slot)
// instead of a table read whose index differs across the warp
__host__ __device__ constexpr unsigned long long cof_word(int w) {
    unsigned long long r = 0;
    for (int i = 0; i < 7; i++) {
        const int q = w * 7 + i;
        if (q >= 24) break;
        const signed char *t = cxt::TOPO_FACE_COF[q / 2][q % 2];
        r |= (unsigned long long)((t[0] + 1) | ((t[1] + 1) << 2) | ((t[2] + 1) << 4) | (t[3] << 6)) << (9 * i);
    }
    return r;
}
__device__ __forceinline__ void face_cof_start(int sl, int j, int &dx, int &dy, int &dz, int &ts) {
    constexpr unsigned long long W0 = cof_word(0), W1 = cof_word(1), W2 = cof_word(2), W3 = cof_word(3);
    const int q = 2 * sl + j, w = q / 7, i = q - 7 * w;
    const unsigned long long word = w == 0 ? W0 : (w == 1 ? W1 : (w == 2 ? W2 : W3));
    const unsigned v = (unsigned)(word >> (9 * i)) & 511u;
    dx = (int)(v & 3u) - 1;
    dy = (int)((v >> 2) & 3u) - 1;
    dz = (int)((v >> 4) & 3u) - 1;
    ts = (int)(v >> 6);
}
static_assert(cxt::TOPO_FACE_NCOF[0] == 2 && cxt::TOPO_FACE_NCOF[5] == 2 && cxt::TOPO_FACE_NCOF[11] == 2,
              "every triangle slot has two cofaces");

// --------------------------------------------------- geometry-mode separatrix checks
// get_false_as_vpath (main_3d.cu:4540-4610) with is_false: for each original
// 2-saddle triangle, its cofaces in search order; along each one's original
// ascending path, the first tetrahedron whose decompressed pairing differs is
// recorded, for the first coface that has one.  get_false_ds_vpath
// (:4837-4959): the reference's walk never advances past the first vertex
// (dec_current_id stays at the start), so each 1-saddle endpoint's
// steepest-descent pairing is compared once, v1 (higher id) first.
//
// The original paths never change during a correction.  They are traced once
// (k_path_trace): every tetrahedron on one gets a bit beside its pairing code
// (bit 18 + slot of the original tcode word), and every 2-saddle the box of
// bricks its paths visit.  A path is false only if a marked tetrahedron's
// pairing differs.  Per brick, two flags say whether it holds such a
// tetrahedron (as), or an original 1-saddle with a differing endpoint (ds);
// the gradient kernels set them with the decompressed field's gradient (a
// changed value reaches exactly the re-paired bricks' anchors).  A
// detection then walks from the 2-saddles whose box holds a flagged brick and looks
// at the 1-saddles of flagged bricks, and at nothing else.
//
// Bound by the reads of the boxes (8 bytes per 2-saddle) and by the latency
// of the walks left over (dependent loads).  Before, every 2-saddle near
// re-paired tiles of 16^3 anchors was walked to its path's end and every 1-saddle
// there checked, in eight kernels with a prefix sum over the tiles: 180 -> 27
// us per detection on a noisy 97 x 61 x 75 field (paths of some hundred
// steps), 677 -> 164 us at 256^3 (cold caches).
// a 2-saddle's box of bricks: x0 x1 (11 bits each), y0 y1 (11), z0 z1 (10); x0 > x1: empty
__device__ __forceinline__ unsigned long long box_pack(int x0, int x1, int y0, int y1, int z0, int z1) {
    return (unsigned long long)x0 | ((unsigned long long)x1 << 11) | ((unsigned long long)y0 << 22) |
           ((unsigned long long)y1 << 33) | ((unsigned long long)z0 << 44) | ((unsigned long long)z1 << 54);
}
__device__ __forceinline__ unsigned long long box_union(unsigned long long a, unsigned long long b) {
    const int ax0 = (int)(a & 2047), ax1 = (int)((a >> 11) & 2047), bx0 = (int)(b & 2047), bx1 = (int)((b >> 11) & 2047);
    if (ax0 > ax1) return b;
    if (bx0 > bx1) return a;
    return box_pack(min(ax0, bx0), max(ax1, bx1), min((int)((a >> 22) & 2047), (int)((b >> 22) & 2047)),
                    max((int)((a >> 33) & 2047), (int)((b >> 33) & 2047)), min((int)((a >> 44) & 1023), (int)((b >> 44) & 1023)),
                    max((int)(a >> 54), (int)(b >> 54)));
}
// does the box hold a flagged brick?  Boxes of more than kBoxBricks bricks (a
// straight path) count as holding one: looking would cost more than walking
constexpr int kBoxBricks = 27;
__device__ __forceinline__ bool box_flagged(const uint8_t *flags, int nbx, int nby, unsigned long long b) {
    const int x0 = (int)(b & 2047), x1 = (int)((b >> 11) & 2047), y0 = (int)((b >> 22) & 2047), y1 = (int)((b >> 33) & 2047),
              z0 = (int)((b >> 44) & 1023), z1 = (int)(b >> 54);
    if (x0 > x1) return false;
    if ((x1 - x0 + 1) * (y1 - y0 + 1) * (z1 - z0 + 1) > kBoxBricks) return true;
    unsigned any = 0;
    for (int z = z0; z <= z1; z++)
        for (int y = y0; y <= y1; y++) {
            const uint8_t *row = flags + (i64)nbx * (y + (i64)nby * z);
            for (int x = x0; x <= x1; x++) any |= row[x];
        }
    return any != 0;
}
// Work items handed out to warps in chunks (a multiple of 32): a warp's first
// chunk is its own index, further ones come from *ticket (zero at launch), so
// that warps that meet long walks do not hold the kernel's end.  Returns the
// chunk's first item.
__device__ __forceinline__ i64 next_chunk(bool &first, i64 chunk, unsigned long long *ticket) {
    const i64 warps = (i64)gridDim.x * (blockDim.x / 32);
    i64 c;
    if (first) {
        c = (i64)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
        first = false;
    } else {
        unsigned long long t = 0;
        if ((threadIdx.x & 31) == 0) t = atomicAdd(ticket, 1ull);
        c = warps + (i64)__shfl_sync(0xffffffffu, t, 0);
    }
    return c * chunk;
}
// chunk size that gives every warp of the grid about eight chunks
__device__ __forceinline__ i64 chunk_size(i64 n, i64 most) {
    const i64 c = (n / ((i64)gridDim.x * (blockDim.x / 32) * 8) + 31) / 32 * 32;
    return c < 32 ? 32 : (c > most ? most : c);
}

// Paths of more than kSegment steps are cut into segments, each an item of its
// own (start, box, slot of its 2-saddle among the ones with such paths, order:
// coface << 25 | index along the path): a detection's longest chain of dependent
// loads is then one segment's, and a long path is looked at only where its bricks are flagged.
constexpr int kSegment = 16;
struct Segment {
    unsigned long long box;
    i64 start;  // tetrahedron code
    uint32_t slot, order;
};
struct LongPaths {
    Segment *seg;
    i64 *sad;                 // per slot: the 2-saddle (anchor * 12 + triangle slot)
    unsigned long long *res;  // per slot: lowest (order << 38 | code) found, ~0: none
    unsigned long long *n;    // [0] segments, [1] slots
    i64 cap_seg, cap_slot;
};
// One lane per 2-saddle, both cofaces one after the other; a lane that is done
// takes the chunk's next 2-saddle.
__global__ void __launch_bounds__(kBlock) k_path_trace(Grid g, const i64 *sad2, const unsigned long long *nsad, i64 capsad, uint32_t *tcP,
                                                      unsigned long long *box, LongPaths L, int shx, int shy, int shz,
                                                      i64 cap, int *err, unsigned long long *ticket) {
    __shared__ AscTab tab;
    load_asc_tab(tab);
    const i64 n = min((i64)*nsad, capsad), chunk = chunk_size(n, 256);
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
    constexpr unsigned long long kEmpty = 1ull;  // x0 = 1 > x1 = 0
    bool first = true;
    for (i64 base = next_chunk(first, chunk, ticket); base < n; base = next_chunk(first, chunk, ticket)) {
        const i64 end = min(n, base + chunk);
        i64 pos = base, item = -1, steps = 0, code = 0, start = 0, start0 = 0;
        int x = 0, y = 0, z = 0, s = 0, j = 0;
        int bx0 = 0, bx1 = 0, by0 = 0, by1 = 0, bz0 = 0, bz1 = 0;  // box of the current segment
        unsigned long long box0 = kEmpty;                            // box of a short first path
        i64 slot = -1;
        unsigned segs = 0;
        bool on = false;  // on a path
        auto reset_box = [&]() { bx0 = 2047, bx1 = 0, by0 = 2047, by1 = 0, bz0 = 1023, bz1 = 0; };
        auto push = [&](unsigned long long b, i64 from, unsigned order) {
            const unsigned long long at = agg_slot(&L.n[0]);
            if ((i64)at < L.cap_seg) L.seg[at] = Segment{b, from, (uint32_t)slot, order};
        };
        while (true) {
            const unsigned want = __ballot_sync(full, item < 0);
            if (want) {
                const i64 my = pos + __popc(want & ((1u << lane) - 1u));
                if (item < 0 && my < end) {
                    item = my;
                    code = sad2[my];
                    j = 0;
                    on = false;
                    slot = -1;
                    reset_box();
                }
                pos = min(end, pos + (i64)__popc(want));
            }
            if (__all_sync(full, item < 0)) break;
            if (item < 0) continue;
            if (!on) {
                if (j == 2) {
                    box[item] = slot >= 0 ? kEmpty : box_union(box0, box_pack(bx0, bx1, by0, by1, bz0, bz1));
                    item = -1;
                    continue;
                }
                box0 = j == 1 ? box_pack(bx0, bx1, by0, by1, bz0, bz1) : kEmpty;
                start0 = start;
                reset_box();
                int vx, vy, vz, dx, dy, dz;
                decode_v(g, code / 12, vx, vy, vz);
                face_cof_start((int)(code % 12), j, dx, dy, dz, s);
                x = vx + dx;
                y = vy + dy;
                z = vz + dz;
                j++;
                steps = 0;
                segs = 0;
                start = tet_code(x + (i64)y * g.W + (i64)z * g.WH, s);
                on = cell_ok(g, x, y, z, 1, 1, 1);
                if (!on) continue;
            }
            const i64 ci = x + (i64)y * g.W + (i64)z * g.WH;
            const uint32_t w = tcP[ci];
            const int p = (int)((w >> (3 * s)) & 7u);
            if (p != 7) {
                const uint32_t mark = 1u << (18 + s);
                if (!(w & mark)) atomicOr(&tcP[ci], mark);
                bx0 = min(bx0, x >> shx);
                bx1 = max(bx1, x >> shx);
                by0 = min(by0, y >> shy);
                by1 = max(by1, y >> shy);
                bz0 = min(bz0, z >> shz);
                bz1 = max(bz1, z >> shz);
                on = asc_move(g, tab, x, y, z, s, p);
                if (++steps > cap) {
                    atomicOr(err, ERR_WALK);
                    on = false;
                }
            } else {
                on = false;
            }
            const bool cut = on && steps % kSegment == 0;
            if (cut && slot < 0) {  // a long path: both cofaces' paths go to the segments
                slot = (i64)agg_slot(&L.n[1]);
                if (slot < L.cap_slot) {
                    L.sad[slot] = code;
                    L.res[slot] = ~0ull;
                }
                if (j == 2) push(box0, start0, 0u);
            }
            if (cut || (!on && slot >= 0)) {
                push(box_pack(bx0, bx1, by0, by1, bz0, bz1), start, ((unsigned)(j - 1) << 25) | segs);
                segs++;
                start = tet_code(x + (i64)y * g.W + (i64)z * g.WH, s);
                reset_box();
            }
        }
    }
}

// an original 1-saddle's first differing endpoint (or -1)
template <int K>
__device__ __forceinline__ i64 ds_differs(const Grid &g, const uint8_t *pvP, const uint8_t *pvQ, i64 v) {
    constexpr int c0 = cxt::TOPO_EDGE_V[K][0], c1 = cxt::TOPO_EDGE_V[K][1];
    const i64 a = v + cxt::ccx(c0) + cxt::ccy(c0) * (i64)g.W + cxt::ccz(c0) * g.WH,
              b = v + cxt::ccx(c1) + cxt::ccy(c1) * (i64)g.W + cxt::ccz(c1) * g.WH;
    const int pa = pvP[a], pb = pvP[b];
    if (pa != 15 && pa != pvQ[a]) return a;
    if (pb != 15 && pb != pvQ[b]) return b;
    return -1;
}
// One detection: the first gridDim.x - ds_blocks blocks take the 2-saddles and
// the segments of long paths, the others the bricks with a differing 1-saddle
// endpoint (strict: none, k_ds_strict does those).
constexpr int kQueue = 512;
__global__ void __launch_bounds__(kBlock) k_path_detect(Grid g, PathFlags F, const i64 *sad2, const unsigned long long *nsad, i64 capsad,
                                                       const unsigned long long *box, const uint32_t *critP,
                                                       const uint32_t *tcQ,
                                                       const uint8_t *pvQ, LongPaths L, PathRec R,
                                                       unsigned long long *ticket, int nbx, int nby, int nbz, int shape_x,
                                                       int shape_y, int shape_z, int ds_blocks) {
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned as_blocks = gridDim.x - (unsigned)ds_blocks;
    if (blockIdx.x >= as_blocks) {
        const i64 nb = (i64)nbx * nby * nbz;
        const i64 w0 = (i64)(blockIdx.x - as_blocks) * (blockDim.x / 32) + warp, ws = (i64)ds_blocks * (blockDim.x / 32);
        for (i64 b0 = w0 * 32; b0 < nb; b0 += ws * 32) {
            unsigned m = __ballot_sync(full, b0 + lane < nb && F.ds[b0 + lane]);
            for (; m; m &= m - 1) {
                const i64 b = b0 + __ffs(m) - 1;
                const int x0 = (int)(b % nbx) * shape_x, y0 = (int)((b / nbx) % nby) * shape_y,
                          z0 = (int)(b / ((i64)nbx * nby)) * shape_z;
                for (int t = lane; t < DMTZ_BRICK; t += 32) {
                    const int x = x0 + t % shape_x, y = y0 + (t / shape_x) % shape_y, z = z0 + t / (shape_x * shape_y);
                    if (x >= g.W || y >= g.H || z >= g.D) continue;
                    const i64 v = x + (i64)y * g.W + (i64)z * g.WH;
                    const uint32_t c = (critP[v] >> 1) & 0x7Fu;
                    if (!c) continue;
                    DMTZ_FOR(7, K, {
                        constexpr int k = decltype(K)::value;
                        if ((c >> k) & 1u) {
                            const i64 e = ds_differs<k>(g, F.pvP, pvQ, v);
                            if (e >= 0) {
                                const unsigned long long at = agg_slot(&R.n[1]);
                                if ((i64)at < R.cap_ds) {
                                    R.ds_edge[at] = edge_code(v, k);
                                    R.ds_vert[at] = e;
                                }
                            }
                        }
                    });
                }
            }
        }
        return;
    }
    __shared__ uint16_t queue[kBlock / 32][kQueue];  // per warp: the chunk's items to walk
    __shared__ AscTab tab;
    load_asc_tab(tab);
    const i64 n2 = min((i64)*nsad, capsad), n = n2 + min((i64)L.n[0], L.cap_seg);  // 2-saddles, then segments
    const i64 warps = (i64)as_blocks * (blockDim.x / 32);
    i64 chunk = (n / (warps * 8) + 31) / 32 * 32;
    chunk = chunk < 32 ? 32 : (chunk > kQueue ? kQueue : chunk);
    bool own = true;
    while (true) {
        i64 c;
        if (own) {
            c = (i64)blockIdx.x * (blockDim.x / 32) + warp;
            own = false;
        } else {
            unsigned long long t = 0;
            if (lane == 0) t = atomicAdd(ticket, 1ull);
            c = warps + (i64)__shfl_sync(full, t, 0);
        }
        const i64 base = c * chunk;
        if (base >= n) return;
        int cnt = 0;
        for (int k = 0; k < (int)chunk; k += 32) {
            const i64 i = base + k + lane;
            const bool d = i < n && box_flagged(F.as, nbx, nby, i < n2 ? box[i] : L.seg[i - n2].box);
            const unsigned m = __ballot_sync(full, d);
            if (d) queue[warp][cnt + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(k + lane);
            cnt += __popc(m);
        }
        __syncwarp();
        // lanes whose walk ended take the next item of the queue.  A 2-saddle's
        // paths (code >= 0) are at most kSegment steps each, and so is a segment (code = -1)
        int pos = 0, item = -1, s = 0, j = 0, x = 0, y = 0, z = 0, steps = 0;
        i64 code = 0, start = 0;
        uint32_t slot = 0, order = 0;
        bool on = false;
        while (true) {
            const unsigned want = __ballot_sync(full, item < 0);
            if (want) {
                const int my = pos + __popc(want & ((1u << lane) - 1u));
                if (item < 0 && my < cnt) {
                    item = queue[warp][my];
                    steps = 0;
                    if (base + item < n2) {
                        code = sad2[base + item];
                        j = 0;
                        on = false;
                    } else {
                        const Segment q = L.seg[base + item - n2];
                        code = -1;
                        j = 2;
                        on = true;
                        slot = q.slot;
                        order = q.order;
                        decode_v(g, q.start >> 5, x, y, z);
                        s = (int)(q.start & 31) - 20;
                    }
                }
                pos = min(cnt, pos + __popc(want));
            }
            if (__all_sync(full, item < 0)) break;
            if (item < 0) continue;
            if (!on) {  // the next coface, or done
                if (j == 2) {
                    item = -1;
                    continue;
                }
                int vx, vy, vz, dx, dy, dz;
                decode_v(g, code / 12, vx, vy, vz);
                face_cof_start((int)(code % 12), j, dx, dy, dz, s);
                x = vx + dx;
                y = vy + dy;
                z = vz + dz;
                j++;
                steps = 0;
                on = cell_ok(g, x, y, z, 1, 1, 1);
                start = tet_code(x + (i64)y * g.W + (i64)z * g.WH, s);
                if (!on) continue;
            }
            const i64 ci = x + (i64)y * g.W + (i64)z * g.WH;
            const uint32_t wp = F.tcP[ci], wq = tcQ[ci];
            const int p = (wp >> (3 * s)) & 7;
            if (p == 7) {
                on = false;
            } else if (p != (int)((wq >> (3 * s)) & 7)) {
                if (code >= 0) {
                    const unsigned long long at = agg_slot(&R.n[0]);
                    if ((i64)at < R.cap_as) {
                        R.as_tet[at] = start;
                        R.as_cur[at] = tet_code(ci, s);
                    }
                } else {
                    atomicMin(&L.res[slot], ((unsigned long long)order << 38) | (unsigned long long)tet_code(ci, s));
                }
                item = -1;
            } else {
                on = asc_move(g, tab, x, y, z, s, p) && ++steps < kSegment;
            }
        }
        __syncwarp();
    }
}

// the records of the 2-saddles with long paths, and their slots for the next detection
__global__ void k_path_long(Grid g, LongPaths L, PathRec R) {
    const i64 n = min((i64)L.n[1], L.cap_slot);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const unsigned long long r = L.res[i];
        if (r == ~0ull) continue;
        L.res[i] = ~0ull;
        const i64 code = L.sad[i], v = code / 12;
        int dx, dy, dz, s;
        face_cof_start((int)(code % 12), (int)(r >> 63), dx, dy, dz, s);  // order's top bit: the coface
        const unsigned long long at = agg_slot(&R.n[0]);
        if ((i64)at < R.cap_as) {
            R.as_tet[at] = tet_code(v + dx + dy * (i64)g.W + dz * g.WH, s);
            R.as_cur[at] = (i64)(r & ((1ull << 38) - 1));
        }
    }
}

// Strict descending check (dmtz_opts.strict_separatrices; no counterpart in
// the reference).  get_false_ds_vpath compares each endpoint's pairing only
// at the first vertex of its path (see above); this check walks the whole
// original descending path of each endpoint of every original 1-saddle (v1,
// the higher id, first; the walk follows the original steepest-descent
// pairing to a minimum) and records the first vertex whose decompressed
// pairing differs, in the same record format, so fix_ds_vpath's rule
// (rule_ds_path) repairs it.  With no record left, every original descending
// separatrix is a decompressed one vertex for vertex, so the descending
// labels of all 1-saddle endpoints agree.
__device__ __forceinline__ i64 dir_offset(const Grid &g, int d) {
    i64 o = 0;
#pragma unroll
    for (int i = 0; i < 14; i++)
        if (d == i) o = g.doff[i];
    return o;
}
// Items are the original 1-saddles (the list of k_crit_list<1, 7>); one lane
// walks one item's first endpoint's path, then, if that is clean, the
// second's, and idle lanes take new items from chunks of 64 handed out by a
// ticket (*ticket, zero at launch): walks are long and uneven, and a lane that
// finished does not wait for the warp's longest walk.
__global__ void k_ds_strict(const __grid_constant__ RuleCtx c, PathRec R, const i64 *sad1, const unsigned long long *nsad1, i64 step_cap,
                            unsigned long long *ticket) {
    const Grid &g = c.g;
    constexpr i64 kChunk = 64;
    // corners (dx + 2 dy + 4 dz) of edge family k, higher id first: bits 6k .. 6k+5
    constexpr uint64_t kEnds = []() {
        uint64_t e = 0;
        for (int k = 0; k < 7; k++)
            e |= (uint64_t)(cxt::TOPO_EDGE_V[k][0] | (cxt::TOPO_EDGE_V[k][1] << 3)) << (6 * k);
        return e;
    }();
    const i64 n = min((i64)*nsad1, R.cap_ds);
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
    i64 pos = 0, end = 0, item = -1, steps = 0, u = 0, second = 0, edge = 0;
    bool first = true, drained = false;
    while (true) {
        const unsigned want = __ballot_sync(full, item < 0 && !drained);
        if (want) {
            if (pos >= end) {  // the warp's chunk is used up: take the next one
                unsigned long long b0 = 0;
                if (lane == 0) b0 = atomicAdd(ticket, (unsigned long long)kChunk);
                pos = (i64)__shfl_sync(full, b0, 0);
                end = min(n, pos + kChunk);
            }
            const i64 my = pos + __popc(want & ((1u << lane) - 1u));
            if (item < 0 && !drained) {
                if (pos >= n) {
                    drained = true;
                } else if (my < end) {
                    const i64 code = sad1[my], a = code / 7;
                    const int k = (int)(code - 7 * a);
                    const int ends = (int)((kEnds >> (6 * k)) & 63u), c0 = ends & 7, c1 = ends >> 3;
                    u = a + (c0 & 1) + ((c0 >> 1) & 1) * (i64)g.W + (c0 >> 2) * g.WH;
                    second = a + (c1 & 1) + ((c1 >> 1) & 1) * (i64)g.W + (c1 >> 2) * g.WH;
                    edge = edge_code(a, k);
                    item = my;
                    first = true;
                    steps = 0;
                }
            }
            pos = min(pos + (i64)__popc(want), end);
        }
        if (__all_sync(full, item < 0 && drained)) break;
        if (item >= 0) {  // one step of the current endpoint's walk
            const int po = c.P.pv[u];
            if (po == 15) {  // an original minimum: this endpoint's path is clean
                if (first) {
                    first = false;
                    u = second;
                    steps = 0;
                } else {
                    item = -1;
                }
            } else if (po != c.Q.pv[u]) {
                const unsigned long long at = agg_slot(R.n + 1);
                if ((i64)at < R.cap_ds) {
                    R.ds_edge[at] = edge;
                    R.ds_vert[at] = u;
                }
                item = -1;
            } else if (++steps > step_cap) {  // a cycle: not a gradient
                atomicOr(c.err, ERR_WALK);
                item = -1;
            } else {
                u += dir_offset(g, po);
            }
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_fix_path(const __grid_constant__ RuleCtx c, const __grid_constant__ PathRec P) {
    __shared__ RuleTab tab;
    let_next();
    const i64 na = min((i64)P.n[0], P.cap_as), nd = min((i64)P.n[1], P.cap_ds);
    const int per = cells_per_warp(na + nd, rule_warps()), lane = threadIdx.x & 31;
    const i64 wa = (na + per - 1) / per, wd = wa + (nd + per - 1) / per;
    constexpr int NW = kBlock / 32;
    if ((i64)blockIdx.x * NW >= wd) return;
    load_rule_tab(tab);
    const Rules R{c, tab};
    for (i64 w = (i64)blockIdx.x * NW + (threadIdx.x >> 5); w < wd; w += (i64)gridDim.x * NW) {
        Lowered o;
        const i64 i = (w < wa ? w : w - wa) * per + lane;
        if (lane < per) {
            if (w < wa) {
                if (i < na) rule_as_path(R, P.as_cur[i], o);
            } else if (i < nd) {
                rule_ds_path(R, P.ds_vert[i], o);
            }
        }
        __syncwarp();
        request_warp(c, o);
    }
}

// --------------------------------------------------------------- value update
// applyDeltaBuffer1 (main_3d.cu:1122-1164) on the requested vertices only.
// The delta is what the reference's buffer holds: get_delta(v), with the
// buffer's "no request" sentinel -2000*range (a request whose delta is not
// above the sentinel leaves the buffer unchanged under edit_type 0).
// Where bricks are marked (mark), a vertex has as many lanes as its reach has bricks
// (see mark_dirty) and the first of them updates it.  (A flag: `c ? BrickMarks{} : B`, with B a
// kernel's grid-constant parameter, bound to the reference faulted where c held.)
__device__ __forceinline__ void apply_requests(const RuleCtx &c, double range, int preserve_type, int update, uint8_t *changed,
                                               double *delta_out, const BrickMarks &B, bool mark, unsigned block,
                                               unsigned blocks) {
    const i64 n = min((i64)*c.reqn, c.reqcap);
    const double sentinel = -2000.0 * range;
    const double tiny = 1e-15 * range;
    double *g = const_cast<double *>(c.gv);
    int *cnt = const_cast<int *>(c.cnt);
    const int lane = threadIdx.x & 31, lanes = mark ? B.lanes : 1, per = 32 / lanes, j = lane % lanes;
    const i64 nw = blockDim.x / 32, step = (i64)blocks * nw * per;
    for (i64 base = ((i64)block * nw + (threadIdx.x >> 5)) * per; base < n; base += step) {
        const i64 i = base + lane / lanes;
        const i64 v = i < n ? c.reqlist[i] : 0;
        double d = 0, f = 0, gv = 0;
        int cv = 0;
        if (i < n) {
            d = get_delta(c, v);
            f = c.f[v];
            gv = g[v];
            cv = cnt[v];
        }
        const bool req = i < n && (c.edit_type == 0 ? (d > sentinel) : (d != sentinel));
        __syncwarp();  // every lane has read what the first one changes
        if (i < n && j == 0) {
            c.reqbits[v >> 5] = 0;  // every bit of this word belongs to listed vertices
            if (delta_out) delta_out[v] = req ? d : sentinel;
            if (req && update) {
                const double lowb = __dsub_rn(f, c.bound);
                if (preserve_type == 0 && fabs(d) > tiny && cv < 5 && fabs(__dsub_rn(f, __dadd_rn(gv, d))) <= c.bound) {
                    g[v] = __dadd_rn(gv, d);
                    cnt[v] = cv + 1;
                    if (c.progress) *c.progress = 1ull;
                } else {
                    cnt[v] = 6;
                    g[v] = lowb;
                    if (c.progress && (cv != 6 || gv != lowb)) *c.progress = 1ull;
                }
                if (changed) changed[v] = 1;
            }
        }
        if (mark) mark_dirty(c.g, B, req && update, v, j);
    }
}
// The blocks of bricks that every n / sample-th request reaches, for a round that re-pairs the
// whole grid and wants to know how much of it the update reached (see sampled_marks).
__device__ __forceinline__ void sample_bricks(const RuleCtx &c, const BrickMarks &B, unsigned block, unsigned blocks) {
    const i64 n = min((i64)*c.reqn, c.reqcap), every = max(n / B.sample, (i64)1), m = (n + every - 1) / every;
    const int lane = threadIdx.x & 31, per = 32 / B.lanes, j = lane % B.lanes;
    const i64 nw = blockDim.x / 32, step = (i64)blocks * nw * per;
    for (i64 base = ((i64)block * nw + (threadIdx.x >> 5)) * per; base < m; base += step) {
        const i64 i = base + lane / B.lanes;
        mark_dirty(c.g, B, i < m, i < m ? c.reqlist[i * every] : 0, j);
    }
}
// SAMPLE: in a round that re-pairs the whole grid; the first blocks sample, beside the others' updates
constexpr unsigned kSampleBlocks = 64;
template <bool SAMPLE>
__global__ void __launch_bounds__(kBlock) k_apply(const __grid_constant__ RuleCtx c, double range, int preserve_type, int update,
                                                 uint8_t *changed, double *delta_out, const __grid_constant__ BrickMarks B) {
    let_next();
    after_previous();
    constexpr unsigned first = SAMPLE ? kSampleBlocks : 0;
    if (SAMPLE && blockIdx.x < first) {
        sample_bricks(c, B, blockIdx.x, first);
        return;
    }
    apply_requests(c, range, preserve_type, update, changed, delta_out, B, !SAMPLE && B.flags, blockIdx.x - first, gridDim.x - first);
}

// ------------------------------------------------------------- stall breaker
// A round whose update changes no value and no edit counter leaves the state
// as it was, so the reference's loop repeats it forever (main_3d.cu:6784 has
// no exit for this; e.g. a false extremum no rule addresses, or requests on
// vertices already at f - bound).  With break_stalls, such a round instead
// sets every vertex within `radius` (per axis) of a vertex of a remaining
// mismatched cell -- or of a separatrix record's tetrahedron or vertex -- back
// to its original value, which is always within the bound, and requests it so
// that the next re-pairing covers it; then the loop goes on.  Rounds that make
// progress are never touched, so runs that converge under the reference's
// rules give the reference's output.
//
// The region is built in spare bits of the per-vertex `changed` bytes (bit 0
// is the edit mark): seeds get bit 1, three separable line dilations grow it
// to the box of half-width `radius` around every seed, and k_snap_mask resets
// the region and clears the bits.  Seed writers all store (bit 0 | 2) to the
// byte, and bit 0 does not change meanwhile, so unordered writes agree.
constexpr uint8_t kSnapSeed = 2, kSnapGrow = 4;
__device__ __forceinline__ void seed_vertex(const Grid &g, uint8_t *m, i64 v) {
    if (v >= 0 && v < g.V) m[v] = (uint8_t)(m[v] | kSnapSeed);
}
// the vertices of a listed cell
__device__ __forceinline__ void seed_cell(const Grid &g, i64 code, uint8_t *m) {
    const i64 v = code >> 5;
    const int b = (int)(code & 31);
    if (b == 0) {
        seed_vertex(g, m, v);
    } else if (b < 8) {
        for (int j = 0; j < 2; j++) seed_vertex(g, m, v + g.coff[TOPO_EDGE_V[b - 1][j]]);
    } else if (b < 20) {
        for (int j = 0; j < 3; j++) seed_vertex(g, m, v + g.coff[TOPO_FACE_V[b - 8][j]]);
    } else {
        for (int j = 0; j < 4; j++) seed_vertex(g, m, v + g.coff[TOPO_TET_V[b - 20][j]]);
    }
}
__global__ void k_seed_cells(Grid g, CpLists L, uint8_t *m) {
    const i64 n0 = min((i64)L.n[0], L.cap[0]), n1 = min((i64)L.n[1], L.cap[1]), n2 = min((i64)L.n[2], L.cap[2]),
              n3 = min((i64)L.n[3], L.cap[3]);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n0 + n1 + n2 + n3; i += (i64)gridDim.x * blockDim.x)
        seed_cell(g, i < n0 ? L.l[0][i] : i < n0 + n1 ? L.l[1][i - n0] : i < n0 + n1 + n2 ? L.l[2][i - n0 - n1]
                                                                                       : L.l[3][i - n0 - n1 - n2], m);
}
__global__ void k_seed_paths(Grid g, PathRec R, uint8_t *m) {
    const i64 na = min((i64)R.n[0], R.cap_as), nd = min((i64)R.n[1], R.cap_ds);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < na + nd; i += (i64)gridDim.x * blockDim.x) {
        if (i < na) seed_cell(g, R.as_cur[i], m);
        else seed_vertex(g, m, R.ds_vert[i - na]);
    }
}
__global__ void k_seed_walls(Grid g, WallRec W, uint8_t *m) {
    const i64 n = min((i64)*W.n, W.cap);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        i64 a, b;
        edge_verts(g, W.edge[i], a, b);
        seed_vertex(g, m, a);
        seed_vertex(g, m, b);
    }
}
// one thread per line along `axis` (0 = x, 1 = y, 2 = z): every position
// within `radius` of a seed of the line becomes a seed
__global__ void k_dilate_axis(Grid g, uint8_t *m, int axis, int radius) {
    const int n = axis == 0 ? g.W : axis == 1 ? g.H : g.D;
    const i64 step = axis == 0 ? 1 : axis == 1 ? (i64)g.W : g.WH;
    const i64 lines = g.V / n;
    for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < lines; t += (i64)gridDim.x * blockDim.x) {
        i64 base;
        if (axis == 0) base = t * g.W;                                  // t = y + H z
        else if (axis == 1) base = (t % g.W) + (t / g.W) * g.WH;        // t = x + W z
        else base = t;                                                  // t = x + W y
        int last = -radius - 1;
        for (int i = 0; i < n; i++) {
            const uint8_t b = m[base + i * step];
            if (b & kSnapSeed) last = i;
            if (i - last <= radius) m[base + i * step] = (uint8_t)(b | kSnapGrow);
        }
        int next = n + radius + 1;
        for (int i = n - 1; i >= 0; i--) {
            uint8_t b = m[base + i * step];
            if (b & kSnapSeed) next = i;
            if (next - i <= radius) b |= kSnapGrow;
            m[base + i * step] = (uint8_t)((b & 1) | ((b & kSnapGrow) ? kSnapSeed : 0));
        }
    }
}
__global__ void k_snap_mask(const __grid_constant__ RuleCtx c, uint8_t *m) {
    double *gv = const_cast<double *>(c.gv);
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < c.g.V; v += (i64)gridDim.x * blockDim.x) {
        const uint8_t b = m[v];
        if (!(b & kSnapSeed)) continue;
        m[v] = (uint8_t)(b & 1);
        if (gv[v] != c.f[v]) {
            gv[v] = c.f[v];
            m[v] = 1;
            lower(c, v);  // a request: the re-pairing looks here
        }
    }
}
// the request bits of the listed vertices back to 0 (k_apply does this for
// the vertices it updates; snapped vertices are only re-paired)
__global__ void k_clear_req(const i64 *reqlist, const unsigned long long *n, i64 cap, uint32_t *reqbits) {
    const i64 m = min((i64)*n, cap);
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (i64)gridDim.x * blockDim.x)
        reqbits[reqlist[i] >> 5] = 0;
}

// filter_vertices / _edges / _faces / _tetrahedras (main_3d.cu:2405-2490):
// every vertex of every original critical cell goes to f - bound
__global__ void k_filter(Grid g, const uint32_t *crit_o, const double *f, double *gv, double bound) {
    i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= g.V) return;
    uint32_t m = crit_o[v];
    if (!m) return;
    int x, y, z;
    decode_v(g, v, x, y, z);
    uint32_t corners = 0;
    if (m & 1u) corners |= 1u;
    for (int k = 0; k < 7; k++)
        if (m & (1u << (1 + k))) corners |= (1u << TOPO_EDGE_V[k][0]) | (1u << TOPO_EDGE_V[k][1]);
    for (int s = 0; s < 12; s++)
        if (m & (1u << (8 + s)))
            corners |= (1u << TOPO_FACE_V[s][0]) | (1u << TOPO_FACE_V[s][1]) | (1u << TOPO_FACE_V[s][2]);
    for (int s = 0; s < 6; s++)
        if (m & (1u << (20 + s)))
            corners |= (1u << TOPO_TET_V[s][0]) | (1u << TOPO_TET_V[s][1]) | (1u << TOPO_TET_V[s][2]) |
                       (1u << TOPO_TET_V[s][3]);
    while (corners) {
        const int c8 = __ffs(corners) - 1;
        corners &= corners - 1;
        const i64 u = v + g.coff[c8];
        gv[u] = __dsub_rn(f[u], bound);  // same value from every writer
    }
}

// --------------------------------------------------------------- manifold labels
// Descending manifold label of a vertex: the minimum its steepest-descent path
// (vertex -> other endpoint of its paired edge, processVertices'
// pairing) reaches.  Ascending label of a tetrahedron: the maximum (unpaired
// tetrahedron) its ascending path (is_false's walk, main_3d.cu:4437-4497)
// reaches, or -1 when the path leaves through the boundary.  Both by pointer
// jumping: lab <- lab[lab] until nothing changes.
//
// I: int32 where every tetrahedron index fits (below 2^31 / 6 vertices), else int64.
template <class I>
__global__ void k_desc_init(Grid g, const uint8_t *pv, I *lab) {
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        const int d = pv[v];
        lab[v] = (I)(d == 15 ? v : v + g.doff[d]);
    }
}
// one thread per anchor, its six tetrahedra
template <class I>
__global__ void __launch_bounds__(kBlock) k_asc_init(Grid g, const uint32_t *tcode, I *lab) {
    __shared__ AscTab tab;
    load_asc_tab(tab);
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        int x, y, z;
        decode_v(g, v, x, y, z);
        const bool cube = cell_ok(g, x, y, z, 1, 1, 1);
        const uint32_t code = tcode[v];
        I out[6];
#pragma unroll
        for (int ts = 0; ts < 6; ts++) {
            const int j = (code >> (3 * ts)) & 7;
            int nx = x, ny = y, nz = z, s = ts;
            if (!cube) out[ts] = -2;                    // no such tetrahedron
            else if (j == 7) out[ts] = (I)(6 * v + ts); // a maximum
            else if (!asc_move(g, tab, nx, ny, nz, s, j)) out[ts] = -1;  // leaves through the boundary
            else out[ts] = (I)((nx + (i64)ny * g.W + (i64)nz * g.WH) * 6 + s);
        }
#pragma unroll
        for (int ts = 0; ts < 6; ts++) lab[6 * v + ts] = out[ts];
    }
}
// Every label to its root, following at most kHops links per element and
// call; *unsettled is set when a root was not reached.  A link read while other threads
// shorten theirs is an older or a newer one of the same path.  (One link per
// call, and a look at the flag from the host after each: 8-10 calls per label
// array.)
constexpr int kHops = 64;
template <class I>
__global__ void __launch_bounds__(kBlock) k_jump(I *lab, i64 n, int *unsettled) {
    int left = 0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const I l = lab[i];
        if (l < 0) continue;
        I r = l;
        int h = 0;
        for (; h < kHops && r >= 0; h++) {
            const I q = lab[r];
            if (q == r) break;
            r = q;
        }
        if (r != l) lab[i] = r;
        left |= h == kHops;
    }
    if (__syncthreads_or(left) && threadIdx.x == 0) atomicOr(unsettled, 1);
}
// reference ids of the tetrahedra's labels (a vertex's label is its id)
template <class I>
__global__ void k_asc_out(Grid g, const I *lab, int32_t *out) {
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        int x, y, z;
        decode_v(g, v, x, y, z);
        if (!cell_ok(g, x, y, z, 1, 1, 1)) continue;
        int32_t *o = out + tet_ref(g, x, y, z, 0);
#pragma unroll
        for (int ts = 0; ts < 6; ts++) {
            const I l = lab[6 * v + ts];
            int32_t r = -1;
            if (l >= 0) {
                const i64 lv = l / 6;
                int lx, ly, lz;
                decode_v(g, lv, lx, ly, lz);
                r = (int32_t)tet_ref(g, lx, ly, lz, (int)(l - 6 * lv));
            }
            o[ts] = r;
        }
    }
}

// exact min / max of a field through its order keys
__global__ void k_minmax(const double *a, i64 n, unsigned long long *kmin, unsigned long long *kmax) {
    unsigned long long lo = ~0ull, hi = 0ull;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const unsigned long long k = okey(a[i]);
        lo = k < lo ? k : lo;
        hi = k > hi ? k : hi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(kmin, lo);
        atomicMax(kmax, hi);
    }
}

// largest |a - b| as an order key
__global__ void k_max_gap(const double *a, const double *b, i64 n, unsigned long long *kmax) {
    double gap = 0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) gap = fmax(gap, fabs(a[i] - b[i]));
    unsigned long long k = okey(gap);
    for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
    if ((threadIdx.x & 31) == 0) atomicMax(kmax, k);
}

__global__ void k_count_u8(const uint8_t *a, i64 n, unsigned long long *out) {
    unsigned long long c = 0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) c += a[i] != 0;
    for (int off = 16; off > 0; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}
__global__ void k_fill_i32(int *p, int val, i64 n) {
    i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = val;
}
__global__ void k_check_finite(const double *a, i64 n, int *bad) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        if (!isfinite(a[i])) atomicOr(bad, 1);
}

}  // namespace dmtz

// =============================================================================
// host side
// =============================================================================
// ----------------------------------------------------- decompression model
// SZ-style error-bounded quantisation of the original field, done on the GPU
// (the reference runs an external compressor and reads its output back,
// main_3d.cu:6331-6356): g = fmin + 2 eps * rint((f - fmin) / (2 eps)); then a
// fraction `frac` of the vertices gets extra uniform noise in [-eps, eps); then
// g is clamped into [f - eps, f + eps].  Random numbers are a counter-based
// hash of (seed, vertex, stream): the splitmix64 finaliser, 53 bits to [0, 1).
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double unit_rand(uint64_t seed, i64 v, int k) {
    const uint64_t h = mix64(seed + 0x9E3779B97F4A7C15ull * (uint64_t)(2 * v + k + 1));
    return (double)(h >> 11) * 0x1.0p-53;
}
__global__ void k_quantize(i64 V, const double *f, double *g, double fmn, double eps, double frac, uint64_t seed) {
    const double w = __dmul_rn(2.0, eps);
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (i64)gridDim.x * blockDim.x) {
        const double fv = f[v];
        double q = w > 0.0 ? __dadd_rn(fmn, __dmul_rn(w, rint(__ddiv_rn(__dsub_rn(fv, fmn), w)))) : fv;
        if (unit_rand(seed, v, 0) < frac)
            q = __dadd_rn(q, __dmul_rn(eps, __dsub_rn(__dmul_rn(2.0, unit_rand(seed, v, 1)), 1.0)));
        const double lo = __dsub_rn(fv, eps), hi = __dadd_rn(fv, eps);
        g[v] = q < lo ? lo : (q > hi ? hi : q);
    }
}

// ----------------------------------------------------- learned-proposal glue
// Network input per vertex (layout in cnn.cuh) and the mismatch byte mm[v]
// (criticality of v's own cells differs between the two gradients).
//
// A slope tanh((f(u) - f(v)) / 4 bound) is the negative of its other end's, so
// a block computes the seven slopes towards larger ids of its vertices and of one
// layer before them, once each, into shared memory, and every vertex gathers its
// fourteen.  Bound by the float64 pipe (a difference, a product and a
// conversion per slope; GB300 has a fraction of other data-centre GPUs'
// float64 units): the quotients are products with the reciprocals, whose
// error (2^-52 relative) is far below the float32 value's; where a
// reciprocal is not finite and normal the host asks for quotients (EXACT).  With
// fourteen quotients per vertex 782 us at 160 x 144 x 128; now 206 us.
//
// Tiles of 32 x 8 x 4, and of 4 x 16 x 16 on grids at most 4 wide in x: 2 x 2000 x 1000
// 10.2 ms a call and 6.7 (7.9 with a thread per vertex), 4 x 1500 x 800 6.4 and 4.2 (7.7).
// the seven stencil directions towards larger ids
__host__ __device__ constexpr int up_dir(int r) { return cxt::dir_by_id(7 + r); }
__host__ __device__ constexpr int opposite_dir(int d) { return d ^ 1; }
template <int TX, int TY, int TZ, bool EXACT>
__global__ void __launch_bounds__(kBlock) k_features(Grid g, const double *f, const double *gv, const uint32_t *critP,
                                                    const uint32_t *critQ, double bound, double inv, double inv4,
                                                    __nv_bfloat16 *feat, uint8_t *mm, int ntx, int nty) {
    // box: one layer towards smaller ids in z and y, one to both sides in x
    // (directions with dz or dy = +1 may have dx = -1)
    constexpr int BX = TX + 2, BY = TY + 1, BZ = TZ + 1, NB = BX * BY * BZ;
    __shared__ __nv_bfloat16 slope[7][NB];
    const int x0 = (int)(blockIdx.x % (unsigned)ntx) * TX, y0 = (int)((blockIdx.x / (unsigned)ntx) % (unsigned)nty) * TY,
              z0 = (int)(blockIdx.x / ((unsigned)ntx * (unsigned)nty)) * TZ;
    for (int e = threadIdx.x; e < NB; e += kBlock) {
        const int x = x0 - 1 + e % BX, y = y0 - 1 + (e / BX) % BY, z = z0 - 1 + e / (BX * BY);
        const bool in = x >= 0 && y >= 0 && z >= 0 && x < g.W && y < g.H && z < g.D;
        const i64 v = in ? x + (i64)y * g.W + (i64)z * g.WH : 0;
        const double fv = f[v];
        DMTZ_FOR(7, R, {
            constexpr int r = decltype(R)::value, d = up_dir(r);
            constexpr int dx = cxt::TOPO_DIRS[d][0], dy = cxt::TOPO_DIRS[d][1], dz = cxt::TOPO_DIRS[d][2];
            float t = 0.f;
            if (in && bound > 0 && inb(g, x + dx, y + dy, z + dz)) {
                const double df = f[v + dx + dy * (i64)g.W + dz * g.WH] - fv;
                t = tanhf((float)(EXACT ? df / (4.0 * bound) : df * inv4));
            }
            slope[r][e] = __float2bfloat16_rn(t);
        });
    }
    __syncthreads();
    for (int t = threadIdx.x; t < TX * TY * TZ; t += kBlock) {
        const int lx = t % TX, ly = (t / TX) % TY, lz = t / (TX * TY);
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        if (x >= g.W || y >= g.H || z >= g.D) continue;
        const i64 v = x + (i64)y * g.W + (i64)z * g.WH;
        const int e = (lx + 1) + BX * ((ly + 1) + BY * (lz + 1));
        const bool mis = critP[v] != critQ[v];
        mm[v] = mis;
        const double dg = gv[v] - f[v];
        const float c0 = bound > 0 ? fminf(fmaxf((float)(EXACT ? dg / bound : dg * inv), -1.f), 1.f) : 0.f;
        uint16_t c[16];
        c[0] = __bfloat16_as_ushort(__float2bfloat16_rn(c0));
        c[1] = mis ? 0x3F80 : 0;  // 1
        DMTZ_FOR(7, R, {
            constexpr int r = decltype(R)::value, d = up_dir(r), o = opposite_dir(d);
            constexpr int dx = cxt::TOPO_DIRS[d][0], dy = cxt::TOPO_DIRS[d][1], dz = cxt::TOPO_DIRS[d][2];
            static_assert(cxt::TOPO_DIRS[o][0] == -dx && cxt::TOPO_DIRS[o][1] == -dy && cxt::TOPO_DIRS[o][2] == -dz, "opposite directions");
            c[2 + d] = __bfloat16_as_ushort(slope[r][e]);
            const uint16_t b = __bfloat16_as_ushort(slope[r][e - dx - dy * BX - dz * BX * BY]);
            c[2 + o] = b ? b ^ 0x8000u : 0;  // the other end's, negated (zero where there is none)
        });
        uint4 *dst = reinterpret_cast<uint4 *>(feat + v * 16);
        auto two = [&](int k) { return (uint32_t)c[k] | ((uint32_t)c[k + 1] << 16); };
        dst[0] = make_uint4(two(0), two(2), two(4), two(6));
        dst[1] = make_uint4(two(8), two(10), two(12), two(14));
    }
}
// dst[v] = max of src over v + k*step, |k| <= 2, along one axis (in-grid)
__global__ void k_dilate(Grid g, int axis, const uint8_t *src, uint8_t *dst) {
    const i64 step = axis == 0 ? 1 : axis == 1 ? (i64)g.W : g.WH;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        int c[3];
        decode_v(g, v, c[0], c[1], c[2]);
        const int n = axis == 0 ? g.W : axis == 1 ? g.H : g.D;
        uint8_t m = 0;
        for (int k = -2; k <= 2; k++) {
            const int q = c[axis] + k;
            if (q >= 0 && q < n) m |= src[v + k * step];
        }
        dst[v] = m;
    }
}
// Proposal at active vertices: g <- f + bound * tanh(o) where that lowers g by
// at least min_drop (absolute; the network's min_drop x bound); a value that
// the reference's own bound test |f - g| <= bound would reject becomes
// f - bound, the value the reference falls back to (main_3d.cu:1133-1141).
// the proposal's edits also go to the request list, so that only the bricks
// around them are re-paired afterwards
__global__ void k_propose(i64 V, const double *f, double *gv, const float *o, const uint8_t *active, double bound,
                          double min_drop, uint8_t *changed, i64 *reqlist, unsigned long long *reqn) {
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (i64)gridDim.x * blockDim.x) {
        if (!active[v]) continue;
        const double fv = f[v], old = gv[v];
        const double p = __dadd_rn(fv, __dmul_rn(bound, (double)tanhf(o[v])));
        if (!(old - p >= min_drop)) continue;  // keep g unless the proposal lowers it enough
        double nv = p;
        if (fabs(__dsub_rn(fv, nv)) > bound) nv = __dsub_rn(fv, bound);
        if (nv != old) {
            gv[v] = nv;
            changed[v] = 1;
            reqlist[agg_slot(reqn)] = v;
        }
    }
}

struct DevField {
    uint8_t *pv = nullptr;
    uint32_t *eup = nullptr;
    uint32_t *fup = nullptr;
    uint32_t *crit = nullptr;
    uint32_t *tcode = nullptr;
};

struct dmtz_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;      // copies that overlap the context stream's work
    cudaEvent_t side_done = nullptr;
    std::string err;
    // sized buffers
    i64 capV = 0, capE = 0, capF = 0, capT = 0, capB = 0;
    double *f = nullptr, *g = nullptr;
    DevField P, Q;
    int *cnt = nullptr;
    uint32_t *reqbits = nullptr;
    i64 *reqlist = nullptr;
    // Mismatch lists and separatrix records.  Sized for the counts that occur,
    // not for every cell: the mismatch lists start at list_frac x cells (at
    // least list_min entries, at most all cells) and grow when a scan
    // overflows them; the path records and the 2-saddle list are sized from
    // the original gradient's saddle counts, which bound them.
    i64 *lists[4] = {nullptr, nullptr, nullptr, nullptr};
    i64 capL[4] = {0, 0, 0, 0};
    double list_frac = 1.0 / 16;
    i64 list_min = 1 << 20;
    i64 *as_tet = nullptr, *as_cur = nullptr, *ds_edge = nullptr, *ds_vert = nullptr;
    i64 capAS = 0, capDS = 0, capSad2 = 0;
    uint32_t *brick_flags = nullptr;  // per brick (a byte each, four to a word): in this round's repair
    int inc_scan = 0;                 // repairs rebuild the mismatch lists incrementally (see KeepOps)
    int strict_ds = 0;                // descending separatrix checks walk whole paths (k_ds_strict)
    i64 *list_tmp[4] = {nullptr, nullptr, nullptr, nullptr};  // rebuilt mismatch lists, capL entries each
    uint32_t *brick_list = nullptr;   // the repair's bricks, capB entries
    unsigned long long *brick_n = nullptr;  // their number
    i64 *sad2 = nullptr;      // original 2-saddle triangles
    i64 *sad1 = nullptr;      // original 1-saddle edges (strict descending checks only)
    i64 capSad1 = 0;
    // separatrix checks (see k_path_detect): the box of bricks of each 2-saddle's
    // paths, and two flags per brick (path_keep: repairs refresh them)
    unsigned long long *path_box = nullptr;
    uint8_t *path_as = nullptr, *path_ds = nullptr;  // one allocation, capB each
    i64 capPB = 0;
    int path_keep = 0;
    Segment *seg = nullptr;  // segments of long paths, capSeg; per 2-saddle with one: capSlot
    i64 *seg_sad = nullptr;
    unsigned long long *seg_res = nullptr;
    i64 capSeg = 0, capSlot = 0;
    i64 *wall_sad = nullptr, *wall_edge = nullptr;  // wall records (preserve_connectors = 1), capWall each
    i64 *wall_next[2] = {nullptr, nullptr};          // 2-saddles handed to the next search tier
    i64 capWall = 0;
    i64 *wall_scratch = nullptr;  // stacks and caches of the larger wall-search tiers
    i64 capWS = 0;
    unsigned long long *counters = nullptr;  // [0..3] cp lists, [4] requests, [5,6] paths, [7] progress,
                                             // [8,9] min/max keys, [10] original 2-saddles, [12] edited
                                             // vertices, [13,14] saddle counts,
                                             // [16] wall records, [17,18] deferred wall searches,
                                             // [20..23] rebuilt mismatch lists, [25,26]
                                             // path segments and their slots, [27] ticket of
                                             // the separatrix walks, [28] original 1-saddles, [29]
                                             // ticket of the strict descending walks, [30] blocks of
                                             // k_round_end that are done
    int *errword = nullptr;
    uint8_t *changed = nullptr;
    int64_t launches = 0;  // kernels launched by the current call
    int tune_shape = 0;    // brick shape (DMTZ_SHAPES) chosen by dmtz_autotune
    int tune_bps = 32;     // sweep blocks per SM
    std::vector<dmtz_ctx *> pool;  // worker contexts of dmtz_correct_batch
    uint8_t *mm = nullptr;         // mismatch bytes of the learned proposal's features
    i64 capMM = 0;
    // results of the calls that hand arrays to the host (pairing arrays, labels):
    // kept between calls up to kWorkKeep bytes, so that a call neither maps nor unmaps memory
    unsigned char *work = nullptr;
    size_t work_bytes = 0;
    unsigned long long *report = nullptr;  // pinned: counts of the last round (k_round_end), hc's layout
    unsigned long long report_seq = 0;       // the last round's end; report[8] once it is done
    std::vector<cudaEvent_t> events;         // of the phase timer
    cudaEvent_t span[2] = {nullptr, nullptr};  // a correction's begin and end
    int short_clusters = 0;        // clusters of k_short_rounds the device holds (0: not asked yet, -1: none)
    int march_blocks = 0;          // blocks of k_grad_march the device holds at once (0: not asked yet)
    void *loopctl = nullptr;       // device copy of the graph loop's control block (kept: a
                                   // cudaFree per call would synchronise the whole device)
};

namespace {

dmtz_status fail(dmtz_ctx *c, dmtz_status s, const std::string &m) {
    if (c) c->err = m;
    return s;
}
#define CK(call)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return fail(ctx, DMTZ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Scratch of one call: take, then cut pieces off it; done gives a large one back.  What is
// kept goes when the context's buffers grow, and when an allocation would fail
// otherwise (dalloc; no call allocates while it uses the scratch).
constexpr size_t kWorkKeep = (size_t)1 << 30;
bool work_free(dmtz_ctx *c) {  // false: there is none
    if (!c->work) return false;
    cudaFree(c->work);
    c->work = nullptr;
    c->work_bytes = 0;
    return true;
}
template <class T>
cudaError_t dalloc(dmtz_ctx *c, T **p, i64 n) {
    return alloc_retry([&]() { return cudaMalloc((void **)p, sizeof(T) * (size_t)std::max<i64>(n, 1)); },
                       [&]() {
                           cudaGetLastError();
                           return work_free(c);
                       });
}

cudaError_t work_take(dmtz_ctx *c, size_t bytes) {
    if (bytes <= c->work_bytes) return cudaSuccess;
    work_free(c);
    const cudaError_t e = cudaMalloc((void **)&c->work, bytes);
    if (e == cudaSuccess) c->work_bytes = bytes;
    return e;
}
void work_done(dmtz_ctx *c) {
    if (c->work_bytes > kWorkKeep) work_free(c);
}
struct WorkDone {  // gives a large scratch back on every way out
    dmtz_ctx *c;
    ~WorkDone() { work_done(c); }
};
size_t work_round(size_t b) { return (b + 255) / 256 * 256; }

void free_field(DevField &d) {
    cudaFree(d.pv); cudaFree(d.eup); cudaFree(d.fup); cudaFree(d.crit); cudaFree(d.tcode);
    d = DevField();
}
void free_all(dmtz_ctx *c) {
    cudaFree(c->f); cudaFree(c->g); free_field(c->P); free_field(c->Q);
    cudaFree(c->cnt); cudaFree(c->reqbits); cudaFree(c->reqlist);
    for (auto &l : c->lists) { cudaFree(l); l = nullptr; }
    for (auto &l : c->list_tmp) { cudaFree(l); l = nullptr; }
    for (auto &k : c->capL) k = 0;
    c->capAS = c->capDS = c->capSad2 = 0;
    cudaFree(c->as_tet); cudaFree(c->as_cur); cudaFree(c->ds_edge); cudaFree(c->ds_vert);
    cudaFree(c->counters); cudaFree(c->errword); cudaFree(c->changed);
    cudaFree(c->sad2); cudaFree(c->brick_flags); cudaFree(c->brick_list);
    cudaFree(c->path_box); cudaFree(c->path_as);
    c->path_box = nullptr; c->path_as = c->path_ds = nullptr;
    cudaFree(c->seg); cudaFree(c->seg_sad); cudaFree(c->seg_res);
    c->seg = nullptr; c->seg_sad = nullptr; c->seg_res = nullptr;
    c->capSeg = c->capSlot = 0;
    c->capPB = 0;
    cudaFree(c->wall_sad); cudaFree(c->wall_edge); cudaFree(c->wall_next[0]); cudaFree(c->wall_next[1]);
    cudaFree(c->wall_scratch);
    c->wall_sad = c->wall_edge = c->wall_next[0] = c->wall_next[1] = c->wall_scratch = nullptr;
    c->capWall = c->capWS = 0;
    cudaFree(c->brick_n);
    c->brick_n = nullptr;
    cudaFree(c->sad1);
    c->sad1 = nullptr;
    c->capSad1 = 0;
    c->sad2 = nullptr; c->brick_flags = nullptr; c->brick_list = nullptr;
    c->f = c->g = nullptr; c->cnt = nullptr; c->reqbits = nullptr; c->reqlist = nullptr;
    c->as_tet = c->as_cur = c->ds_edge = c->ds_vert = nullptr; c->counters = nullptr;
    c->errword = nullptr; c->changed = nullptr;
    c->capV = c->capE = c->capF = c->capT = c->capB = 0;
}

dmtz_status alloc_field(dmtz_ctx *ctx, DevField &d, i64 V) {
    CK(dalloc(ctx, &d.pv, V)); CK(dalloc(ctx, &d.eup, V)); CK(dalloc(ctx, &d.fup, V)); CK(dalloc(ctx, &d.crit, V)); CK(dalloc(ctx, &d.tcode, V));
    return DMTZ_OK;
}

i64 bricks_of(const Grid &g, int shape, int &nbx, int &nby, int &nbz);

// capacity a mismatch list of a dimension with `cells` cells starts with
i64 lean_cap(const dmtz_ctx *ctx, i64 cells) {
    const i64 want = std::max<i64>(ctx->list_min, (i64)((double)cells * ctx->list_frac));
    return std::max<i64>(1, std::min<i64>(cells, want));
}

dmtz_status ensure_lists(dmtz_ctx *ctx, const Grid &g) {
    const i64 cells[4] = {g.V, g.E, g.F, g.T};
    for (int k = 0; k < 4; k++) {
        if (ctx->lists[k]) continue;
        const i64 cap = lean_cap(ctx, cells[k]);
        cudaFree(ctx->list_tmp[k]);
        ctx->list_tmp[k] = nullptr;
        CK(dalloc(ctx, &ctx->lists[k], cap));
        CK(dalloc(ctx, &ctx->list_tmp[k], cap));
        ctx->capL[k] = cap;
    }
    return DMTZ_OK;
}

dmtz_status ensure(dmtz_ctx *ctx, const Grid &g) {
    int nbx, nby, nbz;
    i64 nbr = 0;
    for (int sh = 0; sh < DMTZ_NSHAPES; sh++) nbr = std::max(nbr, bricks_of(g, sh, nbx, nby, nbz));
    if (g.V <= ctx->capV && g.E <= ctx->capE && g.F <= ctx->capF && g.T <= ctx->capT && nbr <= ctx->capB)
        return ensure_lists(ctx, g);
    free_all(ctx);
    work_free(ctx);
    const i64 V = g.V;
    CK(dalloc(ctx, &ctx->f, V)); CK(dalloc(ctx, &ctx->g, V));
    dmtz_status s;
    if ((s = alloc_field(ctx, ctx->P, V)) != DMTZ_OK) return s;
    if ((s = alloc_field(ctx, ctx->Q, V)) != DMTZ_OK) return s;
    CK(dalloc(ctx, &ctx->cnt, V));
    CK(dalloc(ctx, &ctx->reqbits, (V + 31) / 32 + 1));
    CK(cudaMemset(ctx->reqbits, 0, sizeof(uint32_t) * (size_t)((V + 31) / 32 + 1)));
    CK(dalloc(ctx, &ctx->reqlist, V));
    CK(dalloc(ctx, &ctx->brick_flags, (nbr + 3) / 4)); CK(dalloc(ctx, &ctx->brick_list, nbr));
    CK(dalloc(ctx, &ctx->path_as, 2 * nbr));
    ctx->path_ds = ctx->path_as + nbr;
    CK(dalloc(ctx, &ctx->brick_n, 8));
    CK(cudaMemset(ctx->brick_flags, 0, sizeof(uint32_t) * (size_t)((nbr + 3) / 4)));
    ctx->capB = nbr;
    CK(dalloc(ctx, &ctx->counters, 32)); CK(dalloc(ctx, &ctx->errword, 1)); CK(dalloc(ctx, &ctx->changed, V));
    ctx->capV = g.V; ctx->capE = g.E; ctx->capF = g.F; ctx->capT = g.T;
    return ensure_lists(ctx, g);
}

// grow mismatch list k to hold `need` entries; its contents are lost, so the
// caller scans again
dmtz_status grow_list(dmtz_ctx *ctx, const Grid &g, int k, i64 need) {
    const i64 cells[4] = {g.V, g.E, g.F, g.T};
    const i64 cap = std::max<i64>(need, std::min<i64>(cells[k], std::max<i64>(need + need / 2, 2 * ctx->capL[k])));
    cudaFree(ctx->lists[k]);
    cudaFree(ctx->list_tmp[k]);
    ctx->lists[k] = ctx->list_tmp[k] = nullptr;
    ctx->capL[k] = 0;
    CK(dalloc(ctx, &ctx->lists[k], cap));
    CK(dalloc(ctx, &ctx->list_tmp[k], cap));
    ctx->capL[k] = cap;
    return DMTZ_OK;
}

FieldState view(const DevField &d, const double *val) {
    FieldState s;
    s.val = val; s.pv = d.pv; s.eup = d.eup; s.fup = d.fup; s.crit = d.crit; s.tcode = d.tcode;
    return s;
}

unsigned persistent_grid();

i64 bricks_of(const Grid &g, int shape, int &nbx, int &nby, int &nbz) {
    nbx = (g.W + DMTZ_SHAPES[shape][0] - 1) / DMTZ_SHAPES[shape][0];
    nby = (g.H + DMTZ_SHAPES[shape][1] - 1) / DMTZ_SHAPES[shape][1];
    nbz = (g.D + DMTZ_SHAPES[shape][2] - 1) / DMTZ_SHAPES[shape][2];
    return (i64)nbx * nby * nbz;
}
// brick coordinates are packed as bx | by << 11 | bz << 22
bool shape_fits(const Grid &g, int shape) {
    int nbx, nby, nbz;
    bricks_of(g, shape, nbx, nby, nbz);
    return nbx <= 2048 && nby <= 2048 && nbz <= 1024;
}

PathFlags path_flags(const dmtz_ctx *ctx) {
    return PathFlags{ctx->path_as, ctx->path_ds, ctx->P.tcode, ctx->P.pv};
}
LongPaths long_paths(const dmtz_ctx *ctx) {
    return LongPaths{ctx->seg, ctx->seg_sad, ctx->seg_res, ctx->counters + 25, ctx->capSeg, ctx->capSlot};
}
// log2 of the brick extents
void shape_shifts(int shape, int sh[3]) {
    for (int k = 0; k < 3; k++) {
        sh[k] = 0;
        while ((1 << sh[k]) < DMTZ_SHAPES[shape][k]) sh[k]++;
    }
}

// blocks of k_grad_bricks: its blocks hold 384 threads or more, so a quarter
// of tune_bps (a count for blocks of 128) fills the SMs twice over
unsigned brick_grid(const dmtz_ctx *ctx, i64 nb) {
    const unsigned cap = (unsigned)(persistent_grid() / 8) * (unsigned)std::max(1, ctx->tune_bps / 4);
    return (unsigned)std::max<i64>(1, std::min<i64>(nb, cap));
}

// the gradient of a set of bricks (and the old mismatch lists' entries, see KeepOps)
void grad_bricks(const Grid &g, const FieldState &s, const BrickList &bl, unsigned grid, cudaStream_t st,
                 const GradOps &O = GradOps{}, const KeepOps &K = KeepOps{}, const int *wanted = nullptr) {
    grid += K.blocks;
    switch (bl.shape) {
    case 1: launch_next(k_grad_bricks<16, 4, 2>, grid, brick_threads<16, 4, 2>(), st, g, s, bl, O, K, wanted); break;
    case 2: launch_next(k_grad_bricks<32, 2, 2>, grid, brick_threads<32, 2, 2>(), st, g, s, bl, O, K, wanted); break;
    default: launch_next(k_grad_bricks<8, 4, 4>, grid, brick_threads<8, 4, 4>(), st, g, s, bl, O, K, wanted); break;
    }
}

BrickList all_bricks(const Grid &g, int shape, i64 &nb) {
    BrickList bl;
    bl.list = nullptr;
    bl.n = nullptr;
    bl.shape = shape;
    nb = bricks_of(g, shape, bl.nbx, bl.nby, bl.nbz);
    bl.dbx = make_fdiv((unsigned long long)bl.nbx);
    bl.dby = make_fdiv((unsigned long long)bl.nby);
    return bl;
}

// The gradient of the whole grid.  Grids whose bricks fit the GPU in one round
// (three blocks of k_grad_bricks per SM) take one latency of that kernel: 16^3
// 6.2 us, against 14.4 us for the march's five pipeline steps; larger ones
// march (64^3: 25 us, 32 us in bricks; 256^3: 823 us, 1656 us in bricks).
// Tiles of 32 x 16 columns and one block of 640 threads per SM (862 us at 256^3
// when they were compared, 43 us at 97 x 61 x 75): with two blocks and 48 registers 935
// and 51 us, 32 x 8 with three blocks 874 and 51, 64 x 8 1035 and 58.
constexpr int kMarchX = 32, kMarchY = 16, kMarchBlocks = 1;
bool grad_marches(const dmtz_ctx *ctx, const Grid &g) {
    i64 nb;
    all_bricks(g, ctx->tune_shape, nb);
    return nb > (i64)(persistent_grid() / 8) * 3;
}
// Not counted in ctx->launches (also used while capturing the graph loop).
void grad_full(dmtz_ctx *ctx, const Grid &g, const FieldState &s, const GradOps &O = GradOps{}) {
    i64 nb;
    const BrickList bl = all_bricks(g, ctx->tune_shape, nb);
    if (!grad_marches(ctx, g)) {
        grad_bricks(g, s, bl, (unsigned)nb, ctx->stream, O);
        return;
    }
    using M = March<kMarchX, kMarchY>;
    auto plain = k_grad_march<kMarchX, kMarchY, kMarchBlocks, false>;
    auto track = k_grad_march<kMarchX, kMarchY, kMarchBlocks, true>;
    if (!ctx->march_blocks) {
        int per_sm = 0;
        cudaFuncSetAttribute(plain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M::smem);
        cudaFuncSetAttribute(track, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M::smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, plain, M::NT, M::smem);
        ctx->march_blocks = std::max(1, per_sm) * (int)(persistent_grid() / 8);
    }
    const int ntx = (g.W + kMarchX - 1) / kMarchX, nty = (g.H + kMarchY - 1) / kMarchY;
    const i64 tiles = (i64)ntx * nty;
    // planes per block: the fewest steps over all waves (a block's pipeline
    // takes four steps more than it has planes)
    int chunk = 1;
    i64 best = -1;
    for (int c = 1; c <= g.D; c++) {
        const i64 waves = (tiles * ((g.D + c - 1) / c) + ctx->march_blocks - 1) / ctx->march_blocks, cost = waves * (c + 4);
        if (best < 0 || cost < best) {
            best = cost;
            chunk = c;
        }
    }
    const i64 blocks = tiles * ((g.D + chunk - 1) / chunk);
    int sh[3];
    shape_shifts(ctx->tune_shape, sh);
    if (O.critP) {
        if (O.F.as) cudaMemsetAsync(O.F.as, 0, 2 * (size_t)ctx->capB, ctx->stream);
        track<<<(unsigned)blocks, M::NT, M::smem, ctx->stream>>>(g, s, ntx, nty, chunk, O, sh[0], sh[1], sh[2], bl.nbx, bl.nby);
    } else {
        plain<<<(unsigned)blocks, M::NT, M::smem, ctx->stream>>>(g, s, ntx, nty, chunk, O, sh[0], sh[1], sh[2], bl.nbx, bl.nby);
    }
}

Lists mismatch_lists(const dmtz_ctx *ctx) {
    Lists L;
    for (int k = 0; k < 4; k++) {
        L.l[k] = ctx->lists[k];
        L.cap[k] = ctx->capL[k];
    }
    L.n = ctx->counters;
    return L;
}
Lists rebuilt_lists(const dmtz_ctx *ctx) {
    Lists T = mismatch_lists(ctx);
    for (int k = 0; k < 4; k++) T.l[k] = ctx->list_tmp[k];
    T.n = ctx->counters + 20;
    return T;
}
// cells a mismatch list holds, as bits of FieldState::crit
uint32_t want_bits(int want_saddles) { return want_saddles ? 0x3FFFFFFu : (1u | (0x3Fu << 20)); }

// mismatch lists of the decompressed gradient against crit_o
void scan_mismatch(dmtz_ctx *ctx, const Grid &g, const uint32_t *crit_d, const uint32_t *crit_o, int want_saddles) {
    cudaMemsetAsync(ctx->counters, 0, 4 * sizeof(unsigned long long), ctx->stream);
    k_mismatch_scan<<<persistent_grid(), kBlock, 0, ctx->stream>>>(g, crit_d, crit_o, mismatch_lists(ctx), want_saddles);
    ctx->launches++;
}

// full gradient of one field (and its mismatch lists when crit_o is given, and
// the bricks' path flags when they are kept)
void run_pairing(dmtz_ctx *ctx, const Grid &g, const FieldState &s, const uint32_t *crit_o, int want_saddles) {
    GradOps O{};
    if (crit_o) {
        cudaMemsetAsync(ctx->counters, 0, 4 * sizeof(unsigned long long), ctx->stream);
        O.T = mismatch_lists(ctx);
        O.critP = crit_o;
        O.want = want_bits(want_saddles);
        if (ctx->path_keep) O.F = path_flags(ctx);
    }
    grad_full(ctx, g, s, O);
    ctx->launches++;
}

BrickMarks brick_marks(const dmtz_ctx *ctx, const Grid &g) {
    BrickMarks B;
    int nbz, sh[3];
    B.flags = ctx->brick_flags;
    B.list = ctx->brick_list;
    B.n = ctx->brick_n;
    bricks_of(g, ctx->tune_shape, B.nbx, B.nby, nbz);
    shape_shifts(ctx->tune_shape, sh);
    B.shx = sh[0];
    B.shy = sh[1];
    B.shz = sh[2];
    B.lanes = std::min(sh[0], std::min(sh[1], sh[2])) >= 2 ? 8 : 32;
    B.sample = 0;
    return B;
}

// no brick marked and none listed
void clear_marks(dmtz_ctx *ctx) {
    cudaMemsetAsync(ctx->brick_n, 0, sizeof(unsigned long long), ctx->stream);
    cudaMemsetAsync(ctx->brick_flags, 0, (size_t)(ctx->capB + 3) / 4 * sizeof(uint32_t), ctx->stream);
}
// what a repair does besides the gradient
void repair_ops(const dmtz_ctx *ctx, const BrickMarks &B, const uint32_t *crit_o, int want_saddles, GradOps &O, KeepOps &K) {
    if (ctx->path_keep || ctx->inc_scan) O.critP = crit_o;
    if (ctx->path_keep) O.F = path_flags(ctx);
    if (ctx->inc_scan) {
        O.T = rebuilt_lists(ctx);
        O.want = want_bits(want_saddles);
        K.L = mismatch_lists(ctx);
        K.fresh = reinterpret_cast<const uint8_t *>(ctx->brick_flags);
        K.shx = B.shx;
        K.shy = B.shy;
        K.shz = B.shz;
        K.nbx = B.nbx;
        K.nby = B.nby;
        K.blocks = persistent_grid() / 8;
    }
}
// Re-pair only the bricks near the vertices the last update requested (marked
// already by k_apply, or else from ctx->reqlist); the mismatch lists are then rebuilt
// into list_tmp (inc_scan; k_round_end takes them back) or scanned for.  The
// marks are clear at the start (k_round_end, or the caller).
void repair_dirty(dmtz_ctx *ctx, const Grid &g, const FieldState &s, const uint32_t *crit_o, int want_saddles, bool marked,
                  const int *wanted = nullptr) {
    const BrickMarks B = brick_marks(ctx, g);
    cudaStream_t st = ctx->stream;
    i64 nb;
    BrickList bl = all_bricks(g, ctx->tune_shape, nb);
    if (!marked) {
        k_mark_dirty<<<persistent_grid(), kBlock, 0, st>>>(g, B, ctx->reqlist, ctx->counters + 4);
        ctx->launches++;
    }
    bl.list = ctx->brick_list;
    bl.n = ctx->brick_n;
    GradOps O{};
    KeepOps K{};
    repair_ops(ctx, B, crit_o, want_saddles, O, K);
    grad_bricks(g, s, bl, brick_grid(ctx, nb), st, O, K, wanted);
    ctx->launches++;
    if (!ctx->inc_scan) scan_mismatch(ctx, g, s.crit, crit_o, want_saddles);
}
// a round's re-pairing when its lists are long (the whole grid, lists and flags in place)
void repair_full(dmtz_ctx *ctx, const Grid &g, const FieldState &s, const uint32_t *crit_o, int want_saddles) {
    run_pairing(ctx, g, s, crit_o, want_saddles);
}
// Lists with at least this many cells, after a round that reached at least as many bricks
// (before the first: any), mean a repair of the whole grid: the update reaches most bricks
// then, and the march's halo is smaller (256^3: 0.82 ms by the march, 1.66 by all bricks, even
// at half of them).  With separatrices, so and never whole, power-law fields with an SZ-like
// error of 1e-4 of the range: 128^3 (16 k bricks) 1.66 and 1.74 ms, 176^3 (43 k) 3.03 and
// 3.20, 256^3 (131 k) 6.73 and 7.45; with uniform noise of 1e-2: 7.5 and 8.2, 15.3 and 17.3,
// 39.9 and 48.2.  The cells alone do not say it: in a Gaussian mixture with uniform noise of 1e-3
// they crowd where the field is flat, and 600 rounds on its extrema took 63 ms at 104^3 (8.8 k
// bricks), 87 at 128^3 and 157 at 176^3 by the cells alone, 32, 42 and 74 so.
// Below 8192 bricks such grids are always repaired by bricks: 64^3 (2048 bricks) within 2 %
// either way, 96^3 (6912) within 4 %, 7 % slower by bricks for extrema in noise everywhere.
i64 heavy_cells(const dmtz_ctx *ctx, const Grid &g) {
    i64 nb;
    all_bricks(g, ctx->tune_shape, nb);
    return nb >= 8192 ? nb / 2 : INT64_MAX;
}
// The marks of a round that re-pairs the whole grid: up to 4096 blocks of bricks, from twice
// as many of the requests.  They are listed and cleared as bricks are (a block's coordinates
// are a brick's, too).  *bricks: how many bricks a block stands for.  (With the bricks of all
// requests 28 rounds at 256^3 took 22.2 ms, with half as many requests as bricks 20.5, so 19.8;
// without marks 19.7.)
BrickMarks sampled_marks(const dmtz_ctx *ctx, const Grid &g, i64 *bricks) {
    BrickMarks B = brick_marks(ctx, g);
    i64 nb, blocks;
    const BrickList bl = all_bricks(g, ctx->tune_shape, nb);
    for (int k = 0;; k++, B.shx++, B.shy++, B.shz++) {
        auto up = [&](int n) { return (i64)((n + (1 << k) - 1) >> k); };
        blocks = up(bl.nbx) * up(bl.nby) * up(bl.nbz);
        if (blocks <= 4096) break;
    }
    B.sample = 2 * blocks;
    *bricks = nb / blocks;
    return B;
}

double key_to_double(unsigned long long k) {
    uint64_t b = (k & 0x8000000000000000ull) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
    double d;
    memcpy(&d, &b, 8);
    return d;
}

// min and max of a device field (exact)
dmtz_status device_minmax(dmtz_ctx *ctx, const double *a, i64 n, double &mn, double &mx) {
    unsigned long long init[2] = {~0ull, 0ull}, out[2];
    CK(cudaMemcpyAsync(ctx->counters + 8, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
    k_minmax<<<persistent_grid(), kBlock, 0, ctx->stream>>>(a, n, ctx->counters + 8, ctx->counters + 9);
    ctx->launches++;
    CK(cudaMemcpyAsync(out, ctx->counters + 8, sizeof(out), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    mn = key_to_double(out[0]);
    mx = key_to_double(out[1]);
    return DMTZ_OK;
}

RuleCtx rule_ctx(dmtz_ctx *ctx, const Grid &g, double bound, int edit_type) {
    RuleCtx c;
    c.g = g;
    c.P = view(ctx->P, ctx->f);
    c.Q = view(ctx->Q, ctx->g);
    c.f = ctx->f;
    c.gv = ctx->g;
    c.cnt = ctx->cnt;
    c.bound = bound;
    c.edit_type = edit_type;
    c.reqbits = ctx->reqbits;
    c.reqlist = ctx->reqlist;
    c.reqn = ctx->counters + 4;
    c.reqcap = g.V;
    c.err = ctx->errword;
    c.progress = ctx->counters + 7;
    return c;
}

// After a scan that left its counts in hc[0..3]: grow every overflowed list
// and scan again (same masks, so the same counts, which now fit).
dmtz_status fit_lists(dmtz_ctx *ctx, const Grid &g, int want_saddles, unsigned long long *hc) {
    bool over = false;
    for (int k = 0; k < 4; k++) {
        if ((i64)hc[k] <= ctx->capL[k]) continue;
        dmtz_status s = grow_list(ctx, g, k, (i64)hc[k]);
        if (s != DMTZ_OK) return s;
        over = true;
    }
    if (!over) return DMTZ_OK;
    scan_mismatch(ctx, g, ctx->Q.crit, ctx->P.crit, want_saddles);
    CK(cudaMemcpyAsync(hc, ctx->counters, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return DMTZ_OK;
}

CpLists cp_lists(const dmtz_ctx *ctx) {
    CpLists L;
    for (int k = 0; k < 4; k++) {
        L.l[k] = ctx->lists[k];
        L.cap[k] = ctx->capL[k];
    }
    L.n = ctx->counters;
    return L;
}

PathRec path_rec(const dmtz_ctx *ctx) {
    return PathRec{ctx->as_tet, ctx->as_cur, ctx->ds_edge, ctx->ds_vert, ctx->counters + 5, ctx->capAS, ctx->capDS};
}

// The original paths' marks, boxes and segments (after the 2-saddle list).
// Room for the segments: what the last field needed, at first one per 16 vertices
// and 2-saddle slot per 64; a trace that needs more is repeated.
dmtz_status trace_paths(dmtz_ctx *ctx, const Grid &g) {
    cudaStream_t st = ctx->stream;
    i64 need_seg = std::max<i64>(g.V / 16, 1024), need_slot = std::max<i64>(g.V / 64, 256);
    int sh[3];
    shape_shifts(ctx->tune_shape, sh);
    while (true) {
        if (need_seg > ctx->capSeg) {
            cudaFree(ctx->seg);
            ctx->seg = nullptr;
            ctx->capSeg = 0;
            CK(dalloc(ctx, &ctx->seg, need_seg));
            ctx->capSeg = need_seg;
        }
        if (need_slot > ctx->capSlot) {
            cudaFree(ctx->seg_sad);
            cudaFree(ctx->seg_res);
            ctx->seg_sad = nullptr;
            ctx->seg_res = nullptr;
            ctx->capSlot = 0;
            CK(dalloc(ctx, &ctx->seg_sad, need_slot));
            CK(dalloc(ctx, &ctx->seg_res, need_slot));
            ctx->capSlot = need_slot;
        }
        CK(cudaMemsetAsync(ctx->counters + 25, 0, 3 * sizeof(unsigned long long), st));  // segments, slots, ticket
        k_path_trace<<<persistent_grid(), kBlock, 0, st>>>(g, ctx->sad2, ctx->counters + 10, ctx->capSad2, ctx->P.tcode,
                                                           ctx->path_box, long_paths(ctx), sh[0], sh[1], sh[2], g.T + 16,
                                                           ctx->errword, ctx->counters + 27);
        ctx->launches++;
        unsigned long long n[2] = {0, 0};
        CK(cudaMemcpyAsync(n, ctx->counters + 25, sizeof(n), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        CK(cudaGetLastError());
        if ((i64)n[0] <= ctx->capSeg && (i64)n[1] <= ctx->capSlot) return DMTZ_OK;
        need_seg = std::max<i64>(need_seg, (i64)n[0]);
        need_slot = std::max<i64>(need_slot, (i64)n[1]);
    }
}

// Separatrix records' buffers, sized by the original saddle counts (each original
// 2-saddle gives at most one ascending record, each 1-saddle at most one descending
// record), the lists of the original saddles, and, where the geometry-mode checks
// will read them, the original paths (after the original pairing).  Connectivity mode
// and the walls do not (a connectivity correction at 256^3: 20.5 ms with the trace, 19.5
// without, and 2 bytes per vertex less)
dmtz_status prep_paths(dmtz_ctx *ctx, const Grid &g, bool trace) {
    cudaStream_t st = ctx->stream;
    CK(cudaMemsetAsync(ctx->counters + 13, 0, 2 * sizeof(unsigned long long), st));
    k_count_saddles<<<persistent_grid(), kBlock, 0, st>>>(g.V, ctx->P.crit, ctx->counters + 13);
    unsigned long long n[2] = {0, 0};
    CK(cudaMemcpyAsync(n, ctx->counters + 13, sizeof(n), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if ((i64)n[0] > ctx->capDS) {
        cudaFree(ctx->ds_edge);
        cudaFree(ctx->ds_vert);
        ctx->ds_edge = ctx->ds_vert = nullptr;
        ctx->capDS = 0;
        CK(dalloc(ctx, &ctx->ds_edge, (i64)n[0]));
        CK(dalloc(ctx, &ctx->ds_vert, (i64)n[0]));
        ctx->capDS = (i64)n[0];
    }
    if ((i64)n[1] > ctx->capAS) {
        cudaFree(ctx->as_tet);
        cudaFree(ctx->as_cur);
        ctx->as_tet = ctx->as_cur = nullptr;
        ctx->capAS = 0;
        CK(dalloc(ctx, &ctx->as_tet, (i64)n[1]));
        CK(dalloc(ctx, &ctx->as_cur, (i64)n[1]));
        ctx->capAS = (i64)n[1];
    }
    // (of its own: a connectivity check grows the records alone)
    if ((i64)n[1] > ctx->capSad2) {
        cudaFree(ctx->sad2);
        ctx->sad2 = nullptr;
        ctx->capSad2 = 0;
        CK(dalloc(ctx, &ctx->sad2, (i64)n[1]));
        ctx->capSad2 = (i64)n[1];
    }
    // buffers exist even when a count is 0 (kernels take their addresses)
    if (!ctx->ds_edge) {
        CK(dalloc(ctx, &ctx->ds_edge, 1));
        CK(dalloc(ctx, &ctx->ds_vert, 1));
    }
    if (!ctx->as_tet) {
        CK(dalloc(ctx, &ctx->as_tet, 1));
        CK(dalloc(ctx, &ctx->as_cur, 1));
    }
    if (!ctx->sad2) CK(dalloc(ctx, &ctx->sad2, 1));
    const i64 nbox = std::max<i64>((i64)n[1], 1);
    if (trace && nbox > ctx->capPB) {
        cudaFree(ctx->path_box);
        ctx->path_box = nullptr;
        ctx->capPB = 0;
        CK(dalloc(ctx, &ctx->path_box, nbox));
        ctx->capPB = nbox;
    }
    CK(cudaMemsetAsync(ctx->counters + 10, 0, sizeof(unsigned long long), st));
    k_crit_list<8, 12><<<persistent_grid(), kBlock, 0, st>>>(g, ctx->P.crit, ctx->sad2, ctx->capSad2,
                                                             ctx->counters + 10);
    if (ctx->strict_ds) {  // the whole-path descending checks walk from the 1-saddle list
        const i64 need = std::max<i64>((i64)n[0], 1);
        if (need > ctx->capSad1) {
            cudaFree(ctx->sad1);
            ctx->sad1 = nullptr;
            ctx->capSad1 = 0;
            CK(dalloc(ctx, &ctx->sad1, need));
            ctx->capSad1 = need;
        }
        CK(cudaMemsetAsync(ctx->counters + 28, 0, sizeof(unsigned long long), st));
        k_crit_list<1, 7><<<persistent_grid(), kBlock, 0, st>>>(g, ctx->P.crit, ctx->sad1, ctx->capSad1,
                                                                ctx->counters + 28);
        ctx->launches++;
    }
    ctx->launches += 2;
    CK(cudaGetLastError());
    return trace ? trace_paths(ctx, g) : DMTZ_OK;
}

// separatrix detection (ascending and descending) into the path records
// geometry mode (conn = 0) or connectivity mode (conn = 1); no launch counting
// (also used while capturing the graph loop)
// (counters 5, 6 and 27 are zero: the caller, or the round's end in the graph loop)
void launch_detect(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, const PathRec &R, unsigned grid, int conn) {
    cudaStream_t st = ctx->stream;
    if (conn) {
        k_conn_as<<<grid, kBlock, 0, st>>>(g, ctx->P.crit, ctx->Q.crit, ctx->P.tcode, ctx->Q.tcode, R,
                                           g.T + 16, ctx->errword);
        k_conn_ds<<<grid, kBlock, 0, st>>>(rc, R, g.V + 16);
    } else {
        int nbx, nby, nbz;
        const int shape = ctx->tune_shape, *sx = DMTZ_SHAPES[shape];
        const i64 nb = bricks_of(g, shape, nbx, nby, nbz);
        const int ds_blocks = ctx->strict_ds ? 0 : (int)std::min<i64>((nb + 255) / 256, grid / 8);
        k_path_detect<<<grid + (unsigned)ds_blocks, kBlock, 0, st>>>(g, path_flags(ctx), ctx->sad2, ctx->counters + 10,
                                                                     ctx->capSad2, ctx->path_box, ctx->P.crit, ctx->Q.tcode,
                                                                     ctx->Q.pv, long_paths(ctx), R, ctx->counters + 27, nbx,
                                                                     nby, nbz, sx[0], sx[1], sx[2], ds_blocks);
        k_path_long<<<grid / 8, kBlock, 0, st>>>(g, long_paths(ctx), R);
        if (ctx->strict_ds) {  // whole-path descending checks of every 1-saddle, into the records
            cudaMemsetAsync(ctx->counters + 29, 0, sizeof(unsigned long long), st);  // the walks' ticket
            k_ds_strict<<<grid, kBlock, 0, st>>>(rc, R, ctx->sad1, ctx->counters + 28, g.V + 16,
                                                 ctx->counters + 29);
        }
    }
}
// kernels one detection launches
int detect_kernels(const dmtz_ctx *ctx, int conn) { return conn ? 2 : (ctx->strict_ds ? 3 : 2); }
void detect_paths(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, const PathRec &R, unsigned grid, int conn = 0) {
    cudaMemsetAsync(ctx->counters + 5, 0, 2 * sizeof(unsigned long long), ctx->stream);
    cudaMemsetAsync(ctx->counters + 27, 0, sizeof(unsigned long long), ctx->stream);
    launch_detect(ctx, g, rc, R, grid, conn);
    ctx->launches += detect_kernels(ctx, conn);
}

// Wall records (preserve_connectors = 1) of the current decompressed gradient:
// every original 2-saddle searched by tiers (see wall_dfs).  Record arrays
// hold one entry per original 2-saddle; the deferred lists likewise.
dmtz_status ensure_walls(dmtz_ctx *ctx) {
    const i64 need = std::max<i64>(ctx->capSad2, 1);
    if (ctx->capWall >= need) return DMTZ_OK;
    cudaFree(ctx->wall_sad); cudaFree(ctx->wall_edge); cudaFree(ctx->wall_next[0]); cudaFree(ctx->wall_next[1]);
    ctx->wall_sad = ctx->wall_edge = ctx->wall_next[0] = ctx->wall_next[1] = nullptr;
    ctx->capWall = 0;
    CK(dalloc(ctx, &ctx->wall_sad, need));
    CK(dalloc(ctx, &ctx->wall_edge, need));
    CK(dalloc(ctx, &ctx->wall_next[0], need));
    CK(dalloc(ctx, &ctx->wall_next[1], need));
    ctx->capWall = need;
    return DMTZ_OK;
}
WallRec wall_rec(dmtz_ctx *ctx) {
    WallRec W;
    W.sad = ctx->wall_sad;
    W.edge = ctx->wall_edge;
    W.n = ctx->counters + 16;
    W.cap = ctx->capWall;
    return W;
}
unsigned persistent_grid();
dmtz_status detect_walls(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, i64 &n_wall) {
    struct Tier {
        int stack_cap, cache_bits;
        long long pop_cap;
    };
    static const Tier tiers[3] = {{2048, 13, 1ll << 16}, {1 << 16, 18, 1ll << 22}, {1 << 21, 23, 1ll << 28}};
    const i64 budget = (i64)32 << 20;  // scratch entries (256 MB)
    cudaStream_t st = ctx->stream;
    dmtz_status s;
    if ((s = ensure_walls(ctx)) != DMTZ_OK) return s;
    const WallRec W = wall_rec(ctx);
    CK(cudaMemsetAsync(ctx->counters + 16, 0, 3 * sizeof(unsigned long long), st));
    k_wall_t1<<<persistent_grid(), kBlock, 0, st>>>(rc, ctx->sad2, ctx->counters + 10, ctx->capSad2, W,
                                                     ctx->wall_next[0], ctx->counters + 17, ctx->capWall);
    ctx->launches++;
    unsigned long long nd = 0;
    CK(cudaMemcpyAsync(&nd, ctx->counters + 17, sizeof(nd), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int cur = 0;
    for (int t = 0; t < 3 && nd > 0; t++) {
        const Tier &T = tiers[t];
        const i64 per = (i64)T.stack_cap + ((i64)1 << T.cache_bits);
        const i64 chunk = std::max<i64>(1, std::min<i64>((i64)nd, budget / per));
        if (ctx->capWS < chunk * per) {
            cudaFree(ctx->wall_scratch);
            ctx->wall_scratch = nullptr;
            ctx->capWS = 0;
            CK(dalloc(ctx, &ctx->wall_scratch, chunk * per));
            ctx->capWS = chunk * per;
        }
        unsigned long long *nnext = ctx->counters + 17 + (cur ^ 1);
        CK(cudaMemsetAsync(nnext, 0, sizeof(unsigned long long), st));
        for (i64 first = 0; first < (i64)nd; first += chunk) {
            const i64 cnt = std::min<i64>(chunk, (i64)nd - first);
            k_wall_tn<<<grid_for(cnt), kBlock, 0, st>>>(rc, ctx->wall_next[cur], first, cnt, W, ctx->wall_next[cur ^ 1],
                                                        nnext, ctx->capWall, ctx->wall_scratch, T.stack_cap,
                                                        T.cache_bits, T.pop_cap);
            ctx->launches++;
        }
        CK(cudaMemcpyAsync(&nd, nnext, sizeof(nd), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        cur ^= 1;
    }
    if (nd > 0) return fail(ctx, DMTZ_ERR_TOO_LARGE, "a wall search outgrew its largest tier (2^21 stack entries)");
    unsigned long long nw = 0;
    CK(cudaMemcpyAsync(&nw, ctx->counters + 16, sizeof(nw), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    CK(cudaGetLastError());
    n_wall = (i64)nw;
    return DMTZ_OK;
}

unsigned persistent_grid() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (unsigned)sms * 8;
}

dmtz_status check_dims(dmtz_ctx *ctx, int W, int H, int D, Grid &g) {
    if (!ctx) return DMTZ_ERR_ARG;
    if (W < 2 || H < 2 || D < 2) return fail(ctx, DMTZ_ERR_ARG, "dims must be >= 2");
    g = make_grid(W, H, D);
    if (!shape_fits(g, 0)) return fail(ctx, DMTZ_ERR_ARG, "dims exceed 16384 x 8192 x 4096");
    if (!shape_fits(g, ctx->tune_shape)) ctx->tune_shape = 0;
    return DMTZ_OK;
}

// NaN / Inf test of a device field (the reference assumes finite input)
dmtz_status check_finite(dmtz_ctx *ctx, const double *d, i64 n) {
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), ctx->stream));
    k_check_finite<<<persistent_grid(), kBlock, 0, ctx->stream>>>(d, n, ctx->errword);
    ctx->launches++;
    int bad = 0;
    CK(cudaMemcpyAsync(&bad, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (bad) return fail(ctx, DMTZ_ERR_ARG, "input contains NaN or Inf");
    return DMTZ_OK;
}

dmtz_status upload(dmtz_ctx *ctx, double *dst, const double *src, i64 n, int on_device) {
    CK(cudaMemcpyAsync(dst, src, sizeof(double) * (size_t)n, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), ctx->stream));
    k_check_finite<<<persistent_grid(), kBlock, 0, ctx->stream>>>(dst, n, ctx->errword);
    ctx->launches++;
    int bad = 0;
    CK(cudaMemcpyAsync(&bad, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (bad) return fail(ctx, DMTZ_ERR_ARG, "input contains NaN or Inf");
    return DMTZ_OK;
}

}  // namespace

// =============================================================================
// C ABI
// =============================================================================
// Link components of every vertex (no counterpart in the reference, which
// classifies cells by the discrete gradient; this is the piecewise-linear
// reading of "min / max / saddle from the lower and upper link").  The
// Freudenthal triangulation is a flag complex, so the link of v has an edge
// between two stencil neighbours exactly when they are adjacent, and a
// triangle for every adjacent triple.  Lower (upper) link: the neighbours
// below (above) v in compare_vertices order (main_3d.cu:1043-1049).
namespace lnk {
__host__ __device__ constexpr uint32_t adj(int i) {
    uint32_t m = 0;
    for (int j = 0; j < 14; j++)
        if (j != i && cxt::cdir(cxt::TOPO_DIRS[i][0] - cxt::TOPO_DIRS[j][0], cxt::TOPO_DIRS[i][1] - cxt::TOPO_DIRS[j][1],
                                cxt::TOPO_DIRS[i][2] - cxt::TOPO_DIRS[j][2]) >= 0)
            m |= 1u << j;
    return m;
}
// the n-th adjacent triple i < j < k (packed i | j << 4 | k << 8), -1 past the end
__host__ __device__ constexpr int tri(int n) {
    for (int i = 0; i < 14; i++)
        for (int j = i + 1; j < 14; j++)
            for (int k = j + 1; k < 14; k++)
                if (((adj(i) >> j) & 1u) && ((adj(i) >> k) & 1u) && ((adj(j) >> k) & 1u) && n-- == 0)
                    return i | (j << 4) | (k << 8);
    return -1;
}
__host__ __device__ constexpr int ntri() {
    int n = 0;
    while (tri(n) >= 0) n++;
    return n;
}
// the neighbours reachable from `seed` inside m
__device__ __forceinline__ uint32_t grow(uint32_t seed, uint32_t m) {
    uint32_t comp = seed, prev = 0;
    while (comp != prev) {
        prev = comp;
        uint32_t nb = comp;
        DMTZ_FOR(14, I, {
            constexpr int i = decltype(I)::value;
            nb |= ((comp >> i) & 1u) ? adj(i) : 0u;
        });
        comp = nb & m;
    }
    return comp;
}
__device__ __forceinline__ int components(uint32_t m) {
    int c = 0;
    while (m) {
        m &= ~grow(m & (0u - m), m);
        c++;
    }
    return c;
}
// Euler characteristic of the link's full subcomplex on m
__device__ __forceinline__ int chi(uint32_t m) {
    int e2 = 0, t = 0;
    DMTZ_FOR(14, I, {
        constexpr int i = decltype(I)::value;
        e2 += ((m >> i) & 1u) ? __popc(adj(i) & m) : 0;
    });
    DMTZ_FOR(ntri(), N, {
        constexpr int p = tri(decltype(N)::value);
        t += (int)((m >> (p & 15)) & (m >> ((p >> 4) & 15)) & (m >> (p >> 8)) & 1u);
    });
    return __popc(m) - e2 / 2 + t;
}
}  // namespace lnk

__global__ void k_link_classes(Grid g, const double *data, uint8_t *out, unsigned long long *counts) {
    long long c[6] = {0, 0, 0, 0, 0, 0};
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        int x, y, z;
        decode_v(g, v, x, y, z);
        const uint64_t kv = okey(data[v]);
        uint32_t lo = 0, up = 0;
        DMTZ_FOR(14, I, {
            constexpr int i = decltype(I)::value;
            constexpr int dx = cxt::TOPO_DIRS[i][0], dy = cxt::TOPO_DIRS[i][1], dz = cxt::TOPO_DIRS[i][2];
            if (inb(g, x + dx, y + dy, z + dz)) {
                const uint64_t kn = okey(data[v + dx + dy * (i64)g.W + dz * g.WH]);
                const bool below = cxt::dir_up(i) ? (kn < kv) : (kn <= kv);
                lo |= below ? (1u << i) : 0u;
                up |= below ? 0u : (1u << i);
            }
        });
        const int cl = lnk::components(lo), cu = lnk::components(up);
        if (out) out[v] = (uint8_t)(cl | (cu << 4));
        c[0] += cl == 0;
        c[1] += cu == 0;
        c[2] += cl == 1 && cu == 1;
        c[3] += cl >= 2 ? cl - 1 : 0;
        c[4] += cu >= 2 ? cu - 1 : 0;
        c[5] += 1 - lnk::chi(lo);
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
        long long x = c[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(counts + k, (unsigned long long)x);
    }
}

// Separatrix agreement of two gradients (measurement and acceptance checks;
// no counterpart in the reference): per original 1-saddle edge, the descending
// labels of its two endpoints, and per original 2-saddle triangle, the
// ascending labels of its cofaces, in the original field (dP, aP) and in the
// decompressed one (dQ, aQ).  out: [0] endpoints compared, [1] equal, [2]
// cofaces compared, [3] equal, [4] anchor cells whose criticality differs.
// A lane walks its own cells (two at most in most vertices), edges and triangles by
// the same loads with offsets from a table: with a branch per cell of the anchor, a
// warp waited for its loads nineteen times (160 x 144 x 129: 181 us, so: 101).
template <class I>
__global__ void __launch_bounds__(kBlock) k_sep_agree(Grid g, const uint32_t *critP, const uint32_t *critQ, const I *dP,
                                                     const I *dQ, const I *aP, const I *aQ, unsigned long long *out) {
    __shared__ RuleTab tab;
    load_rule_tab(tab);
    unsigned long long c[5] = {0, 0, 0, 0, 0};
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += (i64)gridDim.x * blockDim.x) {
        const uint32_t cp = critP[v];
        c[4] += __popc(cp ^ critQ[v]);
        uint32_t m = (cp >> 1) & 0x7FFFFu;  // 7 edges, 12 triangles
        if (!m) continue;
        int x, y, z;
        decode_v(g, v, x, y, z);
        for (; m; m &= m - 1) {
            const int b = __ffs(m) - 1;
            const bool edge = b < 7;
            const I *p = edge ? dP : aP, *q = edge ? dQ : aQ;
            i64 at[2];
            bool in[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                // an edge's corner, or a triangle's coface (offset + 1, two bits each; slot)
                const unsigned e = edge ? tab.edge[b] >> (3 * j) : tab.fcof[(b - 7) * 2 + j];
                const int dx = edge ? e & 1u : (int)(e & 3u) - 1, dy = edge ? (e >> 1) & 1u : (int)((e >> 2) & 3u) - 1,
                          dz = edge ? (e >> 2) & 1u : (int)((e >> 4) & 3u) - 1;
                const i64 u = v + dx + dy * (i64)g.W + dz * g.WH;
                in[j] = edge || cell_ok(g, x + dx, y + dy, z + dz, 1, 1, 1);
                at[j] = edge ? u : u * 6 + (int)(e >> 6);
            }
            I l[4];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                l[2 * j] = in[j] ? p[at[j]] : 0;
                l[2 * j + 1] = in[j] ? q[at[j]] : 0;
            }
            const unsigned n = in[0] + in[1], same = (in[0] && l[0] == l[1]) + (in[1] && l[2] == l[3]);
            c[0] += edge ? n : 0u;
            c[1] += edge ? same : 0u;
            c[2] += edge ? 0u : n;
            c[3] += edge ? 0u : same;
        }
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
        unsigned long long x = c[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(out + k, x);
    }
}

extern "C" {

dmtz_status dmtz_ctx_create(dmtz_ctx **out, int device) {
    if (!out) return DMTZ_ERR_ARG;
    *out = nullptr;
    dmtz_ctx *ctx = new dmtz_ctx();
    ctx->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete ctx;
        return DMTZ_ERR_CUDA;
    }
    *out = ctx;
    return DMTZ_OK;
}

void dmtz_ctx_destroy(dmtz_ctx *ctx) {
    if (!ctx) return;
    for (dmtz_ctx *w : ctx->pool) dmtz_ctx_destroy(w);
    ctx->pool.clear();
    cudaSetDevice(ctx->device);
    free_all(ctx);
    cudaFree(ctx->mm);
    cudaFree(ctx->loopctl);
    cudaFree(ctx->work);
    cudaFreeHost(ctx->report);
    for (cudaEvent_t e : ctx->events) cudaEventDestroy(e);
    for (cudaEvent_t e : ctx->span)
        if (e) cudaEventDestroy(e);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    if (ctx->side) cudaStreamDestroy(ctx->side);
    if (ctx->side_done) cudaEventDestroy(ctx->side_done);
    delete ctx;
}

const char *dmtz_last_error(const dmtz_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

dmtz_status dmtz_cell_counts(int W, int H, int D, int64_t out[4]) {
    if (W < 2 || H < 2 || D < 2 || !out) return DMTZ_ERR_ARG;
    Grid g = make_grid(W, H, D);
    out[0] = g.V; out[1] = g.E; out[2] = g.F; out[3] = g.T;
    return DMTZ_OK;
}

dmtz_status dmtz_extract(dmtz_ctx *ctx, int W, int H, int D, const double *data, int on_device, int32_t *PV,
                         int32_t *PE, int32_t *PF, int32_t *PT) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (g.F >= INT32_MAX) return fail(ctx, DMTZ_ERR_ARG, "grid too large for 32-bit reference ids");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, data, g.V, on_device)) != DMTZ_OK) return s;
    FieldState fs = view(ctx->P, ctx->f);
    run_pairing(ctx, g, fs, nullptr, 1);
    int32_t *d[4];
    const i64 n[4] = {g.V, g.E, g.F, g.T};
    size_t at[5] = {0, 0, 0, 0, 0};
    for (int k = 0; k < 4; k++) at[k + 1] = at[k] + work_round(sizeof(int32_t) * (size_t)n[k]);
    WorkDone done{ctx};
    CK(work_take(ctx, at[4]));
    for (int k = 0; k < 4; k++) d[k] = reinterpret_cast<int32_t *>(ctx->work + at[k]);
    k_export<<<grid_for(g.V), kBlock, 0, ctx->stream>>>(g, fs, d[0], d[1], d[2], d[3]);
    int32_t *h[4] = {PV, PE, PF, PT};
    for (int k = 0; k < 4; k++)
        CK(cudaMemcpyAsync(h[k], d[k], sizeof(int32_t) * (size_t)n[k], cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaGetLastError());
    return DMTZ_OK;
}

// shared set-up of the two complexes for the parity entry points
// (paths: with the records' buffers and the saddle lists; and the original paths and the bricks' path flags)
enum { NO_PATHS = 0, PATH_LISTS, PATHS_TRACED };
static dmtz_status setup_pair(dmtz_ctx *ctx, const Grid &g, const double *orig, const double *decp, int paths = NO_PATHS) {
    dmtz_status s;
    ctx->path_keep = 0;
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, orig, g.V, 0)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->g, decp, g.V, 0)) != DMTZ_OK) return s;
    run_pairing(ctx, g, view(ctx->P, ctx->f), nullptr, 1);
    if (paths) {
        CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), ctx->stream));
        if ((s = prep_paths(ctx, g, paths == PATHS_TRACED)) != DMTZ_OK) return s;
        ctx->path_keep = paths == PATHS_TRACED;
    }
    run_pairing(ctx, g, view(ctx->Q, ctx->g), ctx->P.crit, 1);
    ctx->path_keep = 0;
    CK(cudaGetLastError());
    unsigned long long hc[4];
    CK(cudaMemcpyAsync(hc, ctx->counters, sizeof(hc), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return fit_lists(ctx, g, 1, hc);
}

// the reference ids of a list's first out.size() cells (their codes are gone then)
static dmtz_status fetch_refs(dmtz_ctx *ctx, const Grid &g, i64 *codes, std::vector<i64> &out) {
    const i64 n = (i64)out.size();
    k_refs<<<std::min(grid_for(n), persistent_grid()), kBlock, 0, ctx->stream>>>(g, codes, n);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(out.data(), codes, sizeof(i64) * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return DMTZ_OK;
}

dmtz_status dmtz_mismatch(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                          int64_t counts[4], int32_t *lmin, int32_t *lsad, int32_t *l2sad, int32_t *lmax) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    CK(cudaSetDevice(ctx->device));
    if ((s = setup_pair(ctx, g, orig, decp)) != DMTZ_OK) return s;
    unsigned long long hc[4];
    CK(cudaMemcpyAsync(hc, ctx->counters, sizeof(hc), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    int32_t *outs[4] = {lmin, lsad, l2sad, lmax};
    for (int k = 0; k < 4; k++) {
        counts[k] = (int64_t)hc[k];
        if (!outs[k] || !hc[k]) continue;
        std::vector<i64> tmp(hc[k]);
        if ((s = fetch_refs(ctx, g, ctx->lists[k], tmp)) != DMTZ_OK) return s;
        std::sort(tmp.begin(), tmp.end());
        for (size_t i = 0; i < tmp.size(); i++) outs[k][i] = (int32_t)tmp[i];
    }
    return DMTZ_OK;
}

static void host_minmax(const double *f, i64 n, double &mn, double &mx) {
    mn = f[0]; mx = f[0];
    for (i64 i = 1; i < n; i++) {
        if (f[i] < mn) mn = f[i];
        if (f[i] > mx) mx = f[i];
    }
}

dmtz_status dmtz_fix_round(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                           const int32_t *edit_counter, double rel_eps, int preserve_saddles, int edit_type,
                           double *delta_out) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    CK(cudaSetDevice(ctx->device));
    if ((s = setup_pair(ctx, g, orig, decp)) != DMTZ_OK) return s;
    double mn, mx;
    host_minmax(orig, g.V, mn, mx);
    const double range = mx - mn, bound = (mx - mn) * rel_eps;
    CK(cudaMemcpyAsync(ctx->cnt, edit_counter, sizeof(int) * (size_t)g.V, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemsetAsync(ctx->counters + 4, 0, sizeof(unsigned long long), ctx->stream));
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), ctx->stream));
    RuleCtx rc = rule_ctx(ctx, g, bound, edit_type);
    k_fix_cp<<<persistent_grid(), kBlock, 0, ctx->stream>>>(rc, cp_lists(ctx), preserve_saddles);
    double *dd = nullptr;
    CK(dalloc(ctx, &dd, g.V));
    const double sentinel = -2000.0 * range;
    std::vector<double> fill((size_t)g.V, sentinel);
    CK(cudaMemcpyAsync(dd, fill.data(), sizeof(double) * (size_t)g.V, cudaMemcpyHostToDevice, ctx->stream));
    // report the deltas the rules requested, without updating the field
    k_apply<false><<<persistent_grid(), kBlock, 0, ctx->stream>>>(rc, range, 0, 0, nullptr, dd, BrickMarks{});
    CK(cudaMemcpyAsync(delta_out, dd, sizeof(double) * (size_t)g.V, cudaMemcpyDeviceToHost, ctx->stream));
    int err = 0;
    CK(cudaMemcpyAsync(&err, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    cudaFree(dd);
    CK(cudaGetLastError());
    if (err & ERR_OOB) return fail(ctx, DMTZ_ERR_OOB, "a fix rule indexed out of range");
    return DMTZ_OK;
}

static dmtz_status path_detect_impl(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                                    int conn, int64_t counts[2], int32_t *as_tet, int32_t *as_cur, int32_t *ds_edge,
                                    int32_t *ds_vert, int strict = 0) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    ctx->strict_ds = strict && !conn;
    CK(cudaSetDevice(ctx->device));
    if ((s = setup_pair(ctx, g, orig, decp, conn ? PATH_LISTS : PATHS_TRACED)) != DMTZ_OK) return s;
    RuleCtx rc = rule_ctx(ctx, g, 0.0, 0);
    unsigned long long hc[2];
    int err = 0;
    for (int attempt = 0; attempt < 2; attempt++) {
        detect_paths(ctx, g, rc, path_rec(ctx), persistent_grid(), conn);
        CK(cudaMemcpyAsync(hc, ctx->counters + 5, sizeof(hc), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaMemcpyAsync(&err, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        // connectivity mode walks from the decompressed 2-saddles, which may
        // outnumber the original ones the records were sized for: grow, redo
        if ((i64)hc[0] <= ctx->capAS && (i64)hc[1] <= ctx->capDS) break;
        if ((i64)hc[0] > ctx->capAS) {
            cudaFree(ctx->as_tet);
            cudaFree(ctx->as_cur);
            ctx->as_tet = ctx->as_cur = nullptr;
            ctx->capAS = 0;
            CK(dalloc(ctx, &ctx->as_tet, (i64)hc[0]));
            CK(dalloc(ctx, &ctx->as_cur, (i64)hc[0]));
            ctx->capAS = (i64)hc[0];
        }
        if ((i64)hc[1] > ctx->capDS) {
            cudaFree(ctx->ds_edge);
            cudaFree(ctx->ds_vert);
            ctx->ds_edge = ctx->ds_vert = nullptr;
            ctx->capDS = 0;
            CK(dalloc(ctx, &ctx->ds_edge, (i64)hc[1]));
            CK(dalloc(ctx, &ctx->ds_vert, (i64)hc[1]));
            ctx->capDS = (i64)hc[1];
        }
    }
    counts[0] = (int64_t)hc[0];
    counts[1] = (int64_t)hc[1];
    // (the second column of the descending records holds vertices, not codes)
    auto fetch = [&](i64 *da, i64 *db, unsigned long long n, int32_t *oa, int32_t *ob, bool vert) -> dmtz_status {
        if (!n || !oa) return DMTZ_OK;
        std::vector<i64> a(n), b(n);
        dmtz_status r = fetch_refs(ctx, g, da, a);
        if (r == DMTZ_OK && !vert) r = fetch_refs(ctx, g, db, b);
        if (r != DMTZ_OK) return r;
        if (vert) CK(cudaMemcpy(b.data(), db, sizeof(i64) * n, cudaMemcpyDeviceToHost));
        std::vector<std::pair<i64, i64>> p(n);
        for (size_t i = 0; i < n; i++) p[i] = {a[i], b[i]};
        sort_records(p);
        for (size_t i = 0; i < n; i++) {
            oa[i] = (int32_t)p[i].first;
            if (ob) ob[i] = (int32_t)p[i].second;
        }
        return DMTZ_OK;
    };
    if ((s = fetch(ctx->as_tet, ctx->as_cur, hc[0], as_tet, as_cur, false)) != DMTZ_OK) return s;
    if ((s = fetch(ctx->ds_edge, ctx->ds_vert, hc[1], ds_edge, ds_vert, true)) != DMTZ_OK) return s;
    if (err & ERR_WALK) return fail(ctx, DMTZ_ERR_CYCLE, "a path walk exceeded its step cap");
    if (err & ERR_OOB) return fail(ctx, DMTZ_ERR_OOB, "a path rule indexed out of range");
    return DMTZ_OK;
}

dmtz_status dmtz_path_detect(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                             int64_t counts[2], int32_t *as_tet, int32_t *as_cur, int32_t *ds_edge,
                             int32_t *ds_vert) {
    return path_detect_impl(ctx, W, H, D, orig, decp, 0, counts, as_tet, as_cur, ds_edge, ds_vert);
}

dmtz_status dmtz_path_detect_strict(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                                    int64_t counts[2], int32_t *as_tet, int32_t *as_cur, int32_t *ds_edge,
                                    int32_t *ds_vert) {
    return path_detect_impl(ctx, W, H, D, orig, decp, 0, counts, as_tet, as_cur, ds_edge, ds_vert, 1);
}

dmtz_status dmtz_path_detect_connectivity(dmtz_ctx *ctx, int W, int H, int D, const double *orig,
                                          const double *decp, int64_t counts[2], int32_t *as_tet, int32_t *as_cur,
                                          int32_t *ds_edge, int32_t *ds_vert) {
    return path_detect_impl(ctx, W, H, D, orig, decp, 1, counts, as_tet, as_cur, ds_edge, ds_vert);
}

dmtz_status dmtz_wall_detect(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                             int64_t *count, int32_t *w_sad, int32_t *w_edge) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!count) return fail(ctx, DMTZ_ERR_ARG, "null count");
    CK(cudaSetDevice(ctx->device));
    if ((s = setup_pair(ctx, g, orig, decp, PATH_LISTS)) != DMTZ_OK) return s;
    RuleCtx rc = rule_ctx(ctx, g, 0.0, 0);
    i64 n = 0;
    if ((s = detect_walls(ctx, g, rc, n)) != DMTZ_OK) return s;
    *count = (int64_t)n;
    if (n > 0 && w_sad) {
        std::vector<i64> a(n), b(n);
        CK(cudaMemcpy(a.data(), ctx->wall_sad, sizeof(i64) * n, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(b.data(), ctx->wall_edge, sizeof(i64) * n, cudaMemcpyDeviceToHost));
        std::vector<std::pair<i64, i64>> p(n);
        for (i64 i = 0; i < n; i++) p[i] = {a[i], b[i]};
        std::sort(p.begin(), p.end());
        for (i64 i = 0; i < n; i++) {
            w_sad[i] = (int32_t)p[i].first;
            if (w_edge) w_edge[i] = (int32_t)p[i].second;
        }
    }
    int err = 0;
    CK(cudaMemcpy(&err, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost));
    if (err & ERR_OOB) return fail(ctx, DMTZ_ERR_OOB, "a wall search indexed out of range");
    return DMTZ_OK;
}

// ----------------------------------------------------------------------------- graph-driven loop
// The host loop of main_3d.cu:6784-7149 as a state machine that runs on the
// device: a CUDA graph holds a WHILE node whose body lets one thread decide the
// state and the loop condition from the device-side counters that the round
// before left (k_round_end), then switches on the state and runs its kernels.
// A pass takes 10 us besides the kernels (6 the loop, 4 the switch).  States:
//   CP     one critical-point round (fix rules, update, re-pair, mismatch)
//   PDF    path phase: detect separatrix records, fix, update, re-pair, mismatch
//   PCHECK detect separatrix records only (the reference's end-of-round check)
//   PFIX   path phase on the records PCHECK just made (the reference detects
//          them again at the start of its next outer iteration; same inputs,
//          same records)
//   CPF    a critical-point round with long lists: the whole grid is re-paired
//   CPS    critical-point rounds with short lists, one after the other (k_short_rounds)
namespace {
enum { LS_CP = 0, LS_PDF = 1, LS_PCHECK = 2, LS_PFIX = 3, LS_CPF = 4, LS_CPS = 5, LS_DONE = 6, LS_STATES = 6 };
// bodies of the loop graph's switch: the last one is CPF's or CPS's (a body more costs 50 us to
// instantiate and destroy, 3 % of a 120 x 89 x 101 field's correction).  Grids that are ever
// repaired whole go without the short rounds: 3 % of a 128^3 Gaussian mixture's 236 rounds
// (uniform noise of 1e-3), nothing where there are few rounds
constexpr int LS_BODIES = 5;
__host__ __device__ inline bool is_cp(int state) { return state == LS_CP || state == LS_CPF || state == LS_CPS; }
struct LoopState {
    int state, pvp, converged, pad;
    long long rounds, max_rounds, outer, cp_rounds, path_rounds;
    long long cc[4];
    long long n_as, n_ds;
    long long cap[4];           // mismatch list capacities
    long long heavy;            // listed cells, and bricks of the round before, from which a round re-pairs the whole grid
    long long marked, block;    // bricks that the last round reached (before any: all); in one of sampled_marks' blocks
    int overflow;       // a scan overflowed a list: stop, grow, scan again, resume at `state`
    int last;           // state of the last body run
    int break_stalls;   // stop when a round changed nothing (the host breaks the stall)
    int stalled;
    int begun;          // a body has run: a round's end has something to end
    int ended;          // and k_short_rounds has ended it
    int pending;        // it left a round's repair to k_grad_bricks
    long long few;      // listed cells up to which rounds are short
};
struct LoopCtl : LoopState {
    long long runs[LS_STATES];  // body executions per state (CPS: rounds)
    long long shorts;           // body executions of CPS
};
}  // namespace

// the state after a body run, from the counters it left
__device__ __forceinline__ LoopState loop_next(LoopState c, const unsigned long long *counters) {
    const int st = c.state;
    if (st != LS_PCHECK)
        for (int k = 0; k < 4; k++) c.cc[k] = (long long)counters[k];
    const long long cells = c.cc[0] + c.cc[1] + c.cc[2] + c.cc[3];
    const bool cp_any = cells > 0;
    const int cp = cells >= c.heavy && c.marked >= c.heavy ? LS_CPF : cells <= c.few ? LS_CPS : LS_CP;
    int next;
    if (is_cp(st)) {
        c.rounds++;
        c.cp_rounds++;
        next = cp_any ? cp : (c.pvp ? LS_PDF : LS_DONE);
    } else if (st == LS_PDF || st == LS_PFIX) {
        c.rounds++;
        c.path_rounds++;
        c.n_as = c.n_ds = 0;
        if (cp_any) {
            c.outer++;
            next = cp;
        } else {
            next = LS_PCHECK;
        }
    } else {
        c.n_as = (long long)counters[5];
        c.n_ds = (long long)counters[6];
        if (c.n_as + c.n_ds > 0) {
            c.outer++;
            next = LS_PFIX;
        } else {
            next = LS_DONE;
        }
    }
    if (next != LS_DONE && c.rounds >= c.max_rounds) {
        c.converged = 0;
        next = LS_DONE;
    }
    c.last = st;
    if (next != LS_DONE && st != LS_PCHECK)
        for (int k = 0; k < 4; k++)
            if (c.cc[k] > c.cap[k]) c.overflow = 1;
    // counters[7]: set by the update when it changed something; a path round
    // counts only if its detection had records (counters[5], [6])
    if (c.break_stalls && next != LS_DONE && counters[7] == 0 &&
        (is_cp(st) || ((st == LS_PDF || st == LS_PFIX) && counters[5] + counters[6] > 0)))
        c.stalled = 1;
    c.state = next;
    return c;
}

// The end of a round: the rebuilt mismatch lists back into the lists (T.n ==
// nullptr: none were rebuilt; entries past a list's capacity were not stored,
// and the count shows the overflow) and the bricks' marks cleared, then the last
// block to finish clears the round's counters and either decides the graph loop's
// next state (ctl) or leaves the counts for the host (report, in pinned memory).
// In the graph it stands before the switch that it sets, so the first one has no
// round to end, and after the last one no state runs.
__global__ void __launch_bounds__(kBlock) k_round_end(const __grid_constant__ Lists T, const __grid_constant__ Lists L, unsigned long long *counters,
                                                     const __grid_constant__ BrickMarks B, LoopCtl *ctl,
                                                     cudaGraphConditionalHandle hwhile, cudaGraphConditionalHandle hswitch,
                                                     unsigned long long *report, unsigned long long seq) {
    __shared__ bool last;
    after_previous();
    const int st = ctl ? ctl->state : LS_CP;
    const bool ends = !ctl || (ctl->begun && !ctl->ended);
    const bool copy = ends && T.n && st != LS_PCHECK && st != LS_CPF;
    const i64 nbrick = (i64)*B.n;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < nbrick; i += (i64)gridDim.x * blockDim.x) {
        const uint32_t e = B.list[i];
        reinterpret_cast<uint8_t *>(B.flags)[(e & 0x7FF) + (i64)B.nbx * (((e >> 11) & 0x7FF) + (i64)B.nby * (e >> 22))] = 0;
    }
    if (copy) {
        const i64 n0 = min((i64)T.n[0], T.cap[0]), n1 = min((i64)T.n[1], T.cap[1]), n2 = min((i64)T.n[2], T.cap[2]),
                  n3 = min((i64)T.n[3], T.cap[3]);
        const i64 tid = (i64)blockIdx.x * blockDim.x + threadIdx.x;
        for (i64 i = tid; i < n0 + n1 + n2 + n3; i += (i64)gridDim.x * blockDim.x) {
            if (i < n0) L.l[0][i] = T.l[0][i];
            else if (i < n0 + n1) L.l[1][i - n0] = T.l[1][i - n0];
            else if (i < n0 + n1 + n2) L.l[2][i - n0 - n1] = T.l[2][i - n0 - n1];
            else L.l[3][i - n0 - n1 - n2] = T.l[3][i - n0 - n1 - n2];
        }
    }
    __syncthreads();  // the block has read T.n and the state
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&counters[30], 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    counters[30] = 0;
    *B.n = 0;
    if (copy)
        for (int k = 0; k < 4; k++) {
            L.n[k] = T.n[k];
            T.n[k] = 0;
        }
    bool stop = false;
    if (ctl) {
        LoopState c = *ctl;
        if (ends) ctl->runs[st]++;
        if (ends && st != LS_PCHECK) c.marked = st == LS_CPF ? nbrick * c.block : nbrick;
        if (ends) c = loop_next(c, counters);
        c.begun = 1;
        c.ended = c.pending = 0;
        static_cast<LoopState &>(*ctl) = c;
        stop = c.state == LS_DONE || c.overflow || c.stalled;
        cudaGraphSetConditional(hswitch, stop ? (unsigned)LS_BODIES : (unsigned)min(c.state, LS_BODIES - 1));
        cudaGraphSetConditional(hwhile, stop ? 0u : 1u);
        if (!stop && (c.state == LS_PDF || c.state == LS_PCHECK)) counters[5] = counters[6] = counters[27] = 0;
    } else {
        for (int k = 0; k < 8; k++) report[k] = counters[k];
        report[14] = (unsigned long long)nbrick;
        __threadfence_system();
        *reinterpret_cast<volatile unsigned long long *>(report + 8) = seq;
    }
    if (!stop) counters[4] = counters[7] = 0;  // a stalled round's requests were applied: the host starts afresh
}

// ----------------------------------------------------------------------------- short rounds
// Critical-point rounds of short lists, one after the other, by one cluster of blocks:
// fix, update, re-pair, lists back, without a launch or the host between them, because
// a round of a few cells is 10 us of dependent loads in 50 us of launches and waits.
// The blocks meet at the cluster's barriers (which order their memory accesses).  The
// loop ends when the lists are empty or hold more than kShortCells (then the whole
// GPU does a round sooner), when a list overflowed, a round changed nothing (stop_stalled), or max_rounds
// have run; with more than kShortBricks bricks marked it leaves the round to the
// kernels that it stands for, after its update (report[10]).  In the loop graph
// (ctl) it is the state CPS and goes on from round to round as k_round_end would.  report: [0..7] the
// counters as after any round, [9] rounds, [11..13] nanoseconds of fix, update and
// the rest, [14] (for few bricks) 0.  Gaussian mixtures with uniform noise, seed 1, without and
// with it: host-driven loops, 16^3 (1e-2) 3.24 and 2.67 ms, 64^3 extrema (1e-3) 11.0 and 10.3;
// graph loop, 97 x 61 x 75 (1e-2) 14.05 and 13.56; a batch of eight the same.  With 384 cells and
// 64 bricks the first two were as fast, but the batch got 3 % slower.
constexpr unsigned kShortBlocks = 16;
constexpr i64 kShortCells = 64, kShortBricks = 160, kShortRounds = 256;  // at most that many per launch
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ unsigned long long nanoseconds() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__global__ void __launch_bounds__((brick_threads<8, 4, 4>()), 2)
    k_short_rounds(const __grid_constant__ RuleCtx c, const __grid_constant__ CpLists CL, const __grid_constant__ Lists L,
                   const __grid_constant__ Lists T, int preserve_saddles, double range, int preserve_type, uint8_t *changed,
                   const __grid_constant__ BrickMarks B, const __grid_constant__ FieldState s, const __grid_constant__ BrickList bl,
                   const __grid_constant__ GradOps O, const __grid_constant__ KeepOps K, unsigned long long *counters,
                   i64 max_rounds, int stop_stalled, LoopCtl *ctl, unsigned long long *report, unsigned long long seq) {
    __shared__ RuleTab tab;
    __shared__ BrickMem<8, 4, 4> M;
    const Grid &g = c.g;
    const unsigned block = blockIdx.x, blocks = gridDim.x;
    const bool first = block == 0 && threadIdx.x == 0;
    const i64 tid = (i64)block * blockDim.x + threadIdx.x, nt = (i64)blocks * blockDim.x;
    load_rule_tab(tab);
    if (ctl) {
        max_rounds = min((i64)(ctl->max_rounds - ctl->rounds), kShortRounds);
        stop_stalled = ctl->break_stalls;
    }
    i64 rounds = 0;
    bool left = false;
    unsigned long long ns[3] = {0, 0, 0}, t0 = nanoseconds(), t1;
    auto lap = [&](int k) {
        t1 = nanoseconds();
        ns[k] += t1 - t0;
        t0 = t1;
    };
    while (true) {
        fix_cells(c, CL, preserve_saddles, tab, true, block, blocks, (i64)blocks * (blockDim.x / 32));
        cluster_barrier();
        lap(0);
        apply_requests(c, range, preserve_type, 1, changed, nullptr, B, true, block, blocks);
        cluster_barrier();
        lap(1);
        rounds++;
        const i64 nb = (i64)__ldcg(B.n);
        left = nb > kShortBricks;
        if (left) break;
        for (i64 b = block; b < nb; b += blocks) {
            grad_brick<8, 4, 4>(g, s, bl, O, b, M);
            __syncthreads();
        }
        keep_lists(g, O, K, block);
        cluster_barrier();
        // the round's end, as k_round_end
        i64 n[4], cells = 0;
        bool over = false;
        for (int k = 0; k < 4; k++) {
            n[k] = (i64)__ldcg(&T.n[k]);
            cells += n[k];
            over |= n[k] > L.cap[k];
            for (i64 i = tid; i < min(n[k], L.cap[k]); i += nt) L.l[k][i] = T.l[k][i];
        }
        for (i64 i = tid; i < nb; i += nt) {
            const uint32_t e = B.list[i];
            reinterpret_cast<uint8_t *>(B.flags)[(e & 0x7FF) + (i64)B.nbx * (((e >> 11) & 0x7FF) + (i64)B.nby * (e >> 22))] = 0;
        }
        const bool moved = __ldcg(&counters[7]) != 0;
        const bool stop = cells == 0 || cells > kShortCells || over || rounds >= max_rounds || (stop_stalled && !moved);
        cluster_barrier();  // every block has read what is cleared now
        if (first) {
            for (int k = 0; k < 4; k++) {
                L.n[k] = (unsigned long long)n[k];
                T.n[k] = 0;
            }
            *B.n = 0;
            if (ctl) {
                ctl->runs[ctl->state]++;
                static_cast<LoopState &>(*ctl) = loop_next(*ctl, counters);
            } else if (stop) {
                for (int k = 0; k < 8; k++) report[k] = counters[k];
            }
            counters[4] = counters[7] = 0;
        }
        cluster_barrier();
        lap(2);
        if (stop) break;
    }
    if (first && ctl) {
        ctl->ended = !left;
        ctl->pending = left;
        ctl->shorts++;
    } else if (first) {
        if (left)
            for (int k = 0; k < 8; k++) report[k] = counters[k];
        report[9] = (unsigned long long)rounds;
        report[10] = left;
        report[14] = 0;  // (few)
        for (int k = 0; k < 3; k++) report[11 + k] = ns[k];
        __threadfence_system();
        *reinterpret_cast<volatile unsigned long long *>(report + 8) = seq;
    }
}

// ----------------------------------------------------------------------------- phase timers
namespace {
enum { PH_PAIR = 0, PH_FIXCP, PH_PATH, PH_FIXPATH, PH_APPLY, PH_SETUP, PH_N };
// Phase times from events on the context's stream: one at each boundary (a phase
// ends where the next begins), from a pool that the context keeps.  reuse() adds up
// what is complete and takes its events back, so a long host-driven loop needs
// about 64 of them (two per phase, created and destroyed in every call: 1 ms of a
// 16^3 field's 48 rounds).
struct PhaseTimer {
    cudaStream_t st;
    std::vector<cudaEvent_t> &pool;
    std::vector<std::pair<int, size_t>> marks;  // phase that begins (PH_N: none), its event
    size_t used = 0;
    double total[PH_N] = {0, 0, 0, 0, 0, 0};
    void mark(int ph) {
        if (used >= 64 && marks.back().first == PH_N) {
            cudaEventSynchronize(pool[used - 1]);
            reuse();
        }
        if (used == pool.size()) {
            cudaEvent_t e;
            cudaEventCreate(&e);
            pool.push_back(e);
        }
        cudaEventRecord(pool[used], st);
        marks.push_back({ph, used++});
    }
    void stop() { mark(PH_N); }
    // the events recorded so far are complete, and no phase is open
    void reuse() {
        for (size_t k = 0; k + 1 < marks.size(); k++) {
            if (marks[k].first == PH_N) continue;
            float t = 0;
            cudaEventElapsedTime(&t, pool[marks[k].second], pool[marks[k + 1].second]);
            total[marks[k].first] += t;
        }
        marks.clear();
        used = 0;
    }
};
}  // namespace

// Can this run's short rounds go to k_short_rounds?  (Lists rebuilt by the repairs,
// the default brick shape, and a device that holds the cluster.)
static bool short_rounds_fit(dmtz_ctx *ctx) {
    if (!ctx->inc_scan || ctx->tune_shape != 0) return false;
    if (!ctx->short_clusters) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kShortBlocks);
        cfg.blockDim = dim3(brick_threads<8, 4, 4>());
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kShortBlocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute((const void *)k_short_rounds, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, k_short_rounds, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        ctx->short_clusters = n > 0 ? n : -1;
    }
    return ctx->short_clusters > 0;
}
// in the loop graph: on grids that are never repaired whole
static bool graph_short_rounds(dmtz_ctx *ctx, const Grid &g) { return heavy_cells(ctx, g) == INT64_MAX && short_rounds_fit(ctx); }
static cudaError_t launch_short_rounds(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, const FieldState &Qs, double range, int ps,
                                       int pt, i64 max_rounds, int stop_stalled, LoopCtl *ctl = nullptr) {
    const BrickMarks B = brick_marks(ctx, g);
    i64 nb;
    BrickList bl = all_bricks(g, ctx->tune_shape, nb);
    bl.list = ctx->brick_list;
    bl.n = ctx->brick_n;
    GradOps O{};
    KeepOps K{};
    repair_ops(ctx, B, ctx->P.crit, ps == 1, O, K);
    K.blocks = kShortBlocks;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kShortBlocks);
    cfg.blockDim = dim3(brick_threads<8, 4, 4>());
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kShortBlocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (!ctl) ctx->report_seq++;
    ctx->launches++;
    return cudaLaunchKernelEx(&cfg, k_short_rounds, rc, cp_lists(ctx), mismatch_lists(ctx), rebuilt_lists(ctx), ps, range, pt,
                              ctx->changed, B, Qs, bl, O, K, ctx->counters, max_rounds, stop_stalled, ctl, ctx->report,
                              ctx->report_seq);
}

// The loop as an executable graph, with the lists' capacities that it was built for.
// Building and instantiating takes 110 us of host time and destroying 60 to 100, so
// the first is done while the set-up's kernels run and the last while the results travel.
struct LoopGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    i64 cap[4] = {0, 0, 0, 0};
    bool fits(const dmtz_ctx *ctx) const {
        for (int k = 0; k < 4; k++)
            if (cap[k] != ctx->capL[k]) return false;
        return exec != nullptr;
    }
    void clear() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    ~LoopGraph() { clear(); }
};
// (a capture: work already on the stream goes on)
static dmtz_status build_graph_loop(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, const PathRec &PR, const FieldState &Qs,
                                    double range, int ps, int pt, int conn, LoopGraph &lg) {
    cudaStream_t st = ctx->stream;
    const unsigned pgrid = persistent_grid();
    const CpLists L = cp_lists(ctx);
    i64 block;
    if (!ctx->loopctl) CK(cudaMalloc(&ctx->loopctl, sizeof(LoopCtl)));
    LoopCtl *dctl = static_cast<LoopCtl *>(ctx->loopctl);
    lg.clear();
    for (int k = 0; k < 4; k++) lg.cap[k] = ctx->capL[k];
    cudaGraph_t &graph = lg.graph;
    cudaGraphExec_t &exec = lg.exec;
    const auto launches = ctx->launches;  // of a capture: none
    dmtz_status res = DMTZ_OK;
    do {
        if (cudaGraphCreate(&graph, 0) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
        cudaGraphConditionalHandle hwhile;
        if (cudaGraphConditionalHandleCreate(&hwhile, graph, 1, cudaGraphCondAssignDefault) != cudaSuccess) {
            res = DMTZ_ERR_CUDA;
            break;
        }
        cudaGraphNodeParams wp = {};
        wp.type = cudaGraphNodeTypeConditional;
        wp.conditional.handle = hwhile;
        wp.conditional.type = cudaGraphCondTypeWhile;
        wp.conditional.size = 1;
        cudaGraphNode_t wnode;
        if (cudaGraphAddNode(&wnode, graph, nullptr, nullptr, 0, &wp) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
        cudaGraph_t body = wp.conditional.phGraph_out[0];
        cudaGraphConditionalHandle hsw;
        if (cudaGraphConditionalHandleCreate(&hsw, body, 0, 0) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
        // body: end the round before and set the switch, then switch over the states
        cudaGraphNode_t n_set, n_sw;
        {
            if (cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
                res = DMTZ_ERR_CUDA;
                break;
            }
            k_round_end<<<pgrid / 8, kBlock, 0, st>>>(ctx->inc_scan ? rebuilt_lists(ctx) : Lists{}, mismatch_lists(ctx),
                                                      ctx->counters, brick_marks(ctx, g), dctl, hwhile, hsw, nullptr, 0);
            cudaGraph_t tmp;
            if (cudaStreamEndCapture(st, &tmp) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
            size_t nn = 1;
            cudaGraphGetNodes(body, &n_set, &nn);
        }
        cudaGraphNodeParams sp = {};
        sp.type = cudaGraphNodeTypeConditional;
        sp.conditional.handle = hsw;
        sp.conditional.type = cudaGraphCondTypeSwitch;
        sp.conditional.size = LS_BODIES;
        if (cudaGraphAddNode(&n_sw, body, &n_set, nullptr, 1, &sp) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
        const bool short_rounds = graph_short_rounds(ctx, g);
        for (int body = 0; body < LS_BODIES && res == DMTZ_OK; body++) {
            cudaGraph_t child = sp.conditional.phGraph_out[body];
            const int state = body == LS_CPF && short_rounds ? LS_CPS : body;
            if (cudaStreamBeginCaptureToGraph(st, child, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
                res = DMTZ_ERR_CUDA;
                break;
            }
            if (state == LS_PDF || state == LS_PCHECK) launch_detect(ctx, g, rc, PR, pgrid, conn);
            if (state == LS_CPS) {
                if (launch_short_rounds(ctx, g, rc, Qs, range, ps, pt, 0, 0, dctl) != cudaSuccess) res = DMTZ_ERR_CUDA;
                repair_dirty(ctx, g, Qs, ctx->P.crit, ps == 1, true, &dctl->pending);
            } else if (state != LS_PCHECK) {
                const bool cp = is_cp(state);
                const int want = cp ? (ps == 1) : 1;
                if (cp) k_fix_cp<<<pgrid, kBlock, 0, st>>>(rc, L, ps);
                else k_fix_path<<<pgrid, kBlock, 0, st>>>(rc, PR);
                launch_next(state == LS_CPF ? k_apply<true> : k_apply<false>, pgrid, kBlock, st, rc, range, pt, 1, ctx->changed, nullptr,
                            state == LS_CPF ? sampled_marks(ctx, g, &block) : brick_marks(ctx, g));
                if (state == LS_CPF) repair_full(ctx, g, Qs, ctx->P.crit, want);
                else repair_dirty(ctx, g, Qs, ctx->P.crit, want, true);
            }
            cudaGraph_t tmp;
            if (cudaStreamEndCapture(st, &tmp) != cudaSuccess) res = DMTZ_ERR_CUDA;
        }
        if (res != DMTZ_OK) break;
        if (cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) { res = DMTZ_ERR_CUDA; break; }
    } while (0);
    ctx->launches = launches;
    if (res != DMTZ_OK) {
        lg.clear();
        cudaGetLastError();
        return fail(ctx, res, "building the loop graph failed");
    }
    return DMTZ_OK;
}
// Run it.  Returns the final LoopCtl in *out.  The states' counters (requests,
// progress, separatrix records) are as the first state needs them.
static dmtz_status run_graph_loop(dmtz_ctx *ctx, const LoopGraph &lg, LoopCtl init, LoopCtl *out) {
    cudaStream_t st = ctx->stream;
    init.begun = init.ended = init.pending = 0;
    CK(cudaMemcpyAsync(ctx->loopctl, &init, sizeof(LoopCtl), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(ctx->counters + 4, 0, sizeof(unsigned long long), st));
    CK(cudaMemsetAsync(ctx->counters + 7, 0, sizeof(unsigned long long), st));
    CK(cudaMemsetAsync(ctx->counters + 27, 0, sizeof(unsigned long long), st));
    if (init.state != LS_PFIX) CK(cudaMemsetAsync(ctx->counters + 5, 0, 2 * sizeof(unsigned long long), st));
    if (cudaGraphLaunch(lg.exec, st) != cudaSuccess ||
        cudaMemcpyAsync(out, ctx->loopctl, sizeof(LoopCtl), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, DMTZ_ERR_CUDA, "running the loop graph failed");
    }
    return DMTZ_OK;
}

// ----------------------------------------------------------------------------- the correction loop
// the round's end of the host-driven loop (its counts then stand in ctx->report once the stream is done)
static void host_round_end(dmtz_ctx *ctx, const Grid &g) {
    launch_next(k_round_end, persistent_grid() / 8, kBlock, ctx->stream, ctx->inc_scan ? rebuilt_lists(ctx) : Lists{},
                mismatch_lists(ctx), ctx->counters, brick_marks(ctx, g), nullptr, cudaGraphConditionalHandle{},
                cudaGraphConditionalHandle{}, ctx->report, ++ctx->report_seq);
    ctx->launches++;
}

// features of (ctx->f, ctx->g) from the current gradients ctx->P / ctx->Q
static dmtz_status features_into(dmtz_ctx *ctx, const Grid &g, double bound, __nv_bfloat16 *feat, uint8_t *active) {
    if (g.V > ctx->capMM) {
        cudaFree(ctx->mm);
        ctx->mm = nullptr;
        ctx->capMM = 0;
        CK(dalloc(ctx, &ctx->mm, g.V));
        ctx->capMM = g.V;
    }
    cudaStream_t st = ctx->stream;
    const unsigned grid = persistent_grid();
    const double inv = 1.0 / bound, inv4 = 1.0 / (4.0 * bound);
    const bool exact = !(std::isnormal(inv) && std::isnormal(inv4)), narrow = g.W <= 4;
    const int tx = narrow ? 4 : 32, ty = narrow ? 16 : 8, tz = narrow ? 16 : 4;
    auto kern = narrow ? (exact ? k_features<4, 16, 16, true> : k_features<4, 16, 16, false>)
                       : (exact ? k_features<32, 8, 4, true> : k_features<32, 8, 4, false>);
    const int ntx = (g.W + tx - 1) / tx, nty = (g.H + ty - 1) / ty, ntz = (g.D + tz - 1) / tz;
    kern<<<(unsigned)((i64)ntx * nty * ntz), kBlock, 0, st>>>(g, ctx->f, ctx->g, ctx->P.crit, ctx->Q.crit, bound, inv, inv4,
                                                             feat, ctx->mm, ntx, nty);
    k_dilate<<<grid, kBlock, 0, st>>>(g, 0, ctx->mm, active);
    k_dilate<<<grid, kBlock, 0, st>>>(g, 1, active, ctx->mm);
    k_dilate<<<grid, kBlock, 0, st>>>(g, 2, ctx->mm, active);
    ctx->launches += 4;
    CK(cudaGetLastError());
    return DMTZ_OK;
}

// Learned warm start: features, network, proposal, then the gradient of the
// edited field (around the edits) and its mismatch lists again.
static dmtz_status learned_start(dmtz_ctx *ctx, dmtz_cnn *net, const Grid &g, double bound) {
    using namespace dmtz_cnn_impl;
    if (device_of(net) != ctx->device) return fail(ctx, DMTZ_ERR_ARG, "network and context on different devices");
    __nv_bfloat16 *feat;
    uint8_t *active;
    float *out;
    dmtz_status s = scratch(net, g.V, &feat, &active, &out);
    if (s != DMTZ_OK) return fail(ctx, s, "network: " + error_of(net));
    if ((s = features_into(ctx, g, bound, feat, active)) != DMTZ_OK) return s;
    s = forward_on(net, g.W, g.H, g.D, feat, out, 0, ctx->stream);
    if (s != DMTZ_OK) return fail(ctx, s, "network: " + error_of(net));
    CK(cudaMemsetAsync(ctx->counters + 4, 0, sizeof(unsigned long long), ctx->stream));
    k_propose<<<persistent_grid(), kBlock, 0, ctx->stream>>>(g.V, ctx->f, ctx->g, out, active, bound,
                                                              (double)min_drop_of(net) * bound, ctx->changed,
                                                              ctx->reqlist, ctx->counters + 4);
    ctx->launches += 5;
    // re-pair only the bricks within the passes' radii of the edited vertices
    // (the mismatch lists are rebuilt by a full scan: the loop has not started)
    repair_dirty(ctx, g, view(ctx->Q, ctx->g), ctx->P.crit, 1, false);
    clear_marks(ctx);
    CK(cudaMemsetAsync(ctx->counters + 4, 0, sizeof(unsigned long long), ctx->stream));
    CK(cudaGetLastError());
    return DMTZ_OK;
}

// a round made no progress: reset the values around the remaining mismatched
// cells (cp = 1) or separatrix records (cp = 0) to the original ones, re-pair
// there, and clear the request bits (see k_snap_mask)
static dmtz_status break_stall(dmtz_ctx *ctx, const Grid &g, const RuleCtx &rc, const PathRec &PR,
                               const FieldState &Qs, int cp, int want_saddles, int64_t nbreaks,
                               const WallRec *WR = nullptr) {
    cudaStream_t st = ctx->stream;
    const unsigned pgrid = persistent_grid();
    // the k-th break resets the box of half-width k around the seeds (the
    // seeds alone first), up to the whole grid, where g = f and every run ends
    const int radius = (int)std::min<int64_t>(nbreaks, std::max(g.W, std::max(g.H, g.D)));
    CK(cudaMemsetAsync(ctx->counters + 4, 0, sizeof(unsigned long long), st));
    if (cp) k_seed_cells<<<pgrid, kBlock, 0, st>>>(g, cp_lists(ctx), ctx->changed);
    else k_seed_paths<<<pgrid, kBlock, 0, st>>>(g, PR, ctx->changed);
    if (!cp && WR) {  // and the wall records' edges
        k_seed_walls<<<pgrid, kBlock, 0, st>>>(g, *WR, ctx->changed);
        ctx->launches++;
    }
    for (int axis = 0; axis < 3; axis++) {
        const int n = axis == 0 ? g.W : axis == 1 ? g.H : g.D;
        k_dilate_axis<<<grid_for(g.V / n), kBlock, 0, st>>>(g, ctx->changed, axis, std::min(radius, n));
    }
    k_snap_mask<<<pgrid, kBlock, 0, st>>>(rc, ctx->changed);
    repair_dirty(ctx, g, Qs, ctx->P.crit, want_saddles, false);
    k_clear_req<<<pgrid, kBlock, 0, st>>>(ctx->reqlist, ctx->counters + 4, g.V, ctx->reqbits);
    host_round_end(ctx, g);
    ctx->launches += 6;
    CK(cudaGetLastError());
    return DMTZ_OK;
}

static dmtz_status correct_impl(dmtz_ctx *ctx, dmtz_cnn *net, int W, int H, int D, const double *orig, double *decp,
                                int on_device, double rel_eps, const dmtz_opts *opts, dmtz_report *rep,
                                int32_t *edit_counter_out) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!opts) return fail(ctx, DMTZ_ERR_ARG, "null options");
    const int ps = opts->preserve_saddles, pvp = opts->preserve_vpath, pg = opts->preserve_geometry,
              filt = opts->filtration, pc = opts->preserve_connectors, pt = opts->preserve_type,
              et = opts->edit_type;
    // wall checks (preserve_connectors = 1) run in the separatrix phase; their
    // searches are sized on the host, so such runs use the host-driven loop
    const bool walls = pc == 1 && pvp == 1;
    const bool use_graph = opts->use_graph && !walls;
    const int conn = (pvp == 1 && pg == 0) ? 1 : 0;  // connectivity-mode separatrices
    if (!(rel_eps >= 0.0) || !std::isfinite(rel_eps)) return fail(ctx, DMTZ_ERR_ARG, "rel_eps must be finite and >= 0");
    const i64 max_rounds = opts->max_rounds > 0 ? opts->max_rounds : 100000;
    ctx->inc_scan = 0;  // full scans until the loop starts
    ctx->path_keep = 0;
    ctx->strict_ds = (opts->strict_separatrices && !conn) ? 1 : 0;
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    cudaStream_t st = ctx->stream;
    if (!ctx->report) {
        CK(cudaHostAlloc((void **)&ctx->report, 16 * sizeof(unsigned long long), cudaHostAllocDefault));
        memset(ctx->report, 0, 16 * sizeof(unsigned long long));
    }
    if (!ctx->span[0]) {
        CK(cudaEventCreate(&ctx->span[0]));
        CK(cudaEventCreate(&ctx->span[1]));
    }
    const cudaEvent_t e0 = ctx->span[0], e1 = ctx->span[1];
    if ((s = upload(ctx, ctx->f, orig, g.V, on_device)) != DMTZ_OK) return s;
    // the decompressed field travels on a second stream while the original
    // field's gradient is computed; the work that reads it waits for it
    if (!ctx->side) {
        CK(cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&ctx->side_done, cudaEventDisableTiming));
    }
    CK(cudaMemcpyAsync(ctx->g, decp, sizeof(double) * (size_t)g.V,
                       on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, ctx->side));
    CK(cudaEventRecord(ctx->side_done, ctx->side));
    // range and bound exactly as the reference computes them (main_3d.cu:6303-6323)
    double mn, mx;
    ctx->launches = 0;
    PhaseTimer pt_{st, ctx->events};
    CK(cudaEventRecord(e0, st));
    pt_.mark(PH_SETUP);
    if ((s = device_minmax(ctx, ctx->f, g.V, mn, mx)) != DMTZ_OK) return s;
    const double bound = (mx - mn) * rel_eps;
    const double range = mx - mn;
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), st));
    CK(cudaMemsetAsync(ctx->changed, 0, (size_t)g.V, st));
    CK(cudaMemsetAsync(ctx->counters, 0, 8 * sizeof(unsigned long long), st));
    CK(cudaMemsetAsync(ctx->counters + 20, 0, 11 * sizeof(unsigned long long), st));
    clear_marks(ctx);
    const FieldState Ps = view(ctx->P, ctx->f), Qs = view(ctx->Q, ctx->g);
    run_pairing(ctx, g, Ps, nullptr, 1);
    if (pvp == 1 && (s = prep_paths(ctx, g, !conn)) != DMTZ_OK) return s;
    CK(cudaStreamWaitEvent(st, ctx->side_done, 0));
    if ((s = check_finite(ctx, ctx->g, g.V)) != DMTZ_OK) return s;
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), st));
    if (filt == 1) {
        k_filter<<<grid_for(g.V), kBlock, 0, st>>>(g, ctx->P.crit, ctx->f, ctx->g, bound);
        ctx->launches++;
    }
    ctx->path_keep = pvp == 1 && !conn;
    run_pairing(ctx, g, Qs, ctx->P.crit, 1);
    k_fill_i32<<<grid_for(g.V), kBlock, 0, st>>>(ctx->cnt, 1, g.V);
    ctx->launches++;
    pt_.stop();
    const unsigned pgrid = persistent_grid();
    RuleCtx rc = rule_ctx(ctx, g, bound, et);
    rc.range = range;
    const PathRec PR = path_rec(ctx);
    // every scan of the loop asks for saddles when preserve_saddles = 1, and none
    // does in runs without separatrix rounds otherwise: the repairs can then rebuild
    // the lists from the re-paired bricks alone
    const int inc = ps == 1 || pvp == 0 ? 1 : 0;
    LoopGraph lg;
    auto fit_graph = [&]() -> dmtz_status {  // (built for lists that the loop itself uses)
        if (lg.fits(ctx)) return DMTZ_OK;
        const int keep = ctx->inc_scan;
        ctx->inc_scan = inc;
        const dmtz_status r = build_graph_loop(ctx, g, rc, PR, Qs, range, ps, pt, conn, lg);
        ctx->inc_scan = keep;
        return r;
    };
    if (use_graph && pvp && (s = fit_graph()) != DMTZ_OK) return s;  // (without separatrix rounds it may not be needed)
    unsigned long long hc[8];
    auto read_counts = [&]() -> dmtz_status {
        CK(cudaMemcpyAsync(hc, ctx->counters, sizeof(hc), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        return DMTZ_OK;
    };
    // counts after a round's end; lists that overflowed grow and are rebuilt
    // (the counts stand in pinned memory as soon as the round's end wrote them, some
    // microseconds before a wait for the stream would return; a launch of the round
    // that failed shows here)
    i64 marked = INT64_MAX;  // bricks of the last round
    auto read_fit = [&](int want_saddles) -> dmtz_status {
        const cudaError_t waited = wait_report(ctx->report + 8, ctx->report_seq, [&]() { return cudaStreamQuery(st); });
        CK(cudaGetLastError());
        CK(waited);
        const volatile unsigned long long *report = ctx->report;
        for (int k = 0; k < 8; k++) hc[k] = report[k];
        marked = (i64)report[14];
        return fit_lists(ctx, g, want_saddles, hc);
    };
    if ((s = read_counts()) != DMTZ_OK || (s = fit_lists(ctx, g, 1, hc)) != DMTZ_OK) return s;
    dmtz_report R;
    memset(&R, 0, sizeof(R));
    for (int k = 0; k < 4; k++) R.initial_mismatch[k] = (int64_t)hc[k];
    if (net) {
        pt_.mark(PH_SETUP);
        if ((s = learned_start(ctx, net, g, bound)) != DMTZ_OK) return s;
        pt_.stop();
        if ((s = read_counts()) != DMTZ_OK || (s = fit_lists(ctx, g, 1, hc)) != DMTZ_OK) return s;
    }
    i64 cc[4] = {(i64)hc[0], (i64)hc[1], (i64)hc[2], (i64)hc[3]};
    i64 n_as = 1, n_ds = 1, n_wall = 1;
    ctx->inc_scan = inc;
    const i64 heavy = heavy_cells(ctx, g);
    i64 block;
    const BrickMarks whole = sampled_marks(ctx, g, &block);
    i64 rounds = 0;
    int converged = 1;
    if (walls && (s = ensure_walls(ctx)) != DMTZ_OK) return s;
    const WallRec WR = wall_rec(ctx);
    auto cp_any = [&]() { return cc[0] > 0 || cc[1] > 0 || cc[2] > 0 || cc[3] > 0; };
    if (use_graph) {
        // same loop, decided on the device (see run_graph_loop)
        LoopCtl c;
        memset(&c, 0, sizeof(c));
        c.pvp = pvp;
        c.converged = 1;
        c.max_rounds = max_rounds;
        c.outer = 1;
        c.break_stalls = opts->break_stalls ? 1 : 0;
        for (int k = 0; k < 4; k++) c.cc[k] = cc[k];
        c.heavy = heavy;
        c.marked = marked;
        c.block = block;
        c.few = graph_short_rounds(ctx, g) ? kShortCells : 0;
        auto cp_state = [&](i64 cells) { return cells >= heavy && marked >= heavy ? LS_CPF : cells <= c.few ? LS_CPS : LS_CP; };
        c.state = cp_any() ? cp_state(cc[0] + cc[1] + cc[2] + cc[3]) : (pvp ? LS_PDF : LS_DONE);
        LoopCtl fin = c;
        if (c.state != LS_DONE) {
            pt_.mark(PH_PAIR);
            LoopCtl cur = c;
            int64_t graphs = 0;
            while (true) {
                graphs++;
                for (int k = 0; k < 4; k++) cur.cap[k] = ctx->capL[k];
                if ((s = fit_graph()) != DMTZ_OK || (s = run_graph_loop(ctx, lg, cur, &fin)) != DMTZ_OK) return s;
                if (!fin.overflow && !fin.stalled) break;
                // a scan outgrew a list: grow it, rebuild the lists and resume
                unsigned long long h4[4];
                for (int k = 0; k < 4; k++) h4[k] = (unsigned long long)fin.cc[k];
                if ((s = fit_lists(ctx, g, is_cp(fin.last) ? (ps == 1) : 1, h4)) != DMTZ_OK) return s;
                cur = fin;
                cur.overflow = 0;
                if (fin.stalled) {  // the round changed nothing: break the stall, then go on
                    const int cpst = is_cp(fin.last);
                    if ((s = break_stall(ctx, g, rc, PR, Qs, cpst, cpst ? (ps == 1) : 1, R.stall_breaks)) != DMTZ_OK)
                        return s;
                    R.stall_breaks++;
                    if ((s = read_fit(cpst ? (ps == 1) : 1)) != DMTZ_OK) return s;
                    cur.marked = marked;
                    cur.stalled = 0;
                    for (int k = 0; k < 4; k++) cur.cc[k] = (long long)hc[k];
                    const bool any = hc[0] || hc[1] || hc[2] || hc[3];
                    if (cpst) {  // on with the critical-point loop, or to a separatrix round
                        cur.state = any ? cp_state(hc[0] + hc[1] + hc[2] + hc[3]) : (pvp ? LS_PDF : LS_DONE);
                    } else {  // a new outer iteration, or the separatrix re-check
                        cur.state = any ? cp_state(hc[0] + hc[1] + hc[2] + hc[3]) : LS_PCHECK;
                        if (any) cur.outer++;
                    }
                    if (cur.state == LS_DONE) {
                        fin = cur;
                        break;
                    }
                }
            }
            pt_.stop();
            // kernels per body run: the round's end, plus each state's own: a fix
            // round is fix + update, then the repair (gradient, and the scan where
            // the lists are not rebuilt), or the whole gradient; short rounds are
            // one kernel and the repair behind it; one end more per graph
            const int64_t det = detect_kernels(ctx, conn);  // separatrix detection kernels
            const int64_t rnd = 2 + 1 + (ctx->inc_scan ? 0 : 1);
            int64_t bodies = 0;
            for (int k = 0; k < LS_STATES; k++) bodies += k == LS_CPS ? 0 : fin.runs[k];
            ctx->launches += graphs + bodies + 3 * fin.shorts + rnd * fin.runs[LS_CP] + (rnd + det) * fin.runs[LS_PDF] +
                             det * fin.runs[LS_PCHECK] + rnd * fin.runs[LS_PFIX] + 3 * fin.runs[LS_CPF];
        }
        R.outer_iterations = fin.outer;
        R.cp_rounds = fin.cp_rounds;
        R.path_rounds = fin.path_rounds;
        for (int k = 0; k < 4; k++) cc[k] = fin.cc[k];
        n_as = fin.n_as;
        n_ds = fin.n_ds;
        n_wall = 0;
        converged = fin.converged;
    }
    // a critical-point round that changed nothing is broken
    auto stalled = [&]() -> dmtz_status {
        if (!opts->break_stalls || hc[7] != 0 || rounds >= max_rounds || !(hc[0] || hc[1] || hc[2] || hc[3])) return DMTZ_OK;
        dmtz_status r = break_stall(ctx, g, rc, PR, Qs, 1, ps == 1, R.stall_breaks);
        if (r != DMTZ_OK) return r;
        R.stall_breaks++;
        return read_fit(ps == 1);
    };
    // separatrix records of the last re-check, still valid while no round ran since
    bool paths_fresh = false;
    while (!use_graph && (n_as > 0 || n_ds > 0 || n_wall > 0 || cp_any())) {
        if (rounds >= max_rounds) {
            converged = 0;
            break;
        }
        R.outer_iterations++;
        while (cp_any()) {
            if (rounds >= max_rounds) break;
            paths_fresh = false;
            if (cc[0] + cc[1] + cc[2] + cc[3] <= kShortCells && short_rounds_fit(ctx)) {
                CK(launch_short_rounds(ctx, g, rc, Qs, range, ps, pt, std::min(max_rounds - rounds, kShortRounds), opts->break_stalls));
                if ((s = read_fit(ps == 1)) != DMTZ_OK) return s;
                const unsigned long long *r = ctx->report;
                rounds += (i64)r[9];
                R.cp_rounds += (i64)r[9];
                pt_.total[PH_FIXCP] += r[11] * 1e-6;
                pt_.total[PH_APPLY] += r[12] * 1e-6;
                pt_.total[PH_PAIR] += r[13] * 1e-6;
                if (r[10]) {  // the last round's repair is left
                    pt_.mark(PH_PAIR);
                    repair_dirty(ctx, g, Qs, ctx->P.crit, ps == 1, true);
                    host_round_end(ctx, g);
                    pt_.stop();
                    if ((s = read_fit(ps == 1)) != DMTZ_OK) return s;
                }
                if ((s = stalled()) != DMTZ_OK) return s;
                for (int k = 0; k < 4; k++) cc[k] = (i64)hc[k];
                continue;
            }
            rounds++;
            R.cp_rounds++;
            const bool full = cc[0] + cc[1] + cc[2] + cc[3] >= heavy && marked >= heavy;
            pt_.mark(PH_FIXCP);
            k_fix_cp<<<pgrid, kBlock, 0, st>>>(rc, cp_lists(ctx), ps);
            pt_.mark(PH_APPLY);
            launch_next(full ? k_apply<true> : k_apply<false>, pgrid, kBlock, st, rc, range, pt, 1, ctx->changed, nullptr,
                        full ? whole : brick_marks(ctx, g));
            ctx->launches += 2;
            pt_.mark(PH_PAIR);
            if (full) {  // lists in place: nothing to take back
                repair_full(ctx, g, Qs, ctx->P.crit, ps == 1);
                const int inc = ctx->inc_scan;
                ctx->inc_scan = 0;
                host_round_end(ctx, g);
                ctx->inc_scan = inc;
            } else {
                repair_dirty(ctx, g, Qs, ctx->P.crit, ps == 1, true);
                host_round_end(ctx, g);
            }
            pt_.stop();
            if ((s = read_fit(ps == 1)) != DMTZ_OK) return s;
            if (full) marked *= block;
            if ((s = stalled()) != DMTZ_OK) return s;
            for (int k = 0; k < 4; k++) cc[k] = (i64)hc[k];
        }
        if (rounds >= max_rounds) {
            converged = 0;
            break;
        }
        if (pvp == 0) break;
        // separatrix phase (main_3d.cu:6943-7148)
        rounds++;
        R.path_rounds++;
        if (!paths_fresh) {  // else the last re-check ran on this same state
            pt_.mark(PH_PATH);
            detect_paths(ctx, g, rc, PR, pgrid, conn);
            if (walls && (s = detect_walls(ctx, g, rc, n_wall)) != DMTZ_OK) return s;
            pt_.stop();
        }
        const i64 walls_fixed = walls ? n_wall : 0;
        paths_fresh = false;
        pt_.mark(PH_FIXPATH);
        k_fix_path<<<pgrid, kBlock, 0, st>>>(rc, PR);
        if (walls_fixed > 0) {
            k_fix_wall<<<pgrid, kBlock, 0, st>>>(rc, WR);
            ctx->launches++;
        }
        pt_.mark(PH_APPLY);
        launch_next(k_apply<false>, pgrid, kBlock, st, rc, range, pt, 1, ctx->changed, nullptr, brick_marks(ctx, g));
        ctx->launches += 2;
        pt_.mark(PH_PAIR);
        repair_dirty(ctx, g, Qs, ctx->P.crit, 1, true);
        host_round_end(ctx, g);
        pt_.stop();
        if ((s = read_fit(1)) != DMTZ_OK) return s;
        if (opts->break_stalls && hc[7] == 0 && rounds < max_rounds && hc[5] + hc[6] + walls_fixed > 0) {
            if ((s = break_stall(ctx, g, rc, PR, Qs, 0, 1, R.stall_breaks, walls_fixed > 0 ? &WR : nullptr)) !=
                DMTZ_OK)
                return s;
            R.stall_breaks++;
            if ((s = read_fit(1)) != DMTZ_OK) return s;
        }
        for (int k = 0; k < 4; k++) cc[k] = (i64)hc[k];
        n_as = n_ds = n_wall = 0;
        if (!cp_any()) {
            pt_.mark(PH_PATH);
            detect_paths(ctx, g, rc, PR, pgrid, conn);
            pt_.stop();
            if ((s = read_counts()) != DMTZ_OK) return s;
            n_as = (i64)hc[5];
            n_ds = (i64)hc[6];
            if (walls && (s = detect_walls(ctx, g, rc, n_wall)) != DMTZ_OK) return s;
            paths_fresh = true;
        }
    }
    ctx->inc_scan = 0;
    CK(cudaEventRecord(e1, st));
    CK(cudaMemsetAsync(ctx->counters + 12, 0, sizeof(unsigned long long), st));
    k_count_u8<<<persistent_grid(), kBlock, 0, st>>>(ctx->changed, g.V, ctx->counters + 12);
    if (on_device) CK(cudaMemcpyAsync(decp, ctx->g, sizeof(double) * (size_t)g.V, cudaMemcpyDeviceToDevice, st));
    lg.clear();
    unsigned long long n_edited = 0;
    CK(cudaMemcpyAsync(&n_edited, ctx->counters + 12, sizeof(n_edited), cudaMemcpyDeviceToHost, st));
    if (!on_device) CK(cudaMemcpyAsync(decp, ctx->g, sizeof(double) * (size_t)g.V, cudaMemcpyDeviceToHost, st));
    if (edit_counter_out)
        CK(cudaMemcpyAsync(edit_counter_out, ctx->cnt, sizeof(int) * (size_t)g.V, cudaMemcpyDeviceToHost, st));
    int err = 0;
    CK(cudaMemcpyAsync(&err, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    CK(cudaGetLastError());
    for (int k = 0; k < 4; k++) R.final_mismatch[k] = cc[k];
    R.final_paths[0] = n_as;
    R.final_paths[1] = n_ds;
    R.final_walls = walls ? n_wall : 0;
    R.converged = converged;
    R.edited_vertices = (int64_t)n_edited;
    R.error_flags = err;
    R.seconds = ms * 1e-3;
    R.kernel_launches = ctx->launches;
    pt_.reuse();
    for (int k = 0; k < PH_N; k++) R.phase_ms[k] = pt_.total[k];
    if (rep) *rep = R;
    if (err & ERR_OOB) return fail(ctx, DMTZ_ERR_OOB, "a fix rule indexed out of range");
    if (err & ERR_WALK) return fail(ctx, DMTZ_ERR_CYCLE, "ascending path walk exceeded its step cap");
    if (!converged) return fail(ctx, DMTZ_ERR_NONCONVERGED, "round cap reached before the complexes agree");
    return DMTZ_OK;
}

dmtz_status dmtz_correct(dmtz_ctx *ctx, int W, int H, int D, const double *orig, double *decp, int on_device,
                         double rel_eps, const dmtz_opts *opts, dmtz_report *rep, int32_t *edit_counter_out) {
    return correct_impl(ctx, nullptr, W, H, D, orig, decp, on_device, rel_eps, opts, rep, edit_counter_out);
}

dmtz_status dmtz_correct_learned(dmtz_ctx *ctx, dmtz_cnn *net, int W, int H, int D, const double *orig,
                                 double *decp, int on_device, double rel_eps, const dmtz_opts *opts,
                                 dmtz_report *rep, int32_t *edit_counter_out) {
    if (!net) return fail(ctx, DMTZ_ERR_ARG, "null network");
    return correct_impl(ctx, net, W, H, D, orig, decp, on_device, rel_eps, opts, rep, edit_counter_out);
}

dmtz_status dmtz_quantize(dmtz_ctx *ctx, int W, int H, int D, const double *orig, double *decp, int on_device,
                          double rel_eps, double noise_frac, uint64_t seed) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!orig || !decp) return fail(ctx, DMTZ_ERR_ARG, "null field");
    if (!(rel_eps >= 0.0) || !std::isfinite(rel_eps) || !(noise_frac >= 0.0 && noise_frac <= 1.0))
        return fail(ctx, DMTZ_ERR_ARG, "rel_eps must be finite and >= 0, noise_frac in [0, 1]");
    CK(cudaSetDevice(ctx->device));
    if (!ctx->counters) {
        CK(dalloc(ctx, &ctx->counters, 32));
        CK(dalloc(ctx, &ctx->errword, 1));
    }
    cudaStream_t st = ctx->stream;
    const double *fd = orig;
    double *gd = decp;
    double *tmp = nullptr;
    if (!on_device) {  // staging buffers for host fields
        CK(dalloc(ctx, &tmp, 2 * g.V));
        CK(cudaMemcpyAsync(tmp, orig, sizeof(double) * (size_t)g.V, cudaMemcpyHostToDevice, st));
        fd = tmp;
        gd = tmp + g.V;
    }
    CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), st));
    k_check_finite<<<persistent_grid(), kBlock, 0, st>>>(fd, g.V, ctx->errword);
    int bad = 0;
    CK(cudaMemcpyAsync(&bad, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, st));
    double mn, mx;
    if ((s = device_minmax(ctx, fd, g.V, mn, mx)) != DMTZ_OK) {
        cudaFree(tmp);
        return s;
    }
    if (bad) {
        cudaFree(tmp);
        return fail(ctx, DMTZ_ERR_ARG, "input contains NaN or Inf");
    }
    k_quantize<<<persistent_grid(), kBlock, 0, st>>>(g.V, fd, gd, mn, (mx - mn) * rel_eps, noise_frac, seed);
    if (!on_device) CK(cudaMemcpyAsync(decp, gd, sizeof(double) * (size_t)g.V, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    cudaFree(tmp);
    CK(cudaGetLastError());
    return DMTZ_OK;
}

dmtz_status dmtz_features(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp, int on_device,
                          double rel_eps, void *feat, uint8_t *active) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!feat || !active || ((uintptr_t)feat & 15)) return fail(ctx, DMTZ_ERR_ARG, "feat must be 16-byte aligned");
    if (!(rel_eps >= 0.0) || !std::isfinite(rel_eps)) return fail(ctx, DMTZ_ERR_ARG, "rel_eps must be finite and >= 0");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, orig, g.V, on_device)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->g, decp, g.V, on_device)) != DMTZ_OK) return s;
    double mn, mx;
    if ((s = device_minmax(ctx, ctx->f, g.V, mn, mx)) != DMTZ_OK) return s;
    run_pairing(ctx, g, view(ctx->P, ctx->f), nullptr, 1);
    run_pairing(ctx, g, view(ctx->Q, ctx->g), nullptr, 1);
    if ((s = features_into(ctx, g, (mx - mn) * rel_eps, static_cast<__nv_bfloat16 *>(feat), active)) != DMTZ_OK)
        return s;
    CK(cudaStreamSynchronize(ctx->stream));
    return DMTZ_OK;
}

}  // extern "C"
// pointer jumping to a fixed point of several label arrays
template <class I>
static dmtz_status jump_to_roots(dmtz_ctx *ctx, I *const *lab, const i64 *n, int arrays) {
    for (int round = 0; round < 64; round++) {
        CK(cudaMemsetAsync(ctx->errword, 0, sizeof(int), ctx->stream));
        for (int k = 0; k < arrays; k++)
            k_jump<I><<<persistent_grid(), kBlock, 0, ctx->stream>>>(lab[k], n[k], ctx->errword);
        int left = 0;
        CK(cudaMemcpyAsync(&left, ctx->errword, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        if (!left) return DMTZ_OK;
    }
    return fail(ctx, DMTZ_ERR_CYCLE, "manifold labels did not settle (cycle in the gradient paths)");
}
extern "C" {

dmtz_status dmtz_labels(dmtz_ctx *ctx, int W, int H, int D, const double *data, int on_device, int32_t *desc,
                        int32_t *asc) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (g.F >= INT32_MAX) return fail(ctx, DMTZ_ERR_ARG, "grid too large for 32-bit reference ids");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, data, g.V, on_device)) != DMTZ_OK) return s;
    run_pairing(ctx, g, view(ctx->P, ctx->f), nullptr, 1);
    // int32 labels: 6 V is below F, and F below 2^31, but for columns of 2 x 2 vertices, which
    // are short.  The vertices' labels are the result itself.
    const size_t nd = work_round(sizeof(int32_t) * (size_t)g.V), na = work_round(sizeof(int32_t) * 6 * (size_t)g.V);
    WorkDone done{ctx};
    CK(work_take(ctx, nd + 2 * na));
    int32_t *dl = reinterpret_cast<int32_t *>(ctx->work), *al = reinterpret_cast<int32_t *>(ctx->work + nd),
            *aout = reinterpret_cast<int32_t *>(ctx->work + nd + na);
    const unsigned pg = persistent_grid();
    k_desc_init<int32_t><<<pg, kBlock, 0, ctx->stream>>>(g, ctx->P.pv, dl);
    k_asc_init<int32_t><<<pg, kBlock, 0, ctx->stream>>>(g, ctx->P.tcode, al);
    int32_t *lab[2] = {dl, al};
    const i64 n[2] = {g.V, 6 * g.V};
    if ((s = jump_to_roots<int32_t>(ctx, lab, n, 2)) != DMTZ_OK) return s;
    k_asc_out<int32_t><<<pg, kBlock, 0, ctx->stream>>>(g, al, aout);
    CK(cudaMemcpyAsync(desc, dl, sizeof(int32_t) * (size_t)g.V, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(asc, aout, sizeof(int32_t) * (size_t)g.T, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaGetLastError());
    return DMTZ_OK;
}

}  // extern "C"
template <class I>
static dmtz_status agreement(dmtz_ctx *ctx, const Grid &g, int64_t out[5]) {
    cudaStream_t st = ctx->stream;
    const size_t nd = work_round(sizeof(I) * (size_t)g.V), na = work_round(sizeof(I) * 6 * (size_t)g.V);
    WorkDone done{ctx};
    if (work_take(ctx, 2 * nd + 2 * na + 256) != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, DMTZ_ERR_CUDA, "cannot allocate label buffers");
    }
    I *lab[4];
    const i64 n[4] = {g.V, g.V, 6 * g.V, 6 * g.V};
    for (int k = 0; k < 4; k++) lab[k] = reinterpret_cast<I *>(ctx->work + (k < 2 ? k * nd : 2 * nd + (k - 2) * na));
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(ctx->work + 2 * nd + 2 * na);
    const unsigned pg = persistent_grid();
    k_desc_init<I><<<pg, kBlock, 0, st>>>(g, ctx->P.pv, lab[0]);
    k_desc_init<I><<<pg, kBlock, 0, st>>>(g, ctx->Q.pv, lab[1]);
    k_asc_init<I><<<pg, kBlock, 0, st>>>(g, ctx->P.tcode, lab[2]);
    k_asc_init<I><<<pg, kBlock, 0, st>>>(g, ctx->Q.tcode, lab[3]);
    const dmtz_status s = jump_to_roots<I>(ctx, lab, n, 4);
    if (s != DMTZ_OK) return s;
    unsigned long long h[5];
    CK(cudaMemsetAsync(cnt, 0, sizeof(h), st));
    k_sep_agree<I><<<pg, kBlock, 0, st>>>(g, ctx->P.crit, ctx->Q.crit, lab[0], lab[1], lab[2], lab[3], cnt);
    CK(cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (int k = 0; k < 5; k++) out[k] = (int64_t)h[k];
    CK(cudaGetLastError());
    return DMTZ_OK;
}
extern "C" {

dmtz_status dmtz_separatrix_agreement(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                                      int on_device, int64_t out[5]) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!out) return fail(ctx, DMTZ_ERR_ARG, "null output");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, orig, g.V, on_device)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->g, decp, g.V, on_device)) != DMTZ_OK) return s;
    run_pairing(ctx, g, view(ctx->P, ctx->f), nullptr, 1);
    run_pairing(ctx, g, view(ctx->Q, ctx->g), nullptr, 1);
    return 6 * g.V <= INT32_MAX ? agreement<int32_t>(ctx, g, out) : agreement<i64>(ctx, g, out);
}

dmtz_status dmtz_link_classes(dmtz_ctx *ctx, int W, int H, int D, const double *data, int on_device, uint8_t *out,
                              int64_t counts[6]) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (!counts) return fail(ctx, DMTZ_ERR_ARG, "null counts");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, data, g.V, on_device)) != DMTZ_OK) return s;
    cudaStream_t st = ctx->stream;
    WorkDone done{ctx};
    if (work_take(ctx, 256 + (out ? (size_t)g.V : 0)) != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, DMTZ_ERR_CUDA, "cannot allocate link buffers");
    }
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(ctx->work);
    uint8_t *dout = out ? ctx->work + 256 : nullptr;
    unsigned long long h[6];
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(h), st);
    k_link_classes<<<persistent_grid(), kBlock, 0, st>>>(g, ctx->f, dout, cnt);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && out) e = cudaMemcpyAsync(out, dout, (size_t)g.V, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(ctx, DMTZ_ERR_CUDA, cudaGetErrorString(e));
    for (int k = 0; k < 6; k++) counts[k] = (int64_t)h[k];
    CK(cudaGetLastError());
    return DMTZ_OK;
}

dmtz_status dmtz_device_name(const dmtz_ctx *ctx, char *buf, int len) {
    if (!ctx || !buf || len < 1) return DMTZ_ERR_ARG;
    cudaDeviceProp p;
    if (cudaGetDeviceProperties(&p, ctx->device) != cudaSuccess) return DMTZ_ERR_CUDA;
    snprintf(buf, (size_t)len, "%s", p.name);
    return DMTZ_OK;
}

dmtz_status dmtz_set_tuning(dmtz_ctx *ctx, int shape, int blocks_per_sm) {
    if (!ctx || shape < 0 || shape >= DMTZ_NSHAPES || blocks_per_sm < 1 || blocks_per_sm > 64) return DMTZ_ERR_ARG;
    ctx->tune_shape = shape;
    ctx->tune_bps = blocks_per_sm;
    return DMTZ_OK;
}

dmtz_status dmtz_set_list_reserve(dmtz_ctx *ctx, double fraction, int64_t min_entries) {
    if (!ctx || !(fraction >= 0.0 && fraction <= 1.0) || min_entries < 1) return DMTZ_ERR_ARG;
    ctx->list_frac = fraction;
    ctx->list_min = min_entries;
    cudaSetDevice(ctx->device);
    for (int k = 0; k < 4; k++) {  // reallocated with the new reserve by the next call
        cudaFree(ctx->lists[k]);
        cudaFree(ctx->list_tmp[k]);
        ctx->lists[k] = ctx->list_tmp[k] = nullptr;
        ctx->capL[k] = 0;
    }
    return DMTZ_OK;
}

dmtz_status dmtz_get_tuning(const dmtz_ctx *ctx, int *shape, int *blocks_per_sm) {
    if (!ctx) return DMTZ_ERR_ARG;
    if (shape) *shape = ctx->tune_shape;
    if (blocks_per_sm) *blocks_per_sm = ctx->tune_bps;
    return DMTZ_OK;
}

// What a choice is worth to corrections: the brick kernel over all bricks is not it, because
// repairs take short lists of bricks, large grids march, and the other shapes lack short
// rounds (64^3 Gaussian mixture, 108 rounds: 5.6 ms with 8 x 4 x 4, 6.7 with 16 x 4 x 2, 7.1
// with 32 x 2 x 2).  So every choice corrects decp for kTuneRounds rounds, with the error
// that decp has as its bound, and another choice than 8 x 4 x 4 and 32 has to be faster by
// kTuneGain.
static constexpr int kTuneRounds = 32;
static constexpr double kTuneGain = 0.02;

dmtz_status dmtz_autotune(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp, int on_device,
                          int best[2], double *best_ms) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, orig, g.V, on_device)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->g, decp, g.V, on_device)) != DMTZ_OK) return s;
    cudaStream_t st = ctx->stream;
    const FieldState Ps = view(ctx->P, ctx->f), Qs = view(ctx->Q, ctx->g);
    run_pairing(ctx, g, Ps, nullptr, 1);
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    static const int bps_opts[4] = {8, 16, 32, 64};
    float sweep[DMTZ_NSHAPES][4];  // ms of the brick kernel over all bricks
    for (int sh = 0; sh < DMTZ_NSHAPES; sh++) {
        if (!shape_fits(g, sh)) continue;
        for (int bi = 0; bi < 4; bi++) {
            ctx->tune_shape = sh;
            ctx->tune_bps = bps_opts[bi];
            i64 nb;
            const BrickList bl = all_bricks(g, sh, nb);
            const unsigned gr = brick_grid(ctx, nb);
            grad_bricks(g, Qs, bl, gr, st);  // warm
            float t_min = 1e30f;
            for (int r = 0; r < 3; r++) {
                CK(cudaEventRecord(e0, st));
                grad_bricks(g, Qs, bl, gr, st);
                CK(cudaEventRecord(e1, st));
                CK(cudaEventSynchronize(e1));
                float t = 0;
                cudaEventElapsedTime(&t, e0, e1);
                t_min = std::min(t_min, t);
            }
            sweep[sh][bi] = t_min;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    double mn, mx;
    unsigned long long gap = 0;
    if ((s = device_minmax(ctx, ctx->f, g.V, mn, mx)) != DMTZ_OK) return s;
    CK(cudaMemsetAsync(ctx->counters + 9, 0, sizeof(gap), st));
    k_max_gap<<<persistent_grid(), kBlock, 0, st>>>(ctx->f, ctx->g, g.V, ctx->counters + 9);
    CK(cudaMemcpyAsync(&gap, ctx->counters + 9, sizeof(gap), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const double rel = key_to_double(gap) / (mx - mn);
    int bs = 0, bb = 2;
    double *copy = nullptr;  // original, decompressed, corrected
    bool can = std::isfinite(rel) && rel > 0;
    if (can && dalloc(ctx, &copy, 3 * g.V) != cudaSuccess) {  // no room for them: the default shape
        cudaGetLastError();
        can = false;
    }
    if (can) {
        const size_t bytes = sizeof(double) * (size_t)g.V;
        cudaMemcpyAsync(copy, ctx->f, bytes, cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(copy + g.V, ctx->g, bytes, cudaMemcpyDeviceToDevice, st);
        const std::string err = ctx->err;
        double best_t = 1e30;
        auto rounds = [&](int sh, int bi) {  // seconds; a first run that takes long is not repeated
            double t = 1e30;
            ctx->tune_shape = sh;
            ctx->tune_bps = bps_opts[bi];
            for (int r = 0; r < 3; r++) {
                dmtz_opts o{};
                dmtz_report rep{};
                o.preserve_saddles = o.preserve_vpath = o.preserve_geometry = o.break_stalls = 1;
                o.max_rounds = kTuneRounds;
                cudaMemcpyAsync(copy + 2 * g.V, copy + g.V, bytes, cudaMemcpyDeviceToDevice, st);
                const dmtz_status q = dmtz_correct(ctx, W, H, D, copy, copy + 2 * g.V, 1, rel, &o, &rep, nullptr);
                if (q != DMTZ_OK && q != DMTZ_ERR_NONCONVERGED) return 1e30;
                t = std::min(t, rep.seconds);
                if (t > 0.05) break;
            }
            return t;
        };
        best_t = rounds(bs, bb);
        for (int sh = 0; sh < DMTZ_NSHAPES; sh++) {
            if (!shape_fits(g, sh)) continue;
            for (int bi = 0; bi < 4; bi++) {
                if (sh == 0 && bi == 2) continue;
                const double t = rounds(sh, bi);
                if (t < (1 - kTuneGain) * best_t) {
                    best_t = t;
                    bs = sh;
                    bb = bi;
                }
            }
        }
        cudaFree(copy);
        ctx->err = err;
    } else {
        for (int bi = 0; bi < 4; bi++)
            if (sweep[0][bi] < sweep[0][bb]) bb = bi;
    }
    ctx->tune_shape = bs;
    ctx->tune_bps = bps_opts[bb];
    if (best) {
        best[0] = bs;
        best[1] = bps_opts[bb];
    }
    if (best_ms) *best_ms = sweep[bs][bb];
    CK(cudaGetLastError());
    return DMTZ_OK;
}

dmtz_status dmtz_correct_batch(dmtz_ctx *ctx, int n, const dmtz_instance *inst, const dmtz_opts *opts,
                               dmtz_report *reports, dmtz_status *status, int workers) {
    if (!ctx || n < 0 || (n > 0 && (!inst || !opts))) return DMTZ_ERR_ARG;
    if (workers < 1) workers = 8;
    workers = std::min(workers, std::max(n, 1));
    while ((int)ctx->pool.size() < workers) {
        dmtz_ctx *w = nullptr;
        const dmtz_status cs = dmtz_ctx_create(&w, ctx->device);
        if (cs != DMTZ_OK) return fail(ctx, cs, "cannot create a worker context");
        ctx->pool.push_back(w);
    }
    // every worker's buffers are sized once for the largest extents of the
    // batch: a reallocation in the middle would free device memory, and
    // cudaFree waits for the whole device, i.e. for the other workers
    int mW = 2, mH = 2, mD = 2;
    for (int i = 0; i < n; i++) {
        mW = std::max(mW, inst[i].W);
        mH = std::max(mH, inst[i].H);
        mD = std::max(mD, inst[i].D);
    }
    Grid gmax;
    if (n > 0 && check_dims(ctx, mW, mH, mD, gmax) == DMTZ_OK) {
        for (int k = 0; k < workers; k++) {
            dmtz_ctx *w = ctx->pool[k];
            w->list_frac = ctx->list_frac;
            w->list_min = ctx->list_min;
            cudaSetDevice(w->device);
            const dmtz_status es = ensure(w, gmax);
            if (es != DMTZ_OK) return fail(ctx, es, "cannot size worker buffers: " + w->err);
        }
    }
    std::atomic<int> next(0);
    std::vector<dmtz_status> st((size_t)n, DMTZ_OK);
    auto work = [&](dmtz_ctx *w) {
        w->tune_shape = ctx->tune_shape;
        w->tune_bps = ctx->tune_bps;
        w->list_frac = ctx->list_frac;
        w->list_min = ctx->list_min;
        std::vector<double> fo, go;
        for (int i = next++; i < n; i = next++) {
            const dmtz_instance &I = inst[i];
            const size_t V = (size_t)std::max(I.W, 0) * (size_t)std::max(I.H, 0) * (size_t)std::max(I.D, 0);
            if (!I.orig || !I.decp || !I.out || V == 0 || (I.dtype != DMTZ_F64 && I.dtype != DMTZ_F32)) {
                st[i] = DMTZ_ERR_ARG;
                continue;
            }
            const double *f64 = (const double *)I.orig;
            if (I.dtype == DMTZ_F32) {  // float32 widens exactly; the correction runs in float64
                fo.resize(V);
                const float *a = (const float *)I.orig, *b = (const float *)I.decp;
                for (size_t k = 0; k < V; k++) {
                    fo[k] = a[k];
                    I.out[k] = b[k];
                }
                f64 = fo.data();
            } else {
                memcpy(I.out, I.decp, V * sizeof(double));
            }
            dmtz_report r;
            st[i] = dmtz_correct(w, I.W, I.H, I.D, f64, I.out, 0, I.rel_eps, opts, &r, nullptr);
            if (reports) reports[i] = r;
        }
    };
    std::vector<std::thread> th;
    for (int k = 0; k < workers; k++) th.emplace_back(work, ctx->pool[k]);
    for (auto &t : th) t.join();
    dmtz_status res = DMTZ_OK;
    for (int i = 0; i < n; i++) {
        if (status) status[i] = st[i];
        if (st[i] != DMTZ_OK && res == DMTZ_OK) {
            res = st[i];
            ctx->err = "instance " + std::to_string(i) + " failed with status " + std::to_string((int)st[i]);
        }
    }
    return res;
}

dmtz_status dmtz_profile_sweep(dmtz_ctx *ctx, int W, int H, int D, const double *orig, const double *decp,
                               int on_device, int reps, double ms[7]) {
    Grid g;
    dmtz_status s = check_dims(ctx, W, H, D, g);
    if (s != DMTZ_OK) return s;
    if (reps < 1) return fail(ctx, DMTZ_ERR_ARG, "reps must be >= 1");
    CK(cudaSetDevice(ctx->device));
    if ((s = ensure(ctx, g)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->f, orig, g.V, on_device)) != DMTZ_OK) return s;
    if ((s = upload(ctx, ctx->g, decp, g.V, on_device)) != DMTZ_OK) return s;
    cudaStream_t st = ctx->stream;
    const FieldState Ps = view(ctx->P, ctx->f), Qs = view(ctx->Q, ctx->g);
    run_pairing(ctx, g, Ps, nullptr, 1);
    run_pairing(ctx, g, Qs, ctx->P.crit, 1);  // warm-up
    cudaEvent_t ev[2];
    for (auto &e : ev) CK(cudaEventCreate(&e));
    CK(cudaEventRecord(ev[0], st));
    for (int r = 0; r < reps; r++) grad_full(ctx, g, Qs);
    CK(cudaEventRecord(ev[1], st));
    CK(cudaEventSynchronize(ev[1]));
    float total = 0;
    cudaEventElapsedTime(&total, ev[0], ev[1]);
    for (auto &e : ev) cudaEventDestroy(e);
    for (int k = 0; k < 7; k++) ms[k] = 0;
    ms[0] = ms[6] = total / reps;  // one kernel does every pass
    CK(cudaGetLastError());
    return DMTZ_OK;
}

}  // extern "C"

// =============================================================================
// allocation-free extraction (dmtz_extract_noalloc)
// =============================================================================
namespace {

// byte layout of the fixed scratch: the FieldState arrays of one field, each
// starting on a 256-byte boundary
constexpr i64 kNaV = DMTZ_NOALLOC_MAX_VERTICES;
constexpr i64 na_round(i64 b) { return (b + 255) / 256 * 256; }
constexpr i64 kNaPv = 0;
constexpr i64 kNaEup = kNaPv + na_round(kNaV * 1);
constexpr i64 kNaFup = kNaEup + na_round(kNaV * 4);
// no criticality array: the export reads the pairing state alone
constexpr i64 kNaBytes = kNaFup + na_round(kNaV * 4);

}  // namespace

// Every array of the gradient state is fully rewritten by the passes before it
// is read, so the contents a previous call left behind need no clearing.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

namespace {
std::mutex g_noalloc_mu;
constexpr int kNaMaxDevices = 64;
void *g_noalloc_addr[kNaMaxDevices] = {};

// device address of the scratch on the current device, looked up once per
// device.  The address belongs to the device's primary context: a
// cudaDeviceReset between calls (which reloads the module) is not supported.
cudaError_t noalloc_scratch(int dev, unsigned char **out) {
    if (dev < 0 || dev >= kNaMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_addr[dev] = p;
    }
    *out = (unsigned char *)g_noalloc_addr[dev];
    return cudaSuccess;
}
}  // namespace

extern "C" dmtz_status dmtz_extract_noalloc(int W, int H, int D, const double *data, int32_t *PV, int32_t *PE,
                                            int32_t *PF, int32_t *PT, void *stream) {
    if (W < 2 || H < 2 || D < 2 || !data || !PV || !PE || !PF || !PT) return DMTZ_ERR_ARG;
    const Grid g = make_grid(W, H, D);
    if (g.V > kNaV) return DMTZ_ERR_TOO_LARGE;
    // an error left by the caller's own earlier work stays the caller's: it is
    // reported, not cleared, and nothing is launched
    if (cudaPeekAtLastError() != cudaSuccess) return DMTZ_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DMTZ_ERR_CUDA;
    unsigned char *base = nullptr;
    if (noalloc_scratch(dev, &base) != cudaSuccess) return DMTZ_ERR_CUDA;
    FieldState s;
    s.val = data;
    s.pv = (uint8_t *)(base + kNaPv);
    s.eup = (uint32_t *)(base + kNaEup);
    s.fup = (uint32_t *)(base + kNaFup);
    s.crit = nullptr;
    s.tcode = nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    i64 nb;
    const BrickList bl = all_bricks(g, 0, nb);
    grad_bricks(g, s, bl, (unsigned)std::max<i64>(1, std::min<i64>(nb, persistent_grid())), st);
    k_export<<<grid_for(g.V), kBlock, 0, st>>>(g, s, PV, PE, PF, PT);
    return cudaGetLastError() == cudaSuccess ? DMTZ_OK : DMTZ_ERR_CUDA;
}
