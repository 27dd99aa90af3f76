// gradient.cuh — the discrete gradient on sm_103a, all five pairing passes and
// the criticality test in one kernel.
//
// Reference: processVertices (main_3d.cu:1930-1988), edgePairingKernel
// (:1990-2113) and trianglePairingKernel (:2197-2316), run in the order
// vertices, edges(a2=0), triangles(a2=0), edges(a2=1), triangles(a2=1).
//
// Every pair the five passes make joins two cells with the same highest
// vertex (in the (value, id) order), so the passes can be restated without
// their sequence.  For a cell c let b(c) be the lowest of the vertices that
// span a coface with it.
//   - A vertex v pairs with the edge to its lowest neighbour, if that is below v.
//   - For a triangle or tetrahedron t call its facet opposite corner j "pointing"
//     when b(facet) is corner j.  If the facet opposite t's lowest corner points,
//     t is paired with it (the a2=0 passes); else, if the facet opposite the second
//     lowest corner points, t is paired with that one (the a2=1 passes: the
//     candidate lies between the facet's lowest and second lowest corner, and t
//     is still free exactly when the first facet does not point).  No other
//     facet pairs with t.
// The remaining conditions of the passes follow: an edge whose candidate is below both ends
// points at a triangle whose lowest corner that candidate is; an edge paired
// with its vertex points, if at all, at a triangle that the a2=0 pass claims; and so on.
//
// So the work per anchor is: 7 argmins over 4 or 6 vertices (edges), 12
// comparisons (triangles), 7 order bits (edges), one argmin over 14 (the
// vertex), all on 64-bit order keys, and then logic on bit vectors: one bit
// per (triangle, its edge) or (tetrahedron, its facet), the twelve triangles or six
// tetrahedra of an anchor side by side in a word.
//
// Three stages, each reading the previous one's words at neighbour anchors:
//   stage 1 (anchors -1 .. S): keys -> pointing bits and order bits
//   stage 2 (anchors -1 .. S-1): the triangles' and tetrahedra's choice
//   stage 3 (anchors 0 .. S-1): edge and triangle codes, criticality
// Vertices outside the grid carry the key ~0, above every real key, so they
// are never chosen; cells that do not exist are masked in stage 3.
//
// Bound by the ALU pipe (64-bit compares and selects: 81 % busy at 128^3, where
// 8 + 17 bytes per vertex are read and written).  One pass per kernel, as the
// reference has them, took 3454 thread instructions per anchor, six stagings
// of the state between the passes and a separate kernel per pass for the
// surface anchors; this takes about 1000.  Measured on GB300, a whole
// gradient: 256^3 3.32 -> 0.82 ms, 120 x 89 x 101 337 -> 72 us, 64^3 25 us,
// 16^3 6.2 us.  A repair also covers less: a changed value reaches anchors
// 2 below to 1 above, where the passes' widest reach was 5 to either side.
#pragma once
#include <algorithm>
#include <utility>

#include "dmtz_common.cuh"

namespace dmtz {
namespace cxt {
#define TOPO_QUAL static constexpr
#include "topology_tables.inc"
#undef TOPO_QUAL

__host__ __device__ constexpr int cdir(int dx, int dy, int dz) {
    return (dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1) ? -1
                                                                         : TOPO_DIR_LUT[(dx + 1) + 3 * (dy + 1) + 9 * (dz + 1)];
}
__host__ __device__ constexpr int ccx(int c) { return c & 1; }
__host__ __device__ constexpr int ccy(int c) { return (c >> 1) & 1; }
__host__ __device__ constexpr int ccz(int c) { return (c >> 2) & 1; }
// Candidates in increasing vertex id order.  Every candidate of a selection
// is the anchor plus a compile-time offset (-1..2 per axis), and ids grow with
// (dz, dy, dx) lexicographically, so visiting candidates in that order and
// keeping the first of equal keys (a strict key comparison) takes the
// smallest id among equal values: the (value, id) tie-break of
// compare_vertices (main_3d.cu:1043-1049) without comparing ids.
__host__ __device__ constexpr int lex3(int x, int y, int z) { return (z + 4) * 64 + (y + 4) * 8 + (x + 4); }
__host__ __device__ constexpr int dir_by_id(int r) {
    for (int i = 0; i < 14; i++) {
        int rank = 0;
        for (int j = 0; j < 14; j++)
            rank += lex3(TOPO_DIRS[j][0], TOPO_DIRS[j][1], TOPO_DIRS[j][2]) <
                    lex3(TOPO_DIRS[i][0], TOPO_DIRS[i][1], TOPO_DIRS[i][2]);
        if (rank == r) return i;
    }
    return -1;
}
__host__ __device__ constexpr bool dir_up(int i) { return lex3(TOPO_DIRS[i][0], TOPO_DIRS[i][1], TOPO_DIRS[i][2]) > lex3(0, 0, 0); }
__host__ __device__ constexpr int edge_cand_by_id(int k, int r) {
    for (int i = 0; i < TOPO_EDGE_NCOF[k]; i++) {
        int rank = 0;
        for (int j = 0; j < TOPO_EDGE_NCOF[k]; j++)
            rank += lex3(TOPO_EDGE_THIRD[k][j][0], TOPO_EDGE_THIRD[k][j][1], TOPO_EDGE_THIRD[k][j][2]) <
                    lex3(TOPO_EDGE_THIRD[k][i][0], TOPO_EDGE_THIRD[k][i][1], TOPO_EDGE_THIRD[k][i][2]);
        if (rank == r) return i;
    }
    return -1;
}

// ------------------------------------------------------------- word layouts
// Every triangle has exactly one face-diagonal edge (families 3, 4, 5); its
// corner opposite that edge gets label 2, the other two labels 0 and 1 (in id
// order, highest first).  A (triangle, edge) incidence is bit 12 label + slot
// of an "A" word for labels 0 and 1, bit slot of a "B" word for label 2, so a
// family's incidences all lie in one word.
__host__ __device__ constexpr bool diag(int k) { return k >= 3 && k <= 5; }
__host__ __device__ constexpr int tri_label(int s, int j) {
    if (diag(TOPO_FACE_EDGE[s][j][3])) return 2;
    int l = 0;
    for (int q = 0; q < j; q++) l += diag(TOPO_FACE_EDGE[s][q][3]) ? 0 : 1;
    return l;
}
__host__ __device__ constexpr int tri_corner_of_label(int s, int l) {
    for (int j = 0; j < 3; j++)
        if (tri_label(s, j) == l) return j;
    return -1;
}
__host__ __device__ constexpr uint32_t tri_bit(int s, int j) {
    return tri_label(s, j) == 2 ? 1u << s : 1u << (12 * tri_label(s, j) + s);
}
// corner index of the triangle that coface i of edge family k is opposite to
__host__ __device__ constexpr int edge_cof_corner(int k, int i) {
    const int s = TOPO_EDGE_COF[k][i][3];
    for (int j = 0; j < 3; j++)
        if (TOPO_FACE_EDGE[s][j][3] == k && TOPO_FACE_EDGE[s][j][4] == i) return j;
    return -1;
}
__host__ __device__ constexpr uint32_t edge_bit(int k, int i) {
    return tri_bit(TOPO_EDGE_COF[k][i][3], edge_cof_corner(k, i));
}
// all incidences of family k
__host__ __device__ constexpr uint32_t edge_mask(int k) {
    uint32_t m = 0;
    for (int i = 0; i < TOPO_EDGE_NCOF[k]; i++) m |= edge_bit(k, i);
    return m;
}
// incidences of family k whose code (coface index + 1) has bit b
__host__ __device__ constexpr uint32_t edge_code_mask(int k, int b) {
    uint32_t m = 0;
    for (int i = 0; i < TOPO_EDGE_NCOF[k]; i++)
        if (((i + 1) >> b) & 1) m |= edge_bit(k, i);
    return m;
}
// incidences (A or B word) whose edge is anchored at the triangle's anchor + corner c
__host__ __device__ constexpr uint32_t tri_at(bool b_word, int c) {
    uint32_t m = 0;
    for (int s = 0; s < 12; s++)
        for (int j = 0; j < 3; j++) {
            const signed char *e = TOPO_FACE_EDGE[s][j];
            if (diag(e[3]) == b_word && e[0] + 2 * e[1] + 4 * e[2] == c) m |= tri_bit(s, j);
        }
    return m;
}
// An edge's order bit says "its lower-id end is below its higher-id end".
// For the edge between the corners labelled 2 and l (opposite label 1 - l):
// bit s is set where that reads the other way round (label 2 has the higher id)
__host__ __device__ constexpr uint32_t tri_flip(int l) {
    uint32_t m = 0;
    for (int s = 0; s < 12; s++)
        if (tri_corner_of_label(s, 2) < tri_corner_of_label(s, l)) m |= 1u << s;
    return m;
}
// (tetrahedron, facet) incidence: bit 6 j + tetrahedron slot, j = the corner
// opposite the facet (by id, highest first)
__host__ __device__ constexpr uint32_t face_bit(int s, int i) {
    const int t = TOPO_FACE_COF[s][i][3];
    for (int j = 0; j < 4; j++)
        if (TOPO_TET_FACE[t][j][3] == s && TOPO_TET_FACE[t][j][4] == i) return 1u << (6 * j + t);
    return 0;
}
__host__ __device__ constexpr uint32_t tet_at(int c) {
    uint32_t m = 0;
    for (int t = 0; t < 6; t++)
        for (int j = 0; j < 4; j++) {
            const signed char *f = TOPO_TET_FACE[t][j];
            if (f[0] + 2 * f[1] + 4 * f[2] == c) m |= 1u << (6 * j + t);
        }
    return m;
}
// (tetrahedron, edge) order bits: bit 6 p + slot, p = the corner pair (0 1),
// (0 2), (0 3), (1 2), (1 3) in word 4; the pair (2 3) in bits 24.. of word 3
__host__ __device__ constexpr int tet_edge_family(int ca, int cb) {
    const int a = ca & ~cb, b = cb & ~ca;
    for (int k = 0; k < 7; k++)
        if ((TOPO_EDGE_V[k][0] == a && TOPO_EDGE_V[k][1] == b) || (TOPO_EDGE_V[k][0] == b && TOPO_EDGE_V[k][1] == a))
            return k;
    return -1;
}
__host__ __device__ constexpr uint32_t tet_order_bits(int word, int family, int c) {  // family / c: -1 = any
    uint32_t m = 0;
    for (int t = 0; t < 6; t++) {
        int p = 0;
        for (int i = 0; i < 4; i++)
            for (int j = i + 1; j < 4; j++, p++) {
                const int ca = TOPO_TET_V[t][i], cb = TOPO_TET_V[t][j];
                if ((family >= 0 && tet_edge_family(ca, cb) != family) || (c >= 0 && (ca & cb) != c)) continue;
                if (p < 5 && word == 4) m |= 1u << (6 * p + t);
                if (p == 5 && word == 3) m |= 1u << (24 + t);
            }
    }
    return m;
}
// edge family of a vertex's direction, and whether the vertex is then the
// edge's higher-id end
__host__ __device__ constexpr int dir_family(int d) {
    for (int k = 0; k < 7; k++) {
        const int p = TOPO_EDGE_V[k][0], q = TOPO_EDGE_V[k][1];
        if (TOPO_CORNER_DIR[p][q] == d || TOPO_CORNER_DIR[q][p] == d) return k;
    }
    return -1;
}
__host__ __device__ constexpr bool dir_from_high(int d) {
    const int k = dir_family(d);
    return TOPO_CORNER_DIR[TOPO_EDGE_V[k][0]][TOPO_EDGE_V[k][1]] == d;
}
// edges (bit k) whose higher-id (hi = 1) or lower-id end is corner c
__host__ __device__ constexpr uint32_t ends_at(int hi, int c) {
    uint32_t m = 0;
    for (int k = 0; k < 7; k++)
        if (TOPO_EDGE_V[k][hi ? 0 : 1] == c) m |= 1u << k;
    return m;
}
__host__ __device__ constexpr uint32_t edges_at(int c) { return ends_at(0, c) | ends_at(1, c); }
// cells that need the anchor's +x (bit 0), +y (1) or +z (2) neighbour
__host__ __device__ constexpr uint32_t edges_over(int axis) {
    uint32_t m = 0;
    for (int k = 0; k < 7; k++)
        if (((TOPO_EDGE_V[k][0] | TOPO_EDGE_V[k][1]) >> axis) & 1) m |= 1u << k;
    return m;
}
__host__ __device__ constexpr uint32_t faces_over(int axis) {
    uint32_t m = 0;
    for (int s = 0; s < 12; s++)
        if (((TOPO_FACE_V[s][0] | TOPO_FACE_V[s][1] | TOPO_FACE_V[s][2]) >> axis) & 1) m |= 1u << s;
    return m;
}
// (tetrahedron, facet) incidences whose bit moves up by d to become the code
// of the facet (coface i of slot s: bit 2 s + i of fup, code i + 1)
__host__ __device__ constexpr int bit_index(uint32_t m) {
    int i = 0;
    while (!((m >> i) & 1u)) i++;
    return i;
}
__host__ __device__ constexpr uint32_t face_move(int d) {
    uint32_t m = 0;
    for (int s = 0; s < 12; s++)
        for (int i = 0; i < 2; i++)
            if (2 * s + i - bit_index(face_bit(s, i)) == d) m |= face_bit(s, i);
    return m;
}
// the first coface's incidence of every triangle slot
__host__ __device__ constexpr uint32_t face_first() {
    uint32_t m = 0;
    for (int s = 0; s < 12; s++) m |= face_bit(s, 0);
    return m;
}
}  // namespace cxt

template <int... Is, class F>
__host__ __device__ __forceinline__ void static_for(std::integer_sequence<int, Is...>, F &&f) {
    (f(std::integral_constant<int, Is>{}), ...);
}
#define DMTZ_FOR(N, VAR, ...) static_for(std::make_integer_sequence<int, N>{}, [&](auto VAR) __VA_ARGS__)

constexpr uint64_t kKeyAbsent = ~0ull;  // key of a vertex outside the grid

// keep the lower of two keys and what goes with it
__host__ __device__ __forceinline__ void take_lower(uint64_t &bk, uint32_t &sel, uint64_t kn, uint32_t c) {
    const bool better = kn < bk;
    bk = better ? kn : bk;
    sel = better ? c : sel;
}

// ------------------------------------------------------------------- stage 1
// Words of one anchor:
//   w.x: pointing bits of its edges, A layout; bits 24..30: edge family of the
//        vertex's pair where the vertex is the edge's higher-id end
//   w.y: pointing bits, B layout; bits 12..23: order bits, B layout; bits
//        24..30: the family where the vertex is the lower-id end
//   w.z: order bits of its edges, A layout; bit 24: its steepest descent is not
//        the original's (set by the kernels that keep PathFlags)
//   w.w: pointing bits of its triangles; bits 24..29: tetrahedron order bits (2 3)
//   w4:  tetrahedron order bits
// km, k0, kp: the anchor's key in the planes z-1, z, z+1, rows ROW apart.
struct StarWords {
    uint32_t x, y, z, w, w4;
    int pv;  // steepest-descent direction, 15 = none
};
template <int ROW>
__host__ __device__ __forceinline__ StarWords grad_stage1(const uint64_t *km, const uint64_t *k0, const uint64_t *kp) {
    auto key = [&](auto X, auto Y, auto Z) -> uint64_t {
        constexpr int x = decltype(X)::value, y = decltype(Y)::value, z = decltype(Z)::value;
        return (z < 0 ? km : z > 0 ? kp : k0)[x + y * ROW];
    };
#define DMTZ_KEY(X, Y, Z) key(std::integral_constant<int, (X)>{}, std::integral_constant<int, (Y)>{}, std::integral_constant<int, (Z)>{})
    StarWords o;
    o.x = o.y = o.z = o.w = o.w4 = 0;
    const uint64_t kv = k0[0];
    // the vertex: its lowest neighbour, if below it.  The reference starts
    // from DBL_MAX with id -1, so a neighbour of that value is never taken.
    {
        uint64_t bk = DMTZ_KEY_DBL_MAX;
        uint32_t sel = 0;  // direction | family bit << 8 (vertex at the higher-id end) or << 16
        bool below = false;
        DMTZ_FOR(14, R, {
            constexpr int r = decltype(R)::value, d = cxt::dir_by_id(r);
            constexpr int dx = cxt::TOPO_DIRS[d][0], dy = cxt::TOPO_DIRS[d][1], dz = cxt::TOPO_DIRS[d][2];
            constexpr uint32_t c = (uint32_t)d | (1u << ((cxt::dir_from_high(d) ? 8 : 16) + cxt::dir_family(d)));
            static_assert(cxt::dir_up(d) == (r >= 7), "seven neighbours have smaller ids");
            const uint64_t kn = DMTZ_KEY(dx, dy, dz);
            take_lower(bk, sel, kn, c);
            if (r == 6) below = bk <= kv;  // the lowest so far has a smaller id: equal values are below
        });
        below |= bk < kv;
        if (!below) sel = 0;
        o.pv = sel ? (int)(sel & 15u) : 15;
        o.x |= (sel << 16) & 0x7F000000u;
        o.y |= (sel << 8) & 0x7F000000u;
    }
    DMTZ_FOR(7, K, {
        constexpr int k = decltype(K)::value;
        constexpr int p = cxt::TOPO_EDGE_V[k][0], q = cxt::TOPO_EDGE_V[k][1];
        constexpr uint32_t m = cxt::edge_mask(k), m3 = cxt::tet_order_bits(3, k, -1), m4 = cxt::tet_order_bits(4, k, -1);
        const bool below = DMTZ_KEY(cxt::ccx(q), cxt::ccy(q), cxt::ccz(q)) <= DMTZ_KEY(cxt::ccx(p), cxt::ccy(p), cxt::ccz(p));
        if (below) {
            if (cxt::diag(k)) o.y |= m << 12;
            else o.z |= m;
            if (m3) o.w |= m3;
            o.w4 |= m4;
        }
        uint64_t bk = kKeyAbsent;
        uint32_t sel = 0;
        DMTZ_FOR(cxt::TOPO_EDGE_NCOF[k], R, {
            constexpr int i = cxt::edge_cand_by_id(k, decltype(R)::value);
            constexpr int tx = cxt::TOPO_EDGE_THIRD[k][i][0], ty = cxt::TOPO_EDGE_THIRD[k][i][1],
                          tz = cxt::TOPO_EDGE_THIRD[k][i][2];
            constexpr uint32_t c = cxt::edge_bit(k, i);
            const uint64_t kn = DMTZ_KEY(tx, ty, tz);
            take_lower(bk, sel, kn, c);
        });
        if (cxt::diag(k)) o.y |= sel;
        else o.x |= sel;
    });
    o.w |= cxt::face_first();
    DMTZ_FOR(12, S, {
        constexpr int s = decltype(S)::value;
        static_assert(cxt::TOPO_FACE_NCOF[s] == 2, "every triangle slot has two cofaces");
        constexpr int ax = cxt::TOPO_FACE_FOURTH[s][0][0], ay = cxt::TOPO_FACE_FOURTH[s][0][1], az = cxt::TOPO_FACE_FOURTH[s][0][2];
        constexpr int bx = cxt::TOPO_FACE_FOURTH[s][1][0], by = cxt::TOPO_FACE_FOURTH[s][1][1], bz = cxt::TOPO_FACE_FOURTH[s][1][2];
        constexpr bool a_first = cxt::lex3(ax, ay, az) < cxt::lex3(bx, by, bz);
        const uint64_t ka = DMTZ_KEY(ax, ay, az), kb = DMTZ_KEY(bx, by, bz);
        if (a_first ? kb < ka : kb <= ka) o.w ^= cxt::face_bit(s, 0) | cxt::face_bit(s, 1);
    });
#undef DMTZ_KEY
    return o;
}

// ------------------------------------------------------------------- stage 2
// The choice of the triangles and tetrahedra of one anchor:
//   pa: the paired edge of each triangle, A layout; bits 24..30: edges (by
//       family) paired with their vertex; bit 31: the vertex is critical
//   pb: the same, B layout; bits 12..23: triangles paired with an edge; bits
//       24..30 (TRACK): edges (by family) with an end whose descent differs
//   r:  the paired facet of each tetrahedron
// w: words of the plane z (w0) and z + 1 (w1) at the anchor, rows ROW apart.
struct CellWords {
    uint32_t pa, pb, r;
};
template <int ROW, bool TRACK = false>
__host__ __device__ __forceinline__ CellWords grad_stage2(const uint4 *w0, const uint4 *w1, const uint32_t *f0,
                                                          const uint32_t *f1) {
    const uint4 a = w0[0], ax = w0[1], ay = w0[ROW], az = w1[0], ayz = w1[ROW];
    static_assert((cxt::tri_at(false, 0) | cxt::tri_at(false, 1) | cxt::tri_at(false, 2) | cxt::tri_at(false, 4) |
                   cxt::tri_at(false, 6)) == 0xFFFFFFu &&
                      (cxt::tri_at(true, 0) | cxt::tri_at(true, 1) | cxt::tri_at(true, 2) | cxt::tri_at(true, 4)) == 0xFFFu &&
                      (cxt::tet_at(0) | cxt::tet_at(1) | cxt::tet_at(2) | cxt::tet_at(4)) == 0xFFFFFFu,
                  "the gathers below reach every incidence");
    constexpr uint32_t v = 24;
    const uint32_t ga = (a.x & cxt::tri_at(false, 0)) |
                        (ax.x & (cxt::tri_at(false, 1) | cxt::ends_at(1, 1) << v)) |
                        (ay.x & (cxt::tri_at(false, 2) | cxt::ends_at(1, 2) << v)) |
                        (az.x & (cxt::tri_at(false, 4) | cxt::ends_at(1, 4) << v)) |
                        (ayz.x & (cxt::tri_at(false, 6) | cxt::ends_at(1, 6) << v));
    constexpr uint32_t b0 = cxt::tri_at(true, 0), b1 = cxt::tri_at(true, 1), b2 = cxt::tri_at(true, 2), b4 = cxt::tri_at(true, 4);
    const uint32_t gb = (a.y & (b0 | b0 << 12 | cxt::ends_at(0, 0) << v)) |
                        (ax.y & (b1 | b1 << 12 | cxt::ends_at(0, 1) << v)) | (ay.y & (b2 | b2 << 12)) |
                        (az.y & (b4 | b4 << 12));
    const uint32_t go = (a.z & cxt::tri_at(false, 0)) | (ax.z & cxt::tri_at(false, 1)) | (ay.z & cxt::tri_at(false, 2)) |
                        (az.z & cxt::tri_at(false, 4)) | (ayz.z & cxt::tri_at(false, 6));
    const uint32_t gx = (a.w & (cxt::tet_at(0) | cxt::tet_order_bits(3, -1, 0))) |
                        (ax.w & (cxt::tet_at(1) | cxt::tet_order_bits(3, -1, 1))) |
                        (ay.w & (cxt::tet_at(2) | cxt::tet_order_bits(3, -1, 2))) |
                        (az.w & (cxt::tet_at(4) | cxt::tet_order_bits(3, -1, 4)));
    static_assert((cxt::tet_order_bits(3, -1, 0) | cxt::tet_order_bits(3, -1, 1) | cxt::tet_order_bits(3, -1, 2) |
                   cxt::tet_order_bits(3, -1, 4)) == 0x3F000000u,
                  "the (2 3) order bits sit at the same anchors as the facets");
    const uint32_t g4 = (f0[0] & cxt::tet_order_bits(4, -1, 0)) | (f0[1] & cxt::tet_order_bits(4, -1, 1)) |
                        (f0[ROW] & cxt::tet_order_bits(4, -1, 2)) | (f0[ROW + 1] & cxt::tet_order_bits(4, -1, 3)) |
                        (f1[0] & cxt::tet_order_bits(4, -1, 4)) | (f1[1] & cxt::tet_order_bits(4, -1, 5)) |
                        (f1[ROW] & cxt::tet_order_bits(4, -1, 6));
    static_assert((cxt::tet_order_bits(4, -1, 0) | cxt::tet_order_bits(4, -1, 1) | cxt::tet_order_bits(4, -1, 2) |
                   cxt::tet_order_bits(4, -1, 3) | cxt::tet_order_bits(4, -1, 4) | cxt::tet_order_bits(4, -1, 5) |
                   cxt::tet_order_bits(4, -1, 6)) == 0x3FFFFFFFu,
                  "every tetrahedron edge is anchored at one of these corners");
    CellWords o;
    {   // triangles: c_ab = corner b below corner a (labels); the facet opposite the
        // lowest corner if it points, else the one opposite the middle corner
        const uint32_t q0 = ga & 0xFFFu, q1 = (ga >> 12) & 0xFFFu, q2 = gb & 0xFFFu;
        const uint32_t c01 = gb >> 12, c02 = (go >> 12) ^ cxt::tri_flip(0), c12 = go ^ cxt::tri_flip(1);
        const uint32_t lo0 = ~c01 & ~c02, lo1 = c01 & ~c12, lo2 = c02 & c12;
        const uint32_t first = (lo0 & q0) | (lo1 & q1) | (lo2 & q2);
        const uint32_t p0 = q0 & (lo0 | ((c01 ^ c02) & ~first)), p1 = q1 & (lo1 | (~(c01 ^ c12) & ~first)),
                       p2 = q2 & (lo2 | ((c02 ^ c12) & ~first));
        const uint32_t vclaim = ((ga | gb) >> v) & 0x7Fu;
        const uint32_t vcrit = ((a.x | a.y) & 0x7F000000u) ? 0u : 0x80000000u;
        o.pa = p0 | (p1 << 12) | (vclaim << v) | vcrit;
        o.pb = p2 | ((p0 | p1 | p2) << 12);
        if (TRACK) {
            uint32_t d = 0;
            if (a.z >> 24) d |= cxt::edges_at(0);
            if (ax.z >> 24) d |= cxt::edges_at(1);
            if (ay.z >> 24) d |= cxt::edges_at(2);
            if (az.z >> 24) d |= cxt::edges_at(4);
            if (ayz.z >> 24) d |= cxt::edges_at(6);
            o.pb |= d << 24;
        }
    }
    {   // tetrahedra, the same with four corners (labels = id order); garbage above
        // bit 5 of the shifted vectors is masked by s
        const uint32_t s0 = gx & 0x3Fu, s1 = (gx >> 6) & 0x3Fu, s2 = (gx >> 12) & 0x3Fu, s3 = (gx >> 18) & 0x3Fu;
        const uint32_t c01 = g4, c02 = g4 >> 6, c03 = g4 >> 12, c12 = g4 >> 18, c13 = g4 >> 24, c23 = gx >> 24;
        const uint32_t l0 = s0 & ~c01 & ~c02 & ~c03, l1 = s1 & c01 & ~c12 & ~c13, l2 = s2 & c02 & c12 & ~c23,
                       l3 = s3 & c03 & c13 & c23;
        const uint32_t free = ~(l0 | l1 | l2 | l3);
        // exactly two of the other three corners above: above0 = ~c01, ~c02, ~c03 and so on
        auto two = [](uint32_t x, uint32_t y, uint32_t z) { return (x & y & ~z) | (x & ~y & z) | (~x & y & z); };
        const uint32_t r0 = l0 | (s0 & free & two(~c01, ~c02, ~c03)), r1 = l1 | (s1 & free & two(c01, ~c12, ~c13)),
                       r2 = l2 | (s2 & free & two(c02, c12, ~c23)), r3 = l3 | (s3 & free & two(c03, c13, c23));
        o.r = r0 | (r1 << 6) | (r2 << 12) | (r3 << 18);
    }
    return o;
}

// six bits to stride 3
__host__ __device__ __forceinline__ uint32_t spread3(uint32_t b) {
    const uint32_t g = (b & 7u) | ((b & 0x38u) << 6);
    return (g | (g << 2) | (g << 4)) & 0x9249u;
}
// ------------------------------------------------------------------- stage 3
// Outputs of one anchor (FieldState's eup, fup, crit, tcode).  c0: the cell words of the anchor's plane at the anchor,
// cm: of the plane below; rows ROW apart.  last: bit per axis, the anchor is on
// the grid's last layer (its cells over that face do not exist).
struct AnchorOut {
    uint32_t eup, fup, crit, tcode;
};
template <int ROW>
__host__ __device__ __forceinline__ AnchorOut grad_stage3(const CellWords *cm, const CellWords *c0, uint32_t last) {
    const CellWords a = c0[0], bx = c0[-1], by = c0[-ROW], bz = cm[0], byz = cm[-ROW];
    uint32_t exE = 0x7Fu, exF = 0xFFFu, exT = 0x3Fu;
    if (last) {
        if (last & 1u) { exE &= ~cxt::edges_over(0); exF &= ~cxt::faces_over(0); }
        if (last & 2u) { exE &= ~cxt::edges_over(1); exF &= ~cxt::faces_over(1); }
        if (last & 4u) { exE &= ~cxt::edges_over(2); exF &= ~cxt::faces_over(2); }
        exT = 0;
    }
    const uint32_t ea = (a.pa & cxt::tri_at(false, 0)) | (bx.pa & cxt::tri_at(false, 1)) | (by.pa & cxt::tri_at(false, 2)) |
                        (bz.pa & cxt::tri_at(false, 4)) | (byz.pa & cxt::tri_at(false, 6));
    const uint32_t eb = (a.pb & cxt::tri_at(true, 0)) | (bx.pb & cxt::tri_at(true, 1)) | (by.pb & cxt::tri_at(true, 2)) |
                        (bz.pb & cxt::tri_at(true, 4));
    const uint32_t fr = (a.r & cxt::tet_at(0)) | (bx.r & cxt::tet_at(1)) | (by.r & cxt::tet_at(2)) | (bz.r & cxt::tet_at(4));
    AnchorOut o;
    uint32_t eup = 0;
    DMTZ_FOR(7, K, {
        constexpr int k = decltype(K)::value;
        const uint32_t e = cxt::diag(k) ? eb : ea;
        constexpr uint32_t m0 = cxt::edge_code_mask(k, 0), m1 = cxt::edge_code_mask(k, 1), m2 = cxt::edge_code_mask(k, 2);
        if (e & m0) eup |= 1u << (3 * k);
        if (e & m1) eup |= 2u << (3 * k);
        if (e & m2) eup |= 4u << (3 * k);
    });
    uint32_t fup = 0;
    DMTZ_FOR(47, I, {  // a triangle's code is one-hot, like its incidences: a bit permutation
        constexpr int d = decltype(I)::value - 23;
        constexpr uint32_t m = cxt::face_move(d);
        if (m) fup |= d >= 0 ? (fr & m) << (d >= 0 ? d : 0) : (fr & m) >> (d < 0 ? -d : 0);
    });
    // one bit per coded edge (stride 3) and triangle (stride 2), packed
    uint32_t upE = (eup | (eup >> 1) | (eup >> 2)) & 0x49249u;
    upE = (upE | (upE >> 2)) & 0x430C3u;
    upE = (upE | (upE >> 4)) & 0x700Fu;
    upE = (upE | (upE >> 8)) & 0x7Fu;
    uint32_t upF = (fup | (fup >> 1)) & 0x555555u;
    upF = (upF | (upF >> 1)) & 0x333333u;
    upF = (upF | (upF >> 2)) & 0x0F0F0Fu;
    upF = ((upF | (upF >> 4)) & 0xFFu) | ((upF >> 8) & 0xF00u);
    if (last) {  // codes of cells that do not exist
        DMTZ_FOR(7, K, {
            constexpr int k = decltype(K)::value;
            if (!((exE >> k) & 1u)) eup &= ~(7u << (3 * k));
        });
        DMTZ_FOR(12, S, {
            constexpr int s = decltype(S)::value;
            if (!((exF >> s) & 1u)) fup &= ~(3u << (2 * s));
        });
    }
    o.eup = eup;
    o.fup = fup;
    const uint32_t r0 = a.r & 0x3Fu, r1 = (a.r >> 6) & 0x3Fu, r2 = (a.r >> 12) & 0x3Fu, r3 = (a.r >> 18) & 0x3Fu;
    const uint32_t none = (~(r0 | r1 | r2 | r3) & 0x3Fu) | (~exT & 0x3Fu);
    o.crit = (a.pa >> 31) | ((exE & ~(upE | (a.pa >> 24))) << 1) | ((exF & ~(upF | (a.pb >> 12))) << 8) |
             ((none & exT) << 20);
    // facet index of each tetrahedron, 7 = unpaired or absent
    o.tcode = spread3(r1 | r3 | none) | (spread3(r2 | r3 | none) << 1) | (spread3(none) << 2);
    return o;
}

// ---------------------------------------------------------------------------
// Bricks.  Anchors are grouped in bricks of 128 (shape chosen by the autotuner,
// 8 x 4 x 4 by default).  A repair runs over an explicit list of bricks
// (packed bx | by << 11 | bz << 22); with list == nullptr the list is every
// brick of the grid.  Blocks stride over the list, so the grid size does not
// depend on its length and the length can stay on the device.
// ---------------------------------------------------------------------------
#define DMTZ_BRICK 128
struct BrickList {
    const uint32_t *list;           // packed brick coordinates, or nullptr for all bricks
    const unsigned long long *n;    // number of listed bricks (device), when list != nullptr
    int nbx, nby, nbz;              // bricks per axis
    int shape;                      // brick shape index (DMTZ_SHAPES)
    FDiv dbx, dby;                  // division by nbx and nby (brick index -> coordinates)
};
// brick shapes (anchors per brick along x, y, z)
#define DMTZ_NSHAPES 3
static const int DMTZ_SHAPES[DMTZ_NSHAPES][3] = {{8, 4, 4}, {16, 4, 2}, {32, 2, 2}};

__device__ __forceinline__ i64 brick_count(const BrickList &bl) {
    return bl.list ? (i64)*bl.n : (i64)bl.nbx * bl.nby * bl.nbz;
}
__device__ __forceinline__ void brick_coords(const BrickList &bl, i64 b, int &bx, int &by, int &bz) {
    if (bl.list) {
        const uint32_t e = bl.list[b];
        bx = e & 0x7FF;
        by = (e >> 11) & 0x7FF;
        bz = e >> 22;
    } else {  // every thread of the block decodes the same index: multiply-high, not division
        const unsigned long long u = (unsigned long long)b, q = fdiv(bl.dbx, u), r = fdiv(bl.dby, q);
        bx = (int)(u - q * (unsigned long long)bl.nbx);
        by = (int)(q - r * (unsigned long long)bl.nby);
        bz = (int)r;
    }
}

// ---------------------------------------------------------------------------
// Cell codes: anchor vertex * 32 + the cell's bit of FieldState::crit (0 the
// vertex, 1..7 edges, 8..19 triangles, 20..25 tetrahedra).
__host__ __device__ __forceinline__ i64 cell_code(i64 anchor, int bit) { return anchor * 32 + bit; }

// The lists of mismatched cells (criticality differs between the two
// gradients), by kind: min, 1-saddle, 2-saddle, max.
struct Lists {
    i64 *l[4];                  // cell codes
    unsigned long long *n;      // 4 counters
    i64 cap[4];                 // capacities; a counter above its capacity = overflow,
                                // the host grows the list and scans again
};
// every lane of a warp appends the mismatched cells d (bits of
// FieldState::crit) of its anchor v, with one atomic per kind and warp
__device__ __forceinline__ void push_warp(const Lists &L, i64 v, uint32_t d) {
    const unsigned full = 0xffffffffu, lane = threadIdx.x & 31u;
    if (!__any_sync(full, d != 0)) return;
    const unsigned long long mine = (unsigned long long)(d & 1u) | ((unsigned long long)__popc(d & 0xFEu) << 16) |
                                    ((unsigned long long)__popc(d & 0xFFF00u) << 32) |
                                    ((unsigned long long)__popc(d & 0x3F00000u) << 48);
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(full, incl, o);
        if (lane >= (unsigned)o) incl += y;
    }
    const unsigned long long total = __shfl_sync(full, incl, 31);
    const unsigned cnt = lane < 4 ? (unsigned)(total >> (16 * lane)) & 0xFFFFu : 0u;
    unsigned long long base = 0;
    if (cnt) base = atomicAdd(&L.n[lane], (unsigned long long)cnt);
    const unsigned long long excl = incl - mine;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        unsigned long long at = __shfl_sync(full, base, k) + ((excl >> (16 * k)) & 0xFFFFull);
        const uint32_t kind = k == 0 ? 1u : k == 1 ? 0xFEu : k == 2 ? 0xFFF00u : 0x3F00000u;
        for (uint32_t m = d & kind; m; m &= m - 1, at++)
            if ((i64)at < L.cap[k]) L.l[k][at] = cell_code(v, __ffs(m) - 1);
    }
}

// Separatrix flags of the bricks (see k_path_detect), refreshed with a brick's gradient.
struct PathFlags {
    uint8_t *as, *ds;            // per brick; nullptr: not kept
    const uint32_t *tcP;         // original tetrahedron codes with path bits (18 + slot)
    const uint8_t *pvP;          // original steepest descent
};
// What a gradient kernel does with its anchors besides storing their state
struct GradOps {
    PathFlags F;
    Lists T;               // receives the anchors' mismatched cells
    const uint32_t *critP; // original criticality; nullptr: no flags, no lists
    uint32_t want;         // cell bits the lists take (0: no lists)
};
// does a tetrahedron on an original path pair differently?
__host__ __device__ __forceinline__ bool tet_path_differs(uint32_t tcP, uint32_t tcQ) {
    const uint32_t x = tcP ^ tcQ, on = tcP >> 18;
    return on && ((x | (x >> 1) | (x >> 2)) & 0x9249u & spread3(on));
}

// Incremental mismatch lists.  A cell's mismatch status changes only where its
// anchor's criticality is recomputed, i.e. in the repair's bricks (marked
// fresh).  The new lists are the old entries outside fresh bricks, appended by
// some extra blocks of the repair, plus what the repair itself finds.  Valid when every scan of
// the run uses the same saddle flag and the old lists were complete (an
// overflow is followed by a full scan before the next round).
struct KeepOps {
    Lists L;               // the old lists
    const uint8_t *fresh;  // per brick
    int shx, shy, shz, nbx, nby;
    unsigned blocks;       // extra blocks; 0: nothing to carry over
};
__device__ __forceinline__ void keep_lists(const Grid &g, const GradOps &O, const KeepOps &K, unsigned block) {
    const bool sad = (O.want & 0xFFFFEu) != 0;  // the run's lists hold saddles
    const i64 n0 = min((i64)K.L.n[0], K.L.cap[0]), n1 = sad ? min((i64)K.L.n[1], K.L.cap[1]) : 0,
              n2 = sad ? min((i64)K.L.n[2], K.L.cap[2]) : 0, n3 = min((i64)K.L.n[3], K.L.cap[3]);
    for (i64 i = (i64)block * blockDim.x + threadIdx.x; i < n0 + n1 + n2 + n3; i += (i64)K.blocks * blockDim.x) {
        const int k = i < n0 ? 0 : i < n0 + n1 ? 1 : i < n0 + n1 + n2 ? 2 : 3;
        const i64 code = K.L.l[k][i - (k > 0 ? n0 : 0) - (k > 1 ? n1 : 0) - (k > 2 ? n2 : 0)];
        int x, y, z;
        decode_v(g, code >> 5, x, y, z);
        if (K.fresh[(x >> K.shx) + (i64)K.nbx * ((y >> K.shy) + (i64)K.nby * (z >> K.shz))]) continue;
        const unsigned long long at = agg_slot(&O.T.n[k]);
        if ((i64)at < O.T.cap[k]) O.T.l[k][at] = code;
    }
}

// The gradient of the listed bricks, one block per brick step.  One thread per
// stage-1 anchor (the brick and one layer around it: 360 of 384 threads for
// 8 x 4 x 4), so each stage is one round; in the later stages the surplus
// warps have nothing to issue.
template <int SX, int SY, int SZ>
__host__ __device__ constexpr int brick_threads() {
    return ((SX + 2) * (SY + 2) * (SZ + 2) + 31) / 32 * 32;
}
template <int SX, int SY, int SZ>
struct BrickMem {
    static constexpr int KX = SX + 4, KY = SY + 4, KZ = SZ + 4, NK = KX * KY * KZ;  // keys: two layers around
    static constexpr int WX = SX + 2, WY = SY + 2, WZ = SZ + 2, NW = WX * WY * WZ;  // star words: one layer around
    static constexpr int CX = SX + 1, CY = SY + 1, CZ = SZ + 1, NC = CX * CY * CZ;  // cell words: one layer below
    uint64_t sk[NK];
    uint4 sw[NW];
    uint32_t sf[NW];
    CellWords sc[NC];
    uint32_t flag;  // bit 0: as, bit 1: ds
};
// one brick, by a block of brick_threads
template <int SX, int SY, int SZ>
__device__ __forceinline__ void grad_brick(const Grid &g, const FieldState &s, const BrickList &bl, const GradOps &O, i64 b,
                                           BrickMem<SX, SY, SZ> &M) {
    static_assert(SX * SY * SZ == DMTZ_BRICK, "a brick is 128 anchors");
    using B = BrickMem<SX, SY, SZ>;
    constexpr int NT = brick_threads<SX, SY, SZ>();
    constexpr int KX = B::KX, KY = B::KY, NK = B::NK, WX = B::WX, WY = B::WY, NW = B::NW, CX = B::CX, CY = B::CY, NC = B::NC;
    const int t = threadIdx.x;
    const int wx = t % WX, wy = (t / WX) % WY, wz = t / (WX * WY);
    const int cx = t % CX, cy = (t / CX) % CY, cz = t / (CX * CY);
    const int ox = t % SX, oy = (t / SX) % SY, oz = t / (SX * SY);
    int bx, by, bz;
    brick_coords(bl, b, bx, by, bz);
    const int x0 = bx * SX, y0 = by * SY, z0 = bz * SZ;
    for (int e = t; e < NK; e += NT) {
        const int ux = x0 - 2 + e % KX, uy = y0 - 2 + (e / KX) % KY, uz = z0 - 2 + e / (KX * KY);
        const bool in = ux >= 0 && uy >= 0 && uz >= 0 && ux < g.W && uy < g.H && uz < g.D;
        M.sk[e] = in ? okey(s.val[ux + (i64)uy * g.W + (i64)uz * g.WH]) : kKeyAbsent;
    }
    // what the flags and lists compare with, loaded with the keys
    uint32_t tcP = 0, critP = 0;
    int pvP = 15;
    if (O.critP) {
        const int x = x0 + wx - 1, y = y0 + wy - 1, z = z0 + wz - 1;
        if (O.F.as && t < NW && x >= 0 && y >= 0 && z >= 0 && x < g.W && y < g.H && z < g.D)
            pvP = O.F.pvP[x + (i64)y * g.W + (i64)z * g.WH];
        if (t < DMTZ_BRICK && x0 + ox < g.W && y0 + oy < g.H && z0 + oz < g.D) {
            const i64 v = (x0 + ox) + (i64)(y0 + oy) * g.W + (i64)(z0 + oz) * g.WH;
            if (O.F.as) tcP = O.F.tcP[v];
            critP = O.critP[v];
        }
    }
    __syncthreads();
    if (t < NW) {
        const uint64_t *k0 = M.sk + (wx + 1) + KX * ((wy + 1) + KY * (wz + 1));
        const StarWords w = grad_stage1<KX>(k0 - KX * KY, k0, k0 + KX * KY);
        M.sw[t] = make_uint4(w.x, w.y, w.z | (pvP != 15 && pvP != w.pv ? 1u << 24 : 0u), w.w);
        M.sf[t] = w.w4;
        const int x = x0 + wx - 1, y = y0 + wy - 1, z = z0 + wz - 1;
        if (wx >= 1 && wy >= 1 && wz >= 1 && wx <= SX && wy <= SY && wz <= SZ && x < g.W && y < g.H && z < g.D)
            s.pv[x + (i64)y * g.W + (i64)z * g.WH] = (uint8_t)w.pv;
    }
    __syncthreads();
    if (t < NC) {
        if (t == 0) M.flag = 0;
        const int i = cx + WX * (cy + WY * cz);
        M.sc[t] = grad_stage2<WX, true>(M.sw + i, M.sw + i + WX * WY, M.sf + i, M.sf + i + WX * WY);
    }
    __syncthreads();
    if (t < DMTZ_BRICK) {
        const int x = x0 + ox, y = y0 + oy, z = z0 + oz;
        const i64 v = x + (i64)y * g.W + (i64)z * g.WH;
        uint32_t differ = 0;
        if (x < g.W && y < g.H && z < g.D) {
            const int i = (ox + 1) + CX * ((oy + 1) + CY * (oz + 1));
            const uint32_t last = (x == g.W - 1 ? 1u : 0u) | (y == g.H - 1 ? 2u : 0u) | (z == g.D - 1 ? 4u : 0u);
            const AnchorOut o = grad_stage3<CX>(M.sc + i - CX * CY, M.sc + i, last);
            s.eup[v] = o.eup;
            s.fup[v] = o.fup;
            if (s.crit) s.crit[v] = o.crit;
            if (s.tcode) s.tcode[v] = o.tcode;
            differ = (o.crit ^ critP) & O.want;
            const uint32_t f = (tet_path_differs(tcP, o.tcode) ? 1u : 0u) | (((critP >> 1) & (M.sc[i].pb >> 24) & 0x7Fu) ? 2u : 0u);
            if (f) atomicOr(&M.flag, f);
        }
        if (O.want) push_warp(O.T, v, differ);
    }
    if (O.F.as) {
        __syncthreads();
        if (t == 0) {
            const i64 b = bx + (i64)bl.nbx * (by + (i64)bl.nby * bz);
            O.F.as[b] = (uint8_t)(M.flag & 1u);
            O.F.ds[b] = (uint8_t)(M.flag >> 1);
        }
    }
}
template <int SX, int SY, int SZ>
__global__ void __launch_bounds__((brick_threads<SX, SY, SZ>()), SX == 8 ? 3 : 2) k_grad_bricks(Grid g, FieldState s, BrickList bl,
                                                                                        const __grid_constant__ GradOps O,
                                                                                        const __grid_constant__ KeepOps K,
                                                                                        const int *wanted) {
    __shared__ BrickMem<SX, SY, SZ> M;
    let_next();
    after_previous();
    if (wanted && !*wanted) return;
    if (blockIdx.x >= gridDim.x - K.blocks) {  // the blocks that carry the old lists over
        keep_lists(g, O, K, blockIdx.x - (gridDim.x - K.blocks));
        return;
    }
    const unsigned n = (unsigned)brick_count(bl);  // (their coordinates fill 32 bits)
    for (unsigned b = blockIdx.x; b < n; b += gridDim.x - K.blocks) {
        grad_brick<SX, SY, SZ>(g, s, bl, O, b, M);
        // the next brick's keys may land now: stage 1 of this one is behind two
        // barriers, and the words stage 3 reads are not written before the next one
    }
}

// The gradient of the whole grid.  A block takes TX x TY columns and marches
// along z over `chunk` planes, so only the x and y halos are recomputed (stage
// 1 runs on (TX+2)(TY+2) of TX TY columns instead of 2.8 times the anchors as
// in bricks of 8 x 4 x 4).  The stages run one behind the other on different
// planes of ring buffers, with one barrier per plane: at step p stage 1 takes plane
// p, stage 2 plane p - 2, stage 3 plane p - 3, and the keys of plane p + 2 arrive.
template <int TX, int TY>
struct March {
    static constexpr int KX = TX + 4, NK = KX * (TY + 4);
    static constexpr int WX = TX + 2, NW = WX * (TY + 2);
    static constexpr int CX = TX + 1, NC = CX * (TY + 1);
    static constexpr int NT = (NW + 31) / 32 * 32;
    static constexpr int NL = (NK + NT - 1) / NT;  // keys a thread loads per plane
    static constexpr size_t smem = 4 * NK * sizeof(uint64_t) + 3 * NW * (sizeof(uint4) + sizeof(uint32_t)) +
                                   3 * NC * sizeof(CellWords);
};
// TRACK: flags and lists as GradOps says (brick flags zero at launch).
template <int TX, int TY, int MINB, bool TRACK>
__global__ void __launch_bounds__((March<TX, TY>::NT), MINB) k_grad_march(Grid g, FieldState s, int ntx, int nty, int chunk,
                                                                          const __grid_constant__ GradOps O, int shx, int shy, int shz, int nbx,
                                                                          int nby) {
    using M = March<TX, TY>;
    constexpr int KX = M::KX, NK = M::NK, WX = M::WX, NW = M::NW, CX = M::CX, NC = M::NC, NT = M::NT, NL = M::NL;
    extern __shared__ __align__(16) unsigned char march_smem[];
    uint4 *sw = reinterpret_cast<uint4 *>(march_smem);                 // [3][NW]
    uint64_t *sk = reinterpret_cast<uint64_t *>(sw + 3 * NW);          // [4][NK]
    uint32_t *sf = reinterpret_cast<uint32_t *>(sk + 4 * NK);          // [3][NW]
    CellWords *sc = reinterpret_cast<CellWords *>(sf + 3 * NW);        // [3][NC]
    const int t = threadIdx.x;
    const int x0 = (int)(blockIdx.x % (unsigned)ntx) * TX, y0 = (int)((blockIdx.x / (unsigned)ntx) % (unsigned)nty) * TY;
    const int z0 = (int)(blockIdx.x / ((unsigned)ntx * (unsigned)nty)) * chunk, z1 = min(z0 + chunk, g.D);
    // the columns whose keys this thread loads
    i64 col[NL];
    bool in[NL];
#pragma unroll
    for (int l = 0; l < NL; l++) {
        const int e = t + l * NT, ux = x0 - 2 + e % KX, uy = y0 - 2 + e / KX;
        in[l] = e < NK && ux >= 0 && uy >= 0 && ux < g.W && uy < g.H;
        col[l] = in[l] ? ux + (i64)uy * g.W : 0;
    }
    auto load_key = [&](int l, int z) -> uint64_t {
        return (in[l] && z >= 0 && z < g.D) ? okey(s.val[col[l] + (i64)z * g.WH]) : kKeyAbsent;
    };
#pragma unroll
    for (int q = 0; q < 3; q++)  // planes z0 - 2, z0 - 1, z0 in slots 0, 1, 2
#pragma unroll
        for (int l = 0; l < NL; l++)
            if (t + l * NT < NK) sk[q * NK + t + l * NT] = load_key(l, z0 - 2 + q);
    // stage 1: this thread's anchor column; its vertex is written if inside the tile
    const int wx = t % WX, wy = t / WX, ki = (wx + 1) + KX * (wy + 1);
    const bool pv_in = t < NW && wx >= 1 && wy >= 1 && wx <= TX && wy <= TY && x0 + wx - 1 < g.W && y0 + wy - 1 < g.H;
    const i64 pv_col = (x0 + wx - 1) + (i64)(y0 + wy - 1) * g.W;
    const bool st1_in = t < NW && x0 + wx >= 1 && y0 + wy >= 1 && x0 + wx - 1 < g.W && y0 + wy - 1 < g.H;
    // stage 2 and stage 3 columns
    const int wi = t % CX + WX * (t / CX);
    const int ox = t % TX, oy = t / TX, x = x0 + ox, y = y0 + oy, ci = (ox + 1) + CX * (oy + 1);
    const bool out_in = t < TX * TY && x < g.W && y < g.H;
    const i64 out_col = x + (i64)y * g.W;
    const uint32_t last_xy = (x == g.W - 1 ? 1u : 0u) | (y == g.H - 1 ? 2u : 0u);
    __syncthreads();
    int s4 = 2, s3 = 0;  // ring slots: keys of plane p + 1 in slot s4 (mod 4), words of plane p in slot s3 (mod 3)
    for (int p = z0 - 1; p <= z1 + 2; p++) {
        uint64_t nk[NL];
#pragma unroll
        for (int l = 0; l < NL; l++) nk[l] = p < z1 ? load_key(l, p + 2) : kKeyAbsent;
        // what the flags and lists compare with
        const i64 v3 = out_col + (i64)(p - 3) * g.WH;
        int pvP = 15;
        uint32_t tcP = 0, critP = 0;
        if (TRACK) {
            if (O.F.as && st1_in && p >= 0 && p < g.D) pvP = O.F.pvP[pv_col + (i64)p * g.WH];
            if (p - 3 >= z0 && out_in) {
                if (O.F.as) tcP = O.F.tcP[v3];
                critP = O.critP[v3];
            }
        }
        const int s3m1 = s3 == 0 ? 2 : s3 - 1, s3m2 = s3m1 == 0 ? 2 : s3m1 - 1;  // slots of planes p - 1, p - 2
        if (p <= z1 && t < NW) {
            const StarWords w = grad_stage1<KX>(sk + ((s4 + 2) & 3) * NK + ki, sk + ((s4 + 3) & 3) * NK + ki, sk + s4 * NK + ki);
            sw[s3 * NW + t] = make_uint4(w.x, w.y, w.z | (TRACK && pvP != 15 && pvP != w.pv ? 1u << 24 : 0u), w.w);
            sf[s3 * NW + t] = w.w4;
            if (pv_in && p >= z0 && p < z1) s.pv[pv_col + (i64)p * g.WH] = (uint8_t)w.pv;
        }
        // cell words of plane q live in the slot star words of plane q had
        if (p - 2 >= z0 - 1 && p - 2 < z1 && t < NC)
            sc[s3m2 * NC + t] = grad_stage2<WX, TRACK>(sw + s3m2 * NW + wi, sw + s3m1 * NW + wi, sf + s3m2 * NW + wi, sf + s3m1 * NW + wi);
        if (p - 3 >= z0 && t < TX * TY) {  // plane p - 3 in slot s3, plane p - 4 in slot s3m1
            const int z = p - 3;
            uint32_t differ = 0;
            if (out_in) {
                const CellWords *c0 = sc + s3 * NC + ci;
                const AnchorOut o = grad_stage3<CX>(sc + s3m1 * NC + ci, c0, last_xy | (z == g.D - 1 ? 4u : 0u));
                s.eup[v3] = o.eup;
                s.fup[v3] = o.fup;
                if (s.crit) s.crit[v3] = o.crit;
                if (s.tcode) s.tcode[v3] = o.tcode;
                if (TRACK) {
                    differ = (o.crit ^ critP) & O.want;
                    const bool as = tet_path_differs(tcP, o.tcode), ds = ((critP >> 1) & (c0->pb >> 24) & 0x7Fu) != 0;
                    if (O.F.as && (as || ds)) {
                        const i64 b = (x >> shx) + (i64)nbx * ((y >> shy) + (i64)nby * (z >> shz));
                        if (as) O.F.as[b] = 1;
                        if (ds) O.F.ds[b] = 1;
                    }
                }
            }
            if (TRACK && O.want) push_warp(O.T, v3, differ);
        }
        s4 = (s4 + 1) & 3;
#pragma unroll
        for (int l = 0; l < NL; l++)
            if (t + l * NT < NK) sk[s4 * NK + t + l * NT] = nk[l];
        s3 = s3 == 2 ? 0 : s3 + 1;
        __syncthreads();
    }
}

}  // namespace dmtz
