// cnn.cu — the learned proposal: a 4-layer 3x3x3 convolutional network with
// BF16 weights/activations and FP32 accumulation on the tensor cores, its
// backward pass, and the loss / optimiser kernels.  No counterpart in the
// reference; it only produces a starting point for the exact correction loop.
//
// Layout: activations channels-last bf16, [vertex][channel], vertex =
// x + W*(y + H*z).  Layers (in -> out channels): 16 -> 32 -> 32 -> 32 -> 16,
// ReLU after the first three; only output channel 0 is used (the other 15
// have zero weights and zero gradients, so they stay zero).  Parameters (f32
// master copy), per layer: weights [27 taps][out][in], then bias [out];
// tap = (dz+1)*9 + (dy+1)*3 + (dx+1).
//
// Kernels (all persistent: one or two blocks per SM loop over tiles):
//   k_conv_tcx  the convolutions (forward and data gradient) on tcgen05: the
//            128 rows of a product are a plane across x, which marches (the
//            default path; see its comment).
//   k_conv_out  the last layer, of which one channel is needed.
//   k_conv_tc  all layers with a box of vertices per MMA chain (tensor path 1;
//            slower than the default at every size, there to compare with).
//   k_conv   the same convolution on mma.sync.m16n8k16 (bf16 in, f32
//            accumulate; tensor path 0, as k_conv_tc).  A block keeps all 27 x out x in weights in shared
//            memory and streams 8x8x4-vertex tiles (+1 halo) through a
//            cp.async double buffer; operands reach registers by ldmatrix.
//            The data gradient is the same kernel with transposed weights,
//            mirrored taps and a ReLU-derivative epilogue.
//   k_wgrad_tc  weight + bias gradient on tcgen05 (the default; see its comment).
//   k_wgrad  the same on mma.sync: per tile, all 27 taps x out x in
//            products reduced over the tile's 256 vertices on the same MMA
//            (operands by ldmatrix.trans from the channels-last tiles);
//            per-block partial sums, then a fixed-order reduction
//            (deterministic).
//   k_loss, k_reduce, k_adam, k_pack: loss, gradient scaling,
//            Adam, bf16 weight refresh.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "cnn.cuh"

typedef __nv_bfloat16 bf16;
typedef long long i64;

namespace {

constexpr int TX = 8, TY = 8, TZ = 4, TV = TX * TY * TZ;  // output tile (256 vertices)
constexpr int HX = TX + 2, HY = TY + 2, HZ = TZ + 2, HALO = HX * HY * HZ;
constexpr int NLAYER = 4;
constexpr int LCIN[NLAYER] = {16, 32, 32, 32};
constexpr int LCOUT[NLAYER] = {32, 32, 32, 16};

constexpr i64 layer_params(int l) { return 27LL * LCOUT[l] * LCIN[l] + LCOUT[l]; }
constexpr i64 layer_offset(int l) { return l == 0 ? 0 : layer_offset(l - 1) + layer_params(l - 1); }
constexpr i64 kParams = layer_offset(NLAYER);

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// 16-byte async copy global -> shared; src_bytes = 0 writes zeros (the source
// address is not read then, but is kept valid anyway)
__device__ __forceinline__ void cp16(void *dst, const void *src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(dst)), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ void ldm4(uint32_t r[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t r[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct Dims {
    int W, H, D, ntx, nty, ntz;
    i64 ntiles;
};
inline Dims make_dims(int W, int H, int D) {
    Dims d{W, H, D, (W + TX - 1) / TX, (H + TY - 1) / TY, (D + TZ - 1) / TZ, 0};
    d.ntiles = (i64)d.ntx * d.nty * d.ntz;
    return d;
}

// Box of EX x EY x EZ vertices starting at (x0, y0, z0) (may stick out of the
// grid: zeros there) of a channels-last tensor with C channels, into shared
// rows of CP = C + 8 bf16 (the 16-byte pad makes ldmatrix conflict-free).
template <int C, int EX, int EY, int EZ>
__device__ __forceinline__ void load_box(bf16 *dst, const bf16 *__restrict__ src, const Dims &d, int x0, int y0,
                                         int z0) {
    constexpr int CP = C + 8, PIECES = C / 8;
    for (int i = threadIdx.x; i < EX * EY * EZ * PIECES; i += blockDim.x) {
        const int row = i / PIECES, piece = i - row * PIECES;
        const int hx = row % EX, hy = (row / EX) % EY, hz = row / (EX * EY);
        const int gx = x0 + hx, gy = y0 + hy, gz = z0 + hz;
        const bool in = gx >= 0 && gx < d.W && gy >= 0 && gy < d.H && gz >= 0 && gz < d.D;
        const bf16 *s = in ? src + ((i64)gx + (i64)gy * d.W + (i64)gz * d.W * d.H) * C + piece * 8 : src;
        cp16(dst + row * CP + piece * 8, s, in ? 16 : 0);
    }
}

__device__ __forceinline__ void tile_origin(const Dims &d, i64 tile, int &x0, int &y0, int &z0) {
    x0 = (int)(tile % d.ntx) * TX;
    y0 = (int)((tile / d.ntx) % d.nty) * TY;
    z0 = (int)(tile / ((i64)d.ntx * d.nty)) * TZ;
}

}  // namespace

namespace {

// ---------------------------------------------------------------- convolution
// out[v][n] = sum_tap sum_c W[tap][n][c] * in[v + off(tap)][c]   (FLIP: v - off)
// MODE 0: + bias, ReLU, bf16 out.  MODE 1: + bias, channel 0 as f32 (the
// proposal).  MODE 2 (data gradient): no bias; zero where aux, the stored
// activation that fed the layer, is not positive (ReLU derivative).
// 8 warps; warp w owns tile vertices 32w..32w+31 (two m16 tiles), all COUT.
template <int CIN, int COUT, int MODE, bool FLIP>
__global__ void __launch_bounds__(256, 1) k_conv(Dims d, const bf16 *__restrict__ in, const bf16 *__restrict__ wt,
                                              const float *__restrict__ bias, void *out,
                                              const bf16 *__restrict__ aux) {
    constexpr int CP = CIN + 8, NT = COUT / 8, KC = CIN / 16;
    static_assert(NT % 2 == 0 && CIN % 16 == 0, "tile shapes");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16 *ws = reinterpret_cast<bf16 *>(smem_raw);  // [27*COUT][CP]
    bf16 *xs0 = ws + 27 * COUT * CP;                 // 2 x [HALO][CP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    for (int i = tid; i < 27 * COUT * (CIN / 8); i += blockDim.x) {
        const int row = i / (CIN / 8), piece = i - row * (CIN / 8);
        cp16(ws + row * CP + piece * 8, wt + (i64)row * CIN + piece * 8, 16);
    }
    // ldmatrix roles.  A (vertices x channels): lane supplies row
    // (lane&7) + 8*((lane>>3)&1) of the m-tile, channel half 8*(lane>>4).
    // B (weights, rows = output channel): n = 8*(lane>>4) + (lane&7) within a
    // pair of n-tiles, channel half 8*((lane>>3)&1).
    int hbase[2];
#pragma unroll
    for (int m = 0; m < 2; m++) {
        const int li = warp * 32 + m * 16 + (lane & 7) + 8 * ((lane >> 3) & 1);
        hbase[m] = (((li >> 6) + 1) * HY + ((li >> 3) & 7) + 1) * HX + (li & 7) + 1;
    }
    const int akofs = 8 * (lane >> 4);
    const int bn = 8 * (lane >> 4) + (lane & 7), bkofs = 8 * ((lane >> 3) & 1);

    i64 tile = blockIdx.x;
    int buf = 0;
    if (tile < d.ntiles) {
        int x0, y0, z0;
        tile_origin(d, tile, x0, y0, z0);
        load_box<CIN, HX, HY, HZ>(xs0, in, d, x0 - 1, y0 - 1, z0 - 1);
    }
    cp_commit();
    for (; tile < d.ntiles; tile += gridDim.x, buf ^= 1) {
        const i64 next = tile + gridDim.x;
        if (next < d.ntiles) {
            int x0, y0, z0;
            tile_origin(d, next, x0, y0, z0);
            load_box<CIN, HX, HY, HZ>(xs0 + (buf ^ 1) * HALO * CP, in, d, x0 - 1, y0 - 1, z0 - 1);
        }
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        const bf16 *xs = xs0 + buf * HALO * CP;
        float acc[2][NT][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[m][n][k] = 0.f;
#pragma unroll 1
        for (int tap = 0; tap < 27; tap++) {
            const int dx = tap % 3 - 1, dy = (tap / 3) % 3 - 1, dzz = tap / 9 - 1;
            const int toff = FLIP ? -((dzz * HY + dy) * HX + dx) : (dzz * HY + dy) * HX + dx;
            const bf16 *wtap = ws + tap * COUT * CP;
#pragma unroll
            for (int kc = 0; kc < KC; kc++) {
                uint32_t a0[4], a1[4];
                ldm4(a0, xs + (hbase[0] + toff) * CP + kc * 16 + akofs);
                ldm4(a1, xs + (hbase[1] + toff) * CP + kc * 16 + akofs);
#pragma unroll
                for (int j = 0; j < NT; j += 2) {
                    uint32_t b[4];
                    ldm4(b, wtap + (j * 8 + bn) * CP + kc * 16 + bkofs);
                    mma16816(acc[0][j], a0, b[0], b[1]);
                    mma16816(acc[1][j], a1, b[0], b[1]);
                    mma16816(acc[0][j + 1], a0, b[2], b[3]);
                    mma16816(acc[1][j + 1], a1, b[2], b[3]);
                }
            }
        }
        // accumulator (m, n, k): vertex row g + 8*(k>>1), channel n*8 + 2t + (k&1)
        int x0, y0, z0;
        tile_origin(d, tile, x0, y0, z0);
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int li = warp * 32 + m * 16 + g + 8 * r;
                const int gx = x0 + (li & 7), gy = y0 + ((li >> 3) & 7), gz = z0 + (li >> 6);
                if (gx >= d.W || gy >= d.H || gz >= d.D) continue;
                const i64 v = gx + (i64)gy * d.W + (i64)gz * d.W * d.H;
                if constexpr (MODE == 1) {
                    if (t == 0) reinterpret_cast<float *>(out)[v] = acc[m][0][2 * r] + bias[0];
                } else {
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int ch = n * 8 + 2 * t;
                    float v0 = acc[m][n][2 * r], v1 = acc[m][n][2 * r + 1];
                    if constexpr (MODE == 0) {
                        v0 = fmaxf(v0 + bias[ch], 0.f);
                        v1 = fmaxf(v1 + bias[ch + 1], 0.f);
                    } else {
                        const __nv_bfloat162 a2 = *reinterpret_cast<const __nv_bfloat162 *>(aux + v * COUT + ch);
                        if (!(__bfloat162float(a2.x) > 0.f)) v0 = 0.f;
                        if (!(__bfloat162float(a2.y) > 0.f)) v1 = 0.f;
                    }
                    *reinterpret_cast<__nv_bfloat162 *>(reinterpret_cast<bf16 *>(out) + v * COUT + ch) =
                        __floats2bfloat162_rn(v0, v1);
                }
                }
            }
        __syncthreads();  // buffer `buf` is refilled two iterations on
    }
    cp_wait<0>();
}

// ------------------------------------------------- convolution on tcgen05
// The same convolution (same modes, FLIP, epilogues) on the 5th-generation
// tensor cores: tcgen05.mma with the accumulator in tensor memory.
//
// GEMM per z-slice of a tile: D[128 vertices][COUT] = sum over 27 taps of
// A_tap[128][CIN] x W_tap[CIN][COUT], K = 16 per instruction.  A tile is
// 8 x 16 x 4 vertices (x, y, z): four slices whose 128 rows are 16 lines of
// 8 x-neighbours.  Its halo box (10 x 18 x 6 vertices) sits in shared memory
// as CIN/8 planes, one per 16-byte group of 8 channels, each plane
// vertex-major (16 bytes per vertex).  In that layout the 8 rows of one
// x-line and one channel group are 128 contiguous bytes: one "core matrix" of
// the no-swizzle K-major operand layout.  A tap's A operand is the box
// shifted by the tap's offset: its descriptor starts at the shifted vertex,
// steps 10 x 16 bytes from one line to the next (stride byte offset) and one
// plane from one channel group to the next (leading byte offset).  Weights
// are stored per tap as [group][out channel][8 channels], the same layout for
// B.  The boxes arrive by TMA; the roles that issue the MMAs and copies and
// run the epilogue are described at k_conv_tc.
constexpr int QX = 8, QY = 16, QZ = 4;  // tile: QZ slices of 128 vertices (one MMA chain each)
constexpr int GX = QX + 2, GY = QY + 2, GZ = QZ + 2, GVOX = GX * GY * GZ;  // halo box
inline Dims make_tc_dims(int W, int H, int D) {
    Dims d{W, H, D, (W + QX - 1) / QX, (H + QY - 1) / QY, (D + QZ - 1) / QZ, 0};
    d.ntiles = (i64)d.ntx * d.nty * d.ntz;
    return d;
}
__device__ __forceinline__ void tc_tile_origin(const Dims &d, i64 tile, int &x0, int &y0, int &z0) {
    x0 = (int)(tile % d.ntx) * QX;
    y0 = (int)((tile / d.ntx) % d.nty) * QY;
    z0 = (int)(tile / ((i64)d.ntx * d.nty)) * QZ;
}
// shared-memory matrix descriptor: no swizzle, start / leading / stride byte
// offsets in 16-byte units, descriptor version 1 (bit 46)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor of kind::f16: f32 accumulator, bf16 A and B, both
// K-major, N = COUT, M = 128
template <int COUT>
__device__ __forceinline__ uint32_t tc_idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COUT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
    uint32_t done = 0;
    for (int it = 0; it < limit && !done; it++)
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity));
    return done != 0;
}
// this warp's 32 accumulator rows, columns 0..N-1 (N = 1, 16 or 32), into r;
// the registers are valid after tmem_wait()
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]) {
    if constexpr (N == 1) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r[0]) : "r"(taddr));
    } else if constexpr (N == 32) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
              "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
              "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
    } else {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
            "[%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
    }
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// The halo box arrives by TMA: the activations are a 4-d tensor (channel,
// x, y, z) with a box of (8 channels, GX, GY, GZ), so one bulk copy per
// 8-channel group writes exactly one plane (vertex-major, 16 bytes per
// vertex), zeros outside the grid.  The box starts at channel 8c (16-byte
// aligned, as a tiled copy's innermost coordinate must be) and at the halo's
// corner (x0-1, y0-1, z0-1), which may be -1.  Planes are padded to a
// multiple of 128 bytes (bulk-copy destinations).
constexpr uint32_t TC_PLANE = ((GVOX * 16 + 127) / 128) * 128;
template <int CIN>
__device__ __forceinline__ void tc_issue_box(const CUtensorMap *tm, uint32_t dst, uint32_t bar, int x0, int y0,
                                             int z0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar),
                 "r"((uint32_t)(CIN / 8 * GVOX * 16)));
#pragma unroll
    for (int c = 0; c < CIN / 8; c++)
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
            "%5}], [%6];\n" ::"r"(dst + c * TC_PLANE),
            "l"(reinterpret_cast<uint64_t>(tm)), "r"(c * 8), "r"(x0 - 1), "r"(y0 - 1), "r"(z0 - 1), "r"(bar)
            : "memory");
}

template <int CIN, int COUT>
constexpr size_t tc_smem() {
    return 128 + (size_t)27 * (CIN / 8) * COUT * 16 + 2 * (size_t)(CIN / 8) * TC_PLANE;
}

// Roles (192 threads): warp 0 lane 0 issues the MMAs, warp 1 lane 0 issues
// the TMA box copies, warps 2..5 run the epilogue (warp w reads accumulator
// lanes 32 (w mod 4) .. 32 (w mod 4) + 31, the quarter tensor memory lets it
// access).  Two box buffers and two accumulator sets (2 x QZ x 32 columns)
// let tile i's MMAs run while tile i-1's epilogue drains its accumulator and
// tile i+1's box arrives.  Barriers, per buffer b:
//   full[b]  the box of the tile using b has landed (TMA complete_tx)
//   mma[b]   that tile's MMAs are done (tcgen05.commit): its accumulator may
//            be read and its box buffer refilled
//   free[b]  the epilogue has read that accumulator (one arrival per
//            epilogue warp)
// Tile i uses b = i mod 2 and completes phase i / 2 of each barrier; every
// wait is bounded, and a role that gives up reports in *err and leaves its
// loop (the others then time out on the phases it no longer completes).
constexpr int kConvThreads = 192;
constexpr int kConvWaitPolls = 1 << 24;
template <int CIN, int COUT, int MODE, bool FLIP>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv_tc(const __grid_constant__ CUtensorMap tmap, Dims d,
                                                           const bf16 *__restrict__ wt, const float *__restrict__ bias,
                                                           void *out, const bf16 *__restrict__ aux, int *err) {
    constexpr int KCH = CIN / 8;
    constexpr uint32_t PLANE = TC_PLANE, WTAP = KCH * COUT * 16, WBYTES = 27 * WTAP, XBYTES = KCH * PLANE;
    constexpr uint32_t ACC_COLS = QZ * 32;  // one accumulator set
    static_assert(CIN % 16 == 0 && (COUT == 16 || COUT == 32), "tile shapes");
    static_assert(WTAP % 128 == 0, "planes stay 128-byte aligned");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t bar_full[2], bar_mma[2], bar_free[2];
    unsigned char *ws = smem_raw + ((128 - (smem_addr(smem_raw) & 127)) & 127);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 27 * COUT * KCH; i += blockDim.x) {
        const int tap = i / (COUT * KCH), rem = i - tap * (COUT * KCH), n = rem / KCH, c = rem - n * KCH;
        cp16(ws + tap * WTAP + c * COUT * 16 + n * 16, wt + ((i64)tap * COUT + n) * CIN + c * 8, 16);
    }
    cp_commit();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_addr(&tmem_slot)),
                     "n"(2 * ACC_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    // barrier addresses by buffer (selected, not indexed: no local-memory array)
    const uint32_t full0 = smem_addr(&bar_full[0]), full1 = smem_addr(&bar_full[1]);
    const uint32_t mma0 = smem_addr(&bar_mma[0]), mma1 = smem_addr(&bar_mma[1]);
    const uint32_t fre0 = smem_addr(&bar_free[0]), fre1 = smem_addr(&bar_free[1]);
    auto full = [&](int b) { return b ? full1 : full0; };
    auto mma = [&](int b) { return b ? mma1 : mma0; };
    auto fre = [&](int b) { return b ? fre1 : fre0; };
    const uint32_t wbase = smem_addr(ws), xbase0 = wbase + WBYTES;
    if (tid == 0) {
#pragma unroll
        for (int b = 0; b < 2; b++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(full(b)));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mma(b)));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(fre(b)));
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    cp_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;\n");  // the weights, for the tensor core
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_slot;
    const i64 first = blockIdx.x, stride = gridDim.x;
    const int ntile = first < d.ntiles ? (int)((d.ntiles - 1 - first) / stride + 1) : 0;
    bool failed = false;

    if (warp == 0) {
        if (lane == 0) {  // MMA issuer
            const uint32_t idesc = tc_idesc<COUT>();
            const uint64_t b0 = smem_desc(wbase, COUT * 16, 128);
            int committed = 0;
            for (int it = 0; it < ntile; it++) {
                const int b = it & 1;
                if (!mbar_wait(full(b), (uint32_t)(it >> 1) & 1u, kConvWaitPolls) ||
                    (it >= 2 && !mbar_wait(fre(b), (uint32_t)((it >> 1) - 1) & 1u, kConvWaitPolls))) {
                    failed = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                // descriptors of every (tap, channel group) differ from the
                // buffer's and the weights' base descriptors only in the
                // start-address field (shared addresses stay below 2^18, so
                // adding the offset in 16-byte units never carries out of it):
                // the unrolled chain adds immediates.  The QZ slices' chains
                // are interleaved so that consecutive MMAs go to different
                // accumulators.
                const uint64_t a0 = smem_desc(xbase0 + b * XBYTES, PLANE, GX * 16);
                const uint32_t acc = tmem + (uint32_t)b * ACC_COLS;
#pragma unroll
                for (int tap = 0; tap < 27; tap++) {
                    // offset + 1 along each axis (FLIP mirrors the tap: -d + 1 = 2 - (d + 1))
                    const int sx = FLIP ? 2 - tap % 3 : tap % 3, sy = FLIP ? 2 - (tap / 3) % 3 : (tap / 3) % 3,
                              sz = FLIP ? 2 - tap / 9 : tap / 9;
                    const uint32_t shift = (uint32_t)((sz * GY + sy) * GX + sx) * 16u;
#pragma unroll
                    for (int kk = 0; kk < KCH / 2; kk++)
#pragma unroll
                        for (int q = 0; q < QZ; q++)
                            tc_mma(acc + (uint32_t)(q * 32), a0 + ((shift + q * GY * GX * 16 + kk * 2 * PLANE) >> 4),
                                   b0 + ((tap * WTAP + kk * 2 * COUT * 16) >> 4), idesc, (tap | kk) != 0);
                }
                asm volatile(
                    "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mma(b)));
                committed = it + 1;
            }
            if (committed > 0)  // every MMA issued is done before the accumulators are released
                mbar_wait(mma((committed - 1) & 1), (uint32_t)((committed - 1) >> 1) & 1u, kConvWaitPolls);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {  // box producer
            int issued = 0;
            for (int it = 0; it < ntile; it++) {
                const int b = it & 1;
                // buffer b was last read by tile it-2's MMAs
                if (it >= 2 && !mbar_wait(mma(b), (uint32_t)((it >> 1) - 1) & 1u, kConvWaitPolls)) {
                    failed = true;
                    break;
                }
                int x0, y0, z0;
                tc_tile_origin(d, first + it * stride, x0, y0, z0);
                tc_issue_box<CIN>(&tmap, xbase0 + b * XBYTES, full(b), x0, y0, z0);
                issued = it + 1;
            }
            // the copies still in flight land before the block leaves
            for (int j = issued - 2; j < issued; j++)
                if (j >= 0) mbar_wait(full(j & 1), (uint32_t)(j >> 1) & 1u, kConvWaitPolls);
        }
        __syncwarp();
    } else {  // epilogue: warps 2..5
        const int quarter = warp & 3;
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
        float bsh[COUT];  // the layer's bias, held in registers (MODE 0 adds all, MODE 1 the first)
#pragma unroll
        for (int c = 0; c < COUT; c++) bsh[c] = MODE == 2 ? 0.f : (MODE == 1 && c > 0 ? 0.f : bias[c]);
        for (int it = 0; it < ntile; it++) {
            const int b = it & 1;
            if (!mbar_wait(mma(b), (uint32_t)(it >> 1) & 1u, kConvWaitPolls)) {
                failed = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            // every slice's rows at once, one wait, and the accumulator set is
            // handed back to the MMA issuer before the arithmetic and stores
            uint32_t raw[QZ][COUT];
#pragma unroll
            for (int zq = 0; zq < QZ; zq++) tmem_ld<COUT>(taddr + (uint32_t)b * ACC_COLS + (uint32_t)(zq * 32), raw[zq]);
            tmem_wait();
            asm volatile("tcgen05.fence::before_thread_sync;\n");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(fre(b)) : "memory");
            int x0, y0, z0;
            tc_tile_origin(d, first + it * stride, x0, y0, z0);
            const int r = quarter * 32 + lane, gx = x0 + (r & 7), gy = y0 + (r >> 3);
#pragma unroll
            for (int zq = 0; zq < QZ; zq++) {  // slice zq of the tile
                const int gz = z0 + zq;
                if (gx < d.W && gy < d.H && gz < d.D) {
                    const i64 v = gx + (i64)gy * d.W + (i64)gz * d.W * d.H;
                    if constexpr (MODE == 1) {
                        reinterpret_cast<float *>(out)[v] = __uint_as_float(raw[zq][0]) + bsh[0];
                    } else {
                        uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<bf16 *>(out) + v * COUT);
                        const uint4 *ax = MODE == 2 ? reinterpret_cast<const uint4 *>(aux + v * COUT) : nullptr;
#pragma unroll
                        for (int q = 0; q < COUT / 8; q++) {
                            uint4 mk = make_uint4(0, 0, 0, 0);
                            if constexpr (MODE == 2) mk = ax[q];
                            const bf16 *mb = reinterpret_cast<const bf16 *>(&mk);
                            uint4 pk;
                            __nv_bfloat162 *p2 = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                            for (int h = 0; h < 4; h++) {
                                const int ch = q * 8 + 2 * h;
                                float v0 = __uint_as_float(raw[zq][ch]), v1 = __uint_as_float(raw[zq][ch + 1]);
                                if constexpr (MODE == 0) {
                                    v0 = fmaxf(v0 + bsh[ch], 0.f);
                                    v1 = fmaxf(v1 + bsh[ch + 1], 0.f);
                                } else {
                                    if (!(__bfloat162float(mb[2 * h]) > 0.f)) v0 = 0.f;
                                    if (!(__bfloat162float(mb[2 * h + 1]) > 0.f)) v1 = 0.f;
                                }
                                p2[h] = __floats2bfloat162_rn(v0, v1);
                            }
                            o[q] = pk;
                        }
                    }
                }
            }
        }
    }
    if (failed) atomicOr(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(2 * ACC_COLS));
}

// ---------------------------------------- convolution on tcgen05, x-taps folded
// The same convolution with wider products, marching along x (or y or z, see
// make_march).  A tile is a column: 8 x 16 vertices of the plane across x (axes
// a and b: y and z, or z and y when that pads fewer rows) are the 128 rows of
// every product.  The input arrives as slices of constant x (10 x 18 vertices
// with the halo), each once.  Slice x contributes to the outputs x + 1, x and
// x - 1 through the taps dx = -1, 0, 1; their weight blocks side by side make one
// MMA of N = 3 COUT per (dy, dz) offset: 9 x CIN/16 MMAs per slice.  The three
// contributions to an output lie in the same lanes of three successive
// slices' accumulators, so the epilogue adds them in registers as it goes.
//
// Blocks take equal contiguous runs of outputs, column after column; a run
// that starts or ends inside a column reads one more slice there.  A vertex is
// one row of CIN channels in shared memory, swizzled over its own width (64 or
// 32 bytes); the swizzle goes by address bits, so an operand may start at any
// row, and a slice is a TMA box whose rows are whole vertices.
//
// Roles: warps 0 and 1 issue the MMAs of every other copy (two slices): the
// tensor pipe takes a product only when one before it is done, so the 400
// cycles that a warp spends on waits and commits would be idle, were there no
// other.  The whole warp walks and one elected lane issues: issued inside a
// branch on the lane, a product took 67 cycles whatever its width.  Warp 2
// brings the copies (full / empty barriers), warps 3..10 the weights, and then
// they run the epilogue, half of the channels of a lane quarter each, from four
// accumulators in turn.  Waits are bounded as in k_conv_tc.
//
// Bound by the products: 59 cycles for N = 96, the rate of back-to-back MMAs of
// that shape, and 47 for N = 48 (and for anything narrower).  161 x 127 x 110,
// against 14 x 8 x 2 tiles with halo boxes, where one lane issued and the shifts
// were warp shuffles: 32 -> 32 76 us (148), 16 -> 32 50 (101), 32 -> 16 59 (128);
// at 100 x 75 x 53 24 (40), 19 (30), 20 (35), data gradients 29 (47) and 23 (45).
// (The output layer, 32 -> 16, has its own kernel since: k_conv_out.)
constexpr int CX_A = 8, CX_B = 16, CX_GA = CX_A + 2, CX_GB = CX_B + 2, CX_NX = 2, CX_ACC = 4, CX_ST = 6;
constexpr int CX_EPI = 8, CX_THREADS = 96 + 32 * CX_EPI;
struct March {
    int n, na, nb;       // extents along the march, a, b
    i64 s, sa, sb;       // their vertex strides
    int t, tp, tq;       // and tap strides: of the march, and of the other axes p before q
    bool along_x() const { return t == 1; }
    int swapped;         // a = q and b = p
    int ta, tb;          // a column's outputs along a and b
    int nta;             // columns along a
    i64 outputs;         // of all columns
};
inline March march_along(int axis, int W, int H, int D, int ta, int tb) {
    const int n[3] = {W, H, D}, tap[3] = {1, 3, 9}, p = axis == 0 ? 1 : 0, q = axis == 2 ? 1 : 2;
    const i64 st[3] = {1, W, (i64)W * H};
    auto up = [](i64 k, i64 m) { return (k + m - 1) / m * m; };
    const bool swap = up(n[q], ta) * up(n[p], tb) < up(n[p], ta) * up(n[q], tb);
    const int a = swap ? q : p, b = swap ? p : q;
    return March{n[axis], n[a],   n[b],   st[axis], st[a], st[b], tap[axis], tap[p],
                 tap[q],  swap,   ta,     tb,       (n[a] + ta - 1) / ta,
                 up(n[a], ta) / ta * (up(n[b], tb) / tb) * n[axis]};
}
// Along x, unless fewer than a third of the columns' rows are vertices then (a grid of
// one or two vertices along y or z, or a few along both) and another axis has fewer
// slices.  Forward passes along x only, and so: 2000 x 1000 x 1 1.37 and 0.39 ms, 1000 x
// 2000 x 2 1.36 and 0.54, 20000 x 3 x 3 0.27 and 0.12 (14 x 8 x 2 tiles with halo boxes: 0.84,
// 0.90 and 0.19); 1000 x 1000 x 3, three eighths: 0.72 (0.88) along x.
inline March make_march(int W, int H, int D, int ta = CX_A, int tb = CX_B) {
    March m = march_along(0, W, H, D, ta, tb);
    if (m.outputs * ta * tb <= 3 * (i64)W * H * D) return m;
    for (int axis = 1; axis < 3; axis++) {
        const March o = march_along(axis, W, H, D, ta, tb);
        if (o.outputs < m.outputs) m = o;
    }
    return m;
}
// the part of a run that lies in one column: outputs [o0, o1) from slices j0..j1
struct Stretch {
    int a0, b0, o0, o1, j0, j1;
    __device__ __forceinline__ Stretch(const March &m, i64 g, i64 end) {
        const i64 col = g / m.n;
        a0 = (int)(col % m.nta) * m.ta;
        b0 = (int)(col / m.nta) * m.tb;
        o0 = (int)(g - col * m.n);
        o1 = (int)min((i64)m.n, o0 + (end - g));
        j0 = max(o0 - 1, 0);
        j1 = min(o1, m.n - 1);
    }
};
template <int CIN>
__host__ __device__ constexpr uint32_t cx_stage() {  // bytes of a copy's slices, to the next 1024
    return (CX_NX * CX_GB * CX_GA * CIN * 2 + 1023) / 1024 * 1024;
}
template <int CIN, int COUT>
constexpr size_t cx_smem() {
    return 1024 + (size_t)CX_ST * cx_stage<CIN>() + (size_t)9 * (CIN / 8) * (3 * COUT) * 16;
}
// descriptor of a K-major operand whose rows are as wide as their swizzle (64
// or 32 bytes), groups of eight rows `group` bytes apart
template <int ROW>
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t addr, uint32_t group) {
    static_assert(ROW == 64 || ROW == 32, "row widths");
    return smem_desc(addr, 16, group) | ((uint64_t)(ROW == 64 ? 4 : 6) << 61);
}
// one lane of a converged warp (elect.sync: always the same one)
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar));
}
struct alignas(32) Vec8 {
    uint32_t v[8];
};
__device__ __forceinline__ Vec8 ld32(const void *p) {  // 32 bytes, issued where it stands
    Vec8 r;
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                   "=r"(r.v[7])
                 : "l"(p));
    return r;
}
__device__ __forceinline__ void st32(void *p, const Vec8 &r) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(r.v[0]), "r"(r.v[1]), "r"(r.v[2]),
                 "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]), "r"(r.v[7])
                 : "memory");
}
// X: the march goes along x (a kernel of its own: with run-time strides 0.6 % of a forward pass)
template <int CIN, int COUT, int MODE, bool FLIP, bool X>
__global__ void __launch_bounds__(CX_THREADS, 1) k_conv_tcx(const __grid_constant__ CUtensorMap tmap, const March m,
                                                          const bf16 *__restrict__ wt, const float *__restrict__ bias,
                                                          bf16 *out, const bf16 *__restrict__ aux, int *err) {
    constexpr int KCH = CIN / 8, N = 3 * COUT, ROW = CIN * 2;
    constexpr uint32_t WGRP = N * 16, LINE = CX_GA * ROW, SLICE = CX_GB * LINE, STAGE = cx_stage<CIN>();
    constexpr uint32_t COLS = 128, ALLOC = CX_ACC * COLS;
    static_assert((CIN == 16 || CIN == 32) && COUT == 32 && MODE != 1, "tile shapes");
    static_assert(ALLOC == 512, "all of the tensor memory");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t bar_full[CX_ST], bar_empty[CX_ST], bar_mma[CX_ACC], bar_free[CX_ACC], bar_w, bar_done;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t ring = (smem_addr(smem_raw) + 1023) & ~1023u, wbase = ring + CX_ST * STAGE;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_addr(&tmem_slot)),
                     "n"(ALLOC));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    auto full = [&](int s) { return smem_addr(&bar_full[s]); };
    auto empty = [&](int s) { return smem_addr(&bar_empty[s]); };
    auto mma = [&](int q) { return smem_addr(&bar_mma[q % CX_ACC]); };
    auto fre = [&](int q) { return smem_addr(&bar_free[q % CX_ACC]); };
    const uint32_t wbar = smem_addr(&bar_w), done = smem_addr(&bar_done);
    if (tid == 0) {
        auto init = [](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(n)); };
        for (int s = 0; s < CX_ST; s++) {
            init(full(s), 1);
            init(empty(s), 1);
        }
        for (int q = 0; q < CX_ACC; q++) {
            init(mma(q), 1);
            init(fre(q), CX_EPI);
        }
        init(wbar, 32 * CX_EPI);
        init(done, 2);
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_slot;
    // this block's run of outputs
    const i64 per = m.outputs / gridDim.x, rest = m.outputs - per * gridDim.x;
    const i64 first = blockIdx.x * per + min((i64)blockIdx.x, rest), end = first + per + (blockIdx.x < rest);
    bool failed = false;

    if (warp < 2) {  // MMA issuers
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t b0 = smem_desc(wbase, WGRP, 128);
        const uint32_t dp = (m.swapped ? LINE : ROW) >> 4, dq = (m.swapped ? ROW : LINE) >> 4;
        if (!mbar_wait(wbar, 0u, kConvWaitPolls)) failed = true;
        int c = 0, q = 0;  // copies and slices so far
        for (i64 g = first; g < end && !failed;) {
            const Stretch t(m, g, end);
            for (int j = t.j0; j <= t.j1 && !failed; j += CX_NX, c++) {
                const int n = min(CX_NX, t.j1 - j + 1), s = c % CX_ST;
                if ((c & 1) == warp) {
                    // the copy, and the accumulators' last readers: a barrier per lane
                    const int mine = lane == 2 && n == 2 ? q + 1 : q;
                    const bool copy = lane == 0 || mine < CX_ACC;
                    if (!__all_sync(0xffffffffu, mbar_wait(copy ? full(s) : fre(mine),
                                                           (uint32_t)(copy ? c / CX_ST : mine / CX_ACC - 1) & 1u,
                                                           kConvWaitPolls))) {
                        failed = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n");
                    if (elect_one()) {
                        for (int e = 0; e < n; e++) {
                            const uint64_t a0 = swizzled_desc<ROW>(ring + s * STAGE + e * SLICE, LINE);
                            const uint32_t acc = tmem + (uint32_t)((q + e) % CX_ACC) * COLS;
#pragma unroll
                            for (int u = 0; u < 9; u++)
#pragma unroll
                                for (int kk = 0; kk < KCH / 2; kk++)
                                    tc_mma(acc, a0 + (u % 3 * dp + u / 3 * dq + kk * 2),
                                           b0 + (((u * KCH + kk * 2) * WGRP) >> 4), idesc, (u | kk) != 0);
                            tc_commit(mma(q + e));
                        }
                        tc_commit(empty(s));
                    }
                    __syncwarp();
                }
                q += n;
            }
            g += t.o1 - t.o0;
        }
        if (elect_one()) tc_commit(done);
        __syncwarp();
        if (!mbar_wait(done, 0u, kConvWaitPolls)) failed = true;  // every MMA issued is done
    } else if (warp == 2) {
        if (lane == 0) {  // copies
            int issued = 0;
            for (i64 g = first; g < end && !failed;) {
                const Stretch t(m, g, end);
                for (int j = t.j0; j <= t.j1; j += CX_NX) {
                    const int s = issued % CX_ST;
                    if (issued >= CX_ST && !mbar_wait(empty(s), (uint32_t)(issued / CX_ST - 1) & 1u, kConvWaitPolls)) {
                        failed = true;
                        break;
                    }
                    const uint32_t bar = full(s);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(CX_NX * SLICE));
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
                        "{%2, %3, %4, %5}], [%6];\n" ::"r"(ring + s * STAGE),
                        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"(t.a0 - 1), "r"(t.b0 - 1), "r"(j), "r"(bar)
                        : "memory");
                    issued++;
                }
                g += t.o1 - t.o0;
            }
            // the copies still in flight land before the block leaves
            for (int j = issued - CX_ST; j < issued; j++)
                if (j >= 0) mbar_wait(full(j % CX_ST), (uint32_t)(j / CX_ST) & 1u, kConvWaitPolls);
        }
        __syncwarp();
    } else {
        // weights: per offset u = (dp + 1) + 3 (dq + 1) and channel group kc, rows
        // n = t COUT + c hold march tap t - 1 of output channel c (mirrored under FLIP)
        unsigned char *ws = smem_raw + (wbase - smem_addr(smem_raw));
        for (int i = tid - 96; i < 9 * KCH * N; i += 32 * CX_EPI) {
            const int u = i / (KCH * N), rem = i - u * (KCH * N), kc = rem / N, n = rem - kc * N;
            const int t = n / COUT, c = n - t * COUT;
            const int at = X ? t + 3 * u : t * m.t + u % 3 * m.tp + u / 3 * m.tq, tap = FLIP ? 26 - at : at;
            cp16(ws + (u * KCH + kc) * WGRP + n * 16, wt + ((i64)tap * COUT + c) * CIN + kc * 8, 16);
        }
        cp_commit();
        cp_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;\n");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(wbar) : "memory");

        // the epilogue: channels [c0, c0 + NC) of lane quarter `quarter`
        constexpr int NC = COUT * 4 / CX_EPI;
        static_assert(NC == 16, "a thread stores 32 bytes");
        const int quarter = warp & 3, half = (warp - 3) >> 2, c0 = half * NC;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
        float bsh[MODE == 2 ? 1 : NC];
        if constexpr (MODE != 2) {
#pragma unroll
            for (int c = 0; c < NC; c++) bsh[c] = bias[c0 + c];
        }
        const int r = quarter * 32 + lane;
        int q = 0;
        for (i64 g = first; g < end && !failed;) {
            const Stretch t(m, g, end);
            const int a = t.a0 + (r & 7), b = t.b0 + (r >> 3);
            const bool row = a < m.na && b < m.nb;
            const i64 v0 = a * m.sa + b * m.sb;
            // contributions of the slices before j: to output j, and to output j - 1
            float next[NC], cur[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) next[c] = cur[c] = 0.f;
            auto store = [&](int o, const Vec8 &mk) {  // cur is complete: output o
                if (!row) return;
                const i64 v = v0 + o * (X ? 1 : m.s);
                Vec8 pk;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    float x0 = cur[2 * i], x1 = cur[2 * i + 1];
                    if constexpr (MODE == 0) {
                        x0 = fmaxf(x0 + bsh[2 * i], 0.f);
                        x1 = fmaxf(x1 + bsh[2 * i + 1], 0.f);
                    } else {
                        if (!(__uint_as_float(mk.v[i] << 16) > 0.f)) x0 = 0.f;
                        if (!(__uint_as_float(mk.v[i] & 0xFFFF0000u) > 0.f)) x1 = 0.f;
                    }
                    const __nv_bfloat162 two = __floats2bfloat162_rn(x0, x1);
                    pk.v[i] = *reinterpret_cast<const uint32_t *>(&two);
                }
                st32(out + v * COUT + c0, pk);
            };
            auto mask = [&](int o) {
                Vec8 mk{};
                if (MODE == 2 && row && o >= t.o0 && o < t.o1) mk = ld32(aux + (v0 + o * (X ? 1 : m.s)) * COUT + c0);
                return mk;
            };
            auto slice = [&](int j, const Vec8 &mk) {
                if (!mbar_wait(mma(q), (uint32_t)(q / CX_ACC) & 1u, kConvWaitPolls)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                const uint32_t at = lanes + (uint32_t)(q % CX_ACC) * COLS;
                uint32_t p0[NC], p1[NC], p2[NC];
                tmem_ld<NC>(at, p0);
                tmem_ld<NC>(at + COUT, p1);
                tmem_ld<NC>(at + 2 * COUT, p2);
                tmem_wait();
                asm volatile("tcgen05.fence::before_thread_sync;\n");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(fre(q)) : "memory");
#pragma unroll
                for (int c = 0; c < NC; c++) cur[c] += __uint_as_float(p2[c]);
                if (j > t.o0) store(j - 1, mk);
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    cur[c] = next[c] + __uint_as_float(p1[c]);
                    next[c] = __uint_as_float(p0[c]);
                }
                q++;
                return true;
            };
            // mk[i] is the mask of output j0 - 1 + i mod 4, loaded three slices before its use
            constexpr int AHEAD = MODE == 2 ? 4 : 1;
            Vec8 mk[AHEAD];
#pragma unroll
            for (int e = 0; e < AHEAD - 1; e++) mk[e] = mask(t.j0 - 1 + e);
            for (int j = t.j0; j <= t.j1 && !failed; j += AHEAD) {
#pragma unroll
                for (int e = 0; e < AHEAD; e++) {
                    if (j + e > t.j1 || failed) break;
                    mk[(e + AHEAD - 1) % AHEAD] = mask(j + e + AHEAD - 2);
                    if (!slice(j + e, mk[e])) failed = true;
                }
            }
            if (t.j1 < t.o1 && !failed) store(t.o1 - 1, mask(t.o1 - 1));  // the column's last output: nothing follows it
            g += t.o1 - t.o0;
        }
    }
    if (failed) atomicOr(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(ALLOC));
}

// ------------------------------------------------- the output layer on tcgen05
// The last convolution needs one output channel, and a product of fewer than 48
// columns takes as long as one of 48.  So the other direction is folded too: the
// columns are the 27 taps (of channel 0; 5 more are zero), and one product per 16
// channels gives what every vertex of a slice adds to its 27 neighbours: 2 MMAs
// per slice instead of 18.  The rows are the slice's 8 x 16 vertices with the
// halo, of which 6 x 14 are outputs; the x contributions are added in registers
// from slice to slice, the nine of the plane through shared memory.
//
// Runs, copies (four slices each, three stages) and waits as in k_conv_tcx; two
// blocks per SM.  Warp 0 issues, warp 1 copies, warps 2..5 are the epilogue; a
// warp whose wait gave up goes on without waiting, so that the others find it at
// their barrier.
//
// Bound by memory: 1.5 times the input through the caches.  161 x 127 x 110: 47 us
// (59 as 18 products of 48 columns); 100 x 75 x 53: 15 (20).  Exchanging four outputs
// at a time changed neither.
constexpr int OL_A = 6, OL_B = 14, OL_ROWS = 128, OL_NX = 4, OL_ST = 3, OL_ACC = 8, OL_COLS = 32, OL_THREADS = 192;
template <int CIN>
struct OutLayer {
    static constexpr uint32_t ROW = CIN * 2, SLICE = OL_ROWS * ROW, STAGE = OL_NX * SLICE, WBYTES = (CIN / 8) * 32 * 16;
    static constexpr size_t smem = 1024 + (size_t)OL_ST * STAGE + WBYTES + 2 * 9 * OL_ROWS * sizeof(float);
};
template <int CIN, int COUT, bool X>
__global__ void __launch_bounds__(OL_THREADS, 2) k_conv_out(const __grid_constant__ CUtensorMap tmap, const March m,
                                                          const bf16 *__restrict__ wt, const float *__restrict__ bias,
                                                          float *__restrict__ out, int *err) {
    using T = OutLayer<CIN>;
    constexpr uint32_t ALLOC = OL_ACC * OL_COLS;
    static_assert(ALLOC == 256 && OL_ACC == 2 * OL_NX, "two copies' accumulators");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t bar_full[OL_ST], bar_empty[OL_ST], bar_mma[2], bar_free[2], bar_done;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t ring = (smem_addr(smem_raw) + 1023) & ~1023u, wbase = ring + OL_ST * T::STAGE;
    unsigned char *ws = smem_raw + (wbase - smem_addr(smem_raw));
    float(*sum)[9][OL_ROWS] = reinterpret_cast<float(*)[9][OL_ROWS]>(ws + T::WBYTES);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_addr(&tmem_slot)),
                     "n"(ALLOC));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    auto full = [&](int s) { return smem_addr(&bar_full[s]); };
    auto empty = [&](int s) { return smem_addr(&bar_empty[s]); };
    auto mma = [&](int c) { return smem_addr(&bar_mma[c & 1]); };
    auto fre = [&](int c) { return smem_addr(&bar_free[c & 1]); };
    const uint32_t done = smem_addr(&bar_done);
    if (tid == 0) {
        auto init = [](uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(n)); };
        for (int s = 0; s < OL_ST; s++) {
            init(full(s), 1);
            init(empty(s), 1);
        }
        for (int c = 0; c < 2; c++) {
            init(mma(c), 1);
            init(fre(c), 4);
        }
        init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    // weights: per channel group, row n = 9 (dm + 1) + 3 (db + 1) + (da + 1) is that tap of output channel 0 (dm: along the march)
    for (int i = tid; i < (CIN / 8) * 32; i += OL_THREADS) {
        const int kc = i / 32, n = i % 32, dm = n / 9, a = n % 3, b = n / 3 % 3;
        const int tp = X ? 3 : m.tp, tq = X ? 9 : m.tq, tap = dm * (X ? 1 : m.t) + (m.swapped ? tq * a + tp * b : tp * a + tq * b);
        const uint4 v = n < 27 ? *reinterpret_cast<const uint4 *>(wt + (i64)tap * COUT * CIN + kc * 8) : make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(ws + i * 16) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;\n");
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_slot;
    const i64 per = m.outputs / gridDim.x, rest = m.outputs - per * gridDim.x;
    const i64 first = blockIdx.x * per + min((i64)blockIdx.x, rest), end = first + per + (blockIdx.x < rest);
    bool failed = false;

    if (warp == 0) {  // MMA issuer; c: copies so far
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t b0 = smem_desc(wbase, 32 * 16, 128);
        int c = 0;
        for (i64 g = first; g < end && !failed;) {
            const Stretch t(m, g, end);
            for (int j = t.j0; j <= t.j1; j += OL_NX, c++) {
                const int n = min(OL_NX, t.j1 - j + 1), s = c % OL_ST;
                const bool copy = lane == 0 || c < 2;  // the copy, and the accumulators' last readers: a barrier per lane
                if (!__all_sync(0xffffffffu, mbar_wait(copy ? full(s) : fre(c), (uint32_t)(copy ? c / OL_ST : c / 2 - 1) & 1u,
                                                       kConvWaitPolls))) {
                    failed = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                if (elect_one()) {
                    for (int e = 0; e < n; e++) {
                        const uint64_t a0 = swizzled_desc<T::ROW>(ring + s * T::STAGE + e * T::SLICE, 8 * T::ROW);
#pragma unroll
                        for (int kk = 0; kk < CIN / 16; kk++)
                            tc_mma(tmem + (uint32_t)((c & 1) * OL_NX + e) * OL_COLS, a0 + kk * 2,
                                   b0 + ((kk * 2 * 32 * 16) >> 4), idesc, kk != 0);
                    }
                    tc_commit(mma(c));
                    tc_commit(empty(s));
                }
                __syncwarp();
            }
            g += t.o1 - t.o0;
        }
        if (elect_one()) tc_commit(done);
        __syncwarp();
        if (!mbar_wait(done, 0u, kConvWaitPolls)) failed = true;  // every MMA issued is done
    } else if (warp == 1) {
        if (lane == 0) {  // copies
            int issued = 0;
            for (i64 g = first; g < end && !failed;) {
                const Stretch t(m, g, end);
                for (int j = t.j0; j <= t.j1; j += OL_NX) {
                    const int s = issued % OL_ST;
                    if (issued >= OL_ST && !mbar_wait(empty(s), (uint32_t)(issued / OL_ST - 1) & 1u, kConvWaitPolls)) {
                        failed = true;
                        break;
                    }
                    const uint32_t bar = full(s);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(T::STAGE));
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
                        "{%2, %3, %4, %5}], [%6];\n" ::"r"(ring + s * T::STAGE),
                        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"(t.a0 - 1), "r"(t.b0 - 1), "r"(j), "r"(bar)
                        : "memory");
                    issued++;
                }
                g += t.o1 - t.o0;
            }
            // the copies still in flight land before the block leaves
            for (int j = issued - OL_ST; j < issued; j++)
                if (j >= 0) mbar_wait(full(j % OL_ST), (uint32_t)(j / OL_ST) & 1u, kConvWaitPolls);
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, r = quarter * 32 + lane, ra = r & 7, rb = r >> 3;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const bool inner = ra >= 1 && ra <= OL_A && rb >= 1 && rb <= OL_B;
        const float b0 = bias[0];
        int c = 0, buf = 0;
        for (i64 g = first; g < end;) {
            const Stretch t(m, g, end);
            const int a = t.a0 + ra - 1, b = t.b0 + rb - 1;
            const bool row = inner && a < m.na && b < m.nb;
            const i64 v0 = a * m.sa + b * m.sb;
            // what this row adds to its nine neighbours' outputs at j (next) and j - 1 (cur), from the slices before j
            float next[9], cur[9];
#pragma unroll
            for (int u = 0; u < 9; u++) next[u] = cur[u] = 0.f;
            auto store = [&](int o) {  // cur is complete: output o
#pragma unroll
                for (int u = 0; u < 9; u++) sum[buf][u][r] = cur[u];
                asm volatile("bar.sync 1, 128;\n" ::: "memory");
                if (row) {
                    float x = 0.f;
#pragma unroll
                    for (int u = 0; u < 9; u++) x += sum[buf][u][r + (u % 3 - 1) + 8 * (u / 3 - 1)];
                    out[v0 + o * (X ? 1 : m.s)] = x + b0;
                }
                buf ^= 1;
            };
            for (int j = t.j0; j <= t.j1; j += OL_NX, c++) {
                const int n = min(OL_NX, t.j1 - j + 1);
                if (!failed && !mbar_wait(mma(c), (uint32_t)(c / 2) & 1u, kConvWaitPolls)) failed = true;
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                for (int e = 0; e < n; e++) {
                    uint32_t p[OL_COLS];
                    tmem_ld<OL_COLS>(lanes + (uint32_t)((c & 1) * OL_NX + e) * OL_COLS, p);
                    tmem_wait();
                    if (e == n - 1) {
                        asm volatile("tcgen05.fence::before_thread_sync;\n");
                        __syncwarp();
                        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(fre(c)) : "memory");
                    }
#pragma unroll
                    for (int u = 0; u < 9; u++) cur[u] += __uint_as_float(p[18 + u]);
                    if (j + e > t.o0) store(j + e - 1);
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        cur[u] = next[u] + __uint_as_float(p[9 + u]);
                        next[u] = __uint_as_float(p[u]);
                    }
                }
            }
            if (t.j1 < t.o1) store(t.o1 - 1);  // the column's last output: nothing follows it
            g += t.o1 - t.o0;
        }
    }
    if (failed) atomicOr(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(ALLOC));
}

// The tensor pipe's own ceiling for one instruction shape: one block per SM
// issues `reps` x 8 back-to-back tcgen05.mma of M = 128, N (32, 48, 64, 96,
// 128 or 256), K = 16 (bf16, f32 accumulators) on zeroed shared-memory
// operands, into the accumulators that fit 256 columns in turn, and waits for
// them (bounded).  A convolution made of
// N = 32 products (32 output channels) cannot run faster than this kernel at
// N = 32; measured on GB300 the rate grows with N up to N = 128.
// operands: A (4 KB) at 0, B (N x 32 bytes, <= 8 KB) at 16 KB; the launch asks
// for more shared memory than two blocks can share, so each SM runs one
constexpr uint32_t kRateOperands = 24 * 1024, kRateSmem = 120 * 1024;
template <int N>
__global__ void __launch_bounds__(128, 1) k_mma_rate(int reps, int *err) {
    extern __shared__ __align__(128) unsigned char rs[];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t mbar;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < (int)(kRateOperands / 4); i += blockDim.x) reinterpret_cast<uint32_t *>(rs)[i] = 0u;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;\n" ::"r"(smem_addr(&tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    const uint32_t bar = smem_addr(&mbar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    asm volatile("fence.proxy.async.shared::cta;\n");
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_slot;
    if (tid == 0) {
        const uint32_t base = smem_addr(rs);
        const uint64_t a = smem_desc(base, 2048, 128), b = smem_desc(base + 16384, N * 16, 128);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
        // accumulators side by side in the 256 columns, each at a multiple of
        // the power of two >= N (as the convolutions place theirs)
        constexpr int step = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256, nacc = 256 / step;
        for (int r = 0; r < reps; r++)
#pragma unroll
            for (int q = 0; q < 8; q++) tc_mma(tmem + (uint32_t)((q % nacc) * step), a, b, idesc, (r | q) != 0);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar));
        if (!mbar_wait(bar, 0u, 1 << 24)) atomicOr(err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;\n" ::"r"(tmem));
}

// ------------------------------------------------------------ weight gradient
// dW[tap][n][c] = sum_v dz[v][n] * act[v + off(tap)][c]; db[n] = sum_v dz[v][n].
// GEMM per tap with M = n, N = c, K = vertices of the tile.  Both operands are
// read transposed from the channels-last tiles by ldmatrix.trans.  16 warps
// share the 27 x (COUT/16) (tap, m-tile) units; each keeps its units'
// accumulators in registers across all tiles of the block, and the block
// writes one partial sum of every parameter of the layer to part[blockIdx.x].
template <int CIN, int COUT>
__global__ void __launch_bounds__(512, 1) k_wgrad(Dims d, const bf16 *__restrict__ act, const bf16 *__restrict__ dz,
                                                  float *__restrict__ part) {
    constexpr int AP = CIN + 8, DP = COUT + 8, NT = CIN / 8, MT = COUT / 16, UNITS = 27 * MT, NW = 16;
    constexpr int UPW = (UNITS + NW - 1) / NW;
    constexpr i64 NPAR = 27LL * COUT * CIN + COUT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16 *as0 = reinterpret_cast<bf16 *>(smem_raw);  // 2 x [HALO][AP]
    bf16 *ds0 = as0 + 2 * HALO * AP;                  // 2 x [TV][DP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    float acc[UPW][NT][4];
#pragma unroll
    for (int u = 0; u < UPW; u++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[u][n][k] = 0.f;
    float bacc = 0.f;
    // ldmatrix.trans roles.  A (dz^T: rows = out channel, k = vertex): lane
    // gives vertex (lane&7) + 8*(lane>>4), channel block 8*((lane>>3)&1).
    // B (act: k = vertex, n = in channel): vertex (lane&7) + 8*((lane>>3)&1),
    // channel block 8*(lane>>4) within a pair of n-tiles.
    const int va = (lane & 7) + 8 * (lane >> 4), ca = 8 * ((lane >> 3) & 1);
    const int vb = (lane & 7) + 8 * ((lane >> 3) & 1), cb = 8 * (lane >> 4);

    i64 tile = blockIdx.x;
    int buf = 0;
    if (tile < d.ntiles) {
        int x0, y0, z0;
        tile_origin(d, tile, x0, y0, z0);
        load_box<CIN, HX, HY, HZ>(as0, act, d, x0 - 1, y0 - 1, z0 - 1);
        load_box<COUT, TX, TY, TZ>(ds0, dz, d, x0, y0, z0);
    }
    cp_commit();
    for (; tile < d.ntiles; tile += gridDim.x, buf ^= 1) {
        const i64 next = tile + gridDim.x;
        if (next < d.ntiles) {
            int x0, y0, z0;
            tile_origin(d, next, x0, y0, z0);
            load_box<CIN, HX, HY, HZ>(as0 + (buf ^ 1) * HALO * AP, act, d, x0 - 1, y0 - 1, z0 - 1);
            load_box<COUT, TX, TY, TZ>(ds0 + (buf ^ 1) * TV * DP, dz, d, x0, y0, z0);
        }
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        const bf16 *as = as0 + buf * HALO * AP, *ds = ds0 + buf * TV * DP;
        if (lane < COUT)
            for (int v = warp * (TV / NW); v < (warp + 1) * (TV / NW); v++) bacc += __bfloat162float(ds[v * DP + lane]);
#pragma unroll
        for (int u = 0; u < UPW; u++) {
            const int unit = warp + u * NW;
            if (unit >= UNITS) continue;
            const int tap = unit / MT, mt = unit - tap * MT;
            const int dx = tap % 3 - 1, dy = (tap / 3) % 3 - 1, dzz = tap / 9 - 1;
            const int toff = (dzz * HY + dy) * HX + dx;
#pragma unroll 4
            for (int ks = 0; ks < TV / 16; ks++) {
                uint32_t a[4];
                ldm4t(a, ds + (ks * 16 + va) * DP + mt * 16 + ca);
                const int lb = ks * 16 + vb;
                const int hb = (((lb >> 6) + 1) * HY + ((lb >> 3) & 7) + 1) * HX + (lb & 7) + 1 + toff;
#pragma unroll
                for (int nt = 0; nt < NT; nt += 2) {
                    uint32_t b[4];
                    ldm4t(b, as + hb * AP + nt * 8 + cb);
                    mma16816(acc[u][nt], a, b[0], b[1]);
                    mma16816(acc[u][nt + 1], a, b[2], b[3]);
                }
            }
        }
        __syncthreads();
    }
    cp_wait<0>();
    float *p = part + (i64)blockIdx.x * NPAR;
#pragma unroll
    for (int u = 0; u < UPW; u++) {
        const int unit = warp + u * NW;
        if (unit >= UNITS) continue;
        const int tap = unit / MT, mt = unit - tap * MT;
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int n0 = mt * 16 + g, c0 = nt * 8 + 2 * t;
            float *q = p + ((i64)tap * COUT + n0) * CIN + c0;
            q[0] = acc[u][nt][0];
            q[1] = acc[u][nt][1];
            q[8 * CIN] = acc[u][nt][2];
            q[8 * CIN + 1] = acc[u][nt][3];
        }
    }
    // bias: fixed-order sum of the 16 warps' partials
    __syncthreads();
    float *red = reinterpret_cast<float *>(smem_raw);
    if (lane < COUT) red[warp * COUT + lane] = bacc;
    __syncthreads();
    if (tid < COUT) {
        float s = 0.f;
        for (int w = 0; w < NW; w++) s += red[w * COUT + tid];
        p[27LL * COUT * CIN + tid] = s;
    }
}

// --------------------------------------------- weight gradient on tcgen05
// The same sums as matrix products with the vertices as K.  With u = v + (0, 0, dz):
//   dW[dx, dy, dz][n][c] = sum_u dz[u - (0, 0, dz)][n] act[u + (dx, dy, 0)][c],
// so one product of M = 3 COUT rows (z shift, n), N = 3 CIN columns (y shift, c)
// and K = 16 vertices of an x-line serves nine taps, and the three x shifts have an
// accumulator each: 27 taps in three products per line.  A tile is 16 x 8 x 2
// vertices; its operands arrive by two TMA copies whose boxes put the lines
// where the products want them, a vertex as one row of its channels, swizzled
// over its own width (64 or 32 bytes):
//   dz  as [y 8][z 4][x 16], z from z0 - 1: three consecutive z lines are M
//   act as [z 2][y 10][x 18], from x0 - 1, y0 - 1: three consecutive y lines
//       are N, an x shift is a row of the start address (the swizzle goes by
//       address bits, so an operand may start at any row)
// Both operands are MN-major: the channels of 8 vertices are one swizzle atom,
// the next 8 vertices the next (stride offset), the next line of the operand
// one leading offset on.  M is 128: the rows past 3 COUT multiply whatever
// follows in the stage and are not read.  Zeros outside the grid make every
// edge right.  The accumulators stay in tensor memory over all tiles of a block
// and are written once, as this block's partial sums.
//
// Roles: warps 0..2 issue one x shift each, so that one's waits are hidden
// behind the others' products and every accumulator has its order; warp 3 brings
// the tiles; warps 4..7 sum the bias gradient from the same tiles and write the
// accumulators at the end.  empty[s] takes the commits of the three issuers and
// one arrival per bias warp.  Waits are bounded as in k_conv_tc.
//
// Bound by the products: 48 per tile at 59 cycles (N = 96), a quarter of their
// rows unused.  100 x 75 x 53: 29 us for 32 -> 32, 23 for 16 -> 32, 27 for 32 ->
// 16 (mma.sync: 98, 68 and 60; 16-byte copy rows and one issuing lane: 35, 30, 30).
constexpr int WG_X = 16, WG_Y = 8, WG_Z = 2, WG_ST = 4, WG_THREADS = 256;
template <int CIN, int COUT>
struct WgradTc {
    static constexpr uint32_t AROW = COUT * 2, ALINE = WG_X * AROW, ABYTES = WG_Y * (WG_Z + 2) * ALINE;
    static constexpr uint32_t BROW = CIN * 2, BLINE = (WG_X + 2) * BROW, BPLANE = (WG_Y + 2) * BLINE, BBYTES = WG_Z * BPLANE;
    static constexpr uint32_t STAGE = (ABYTES + BBYTES + 1023) / 1024 * 1024;
    static constexpr uint32_t N = 3 * CIN, COLS = N <= 64 ? 64 : 128, ALLOC = 3 * COLS <= 256 ? 256 : 512;
    static constexpr size_t smem = 1024 + (size_t)WG_ST * STAGE;
    // the rows past 3 COUT of the last line stay inside the stage
    static_assert(ABYTES - 3 * ALINE + (128 / COUT) * ALINE <= STAGE, "operand reads stay inside the stage");
    static_assert(ABYTES % 1024 == 0, "both boxes start on a swizzle pattern");
};
// descriptor of an MN-major operand of such rows, `line` bytes from one line to the next
template <int ROW>
__device__ __forceinline__ uint64_t lines_desc(uint32_t addr, uint32_t line) {
    static_assert(ROW == 64 || ROW == 32, "row widths");
    return smem_desc(addr, line, 8 * ROW) | ((uint64_t)(ROW == 64 ? 4 : 6) << 61);
}
template <int CIN, int COUT>
__global__ void __launch_bounds__(WG_THREADS, 1) k_wgrad_tc(const __grid_constant__ CUtensorMap tdz,
                                                            const __grid_constant__ CUtensorMap tact, int ntx, int nty,
                                                            i64 ntiles, float *__restrict__ part, int *err) {
    using T = WgradTc<CIN, COUT>;
    constexpr i64 NPAR = 27LL * COUT * CIN + COUT;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t bar_full[WG_ST], bar_empty[WG_ST], bar_done;
    __shared__ float red[4][COUT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_addr(smem_raw) + 1023) & ~1023u;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_slot)),
                     "n"(T::ALLOC));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    auto full = [&](int s) { return smem_addr(&bar_full[s]); };
    auto empty = [&](int s) { return smem_addr(&bar_empty[s]); };
    const uint32_t done = smem_addr(&bar_done);
    if (tid == 0) {
        for (int s = 0; s < WG_ST; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(full(s)));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 7;\n" ::"r"(empty(s)));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 3;\n" ::"r"(done));
        asm volatile("fence.mbarrier_init.release.cluster;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_slot;
    // this block's run of tiles, x fastest
    const i64 per = ntiles / gridDim.x, rest = ntiles - per * gridDim.x;
    const i64 first = blockIdx.x * per + min((i64)blockIdx.x, rest);
    const int ntile = (int)per + (blockIdx.x < rest);
    bool failed = false;

    if (warp < 3) {  // MMA issuers, one x shift each
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((T::N >> 3) << 17) |
                               ((uint32_t)(128 >> 4) << 24);
        int s = 0;
        uint32_t ph = 0;
        for (int it = 0; it < ntile; it++) {
            if (!__all_sync(0xffffffffu, mbar_wait(full(s), ph, kConvWaitPolls))) {
                failed = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            if (elect_one()) {
                const uint32_t ab = base + (uint32_t)s * T::STAGE;
                const uint64_t a0 = lines_desc<T::AROW>(ab, T::ALINE),
                               b0 = lines_desc<T::BROW>(ab + T::ABYTES + warp * T::BROW, T::BLINE);
#pragma unroll
                for (int q = 0; q < WG_Z; q++)
#pragma unroll
                    for (int y = 0; y < WG_Y; y++)
                        tc_mma(tmem + (uint32_t)warp * T::COLS, a0 + (((y * (WG_Z + 2) + q) * T::ALINE) >> 4),
                               b0 + ((q * T::BPLANE + y * T::BLINE) >> 4), idesc, (it | q | y) != 0);
                tc_commit(empty(s));
            }
            __syncwarp();
            if (++s == WG_ST) {
                s = 0;
                ph ^= 1;
            }
        }
        if (elect_one()) tc_commit(done);
        __syncwarp();
        if (!mbar_wait(done, 0u, kConvWaitPolls)) failed = true;  // every MMA issued is done
    } else if (warp == 3) {
        if (lane == 0) {  // operand producer
            int issued = 0, s = 0;
            uint32_t ph = 0;
            int x = (int)(first % ntx), y = (int)((first / ntx) % nty), z = (int)(first / ((i64)ntx * nty));
            for (int it = 0; it < ntile; it++) {
                if (it >= WG_ST && !mbar_wait(empty(s), ph ^ 1u, kConvWaitPolls)) {
                    failed = true;
                    break;
                }
                const uint32_t dst = base + (uint32_t)s * T::STAGE, bar = full(s);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(T::ABYTES + T::BBYTES));
                asm volatile(
                    "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
                    "{%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
                    "l"(reinterpret_cast<uint64_t>(&tdz)), "r"(0), "r"(x * WG_X), "r"(z * WG_Z - 1), "r"(y * WG_Y), "r"(bar)
                    : "memory");
                asm volatile(
                    "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
                    "{%2, %3, %4, %5}], [%6];\n" ::"r"(dst + T::ABYTES),
                    "l"(reinterpret_cast<uint64_t>(&tact)), "r"(0), "r"(x * WG_X - 1), "r"(y * WG_Y - 1), "r"(z * WG_Z), "r"(bar)
                    : "memory");
                issued = it + 1;
                if (++s == WG_ST) {
                    s = 0;
                    ph ^= 1;
                }
                if (++x == ntx) {
                    x = 0;
                    if (++y == nty) {
                        y = 0;
                        z++;
                    }
                }
            }
            // the copies still in flight land before the block leaves
            for (int j = issued - WG_ST; j < issued; j++)
                if (j >= 0) mbar_wait(full(j % WG_ST), (uint32_t)(j / WG_ST) & 1u, kConvWaitPolls);
        }
        __syncwarp();
    } else {  // bias gradient, then the accumulators
        const int w = warp - 4;
        float b[COUT];
#pragma unroll
        for (int c = 0; c < COUT; c++) b[c] = 0.f;
        int s = 0;
        uint32_t ph = 0;
        for (int it = 0; it < ntile; it++) {
            if (!mbar_wait(full(s), ph, kConvWaitPolls)) {
                failed = true;
                break;
            }
            // lines 2 w and 2 w + 1 of both planes: lane = x + 16 * plane; the row's
            // 16-byte chunks are permuted by the address bits above a pair of rows
            const uint32_t row = (uint32_t)((lane >> 4) + 1) * T::ALINE + (lane & 15) * T::AROW;
            const uint32_t ab = base + (uint32_t)s * T::STAGE + row, turn = (row >> 7) & (COUT / 8 - 1);
#pragma unroll
            for (int y = 0; y < 2; y++)
#pragma unroll
                for (int gch = 0; gch < COUT / 8; gch++) {
                    uint32_t r[4];
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                                 : "r"(ab + (uint32_t)(2 * w + y) * ((WG_Z + 2) * T::ALINE) + ((gch ^ turn) << 4)));
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        b[gch * 8 + 2 * k] += __uint_as_float(r[k] << 16);
                        b[gch * 8 + 2 * k + 1] += __uint_as_float(r[k] & 0xFFFF0000u);
                    }
                }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(empty(s)) : "memory");
            if (++s == WG_ST) {
                s = 0;
                ph ^= 1;
            }
        }
#pragma unroll
        for (int c = 0; c < COUT; c++) {
            for (int o = 16; o > 0; o >>= 1) b[c] += __shfl_xor_sync(0xffffffffu, b[c], o);
            if (lane == 0) red[w][c] = b[c];
        }
        if (!mbar_wait(done, 0u, kConvWaitPolls)) failed = true;
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        const int quarter = warp & 3, row = quarter * 32 + lane, sh = row / COUT, n = row % COUT;
        float *p = part + (i64)blockIdx.x * NPAR;
        if (quarter * 32 < 3 * COUT) {  // whole warps: the loads are warp-wide
#pragma unroll 1
            for (int tx = 0; tx < 3; tx++)
#pragma unroll 1
                for (int ty = 0; ty < 3; ty++) {
                    uint32_t r[CIN];
                    tmem_ld<CIN>(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)tx * T::COLS + (uint32_t)ty * CIN, r);
                    tmem_wait();
                    if (sh < 3) {  // z shift sh holds dz = 1 - sh
                        float4 *q = reinterpret_cast<float4 *>(p + ((i64)((2 - sh) * 9 + ty * 3 + tx) * COUT + n) * CIN);
#pragma unroll
                        for (int k = 0; k < CIN / 4; k++)
                            q[k] = make_float4(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]),
                                               __uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]));
                    }
                }
        }
    }
    if (failed) atomicOr(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (tid < COUT)
        part[(i64)blockIdx.x * NPAR + 27LL * COUT * CIN + tid] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(T::ALLOC));
}

// grad[i] = scale * sum over blocks of part[b][i], in a fixed order: eight
// threads per parameter take every eighth block, then their sums are added
// pairwise.  One launch for all layers, whose sums lie one after the other (one
// thread per parameter and a launch per layer: 304 loads in turn, 4 x 19 us; so:
// 15 us)
constexpr int kRedWays = 8;
struct Partials {
    const float *part[NLAYER];
    int nblk[NLAYER], first[NLAYER + 1];  // blocks that wrote; first block here
    i64 n[NLAYER], grad[NLAYER];
};
__global__ void __launch_bounds__(256) k_reduce(const Partials p, const float *__restrict__ scale, float *__restrict__ grad) {
    __shared__ float sm[kRedWays][32];
    int l = 0;
    while ((int)blockIdx.x >= p.first[l + 1]) l++;
    const float *part = p.part[l];
    const int nblk = p.nblk[l], col = threadIdx.x & 31, way = threadIdx.x >> 5;
    const i64 n = p.n[l], i = (i64)((int)blockIdx.x - p.first[l]) * 32 + col;
    float s = 0.f;
    if (i < n) {
#pragma unroll 8
        for (int b = way; b < nblk; b += kRedWays) s += part[(i64)b * n + i];
    }
    sm[way][col] = s;
    __syncthreads();
    if (way == 0 && i < n) {
        const float a = (sm[0][col] + sm[1][col]) + (sm[2][col] + sm[3][col]);
        const float b = (sm[4][col] + sm[5][col]) + (sm[6][col] + sm[7][col]);
        grad[p.grad[l] + i] = (a + b) * *scale;
    }
}

// ------------------------------------------------------------------- the loss
// Weighted over vertices (weight = the byte active[v], 0 = ignored):
// L = sum w (tanh(o) - target)^2 / sum w.  Writes dL/do without the 1/sum w
// factor (applied by k_reduce) into channel 0 of dz (16 channels, the others
// 0), and per-block (weighted sum, sum of weights) partials; the block that
// finishes last adds those in a fixed order: res[0] = mean loss, res[1] = sum of
// weights, scale = 1 / that (0 if none).  (Added by one thread of a kernel of
// its own: 14 + 109 us at 100 x 75 x 53; so: 13)
constexpr int kLossBlocks = 608;  // few: the blocks' sums are in double precision, which is slow here
__global__ void __launch_bounds__(256) k_loss(i64 V, const float *__restrict__ o, const float *__restrict__ target,
                                              const uint8_t *__restrict__ active, bf16 *__restrict__ dz,
                                              double *__restrict__ part, unsigned *__restrict__ ticket,
                                              double *__restrict__ res, float *__restrict__ scale) {
    double ls = 0.0;
    i64 cnt = 0;  // whole weights
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (i64)gridDim.x * blockDim.x) {
        float gval = 0.f;
        const float w = (float)active[v];
        if (w > 0.f) {
            const float y = tanhf(o[v]);
            const float e = y - target[v];
            ls += (double)w * e * e;
            cnt += active[v];
            gval = 2.f * w * e * (1.f - y * y);
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(gval, 0.f);
        st32(dz + v * 16, Vec8{{*reinterpret_cast<const uint32_t *>(&lo), 0u, 0u, 0u, 0u, 0u, 0u, 0u}});
    }
    __shared__ double sl[256];
    __shared__ i64 sc[256];
    __shared__ unsigned turn;
    for (int off = 16; off > 0; off >>= 1) {
        ls += __shfl_down_sync(0xffffffffu, ls, off);
        cnt += __shfl_down_sync(0xffffffffu, cnt, off);
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        sl[w] = ls;
        sc[w] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0;
        i64 b = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            a += sl[i];
            b += sc[i];
        }
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = (double)b;
        __threadfence();
        turn = atomicAdd(ticket, 1u);
    }
    __syncthreads();
    if (turn != gridDim.x - 1) return;
    __threadfence();
    double a = 0.0;
    i64 n = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 256) {
        a += __ldcg(part + 2 * i);
        n += (i64)__ldcg(part + 2 * i + 1);
    }
    sl[threadIdx.x] = a;
    sc[threadIdx.x] = n;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) {
            sl[threadIdx.x] += sl[threadIdx.x + k];
            sc[threadIdx.x] += sc[threadIdx.x + k];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    a = sl[0];
    const double b = (double)sc[0];
    res[0] = b > 0 ? a / b : 0.0;
    res[1] = b;
    *scale = b > 0 ? (float)(1.0 / b) : 0.f;
    *ticket = 0u;
}

// ------------------------------------------------------------ Adam + weights
__global__ void k_adam(i64 n, float *__restrict__ w, const float *__restrict__ gr, float *__restrict__ m1,
                       float *__restrict__ m2, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const float gv = gr[i];
        const float a = b1 * m1[i] + (1.f - b1) * gv;
        const float b = b2 * m2[i] + (1.f - b2) * gv * gv;
        m1[i] = a;
        m2[i] = b;
        w[i] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
    }
}
// bf16 copies of one layer's weights: forward [tap][n][c] and transposed
// [tap][c][n] (for the data gradient)
__global__ void k_pack(const float *__restrict__ w, int cin, int cout, bf16 *__restrict__ wf, bf16 *__restrict__ wt) {
    const int n = 27 * cin * cout;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = i % cin, no = (i / cin) % cout, tap = i / (cin * cout);
        const bf16 b = __float2bfloat16_rn(w[i]);
        wf[i] = b;
        wt[((i64)tap * cin + c) * cout + no] = b;
    }
}

}  // namespace

// ====================================================================== host
struct dmtz_cnn {
    float min_drop = 0.5f;  // proposal applied only where it lowers g by >= min_drop * bound
    int device = 0;
    int nsm = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    float *w = nullptr, *grad = nullptr, *m1 = nullptr, *m2 = nullptr;  // kParams each
    bf16 *wf = nullptr, *wt = nullptr;  // bf16 weights, forward and transposed, per layer at woff[l]
    float *part = nullptr;              // weight-gradient partials: nsm x all layers, or 2 nsm x one layer (mma.sync); from the first training pass on
    double *lpart = nullptr, *lres = nullptr;
    float *scale = nullptr;
    i64 step = 0;
    // activations of the last forward pass (a[2] aliases a[0] unless kept for training)
    i64 capV = 0;
    bool cap_train = false;
    bf16 *a[3] = {nullptr, nullptr, nullptr};
    bf16 *dz4 = nullptr, *gA = nullptr, *gB = nullptr;
    int lastW = 0, lastH = 0, lastD = 0, last_train = 0;
    const bf16 *last_feat = nullptr;
    const float *last_out = nullptr;
    // convolutions on tcgen05, three taps per product (2, the default) or one (1), or on mma.sync (0)
    int tensor_path = 2;
    unsigned *lticket = nullptr;
    std::map<const void *, int> per_sm;  // blocks of a kernel that an SM holds
    int *tc_err = nullptr;  // set by a tcgen05 convolution whose wait timed out
    // warm-start scratch
    i64 capS = 0;
    bf16 *feat = nullptr;
    uint8_t *active = nullptr;
    float *out = nullptr;
};

namespace {

i64 woff(int l) {
    i64 o = 0;
    for (int k = 0; k < l; k++) o += 27LL * LCIN[k] * LCOUT[k];
    return o;
}
constexpr i64 kWeights = 27LL * (16 * 32 + 32 * 32 + 32 * 32 + 32 * 16);

dmtz_status nfail(dmtz_cnn *n, dmtz_status s, const std::string &m) {
    if (n) n->err = m;
    return s;
}
#define NCK(call)                                                                                 \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess)                                                                    \
            return nfail(net, DMTZ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
cudaError_t nalloc(T **p, i64 n) {
    return cudaMalloc((void **)p, sizeof(T) * (size_t)std::max<i64>(n, 1));
}

uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

template <int CIN, int COUT, int MODE, bool FLIP>
constexpr size_t conv_smem() {
    return (size_t)(27 * COUT * (CIN + 8) + 2 * HALO * (CIN + 8)) * sizeof(bf16);
}
template <int CIN, int COUT>
constexpr size_t wgrad_smem() {
    return (size_t)(2 * HALO * (CIN + 8) + 2 * TV * (COUT + 8)) * sizeof(bf16);
}

// launches a persistent kernel with as many blocks as fit on the GPU (at most
// one per tile); the dynamic shared-memory limit is raised once per kernel
template <class K>
dmtz_status launch_persistent(dmtz_cnn *net, K kernel, int threads, size_t smem, i64 ntiles, int cap_blocks,
                              int *used_blocks, cudaStream_t st, void **args) {
    int &per_sm = net->per_sm[(const void *)kernel];  // asked for once: the shared memory depends on the kernel alone
    if (per_sm < 1) {
        NCK(cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        NCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
        if (per_sm < 1) return nfail(net, DMTZ_ERR_CUDA, "convolution kernel does not fit on an SM");
    }
    i64 blocks = std::min<i64>(ntiles, (i64)per_sm * net->nsm);
    if (cap_blocks > 0) blocks = std::min<i64>(blocks, cap_blocks);
    blocks = std::max<i64>(blocks, 1);
    if (used_blocks) *used_blocks = (int)blocks;
    NCK(cudaLaunchKernel((const void *)kernel, dim3((unsigned)blocks), dim3(threads), args, smem, st));
    return DMTZ_OK;
}

// the CUDA driver's tensor-map encoder, looked up once through the runtime
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    return encode;
}
dmtz_status encode_map(dmtz_cnn *net, CUtensorMap *tm, const bf16 *act, int rank, const cuuint64_t *dims,
                       const cuuint64_t *strides, const cuuint32_t *box,
                       CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE) {
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const auto encode = tensor_map_encoder();
    if (!encode) return nfail(net, DMTZ_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const CUresult r = encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<bf16 *>(act), dims, strides,
                              box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return nfail(net, DMTZ_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    return DMTZ_OK;
}
// tensor map of a channels-last bf16 activation tensor for k_conv_tc's boxes
dmtz_status box_map(dmtz_cnn *net, CUtensorMap *tm, const bf16 *act, int C, int W, int H, int D) {
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)C * 2 * W, (cuuint64_t)C * 2 * W * H};
    const cuuint32_t box[4] = {8, GX, GY, GZ};
    return encode_map(net, tm, act, 4, dims, strides, box);
}
// and for k_conv_tcx's and k_conv_out's slices with their halo: whole vertices, axes (channel, a, b, march)
dmtz_status slice_map(dmtz_cnn *net, CUtensorMap *tm, const bf16 *act, int C, const March &m, int nx) {
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)m.na, (cuuint64_t)m.nb, (cuuint64_t)m.n}, row = (cuuint64_t)C * 2;
    const cuuint64_t strides[3] = {row * m.sa, row * m.sb, row * m.s};
    const cuuint32_t box[4] = {(cuuint32_t)C, (cuuint32_t)m.ta + 2, (cuuint32_t)m.tb + 2, (cuuint32_t)nx};
    return encode_map(net, tm, act, 4, dims, strides, box, C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}
// and for k_wgrad_tc's lines: whole vertices, axes (channel, x, third, fourth);
// z_inner: third = z and fourth = y, else the other way round
dmtz_status line_map(dmtz_cnn *net, CUtensorMap *tm, const bf16 *act, int C, const Dims &d, bool z_inner, int bx, int b3,
                     int b4) {
    const cuuint64_t sx = (cuuint64_t)C * 2, sy = sx * d.W, sz = sy * d.H;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)d.W, (cuuint64_t)(z_inner ? d.D : d.H), (cuuint64_t)(z_inner ? d.H : d.D)};
    const cuuint64_t strides[3] = {sx, z_inner ? sz : sy, z_inner ? sy : sz};
    const cuuint32_t box[4] = {(cuuint32_t)C, (cuuint32_t)bx, (cuuint32_t)b3, (cuuint32_t)b4};
    return encode_map(net, tm, act, 4, dims, strides, box, C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

template <int CIN, int COUT, int MODE, bool FLIP>
dmtz_status conv(dmtz_cnn *net, const Dims &d, const bf16 *in, const bf16 *w, const float *bias, void *out,
                 const bf16 *aux, cudaStream_t st) {
    if (net->tensor_path == 2) {
        CUtensorMap tm;
        dmtz_status s;
        int *err = net->tc_err;
        if constexpr (MODE == 1) {
            March m = make_march(d.W, d.H, d.D, OL_A, OL_B);
            if ((s = slice_map(net, &tm, in, CIN, m, OL_NX)) != DMTZ_OK) return s;
            void *args[] = {&tm, &m, &w, &bias, &out, &err};
            auto kernel = m.along_x() ? k_conv_out<CIN, COUT, true> : k_conv_out<CIN, COUT, false>;
            return launch_persistent(net, kernel, OL_THREADS, OutLayer<CIN>::smem, m.outputs, 2 * net->nsm, nullptr, st, args);
        } else {
            March m = make_march(d.W, d.H, d.D);
            if ((s = slice_map(net, &tm, in, CIN, m, CX_NX)) != DMTZ_OK) return s;
            void *args[] = {&tm, &m, &w, &bias, &out, &aux, &err};
            auto kernel = m.along_x() ? k_conv_tcx<CIN, COUT, MODE, FLIP, true> : k_conv_tcx<CIN, COUT, MODE, FLIP, false>;
            return launch_persistent(net, kernel, CX_THREADS, cx_smem<CIN, COUT>(), m.outputs, net->nsm, nullptr, st, args);
        }
    }
    if (net->tensor_path) {
        Dims dt = make_tc_dims(d.W, d.H, d.D);
        CUtensorMap tm;
        dmtz_status s = box_map(net, &tm, in, CIN, d.W, d.H, d.D);
        if (s != DMTZ_OK) return s;
        int *err = net->tc_err;
        void *args[] = {&tm, &dt, &w, &bias, &out, &aux, &err};
        return launch_persistent(net, k_conv_tc<CIN, COUT, MODE, FLIP>, kConvThreads, tc_smem<CIN, COUT>(), dt.ntiles, 0,
                                 nullptr, st, args);
    }
    Dims dd = d;
    void *args[] = {&dd, &in, &w, &bias, &out, &aux};
    return launch_persistent(net, k_conv<CIN, COUT, MODE, FLIP>, 256, conv_smem<CIN, COUT, MODE, FLIP>(), d.ntiles, 0,
                             nullptr, st, args);
}

// gradients of layers [from, to) from their blocks' partial sums
dmtz_status reduce(dmtz_cnn *net, Partials &p, int from, int to, cudaStream_t st) {
    int blocks = 0;
    for (int l = 0; l < NLAYER; l++) {
        p.first[l] = blocks;
        p.grad[l] = layer_offset(l);
        p.n[l] = layer_params(l);
        if (l >= from && l < to) blocks += (int)((p.n[l] + 31) / 32);
    }
    p.first[NLAYER] = blocks;
    k_reduce<<<blocks, 256, 0, st>>>(p, net->scale, net->grad);
    NCK(cudaGetLastError());
    return DMTZ_OK;
}
// the blocks' partial sums of a layer; on the tcgen05 paths the caller reduces
// all layers at once
template <int CIN, int COUT>
dmtz_status wgrad(dmtz_cnn *net, const Dims &d, const bf16 *act, const bf16 *dz, int layer, Partials &p, cudaStream_t st) {
    float *part = net->part;
    int used = 0;
    dmtz_status s;
    if (net->tensor_path) {
        part += net->nsm * layer_offset(layer);
        CUtensorMap tdz, tact;
        if ((s = line_map(net, &tdz, dz, COUT, d, true, WG_X, WG_Z + 2, WG_Y)) != DMTZ_OK ||
            (s = line_map(net, &tact, act, CIN, d, false, WG_X + 2, WG_Y + 2, WG_Z)) != DMTZ_OK)
            return s;
        int ntx = (d.W + WG_X - 1) / WG_X, nty = (d.H + WG_Y - 1) / WG_Y, *err = net->tc_err;
        i64 ntiles = (i64)ntx * nty * ((d.D + WG_Z - 1) / WG_Z);
        void *args[] = {&tdz, &tact, &ntx, &nty, &ntiles, &part, &err};
        s = launch_persistent(net, k_wgrad_tc<CIN, COUT>, WG_THREADS, WgradTc<CIN, COUT>::smem, ntiles, net->nsm, &used,
                              st, args);
    } else {
        Dims dd = d;
        void *args[] = {&dd, &act, &dz, &part};
        s = launch_persistent(net, k_wgrad<CIN, COUT>, 512, wgrad_smem<CIN, COUT>(), d.ntiles, 2 * net->nsm, &used, st,
                              args);
    }
    if (s != DMTZ_OK) return s;
    p.part[layer] = part;
    p.nblk[layer] = used;
    return net->tensor_path ? DMTZ_OK : reduce(net, p, layer, layer + 1, st);
}

dmtz_status pack(dmtz_cnn *net, cudaStream_t st) {
    for (int l = 0; l < NLAYER; l++) {
        k_pack<<<64, 256, 0, st>>>(net->w + layer_offset(l), LCIN[l], LCOUT[l], net->wf + woff(l), net->wt + woff(l));
    }
    NCK(cudaGetLastError());
    return DMTZ_OK;
}

dmtz_status ensure_act(dmtz_cnn *net, i64 V, bool train) {
    if (train && !net->part) NCK(nalloc(&net->part, net->nsm * kParams));  // (50 MB that inference does without)
    if (V <= net->capV && (!train || net->cap_train)) return DMTZ_OK;
    cudaFree(net->a[0]);
    cudaFree(net->a[1]);
    if (net->cap_train) cudaFree(net->a[2]);
    cudaFree(net->dz4);
    cudaFree(net->gA);
    cudaFree(net->gB);
    net->a[0] = net->a[1] = net->a[2] = net->dz4 = net->gA = net->gB = nullptr;
    net->capV = 0;
    net->cap_train = false;
    const i64 cap = std::max(V, net->capV);
    NCK(nalloc(&net->a[0], cap * 32));
    NCK(nalloc(&net->a[1], cap * 32));
    if (train) {
        NCK(nalloc(&net->a[2], cap * 32));
        NCK(nalloc(&net->dz4, cap * 16));
        NCK(nalloc(&net->gA, cap * 32));
        NCK(nalloc(&net->gB, cap * 32));
    } else {
        net->a[2] = net->a[0];
    }
    net->capV = cap;
    net->cap_train = train;
    return DMTZ_OK;
}

dmtz_status check_grid(dmtz_cnn *net, int W, int H, int D) {
    if (!net) return DMTZ_ERR_ARG;
    if (W < 1 || H < 1 || D < 1) return nfail(net, DMTZ_ERR_ARG, "grid dimensions must be >= 1");
    if ((i64)W * H * D > (1LL << 40)) return nfail(net, DMTZ_ERR_ARG, "grid too large");
    return DMTZ_OK;
}

}  // namespace

namespace dmtz_cnn_impl {

const std::string &error_of(const dmtz_cnn *net) { return net->err; }
int device_of(const dmtz_cnn *net) { return net->device; }
float min_drop_of(const dmtz_cnn *net) { return net->min_drop; }

dmtz_status forward_on(dmtz_cnn *net, int W, int H, int D, const bf16 *feat, float *out, int train,
                       cudaStream_t st) {
    dmtz_status s = check_grid(net, W, H, D);
    if (s != DMTZ_OK) return s;
    if (!feat || !out || ((uintptr_t)feat & 15)) return nfail(net, DMTZ_ERR_ARG, "features must be 16-byte aligned");
    NCK(cudaSetDevice(net->device));
    const Dims d = make_dims(W, H, D);
    const i64 V = (i64)W * H * D;
    if ((s = ensure_act(net, V, train != 0)) != DMTZ_OK) return s;
    bf16 *a1 = net->a[0], *a2 = net->a[1], *a3 = net->a[2];
    const float *w = net->w;
    if ((s = conv<16, 32, 0, false>(net, d, feat, net->wf + woff(0), w + layer_offset(0) + 27 * 32 * 16, a1, nullptr,
                                    st)) != DMTZ_OK)
        return s;
    if ((s = conv<32, 32, 0, false>(net, d, a1, net->wf + woff(1), w + layer_offset(1) + 27 * 32 * 32, a2, nullptr,
                                    st)) != DMTZ_OK)
        return s;
    if ((s = conv<32, 32, 0, false>(net, d, a2, net->wf + woff(2), w + layer_offset(2) + 27 * 32 * 32, a3, nullptr,
                                    st)) != DMTZ_OK)
        return s;
    if ((s = conv<32, 16, 1, false>(net, d, a3, net->wf + woff(3), w + layer_offset(3) + 27 * 16 * 32, out, nullptr,
                                    st)) != DMTZ_OK)
        return s;
    net->lastW = W;
    net->lastH = H;
    net->lastD = D;
    net->last_train = train != 0;
    net->last_feat = feat;
    net->last_out = out;
    return DMTZ_OK;
}

dmtz_status scratch(dmtz_cnn *net, int64_t V, bf16 **feat, uint8_t **active, float **out) {
    if (V > net->capS) {
        cudaFree(net->feat);
        cudaFree(net->active);
        cudaFree(net->out);
        net->feat = nullptr;
        net->active = nullptr;
        net->out = nullptr;
        net->capS = 0;
        NCK(nalloc(&net->feat, V * kFeat));
        NCK(nalloc(&net->active, V));
        NCK(nalloc(&net->out, V));
        net->capS = V;
    }
    *feat = net->feat;
    *active = net->active;
    *out = net->out;
    return DMTZ_OK;
}

}  // namespace dmtz_cnn_impl

using dmtz_cnn_impl::forward_on;

extern "C" {

int64_t dmtz_cnn_num_params(void) { return kParams; }

dmtz_status dmtz_cnn_create(dmtz_cnn **out, int device, uint64_t seed) {
    if (!out) return DMTZ_ERR_ARG;
    *out = nullptr;
    dmtz_cnn *net = new dmtz_cnn();
    net->device = device;
    auto bail = [&](dmtz_status s) {
        dmtz_cnn_destroy(net);
        return s;
    };
    if (cudaSetDevice(device) != cudaSuccess) return bail(DMTZ_ERR_CUDA);
    if (cudaDeviceGetAttribute(&net->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return bail(DMTZ_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(DMTZ_ERR_CUDA);
    if (nalloc(&net->w, kParams) || nalloc(&net->grad, kParams) || nalloc(&net->m1, kParams) ||
        nalloc(&net->m2, kParams) || nalloc(&net->wf, kWeights) || nalloc(&net->wt, kWeights) ||
        nalloc(&net->lpart, 2 * kLossBlocks) || nalloc(&net->lres, 3) || nalloc(&net->scale, 1))
        return bail(DMTZ_ERR_CUDA);
    net->tc_err = reinterpret_cast<int *>(net->lres + 2);  // behind the loss, so that one copy brings both
    net->lticket = reinterpret_cast<unsigned *>(net->lres + 2) + 1;
    if (cudaMemset(net->tc_err, 0, sizeof(double)) != cudaSuccess) return bail(DMTZ_ERR_CUDA);
    // He-uniform weights (bound sqrt(6 / fan_in)); the output layer 0.1x and
    // only its channel 0 nonzero; zero biases
    std::vector<float> h((size_t)kParams, 0.f);
    uint64_t s = seed ^ 0x6A09E667F3BCC909ull;
    for (int l = 0; l < NLAYER; l++) {
        const double b = std::sqrt(6.0 / (27.0 * LCIN[l])) * (l == NLAYER - 1 ? 0.1 : 1.0);
        float *p = h.data() + layer_offset(l);
        for (int tap = 0; tap < 27; tap++)
            for (int n = 0; n < LCOUT[l]; n++)
                for (int c = 0; c < LCIN[l]; c++) {
                    const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
                    const bool live = l < NLAYER - 1 || n == 0;
                    p[((i64)tap * LCOUT[l] + n) * LCIN[l] + c] = live ? (float)((2.0 * u - 1.0) * b) : 0.f;
                }
    }
    if (dmtz_cnn_set_params(net, h.data()) != DMTZ_OK) return bail(DMTZ_ERR_CUDA);
    *out = net;
    return DMTZ_OK;
}

void dmtz_cnn_destroy(dmtz_cnn *net) {
    if (!net) return;
    cudaSetDevice(net->device);
    if (net->stream) cudaStreamSynchronize(net->stream);
    for (void *p : {(void *)net->w, (void *)net->grad, (void *)net->m1, (void *)net->m2, (void *)net->wf,
                    (void *)net->wt, (void *)net->part, (void *)net->lpart, (void *)net->lres, (void *)net->scale,
                    (void *)net->a[0], (void *)net->a[1], (void *)net->dz4, (void *)net->gA, (void *)net->gB,
                    (void *)net->feat, (void *)net->active, (void *)net->out})
        cudaFree(p);
    if (net->cap_train) cudaFree(net->a[2]);
    if (net->stream) cudaStreamDestroy(net->stream);
    delete net;
}

const char *dmtz_cnn_last_error(const dmtz_cnn *net) { return net ? net->err.c_str() : "null network"; }

dmtz_status dmtz_cnn_set_min_drop(dmtz_cnn *net, float min_drop) {
    if (!net) return DMTZ_ERR_ARG;
    if (!(min_drop >= 0.f) || !(min_drop <= 2.f)) return nfail(net, DMTZ_ERR_ARG, "min_drop must be in [0, 2]");
    net->min_drop = min_drop;
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_set_params(dmtz_cnn *net, const float *host) {
    if (!net || !host) return DMTZ_ERR_ARG;
    NCK(cudaSetDevice(net->device));
    NCK(cudaMemcpyAsync(net->w, host, sizeof(float) * kParams, cudaMemcpyHostToDevice, net->stream));
    NCK(cudaMemsetAsync(net->m1, 0, sizeof(float) * kParams, net->stream));
    NCK(cudaMemsetAsync(net->m2, 0, sizeof(float) * kParams, net->stream));
    NCK(cudaMemsetAsync(net->grad, 0, sizeof(float) * kParams, net->stream));
    net->step = 0;
    dmtz_status s = pack(net, net->stream);
    if (s != DMTZ_OK) return s;
    NCK(cudaStreamSynchronize(net->stream));
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_get_params(dmtz_cnn *net, float *host) {
    if (!net || !host) return DMTZ_ERR_ARG;
    NCK(cudaSetDevice(net->device));
    NCK(cudaMemcpyAsync(host, net->w, sizeof(float) * kParams, cudaMemcpyDeviceToHost, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_get_grads(dmtz_cnn *net, float *host) {
    if (!net || !host) return DMTZ_ERR_ARG;
    NCK(cudaSetDevice(net->device));
    NCK(cudaMemcpyAsync(host, net->grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    return DMTZ_OK;
}

// a tcgen05 convolution whose completion wait timed out leaves a flag (the
// kernel itself returns); the synchronous calls report it
// (res: the loss and its weight as well; waits for the network's stream)
static dmtz_status check_tc(dmtz_cnn *net, double *res = nullptr) {
    double h[3];
    NCK(cudaMemcpyAsync(h, net->lres, sizeof(h), cudaMemcpyDeviceToHost, net->stream));
    NCK(cudaStreamSynchronize(net->stream));
    int e;
    memcpy(&e, h + 2, sizeof(e));
    if (e) {
        NCK(cudaMemset(net->tc_err, 0, sizeof(int)));
        return nfail(net, DMTZ_ERR_CUDA, "a tensor-core convolution timed out waiting for its MMAs");
    }
    if (res) *res = h[0];
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_set_tensor_path(dmtz_cnn *net, int path) {
    if (!net || path < 0 || path > 2) return DMTZ_ERR_ARG;
    net->tensor_path = path;
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_mma_ceiling(dmtz_cnn *net, int n, int reps, double *tflops) {
    // the shapes are compile-time constants: the issuing thread does no arithmetic between MMAs
    void (*kern)(int, int *) = n == 32 ? k_mma_rate<32> : n == 48 ? k_mma_rate<48> : n == 64 ? k_mma_rate<64>
                             : n == 96 ? k_mma_rate<96> : n == 128 ? k_mma_rate<128> : n == 256 ? k_mma_rate<256>
                                                                                                 : nullptr;
    if (!net || !tflops || reps < 1 || reps > (1 << 16) || !kern) return DMTZ_ERR_ARG;
    NCK(cudaSetDevice(net->device));
    cudaStream_t st = net->stream;
    NCK(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRateSmem));
    int *err = nullptr;
    NCK(cudaMalloc(&err, sizeof(int)));
    cudaEvent_t e[2];
    cudaEventCreate(&e[0]);
    cudaEventCreate(&e[1]);
    cudaMemsetAsync(err, 0, sizeof(int), st);
    kern<<<net->nsm, 128, kRateSmem, st>>>(reps, err);  // warm-up
    cudaEventRecord(e[0], st);
    kern<<<net->nsm, 128, kRateSmem, st>>>(reps, err);
    cudaEventRecord(e[1], st);
    int herr = 0;
    cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    const cudaError_t ce = cudaStreamSynchronize(st);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e[0], e[1]);
    cudaEventDestroy(e[0]);
    cudaEventDestroy(e[1]);
    cudaFree(err);
    if (ce != cudaSuccess) return nfail(net, DMTZ_ERR_CUDA, std::string("k_mma_rate: ") + cudaGetErrorString(ce));
    if (herr) return nfail(net, DMTZ_ERR_CUDA, "k_mma_rate: the MMAs did not complete in time");
    *tflops = 2.0 * 128 * n * 16 * 8.0 * reps * net->nsm / (ms * 1e-3) / 1e12;
    return DMTZ_OK;
}

dmtz_status dmtz_cnn_forward(dmtz_cnn *net, int W, int H, int D, const void *feat, float *out, int train) {
    if (!net) return DMTZ_ERR_ARG;
    dmtz_status s = forward_on(net, W, H, D, static_cast<const bf16 *>(feat), out, train, net->stream);
    if (s != DMTZ_OK) return s;
    return check_tc(net);
}

dmtz_status dmtz_cnn_backward(dmtz_cnn *net, int W, int H, int D, const float *target, const uint8_t *active,
                              double *loss) {
    dmtz_status s = check_grid(net, W, H, D);
    if (s != DMTZ_OK) return s;
    if (!target || !active) return nfail(net, DMTZ_ERR_ARG, "null target or mask");
    if (!net->last_train || net->lastW != W || net->lastH != H || net->lastD != D)
        return nfail(net, DMTZ_ERR_ARG, "backward needs a training forward pass on the same grid");
    NCK(cudaSetDevice(net->device));
    cudaStream_t st = net->stream;
    const Dims d = make_dims(W, H, D);
    const i64 V = (i64)W * H * D;
    k_loss<<<kLossBlocks, 256, 0, st>>>(V, net->last_out, target, active, net->dz4, net->lpart, net->lticket, net->lres,
                                         net->scale);
    NCK(cudaGetLastError());
    bf16 *a1 = net->a[0], *a2 = net->a[1], *a3 = net->a[2];
    Partials p{};
    // layer 4: data gradient into a3's space (ReLU mask of a3), weight gradient
    if ((s = conv<16, 32, 2, true>(net, d, net->dz4, net->wt + woff(3), nullptr, net->gA, a3, st)) != DMTZ_OK) return s;
    if ((s = wgrad<32, 16>(net, d, a3, net->dz4, 3, p, st)) != DMTZ_OK) return s;
    // layer 3
    if ((s = conv<32, 32, 2, true>(net, d, net->gA, net->wt + woff(2), nullptr, net->gB, a2, st)) != DMTZ_OK) return s;
    if ((s = wgrad<32, 32>(net, d, a2, net->gA, 2, p, st)) != DMTZ_OK) return s;
    // layer 2
    if ((s = conv<32, 32, 2, true>(net, d, net->gB, net->wt + woff(1), nullptr, net->gA, a1, st)) != DMTZ_OK) return s;
    if ((s = wgrad<32, 32>(net, d, a1, net->gB, 1, p, st)) != DMTZ_OK) return s;
    // layer 1 (no data gradient of the features)
    if ((s = wgrad<16, 32>(net, d, net->last_feat, net->gA, 0, p, st)) != DMTZ_OK) return s;
    if (net->tensor_path && (s = reduce(net, p, 0, NLAYER, st)) != DMTZ_OK) return s;
    return check_tc(net, loss);
}

dmtz_status dmtz_cnn_step(dmtz_cnn *net, float lr) {
    if (!net) return DMTZ_ERR_ARG;
    if (!(lr >= 0.f) || !std::isfinite(lr)) return nfail(net, DMTZ_ERR_ARG, "learning rate must be finite, >= 0");
    NCK(cudaSetDevice(net->device));
    net->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = (float)(1.0 - std::pow((double)b1, (double)net->step));
    const float c2 = (float)(1.0 - std::pow((double)b2, (double)net->step));
    k_adam<<<(unsigned)((kParams + 255) / 256), 256, 0, net->stream>>>(kParams, net->w, net->grad, net->m1, net->m2,
                                                                       lr, b1, b2, 1e-8f, c1, c2);
    NCK(cudaGetLastError());
    dmtz_status s = pack(net, net->stream);
    if (s != DMTZ_OK) return s;
    NCK(cudaStreamSynchronize(net->stream));
    return DMTZ_OK;
}

}  // extern "C"

extern "C" dmtz_status dmtz_cnn_profile(dmtz_cnn *net, int W, int H, int D, const void *feat, float *out,
                                        const float *target, const uint8_t *active, int reps, double ms[4]) {
    dmtz_status s = check_grid(net, W, H, D);
    if (s != DMTZ_OK) return s;
    if (!ms || reps < 1 || !target || !active) return nfail(net, DMTZ_ERR_ARG, "bad profile arguments");
    NCK(cudaSetDevice(net->device));
    cudaStream_t st = net->stream;
    const bf16 *fb = static_cast<const bf16 *>(feat);
    cudaEvent_t e[2];
    NCK(cudaEventCreate(&e[0]));
    NCK(cudaEventCreate(&e[1]));
    float t = 0.f;
    auto timed = [&](auto &&body, double &acc) -> dmtz_status {
        NCK(cudaEventRecord(e[0], st));
        for (int r = 0; r < reps; r++) {
            dmtz_status q = body();
            if (q != DMTZ_OK) return q;
        }
        NCK(cudaEventRecord(e[1], st));
        NCK(cudaEventSynchronize(e[1]));
        NCK(cudaEventElapsedTime(&t, e[0], e[1]));
        acc = (double)t / reps;
        return DMTZ_OK;
    };
    // the training steps are undone afterwards: weights, Adam moments and step count
    float *keep = nullptr;
    NCK(nalloc(&keep, 3 * kParams));
    NCK(cudaMemcpyAsync(keep, net->w, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st));
    NCK(cudaMemcpyAsync(keep + kParams, net->m1, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st));
    NCK(cudaMemcpyAsync(keep + 2 * kParams, net->m2, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st));
    const i64 step0 = net->step;
    const Dims d = make_dims(W, H, D);
    if ((s = forward_on(net, W, H, D, fb, out, 1, st)) != DMTZ_OK) return s;  // warm-up, sizes buffers
    NCK(cudaStreamSynchronize(st));
    s = timed([&]() { return forward_on(net, W, H, D, fb, out, 0, st); }, ms[0]);
    if (s == DMTZ_OK)
        s = timed(
            [&]() {
                dmtz_status q = forward_on(net, W, H, D, fb, out, 1, st);
                if (q == DMTZ_OK) q = dmtz_cnn_backward(net, W, H, D, target, active, nullptr);
                if (q == DMTZ_OK) q = dmtz_cnn_step(net, 0.f);
                return q;
            },
            ms[1]);
    if (s == DMTZ_OK)
        s = timed(
            [&]() {
                return conv<32, 32, 0, false>(net, d, net->a[0], net->wf + woff(1),
                                              net->w + layer_offset(1) + 27 * 32 * 32, net->a[1], nullptr, st);
            },
            ms[2]);
    if (s == DMTZ_OK)
        s = timed(
            [&]() {
                Partials p{};
                const dmtz_status r = wgrad<32, 32>(net, d, net->a[1], net->gB, 2, p, st);
                return r == DMTZ_OK && net->tensor_path ? reduce(net, p, 2, 3, st) : r;
            },
            ms[3]);
    cudaEventDestroy(e[0]);
    cudaEventDestroy(e[1]);
    cudaMemcpyAsync(net->w, keep, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(net->m1, keep + kParams, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(net->m2, keep + 2 * kParams, sizeof(float) * kParams, cudaMemcpyDeviceToDevice, st);
    net->step = step0;
    const dmtz_status sp = pack(net, st);
    NCK(cudaStreamSynchronize(st));
    cudaFree(keep);
    return s != DMTZ_OK ? s : sp;
}
