// The three stages of gradient.cuh on the host, over a whole grid at once:
// reads "W H D" and W*H*D doubles from argv[1], writes pv (u8), eup, fup, crit,
// tcode (u32) of every anchor to argv[2].
#include <cstdio>
#include <vector>

#include "../../dmtz_gb300/csrc/gradient.cuh"

using namespace dmtz;

constexpr int ROW = 64;  // row length of every padded array; grids up to 60 wide

int main(int argc, char **argv) {
    int d[3];
    FILE *in = argc > 2 ? fopen(argv[1], "rb") : nullptr;
    if (!in || fread(d, 4, 3, in) != 3 || d[0] + 4 > ROW) return 2;
    const int W = d[0], H = d[1], D = d[2];
    std::vector<double> f((size_t)W * H * D);
    if (fread(f.data(), 8, f.size(), in) != f.size()) return 2;
    const int PL = ROW * (H + 4);
    auto at = [&](int x, int y, int z) { return (x + 2) + ROW * (y + 2) + PL * (z + 2); };
    const size_t n = (size_t)PL * (D + 4);
    std::vector<uint64_t> key(n, kKeyAbsent);
    std::vector<uint4> w(n);
    std::vector<uint32_t> w4(n);
    std::vector<CellWords> c(n);
    for (int z = 0; z < D; z++)
        for (int y = 0; y < H; y++)
            for (int x = 0; x < W; x++) key[at(x, y, z)] = okey(f[x + (size_t)W * (y + (size_t)H * z)]);
    std::vector<uint8_t> pv(f.size());
    std::vector<uint32_t> out[4];
    for (auto &o : out) o.resize(f.size());
    for (int z = -1; z <= D; z++)
        for (int y = -1; y <= H; y++)
            for (int x = -1; x <= W; x++) {
                const uint64_t *k = key.data() + at(x, y, z);
                const StarWords s = grad_stage1<ROW>(k - PL, k, k + PL);
                w[at(x, y, z)] = make_uint4(s.x, s.y, s.z, s.w);
                w4[at(x, y, z)] = s.w4;
                if (x >= 0 && y >= 0 && z >= 0 && x < W && y < H && z < D) pv[x + (size_t)W * (y + (size_t)H * z)] = (uint8_t)s.pv;
            }
    for (int z = -1; z < D; z++)
        for (int y = -1; y < H; y++)
            for (int x = -1; x < W; x++) {
                const int i = at(x, y, z);
                c[i] = grad_stage2<ROW>(&w[i], &w[i + PL], &w4[i], &w4[i + PL]);
            }
    for (int z = 0; z < D; z++)
        for (int y = 0; y < H; y++)
            for (int x = 0; x < W; x++) {
                const int i = at(x, y, z);
                const AnchorOut o = grad_stage3<ROW>(&c[i - PL], &c[i], (x == W - 1) | (y == H - 1) << 1 | (z == D - 1) << 2);
                const size_t v = x + (size_t)W * (y + (size_t)H * z);
                out[0][v] = o.eup; out[1][v] = o.fup; out[2][v] = o.crit; out[3][v] = o.tcode;
            }
    FILE *of = fopen(argv[2], "wb");
    if (!of) return 2;
    fwrite(pv.data(), 1, pv.size(), of);
    for (auto &o : out) fwrite(o.data(), 4, o.size(), of);
    return fclose(of);
}
