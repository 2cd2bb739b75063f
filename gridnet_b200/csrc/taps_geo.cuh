// Geometry and building blocks of the kernel that adds a neuron's taps in the order of their numbers (step_taps.cu): how the
// 32 lanes of a warp split an 8^3 region, where the cells lie in the tile, and the 27-tap sum.
#pragma once
#include "quad_geo.cuh"

namespace gn {

// A lane owns the 4 x 1 x 4 patch z = 4 zp .. 4 zp + 3, x = 4 h .. 4 h + 3 of row y. Its window is 6 x 3 x 6 cells, 108 for 16
// neurons (the 2 x 2 x 4 patches of quad_geo.cuh have 96), but nothing is mirrored: every neuron meets its taps in
// ascending order, all cells of the window lie at fixed distances from its corner, and one register addresses them. The
// eight lanes of a quarter-warp are eight rows; the layouts put these on eight different 16-byte banks.
struct TapLane {
    int y, h, zp;
    __device__ __forceinline__ explicit TapLane(int lane) : y(lane & 7), h((lane >> 3) & 1), zp(lane >> 4) {}
};

template <int SUB>
struct TapGeo;

// TEAM: warps per quarter of tensor memory; NBUF: tile buffers per team. A third buffer fits but leaves nothing of the SM's memory
// for the first-level cache (64^3 x 64, 4 x 12: 1616 us with three, 1553 with two).
// Block 8: rows of 11 cells, the last one beyond the tile (11 y mod 8 takes eight values), fetched by bulk tensor copy. A third
// warp, with 168 registers, brought nothing: two keep the FMA pipe as busy as its operands allow (64^3 x 64, 4 x 12: 1667 us).
template <>
struct TapGeo<8> {
    static constexpr int ROW = 11, PLANE = 110, CELLS = 1100, BUF_BYTES = 17664, TEAM = 2, NBUF = 2;
    __device__ static int corner(const TapLane &L) { return 4 * L.zp * PLANE + L.y * ROW + 4 * L.h; }
};

// Block 4: eight 6^3 tiles in the order (z, x, y), 217 cells from one to the next: rows differ by 6 y mod 8 (0, 6, 4, 2) and
// the two tiles along y by 1. Bulk tensor copies go to multiples of 8 cells only, so these are fetched cell by cell.
template <>
struct TapGeo<4> {
    static constexpr int ROW = 6, PLANE = 36, TILE = 217, BUF_BYTES = 8 * TILE * 16, TEAM = 2, NBUF = 2;
    __device__ static int corner(const TapLane &L) { return ((L.zp * 2 + L.h) * 2 + (L.y >> 2)) * TILE + (L.y & 3) * ROW; }
};

// The 27-tap sums of the lane's 16 neurons for four samples, acc[dz][o][sample pair]: the bias, then taps 0 .. 26 one after the
// other, as the register-patch kernels do it (step_fast.cu), which makes the sums the same bits. win: the window's corner.
// done(n, o, scale, centre) is called when neuron (n, o) has its sum, between the FMAs of the planes that follow, so that the
// activation functions (MUFU) run under them.
template <int SUB, typename Done>
__device__ __forceinline__ void tap_stencil(unsigned win, unsigned tm, u64 (&acc)[4][4][2], const u64 (&own)[4][4][2], Done done)
{
    using G = TapGeo<SUB>;
    float wb[2][12], sc[2][4];
    {
        float first[16];
        tmem_ld16(tm + quad::COL_BIAS, first);
        tmem_wait_ld16(first);
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int o = 0; o < 4; ++o) acc[n][o][0] = acc[n][o][1] = pack2(first[n * 4 + o], first[n * 4 + o]);
    }
    tmem_ld8(tm, wb[0]);
    tmem_ld4(tm + 8, wb[0] + 8);
    int use = 0;
#pragma unroll
    for (int rz = 0; rz < 6; ++rz) {
        int at = 0, fin = 0;  // uses of this plane, neurons of plane rz - 3 that are finished
        const int uses = 3 * (rz < 3 ? rz + 1 : 6 - rz);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            u64 v[6][2];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                if (b == 1 && rz >= 1 && rz <= 4 && j >= 1 && j <= 4) v[j][0] = own[rz - 1][j - 1][0], v[j][1] = own[rz - 1][j - 1][1];
                else lds128u(win + (unsigned)(rz * G::PLANE + b * G::ROW + j) * 16u, v[j][0], v[j][1]);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int a = rz - n;
                if (a < 0 || a > 2) continue;
                float *wp = wb[use & 1];
                tmem_wait_ld12(wp);
                if (rz >= 3 && at == 0) tmem_use4(sc[rz & 1]);  // asked for before: that wait covered it
                if (use + 1 < 36) {
                    tmem_ld8(tm + (use + 1) * 12, wb[(use & 1) ^ 1]);
                    tmem_ld4(tm + (use + 1) * 12 + 8, wb[(use & 1) ^ 1] + 8);
                }
                ++use, ++at;
                if (rz >= 2 && at == uses) tmem_ld4(tm + quad::COL_SCALE + (rz - 2) * 4, sc[(rz + 1) & 1]);
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        const u64 ww = pack2(wp[c * 4 + o], wp[c * 4 + o]);
                        ffma2(acc[n][o][0], v[o + c][0], ww);
                        ffma2(acc[n][o][1], v[o + c][1], ww);
                    }
                if (rz >= 3)
#pragma unroll
                    for (int e = 4 * at / uses; fin < e; ++fin) done(rz - 3, fin, sc[rz & 1][fin]);
            }
        }
    }
    tmem_wait_ld4(sc[0]);
#pragma unroll
    for (int o = 0; o < 4; ++o) done(3, o, sc[0][o]);
}

// The sum (j = 0) and the sum of squares (j = 1) of a region's values for the quad's samples s = 0 .. 3: on return lanes with
// l = lane & 15 hold value j = l & 1 of sample s = (l >> 1 & 1) * 2 + (l >> 3). As in step_fast.cu the 128 values of two
// planes are added in float, in that kernel's order (2 x 2 in y and x, then over z, y and x), and the four pairs of planes
// in double: the statistics of a step are the same whichever kernel ran it.
__device__ __forceinline__ double tap_region_sums(const u64 (&v)[4][4][2], int lane)
{
    const bool y0 = lane & 1, y1 = lane & 2, y2 = lane & 4, h = lane & 8;
    // [dz][x pair][sample]: sums in the lanes of even rows, squares in those of odd rows
    float a[4][2][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const u64 lo = v[n][2 * p][k], hi = v[n][2 * p + 1][k];
                float s[2], q[2];
                unpack2(fadd2(lo, hi), s[0], s[1]);
                unpack2(ffma2r(lo, lo, fmul2(hi, hi)), q[0], q[1]);
#pragma unroll
                for (int i = 0; i < 2; ++i) a[n][p][2 * k + i] = (y0 ? q[i] : s[i]) + __shfl_xor_sync(0xffffffffu, y0 ? s[i] : q[i], 1);
            }
    float b[2][4], c[2][2], d[2];  // [x pair][sample]
#pragma unroll
    for (int p = 0; p < 2; ++p) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // planes 0 and 1, 2 and 3; then rows four apart, after which a lane has one pair of planes
            const float z0 = a[0][p][i] + a[1][p][i], z1 = a[2][p][i] + a[3][p][i];
            b[p][i] = (y2 ? z1 : z0) + __shfl_xor_sync(0xffffffffu, y2 ? z0 : z1, 4);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) c[p][i] = (y1 ? b[p][i + 2] : b[p][i]) + __shfl_xor_sync(0xffffffffu, y1 ? b[p][i] : b[p][i + 2], 2);
        d[p] = (h ? c[p][1] : c[p][0]) + __shfl_xor_sync(0xffffffffu, h ? c[p][0] : c[p][1], 8);
    }
    double r = (double)(d[0] + d[1]);
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    r += __shfl_xor_sync(0xffffffffu, r, 16);
    return r;
}

}  // namespace gn
