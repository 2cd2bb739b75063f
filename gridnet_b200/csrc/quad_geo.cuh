// Geometry and building blocks shared by the quad kernels (step_quad.cu, step_quad_bwd.cu, step_quad_gated.cu): how the 32 lanes of a warp split an 8^3
// region of the grid, where a lane's window lies in the tile, the order of the weights in tensor memory, and the
// 27-tap sum itself.
#pragma once
#include "packed.cuh"
#include "tmem.cuh"

namespace gn {

namespace quad {
constexpr int QUARTERS = 4;
constexpr unsigned kSpinLimit = 1u << 20;
// columns of tensor memory: 36 uses of 12 weights, then 16 biases, 16 scales, 16 weight sums (per-block normalisation)
constexpr int COL_BIAS = 432, COL_SCALE = 448, COL_WSUM = 464;
// what the 27-tap sums start from: what is there, or minus the tile's mean times the weight sum
enum Mode { ADD, NORMED };
}  // namespace quad

// A region's tile buffer, in cells of 16 bytes (four samples).
template <int SUB>
struct QuadGeo;

// TEAM: warps per quarter of tensor memory; NBUF: tile buffers per team of step_quad.cu. Block 8: the region is one block, its tile
// 10 x 10 x 10 cells.
template <>
struct QuadGeo<8> {
    static constexpr int SIDE = 10, ROW = 10, PLANE = 100, CELLS = 1000, BUF_BYTES = 16000, TEAM = 2, NBUF = 2;
    __device__ static void cell(int c, int &cz, int &cy, int &cx)
    {
        cx = c % 10, cy = (c / 10) % 10, cz = c / 100;
    }
};

// Block 4: eight blocks, each with its own 6^3 tile
template <>
struct QuadGeo<4> {
    static constexpr int SIDE = 6, ROW = 6, PLANE = 36, SUBCELLS = 216, CELLS = 8 * SUBCELLS, BUF_BYTES = CELLS * 16, TEAM = 2, NBUF = 2;
    __device__ static void cell(int c, int &cz, int &cy, int &cx)
    {
        const int sub = c / SUBCELLS, l = c % SUBCELLS;
        cx = (sub & 1) * 4 + l % 6, cy = ((sub >> 1) & 1) * 4 + (l / 6) % 6, cz = (sub >> 2) * 4 + l / 36;
    }
};

// What a lane owns: the 2 x 2 x 4 patch at z = z0 + dz, y = y0 + ysgn * dy, x = 4 h + (h ? 3 - o : o) of the region,
// and the tile cell of its window's corner, from which the window extends by + PLANE per z, ysgn * ROW per y and
// xsgn per x. The upper x half and the upper y half walk inwards from the far end: with dense rows of 10 (or 6)
// cells the 8 lanes of a quarter-warp then hit 8 different 16-byte banks in every load and store of a cell.
template <int SUB>
struct QuadLane {
    int h, z0, y0, ysgn, xsgn, cell0;
    __device__ __forceinline__ explicit QuadLane(int lane)
    {
        using G = QuadGeo<SUB>;
        h = lane & 1;
        const int yp = (lane >> 1) & 3, zp = lane >> 3, my = yp >> 1, e = yp & 1;
        z0 = 2 * zp;
        xsgn = h ? -1 : 1;
        y0 = my ? 7 - 2 * e : 2 * e;
        ysgn = my ? -1 : 1;
        const int row = my ? G::SIDE - 1 - 2 * e : 2 * e, col = h ? G::SIDE - 1 : 0;
        if (SUB == 8) cell0 = 2 * zp * G::PLANE + row * G::ROW + col;
        else cell0 = (((zp >> 1) * 2 + my) * 2 + h) * 216 + 2 * (zp & 1) * G::PLANE + row * G::ROW + col;
    }
};

__device__ __forceinline__ float4 lds128(unsigned a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts128(unsigned a, float4 v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void sts128u(unsigned a, u64 lo, u64 hi)
{
    asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(a), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ void lds128u(unsigned a, u64 &lo, u64 &hi)
{
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "r"(a));
}
__device__ __forceinline__ void stg128(float *p, u64 lo, u64 hi)
{
    asm volatile("st.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ void st_release_shared(unsigned a, int v)
{
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_shared(unsigned a)
{
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// 16 bytes to shared memory, asynchronously
__device__ __forceinline__ void cp_async16(unsigned dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// ---- a lane's 16 cells in an IL4 tensor. base: its first cell row (dz = dy = 0) at x = 4 h, the lower end of its x half;
// zstr, ystr: floats to the next row in z and (signed) in y. 32 bytes, a whole sector, per access: cells one by one, the
// two halves of a sector go to memory separately.
__device__ __forceinline__ void stg256(float *p, u64 a, u64 b, u64 c, u64 d)
{
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}
__device__ __forceinline__ void ldg256(const float *p, u64 &a, u64 &b, u64 &c, u64 &d)
{
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p) : "memory");
}
// two x-neighbours (o = 2 j, 2 j + 1) of neuron row n
__device__ __forceinline__ void quad_store2(float *base, int n, int j, long long zstr, long long ystr, int h, const u64 (&v)[4][2])
{
    float *p = base + (n >> 1) * zstr + (n & 1) * ystr + 8 * (j ^ h);
    const u64 *lo = v[2 * j], *hi = v[2 * j + 1];
    stg256(p, h ? hi[0] : lo[0], h ? hi[1] : lo[1], h ? lo[0] : hi[0], h ? lo[1] : hi[1]);
}
__device__ __forceinline__ void quad_store(float *base, long long zstr, long long ystr, int h, const u64 (&v)[4][4][2])
{
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) quad_store2(base, n, j, zstr, ystr, h, v[n]);
}
__device__ __forceinline__ void quad_load2(const float *base, int n, int j, long long zstr, long long ystr, int h, u64 (&v)[4][2])
{
    u64 a, b, c, d;
    ldg256(base + (n >> 1) * zstr + (n & 1) * ystr + 8 * (j ^ h), a, b, c, d);
    v[2 * j][0] = h ? c : a;
    v[2 * j][1] = h ? d : b;
    v[2 * j + 1][0] = h ? a : c;
    v[2 * j + 1][1] = h ? b : d;
}
__device__ __forceinline__ void quad_load(const float *base, long long zstr, long long ystr, int h, u64 (&v)[4][4][2])
{
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) quad_load2(base, n, j, zstr, ystr, h, v[n]);
}
// ---- a region's 512 cells, staged in shared memory by whole lines: cell (z, y, x) at unit (8 z + y) 8 + (x ^ (y >> 1)) of 16
// bytes. The swizzle keeps both the copies (8 lanes to a row) and the reads of a lane's own cells free of bank conflicts.
// src: the region's first cell; cells of planes z0 .. z0 + nz - 1, 4 rows per instruction.
template <int Z0, int NZ>
__device__ __forceinline__ void quad_stage(unsigned stage, const float *src, long long zstr, int K, int lane)
{
    const int y = lane >> 3, x = lane & 7;
    const float *s = src + ((long long)y * K + x) * 4 + Z0 * zstr;
#pragma unroll
    for (int k = 2 * Z0; k < 2 * (Z0 + NZ); ++k) {
        const int yy = y + 4 * (k & 1);
        cp_async16(stage + (unsigned)(((k >> 1) * 8 + yy) * 8 + (x ^ (yy >> 1))) * 16u, s + (k & 1) * 16ll * K + ((k >> 1) - Z0) * zstr);
    }
}
// offset of a lane's own cell (n = (dz, dy), o) in such a staging area: row(n) + ((o ^ e) * 16)
template <int SUB>
struct QuadStage {
    unsigned row0, e;
    int ys;
    __device__ __forceinline__ explicit QuadStage(const QuadLane<SUB> &L)
    {
        row0 = (unsigned)(L.z0 * 8 + L.y0) * 128u;
        e = (L.h ? 7u : 0u) ^ (unsigned)(L.y0 >> 1);
        ys = L.ysgn * 128;
    }
    __device__ __forceinline__ unsigned at(int n, int o) const { return row0 + (n >> 1) * 1024u + (unsigned)((n & 1) * ys) + (((unsigned)o ^ e) << 4); }
};

// the warps of a team
template <int TEAM>
__device__ __forceinline__ void team_sync(int quarter)
{
    asm volatile("bar.sync %0, %1;" ::"r"(quarter + 1), "n"(32 * TEAM) : "memory");
}

// Items (regions x quads) are split over the quarters of ctas CTAs in whole multiples of this: two where that leaves the longest quarter
// no longer. A region that a quarter has an odd number of quads of ends with a warp on its own, at 3100 cycles an iteration instead of
// 2820 each for two, so pairs that never straddle a change of region gain where the longest quarter has an even number of items
// (64^3 x 64: 14). Where it has an odd number, pairs make it one item longer, and where there are no more items than quarters they leave
// half of these without work. us of a training loop of 2 x 8 iterations, one by one / in pairs: 32^3 x 8 348 / 386, x 64 718 / 648,
// 64^3 x 16 1316 / 1236, x 64 3668 / 3619; of inference, 4 x 8: 32^3 x 32 141 / 173, x 64 222 / 193, x 96 271 / 309, 64^3 x 32 588 / 629.
inline int quad_split_unit(long long nitems, long long ctas, int Q)
{
    const long long quarters = ctas * quad::QUARTERS, longest = (nitems + quarters - 1) / quarters;
    return Q % 2 == 0 && longest % 2 == 0 ? 2 : 1;
}

// Parameters of a region, packed in the order quad_stencil uses them (quad_pack; tap_stencil: tap_pack): 116 vectors of four words per
// lane, lane-contiguous (512 bytes per vector and warp).
namespace quad {
constexpr int VECS = 116, PACK_F = VECS * 128;  // floats per region
}
template <int N>
__device__ __forceinline__ void quad_fetch(const float4 *src, float (&r)[4 * N])
{
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float4 v = src[k * 32];  // not __ldg: the kernel before may be writing it still
        r[4 * k + 0] = v.x, r[4 * k + 1] = v.y, r[4 * k + 2] = v.z, r[4 * k + 3] = v.w;
    }
}
template <int N>
__device__ __forceinline__ void quad_put(unsigned col, const float (&r)[4 * N])
{
    int k = 0;
#pragma unroll
    for (; k + 4 <= N; k += 4) tmem_st16(col + 4 * k, r + 4 * k);
    if (N & 2) {
        tmem_st8(col + 4 * k, r + 4 * k);
        k += 2;
    }
    if (N & 1) tmem_st4(col + 4 * k, r + 4 * k);
}
// -> tensor memory, by the two warps of a quarter, each its half of the vectors in two goes: the loads of the first, then
// between(), after which the region before may be overwritten, then the rest.
template <typename Between>
__device__ __forceinline__ void quad_load_params(const float *packed, int role, int lane, unsigned tm, Between between)
{
    constexpr int N = quad::VECS / 4;
    const float4 *src = reinterpret_cast<const float4 *>(packed) + role * (2 * N) * 32 + lane;
    tm += role * (8 * N);
    float r[4 * N];
    quad_fetch<N>(src, r);
    between();
    quad_put<N>(tm, r);
    quad_fetch<N>(src + N * 32, r);
    quad_put<N>(tm + 4 * N, r);
}
__device__ __forceinline__ void quad_load_params(const float *packed, int role, int lane, unsigned tm)
{
    quad_load_params(packed, role, lane, tm, [] {});
}

// the weight sums of per-block normalisation (quad_wsum), by one warp of the team
__device__ __forceinline__ void quad_load_wsum(const float *wsum, int region, int lane, unsigned tm)
{
    const float4 *src = reinterpret_cast<const float4 *>(wsum) + (size_t)region * 128 + lane;
    float r[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 v = src[k * 32];  // not __ldg: the kernel before may be writing it still
        r[4 * k + 0] = v.x, r[4 * k + 1] = v.y, r[4 * k + 2] = v.z, r[4 * k + 3] = v.w;
    }
    tmem_st16(tm + quad::COL_WSUM, r);
}

// The 27-tap sums of the lane's 16 neurons for four samples, acc[n = (dz, dy)][o][sample pair] += sum.
//   NORMED: acc starts at negm (minus the mean of the tile) times the sum of the neuron's weights, and done(n, o, scale, bias,
//   centre), which adds the bias, is called when a sum is complete - for the neurons of dy = 0 between the FMAs of the last
//   window rows, so that their activation functions (MUFU) run under them. ADD: acc is added to, and done is not called.
//   rows[ry]: where window row ry of plane 0, column 0 starts; PLANE: cells from one plane to the next; dx: bytes from
//   one column to the next.
template <int PLANE, quad::Mode MODE, typename Done>
__device__ __forceinline__ void quad_stencil(const unsigned (&rows)[4], int dx, unsigned tm, u64 (&acc)[4][4][2], const u64 (&negm)[2],
                                             Done done)
{
    constexpr bool NORMED = MODE == quad::NORMED;
    float wb[2][12], sc[2][4], bi[2][4];
    auto finish = [&](int n, int o, float s, float b) {
        u64 c0, c1;
        lds128u(rows[1 + (n & 1)] + (unsigned)((1 + o) * dx) + (1 + (n >> 1)) * PLANE * 16u, c0, c1);
        done(n, o, s, b, c0, c1);
    };
    if (NORMED) {
        float first[16];
        tmem_ld16(tm + quad::COL_WSUM, first);
        tmem_wait_ld16(first);
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const u64 f2 = pack2(first[n * 4 + o], first[n * 4 + o]);
#pragma unroll
                for (int k = 0; k < 2; ++k) acc[n][o][k] = fmul2(f2, negm[k]);
            }
    }
    tmem_ld8(tm, wb[0]);
    tmem_ld4(tm + 8, wb[0] + 8);
    int use = 0, fin = 0;
#pragma unroll
    for (int ry = 0; ry < 4; ++ry) {
        unsigned a6[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) a6[j] = rows[ry] + (unsigned)(j * dx);
#pragma unroll
        for (int rz = 0; rz < 4; ++rz) {
            u64 v[6][2];
#pragma unroll
            for (int j = 0; j < 6; ++j) lds128u(a6[j] + rz * PLANE * 16u, v[j][0], v[j][1]);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int a = rz - (n >> 1), b = ry - (n & 1);
                if (a < 0 || a > 2 || b < 0 || b > 2) continue;
                float *wp = wb[use & 1];
                tmem_wait_ld12(wp);
                if (NORMED && use == 30) {  // asked for before: that wait covered it
                    tmem_use8(sc[0]);
                    tmem_use8(bi[0]);
                }
                if (use + 1 < 36) {
                    tmem_ld8(tm + (use + 1) * 12, wb[(use & 1) ^ 1]);
                    tmem_ld4(tm + (use + 1) * 12 + 8, wb[(use & 1) ^ 1] + 8);
                }
                if (NORMED && use == 29) {
                    tmem_ld4(tm + quad::COL_SCALE, sc[0]);
                    tmem_ld4(tm + quad::COL_SCALE + 8, sc[1]);
                    tmem_ld4(tm + quad::COL_BIAS, bi[0]);
                    tmem_ld4(tm + quad::COL_BIAS + 8, bi[1]);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        const u64 ww = pack2(wp[c * 4 + o], wp[c * 4 + o]);
                        ffma2(acc[n][o][0], v[o + c][0], ww);
                        ffma2(acc[n][o][1], v[o + c][1], ww);
                    }
                ++use;
                if (NORMED && ry == 3)
#pragma unroll
                    for (int e = (use - 30) * 8 / 6; fin < e; ++fin)
                        finish((fin >> 2) * 2, fin & 3, sc[fin >> 2][fin & 3], bi[fin >> 2][fin & 3]);
            }
        }
    }
    if (NORMED) {
        tmem_ld4(tm + quad::COL_SCALE + 4, sc[0]);
        tmem_ld4(tm + quad::COL_SCALE + 12, sc[1]);
        tmem_ld4(tm + quad::COL_BIAS + 4, bi[0]);
        tmem_ld4(tm + quad::COL_BIAS + 12, bi[1]);
        tmem_wait_ld8(sc[0]);
        tmem_use8(bi[0]);
#pragma unroll
        for (int e = 0; e < 8; ++e) finish((e >> 2) * 2 + 1, e & 3, sc[e >> 2][e & 3], bi[e >> 2][e & 3]);
    }
}

// Adds eight values over the warp; afterwards lanes 4 j .. 4 j + 3 all hold the sum of value j.
template <typename T>
__device__ __forceinline__ T quad_reduce8(const T (&v)[8], int lane)
{
    T a[4], b[2], c;
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = (h16 ? v[k + 4] : v[k]) + __shfl_xor_sync(0xffffffffu, h16 ? v[k] : v[k + 4], 16);
#pragma unroll
    for (int k = 0; k < 2; ++k) b[k] = (h8 ? a[k + 2] : a[k]) + __shfl_xor_sync(0xffffffffu, h8 ? a[k] : a[k + 2], 8);
    c = (h4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h4 ? b[0] : b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;
}

// Adds eight values over the lanes that share a tile (block 8: the warp, block 4: the four lanes of a sub-block); every
// lane gets all eight sums. T: what the lanes' values are added in.
template <int SUB, typename T = float>
__device__ __forceinline__ void quad_tile_sum8(float (&f)[8], int lane)
{
    T v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = (T)f[k];
    if (SUB == 8) {
        const float r = (float)quad_reduce8(v, lane);
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = __shfl_sync(0xffffffffu, r, 4 * k);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], 8);
            f[k] = (float)v[k];
        }
    }
}
// The tile of a lane among all blocks of the grid (block 8: the region, block 4: eight per region), and the lane that
// writes what the lanes of a tile have in common.
template <int SUB>
__device__ __forceinline__ int quad_tile_of(const QuadLane<SUB> &L, int region)
{
    return SUB == 8 ? region : region * 8 + ((L.z0 >> 2) * 2 + (L.y0 >> 2)) * 2 + L.h;
}
template <int SUB>
__device__ __forceinline__ bool quad_tile_leader(int lane) { return SUB == 8 ? lane == 0 : (lane & 10) == 0; }
// Per-block normalisation keeps, for every iteration, quad and tile, four vectors over the quad's samples
enum QuadStat { QS_MEAN, QS_INV /* 1 / (std + eps) */, QS_STD, QS_STDEPS, QS_COUNT };

}  // namespace gn
