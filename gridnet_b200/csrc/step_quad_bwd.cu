// Backward of the block-local update with the quad mapping (float, block 8 and 4, with and without per-block normalisation): the
// decomposition of step_bwd_fast.cu on the layout and the work split of step_quad.cu.
//
//   reverse  quad_reverse_k: walks the inner iterations backwards. delta_t = act'(h_t) g s; what flows back inside a block
//            is the 27-tap sum over the delta tile with transposed weights, read from tensor memory. The gradient of the
//            whole-grid normalisation that follows the step is applied to g on the way in, so the normalised gradient
//            never exists in memory.
//   wgrad    quad_wgrad_k: dW[n][t] += x_t[n + o_t] delta_t[n], accumulated in registers over quads and iterations. Chunks of
//            the batch leave their sums in parts of their own, which quad_finish_k adds up in chunk order: no
//            atomics, the same bits every time.
//   border   quad_border_k: the part of grad_x that crosses block borders, from the per-neuron sums of deltas.
//   norms    quad_norm_sums_k: one pass over the step's output and the gradient of its normalised form gives the
//            per-sample sums of the LayerNorm gradient and the gradients of its weight and bias.
//
// Reference semantics: the gradient of gridnet/backend_torch.py:61-142 and of
// torch.nn.LayerNorm((M,N,K)) (gridnet/scripts/train_mnist.py:54,62-64); the kernel this stands in for is
// gridnet_cuda_backward_kernel, src/gridnet_cuda_kernels.cu:202-450.
#include <cooperative_groups.h>
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "quad_geo.cuh"
#include "tmem.cuh"

namespace gn {

// ------------------------------------------------------------------------------------------- reverse sweep
namespace quadrev {
// delta tile of a region: 10 planes of 8 rows of 10 cells. The outer planes and columns are zero; rows beyond the region
// are read as the nearest row and meet zero weights.
// Before an item, the gradient of its output is fetched into the tile's own cells; pre-activations arrive in a staging area,
// with per-block normalisation the activations in a second one and the iteration's statistics behind it. The tiles of
// neighbouring warps share a zero plane, without which that would not fit.
constexpr int ROW = 10, PLANE = 80, CELLS = 800, TILE_BYTES = 9 * PLANE * 16, STAGE_BYTES = 512 * 16, TEAM = 2, WARPS = 4 * TEAM;
constexpr int TILES_BYTES = WARPS * TILE_BYTES + PLANE * 16;
constexpr int STATS_BYTES = 8 * QS_COUNT * 16;  // block 4: eight tiles
enum In { PLAIN, GRID_NORM /* the output went through a whole-grid norm */, BLOCK_NORM /* the sums' inputs were normalised per block */ };
template <In IN>
struct Bytes {
    static constexpr int STAGE = IN == BLOCK_NORM ? 2 * STAGE_BYTES + STATS_BYTES : STAGE_BYTES, SMEM = TILES_BYTES + WARPS * STAGE;
    static_assert(SMEM <= 232448 - 1024, "shared memory of one SM");
};
}  // namespace quadrev

struct QuadRevParams {
    const float *packed;           // transposed weights; GRID_NORM: the norm's weight in the place of the biases
    const float *g;                // gradient of the step's output (GRID_NORM: of its normalised output), IL4
    const float *raw;              // GRID_NORM, BLOCK_NORM: the step's output, IL4
    const float2 *stats, *ac;      // GRID_NORM: [4 Q] (mean, rstd) and (sum g gamma, sum g gamma xhat) / P
    const float *wsum;             // BLOCK_NORM: as in step_fwd_quad
    const float4 *tile_stats;      // BLOCK_NORM: [inner][Q][tiles][QS_COUNT]
    float4 *hterm;                 // BLOCK_NORM: [Q][tiles][2] F, E
    const float *h;                // [inner] pre-activations, IL4
    float *delta, *dsum, *gx;      // [inner], one, one IL4 tensors
    float *dsq;                    // [Q][P] gradient terms of the residual scale, summed over the quad and the iterations
    int M, N, K, Q, inner;
    int params_old;                // the kernel before this one did not write packed (or wsum)
    int unit;                      // quad_split_unit
    long long nitems;
};

// BLOCK_NORM: the input of iteration t's sums was (tile - mean) inv with inv = 1 / (std + eps). With Gin the gradient of that
// input, a tile cell's gradient is inv Gin - P1 - P2 (x - mean), P1 = inv sum(Gin) / cells, P2 = inv sum(Gin in) /
// (cells std), and both sums are sums over the block's neurons: sum(Gin) = sum raw W (W the neuron's weights added up), sum(Gin
// in) = sum raw (h - bias), raw the delta before it is scaled by inv. The deltas that are stored and summed are the scaled
// ones, so the other kernels see inv Gin. The lanes that share a tile add the two sums up by shuffles; what the halo
// cells owe, F + E x with F = sum_t (P1 - P2 mean), E = sum_t P2, goes (negated) to the border kernel. The activations x_t are
// walked back from the step's output, x_t = x_(t+1) - scale act(h_t).
// What bounds it: latency. Of 42 k cycles that an item of two iterations takes at 128^3 x 32 the transposed sums are 13 k, deltas 8.5 k, its
// first loads 8.8 k (asked for to L2 a stencil ahead; a staging area of their own would take the first-level cache's room and was
// slower), its stores 4.7 k. Warps take the next item when they are free; a region's first half of parameters is loaded ahead of the barrier,
// the first region's while the kernel before still runs: 626 -> 571 us.
template <int SUB, int ACT, quadrev::In IN>
__global__ void __launch_bounds__(256, 1) quad_reverse_k(const QuadRevParams p)
{
    using namespace quad;
    using namespace quadrev;
    constexpr bool NORM_IN = IN == GRID_NORM, BN = IN == BLOCK_NORM;
    constexpr float PER_CELL = SUB == 8 ? 1.0f / 1000 : 1.0f / 216;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ unsigned tmem_slot;
    __shared__ int claimed[QUARTERS];  // items of the team that warps have taken
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid < QUARTERS) claimed[tid] = 0;
    const unsigned tile = smem_u32(smem) + warp * TILE_BYTES, stage = smem_u32(smem) + TILES_BYTES + warp * Bytes<IN>::STAGE;
    const unsigned stage_x = stage + STAGE_BYTES, stage_s = stage_x + STAGE_BYTES;  // BN
    for (int c = lane; c < CELLS; c += 32) sts128u(tile + c * 16, 0, 0);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<SUB> L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K, T4 = (size_t)p.Q * P * 4;  // floats of an IL4 tensor
    const long long worker = (long long)blockIdx.x * QUARTERS + quarter, nworkers = (long long)gridDim.x * QUARTERS;
    const unsigned n0 = (unsigned)(p.nitems / p.unit * worker / nworkers * p.unit);
    const int cnt = (int)(p.nitems / p.unit * (worker + 1) / nworkers * p.unit - n0);
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K;
    const long long zstr = wzs * 4, ystr = wys * 4;
    const int dx = L.xsgn * 16;
    const QuadStage<SUB> S(L);

    // this lane's window rows in the tile (plane 0, column 0)
    unsigned rows[4];
#pragma unroll
    for (int ry = 0; ry < 4; ++ry) {
        int y = L.y0 + L.ysgn * (ry - 1);
        y = y < 0 ? 0 : (y > 7 ? 7 : y);
        rows[ry] = tile + (unsigned)(L.z0 * PLANE + y * ROW + (L.h ? 9 : 0)) * 16u;
    }
    const unsigned mine = rows[1] + (unsigned)dx + PLANE * 16u;  // own cell (0, 0, 0)
    auto own_cell = [&](int n, int o) { return mine + (unsigned)((n & 1) * L.ysgn * ROW * 16 + o * dx) + (n >> 1) * PLANE * 16u; };
    // first cell of the region of the team's item i in an IL4 tensor
    auto corner_of = [&](int i) {
        const unsigned n = n0 + i, blk = n / (unsigned)p.Q, q = n - blk * p.Q;
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        return ((size_t)q * P + ((size_t)(bz * 8) * p.N + by * 8) * p.K + bx * 8) * 4;
    };
    const size_t ntiles = (size_t)nbx * nby * (p.M >> 3) * (SUB == 8 ? 1 : 8);
    // pre-activations of iteration t of the team's item i (BN: and the statistics of its tiles)
    auto fetch_h = [&](int i, size_t corner, int t) {
        quad_stage<0, 8>(stage, p.h + (size_t)t * T4 + corner, zstr, p.K, lane);
        if (BN) {
            const unsigned n = n0 + i, blk = n / (unsigned)p.Q, q = n - blk * p.Q;
            const float4 *src = p.tile_stats + (((size_t)t * p.Q + q) * ntiles + (size_t)blk * (SUB == 8 ? 1 : 8)) * QS_COUNT;
            if (lane < (SUB == 8 ? 1 : 8) * QS_COUNT) cp_async16(stage_s + lane * 16, src + lane);
        }
    };
    auto fetch_x = [&](size_t corner) { quad_stage<0, 8>(stage_x, p.raw + corner, zstr, p.K, lane); };
    auto fetch_g = [&](size_t corner) {
        const int y = lane >> 3, x = lane & 7;
        const float *src = p.g + corner + ((long long)y * p.K + x) * 4;
#pragma unroll
        for (int k = 0; k < 16; ++k)
            cp_async16(tile + (unsigned)(((k >> 1) + 1) * PLANE + (y + 4 * (k & 1)) * ROW + x + 1) * 16u, src + (k & 1) * 16ll * p.K + (k >> 1) * zstr);
    };
    // what an item starts with, 64 lines each, on its way to L2
    auto expect = [&](size_t corner) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const size_t row = corner + ((lane >> 3) + 4 * k) * zstr + (lane & 7) * 4ll * p.K;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.g + row));
            if (NORM_IN) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.raw + row));
        }
    };
    auto claim = [&]() {
        int i = 0;
        if (lane == 0) i = atomicAdd(&claimed[quarter], 1);
        return __shfl_sync(0xffffffffu, i, 0);
    };
    const size_t to_own = (((size_t)L.z0 * p.N + L.y0) * p.K + 4 * L.h) * 4;  // corner -> this lane's cells
    int i = claim();  // the item in work
    auto begin = [&]() {
        previous_done();
        __syncwarp();
        if (i < cnt) {
            fetch_g(corner_of(i));
            fetch_h(i, corner_of(i), p.inner - 1);
            if (BN) fetch_x(corner_of(i));
            if (NORM_IN) expect(corner_of(i));
        }
    };
    if (!p.params_old || cnt == 0) begin();  // else the first region's parameters come first

    int blk = (int)(n0 / (unsigned)p.Q), q0 = (int)(n0 - (unsigned)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);
        quad_load_params(p.packed + (size_t)blk * PACK_F, role, lane, tm, [&] {
            if (i0 > 0) {
                tmem_fence_before();
                team_sync<TEAM>(quarter);  // the other warp no longer reads the old region's weights
                tmem_fence_after();
            }
        });
        if (BN && role == 0) quad_load_wsum(p.wsum, blk, lane, tm);
        tmem_wait_st();
        if (i0 == 0 && p.params_old) begin();
        tmem_fence_before();
        team_sync<TEAM>(quarter);
        tmem_fence_after();
        if (i0 + here < cnt) {
            const unsigned char *nx = reinterpret_cast<const unsigned char *>(p.packed + (size_t)(blk + 1) * PACK_F);
            for (int c = role * 32 + lane; c < PACK_F * 4 / 128; c += 32 * TEAM) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c * 128));
            __syncwarp();
        }
        const unsigned my_stats = stage_s + (SUB == 8 ? 0 : (unsigned)quad_tile_of(L, 0)) * (QS_COUNT * 16);
        for (int next = 0; i < i0 + here; i = next) {
            const int q = q0 + i - i0;
            const size_t corner = corner_of(i), own = corner + to_own;
            u64 g[4][4][2], dsum[4][4][2];
            float dsa[4][4];
            {
                // everything the item starts with is asked for at once
                u64 r[4][4][2];
                float2 m4[4], a4[4];
                float gm[16];
                if (NORM_IN) {
                    quad_load(p.raw + own, zstr, ystr, L.h, r);
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        m4[s] = p.stats[4 * q + s];
                        a4[s] = p.ac[4 * q + s];
                    }
                    tmem_ld16(tm + COL_BIAS, gm);
                }
                cp_async_wait_all();
                if (NORM_IN) tmem_wait_ld16(gm);
                __syncwarp();
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o) lds128u(own_cell(n, o), g[n][o][0], g[n][o][1]);
                if (NORM_IN) {
                    // gradient of (x - mean) rstd gamma + beta: rstd (g gamma - a - xhat c)
#pragma unroll
                    for (int k2 = 0; k2 < 2; ++k2) {
                        const float2 m0 = m4[2 * k2], m1 = m4[2 * k2 + 1], a0 = a4[2 * k2], a1 = a4[2 * k2 + 1];
                        const u64 mu = pack2(-m0.x, -m1.x), rs = pack2(m0.y, m1.y), ma = pack2(-a0.x, -a1.x), mc = pack2(-a0.y, -a1.y);
#pragma unroll
                        for (int n = 0; n < 4; ++n)
#pragma unroll
                            for (int o = 0; o < 4; ++o) {
                                const u64 xh = fmul2(fadd2(r[n][o][k2], mu), rs);
                                const u64 gg = ffma2r(g[n][o][k2], pack2(gm[n * 4 + o], gm[n * 4 + o]), ma);
                                g[n][o][k2] = fmul2(ffma2r(xh, mc, gg), rs);
                            }
                    }
                }
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    dsum[n][o][0] = dsum[n][o][1] = 0;
                    dsa[n][o] = 0.0f;
                }
            u64 hf[2] = {0, 0}, he[2] = {0, 0};  // BN: F and E
            size_t ahead = 0;                    // corner of the next item
            for (int t = p.inner - 1; t >= 0; --t) {
                float sc[16];
                if (!BN) tmem_ld16(tm + COL_SCALE, sc);
                cp_async_wait_all();
                if (!BN) tmem_wait_ld16(sc);
                __syncwarp();  // everyone's part of h_t has landed
                u64 inv[2] = {0, 0}, pa[2] = {0, 0}, pc[2] = {0, 0};
                if (BN) lds128u(my_stats + QS_INV * 16, inv[0], inv[1]);
                // Row by row: loads, arithmetic and stores of a row of four cells each overlap with themselves (cell by cell,
                // a load waits for the store before it); more rows at a time spill (0.64 ms by one row, 0.67 by two, 0.71 by
                // four, at 128^3 with two inner iterations and batch 32).
                float *const dt = p.delta + (size_t)t * T4 + own;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    u64 h[4][2], x[4][2];
                    float bw[16];  // BN: bias and scale, weight sum
                    if (BN) {
                        tmem_ld4(tm + COL_BIAS + n * 4, bw);
                        tmem_ld4(tm + COL_SCALE + n * 4, bw + 4);
                        tmem_ld4(tm + COL_WSUM + n * 4, bw + 8);
                    }
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        lds128u(stage + S.at(n, o), h[o][0], h[o][1]);
                        if (BN) lds128u(stage_x + S.at(n, o), x[o][0], x[o][1]);
                    }
                    if (BN) {
                        tmem_wait_ld12(bw);
#pragma unroll
                        for (int o = 0; o < 4; ++o) sc[n * 4 + o] = bw[4 + o];
                    }
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        u64 f0, f1, d0, d1;
                        act_both2<ACT>(h[o][0], f0, d0);
                        act_both2<ACT>(h[o][1], f1, d1);
                        float s0, s1;
                        unpack2(ffma2r(f0, g[n][o][0], fmul2(f1, g[n][o][1])), s0, s1);
                        dsa[n][o] += s0 + s1;
                        const u64 s2 = pack2(sc[n * 4 + o], sc[n * 4 + o]);
                        if (BN) {
                            const u64 nb = pack2(-bw[o], -bw[o]), w2 = pack2(bw[8 + o], bw[8 + o]), ns = pack2(-sc[n * 4 + o], -sc[n * 4 + o]);
                            const u64 r0 = fmul2(fmul2(d0, g[n][o][0]), s2), r1 = fmul2(fmul2(d1, g[n][o][1]), s2);
                            ffma2(pa[0], r0, w2);
                            ffma2(pa[1], r1, w2);
                            ffma2(pc[0], r0, fadd2(h[o][0], nb));
                            ffma2(pc[1], r1, fadd2(h[o][1], nb));
                            ffma2(x[o][0], f0, ns);
                            ffma2(x[o][1], f1, ns);
                            sts128u(stage_x + S.at(n, o), x[o][0], x[o][1]);
                            h[o][0] = fmul2(r0, inv[0]);
                            h[o][1] = fmul2(r1, inv[1]);
                        } else {
                            h[o][0] = fmul2(fmul2(d0, g[n][o][0]), s2);
                            h[o][1] = fmul2(fmul2(d1, g[n][o][1]), s2);
                        }
                        dsum[n][o][0] = fadd2(dsum[n][o][0], h[o][0]);
                        dsum[n][o][1] = fadd2(dsum[n][o][1], h[o][1]);
                    }
#pragma unroll
                    for (int o = 0; o < 4; ++o) sts128u(own_cell(n, o), h[o][0], h[o][1]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) quad_store2(dt, n, j, zstr, ystr, L.h, h);
                }
                if (BN) {
                    u64 mean[2], sd[2];
                    lds128u(my_stats + QS_MEAN * 16, mean[0], mean[1]);
                    lds128u(my_stats + QS_STD * 16, sd[0], sd[1]);
                    float v[8];
                    unpack2(pa[0], v[0], v[1]);
                    unpack2(pa[1], v[2], v[3]);
                    unpack2(pc[0], v[4], v[5]);
                    unpack2(pc[1], v[6], v[7]);
                    quad_tile_sum8<SUB>(v, lane);
                    u64 np1[2], np2[2];  // -(P1 - P2 mean), -P2
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        float i0, i1, s0, s1;
                        unpack2(inv[j], i0, i1);
                        unpack2(sd[j], s0, s1);
                        // a constant tile has no deviation to divide by, and nothing is as far from its mean as to need it
                        const float e0 = s0 > 0.0f ? -v[4 + 2 * j] * i0 / (s0 * (1.0f / PER_CELL)) : 0.0f;
                        const float e1 = s1 > 0.0f ? -v[5 + 2 * j] * i1 / (s1 * (1.0f / PER_CELL)) : 0.0f;
                        np2[j] = pack2(e0, e1);
                        const u64 p1 = pack2(v[2 * j] * i0 * -PER_CELL, v[2 * j + 1] * i1 * -PER_CELL);
                        np1[j] = ffma2r(fmul2(np2[j], pack2(-1.0f, -1.0f)), mean[j], p1);
                        hf[j] = fadd2(hf[j], np1[j]);
                        he[j] = fadd2(he[j], np2[j]);
                    }
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        u64 x[4][2];
#pragma unroll
                        for (int o = 0; o < 4; ++o) lds128u(stage_x + S.at(n, o), x[o][0], x[o][1]);
#pragma unroll
                        for (int o = 0; o < 4; ++o)
#pragma unroll
                            for (int j = 0; j < 2; ++j) g[n][o][j] = fadd2(g[n][o][j], ffma2r(x[o][j], np2[j], np1[j]));
                    }
                }
                __syncwarp();  // the delta tile is complete, h_t has been read
                if (t > 0) {
                    fetch_h(i, corner, t - 1);
                } else {
                    next = claim();
                    if (next < cnt) {
                        ahead = corner_of(next);
                        fetch_h(next, ahead, p.inner - 1);
                        if (BN) fetch_x(ahead);
                        expect(ahead);
                    }
                }
                quad_stencil<PLANE, ADD>(rows, dx, tm, g, inv, [](int, int, float, float, u64, u64) {});
                __syncwarp();  // ... and has been read
            }
            if (next < cnt) fetch_g(ahead);
            if (BN && quad_tile_leader<SUB>(lane)) {
                float4 *to = p.hterm + ((size_t)q * ntiles + quad_tile_of(L, blk)) * 2;
                float v[8];
                unpack2(hf[0], v[0], v[1]);
                unpack2(hf[1], v[2], v[3]);
                unpack2(he[0], v[4], v[5]);
                unpack2(he[1], v[6], v[7]);
                to[0] = make_float4(v[0], v[1], v[2], v[3]);
                to[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
            __syncwarp();
            quad_store(p.gx + own, zstr, ystr, L.h, g);
            quad_store(p.dsum + own, zstr, ystr, L.h, dsum);
            // four x-neighbours at a time, in ascending order
            float *const dq = p.dsq + own / 4;
#pragma unroll
            for (int n = 0; n < 4; ++n)
                *reinterpret_cast<float4 *>(dq + (n >> 1) * wzs + (n & 1) * wys) =
                    L.h ? make_float4(dsa[n][3], dsa[n][2], dsa[n][1], dsa[n][0]) : make_float4(dsa[n][0], dsa[n][1], dsa[n][2], dsa[n][3]);
        }
        i0 += here;
        q0 = 0;
        ++blk;
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free_all(tmem_slot);
}

// ---------------------------------------------------------------------------------------- weight gradients
// One CTA of 128 threads per region and chunk of quads. A thread owns a 2 x 2 x 1 (z, y, x) patch and keeps its 4 x 27 sums
// in registers from the first quad to the last; a quarter-warp reads whole rows of cells, so every shared-memory access is
// free of bank conflicts. Per iteration and quad 48 cells serve 4 x 27 x 4 FMAs: 2.25 per wavefront, half of what the
// 2 x 2 x 4 patches of the other kernels get, but those would need their 432 sums in tensor memory, and reading, adding to
// and writing back sums there was 3 to 4 times slower than this (128^3, two inner iterations, batch 32: 0.77 - 0.97 ms).
// The step's input tile arrives by bulk tensor copy and is normalised in place; activations between iterations are rebuilt
// from it and the pre-activations. Two tiles take turns over the iterations, one barrier each (block 4 with one tile, updated in
// place between two barriers: 64^3 x 128, 8 x 16 with gradients 39.9 ms, with two 38.8). Deltas and pre-activations arrive
// an iteration ahead, what else a quad needs a quad ahead, each thread its own (128^3 x 32, 2 x 16: 30.35 -> 30.05 ms).
// What bounds it: 61 % of the shared-memory pipe, 1300 of 2900 cycles per iteration in the window sums, the rest deltas, activations and
// copies between two barriers (block 4: 956 us a step at 64^3 x 128, now 823; 128^3 x 32 518, now 486). Computing the activations under the
// window sums takes a second copy of these: 1 % faster at 128^3, 2 % slower at 32^3, where kernels are over before their code has
// arrived.
namespace quadwg {
constexpr int CTAS = 2;  // per SM: 255 registers (three with 168 spill, and are no faster)
constexpr int THREADS = 128, OWN = 4 * THREADS * 16;  // bytes of one staging area: a thread's four cells
constexpr int GRAD_F = (27 * 4 + 8) * THREADS;        // floats per region and chunk: weights, biases, scales
template <int SUB>
struct Lay {
    static constexpr int NT = 2;  // tiles
    static constexpr int TILE = (QuadGeo<SUB>::BUF_BYTES + 127) / 128 * 128;
    static constexpr int DSQ = NT * TILE + 3 * OWN;  // a quad's terms of the scale gradient, each thread its own four
    static constexpr int IST = DSQ + THREADS * 16;   // and, each warp its own copy, its statistics
    static constexpr int SCALE = IST + THREADS;      // residual scales, each thread its own four
    static constexpr int GB = SCALE + THREADS * 16;  // normalise-on-load: the region's (gamma, beta) table
    static constexpr int NSTAT = (SUB == 8 ? 1 : 8) * QS_COUNT;  // per-block normalisation, there: two iterations' statistics
    static constexpr int smem(bool fuse, bool norm) { return GB + (fuse ? QuadGeo<SUB>::CELLS * 8 : 0) + (norm ? 2 * NSTAT * 16 : 0); }
};
// thread -> patch. Block 8: lanes of a quarter-warp are the eight x; block 4: four x and two y patches (two rows of six
// cells further is four banks further)
template <int SUB>
struct Patch {
    int x, yp, zp, cell0;
    __device__ __forceinline__ explicit Patch(int tid)
    {
        using G = QuadGeo<SUB>;
        const int l = tid & 31;
        zp = tid >> 5;
        if (SUB == 8) {
            x = l & 7;
            yp = l >> 3;
            cell0 = 2 * zp * G::PLANE + 2 * yp * G::ROW + x;
        } else {
            x = (l & 3) | ((l >> 3) & 1) << 2;
            yp = ((l >> 2) & 1) | (l >> 4) << 1;
            cell0 = (((zp >> 1) * 2 + (yp >> 1)) * 2 + (x >> 2)) * 216 + 2 * (zp & 1) * G::PLANE + 2 * (yp & 1) * G::ROW + (x & 3);
        }
    }
};
}  // namespace quadwg

struct QuadWgradParams {
    const float2 *gbt;       // FUSE_IN: as in step_fwd_quad
    const float2 *in_stats;
    const float *delta, *h;  // [inner] IL4
    const float *scale;      // [M][N][K]
    const float *dsq;        // [Q][P]
    const float4 *tile_stats;  // NORM: [inner][Q][tiles][QS_COUNT]
    const float *delta2;       // GATED: of the gate
    float *gpk;              // [chunks][regions][GRAD_F]
    int accumulate;          // add to what is there
    int *error_flag;
    int M, N, K, Q, inner, qpc;
};

// NORM: per-block normalisation. The deltas are already scaled by 1 / (std + eps). The tile is kept relative to its mean before the
// first iteration, v - c, and sum delta (v - mean_t) = sum delta (v - c) - sum delta (mean_t - c): the second sum is one
// number per neuron, taken off all its 27 sums at the end. The bias gradient wants the unscaled delta back.
// GATED: blockIdx.z picks the branch; h holds the activations after each iteration (they were kept), there is no scale.
template <int SUB, int ACT, bool FUSE_IN, bool NORM, bool GATED>
__global__ void __launch_bounds__(quadwg::THREADS, quadwg::CTAS) quad_wgrad_k(const __grid_constant__ CUtensorMap in_map, const QuadWgradParams p)
{
    using namespace quadwg;
    using G = QuadGeo<SUB>;
    using Y = Lay<SUB>;
    constexpr int NT = Y::NT;
    constexpr unsigned kSpin = quad::kSpinLimit;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[NT];
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < NT; ++i) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    __syncthreads();
    const Patch<SUB> T(tid);
    const int nbx = p.K >> 3, nby = p.N >> 3, blk = blockIdx.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)p.M * p.N * p.K, T4 = (size_t)p.Q * P * 4;
    const unsigned tiles = smem_u32(smem), stage_d = tiles + NT * Y::TILE + tid * 16, stage_h = stage_d + 2 * OWN;
    const unsigned bar0 = smem_u32(bars);
    const size_t g0 = ((size_t)(bz * 8 + 2 * T.zp) * p.N + (by * 8 + 2 * T.yp)) * p.K + bx * 8 + T.x;
    const size_t zs = (size_t)p.N * p.K;
    const int q0 = blockIdx.y * p.qpc, q1 = min(p.Q, q0 + p.qpc);
    bool failed = false;
    constexpr int STEPS = (G::CELLS + THREADS - 1) / THREADS;
    unsigned halo = 0;  // bit c: cell c * THREADS + tid of the tile is a halo cell
    for (int c = 0; c < STEPS; ++c) {
        const int l = (c * THREADS + tid) % (SUB == 8 ? 1000 : 216), x = l % G::SIDE, y = l / G::SIDE % G::SIDE, z = l / G::SIDE / G::SIDE;
        if (z == 0 || z == G::SIDE - 1 || y == 0 || y == G::SIDE - 1 || x == 0 || x == G::SIDE - 1) halo |= 1u << c;
    }

    auto issue = [&](int q, int buf) {
        const unsigned tile = tiles + buf * Y::TILE, bar = bar0 + 8 * buf;
        fence_proxy_async();
        mbar_expect_tx(bar, G::CELLS * 16);
        if (SUB == 8) {
            tma_load_4d(tile, &in_map, bar, (bx * 8 - 1) * 4, by * 8 - 1, bz * 8 - 1, q);
        } else {
            for (int sub = 0; sub < 8; ++sub)
                tma_load_4d(tile + sub * 216 * 16, &in_map, bar, (bx * 8 + (sub & 1) * 4 - 1) * 4, by * 8 + ((sub >> 1) & 1) * 4 - 1,
                            bz * 8 + (sub >> 2) * 4 - 1, q);
        }
    };
    auto fetch = [&](unsigned dst, const float *src) {  // this thread's four cells
#pragma unroll
        for (int n = 0; n < 4; ++n) cp_async16(dst + n * (THREADS * 16), src + ((n >> 1) * zs + (n & 1) * (size_t)p.K) * 4);
    };
    const unsigned stats0 = tiles + Y::GB;  // NORM: [2][tile][QS_COUNT]
    const unsigned my_tile = SUB == 8 ? 0u : (unsigned)(((T.zp >> 1) * 2 + (T.yp >> 1)) * 2 + (T.x >> 2)) * (QS_COUNT * 16);
    auto fetch_stats = [&](int buf, int q, int it) {
        if (NORM && tid < Y::NSTAT)
            cp_async16(stats0 + buf * (Y::NSTAT * 16) + tid * 16, p.tile_stats + (((size_t)it * p.Q + q) * gridDim.x + blk) * Y::NSTAT + tid);
    };
    auto at = [&](const float *t, int q, int it) { return t + (size_t)it * T4 + ((size_t)q * P + g0) * 4; };
    // what a quad starts with, a quad ahead: its scale terms and statistics
    const unsigned my_dsq = tiles + Y::DSQ + tid * 16, my_ist = tiles + Y::IST + (tid >> 5) * 32;
    auto fetch_quad = [&](int q) {
        if (!GATED) {
            const float *s = p.dsq + (size_t)q * P + g0;
#pragma unroll
            for (int n = 0; n < 4; ++n) cp_async4(my_dsq + 4 * n, s + (n >> 1) * zs + (n & 1) * (size_t)p.K);
        }
        // four lanes: asynchronous copies of one address by all lanes are a request each (128^3: the step three times as long). A pair
        // each: that is how a caller's statistics are aligned
        if (FUSE_IN && (tid & 31) < 4) cp_async8(my_ist + (tid & 31) * 8, p.in_stats + 4 * q + (tid & 31));
    };

    // sums: sg[dy = 0 at ry = 0, dy = 1 at ry = 3][dz][a][c], sp[ry = 1, 2][dz][a][c] = (dy = 0, dy = 1)
    float sg[2][2][3][3];
    u64 sp[2][2][3][3];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    sg[i][j][a][c] = 0.0f;
                    sp[i][j][a][c] = 0;
                }
    u64 db[2] = {0, 0}, ds[2] = {0, 0};  // [dz]: (dy = 0, dy = 1)
    u64 off[2] = {0, 0};                 // NORM: sum delta (mean_t - c)

    int buf_x = 0, buf_d = 0;
    unsigned landed = 0;  // bit b: phase of tile b's barrier
    const float2 *const gbs = reinterpret_cast<const float2 *>(smem + Y::GB);
    if (FUSE_IN) {
        const unsigned char *src = reinterpret_cast<const unsigned char *>(p.gbt + (size_t)blk * G::CELLS);
        for (int c = tid; c < G::CELLS / 2; c += THREADS) cp_async16(tiles + Y::GB + c * 16, src + c * 16);
        cp_async_wait_all();
        __syncthreads();
    }
    const unsigned my_scale = tiles + Y::SCALE + tid * 16;
    if (!GATED && p.inner > 1) {
        const float *s = p.scale + g0;
        sts128(my_scale, make_float4(s[0], s[p.K], s[zs], s[zs + p.K]));
    }
    previous_done();
    if (tid == 0) issue(q0, 0);
    fetch_quad(q0);
    const float *const delta = GATED && blockIdx.z ? p.delta2 : p.delta;
    // deltas are asked for in the order (quad, iteration), pre-activations likewise without the last iteration
    const float *d_next = at(delta, q0, 0), *h_next = at(p.h, q0, 0);
    const long long next_quad = 4 * (long long)P;
    fetch(stage_d, d_next);
    fetch_stats(0, q0, 0);
    if (p.inner > 1) fetch(stage_h, h_next);
    const unsigned own0 = (unsigned)(T.cell0 + G::PLANE + G::ROW + 1) * 16u;

    for (int q = q0; q < q1; ++q) {
        if (!mbar_wait_bounded(bar0 + 8 * buf_x, (landed >> buf_x) & 1u, kSpin)) failed = true;
        landed ^= 1u << buf_x;
        const bool two = p.inner > 1;
        cp_async_wait_all();  // the quad's statistics, the first iteration's
        if (FUSE_IN) __syncwarp();
        if (two || NORM) __syncthreads();  // nobody reads the other tile any more: it gets the new halo
        float4 pivot = make_float4(0.f, 0.f, 0.f, 0.f);
        if (NORM) pivot = lds128(stats0 + buf_d * (Y::NSTAT * 16) + my_tile + QS_MEAN * 16);
        if (FUSE_IN || two || NORM) {
            const unsigned tile = tiles + buf_x * Y::TILE, other = tiles + (buf_x ^ 1) * Y::TILE;
            u64 na[2], nb[2];
            if (FUSE_IN) {
                const float4 m01 = lds128(my_ist), m23 = lds128(my_ist + 16);
                na[0] = pack2(m01.y, m01.w);
                na[1] = pack2(m23.y, m23.w);
                nb[0] = pack2(-m01.x, -m01.z);
                nb[1] = pack2(-m23.x, -m23.z);
            }
            constexpr int BATCH = SUB == 8 ? 8 : 7;
#pragma unroll 1
            for (int c0 = 0; c0 < STEPS; c0 += BATCH) {
                u64 v[BATCH][2];
                float2 g2[BATCH];
#pragma unroll
                for (int c = 0; c < BATCH; ++c) {
                    const int i = (c0 + c) * THREADS + tid;
                    if (i < G::CELLS) {
                        if (FUSE_IN) g2[c] = gbs[i];
                        lds128u(tile + i * 16, v[c][0], v[c][1]);
                    }
                }
#pragma unroll
                for (int c = 0; c < BATCH; ++c) {
                    const int i = (c0 + c) * THREADS + tid;
                    if (i < G::CELLS) {
                        if (FUSE_IN) {
                            const u64 gg = pack2(g2[c].x, g2[c].x), bb = pack2(g2[c].y, g2[c].y);
                            v[c][0] = ffma2r(fmul2(fadd2(v[c][0], nb[0]), na[0]), gg, bb);
                            v[c][1] = ffma2r(fmul2(fadd2(v[c][1], nb[1]), na[1]), gg, bb);
                            sts128u(tile + i * 16, v[c][0], v[c][1]);
                        }
                        if (NORM) {
                            u64 m0, m1;
                            lds128u(stats0 + buf_d * (Y::NSTAT * 16) + (SUB == 8 ? 0 : i / 216 * (QS_COUNT * 16)) + QS_MEAN * 16, m0, m1);
                            v[c][0] = ffma2r(m0, pack2(-1.0f, -1.0f), v[c][0]);
                            v[c][1] = ffma2r(m1, pack2(-1.0f, -1.0f), v[c][1]);
                            sts128u(tile + i * 16, v[c][0], v[c][1]);
                        }
                        if (two && (halo >> (c0 + c) & 1)) sts128u(other + i * 16, v[c][0], v[c][1]);
                    }
                }
            }
        }
        for (int t = 0; t < p.inner; ++t) {
            const bool last = t + 1 == p.inner;
            const unsigned tile = tiles + buf_x * Y::TILE;
            cp_async_wait_all();
            __syncthreads();  // the tile is complete; nobody is an iteration behind
            u64 dp[2][4];     // deltas [dz][sample]: (dy = 0, dy = 1)
#pragma unroll
            for (int dz = 0; dz < 2; ++dz) {
                const float4 a = lds128(stage_d + buf_d * OWN + (2 * dz) * (THREADS * 16)), b = lds128(stage_d + buf_d * OWN + (2 * dz + 1) * (THREADS * 16));
                dp[dz][0] = pack2(a.x, b.x);
                dp[dz][1] = pack2(a.y, b.y);
                dp[dz][2] = pack2(a.z, b.z);
                dp[dz][3] = pack2(a.w, b.w);
            }
            float4 unscale = make_float4(1.f, 1.f, 1.f, 1.f), shift = unscale;  // NORM
            if (NORM) {
                const unsigned st = stats0 + buf_d * (Y::NSTAT * 16) + my_tile;
                unscale = lds128(st + QS_STDEPS * 16);
                shift = lds128(st + QS_MEAN * 16);
                shift.x -= pivot.x, shift.y -= pivot.y, shift.z -= pivot.z, shift.w -= pivot.w;
            }
            if (!last) {  // the activations of iteration t + 1 -> the other tile. All loads first: a load waits for a store before it
                const unsigned to = tiles + (buf_x ^ 1) * Y::TILE;
                auto cell = [&](int n) { return own0 + (unsigned)((n >> 1) * G::PLANE + (n & 1) * G::ROW) * 16u; };
                u64 h[4][2], x[4][2];
                float4 sc = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!GATED) sc = lds128(my_scale);
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    lds128u(stage_h + n * (THREADS * 16), h[n][0], h[n][1]);
                    if (!GATED) lds128u(tile + cell(n), x[n][0], x[n][1]);
                }
                const float s4[4] = {sc.x, sc.y, sc.z, sc.w};
                if (!GATED)
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int k = 0; k < 2; ++k) h[n][k] = act_residual2<ACT>(h[n][k], s4[n], x[n][k]);
#pragma unroll
                for (int n = 0; n < 4; ++n) sts128u(to + cell(n), h[n][0], h[n][1]);
            }
            if (t == 0) {
                if (!GATED) {
                    const float4 v = lds128(my_dsq);
                    ds[0] = fadd2(ds[0], pack2(v.x, v.y));
                    ds[1] = fadd2(ds[1], pack2(v.z, v.w));
                }
                if (q + 1 < q1) fetch_quad(q + 1);  // every warp has passed a barrier since it read the quad's statistics
            }
            // the next iteration's data
            if (!last) {
                d_next += T4;
                fetch(stage_d + (buf_d ^ 1) * OWN, d_next);
                fetch_stats(buf_d ^ 1, q, t + 1);
                if (t + 2 < p.inner) {
                    h_next += T4;
                    fetch(stage_h, h_next);
                }
            } else if (q + 1 < q1) {
                d_next += next_quad - (p.inner - 1) * (long long)T4;
                fetch(stage_d + (buf_d ^ 1) * OWN, d_next);
                fetch_stats(buf_d ^ 1, q + 1, 0);
                if (p.inner > 1) {
                    h_next += next_quad - (p.inner - 2) * (long long)T4;
                    fetch(stage_h, h_next);
                }
                if (tid == 0) issue(q + 1, buf_x ^ 1);
            }
#pragma unroll
            for (int dz = 0; dz < 2; ++dz) {
                if (NORM) {
                    const float us[4] = {unscale.x, unscale.y, unscale.z, unscale.w}, sh[4] = {shift.x, shift.y, shift.z, shift.w};
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        ffma2(db[dz], dp[dz][s], pack2(us[s], us[s]));
                        ffma2(off[dz], dp[dz][s], pack2(sh[s], sh[s]));
                    }
                } else {
                    db[dz] = fadd2(db[dz], fadd2(fadd2(dp[dz][0], dp[dz][1]), fadd2(dp[dz][2], dp[dz][3])));
                }
            }
            const unsigned win = tile + T.cell0 * 16u;
#pragma unroll
            for (int rz = 0; rz < 4; ++rz)
#pragma unroll
                for (int ry = 0; ry < 4; ++ry)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float4 v = lds128(win + (unsigned)(rz * G::PLANE + ry * G::ROW + c) * 16u);
                        const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int dz = 0; dz < 2; ++dz) {
                            const int a = rz - dz;
                            if (a < 0 || a > 2) continue;
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                if (ry == 1 || ry == 2) {
                                    ffma2(sp[ry - 1][dz][a][c], dp[dz][s], pack2(vs[s], vs[s]));
                                } else {
                                    float lo, hi;
                                    unpack2(dp[dz][s], lo, hi);
                                    sg[ry ? 1 : 0][dz][a][c] = fmaf(vs[s], ry ? hi : lo, sg[ry ? 1 : 0][dz][a][c]);
                                }
                            }
                        }
                    }
            buf_x ^= 1;
            buf_d ^= 1;
        }
    }
    // ---- sums -> this chunk's part: [tap][n] then [bias | scale][n], 128 threads each
    float *const dst = p.gpk + (((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blk) * GRAD_F + tid;
    auto put = [&](int k, float v) { dst[k * THREADS] = p.accumulate ? dst[k * THREADS] + v : v; };
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        float off0 = 0.0f, off1 = 0.0f;
        if (NORM) unpack2(off[dz], off0, off1);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                // window row ry is tap row b = ry - dy of neuron row dy
                put((a * 9 + 0 + c) * 4 + dz * 2 + 0, sg[0][dz][a][c] - off0);
                put((a * 9 + 6 + c) * 4 + dz * 2 + 1, sg[1][dz][a][c] - off1);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float lo, hi;
                    unpack2(sp[r][dz][a][c], lo, hi);
                    put((a * 9 + (r + 1) * 3 + c) * 4 + dz * 2 + 0, lo - off0);
                    put((a * 9 + r * 3 + c) * 4 + dz * 2 + 1, hi - off1);
                }
            }
    }
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        float lo, hi;
        unpack2(db[dz], lo, hi);
        put(108 + dz * 2, lo);
        put(109 + dz * 2, hi);
        if (GATED) continue;
        unpack2(ds[dz], lo, hi);
        put(112 + dz * 2, lo);
        put(113 + dz * 2, hi);
    }
    if (failed && p.error_flag) *p.error_flag = 1;
}

// The chunks' sums in chunk order -> gradients in the layout of the parameters. Two regions per CTA
// of 256 threads, four CTAs side by side, branch after branch;
// the CTAs after those put the input's gradient back into the grid's own layout.
constexpr int kUnpack = 29;  // of the 116 values per thread
template <int SUB>
__global__ void __launch_bounds__(256) quad_finish_k(const float *gpk, float *gw, float *gb, float *gs, const float4 *il, float *x, int B, int M,
                                                     int N, int K, int chunks, int branches, unsigned grads, unsigned parts)
{
    using namespace quadwg;
    previous_done();
    if (blockIdx.x >= grads) {
        const unsigned i = blockIdx.x - grads;
        const size_t P = (size_t)M * N * K, c = (size_t)(i % parts) * 256 + threadIdx.x;
        const int q = i / parts;
        if (c >= P) return;
        const float4 v = il[(size_t)q * P + c];
        const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (4 * q + s < B) x[(size_t)(4 * q + s) * P + c] = vs[s];
        return;
    }
    const int tid = threadIdx.x & 127, regions = (M >> 3) * (N >> 3) * (K >> 3);
    const unsigned per = grads / branches, cta = blockIdx.x % per, branch = blockIdx.x / per;
    const Patch<SUB> T(tid);
    const int nbx = K >> 3, nby = N >> 3, blk = cta / (116 / kUnpack) * 2 + (threadIdx.x >> 7);
    if (blk >= regions) return;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const size_t g0 = ((size_t)(bz * 8 + 2 * T.zp) * N + (by * 8 + 2 * T.yp)) * K + bx * 8 + T.x;
    const float *src = gpk + ((size_t)branch * chunks * regions + blk) * GRAD_F + tid;
    const size_t step = (size_t)regions * GRAD_F;
    const int k0 = cta % (116 / kUnpack) * kUnpack;
    // chunk after chunk, so that a thread has 29 loads in flight
    float v[kUnpack];
#pragma unroll
    for (int i = 0; i < kUnpack; ++i) v[i] = src[(k0 + i) * THREADS];
    for (int c = 1; c < chunks; ++c) {
        src += step;
#pragma unroll
        for (int i = 0; i < kUnpack; ++i) v[i] += src[(k0 + i) * THREADS];
    }
#pragma unroll
    for (int i = 0; i < kUnpack; ++i) {
        const int k = k0 + i, n = k & 3;
        if (branches > 1 && k >= 112) break;  // no scale
        float *dst = k < 108 ? gw + ((size_t)(k >> 2) * branches + branch) * P : (k < 112 ? gb + branch * P : gs);
        dst[g0 + (size_t)(n >> 1) * N * K + (size_t)(n & 1) * K] = v[i];
    }
}

// ------------------------------------------------------------------------- gradient across block borders
// As bwd_border8_k / bwd_halo8_k (step_bwd_fast.cu), four samples at a time: a cell of a quad is 16 bytes, so even the
// x faces use half of every sector they touch.
// Block 8: three groups of 128 threads, one per axis; a thread owns one cell of the two faces and the nine taps that cross
// that face (a tap that crosses several faces belongs to the first axis in the order z, y, x); then one thread per surface
// cell adds the up to three partial sums to grad_x in that order. Only the shell of 488 cells around the region is fetched,
// face by face: what a group reads is dense, so there are no bank conflicts and a thread needs one base address. Bound by
// memory latency: everything a quad needs is asked for two quads ahead by asynchronous copies, which need no registers,
// so that three CTAs fit on an SM (with the 10^3 tile and register prefetch two did: 72 us, now 40, at 64^3, batch 64).
__device__ __forceinline__ float4 fma4(float w, float4 v, float4 a)
{
    return make_float4(fmaf(w, v.x, a.x), fmaf(w, v.y, a.y), fmaf(w, v.z, a.z), fmaf(w, v.w, a.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// NORM (per-block normalisation): a cell also owes F + E x to the statistics of every tile that it is a halo cell of
// (quad_reverse_k). The (negated) terms of the surrounding tiles, 3^3 regions or 4^3 blocks of 4, come with the quad.
namespace quadborder {
constexpr int TS = 1000;               // block 4: cells of a tile
constexpr int SHELL = 500;             // block 8: cells of a shell, padded for taps that do not count
constexpr int SURFACE = 296, DIRS = 27;
template <int SUB>
struct Terms {
    static constexpr int SIDE = SUB == 8 ? 3 : 4, COUNT = SIDE * SIDE * SIDE;
    // the tile this thread fetches, -1: none, or outside the grid
    __device__ static int tile(int slot, int bx, int by, int bz, int M, int N, int K)
    {
        if (slot >= COUNT) return -1;
        const int tx = bx * (8 / SUB) + slot % SIDE - 1, ty = by * (8 / SUB) + slot / SIDE % SIDE - 1, tz = bz * (8 / SUB) + slot / SIDE / SIDE - 1;
        if (tx < 0 || ty < 0 || tz < 0 || tx >= K / SUB || ty >= N / SUB || tz >= M / SUB) return -1;
        if (SUB == 8) return (tz * (N / 8) + ty) * (K / 8) + tx;
        return (((tz >> 1) * (N / 8) + (ty >> 1)) * (K / 8) + (tx >> 1)) * 8 + ((tz & 1) * 2 + (ty & 1)) * 2 + (tx & 1);
    }
    // sum over the tiles that contain a cell of tile `own` as halo, the cell lying on the faces (dz, dy, dx)
    __device__ static float4 along(const float4 *t, int own, int dz, int dy, int dx)
    {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int m = 1; m < 8; ++m)
            if ((!(m & 4) || dz) && (!(m & 2) || dy) && (!(m & 1) || dx)) {
                const float4 f = t[2 * (own + ((m & 4 ? dz : 0) * SIDE + (m & 2 ? dy : 0)) * SIDE + (m & 1 ? dx : 0))];
                a.x += f.x, a.y += f.y, a.z += f.z, a.w += f.w;
            }
        return a;
    }
    // F + E v of the region's cell (z, y, x)
    __device__ static float4 sum(const float4 *t, int z, int y, int x, float4 v)
    {
        const int qz = z % SUB, qy = y % SUB, qx = x % SUB;
        const int dz = qz == 0 ? -1 : (qz == SUB - 1 ? 1 : 0), dy = qy == 0 ? -1 : (qy == SUB - 1 ? 1 : 0), dx = qx == 0 ? -1 : (qx == SUB - 1 ? 1 : 0);
        const int own = ((z / SUB + 1) * SIDE + y / SUB + 1) * SIDE + x / SUB + 1;
        const float4 f = along(t, own, dz, dy, dx), e = along(t + 1, own, dz, dy, dx);
        return make_float4(fmaf(e.x, v.x, f.x), fmaf(e.y, v.y, f.y), fmaf(e.z, v.z, f.z), fmaf(e.w, v.w, f.w));
    }
};
}  // namespace quadborder

// SUMS: the sums of the LayerNorm gradient of the step before, whose output is this step's input, in the same pass (see
// quad_norm_sums_k), since the gradient is in the CTA's hands anyway. A thread has a cell of the surface or
// the interior, the first 128 a second one; the CTAs of a region are a cluster, which adds up the gradients of gamma and beta
// in the order of their ranks. When: quad_border_takes_sums.
enum BorderSums { NO_SUMS, SUMS };
struct BorderParams {
    const float *w;
    const float4 *dsum, *dsum2;  // BR == 2: of the gate
    float4 *gx;
    const float4 *x;             // NORM: the step's input; sums: the norm's, IL4
    const float4 *hterm;         // NORM
    const float *gamma;
    const float2 *stats;
    double2 *partials;           // sums: [4 Q][regions]
    float *ggamma, *gbeta;
    int accumulate, Q, M, N, K, qpc;
};
// cell s of a region: 0 .. 295 on its surface, then the interior
__device__ __forceinline__ void border_cell(int s, int &z, int &y, int &x)
{
    if (s < 128) {
        z = (s >> 6) * 7, y = (s >> 3) & 7, x = s & 7;
    } else if (s < 224) {
        const int j = s - 128;
        y = (j / 48) * 7, z = 1 + (j % 48) / 8, x = j & 7;
    } else if (s < 296) {
        const int j = s - 224;
        x = (j / 36) * 7, z = 1 + (j % 36) / 6, y = 1 + j % 6;
    } else {
        const int j = s - 296;
        z = 1 + j / 36, y = 1 + j / 6 % 6, x = 1 + j % 6;
    }
}
namespace quadborder {
template <bool NORM, int BR, BorderSums S>
struct Room {
    static constexpr int RING = S != NO_SUMS && BR == 2 ? 2 : 3;      // quads in flight
    static constexpr int CELLS = S == NO_SUMS ? SURFACE : 512;        // a quad's grad_x, and as many of each further tensor
    static constexpr int TENSORS = S == SUMS || NORM ? 2 : 1;
    static constexpr int BYTES = (RING * (BR * SHELL + TENSORS * CELLS) + 2 * BR * 384) * 16;
    static constexpr int CTAS = S == NO_SUMS && BR == 1 ? 3 : 2;
};
}  // namespace quadborder

template <bool NORM, int BR, BorderSums S>
__global__ void __launch_bounds__(384, quadborder::Room<NORM, BR, S>::CTAS) quad_border8_k(const BorderParams p)
{
    using namespace quadborder;
    using T = Terms<8>;
    using R = Room<NORM, BR, S>;
    static_assert(S == NO_SUMS || !NORM, "");
    constexpr int THREADS = 384, RING = R::RING, CELLS = R::CELLS, AHEAD = RING - 1, QB = 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4 *const shell = reinterpret_cast<float4 *>(smem_raw);  // [RING][BR][SHELL]
    float4 *const part = shell + RING * BR * SHELL;              // [2][BR][3][128]
    float4 *const mine = part + 2 * BR * 3 * 128;                // [tensor][RING][CELLS] grad_x, then x
    __shared__ float4 terms[NORM ? RING : 1][2 * T::COUNT], dirs[NORM ? 2 : 1][2 * DIRS];
    __shared__ double red[S != NO_SUMS ? QB : 1][THREADS / 32][8];
    __shared__ float4 quad_stats[S != NO_SUMS ? RING : 1][2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int M = p.M, N = p.N, K = p.K, nbx = K >> 3, nby = N >> 3;
    const unsigned blk = blockIdx.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const long long origin = ((long long)(bz * 8 - 1) * N + (by * 8 - 1)) * K + (bx * 8 - 1);
    for (int i = tid; i < RING * BR * SHELL; i += THREADS) shell[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // shell cells this thread fetches: z faces 2 x 10 x 10, then y faces 2 x 8 x 10, then x faces 2 x 8 x 8
    int rel[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = tid + j * THREADS;
        int cz, cy, cx;
        if (i < 200) {
            cz = i / 100 * 9, cy = i % 100 / 10, cx = i % 10;
        } else if (i < 360) {
            const int e = i - 200;
            cz = 1 + e % 80 / 10, cy = e / 80 * 9, cx = e % 10;
        } else {
            const int e = i - 360;
            cz = 1 + e % 64 / 8, cy = 1 + e % 8, cx = e / 64 * 9;
        }
        const int gz = bz * 8 + cz - 1, gy = by * 8 + cy - 1, gxx = bx * 8 + cx - 1;
        const bool in = i < 488 && gz >= 0 && gz < M && gy >= 0 && gy < N && gxx >= 0 && gxx < K;
        rel[j] = in ? (cz * N + cy) * K + cx : -1;
    }
    // role 1: one cell of one face, (u, v) its coordinates along the other two axes
    const int axis = tid >> 7, fc = tid & 127, side = fc >> 6, u = (fc >> 3) & 7, v = fc & 7;
    const int across = side == 0 ? 1 : -1;
    float wf[BR][9];
    {
        const int lz = axis == 0 ? side * 7 : u, ly = axis == 0 ? u : (axis == 1 ? side * 7 : v), lx = axis == 2 ? side * 7 : v;
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            const int d1 = e / 3 - 1, d2 = e % 3 - 1;
            const int dz = axis == 0 ? across : d1, dy = axis == 0 ? d1 : (axis == 1 ? across : d2), dx = axis == 2 ? across : d2;
            const bool owned = (axis == 0 || (u - d1 >= 0 && u - d1 < 8)) && (axis < 2 || (v - d2 >= 0 && v - d2 < 8));
            const int nz = bz * 8 + lz - dz, ny = by * 8 + ly - dy, nx = bx * 8 + lx - dx;
            const bool ok = owned && nz >= 0 && nz < M && ny >= 0 && ny < N && nx >= 0 && nx < K;
#pragma unroll
            for (int k = 0; k < BR; ++k)
                wf[k][e] = ok ? p.w[((size_t)((dz + 1) * 9 + (dy + 1) * 3 + dx + 1) * BR + k) * P + ((size_t)nz * N + ny) * K + nx] : 0.0f;
        }
    }
    const int row = axis == 2 ? 8 : 10;
    const int base = axis == 0 ? side * 100 + (u + 1) * 10 + v + 1 : (axis == 1 ? 200 + side * 80 + u * 10 + v + 1 : 360 + side * 64 + u * 8 + v);
    // role 2: one surface cell; sums: or one of the interior, and the interior's others
    const bool surface = tid < SURFACE, active = S != NO_SUMS || surface, second = S != NO_SUMS && tid < 512 - THREADS;
    auto place = [&](int s) {
        int z, y, x;
        border_cell(s, z, y, x);
        return ((size_t)(bz * 8 + z) * N + by * 8 + y) * K + bx * 8 + x;
    };
    int sz, sy, sx;
    border_cell(tid, sz, sy, sx);
    const size_t c = active ? place(tid) : 0, c2 = second ? place(THREADS + tid) : 0;
    const bool on_z = surface && (sz == 0 || sz == 7), on_y = surface && (sy == 0 || sy == 7), on_x = surface && (sx == 0 || sx == 7);
    const int pz = (sz / 7) * 64 + sy * 8 + sx, py = 128 + (sy / 7) * 64 + sz * 8 + sx, px = 256 + (sx / 7) * 64 + sz * 8 + sy;
    const int my_dir = ((on_z ? sz / 7 * 2 : 1) * 3 + (on_y ? sy / 7 * 2 : 1)) * 3 + (on_x ? sx / 7 * 2 : 1);
    float gm[2] = {0.f, 0.f}, dg[2] = {0.f, 0.f}, db[2] = {0.f, 0.f};  // sums: of the two cells
    if (S != NO_SUMS) {
        gm[0] = p.gamma[c];
        if (second) gm[1] = p.gamma[c2];
    }

    const int Q = p.Q, q0 = blockIdx.y * p.qpc, q1 = min(Q, q0 + p.qpc);
    const unsigned shell0 = smem_u32(shell) + tid * 16, mine0 = smem_u32(mine) + tid * 16;
    const int my_term = NORM ? T::tile(tid >> 1, bx, by, bz, M, N, K) : -1;
    if (NORM && tid < 2 * T::COUNT)
        for (int r = 0; r < RING; ++r) terms[r][tid] = make_float4(0.f, 0.f, 0.f, 0.f);
    int slot = 0;  // ring slot of the quad in work
    auto fetch = [&](int q, int r) {
        if (q < q1) {
#pragma unroll
            for (int k = 0; k < BR; ++k) {
                const float4 *src = (k ? p.dsum2 : p.dsum) + (size_t)q * P + origin;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (rel[j] >= 0) cp_async16(shell0 + (unsigned)((r * BR + k) * SHELL + j * THREADS) * 16u, src + rel[j]);
            }
            const float4 *const tensors[2] = {p.gx, p.x};
#pragma unroll
            for (int k = 0; k < R::TENSORS; ++k) {
                if (active) cp_async16(mine0 + (unsigned)((k * RING + r) * CELLS) * 16u, tensors[k] + (size_t)q * P + c);
                if (second) cp_async16(mine0 + (unsigned)((k * RING + r) * CELLS + THREADS) * 16u, tensors[k] + (size_t)q * P + c2);
            }
            if (NORM && my_term >= 0) cp_async16(smem_u32(&terms[r][tid]), p.hterm + ((size_t)q * gridDim.x + my_term) * 2 + (tid & 1));
            if (S != NO_SUMS && tid < 4) cp_async8(smem_u32(&quad_stats[r][0]) + tid * 8, p.stats + 4 * q + tid);  // a caller's: 8-byte aligned
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();  // the shells are zeroed
    previous_done();
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) fetch(q0 + k, k);
    for (int q = q0; q < q1; ++q) {
        const int par = q & 1;
        asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
        __syncthreads();  // quad q has landed; the shell of quad q - 1 has been read
        fetch(q + AHEAD, slot == 0 ? RING - 1 : slot - 1);
#pragma unroll
        for (int k = 0; k < BR; ++k) {
            const float4 *sh = shell + (slot * BR + k) * SHELL + base;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 9; ++e) s = fma4(wf[k][e], sh[-(e / 3 - 1) * row - (e % 3 - 1)], s);
            part[(par * BR + k) * 384 + tid] = s;
        }
        if (NORM && tid < 2 * DIRS) {
            const int d = tid >> 1;
            dirs[par][tid] = T::along(&terms[slot][tid & 1], 13, d / 9 - 1, d / 3 % 3 - 1, d % 3 - 1);
        }
        __syncthreads();
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (active) acc = mine[slot * CELLS + tid];
        if (surface) {
            if (NORM) {
                const float4 xv = mine[(RING + slot) * CELLS + tid], f = dirs[par][2 * my_dir], e = dirs[par][2 * my_dir + 1];
                acc.x += fmaf(e.x, xv.x, f.x), acc.y += fmaf(e.y, xv.y, f.y), acc.z += fmaf(e.z, xv.z, f.z), acc.w += fmaf(e.w, xv.w, f.w);
            }
#pragma unroll
            for (int k = 0; k < BR; ++k) {
                const float4 *from = part + (par * BR + k) * 384;
                if (on_z) acc = add4(acc, from[pz]);
                if (on_y) acc = add4(acc, from[py]);
                if (on_x) acc = add4(acc, from[px]);
            }
            p.gx[(size_t)q * P + c] = acc;
        }
        if constexpr (S != NO_SUMS) {
            double sum[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
            const float4 m01 = quad_stats[slot][0], m23 = quad_stats[slot][1];
            const float mean[4] = {m01.x, m01.z, m23.x, m23.z}, rstd[4] = {m01.y, m01.w, m23.y, m23.w};
            auto add = [&](int i, float4 g, const float4 *at) {
                const float4 xv = at[RING * CELLS];
                const float gs[4] = {g.x, g.y, g.z, g.w}, xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float xh = (xs[s] - mean[s]) * rstd[s], gg = gs[s] * gm[i];
                    sum[s] += (double)gg;
                    sum[4 + s] += (double)(gg * xh);
                    dg[i] = fmaf(gs[s], xh, dg[i]);
                    db[i] += gs[s];
                }
            };
            add(0, acc, mine + slot * CELLS + tid);
            if (second) add(1, mine[slot * CELLS + THREADS + tid], mine + slot * CELLS + THREADS + tid);  // whole warps
            const double r = quad_reduce8(sum, lane);
            const int b = (q - q0) % QB;
            if ((lane & 3) == 0) red[b][warp][lane >> 2] = r;
            if (b == QB - 1 || q + 1 == q1) {
                __syncthreads();
                if (tid < (b + 1) * 8) {
                    double s = 0.0;
#pragma unroll
                    for (int k = 0; k < THREADS / 32; ++k) s += red[tid >> 3][k][tid & 7];
                    const int j = tid & 7;  // value j: a of samples 0..3, then c
                    reinterpret_cast<double *>(p.partials + (size_t)(4 * (q - b + (tid >> 3)) + (j & 3)) * gridDim.x + blk)[j >> 2] = s;
                }
            }
        }
        slot = slot == RING - 1 ? 0 : slot + 1;
    }
    if constexpr (S != NO_SUMS) {
        auto put = [&](size_t at, float *to, float v) { to[at] = p.accumulate ? to[at] + v : v; };
        if (gridDim.y == 1) {
            put(c, p.ggamma, dg[0]);
            put(c, p.gbeta, db[0]);
            if (second) {
                put(c2, p.ggamma, dg[1]);
                put(c2, p.gbeta, db[1]);
            }
            return;
        }
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        float *const own = reinterpret_cast<float *>(part);  // [2][512]; the partial sums of the borders have been read:
        __syncthreads();
        own[tid] = dg[0], own[512 + tid] = db[0];
        if (second) own[THREADS + tid] = dg[1], own[512 + THREADS + tid] = db[1];
        cluster.sync();
        for (unsigned i = blockIdx.y * THREADS + tid; i < 1024; i += gridDim.y * THREADS) {
            float s = 0.0f;
            for (unsigned r = 0; r < gridDim.y; ++r) s += *cluster.map_shared_rank(own + i, r);
            put(place(i & 511), i < 512 ? p.ggamma : p.gbeta, s);
        }
        cluster.sync();  // nobody leaves while its sums are being read
    }
}

// Block 4: one thread per cell of the region, all 27 taps; sources in the cell's own block carry a zero weight.
template <bool NORM>
__global__ void __launch_bounds__(512, 2) quad_border4_k(const float *__restrict__ w, const float4 *dsum, float4 *gx, const float4 *x_il4,
                                                         const float4 *hterm, int Q, int M, int N, int K, int qpc)
{
    using T = quadborder::Terms<4>;
    __shared__ float4 terms[NORM ? 2 : 1][2 * T::COUNT];
    using namespace quadborder;
    constexpr int THREADS = 512, SLOTS = 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4 *const tile = reinterpret_cast<float4 *>(smem_raw);  // [2][TS]
    const int tid = threadIdx.x;
    const int nbx = K >> 3, nby = N >> 3;
    const unsigned blk = blockIdx.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const long long origin = ((long long)(bz * 8 - 1) * N + (by * 8 - 1)) * K + (bx * 8 - 1);
    for (int i = tid; i < 2 * TS; i += THREADS) tile[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    int tof[SLOTS], rel[SLOTS];
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        const int i = tid + j * THREADS;
        tof[j] = -1;
        rel[j] = 0;
        if (i < TS) {
            const int cx = i % 10, cy = (i / 10) % 10, cz = i / 100;
            const int gz = bz * 8 + cz - 1, gy = by * 8 + cy - 1, gxx = bx * 8 + cx - 1;
            if (gz >= 0 && gz < M && gy >= 0 && gy < N && gxx >= 0 && gxx < K) {
                tof[j] = i;
                rel[j] = (cz * N + cy) * K + cx;
            }
        }
    }
    const int lz = tid >> 6, ly = (tid >> 3) & 7, lx = tid & 7;
    const int qz = lz & 3, qy = ly & 3, qx = lx & 3;
    const bool active = !(qz > 0 && qz < 3 && qy > 0 && qy < 3 && qx > 0 && qx < 3);  // the core of a block has no outside neighbour
    const int z = bz * 8 + lz, y = by * 8 + ly, x = bx * 8 + lx;
    const size_t c = ((size_t)z * N + y) * K + x;
    float wd[27];
#pragma unroll
    for (int t = 0; t < 27; ++t) {
        const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
        const int nz = z - dz, ny = y - dy, nx = x - dx;
        const bool other = active && ((nz >> 2) != (z >> 2) || (ny >> 2) != (y >> 2) || (nx >> 2) != (x >> 2)) && nz >= 0 && nz < M &&
                           ny >= 0 && ny < N && nx >= 0 && nx < K;
        wd[t] = other ? w[(size_t)t * P + ((size_t)nz * N + ny) * K + nx] : 0.0f;
    }
    const int tbase = (lz + 1) * 100 + (ly + 1) * 10 + (lx + 1);
    const int q0 = blockIdx.y * qpc, q1 = min(Q, q0 + qpc);
    const int my_term = NORM ? T::tile(tid >> 1, bx, by, bz, M, N, K) : -1;
    const size_t ntiles = (size_t)gridDim.x * 8;
    float4 pt = make_float4(0.f, 0.f, 0.f, 0.f), xnext = pt;
    float4 pf[SLOTS], gnext = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int q) {
        if (q < q1) {
            const float4 *src = dsum + (size_t)q * P + origin;
#pragma unroll
            for (int j = 0; j < SLOTS; ++j)
                if (tof[j] >= 0) pf[j] = src[rel[j]];
            if (NORM && my_term >= 0) pt = hterm[((size_t)q * ntiles + my_term) * 2 + (tid & 1)];
        }
    };
    previous_done();
    fetch(q0);
    if (active && q0 < q1) gnext = gx[(size_t)q0 * P + c];
    if (NORM && active && q0 < q1) xnext = x_il4[(size_t)q0 * P + c];
    __syncthreads();
    for (int q = q0; q < q1; ++q) {
        float4 *tl = tile + (q & 1) * TS;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j)
            if (tof[j] >= 0) tl[tof[j]] = pf[j];
        if (NORM && tid < 2 * T::COUNT) terms[q & 1][tid] = pt;
        fetch(q + 1);
        float4 acc = gnext;
        const float4 xv = xnext;
        if (active && q + 1 < q1) gnext = gx[(size_t)(q + 1) * P + c];
        if (NORM && active && q + 1 < q1) xnext = x_il4[(size_t)(q + 1) * P + c];
        __syncthreads();  // the other tile may still be read by slower threads; it is rewritten after the next barrier
        if (active) {
            if (NORM) acc = add4(acc, T::sum(terms[q & 1], lz, ly, lx, xv));
#pragma unroll
            for (int t = 0; t < 27; ++t) {
                const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
                acc = fma4(wd[t], tl[tbase - (dz * 100 + dy * 10 + dx)], acc);
            }
            gx[(size_t)q * P + c] = acc;
        }
    }
}

// ------------------------------------------------------------------------------------------ whole-grid norm
// Gradient of y = (x - mean) rstd gamma + beta, first pass: per sample a = sum g gamma and c = sum g gamma xhat, and the
// gradients of gamma and beta, which need no second look at the batch. A thread owns CPT cells and walks the quads. The
// eight sums of a quad are added in double from the single value on, as in norm_bwd_partial_k (norm.cu). SUB_G: the gradient is
// g - sub (residual form of the loop).
// On a small grid the quads are split over the CTAs of a cluster, which add up their gradients of gamma and beta in
// the order of their ranks (32^3 x 64: with its launch 14.1 us with one CTA for 16 quads, 11.6 with a cluster of eight that starts early).
template <int CPT, bool SUB_G>
__global__ void __launch_bounds__(256) quad_norm_sums_k(const float4 *x, const float4 *g, const float4 *sub, const float *gamma, const float2 *stats,
                                                        double2 *partials, int nparts, float *ggamma, float *gbeta, int accumulate, int Q,
                                                        int qpc, size_t P)
{
    constexpr int QB = 16;                     // quads between two block-wide sums
    constexpr int AT_ONCE = CPT == 1 ? 4 : 2;  // quads whose loads are in flight
    __shared__ double red[QB][8][8];
    __shared__ float part[2][CPT * 256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t c0 = (size_t)blockIdx.x * (256 * CPT) + tid;
    float gm[CPT], dg[CPT], db[CPT];
    previous_done();
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        gm[k] = c0 + k * 256 < P ? gamma[c0 + k * 256] : 0.0f;
        dg[k] = db[k] = 0.0f;
    }
    const int q0 = blockIdx.y * qpc, q1 = min(Q, q0 + qpc);
    for (int qb = q0; qb < q1; qb += QB) {
        const int qe = min(q1, qb + QB);
#pragma unroll AT_ONCE
        for (int q = qb; q < qe; ++q) {
            float4 xv[CPT], gv[CPT];
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const size_t i = (size_t)q * P + c0 + k * 256;
                xv[k] = gv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c0 + k * 256 < P) {
                    xv[k] = x[i];
                    gv[k] = g[i];
                    if (SUB_G) {
                        const float4 s = sub[i];
                        gv[k].x -= s.x, gv[k].y -= s.y, gv[k].z -= s.z, gv[k].w -= s.w;
                    }
                }
            }
            double v[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
            float2 mr[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) mr[s] = stats[4 * q + s];
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const float xs[4] = {xv[k].x, xv[k].y, xv[k].z, xv[k].w}, gs[4] = {gv[k].x, gv[k].y, gv[k].z, gv[k].w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float xh = (xs[s] - mr[s].x) * mr[s].y, gg = gs[s] * gm[k];
                    v[s] += (double)gg;
                    v[4 + s] += (double)(gg * xh);
                    dg[k] = fmaf(gs[s], xh, dg[k]);
                    db[k] += gs[s];
                }
            }
            const double r = quad_reduce8(v, lane);
            if ((lane & 3) == 0) red[q - qb][warp][lane >> 2] = r;
        }
        __syncthreads();
        for (int e = tid; e < (qe - qb) * 8; e += 256) {
            double s = 0.0;
#pragma unroll
            for (int w8 = 0; w8 < 8; ++w8) s += red[e >> 3][w8][e & 7];
            const int j = e & 7;  // value j: a of samples 0..3, then c
            reinterpret_cast<double *>(partials + (size_t)(4 * (qb + (e >> 3)) + (j & 3)) * nparts + blockIdx.x)[j >> 2] = s;
        }
        __syncthreads();
    }
    auto put = [&](size_t c, float *to, float v) {
        if (c < P) to[c] = accumulate ? to[c] + v : v;
    };
    if (gridDim.y == 1) {
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            put(c0 + k * 256, ggamma, dg[k]);
            put(c0 + k * 256, gbeta, db[k]);
        }
        return;
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        part[0][k * 256 + tid] = dg[k];
        part[1][k * 256 + tid] = db[k];
    }
    cluster.sync();
    for (unsigned i = blockIdx.y * 256 + tid; i < 2 * CPT * 256; i += gridDim.y * 256) {
        float v = 0.0f;
        for (unsigned r = 0; r < gridDim.y; ++r) v += *cluster.map_shared_rank(&part[0][0] + i, r);
        put((size_t)blockIdx.x * (256 * CPT) + i % (CPT * 256), i < CPT * 256 ? ggamma : gbeta, v);
    }
    cluster.sync();  // nobody leaves while its part is being read
}

// grid 4 Q: (a, c) / P from the partial sums, in a fixed order
__global__ void __launch_bounds__(256) quad_norm_ac_k(const double2 *partials, int nparts, float2 *ac, size_t P)
{
    __shared__ double red[33];
    previous_done();
    const double2 *ps = partials + (size_t)blockIdx.x * nparts;
    double a = 0.0, c = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nparts; i += 256) {
        const double2 v = ps[i];
        a += v.x;
        c += v.y;
    }
    a = block_sum(a, red);
    c = block_sum(c, red);
    if (threadIdx.x == 0) ac[blockIdx.x] = make_float2((float)(a / (double)P), (float)(c / (double)P));
}

// Residual form of the loop, backward: n = norm(h), h' = h + net(n) - n. gn = gradient that the step sent back to n;
// out = gu + rstd ((gn - gu) gamma - a - xhat c), gu = gradient of h'. out may be gu.
__global__ void __launch_bounds__(256) quad_norm_residual_apply_k(const float4 *h, const float4 *gn, const float4 *gu, const float *gamma,
                                                                  const float2 *stats, const float2 *ac, float4 *out, size_t P, unsigned parts)
{
    previous_done();
    const unsigned q = blockIdx.x / parts;
    const size_t c = (size_t)(blockIdx.x - q * parts) * 256 + threadIdx.x;
    if (c >= P) return;
    const size_t i = (size_t)q * P + c;
    const float gm = gamma[c];
    const float4 hv = h[i], nv = gn[i], uv = gu[i];
    const float hs[4] = {hv.x, hv.y, hv.z, hv.w}, ns[4] = {nv.x, nv.y, nv.z, nv.w}, us[4] = {uv.x, uv.y, uv.z, uv.w};
    float o[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float2 mr = stats[4 * q + s], k = ac[4 * q + s];
        const float xh = (hs[s] - mr.x) * mr.y;
        o[s] = us[s] + mr.y * ((ns[s] - us[s]) * gm - k.x - xh * k.y);
    }
    out[i] = make_float4(o[0], o[1], o[2], o[3]);
}

// Residual form, forward: out = h + (y - norm(h)), and the per-sample partial sums of out (out may be y). With y and out
// null only the sums of h are taken (the statistics of the loop's first input). As in norm_residual_combine_k and
// norm_partial_stats_k (norm.cu) four x-neighbours are added in float, everything above in double: neighbouring lanes hold
// neighbouring cells, and of the sums that four lanes then share each goes on with one sample's. P is a multiple of 512.
__global__ void __launch_bounds__(256) quad_residual_combine_k(const float4 *h, const float4 *y, const float *gamma, const float *beta,
                                                               const float2 *stats, float4 *out, double2 *partials, unsigned nparts, size_t P)
{
    constexpr int CPT = 4;
    __shared__ double red[8][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned q = blockIdx.x / nparts, part = blockIdx.x - q * nparts;
    const size_t c0 = (size_t)part * (256 * CPT) + tid;
    float2 mr[4];
    previous_done();
    if (y) {
#pragma unroll
        for (int s = 0; s < 4; ++s) mr[s] = stats[4 * q + s];
    }
    float o[CPT][4];
    {
        float4 hv[CPT], yv[CPT];
        float g[CPT], b[CPT];
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const size_t c = c0 + k * 256, i = (size_t)q * P + c;
            hv[k] = yv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            g[k] = b[k] = 0.0f;
            if (c < P) {  // the whole CTA
                hv[k] = h[i];
                if (y) {
                    yv[k] = y[i];
                    g[k] = gamma[c], b[k] = beta[c];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const size_t c = c0 + k * 256;
            const float hs[4] = {hv[k].x, hv[k].y, hv[k].z, hv[k].w}, ys[4] = {yv[k].x, yv[k].y, yv[k].z, yv[k].w};
#pragma unroll
            for (int s = 0; s < 4; ++s) o[k][s] = y ? hs[s] + (ys[s] - fmaf((hs[s] - mr[s].x) * mr[s].y, g[k], b[k])) : hs[s];
            if (y && c < P) out[(size_t)q * P + c] = make_float4(o[k][0], o[k][1], o[k][2], o[k][3]);
            if (c >= P) o[k][0] = o[k][1] = o[k][2] = o[k][3] = 0.0f;
        }
    }
    double sum = 0.0, squares = 0.0;  // of sample lane & 3
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        float a[4], b[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const float other = __shfl_xor_sync(0xffffffffu, o[k][s], 1), lo = lane & 1 ? other : o[k][s], hi = lane & 1 ? o[k][s] : other;
            a[s] = lo + hi;
            b[s] = fmaf(lo, lo, hi * hi);
            a[s] += __shfl_xor_sync(0xffffffffu, a[s], 2);
            b[s] += __shfl_xor_sync(0xffffffffu, b[s], 2);
        }
        sum += (double)(lane & 2 ? (lane & 1 ? a[3] : a[2]) : (lane & 1 ? a[1] : a[0]));
        squares += (double)(lane & 2 ? (lane & 1 ? b[3] : b[2]) : (lane & 1 ? b[1] : b[0]));
    }
#pragma unroll
    for (int m = 4; m < 32; m *= 2) {
        sum += __shfl_xor_sync(0xffffffffu, sum, m);
        squares += __shfl_xor_sync(0xffffffffu, squares, m);
    }
    if (lane < 4) {
        red[warp][lane] = sum;
        red[warp][4 + lane] = squares;
    }
    __syncthreads();
    if (tid < 8) {
        double s = 0.0;
#pragma unroll
        for (int w8 = 0; w8 < 8; ++w8) s += red[w8][tid];
        reinterpret_cast<double *>(partials + (size_t)(4 * q + (tid & 3)) * nparts + part)[tid >> 2] = s;
    }
}

// ------------------------------------------------------------------------------------------------ host side
template <typename Kern>
static int smem_once(Kern kern, int bytes, unsigned long long *mask, const char *what)
{
    if (!first_use_on_device(mask)) return GN_OK;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) {
        record_cuda_error(e, what);
        return GN_ERR_CUDA;
    }
    return GN_OK;
}

static long long regions_of(int M, int N, int K) { return (long long)(M / 8) * (N / 8) * (K / 8); }

template <int SUB, int ACT, quadrev::In IN>
static int launch_reverse_in(const QuadRevParams &p, unsigned ctas, cudaStream_t st)
{
    constexpr int smem = quadrev::Bytes<IN>::SMEM;
    static unsigned long long done = 0;
    const int rc = smem_once(quad_reverse_k<SUB, ACT, IN>, smem, &done, "cudaFuncSetAttribute(quad_reverse_k)");
    if (rc != GN_OK) return rc;
    launch_after(quad_reverse_k<SUB, ACT, IN>, ctas, 256, smem, st, p);
    return check_launch("quad_reverse");
}
template <int SUB, int ACT>
static int launch_reverse_one(const QuadRevParams &p, unsigned ctas, cudaStream_t st)
{
    if (p.tile_stats) return launch_reverse_in<SUB, ACT, quadrev::BLOCK_NORM>(p, ctas, st);
    return p.raw ? launch_reverse_in<SUB, ACT, quadrev::GRID_NORM>(p, ctas, st) : launch_reverse_in<SUB, ACT, quadrev::PLAIN>(p, ctas, st);
}

template <int SUB>
static int launch_reverse_sub(const QuadRevParams &p, unsigned ctas, int act, cudaStream_t st)
{
    switch (act) {
    case GN_ACT_RELU: return launch_reverse_one<SUB, GN_ACT_RELU>(p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_reverse_one<SUB, GN_ACT_LEAKY_RELU>(p, ctas, st);
    case GN_ACT_SILU: return launch_reverse_one<SUB, GN_ACT_SILU>(p, ctas, st);
    default: return launch_reverse_one<SUB, GN_ACT_TANH>(p, ctas, st);
    }
}

int launch_quad_reverse(const QuadReverse &a, int act, cudaStream_t st)
{
    QuadRevParams p{};
    p.packed = a.packed_t; p.params_old = a.params_old; p.g = a.g; p.raw = a.raw; p.stats = a.stats; p.ac = a.ac; p.h = a.h;
    p.wsum = a.wsum; p.tile_stats = a.tile_stats; p.hterm = a.hterm;
    p.delta = a.delta; p.dsum = a.dsum; p.gx = a.gx; p.dsq = a.dsq;
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = regions_of(a.M, a.N, a.K) * a.Q;
    long long ctas = (p.nitems + quad::QUARTERS - 1) / quad::QUARTERS;
    if (ctas > sm_count()) ctas = sm_count();
    p.unit = quad_split_unit(p.nitems, ctas, p.Q);
    return a.block == 8 ? launch_reverse_sub<8>(p, (unsigned)ctas, act, st) : launch_reverse_sub<4>(p, (unsigned)ctas, act, st);
}

// Into how many chunks the quads of a region go: as many as fill the two CTAs that an SM holds evenly. A chunk costs its CTA about
// two quads' time (tile latency, sums out) and its part of the gradient, 59 KB, is written and added up once.
static int wgrad_chunks(long long regions, int Q, int branches)
{
    const int c = pick_batch_chunks_balanced(regions * branches, Q, quadwg::CTAS, 2.0, 16);
    const int qpc = (Q + c - 1) / c;
    return (Q + qpc - 1) / qpc;
}

size_t quad_grad_floats(int M, int N, int K, int Q, int branches)
{
    const long long regions = regions_of(M, N, K);
    return (size_t)branches * wgrad_chunks(regions, Q, branches) * regions * quadwg::GRAD_F;
}

template <int SUB, int ACT, bool FUSE_IN, bool NORM, bool GATED = false>
static int launch_wgrad_in(const CUtensorMap &map, const QuadWgradParams &p, dim3 grid, cudaStream_t st)
{
    constexpr int smem = quadwg::Lay<SUB>::smem(FUSE_IN, NORM);
    static unsigned long long done = 0;
    const int rc = smem_once(quad_wgrad_k<SUB, ACT, FUSE_IN, NORM, GATED>, smem, &done, "cudaFuncSetAttribute(quad_wgrad_k)");
    if (rc != GN_OK) return rc;
    launch_after(quad_wgrad_k<SUB, ACT, FUSE_IN, NORM, GATED>, grid, quadwg::THREADS, smem, st, map, p);
    return check_launch("quad_wgrad");
}
template <int SUB, int ACT>
static int launch_wgrad_one(const CUtensorMap &map, const QuadWgradParams &p, dim3 grid, cudaStream_t st)
{
    if (p.tile_stats) return launch_wgrad_in<SUB, ACT, false, true>(map, p, grid, st);
    return p.in_stats ? launch_wgrad_in<SUB, ACT, true, false>(map, p, grid, st) : launch_wgrad_in<SUB, ACT, false, false>(map, p, grid, st);
}

template <int SUB>
static int launch_wgrad_sub(const CUtensorMap &map, const QuadWgradParams &p, dim3 grid, int act, cudaStream_t st)
{
    switch (act) {
    case GN_ACT_RELU: return launch_wgrad_one<SUB, GN_ACT_RELU>(map, p, grid, st);
    case GN_ACT_LEAKY_RELU: return launch_wgrad_one<SUB, GN_ACT_LEAKY_RELU>(map, p, grid, st);
    case GN_ACT_SILU: return launch_wgrad_one<SUB, GN_ACT_SILU>(map, p, grid, st);
    default: return launch_wgrad_one<SUB, GN_ACT_TANH>(map, p, grid, st);
    }
}

int launch_quad_wgrad(const QuadWgrad &a, int act, cudaStream_t st)
{
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (a.tile_stats && a.in_stats) return GN_ERR_UNSUPPORTED;
    const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, a.block);
    if (rc != GN_OK) return rc;
    QuadWgradParams p{};
    p.gbt = a.gbt; p.in_stats = a.in_stats; p.delta = a.delta; p.h = a.h; p.scale = a.scale; p.dsq = a.dsq; p.gpk = a.gpk;
    p.tile_stats = a.tile_stats; p.delta2 = a.delta2;
    p.accumulate = a.accumulate;
    p.error_flag = a.error_flag ? a.error_flag : device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    const long long regions = regions_of(a.M, a.N, a.K);
    const int branches = a.delta2 ? 2 : 1, chunks = wgrad_chunks(regions, a.Q, branches);
    p.qpc = (a.Q + chunks - 1) / chunks;
    const dim3 grid((unsigned)regions, (unsigned)chunks, branches);
    if (a.delta2) {
        if (a.block != 8 || a.tile_stats) return GN_ERR_UNSUPPORTED;
        return a.in_stats ? launch_wgrad_in<8, GN_ACT_RELU, true, false, true>(map, p, grid, st)
                          : launch_wgrad_in<8, GN_ACT_RELU, false, false, true>(map, p, grid, st);
    }
    return a.block == 8 ? launch_wgrad_sub<8>(map, p, grid, act, st) : launch_wgrad_sub<4>(map, p, grid, act, st);
}

int launch_quad_finish(const float *gpk, float *gw, float *gb, float *gs, const float *il, float *x, int B, int M, int N, int K, int block,
                       int branches, cudaStream_t st)
{
    const long long regions = regions_of(M, N, K);
    const int chunks = wgrad_chunks(regions, (B + 3) / 4, branches);
    const unsigned grads = (unsigned)(branches * ((regions + 1) / 2) * (116 / kUnpack)), parts = (unsigned)(((long long)M * N * K + 255) / 256);
    const unsigned long long n = grads + (il ? (unsigned long long)parts * ((B + 3) / 4) : 0);
    if (n >= 1ull << 31) return GN_ERR_UNSUPPORTED;
    const float4 *const i4 = reinterpret_cast<const float4 *>(il);
    if (block == 8) launch_after(quad_finish_k<8>, (unsigned)n, 256, 0, st, gpk, gw, gb, gs, i4, x, B, M, N, K, chunks, branches, grads, parts);
    else launch_after(quad_finish_k<4>, (unsigned)n, 256, 0, st, gpk, gw, gb, gs, i4, x, B, M, N, K, chunks, branches, grads, parts);
    return check_launch("quad_finish");
}

template <bool NORM, int BR, BorderSums S>
static int launch_border8(BorderParams p, cudaStream_t st)
{
    using R = quadborder::Room<NORM, BR, S>;
    const long long nb = regions_of(p.M, p.N, p.K);
    const int chunks = pick_batch_chunks_balanced(nb, p.Q, R::CTAS, 4.0, S == NO_SUMS ? 32 : 8);  // sums: a cluster
    p.qpc = (p.Q + chunks - 1) / chunks;
    const dim3 grid((unsigned)nb, (unsigned)((p.Q + p.qpc - 1) / p.qpc));
    static unsigned long long done = 0;
    const int rc = smem_once(quad_border8_k<NORM, BR, S>, R::BYTES, &done, "cudaFuncSetAttribute(quad_border8_k)");
    if (rc != GN_OK) return rc;
    launch_after_cluster(S == NO_SUMS ? 1 : grid.y, quad_border8_k<NORM, BR, S>, grid, 384, R::BYTES, st, p);
    return check_launch("quad_border");
}

template <bool NORM>
static int launch_border4(const BorderParams &p, cudaStream_t st)
{
    constexpr int smem = 2 * quadborder::TS * 16;
    const long long nb = regions_of(p.M, p.N, p.K);
    const int chunks = pick_batch_chunks_balanced(nb, p.Q, 2, 4.0, 32), qpc = (p.Q + chunks - 1) / chunks;
    const dim3 grid((unsigned)nb, (unsigned)((p.Q + qpc - 1) / qpc));
    static unsigned long long done = 0;
    const int rc = smem_once(quad_border4_k<NORM>, smem, &done, "cudaFuncSetAttribute(quad_border4_k)");
    if (rc != GN_OK) return rc;
    launch_after(quad_border4_k<NORM>, grid, 512, smem, st, p.w, p.dsum, p.gx, p.x, p.hterm, p.Q, p.M, p.N, p.K, qpc);
    return check_launch("quad_border");
}

// Whether the sums are better taken in the border pass: where a region per SM is all there is, a kernel is mostly its launch and its
// latency. us of a training loop of 2 x 8 iterations, apart / together: 32^3 (64 regions) x 16 460 / 454, x 64 689 / 657, x 128
// 1130 / 1093, gated x 64 1416 / 1377; 64^3 (512) x 4 636 / 647, x 16 1264 / 1270, x 64 3726 / 3724; 128^3 (4096) x 4 4228 / 4448. Two
// CTAs per SM instead of three, and eight times the warp sums per cell, are what it costs.
bool quad_border_takes_sums(int M, int N, int K, int block) { return block == 8 && regions_of(M, N, K) <= sm_count(); }

int launch_quad_border(const QuadBorder &a, cudaStream_t st)
{
    BorderParams p{};
    p.w = a.w; p.dsum = reinterpret_cast<const float4 *>(a.dsum); p.dsum2 = reinterpret_cast<const float4 *>(a.dsum2);
    p.gx = reinterpret_cast<float4 *>(a.gx); p.x = reinterpret_cast<const float4 *>(a.x_il4); p.hterm = a.hterm;
    p.gamma = a.gamma; p.stats = a.stats; p.partials = a.partials;
    p.ggamma = a.ggamma; p.gbeta = a.gbeta; p.accumulate = a.accumulate;
    p.Q = a.Q; p.M = a.M; p.N = a.N; p.K = a.K;
    const bool sums = a.gamma != nullptr;
    if ((a.dsum2 && (a.block != 8 || a.hterm)) || (sums && (a.block != 8 || a.hterm))) return GN_ERR_UNSUPPORTED;
    if (a.block == 4) return a.hterm ? launch_border4<true>(p, st) : launch_border4<false>(p, st);
    if (!sums) {
        if (a.hterm) return launch_border8<true, 1, NO_SUMS>(p, st);
        return a.dsum2 ? launch_border8<false, 2, NO_SUMS>(p, st) : launch_border8<false, 1, NO_SUMS>(p, st);
    }
    const int rc = a.dsum2 ? launch_border8<false, 2, SUMS>(p, st) : launch_border8<false, 1, SUMS>(p, st);
    if (rc != GN_OK) return rc;
    const long long P = (long long)a.M * a.N * a.K;
    launch_after(quad_norm_ac_k, 4 * a.Q, 256, 0, st, (const double2 *)a.partials, (int)regions_of(a.M, a.N, a.K), a.ac, (size_t)P);
    return check_launch("quad_norm_ac");
}

int quad_norm_parts(long long P)
{
    // four cells per thread where that still gives every SM a few CTAs, else one
    return (int)(P >= 4LL * 256 * 4 * sm_count() ? (P + 1023) / 1024 : (P + 255) / 256);
}

int launch_quad_norm_sums(const float *x, const float *g, const float *sub, const float *gamma, const float2 *stats, double2 *partials,
                          float *ggamma, float *gbeta, int accumulate, float2 *ac, int Q, long long P, cudaStream_t st)
{
    const int nparts = quad_norm_parts(P);
    const float4 *x4 = reinterpret_cast<const float4 *>(x), *g4 = reinterpret_cast<const float4 *>(g), *s4 = reinterpret_cast<const float4 *>(sub);
    const bool wide = (long long)nparts * 256 < P;
    // enough CTAs for a few per SM, by splitting the quads where the cells do not give them
    int chunks = 1;
    while (chunks < 8 && 2 * chunks <= Q && (long long)nparts * chunks < 4LL * sm_count()) chunks *= 2;
    const int qpc = (Q + chunks - 1) / chunks;
#define SUMS_(C, S)                                                                                                                     \
    launch_after_cluster(chunks, quad_norm_sums_k<C, S>, dim3(nparts, chunks), 256, 0, st, x4, g4, s4, gamma, stats, partials, nparts, \
                         ggamma, gbeta, accumulate, Q, qpc, (size_t)P)
    if (wide && sub) SUMS_(4, true);
    else if (wide) SUMS_(4, false);
    else if (sub) SUMS_(1, true);
    else SUMS_(1, false);
#undef SUMS_
    launch_after(quad_norm_ac_k, 4 * Q, 256, 0, st, partials, nparts, ac, (size_t)P);
    return check_launch("quad_norm_sums");
}

int launch_quad_norm_residual_apply(const float *h, const float *gn, const float *gu, const float *gamma, const float2 *stats, const float2 *ac,
                                    float *out, int Q, long long P, cudaStream_t st)
{
    const unsigned parts = (unsigned)((P + 255) / 256);
    if ((unsigned long long)parts * Q >= 1ull << 31) return GN_ERR_UNSUPPORTED;
    launch_after(quad_norm_residual_apply_k, parts * (unsigned)Q, 256, 0, st, reinterpret_cast<const float4 *>(h), reinterpret_cast<const float4 *>(gn),
                 reinterpret_cast<const float4 *>(gu), gamma, stats, ac, reinterpret_cast<float4 *>(out), (size_t)P, parts);
    return check_launch("quad_norm_residual_apply");
}

int quad_combine_parts(long long P) { return (int)((P + 1023) / 1024); }

int launch_quad_residual_combine(const float *h, const float *y, const float *gamma, const float *beta, const float2 *stats, float *out,
                                 double2 *partials, int Q, long long P, cudaStream_t st)
{
    const unsigned parts = (unsigned)quad_combine_parts(P);
    if ((unsigned long long)parts * Q >= 1ull << 31) return GN_ERR_UNSUPPORTED;
    launch_after(quad_residual_combine_k, parts * (unsigned)Q, 256, 0, st, reinterpret_cast<const float4 *>(h), reinterpret_cast<const float4 *>(y), gamma,
                 beta, stats, reinterpret_cast<float4 *>(out), partials, parts, (size_t)P);
    return check_launch("quad_residual_combine");
}

}  // namespace gn
