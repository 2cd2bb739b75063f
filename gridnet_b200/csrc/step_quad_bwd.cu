// Backward of the block-local update with the quad mapping (float, block 8 and 4, per-block normalisation off): the
// decomposition of step_bwd_fast.cu on the layout and the work split of step_quad.cu.
//
//   reverse  quad_reverse_k: walks the inner iterations backwards. delta_t = act'(h_t) g s; what flows back inside a block
//            is the 27-tap sum over the delta tile with transposed weights, read from tensor memory. The gradient of the
//            whole-grid normalisation that follows the step is applied to g on the way in, so the normalised gradient
//            never exists in memory.
//   wgrad    quad_wgrad_k: dW[n][t] += x_t[n + o_t] delta_t[n]. The 432 sums per lane live in tensor memory and are
//            read, added to and written back twelve at a time; a team's two warps work on the same item, each on one half
//            of the window rows. Sums go to the slot of (region, team) and are added up in team order by
//            quad_unpack_grads_k: no atomics, the same bits every time.
//   border   quad_border_k: the part of grad_x that crosses block borders, from the per-neuron sums of deltas.
//   norms    quad_norm_sums_k: one pass over the step's output and the gradient of its normalised form gives the
//            per-sample sums of the LayerNorm gradient and the gradients of its weight and bias.
//
// Reference semantics: the gradient of gridnet/backend_torch.py:61-142 with normalize=False and of
// torch.nn.LayerNorm((M,N,K)) (gridnet/scripts/train_mnist.py:54,62-64); the kernel this stands in for is
// gridnet_cuda_backward_kernel, src/gridnet_cuda_kernels.cu:202-450.
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
// Before an item, the gradient of its output is fetched into the tile's own cells; pre-activations arrive in a staging area.
constexpr int ROW = 10, PLANE = 80, CELLS = 800, TILE_BYTES = CELLS * 16, STAGE_BYTES = 512 * 16;
constexpr int WARP_BYTES = TILE_BYTES + STAGE_BYTES, TEAM = 2;
constexpr int SMEM_BYTES = 4 * TEAM * WARP_BYTES;
}  // namespace quadrev

struct QuadRevParams {
    const float *packed;           // transposed weights; NORM_IN: the norm's weight in the place of the biases
    const float *g;                // gradient of the step's output (NORM_IN: of its normalised output), IL4
    const float *raw;              // NORM_IN: the step's output, IL4
    const float2 *stats, *ac;      // NORM_IN: [4 Q] (mean, rstd) and (sum g gamma, sum g gamma xhat) / P
    const float *h;                // [inner] pre-activations, IL4
    float *delta, *dsum, *gx;      // [inner], one, one IL4 tensors
    float *dsq;                    // [Q][P] gradient terms of the residual scale, summed over the quad and the iterations
    int M, N, K, Q, inner;
    long long nitems;
};

template <int ACT>
__device__ __forceinline__ void act_both2(u64 h, u64 &f, u64 &d)
{
    if (ACT == GN_ACT_SILU) {
        const u64 t = fmul2(h, pack2(-1.4426950408889634f, -1.4426950408889634f));
        float t0, t1, e0, e1, r0, r1, d0, d1;
        unpack2(t, t0, t1);
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
        unpack2(fadd2(pack2(e0, e1), pack2(1.0f, 1.0f)), d0, d1);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
        const u64 r = pack2(r0, r1);
        f = fmul2(h, r);
        d = ffma2r(f, ffma2r(r, pack2(-1.0f, -1.0f), pack2(1.0f, 1.0f)), r);  // sg (1 + h (1 - sg))
        return;
    }
    float h0, h1, f0, f1, d0, d1;
    unpack2(h, h0, h1);
    Act<ACT, float>::both(h0, f0, d0);
    Act<ACT, float>::both(h1, f1, d1);
    f = pack2(f0, f1);
    d = pack2(d0, d1);
}

template <int SUB, int ACT, bool NORM_IN>
__global__ void __launch_bounds__(256, 1) quad_reverse_k(const QuadRevParams p)
{
    using namespace quad;
    using namespace quadrev;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    const unsigned tile = smem_u32(smem) + warp * WARP_BYTES, stage = tile + TILE_BYTES;
    for (int c = lane; c < CELLS; c += 32) sts128u(tile + c * 16, 0, 0);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<SUB> L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K, T4 = (size_t)p.Q * P * 4;  // floats of an IL4 tensor
    const long long worker = (long long)blockIdx.x * QUARTERS + quarter, nworkers = (long long)gridDim.x * QUARTERS;
    const long long n0 = p.nitems * worker / nworkers;
    const int cnt = (int)(p.nitems * (worker + 1) / nworkers - n0);
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
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        return ((size_t)q * P + ((size_t)(bz * 8) * p.N + by * 8) * p.K + bx * 8) * 4;
    };
    auto fetch_h = [&](size_t corner, int t) { quad_stage<0, 8>(stage, p.h + (size_t)t * T4 + corner, zstr, p.K, lane); };
    auto fetch_g = [&](size_t corner) {
        const int y = lane >> 3, x = lane & 7;
        const float *src = p.g + corner + ((long long)y * p.K + x) * 4;
#pragma unroll
        for (int k = 0; k < 16; ++k)
            cp_async16(tile + (unsigned)(((k >> 1) + 1) * PLANE + (y + 4 * (k & 1)) * ROW + x + 1) * 16u, src + (k & 1) * 16ll * p.K + (k >> 1) * zstr);
    };
    auto prefetch_rows = [&](const float *t, size_t corner) {  // a region's 64 rows of 128 bytes on their way to L2
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int r = lane + 32 * k;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(t + corner + (r >> 3) * zstr + (long long)(r & 7) * p.K * 4));
        }
    };
    const size_t to_own = (((size_t)L.z0 * p.N + L.y0) * p.K + 4 * L.h) * 4;  // corner -> this lane's cells
    __syncwarp();
    if (role < cnt) {
        fetch_g(corner_of(role));
        fetch_h(corner_of(role), p.inner - 1);
    }

    int blk = (int)(n0 / p.Q), q0 = (int)(n0 - (long long)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);
        if (i0 > 0) {
            tmem_fence_before();
            team_sync<TEAM>(quarter);
            tmem_fence_after();
        }
        quad_load_params(p.packed + (size_t)blk * PACK_F, role, lane, tm);
        tmem_wait_st();
        tmem_fence_before();
        team_sync<TEAM>(quarter);
        tmem_fence_after();
        if (i0 + here < cnt) {
            const unsigned char *nx = reinterpret_cast<const unsigned char *>(p.packed + (size_t)(blk + 1) * PACK_F);
            for (int c = role * 32 + lane; c < PACK_F * 4 / 128; c += 32 * TEAM) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c * 128));
            __syncwarp();
        }
        for (int k = (role + TEAM - i0 % TEAM) % TEAM; k < here; k += TEAM) {
            const int i = i0 + k, q = q0 + k;
            const size_t corner = corner_of(i), own = corner + to_own;
            u64 g[4][4][2], dsum[4][4][2];
            float dsa[4][4];
            u64 r[4][4][2];
            if (NORM_IN) quad_load(p.raw + own, zstr, ystr, L.h, r);
            if (i + TEAM < cnt) {
                const size_t next = corner_of(i + TEAM);
                prefetch_rows(p.g, next);
                if (NORM_IN) prefetch_rows(p.raw, next);
            }
            cp_async_wait_all();
            __syncwarp();
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int o = 0; o < 4; ++o) lds128u(own_cell(n, o), g[n][o][0], g[n][o][1]);
            if (NORM_IN) {
                // gradient of (x - mean) rstd gamma + beta: rstd (g gamma - a - xhat c)
                u64 mu[2], rs[2], ma[2], mc[2];
#pragma unroll
                for (int k2 = 0; k2 < 2; ++k2) {
                    const float2 m0 = p.stats[4 * q + 2 * k2], m1 = p.stats[4 * q + 2 * k2 + 1];
                    const float2 a0 = p.ac[4 * q + 2 * k2], a1 = p.ac[4 * q + 2 * k2 + 1];
                    mu[k2] = pack2(-m0.x, -m1.x);
                    rs[k2] = pack2(m0.y, m1.y);
                    ma[k2] = pack2(-a0.x, -a1.x);
                    mc[k2] = pack2(-a0.y, -a1.y);
                }
                float gm[16];
                tmem_ld16(tm + COL_BIAS, gm);
                tmem_wait_ld16(gm);
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o)
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            const u64 xh = fmul2(fadd2(r[n][o][k2], mu[k2]), rs[k2]);
                            const u64 gg = ffma2r(g[n][o][k2], pack2(gm[n * 4 + o], gm[n * 4 + o]), ma[k2]);
                            g[n][o][k2] = fmul2(ffma2r(xh, mc[k2], gg), rs[k2]);
                        }
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    dsum[n][o][0] = dsum[n][o][1] = 0;
                    dsa[n][o] = 0.0f;
                }
            for (int t = p.inner - 1; t >= 0; --t) {
                float sc[16];
                tmem_ld16(tm + COL_SCALE, sc);
                cp_async_wait_all();
                tmem_wait_ld16(sc);
                __syncwarp();  // everyone's part of h_t has landed
                float *const dt = p.delta + (size_t)t * T4 + own;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    u64 dl[4][2];
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        u64 h0, h1, f0, f1, d0, d1;
                        lds128u(stage + S.at(n, o), h0, h1);
                        act_both2<ACT>(h0, f0, d0);
                        act_both2<ACT>(h1, f1, d1);
                        float s0, s1;
                        unpack2(ffma2r(f0, g[n][o][0], fmul2(f1, g[n][o][1])), s0, s1);
                        dsa[n][o] += s0 + s1;
                        const u64 s2 = pack2(sc[n * 4 + o], sc[n * 4 + o]);
                        dl[o][0] = fmul2(fmul2(d0, g[n][o][0]), s2);
                        dl[o][1] = fmul2(fmul2(d1, g[n][o][1]), s2);
                        dsum[n][o][0] = fadd2(dsum[n][o][0], dl[o][0]);
                        dsum[n][o][1] = fadd2(dsum[n][o][1], dl[o][1]);
                        sts128u(own_cell(n, o), dl[o][0], dl[o][1]);
                    }
                    quad_store2(dt, n, 0, zstr, ystr, L.h, dl);
                    quad_store2(dt, n, 1, zstr, ystr, L.h, dl);
                }
                __syncwarp();  // the delta tile is complete, h_t has been read
                if (t > 0) fetch_h(corner, t - 1);
                else if (i + TEAM < cnt) fetch_h(corner_of(i + TEAM), p.inner - 1);
                quad_stencil<PLANE, false>(rows, dx, tm, g, [](int, int, float, u64, u64) {});
                __syncwarp();  // ... and has been read
            }
            if (i + TEAM < cnt) fetch_g(corner_of(i + TEAM));
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
// What a team has in shared memory: tiles of the step's input with its halo (block 8: two, which take turns over the
// inner iterations so that one barrier per iteration is enough; block 4: one, updated in place between two), two staging
// areas for deltas and one for pre-activations.
namespace quadwg {
constexpr int TEAM = 2, STAGE_BYTES = 512 * 16;
template <int SUB>
struct Lay {
    static constexpr int NT = SUB == 8 ? 2 : 1;
    static constexpr int TEAM_BYTES = NT * QuadGeo<SUB>::BUF_BYTES + 3 * STAGE_BYTES;
    static constexpr int SMEM = 4 * TEAM_BYTES;
};
}  // namespace quadwg

struct QuadWgradParams {
    const float2 *gbt;       // FUSE_IN: as in step_fwd_quad
    const float2 *in_stats;
    const float *delta, *h;  // [inner] IL4
    const float *scale;      // [M][N][K]
    const float *dsq;        // [Q][P]
    float *gpk;              // [slots][regions][PACK_F]
    int accumulate;          // add to what the slots hold
    int *error_flag;
    int M, N, K, Q, inner, regions;
    long long nitems;
};

// first team that works on an item >= n, when nitems items are cut into nteams contiguous ranges
__host__ __device__ __forceinline__ long long quad_team_of(long long n, long long nitems, long long nteams)
{
    return ((n + 1) * nteams - 1) / nitems;
}

// The sums of a warp: half of the window rows. In the two inner row pairs (ry = 1, 2) a window row is read by both neuron
// rows dy = 0, 1: their sums are neighbours in tensor memory ("pair units", 24 columns: [c][o][dy]) and take packed FMAs
// with the cell's value as the scalar operand. The outer rows (ry = 0, 3) serve one neuron row ("single units", 12
// columns: [c][o]). Half 0: six single units, then six pair units; half 1 the other way round.
template <int COLS>
__device__ __forceinline__ void quad_ld_cols(unsigned a, float *r)
{
    if (COLS == 24) {
        tmem_ld16(a, r);
        tmem_ld8(a + 16, r + 16);
    } else {
        tmem_ld8(a, r);
        tmem_ld4(a + 8, r + 8);
    }
}

// One iteration: every sum += window cell * delta, four samples. dp[dz][o][s]: deltas of (dy = 0, dy = 1).
// Bound by FMA issue: 288 packed and 288 scalar FMAs per warp. Three register buffers per unit in flight: a unit's sums
// are asked for while the one before is worked on and are still being written back while the next one is.
template <int PLANE, int HALF>
__device__ __forceinline__ void quad_wgrad_rows(const unsigned (&rows)[4], int dx, unsigned tm, const u64 (&dp)[2][4][4])
{
    const unsigned t0 = tm + HALF * 216;
    float wb[2][24];
    tmem_wait_st();  // the previous iteration's sums are in place
    if (HALF == 0) quad_ld_cols<12>(t0, wb[0]);
    else quad_ld_cols<24>(t0, wb[0]);
    int unit = 0, col = 0;
#pragma unroll
    for (int ry = 2 * HALF; ry < 2 * HALF + 2; ++ry) {
        const bool pair = ry == 1 || ry == 2;
        unsigned a6[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) a6[j] = rows[ry] + (unsigned)(j * dx);
#pragma unroll
        for (int rz = 0; rz < 4; ++rz) {
            float4 v[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) v[j] = lds128(a6[j] + rz * PLANE * 16u);
#pragma unroll
            for (int dz = 0; dz < 2; ++dz) {
                if (rz - dz < 0 || rz - dz > 2) continue;
                float *wp = wb[unit % 2], *wn = wb[(unit + 1) % 2];
                const int cols = pair ? 24 : 12, next = col + cols;
                tmem_wait_ld12(wp);
                if (pair) tmem_use12(wp + 12);
                if (unit + 1 < 12) {
                    const bool next_pair = HALF == 0 ? unit + 1 >= 6 : unit + 1 < 6;
                    if (next_pair) quad_ld_cols<24>(t0 + next, wn);
                    else quad_ld_cols<12>(t0 + next, wn);
                }
                if (pair) {
                    u64 acc[12];
#pragma unroll
                    for (int k = 0; k < 12; ++k) acc[k] = pack2(wp[2 * k], wp[2 * k + 1]);
#pragma unroll
                    for (int s = 0; s < 4; ++s)
#pragma unroll
                        for (int c = 0; c < 3; ++c)
#pragma unroll
                            for (int o = 0; o < 4; ++o) {
                                const float4 &vv = v[o + c];
                                const float x = s == 0 ? vv.x : (s == 1 ? vv.y : (s == 2 ? vv.z : vv.w));
                                ffma2(acc[c * 4 + o], dp[dz][o][s], pack2(x, x));
                            }
#pragma unroll
                    for (int k = 0; k < 12; ++k) unpack2(acc[k], wp[2 * k], wp[2 * k + 1]);
                    tmem_st16(t0 + col, wp);
                    tmem_st8(t0 + col + 16, wp + 16);
                } else {
#pragma unroll
                    for (int s = 0; s < 4; ++s)
#pragma unroll
                        for (int c = 0; c < 3; ++c)
#pragma unroll
                            for (int o = 0; o < 4; ++o) {
                                const float4 &vv = v[o + c];
                                const float x = s == 0 ? vv.x : (s == 1 ? vv.y : (s == 2 ? vv.z : vv.w));
                                float lo, hi;
                                unpack2(dp[dz][o][s], lo, hi);
                                wp[c * 4 + o] = fmaf(x, HALF == 0 ? lo : hi, wp[c * 4 + o]);
                            }
                    tmem_st8(t0 + col, wp);
                    tmem_st4(t0 + col + 8, wp + 8);
                }
                ++unit;
                col = next;
            }
        }
    }
}

// 72 of a warp's 216 sums (six single units, or three pair units) -> (or onto) 18 vectors of the packed gradient
template <bool PAIR>
__device__ __forceinline__ void quad_flush72(float4 *o, unsigned col, bool accumulate)
{
    float r[72];
    float4 old[18];
#pragma unroll
    for (int k = 0; k < 3; ++k) quad_ld_cols<24>(col + k * 24, r + k * 24);
#pragma unroll
    for (int v = 0; v < 18; ++v) old[v] = accumulate ? o[v * 32] : make_float4(0.f, 0.f, 0.f, 0.f);
    tmem_wait_ld12(r);
#pragma unroll
    for (int k = 1; k < 6; ++k) tmem_use12(r + 12 * k);
#pragma unroll
    for (int v = 0; v < 18; ++v) {
        // pair unit j: vectors 6 j + 3 dy + c, columns 24 j + (4 c + o) 2 + dy
        const int j = v / 6, dy = v % 6 / 3, c = v % 3;
        float e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = PAIR ? r[24 * j + (4 * c + i) * 2 + dy] : r[4 * v + i];
        o[v * 32] = make_float4(e[0] + old[v].x, e[1] + old[v].y, e[2] + old[v].z, e[3] + old[v].w);
    }
}

template <int SUB, int ACT, bool FUSE_IN>
__global__ void __launch_bounds__(256, 1) quad_wgrad_k(const __grid_constant__ CUtensorMap in_map, const QuadWgradParams p)
{
    using namespace quad;
    using G = QuadGeo<SUB>;
    using Y = quadwg::Lay<SUB>;
    constexpr int TEAM = quadwg::TEAM, NT = Y::NT, SB = quadwg::STAGE_BYTES;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[QUARTERS * NT];
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid == 0) {
        for (int i = 0; i < QUARTERS * NT; ++i) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<SUB> L(lane);
    const QuadStage<SUB> S(L);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K, T4 = (size_t)p.Q * P * 4;
    const long long nteams = (long long)gridDim.x * QUARTERS, team = (long long)blockIdx.x * QUARTERS + quarter;
    const long long n0 = p.nitems * team / nteams;
    const int cnt = (int)(p.nitems * (team + 1) / nteams - n0);
    const unsigned tiles = smem_u32(smem) + quarter * Y::TEAM_BYTES;
    const unsigned stage_d = tiles + NT * G::BUF_BYTES, stage_h = stage_d + 2 * SB;
    const unsigned bar0 = smem_u32(&bars[quarter * NT]);
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K, zstr = wzs * 4;
    const int dx = L.xsgn * 16;
    const unsigned own0 = (unsigned)(L.cell0 * 16 + dx + L.ysgn * G::ROW * 16) + G::PLANE * 16u;  // own cell (0, 0, 0) in a tile
    bool failed = false;

    // normalise pass: this thread's cells are first, first + 64, ...; which of them are halo (kept in both tiles)
    const int first = role * 32 + lane;
    constexpr int STEPS = (G::CELLS + 63) / 64;
    unsigned halo = 0;
    if (NT == 2) {
        for (int c = 0; c < STEPS; ++c) {
            int cz, cy, cx;
            G::cell(first + 64 * c, cz, cy, cx);
            if (cz == 0 || cz == 9 || cy == 0 || cy == 9 || cx == 0 || cx == 9) halo |= 1u << c;
        }
    }

    auto issue = [&](int i, int buf) {  // one lane: tile of item i
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const unsigned tile = tiles + buf * G::BUF_BYTES, bar = bar0 + 8 * buf;
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
    auto corner_of = [&](int i) {
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        return ((size_t)q * P + ((size_t)(bz * 8) * p.N + by * 8) * p.K + bx * 8) * 4;
    };
    // Deltas of iteration t -> staging area `buf`: each warp brings half of the planes, the team barrier shares them.
    // Pre-activations h_t: each warp the planes whose neurons it updates (dz = role), for itself alone.
    auto fetch_d = [&](size_t corner, int t, int buf) {
        quad_stage4(stage_d + buf * SB, p.delta + (size_t)t * T4 + corner, zstr, p.K, lane, role * 4, 1);
    };
    auto fetch_h = [&](size_t corner, int t) {
        quad_stage4(stage_h, p.h + (size_t)t * T4 + corner, zstr, p.K, lane, role, 2);
    };
    int buf_x = 0, buf_d = 0;     // tile and delta area of the iteration at hand
    unsigned landed[NT] = {};     // phases of the tile barriers
    if (cnt > 0) {
        if (role == 0 && lane == 0) issue(0, 0);
        __syncwarp();
        fetch_d(corner_of(0), 0, 0);
        if (p.inner > 1) fetch_h(corner_of(0), 0);
    }

    int blk = (int)(n0 / p.Q), q0 = (int)(n0 - (long long)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + L.z0) * p.N + (by * 8 + L.y0)) * p.K + bx * 8 + (L.h ? 7 : 0);
        {
            float z[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) z[k] = 0.0f;
#pragma unroll
            for (int k = 0; k < 13; ++k) tmem_st16(tm + role * 216 + k * 16, z);
            tmem_st8(tm + role * 216 + 208, z);
        }
        float dacc[4][4];  // role 0: bias gradient, role 1: gradient of the residual scale
        float sc[2][4];    // scales of the neurons this warp updates between iterations
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int o = 0; o < 4; ++o) dacc[n][o] = 0.0f;
        if (p.inner > 1) {
#pragma unroll
            for (int dy = 0; dy < 2; ++dy)
#pragma unroll
                for (int o = 0; o < 4; ++o) sc[dy][o] = __ldg(p.scale + g0 + role * wzs + dy * wys + o * L.xsgn);
        }

        for (int k = 0; k < here; ++k) {
            const int i = i0 + k, q = q0 + k;
            const size_t corner = corner_of(i);
            if (role == 1) {
                const float *dq = p.dsq + corner / 4 + ((size_t)L.z0 * p.N + L.y0) * p.K + 4 * L.h;
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float4 v = *reinterpret_cast<const float4 *>(dq + (n >> 1) * wzs + (n & 1) * wys);
                    dacc[n][0] += L.h ? v.w : v.x;
                    dacc[n][1] += L.h ? v.z : v.y;
                    dacc[n][2] += L.h ? v.y : v.z;
                    dacc[n][3] += L.h ? v.x : v.w;
                }
            }
            {
                const unsigned tile = tiles + buf_x * G::BUF_BYTES, other = tiles + (buf_x ^ 1) * G::BUF_BYTES;
                constexpr int BATCH = SUB == 8 ? 16 : 14;
                float2 g2[FUSE_IN ? BATCH : 1];
                const float2 *gp = FUSE_IN ? p.gbt + (size_t)blk * G::CELLS + first : nullptr;
                u64 na[2], nb[2];
                if (FUSE_IN) {  // (gamma, beta) of the first batch: in flight while the tile is waited for
#pragma unroll
                    for (int c = 0; c < BATCH; ++c)
                        if (c * 64 + first < G::CELLS) g2[c] = ld_pinned2(reinterpret_cast<const float *>(gp + c * 64));
                    float2 mr[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) mr[s] = p.in_stats[4 * q + s];
                    na[0] = pack2(mr[0].y, mr[1].y);
                    na[1] = pack2(mr[2].y, mr[3].y);
                    nb[0] = pack2(-mr[0].x * mr[0].y, -mr[1].x * mr[1].y);
                    nb[1] = pack2(-mr[2].x * mr[2].y, -mr[3].x * mr[3].y);
                }
                if (!mbar_wait_bounded(bar0 + 8 * buf_x, landed[buf_x] & 1u, kSpinLimit)) failed = true;
                if (NT == 1 || buf_x == 0) ++landed[0];
                else ++landed[NT - 1];
                __syncwarp();
                if (NT == 2 && p.inner > 1) team_sync<TEAM>(quarter);  // nobody reads the other tile any more: it gets the new halo
                if (FUSE_IN || (NT == 2 && p.inner > 1)) {
#pragma unroll 1
                    for (int c0 = 0; c0 < STEPS; c0 += BATCH) {
                        const unsigned a = (unsigned)(c0 * 64 + first) * 16u;
                        u64 v[BATCH][2];
#pragma unroll
                        for (int c = 0; c < BATCH; ++c)
                            if ((c0 + c) * 64 + first < G::CELLS) {
                                if (FUSE_IN && c0 > 0) g2[c] = ld_pinned2(reinterpret_cast<const float *>(gp + (c0 + c) * 64));
                                lds128u(tile + a + c * 1024, v[c][0], v[c][1]);
                            }
#pragma unroll
                        for (int c = 0; c < BATCH; ++c)
                            if ((c0 + c) * 64 + first < G::CELLS) {
                                if (FUSE_IN) {
                                    const u64 gg = pack2(g2[c].x, g2[c].x), bb = pack2(g2[c].y, g2[c].y);
                                    v[c][0] = ffma2r(ffma2r(v[c][0], na[0], nb[0]), gg, bb);
                                    v[c][1] = ffma2r(ffma2r(v[c][1], na[1], nb[1]), gg, bb);
                                    sts128u(tile + a + c * 1024, v[c][0], v[c][1]);
                                }
                                if (NT == 2 && p.inner > 1 && (halo >> (c0 + c) & 1u)) sts128u(other + a + c * 1024, v[c][0], v[c][1]);
                            }
                    }
                }
            }
            for (int t = 0; t < p.inner; ++t) {
                const bool last = t + 1 == p.inner;
                const unsigned tile = tiles + buf_x * G::BUF_BYTES;
                cp_async_wait_all();
                __syncwarp();
                team_sync<TEAM>(quarter);  // staged data and the tile's new values are visible; nobody is an iteration behind
                u64 dp[2][4][4];
#pragma unroll
                for (int dz = 0; dz < 2; ++dz)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        const float4 a = lds128(stage_d + buf_d * SB + S.at(dz * 2, o)), b = lds128(stage_d + buf_d * SB + S.at(dz * 2 + 1, o));
                        dp[dz][o][0] = pack2(a.x, b.x);
                        dp[dz][o][1] = pack2(a.y, b.y);
                        dp[dz][o][2] = pack2(a.z, b.z);
                        dp[dz][o][3] = pack2(a.w, b.w);
                    }
                // the activations that this warp's neurons turn into: block 8 those of iteration t + 1, into the other tile;
                // block 4 those of iteration t, in place
                if (NT == 2 ? !last : t > 0) {
                    const unsigned to = NT == 2 ? tiles + (buf_x ^ 1) * G::BUF_BYTES : tile;
#pragma unroll
                    for (int dy = 0; dy < 2; ++dy)
#pragma unroll
                        for (int o = 0; o < 4; ++o) {
                            const unsigned c = own0 + (unsigned)(dy * L.ysgn * G::ROW * 16 + o * dx) + role * (G::PLANE * 16u);
                            u64 h0, h1, x0, x1;
                            lds128u(stage_h + S.at(role * 2 + dy, o), h0, h1);
                            lds128u(tile + c, x0, x1);
                            sts128u(to + c, act_residual2<ACT>(h0, sc[dy][o], x0), act_residual2<ACT>(h1, sc[dy][o], x1));
                        }
                    __syncwarp();
                }
                if (NT == 1) team_sync<TEAM>(quarter);  // the tile is complete
                // next iteration's data
                if (!last) {
                    fetch_d(corner, t + 1, buf_d ^ 1);
                    if (NT == 2 ? t + 2 < p.inner : true) fetch_h(corner, NT == 2 ? t + 1 : t);
                } else if (i + 1 < cnt) {
                    const size_t next = corner_of(i + 1);
                    fetch_d(next, 0, buf_d ^ 1);
                    if (NT == 2 && p.inner > 1) fetch_h(next, 0);
                    if (NT == 2 && role == 0 && lane == 0) issue(i + 1, buf_x ^ 1);
                    __syncwarp();
                }
                unsigned rows[4];
#pragma unroll
                for (int ry = 0; ry < 4; ++ry) rows[ry] = tile + (unsigned)(L.cell0 * 16 + ry * L.ysgn * G::ROW * 16);
                if (role == 0) {
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int o = 0; o < 4; ++o) {
                            float e[4];
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                float lo, hi;
                                unpack2(dp[n >> 1][o][s], lo, hi);
                                e[s] = n & 1 ? hi : lo;
                            }
                            dacc[n][o] += (e[0] + e[1]) + (e[2] + e[3]);
                        }
                    quad_wgrad_rows<G::PLANE, 0>(rows, dx, tm, dp);
                } else {
                    quad_wgrad_rows<G::PLANE, 1>(rows, dx, tm, dp);
                }
                __syncwarp();
                if (NT == 2) buf_x ^= 1;
                buf_d ^= 1;
            }
            if (NT == 1) {
                team_sync<TEAM>(quarter);
                if (role == 0 && lane == 0 && i + 1 < cnt) issue(i + 1, 0);
                __syncwarp();
            }
        }

        // ---- the region's sums -> this team's slot
        const long long slot = team - quad_team_of((long long)blk * p.Q, p.nitems, nteams);
        float4 *dst = reinterpret_cast<float4 *>(p.gpk + ((size_t)slot * p.regions + blk) * PACK_F) + lane;
        tmem_wait_st();
        // half 0: single units first, half 1: last
        quad_flush72<false>(dst + role * 90 * 32, tm + role * 360, p.accumulate);
#pragma unroll 1
        for (int b = 0; b < 2; ++b) {
            const int at = 1 + role * 2 + b;  // in batches of 72 columns, 18 vectors
            quad_flush72<true>(dst + at * 18 * 32, tm + at * 72, p.accumulate);
        }
        float4 *o4 = dst + (108 + role * 4) * 32, old[4];
        if (p.accumulate) {
#pragma unroll
            for (int n = 0; n < 4; ++n) old[n] = o4[n * 32];
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            float4 x = make_float4(dacc[n][0], dacc[n][1], dacc[n][2], dacc[n][3]);
            if (p.accumulate) x.x += old[n].x, x.y += old[n].y, x.z += old[n].z, x.w += old[n].w;
            o4[n * 32] = x;
        }
        __syncwarp();
        i0 += here;
        q0 = 0;
        ++blk;
    }
    if (failed && p.error_flag) *p.error_flag = 1;
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free_all(tmem_slot);
}

// Sums of the teams' slots in team order -> gradients in the layout of the parameters. One CTA per region.
template <int SUB>
__global__ void __launch_bounds__(256) quad_unpack_grads_k(const float *__restrict__ gpk, float *__restrict__ gw, float *__restrict__ gb,
                                                           float *__restrict__ gs, int M, int N, int K, int Q, long long nteams)
{
    __shared__ unsigned char uses[36];
    if (threadIdx.x == 0) {
        int k = 0;
        for (int ry = 0; ry < 4; ++ry)
            for (int rz = 0; rz < 4; ++rz)
                for (int n = 0; n < 4; ++n) {
                    const int a = rz - (n >> 1), bb = ry - (n & 1);
                    if (a >= 0 && a <= 2 && bb >= 0 && bb <= 2) uses[k++] = (unsigned char)((a * 3 + bb) | n << 4);
                }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const QuadLane<SUB> L(lane);
    const int nbx = K >> 3, nby = N >> 3, blk = blockIdx.x, regions = gridDim.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const size_t g0 = ((size_t)(bz * 8 + L.z0) * N + (by * 8 + L.y0)) * K + bx * 8 + 4 * L.h;
    const long long zs = (long long)N * K, ys = (long long)L.ysgn * K;
    const long long nitems = (long long)regions * Q;
    const int slots = (int)(quad_team_of((long long)(blk + 1) * Q - 1, nitems, nteams) - quad_team_of((long long)blk * Q, nitems, nteams)) + 1;
#pragma unroll 2
    for (int v = threadIdx.x >> 5; v < quad::VECS; v += 8) {
        const float4 *src = reinterpret_cast<const float4 *>(gpk + (size_t)blk * quad::PACK_F) + v * 32 + lane;
        float4 r = *src;
        for (int k = 1; k < slots; ++k) {
            const float4 e = src[(size_t)k * regions * (quad::PACK_F / 4)];
            r.x += e.x, r.y += e.y, r.z += e.z, r.w += e.w;
        }
        if (L.h) r = make_float4(r.w, r.z, r.y, r.x);
        int n;
        float *dst;
        if (v < 108) {
            const int u = uses[v / 3], c = v % 3;
            n = u >> 4;
            const int tb = (u & 15) % 3;
            dst = gw + (size_t)((u & 15) / 3 * 9 + (L.ysgn < 0 ? 2 - tb : tb) * 3 + (L.h ? 2 - c : c)) * P;
        } else {
            n = v & 3;
            dst = v < 112 ? gb : gs;
        }
        dst += g0 + (n >> 1) * zs + (n & 1) * ys;
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            *reinterpret_cast<float4 *>(dst) = r;
        } else {
            dst[0] = r.x, dst[1] = r.y, dst[2] = r.z, dst[3] = r.w;
        }
    }
}

// ------------------------------------------------------------------------- gradient across block borders
// As bwd_border8_k / bwd_halo8_k (step_bwd_fast.cu), four samples at a time: a cell of a quad is 16 bytes, so even the
// x faces use half of every sector they touch.
// Block 8: three groups of 128 threads, one per axis; a thread owns one cell of the two faces and the nine taps that cross
// that face (a tap that crosses several faces belongs to the first axis in the order z, y, x); then one thread per surface
// cell adds the up to three partial sums to grad_x in that order.
__device__ __forceinline__ float4 fma4(float w, float4 v, float4 a)
{
    return make_float4(fmaf(w, v.x, a.x), fmaf(w, v.y, a.y), fmaf(w, v.z, a.z), fmaf(w, v.w, a.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

namespace quadborder {
constexpr int TS = 1000;
}

__global__ void __launch_bounds__(384) quad_border8_k(const float *__restrict__ w, const float4 *__restrict__ dsum, float4 *__restrict__ gx,
                                                      int Q, int M, int N, int K, int qpc)
{
    using namespace quadborder;
    constexpr int THREADS = 384, SLOTS = 3;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4 *const tile = reinterpret_cast<float4 *>(smem_raw);                   // [2][TS]
    float4 *const part = reinterpret_cast<float4 *>(smem_raw) + 2 * TS;          // [2][3][128]
    const int tid = threadIdx.x;
    const int nbx = K >> 3, nby = N >> 3;
    const unsigned blk = blockIdx.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const long long origin = ((long long)(bz * 8 - 1) * N + (by * 8 - 1)) * K + (bx * 8 - 1);
    for (int i = tid; i < 2 * TS; i += THREADS) tile[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // shell cells this thread fetches: tile offset and offset from the tile's origin
    int tof[SLOTS], rel[SLOTS];
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        const int i = tid + j * THREADS;
        tof[j] = -1;
        rel[j] = 0;
        if (i < TS) {
            const int cx = i % 10, cy = (i / 10) % 10, cz = i / 100;
            const int gz = bz * 8 + cz - 1, gy = by * 8 + cy - 1, gxx = bx * 8 + cx - 1;
            const bool shell = cx == 0 || cx == 9 || cy == 0 || cy == 9 || cz == 0 || cz == 9;
            if (shell && gz >= 0 && gz < M && gy >= 0 && gy < N && gxx >= 0 && gxx < K) {
                tof[j] = i;
                rel[j] = (cz * N + cy) * K + cx;
            }
        }
    }
    // role 1: one cell of one face
    const int axis = tid >> 7, fc = tid & 127, side = fc >> 6, u = (fc >> 3) & 7, v = fc & 7;
    int l[3];
    l[axis] = side * 7;
    l[axis == 0 ? 1 : 0] = u;
    l[axis == 2 ? 1 : 2] = v;
    const int dcross = side == 0 ? 1 : -1;
    float wf[9];
    int toff[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        int d[3];
        d[axis] = dcross;
        d[axis == 0 ? 1 : 0] = q / 3 - 1;
        d[axis == 2 ? 1 : 2] = q % 3 - 1;
        bool owned = true;
        for (int a = 0; a < axis; ++a) {
            const int s = l[a] - d[a];
            if (s < 0 || s > 7) owned = false;
        }
        const int nz = bz * 8 + l[0] - d[0], ny = by * 8 + l[1] - d[1], nx = bx * 8 + l[2] - d[2];
        const bool ok = owned && nz >= 0 && nz < M && ny >= 0 && ny < N && nx >= 0 && nx < K;
        const int t = (d[0] + 1) * 9 + (d[1] + 1) * 3 + (d[2] + 1);
        wf[q] = ok ? w[(size_t)t * P + ((size_t)nz * N + ny) * K + nx] : 0.0f;
        toff[q] = (l[0] + 1 - d[0]) * 100 + (l[1] + 1 - d[1]) * 10 + (l[2] + 1 - d[2]);
    }
    // role 2: one surface cell
    int sz = 0, sy = 0, sx = 0;
    const bool active = tid < 296;
    if (tid < 128) {
        sz = (tid >> 6) * 7; sy = (tid >> 3) & 7; sx = tid & 7;
    } else if (tid < 224) {
        const int j = tid - 128;
        sy = (j / 48) * 7; sz = 1 + (j % 48) / 8; sx = j & 7;
    } else if (active) {
        const int j = tid - 224;
        sx = (j / 36) * 7; sz = 1 + (j % 36) / 6; sy = 1 + j % 6;
    }
    const size_t c = ((size_t)(bz * 8 + sz) * N + by * 8 + sy) * K + bx * 8 + sx;
    const int pz = (sz == 0 || sz == 7) ? (sz / 7) * 64 + sy * 8 + sx : -1;
    const int py = (sy == 0 || sy == 7) ? (sy / 7) * 64 + sz * 8 + sx : -1;
    const int px = (sx == 0 || sx == 7) ? (sx / 7) * 64 + sz * 8 + sy : -1;

    const int q0 = blockIdx.y * qpc, q1 = min(Q, q0 + qpc);
    float4 pf[SLOTS], gnext = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int q) {
        if (q < q1) {
            const float4 *src = dsum + (size_t)q * P + origin;
#pragma unroll
            for (int j = 0; j < SLOTS; ++j)
                if (tof[j] >= 0) pf[j] = __ldg(src + rel[j]);
        }
    };
    fetch(q0);
    if (active && q0 < q1) gnext = gx[(size_t)q0 * P + c];
    __syncthreads();
    for (int q = q0; q < q1; ++q) {
        const int par = q & 1;
        float4 *tl = tile + par * TS;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j)
            if (tof[j] >= 0) tl[tof[j]] = pf[j];
        fetch(q + 1);
        float4 acc = gnext;
        if (active && q + 1 < q1) gnext = gx[(size_t)(q + 1) * P + c];
        __syncthreads();
        {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 9; ++e) s = fma4(wf[e], tl[toff[e]], s);
            part[(par * 3 + axis) * 128 + fc] = s;
        }
        __syncthreads();
        if (active) {
            if (pz >= 0) acc = add4(acc, part[(par * 3 + 0) * 128 + pz]);
            if (py >= 0) acc = add4(acc, part[(par * 3 + 1) * 128 + py]);
            if (px >= 0) acc = add4(acc, part[(par * 3 + 2) * 128 + px]);
            gx[(size_t)q * P + c] = acc;
        }
    }
}

// Block 4: one thread per cell of the region, all 27 taps; sources in the cell's own block carry a zero weight.
__global__ void __launch_bounds__(512) quad_border4_k(const float *__restrict__ w, const float4 *__restrict__ dsum, float4 *__restrict__ gx,
                                                      int Q, int M, int N, int K, int qpc)
{
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
    float4 pf[SLOTS], gnext = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int q) {
        if (q < q1) {
            const float4 *src = dsum + (size_t)q * P + origin;
#pragma unroll
            for (int j = 0; j < SLOTS; ++j)
                if (tof[j] >= 0) pf[j] = __ldg(src + rel[j]);
        }
    };
    fetch(q0);
    if (active && q0 < q1) gnext = gx[(size_t)q0 * P + c];
    __syncthreads();
    for (int q = q0; q < q1; ++q) {
        float4 *tl = tile + (q & 1) * TS;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j)
            if (tof[j] >= 0) tl[tof[j]] = pf[j];
        fetch(q + 1);
        float4 acc = gnext;
        if (active && q + 1 < q1) gnext = gx[(size_t)(q + 1) * P + c];
        __syncthreads();  // the other tile may still be read by slower threads; it is rewritten after the next barrier
        if (active) {
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
// gradients of gamma and beta, which need no second look at the batch. A thread owns CPT cells and walks the quads; the
// eight sums of a quad are added over the warp in float (32 CPT values), above that in double. SUB_G: the gradient is
// g - sub (residual form of the loop).
template <int CPT, bool SUB_G>
__global__ void __launch_bounds__(256) quad_norm_sums_k(const float4 *__restrict__ x, const float4 *__restrict__ g,
                                                        const float4 *__restrict__ sub, const float *__restrict__ gamma,
                                                        const float2 *__restrict__ stats, double2 *__restrict__ partials, int nparts,
                                                        float *__restrict__ ggamma, float *__restrict__ gbeta, int accumulate, int Q,
                                                        size_t P)
{
    constexpr int QB = 16;  // quads between two block-wide sums
    __shared__ float red[QB][8][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t c0 = (size_t)blockIdx.x * (256 * CPT) + tid;
    float gm[CPT], dg[CPT], db[CPT];
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        gm[k] = c0 + k * 256 < P ? gamma[c0 + k * 256] : 0.0f;
        dg[k] = db[k] = 0.0f;
    }
    for (int qb = 0; qb < Q; qb += QB) {
        const int qe = min(Q, qb + QB);
#pragma unroll 2
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
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            float2 mr[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) mr[s] = __ldg(stats + 4 * q + s);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const float xs[4] = {xv[k].x, xv[k].y, xv[k].z, xv[k].w}, gs[4] = {gv[k].x, gv[k].y, gv[k].z, gv[k].w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float xh = (xs[s] - mr[s].x) * mr[s].y, gg = gs[s] * gm[k];
                    v[s] += gg;
                    v[4 + s] = fmaf(gg, xh, v[4 + s]);
                    dg[k] = fmaf(gs[s], xh, dg[k]);
                    db[k] += gs[s];
                }
            }
            const float r = quad_reduce8(v, lane);
            if ((lane & 3) == 0) red[q - qb][warp][lane >> 2] = r;
        }
        __syncthreads();
        for (int e = tid; e < (qe - qb) * 8; e += 256) {
            double s = 0.0;
#pragma unroll
            for (int w8 = 0; w8 < 8; ++w8) s += (double)red[e >> 3][w8][e & 7];
            const int j = e & 7;  // value j: a of samples 0..3, then c
            reinterpret_cast<double *>(partials + (size_t)(4 * (qb + (e >> 3)) + (j & 3)) * nparts + blockIdx.x)[j >> 2] = s;
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k)
        if (c0 + k * 256 < P) {
            ggamma[c0 + k * 256] = accumulate ? ggamma[c0 + k * 256] + dg[k] : dg[k];
            gbeta[c0 + k * 256] = accumulate ? gbeta[c0 + k * 256] + db[k] : db[k];
        }
}

// grid 4 Q: (a, c) / P from the partial sums, in a fixed order
__global__ void __launch_bounds__(256) quad_norm_ac_k(const double2 *__restrict__ partials, int nparts, float2 *__restrict__ ac, size_t P)
{
    __shared__ double red[33];
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
__global__ void __launch_bounds__(256) quad_norm_residual_apply_k(const float4 *__restrict__ h, const float4 *__restrict__ gn, const float4 *gu,
                                                                  const float *__restrict__ gamma, const float2 *__restrict__ stats,
                                                                  const float2 *__restrict__ ac, float4 *out, size_t P)
{
    const size_t c = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= P) return;
    const int q = blockIdx.y;
    const size_t i = (size_t)q * P + c;
    const float gm = gamma[c];
    const float4 hv = h[i], nv = gn[i], uv = gu[i];
    const float hs[4] = {hv.x, hv.y, hv.z, hv.w}, ns[4] = {nv.x, nv.y, nv.z, nv.w}, us[4] = {uv.x, uv.y, uv.z, uv.w};
    float o[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float2 mr = __ldg(stats + 4 * q + s), k = __ldg(ac + 4 * q + s);
        const float xh = (hs[s] - mr.x) * mr.y;
        o[s] = us[s] + mr.y * ((ns[s] - us[s]) * gm - k.x - xh * k.y);
    }
    out[i] = make_float4(o[0], o[1], o[2], o[3]);
}

// Residual form, forward: out = h + (y - norm(h)), and the per-sample partial sums of out (out may be y). With y and out
// null only the sums of h are taken (the statistics of the loop's first input).
__global__ void __launch_bounds__(256) quad_residual_combine_k(const float4 *__restrict__ h, const float4 *y, const float *__restrict__ gamma,
                                                               const float *__restrict__ beta, const float2 *__restrict__ stats, float4 *out,
                                                               double2 *__restrict__ partials, int nparts, size_t P)
{
    constexpr int CPT = 4;
    __shared__ float red[8][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = blockIdx.y;
    const size_t c0 = (size_t)blockIdx.x * (256 * CPT) + tid;
    float2 mr[4];
    if (y) {
#pragma unroll
        for (int s = 0; s < 4; ++s) mr[s] = __ldg(stats + 4 * q + s);
    }
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const size_t c = c0 + k * 256;
        if (c < P) {
            const size_t i = (size_t)q * P + c;
            const float4 hv = h[i];
            float o[4] = {hv.x, hv.y, hv.z, hv.w};
            if (y) {
                const float4 yv = y[i];
                const float ys[4] = {yv.x, yv.y, yv.z, yv.w};
                const float g = gamma[c], b = beta[c];
#pragma unroll
                for (int s = 0; s < 4; ++s) o[s] = o[s] + (ys[s] - fmaf((o[s] - mr[s].x) * mr[s].y, g, b));
                out[i] = make_float4(o[0], o[1], o[2], o[3]);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                v[s] += o[s];
                v[4 + s] = fmaf(o[s], o[s], v[4 + s]);
            }
        }
    }
    const float r = quad_reduce8(v, lane);
    if ((lane & 3) == 0) red[warp][lane >> 2] = r;
    __syncthreads();
    if (tid < 8) {
        double s = 0.0;
#pragma unroll
        for (int w8 = 0; w8 < 8; ++w8) s += (double)red[w8][tid];
        reinterpret_cast<double *>(partials + (size_t)(4 * q + (tid & 3)) * nparts + blockIdx.x)[tid >> 2] = s;
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

template <int SUB, int ACT>
static int launch_reverse_one(const QuadRevParams &p, unsigned ctas, cudaStream_t st)
{
    static unsigned long long done[2] = {};
    int rc;
    if (p.raw) {
        rc = smem_once(quad_reverse_k<SUB, ACT, true>, quadrev::SMEM_BYTES, &done[1], "cudaFuncSetAttribute(quad_reverse_k)");
        if (rc != GN_OK) return rc;
        quad_reverse_k<SUB, ACT, true><<<ctas, 256, quadrev::SMEM_BYTES, st>>>(p);
    } else {
        rc = smem_once(quad_reverse_k<SUB, ACT, false>, quadrev::SMEM_BYTES, &done[0], "cudaFuncSetAttribute(quad_reverse_k)");
        if (rc != GN_OK) return rc;
        quad_reverse_k<SUB, ACT, false><<<ctas, 256, quadrev::SMEM_BYTES, st>>>(p);
    }
    return check_launch("quad_reverse");
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
    p.packed = a.packed_t; p.g = a.g; p.raw = a.raw; p.stats = a.stats; p.ac = a.ac; p.h = a.h;
    p.delta = a.delta; p.dsum = a.dsum; p.gx = a.gx; p.dsq = a.dsq;
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = regions_of(a.M, a.N, a.K) * a.Q;
    long long ctas = (p.nitems + quad::QUARTERS - 1) / quad::QUARTERS;
    if (ctas > sm_count()) ctas = sm_count();
    return a.block == 8 ? launch_reverse_sub<8>(p, (unsigned)ctas, act, st) : launch_reverse_sub<4>(p, (unsigned)ctas, act, st);
}

// CTAs of the weight-gradient kernel: every team writes (or adds to) 59 KB per region it touches, so small problems use
// teams of at least two items
static unsigned wgrad_ctas(long long nitems)
{
    long long ctas = (nitems + 2 * quad::QUARTERS - 1) / (2 * quad::QUARTERS);
    if (ctas > sm_count()) ctas = sm_count();
    return (unsigned)(ctas < 1 ? 1 : ctas);
}

size_t quad_grad_floats(int M, int N, int K, int Q)
{
    const long long regions = regions_of(M, N, K), nitems = regions * Q;
    const long long nteams = (long long)wgrad_ctas(nitems) * quad::QUARTERS;
    long long slots = 1;
    for (long long r = 0; r < regions; ++r) {
        const long long s = quad_team_of((r + 1) * Q - 1, nitems, nteams) - quad_team_of(r * Q, nitems, nteams) + 1;
        if (s > slots) slots = s;
    }
    return (size_t)slots * regions * quad::PACK_F;
}

template <int SUB, int ACT>
static int launch_wgrad_one(const CUtensorMap &map, const QuadWgradParams &p, unsigned ctas, cudaStream_t st)
{
    static unsigned long long done[2] = {};
    constexpr int smem = quadwg::Lay<SUB>::SMEM;
    static_assert(smem <= 232448 - 2048, "shared memory budget of one SM");
    int rc;
    if (p.in_stats) {
        rc = smem_once(quad_wgrad_k<SUB, ACT, true>, smem, &done[1], "cudaFuncSetAttribute(quad_wgrad_k)");
        if (rc != GN_OK) return rc;
        quad_wgrad_k<SUB, ACT, true><<<ctas, 256, smem, st>>>(map, p);
    } else {
        rc = smem_once(quad_wgrad_k<SUB, ACT, false>, smem, &done[0], "cudaFuncSetAttribute(quad_wgrad_k)");
        if (rc != GN_OK) return rc;
        quad_wgrad_k<SUB, ACT, false><<<ctas, 256, smem, st>>>(map, p);
    }
    return check_launch("quad_wgrad");
}

template <int SUB>
static int launch_wgrad_sub(const CUtensorMap &map, const QuadWgradParams &p, unsigned ctas, int act, cudaStream_t st)
{
    switch (act) {
    case GN_ACT_RELU: return launch_wgrad_one<SUB, GN_ACT_RELU>(map, p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_wgrad_one<SUB, GN_ACT_LEAKY_RELU>(map, p, ctas, st);
    case GN_ACT_SILU: return launch_wgrad_one<SUB, GN_ACT_SILU>(map, p, ctas, st);
    default: return launch_wgrad_one<SUB, GN_ACT_TANH>(map, p, ctas, st);
    }
}

int launch_quad_wgrad(const QuadWgrad &a, int act, cudaStream_t st)
{
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, a.block);
    if (rc != GN_OK) return rc;
    QuadWgradParams p{};
    p.gbt = a.gbt; p.in_stats = a.in_stats; p.delta = a.delta; p.h = a.h; p.scale = a.scale; p.dsq = a.dsq; p.gpk = a.gpk;
    p.accumulate = a.accumulate;
    p.error_flag = a.error_flag ? a.error_flag : device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.regions = (int)regions_of(a.M, a.N, a.K);
    p.nitems = (long long)p.regions * a.Q;
    const unsigned ctas = wgrad_ctas(p.nitems);
    return a.block == 8 ? launch_wgrad_sub<8>(map, p, ctas, act, st) : launch_wgrad_sub<4>(map, p, ctas, act, st);
}

int launch_quad_unpack_grads(const float *gpk, float *gw, float *gb, float *gs, int M, int N, int K, int Q, int block, cudaStream_t st)
{
    const long long regions = regions_of(M, N, K);
    const long long nteams = (long long)wgrad_ctas(regions * Q) * quad::QUARTERS;
    if (block == 8) quad_unpack_grads_k<8><<<(unsigned)regions, 256, 0, st>>>(gpk, gw, gb, gs, M, N, K, Q, nteams);
    else quad_unpack_grads_k<4><<<(unsigned)regions, 256, 0, st>>>(gpk, gw, gb, gs, M, N, K, Q, nteams);
    return check_launch("quad_unpack_grads");
}

int launch_quad_border(const float *w, const float *dsum, float *gx, int M, int N, int K, int Q, int block, cudaStream_t st)
{
    const long long nb = regions_of(M, N, K);
    const int ctas_per_sm = block == 8 ? 4 : 3;
    const int chunks = pick_batch_chunks_balanced(nb, Q, ctas_per_sm, 4.0, 32);
    const int qpc = (Q + chunks - 1) / chunks;
    dim3 grid((unsigned)nb, (unsigned)((Q + qpc - 1) / qpc));
    static unsigned long long done[2] = {};
    if (block == 8) {
        constexpr int smem = (2 * quadborder::TS + 2 * 3 * 128) * 16;
        const int rc = smem_once(quad_border8_k, smem, &done[0], "cudaFuncSetAttribute(quad_border8_k)");
        if (rc != GN_OK) return rc;
        quad_border8_k<<<grid, 384, smem, st>>>(w, reinterpret_cast<const float4 *>(dsum), reinterpret_cast<float4 *>(gx), Q, M, N, K, qpc);
    } else {
        constexpr int smem = 2 * quadborder::TS * 16;
        const int rc = smem_once(quad_border4_k, smem, &done[1], "cudaFuncSetAttribute(quad_border4_k)");
        if (rc != GN_OK) return rc;
        quad_border4_k<<<grid, 512, smem, st>>>(w, reinterpret_cast<const float4 *>(dsum), reinterpret_cast<float4 *>(gx), Q, M, N, K, qpc);
    }
    return check_launch("quad_border");
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
#define SUMS_(C, S) quad_norm_sums_k<C, S><<<nparts, 256, 0, st>>>(x4, g4, s4, gamma, stats, partials, nparts, ggamma, gbeta, accumulate, Q, (size_t)P)
    if (wide && sub) SUMS_(4, true);
    else if (wide) SUMS_(4, false);
    else if (sub) SUMS_(1, true);
    else SUMS_(1, false);
#undef SUMS_
    quad_norm_ac_k<<<4 * Q, 256, 0, st>>>(partials, nparts, ac, (size_t)P);
    return check_launch("quad_norm_sums");
}

int launch_quad_norm_residual_apply(const float *h, const float *gn, const float *gu, const float *gamma, const float2 *stats, const float2 *ac,
                                    float *out, int Q, long long P, cudaStream_t st)
{
    dim3 grid((unsigned)((P + 255) / 256), (unsigned)Q);
    quad_norm_residual_apply_k<<<grid, 256, 0, st>>>(reinterpret_cast<const float4 *>(h), reinterpret_cast<const float4 *>(gn),
                                                     reinterpret_cast<const float4 *>(gu), gamma, stats, ac, reinterpret_cast<float4 *>(out), (size_t)P);
    return check_launch("quad_norm_residual_apply");
}

int quad_combine_parts(long long P) { return (int)((P + 1023) / 1024); }

int launch_quad_residual_combine(const float *h, const float *y, const float *gamma, const float *beta, const float2 *stats, float *out,
                                 double2 *partials, int Q, long long P, cudaStream_t st)
{
    dim3 grid((unsigned)quad_combine_parts(P), (unsigned)Q);
    quad_residual_combine_k<<<grid, 256, 0, st>>>(reinterpret_cast<const float4 *>(h), reinterpret_cast<const float4 *>(y), gamma, beta, stats,
                                                  reinterpret_cast<float4 *>(out), partials, quad_combine_parts(P), (size_t)P);
    return check_launch("quad_residual_combine");
}

}  // namespace gn
