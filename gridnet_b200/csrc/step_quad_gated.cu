// Gated update with the weights in tensor memory and four samples per lane (float, block 8):
//   gate = sigmoid(sum_t x[n + o_t] w[t][1][n] + b[1][n])
//   x[n] <- gate x[n] + (1 - gate) act(sum_t x[n + o_t] w[t][0][n] + b[0][n])
// (gridnet/backend_torch.py:145-267; the kernels this stands in for are src/gridnet_cuda_kernels.cu:452-560.)
//
// A gated neuron has 54 weights, twice what a lane's tensor memory holds for the 16 neurons of the mapping of
// step_quad.cu. So two warps in different quarters of tensor memory work on a region and quad together, one per branch: each
// runs the 27-tap sums of its branch over the shared tile exactly as the plain kernel does, then they exchange half of their
// sums through shared memory, and each finishes half of the neurons (the even and the odd z planes). That costs 32
// shared-memory accesses per lane and iteration beside the 96 of the window, the same as in the plain kernel. Four such pairs per SM; the
// two pairs that share a region take its quads in turn, one's exchange under the other's sums.
//
// Bound by the shared-memory pipe like the plain kernel (4.5 FMAs per wavefront of the window). At 32^3, two inner
// iterations, batch 64: forward 38 us with what the backward pass needs written out and statistics in double above four values (34 with
// floats of 256; register-patch kernel: 38), reverse sweep 53 us (57).
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "quad_geo.cuh"
#include "tmem.cuh"

namespace gn {

namespace quadgate {
using G = QuadGeo<8>;
constexpr int NBUF = 4, TEAMS = 2, PAIRS = 4;
constexpr int XCH_BYTES = 2 * 8 * 512;  // of a pair: eight cells per lane from each branch
constexpr int FWD_SMEM(bool fuse) { return TEAMS * NBUF * G::BUF_BYTES + PAIRS * XCH_BYTES + (fuse ? TEAMS * G::CELLS * 8 : 0); }
// reverse sweep: a delta tile per warp (as in quad_reverse_k), staging for half a region's hv, hg and x per warp, exchange
constexpr int RROW = 10, RPLANE = 80, RTILE = 9 * RPLANE * 16, RTILES = 8 * RTILE + RPLANE * 16;
constexpr int HALF = 4 * 64 * 16, STAGE = 3 * HALF;
constexpr int REV_SMEM = RTILES + 8 * STAGE + PAIRS * XCH_BYTES;
static_assert(REV_SMEM <= 232448 - 1024, "shared memory of one SM");
}  // namespace quadgate

// the two warps of a pair (barriers 1 .. 4), the four warps of a team (5, 6)
__device__ __forceinline__ void pair_sync(int pair)
{
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
}
__device__ __forceinline__ void gate_team_sync(int team)
{
    __syncwarp();
    asm volatile("bar.sync %0, 128;" ::"r"(team + 5) : "memory");
}

// 1 / (1 + 2^(-h log2 e)); as sigmoid_ (common.cuh), whose cap the reciprocal of infinity makes unnecessary
__device__ __forceinline__ u64 sigmoid2(u64 h)
{
    float t0, t1, e0, e1, d0, d1, r0, r1;
    unpack2(fmul2(h, pack2(-1.4426950408889634f, -1.4426950408889634f)), t0, t1);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
    unpack2(fadd2(pack2(e0, e1), pack2(1.0f, 1.0f)), d0, d1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
    return pack2(r0, r1);
}
__device__ __forceinline__ u64 one_minus2(u64 a) { return ffma2r(a, pack2(-1.0f, -1.0f), pack2(1.0f, 1.0f)); }

struct QuadGateParams {
    const float *packed;     // [branch][regions][PACK_F]
    const float2 *gbt;       // FUSE_IN: as in step_fwd_quad
    const float2 *in_stats;
    double2 *out_partials;   // [4 Q][nparts]: slots 2 region + branch; nullptr: not wanted
    int nparts;
    float *y;                // IL4
    float *save_v, *save_g, *save_x;  // SAVE: [inner] IL4 tensors: the two pre-activations, the activations that went in
    int *error_flag;
    int M, N, K, Q, inner;
    int params_old;         // the kernel before this one did not write packed or gbt
    long long nitems;
};

template <int ACT, bool FUSE_IN, bool SAVE>
__global__ void __launch_bounds__(256, 1) quad_gated_fwd_k(const __grid_constant__ CUtensorMap in_map, const QuadGateParams p)
{
    using namespace quad;
    using namespace quadgate;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[TEAMS * NBUF];
    __shared__ int issued[TEAMS * NBUF];  // which item's copy into this buffer has been started last
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2, branch = quarter & 1, team = quarter >> 1, pair = team * 2 + role;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid == 0) {
        for (int i = 0; i < TEAMS * NBUF; ++i) {
            mbar_init(smem_u32(&bars[i]), 1);
            issued[i] = -1;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<8> L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K, regions = (size_t)nbx * nby * (p.M >> 3);
    const long long worker = (long long)blockIdx.x * TEAMS + team, nworkers = (long long)gridDim.x * TEAMS;
    const long long n0 = p.nitems * worker / nworkers;
    const int cnt = (int)(p.nitems * (worker + 1) / nworkers - n0);
    const unsigned bar0 = smem_u32(&bars[team * NBUF]), issued0 = smem_u32(&issued[team * NBUF]);
    const unsigned tiles = smem_u32(smem) + team * (NBUF * G::BUF_BYTES);
    const unsigned xch = smem_u32(smem) + TEAMS * NBUF * G::BUF_BYTES + pair * XCH_BYTES + lane * 16;  // + branch * 4096: written by
    float2 *const gbs = reinterpret_cast<float2 *>(smem + TEAMS * NBUF * G::BUF_BYTES + PAIRS * XCH_BYTES) + team * G::CELLS;
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K;
    const long long zstr = wzs * 4, ystr = wys * 4;
    bool failed = false;

    auto issue = [&](int i) {  // one lane: fetch the tile of the team's item i
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const unsigned bar = bar0 + 8 * (i % NBUF);
        fence_proxy_async();
        mbar_expect_tx(bar, G::CELLS * 16);
        tma_load_4d(tiles + (i % NBUF) * G::BUF_BYTES, &in_map, bar, (bx * 8 - 1) * 4, by * 8 - 1, bz * 8 - 1, q);
        st_release_shared(issued0 + 4 * (i % NBUF), i);
    };
    auto wait_tile = [&](int i) {  // see step_fwd_quad
        unsigned spins = 0;
        while (ld_acquire_shared(issued0 + 4 * (i % NBUF)) != i && ++spins < kSpinLimit) {}
        if (spins >= kSpinLimit || !mbar_wait_bounded(bar0 + 8 * (i % NBUF), (unsigned)(i / NBUF) & 1u, kSpinLimit)) failed = true;
        __syncwarp();
    };
    auto begin = [&]() {
        previous_done();
        if (branch == 0 && role == 0 && lane == 0)
            for (int i = 0; i < NBUF && i < cnt; ++i) issue(i);
        __syncwarp();
    };
    if (!p.params_old || cnt == 0) begin();  // else the first region's parameters come first

    int blk = (int)(n0 / p.Q), q0 = (int)(n0 - (long long)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + L.z0) * p.N + (by * 8 + L.y0)) * p.K + bx * 8 + 4 * L.h;
        if (i0 > 0) {
            tmem_fence_before();
            gate_team_sync(team);  // nobody reads the old region's weights or table any more
            tmem_fence_after();
        }
        if (FUSE_IN) {
            const unsigned char *src = reinterpret_cast<const unsigned char *>(p.gbt + (size_t)blk * G::CELLS);
            for (int c = (branch * 2 + role) * 32 + lane; c < G::CELLS / 2; c += 128) cp_async16(smem_u32(gbs) + c * 16, src + c * 16);
            __syncwarp();
        }
        quad_load_params(p.packed + (branch * regions + blk) * PACK_F, role, lane, tm);
        tmem_wait_st();
        if (FUSE_IN) cp_async_wait_all();
        if (i0 == 0 && p.params_old) begin();
        tmem_fence_before();
        gate_team_sync(team);
        tmem_fence_after();

        for (int k = (role + 2 - i0 % 2) % 2; k < here; k += 2) {
            const int i = i0 + k, q = q0 + k;
            const unsigned tile = tiles + (i % NBUF) * G::BUF_BYTES;
            if (FUSE_IN) {
                u64 na[2], nb[2];
                {
                    float2 mr[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) mr[s] = p.in_stats[4 * q + s];
                    na[0] = pack2(mr[0].y, mr[1].y);
                    na[1] = pack2(mr[2].y, mr[3].y);
                    nb[0] = pack2(-mr[0].x, -mr[1].x);
                    nb[1] = pack2(-mr[2].x, -mr[3].x);
                }
                wait_tile(i);
                u64 v[16][2];
                float2 g2[16];
                const int c0 = branch * 32 + lane;
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c0 + c * 64 < G::CELLS) {
                        g2[c] = gbs[c0 + c * 64];
                        lds128u(tile + (c0 + c * 64) * 16, v[c][0], v[c][1]);
                    }
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c0 + c * 64 < G::CELLS) {
                        const u64 gg = pack2(g2[c].x, g2[c].x), bb = pack2(g2[c].y, g2[c].y);
                        sts128u(tile + (c0 + c * 64) * 16, ffma2r(fmul2(fadd2(v[c][0], nb[0]), na[0]), gg, bb), ffma2r(fmul2(fadd2(v[c][1], nb[1]), na[1]), gg, bb));
                    }
                pair_sync(pair);
            } else {
                wait_tile(i);
            }
            const unsigned win = tile + L.cell0 * 16u;
            unsigned rows[4];
#pragma unroll
            for (int ry = 0; ry < 4; ++ry) rows[ry] = win + (unsigned)(ry * L.ysgn * G::ROW * 16);
            auto own_cell = [&](int n, int o) {
                return win + (unsigned)((1 + o) * L.xsgn * 16 + (1 + (n & 1)) * L.ysgn * G::ROW * 16) + (1 + (n >> 1)) * G::PLANE * 16u;
            };
            const size_t own = ((size_t)q * P + g0) * 4, T4 = (size_t)p.Q * P * 4;
            for (int t = 0; t < p.inner; ++t) {
                u64 acc[4][4][2];
                {
                    float bias[16];
                    tmem_ld16(tm + COL_BIAS, bias);
                    tmem_wait_ld16(bias);
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int o = 0; o < 4; ++o) acc[n][o][0] = acc[n][o][1] = pack2(bias[n * 4 + o], bias[n * 4 + o]);
                }
                const u64 none[2] = {0, 0};
                quad_stencil<G::PLANE, ADD>(rows, L.xsgn * 16, tm, acc, none, [](int, int, float, float, u64, u64) {});
                // rows n = 0, 1 (the even planes) are finished by branch 0, n = 2, 3 by branch 1
                u64 mine[2][4][2], his[2][4][2];
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        const unsigned to = xch + branch * 4096 + (r * 4 + o) * 512;
                        if (branch) sts128u(to, acc[r][o][0], acc[r][o][1]);
                        else sts128u(to, acc[2 + r][o][0], acc[2 + r][o][1]);
                        mine[r][o][0] = branch ? acc[2 + r][o][0] : acc[r][o][0];
                        mine[r][o][1] = branch ? acc[2 + r][o][1] : acc[r][o][1];
                    }
                if (SAVE) quad_store((branch ? p.save_g : p.save_v) + t * T4 + own, zstr, ystr, L.h, acc);
                pair_sync(pair);  // both have read their windows, the sums are there
                const bool last = t + 1 == p.inner;
                u64 x[2][4][2];
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        lds128u(xch + (branch ^ 1) * 4096 + (r * 4 + o) * 512, his[r][o][0], his[r][o][1]);
                        lds128u(own_cell(2 * branch + r, o), x[r][o][0], x[r][o][1]);
                    }
                float *const half = (SAVE ? p.save_x + t * T4 : p.y) + own + branch * zstr;
                if (SAVE)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int j = 0; j < 2; ++j) quad_store2(half, r, j, zstr, ystr, L.h, x[r]);
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int o = 0; o < 4; ++o)
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            const u64 hv = branch ? his[r][o][k2] : mine[r][o][k2], hg = branch ? mine[r][o][k2] : his[r][o][k2];
                            const u64 gate = sigmoid2(hg);
                            float h0, h1;
                            unpack2(hv, h0, h1);
                            const u64 a = pack2(Act<ACT, float>::fwd(h0), Act<ACT, float>::fwd(h1));
                            x[r][o][k2] = ffma2r(gate, x[r][o][k2], fmul2(one_minus2(gate), a));
                        }
                if (!last) {
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int o = 0; o < 4; ++o) sts128u(own_cell(2 * branch + r, o), x[r][o][0], x[r][o][1]);
                    pair_sync(pair);  // the tile is complete
                } else {
                    float *const to = p.y + own + branch * zstr;
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int j = 0; j < 2; ++j) quad_store2(to, r, j, zstr, ystr, L.h, x[r]);
                    if (p.out_partials) {
                        // four x-neighbours in float, everything above in double, as norm_partial_stats_k (norm.cu)
                        double v[8];
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            float f[2][2][2];  // [row][sum | squares][sample]
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                u64 a[4];
#pragma unroll
                                for (int o = 0; o < 4; ++o) a[o] = x[r][L.h ? 3 - o : o][k2];
                                unpack2(fadd2(fadd2(a[0], a[1]), fadd2(a[2], a[3])), f[r][0][0], f[r][0][1]);
                                unpack2(fadd2(ffma2r(a[0], a[0], fmul2(a[1], a[1])), ffma2r(a[2], a[2], fmul2(a[3], a[3]))), f[r][1][0], f[r][1][1]);
                            }
#pragma unroll
                            for (int j = 0; j < 2; ++j)
#pragma unroll
                                for (int i = 0; i < 2; ++i) v[4 * j + 2 * k2 + i] = (double)f[0][j][i] + (double)f[1][j][i];
                        }
                        const double r = quad_reduce8(v, lane);
                        if ((lane & 3) == 0)
                            reinterpret_cast<double *>(p.out_partials + (size_t)(4 * q + ((lane >> 2) & 3)) * p.nparts + 2 * blk + branch)[lane >> 4] = r;
                    }
                    pair_sync(pair);  // the tile is dead
                    if (branch == 0 && lane == 0 && i + NBUF < cnt) issue(i + NBUF);
                    __syncwarp();
                }
            }
        }
        i0 += here;
        q0 = 0;
        ++blk;
    }
    if (failed && p.error_flag) *p.error_flag = 1;
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free_all(tmem_slot);
}

struct QuadGateRevParams {
    const float *packed;           // [branch][regions][PACK_F], transposed
    const float *gamma;            // the whole-grid norm that followed the step
    const float *g, *raw;          // gradient of the normalised output, the step's output, IL4
    const float2 *stats, *ac;
    const float *hv, *hg, *x;      // [inner] IL4
    float *delta_v, *delta_g;      // [inner] IL4
    float *dsum_v, *dsum_g, *gx;   // IL4
    int M, N, K, Q, inner;
    long long nitems;
};

// The inner iterations backwards. With a = act(hv): delta_v = g (1 - gate) act'(hv), delta_g = g (x - a) gate (1 - gate), and
// g <- gate g + what the two transposed sums over delta_v and delta_g bring. Each warp of a pair makes both deltas of half the neurons and
// runs the transposed sum of its branch over the whole region; they exchange half of those sums.
template <int ACT>
__global__ void __launch_bounds__(256, 1) quad_gated_reverse_k(const QuadGateRevParams p)
{
    using namespace quad;
    using namespace quadgate;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2, branch = quarter & 1, team = quarter >> 1, pair = team * 2 + role;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    for (int c = tid; c < RTILES / 16; c += 256) sts128u(smem_u32(smem) + c * 16, 0, 0);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);
    const unsigned tile_v = smem_u32(smem) + pair * 2 * RTILE, tile = tile_v + branch * RTILE;
    const unsigned stage = smem_u32(smem) + RTILES + (pair * 2 + branch) * STAGE;
    const unsigned xch = smem_u32(smem) + RTILES + 8 * STAGE + pair * XCH_BYTES + lane * 16;

    const QuadLane<8> L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K, T4 = (size_t)p.Q * P * 4, regions = (size_t)nbx * nby * (p.M >> 3);
    const long long worker = (long long)blockIdx.x * TEAMS + team, nworkers = (long long)gridDim.x * TEAMS;
    const long long n0 = p.nitems * worker / nworkers;
    const int cnt = (int)(p.nitems * (worker + 1) / nworkers - n0);
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K;
    const long long zstr = wzs * 4, ystr = wys * 4;
    const int dx = L.xsgn * 16;
    unsigned rows[4];  // window rows, plane 0, column 0, relative to a tile
#pragma unroll
    for (int ry = 0; ry < 4; ++ry) {
        int y = L.y0 + L.ysgn * (ry - 1);
        y = y < 0 ? 0 : (y > 7 ? 7 : y);
        rows[ry] = (unsigned)(L.z0 * RPLANE + y * RROW + (L.h ? 9 : 0)) * 16u;
    }
    // own cell of half row r (plane 2 zp + branch, y row r) relative to a tile, and in the staging area of the half region
    const unsigned cell0 = rows[1] + (unsigned)dx + (1 + branch) * RPLANE * 16u;
    auto own_cell = [&](int r, int o) { return cell0 + (unsigned)(r * L.ysgn * RROW * 16 + o * dx); };
    const unsigned s_row = (unsigned)((L.z0 >> 1) * 8 + L.y0) * 128u, s_e = (L.h ? 7u : 0u) ^ (unsigned)(L.y0 >> 1);
    auto staged = [&](int r, int o) { return s_row + (unsigned)(r * L.ysgn * 128) + (((unsigned)o ^ s_e) << 4); };
    auto corner_of = [&](int i) {  // first cell of the half region's first row in an IL4 tensor
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        return ((size_t)q * P + ((size_t)(bz * 8 + branch) * p.N + by * 8) * p.K + bx * 8) * 4;
    };
    auto fetch_half = [&](unsigned to, const float *src) {
        const int y = lane >> 3, xx = lane & 7;
        const float *s = src + ((long long)y * p.K + xx) * 4;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int yy = y + 4 * (k & 1);
            cp_async16(to + (unsigned)(((k >> 1) * 8 + yy) * 8 + (xx ^ (yy >> 1))) * 16u, s + (k & 1) * 16ll * p.K + (k >> 1) * 2 * zstr);
        }
    };
    auto fetch = [&](size_t corner, int t) {
        fetch_half(stage, p.hv + t * T4 + corner);
        fetch_half(stage + HALF, p.hg + t * T4 + corner);
        fetch_half(stage + 2 * HALF, p.x + t * T4 + corner);
    };
    int blk = (int)(n0 / p.Q), q0 = (int)(n0 - (long long)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + L.z0 + branch) * p.N + (by * 8 + L.y0)) * p.K + bx * 8 + 4 * L.h;  // own half, native layout
        if (i0 > 0) {
            tmem_fence_before();
            gate_team_sync(team);
            tmem_fence_after();
        }
        quad_load_params(p.packed + (branch * regions + blk) * PACK_F, role, lane, tm);  // at least two kernels old
        tmem_wait_st();
        if (i0 == 0) {
            previous_done();
            if (role < cnt) fetch(corner_of(role), p.inner - 1);
            __syncwarp();
        }
        tmem_fence_before();
        gate_team_sync(team);
        tmem_fence_after();
        for (int k = (role + 2 - i0 % 2) % 2; k < here; k += 2) {
            const int i = i0 + k, q = q0 + k;
            const size_t own = ((size_t)q * P + g0) * 4;
            u64 g[2][4][2], sv[2][4][2], sg[2][4][2];
            {
                // gradient of (y - mean) rstd gamma + beta: rstd (g gamma - a - yhat c)
                u64 y[2][4][2];
                float gm[2][4];
                float2 m4[4], a4[4];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        quad_load2(p.g + own, r, j, zstr, ystr, L.h, g[r]);
                        quad_load2(p.raw + own, r, j, zstr, ystr, L.h, y[r]);
                    }
#pragma unroll
                    for (int o = 0; o < 4; ++o) gm[r][o] = p.gamma[g0 + r * wys + (L.h ? 3 - o : o)];
                }
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    m4[s] = p.stats[4 * q + s];
                    a4[s] = p.ac[4 * q + s];
                }
#pragma unroll
                for (int k2 = 0; k2 < 2; ++k2) {
                    const float2 m0 = m4[2 * k2], m1 = m4[2 * k2 + 1], a0 = a4[2 * k2], a1 = a4[2 * k2 + 1];
                    const u64 mu = pack2(-m0.x, -m1.x), rs = pack2(m0.y, m1.y), ma = pack2(-a0.x, -a1.x), mc = pack2(-a0.y, -a1.y);
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int o = 0; o < 4; ++o) {
                            const u64 yh = fmul2(fadd2(y[r][o][k2], mu), rs);
                            const u64 gg = ffma2r(g[r][o][k2], pack2(gm[r][o], gm[r][o]), ma);
                            g[r][o][k2] = fmul2(ffma2r(yh, mc, gg), rs);
                            sv[r][o][k2] = sg[r][o][k2] = 0;
                        }
                }
            }
            for (int t = p.inner - 1; t >= 0; --t) {
                cp_async_wait_all();
                __syncwarp();
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    u64 hv[4][2], hg[4][2], x[4][2];
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        lds128u(stage + staged(r, o), hv[o][0], hv[o][1]);
                        lds128u(stage + HALF + staged(r, o), hg[o][0], hg[o][1]);
                        lds128u(stage + 2 * HALF + staged(r, o), x[o][0], x[o][1]);
                    }
#pragma unroll
                    for (int o = 0; o < 4; ++o)
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            u64 a, da;
                            act_both2<ACT>(hv[o][k2], a, da);
                            const u64 gate = sigmoid2(hg[o][k2]);
                            const u64 rest = fmul2(g[r][o][k2], one_minus2(gate));  // g (1 - gate)
                            hv[o][k2] = fmul2(rest, da);
                            hg[o][k2] = fmul2(fmul2(rest, gate), ffma2r(a, pack2(-1.0f, -1.0f), x[o][k2]));
                            sv[r][o][k2] = fadd2(sv[r][o][k2], hv[o][k2]);
                            sg[r][o][k2] = fadd2(sg[r][o][k2], hg[o][k2]);
                            g[r][o][k2] = fmul2(g[r][o][k2], gate);
                        }
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        sts128u(tile_v + own_cell(r, o), hv[o][0], hv[o][1]);
                        sts128u(tile_v + RTILE + own_cell(r, o), hg[o][0], hg[o][1]);
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        quad_store2(p.delta_v + t * T4 + own, r, j, zstr, ystr, L.h, hv);
                        quad_store2(p.delta_g + t * T4 + own, r, j, zstr, ystr, L.h, hg);
                    }
                }
                pair_sync(pair);  // both delta tiles are complete; what was staged has been read
                if (t > 0) fetch(corner_of(i), t - 1);
                else if (i + 2 < cnt) fetch(corner_of(i + 2), p.inner - 1);
                u64 acc[4][4][2];
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o) acc[n][o][0] = acc[n][o][1] = 0;
                unsigned at[4];
#pragma unroll
                for (int ry = 0; ry < 4; ++ry) at[ry] = tile + rows[ry];
                const u64 none[2] = {0, 0};
                __syncwarp();
                quad_stencil<RPLANE, ADD>(at, dx, tm, acc, none, [](int, int, float, float, u64, u64) {});
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        const unsigned to = xch + branch * 4096 + (r * 4 + o) * 512;
                        if (branch) sts128u(to, acc[r][o][0], acc[r][o][1]);
                        else sts128u(to, acc[2 + r][o][0], acc[2 + r][o][1]);
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) g[r][o][k2] = fadd2(g[r][o][k2], branch ? acc[2 + r][o][k2] : acc[r][o][k2]);
                    }
                pair_sync(pair);  // both have read their tiles, the sums are there
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        u64 h[2];
                        lds128u(xch + (branch ^ 1) * 4096 + (r * 4 + o) * 512, h[0], h[1]);
                        g[r][o][0] = fadd2(g[r][o][0], h[0]);
                        g[r][o][1] = fadd2(g[r][o][1], h[1]);
                    }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    quad_store2(p.gx + own, r, j, zstr, ystr, L.h, g[r]);
                    quad_store2(p.dsum_v + own, r, j, zstr, ystr, L.h, sv[r]);
                    quad_store2(p.dsum_g + own, r, j, zstr, ystr, L.h, sg[r]);
                }
        }
        i0 += here;
        q0 = 0;
        ++blk;
    }
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free_all(tmem_slot);
}

// ------------------------------------------------------------------------------------------------ host side
template <typename Kern>
static int set_smem(Kern kern, int bytes, unsigned long long *mask)
{
    if (!first_use_on_device(mask)) return GN_OK;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) return GN_OK;
    record_cuda_error(e, "cudaFuncSetAttribute(quad_gated)");
    return GN_ERR_CUDA;
}

static unsigned gate_ctas(long long nitems)
{
    const long long c = (nitems + quadgate::TEAMS - 1) / quadgate::TEAMS;
    return (unsigned)(c < sm_count() ? c : sm_count());
}

template <int ACT, bool FUSE_IN, bool SAVE>
static int launch_fwd_one(const CUtensorMap &map, const QuadGateParams &p, cudaStream_t st)
{
    constexpr int smem = quadgate::FWD_SMEM(FUSE_IN);
    static unsigned long long done = 0;
    const int rc = set_smem(quad_gated_fwd_k<ACT, FUSE_IN, SAVE>, smem, &done);
    if (rc != GN_OK) return rc;
    launch_after(quad_gated_fwd_k<ACT, FUSE_IN, SAVE>, gate_ctas(p.nitems), 256, smem, st, map, p);
    return check_launch("quad_gated_fwd");
}
template <int ACT>
static int launch_fwd_act(const CUtensorMap &map, const QuadGateParams &p, cudaStream_t st)
{
    if (p.save_v) return p.in_stats ? launch_fwd_one<ACT, true, true>(map, p, st) : launch_fwd_one<ACT, false, true>(map, p, st);
    return p.in_stats ? launch_fwd_one<ACT, true, false>(map, p, st) : launch_fwd_one<ACT, false, false>(map, p, st);
}

int launch_quad_gated_fwd(const QuadGated &a, int act, cudaStream_t st)
{
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, 8);
    if (rc != GN_OK) return rc;
    QuadGateParams p{};
    p.packed = a.packed; p.params_old = a.params_old; p.gbt = a.gbt; p.in_stats = a.in_stats; p.out_partials = a.out_partials; p.nparts = a.nparts; p.y = a.out_il4;
    p.save_v = a.hv; p.save_g = a.hg; p.save_x = a.x;
    p.error_flag = device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = (long long)(a.M / 8) * (a.N / 8) * (a.K / 8) * a.Q;
    switch (act) {
    case GN_ACT_RELU: return launch_fwd_act<GN_ACT_RELU>(map, p, st);
    case GN_ACT_LEAKY_RELU: return launch_fwd_act<GN_ACT_LEAKY_RELU>(map, p, st);
    case GN_ACT_SILU: return launch_fwd_act<GN_ACT_SILU>(map, p, st);
    default: return launch_fwd_act<GN_ACT_TANH>(map, p, st);
    }
}

template <int ACT>
static int launch_rev_act(const QuadGateRevParams &p, cudaStream_t st)
{
    static unsigned long long done = 0;
    const int rc = set_smem(quad_gated_reverse_k<ACT>, quadgate::REV_SMEM, &done);
    if (rc != GN_OK) return rc;
    launch_after(quad_gated_reverse_k<ACT>, gate_ctas(p.nitems), 256, quadgate::REV_SMEM, st, p);
    return check_launch("quad_gated_reverse");
}

int launch_quad_gated_reverse(const QuadGatedReverse &a, int act, cudaStream_t st)
{
    QuadGateRevParams p{};
    p.packed = a.packed_t; p.gamma = a.gamma; p.g = a.g; p.raw = a.raw; p.stats = a.stats; p.ac = a.ac;
    p.hv = a.hv; p.hg = a.hg; p.x = a.x;
    p.delta_v = a.delta_v; p.delta_g = a.delta_g; p.dsum_v = a.dsum_v; p.dsum_g = a.dsum_g; p.gx = a.gx;
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = (long long)(a.M / 8) * (a.N / 8) * (a.K / 8) * a.Q;
    switch (act) {
    case GN_ACT_RELU: return launch_rev_act<GN_ACT_RELU>(p, st);
    case GN_ACT_LEAKY_RELU: return launch_rev_act<GN_ACT_LEAKY_RELU>(p, st);
    case GN_ACT_SILU: return launch_rev_act<GN_ACT_SILU>(p, st);
    default: return launch_rev_act<GN_ACT_TANH>(p, st);
    }
}

}  // namespace gn
