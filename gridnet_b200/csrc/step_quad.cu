// "Quad" kernels: float forward of the block-local update (block 8 and 4) with the weights in tensor memory and four
// samples per lane. This file has the step with per-block normalisation and what all quad kernels share: re-ordering of
// parameters and activations. step_taps.cu has the step without it.
//
// The register-patch kernel (step_fast.cu) keeps 108 weights per thread in registers and pays 2.25 FMAs per
// shared-memory wavefront; the large-batch kernel (step_pair64.cu) fetches the weights from shared memory and pays
// about 2.9. Here the weights do not touch the shared-memory data pipe at all: a warp handles a whole 8^3 region for
// four samples, a lane owns a 2 x 2 x 4 (z, y, x) patch of neurons, and its 16 x 27 weights, biases and scales are
// 464 of the 512 words that tensor memory has per lane. They are read back in steps of 12 words, a stencil step
// ahead, and each is used for the lane's four samples. A window is 4 x 4 x 6 cells for 16 neurons: 4.5 FMAs per
// wavefront, the most that any split of an 8^3 region over 32 lanes gives.
//
//   * Layout ("IL4"): activations between the steps are interleaved by four samples, [B/4][M][N][K][4], so that a
//     cell of a quad is one 128-bit access and FMAs are packed (fma.rn.f32x2) over sample pairs; a weight is the
//     scalar operand of both.
//   * A warp is on its own: its tile (10 x 10 x 10 cells) is read and written by no other warp, so the
//     inner iterations need no barrier beyond __syncwarp, and new values go back into the tile in place.
//   * Bank conflicts: none, see QuadLane in quad_geo.cuh.
//   * Two warps (w, w + 4) share a quarter of tensor memory and therefore a region: each takes the next of its quads when it
//     is free (its tile may have to wait for the buffer that the other warp is done with last). Each such team has its own
//     contiguous range of (region, quad) items, and meets (named barrier) only to exchange the weights at a new region. The
//     two warps sit on the same scheduler, so one's activation functions (MUFU) overlap the other's FMAs.
//   * Tiles arrive by bulk tensor copy (zero fill outside the grid) into two buffers per team. With a third one the kernel was
//     slower, the first-level cache being what is left; so it was with the next region's parameters prefetched to L2 (64^3 x 64,
//     two iterations, kept for a backward pass: 120 us with both, 114 without).
//
// Reference semantics: gridnet/backend_torch.py:61-142; the kernel it stands in for is
// gridnet_cuda_forward_kernel, src/gridnet_cuda_kernels.cu:101-200.
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "quad_geo.cuh"
#include "taps_geo.cuh"
#include "tmem.cuh"

namespace gn {

struct QuadParams {
    const float *packed;     // [regions][quad::PACK_F]
    const float *wsum;       // the neurons' weight sums, [regions][4][32] vectors
    float4 *tile_stats;      // SAVE: [inner][Q][tiles][QS_COUNT]
    float eps;
    float *y;                // IL4; nullptr: not wanted (replay)
    float *save_h;           // SAVE: [inner][Q][P][4]
    int *error_flag;
    int M, N, K, Q, inner;
    long long nitems;        // regions * Q
    int unit;                // quad_split_unit
};

// SAVE: keep every iteration's pre-activations for the backward pass (which gets the activations in between from them and
// the step's input).
// Per-block normalisation (the reference's normalize=True, gridnet/backend_torch.py:92-97): the input of an
// iteration's sums is (tile - mean) / (std + eps) over all cells of the block's tile, the residual stays as it is. A tile
// belongs to one warp, so the statistics need only shuffles. The landed tile is read once for its mean c and once more
// to subtract it and to take the sums over its halo, which no iteration changes; from then on the tile holds v - c, so
// that neither the variance nor sum w v - mean sum w cancels. Each iteration adds up the values it has just computed
// while they are still in registers.
template <int SUB, int ACT, bool SAVE>
__global__ void __launch_bounds__(128 * QuadGeo<SUB>::TEAM, 1)
    step_fwd_quad(const __grid_constant__ CUtensorMap in_map, const QuadParams p)
{
    using namespace quad;
    using G = QuadGeo<SUB>;
    constexpr int TEAM = G::TEAM, NBUF = G::NBUF;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[QUARTERS * G::NBUF];
    __shared__ int issued[QUARTERS * G::NBUF];  // which item's copy into this buffer has been started last
    __shared__ int claimed[QUARTERS];           // items of the team that warps have taken
    __shared__ unsigned tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid == 0) {
        for (int i = 0; i < QUARTERS * G::NBUF; ++i) {
            mbar_init(smem_u32(&bars[i]), 1);
            issued[i] = -1;
        }
        for (int i = 0; i < QUARTERS; ++i) claimed[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<SUB> L(lane);
    // The lane's share of its tile's cells, first + STRIDE k; four lanes share a block-4 tile, and the first two
    // bits of a quarter-warp's tiles are spread over the banks. Bit k of inside: cell k is no halo.
    constexpr int TILE_CELLS = SUB == 8 ? G::CELLS : 216, STRIDE = SUB == 8 ? 32 : 4, SHARE = (TILE_CELLS + STRIDE - 1) / STRIDE;
    const int my = L.ysgn < 0, turn = SUB == 8 ? 0 : 2 * (2 * my + L.h);
    const int first = SUB == 8 ? lane : ((lane >> 1) & 1) + ((lane >> 3) & 1) * 2 + turn;
    const unsigned tile_off = SUB == 8 ? 0u : (unsigned)(((L.z0 >> 2) * 2 + (L.y0 >> 2)) * 2 + L.h) * (TILE_CELLS * 16u);
    unsigned long long inside = 0;
    for (int k = 0; k < SHARE; ++k) {
        int c = first + STRIDE * k;
        if (SUB == 4 && c >= TILE_CELLS) c -= TILE_CELLS;
        const int cx = c % G::SIDE, cy = c / G::SIDE % G::SIDE, cz = c / G::SIDE / G::SIDE;
        if (cx > 0 && cx < G::SIDE - 1 && cy > 0 && cy < G::SIDE - 1 && cz > 0 && cz < G::SIDE - 1) inside |= 1ull << k;
    }
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K;
    const long long worker = (long long)blockIdx.x * QUARTERS + quarter, nworkers = (long long)gridDim.x * QUARTERS;
    const unsigned n0 = (unsigned)(p.nitems / p.unit * worker / nworkers * p.unit);
    const int cnt = (int)(p.nitems / p.unit * (worker + 1) / nworkers * p.unit - n0);
    const unsigned bar0 = smem_u32(&bars[quarter * NBUF]), issued0 = smem_u32(&issued[quarter * NBUF]);
    const unsigned tiles = smem_u32(smem) + quarter * (NBUF * G::BUF_BYTES);
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K;
    bool failed = false;

    // one lane: fetch the tile of the team's item i into its buffer
    auto issue = [&](int i) {
        const unsigned n = n0 + i, blk = n / (unsigned)p.Q;
        const int q = (int)(n - blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const unsigned tile = tiles + (i % NBUF) * G::BUF_BYTES, bar = bar0 + 8 * (i % NBUF);
        fence_proxy_async();  // earlier accesses to the buffer precede the bulk copies' writes
        mbar_expect_tx(bar, G::CELLS * 16);
        if (SUB == 8) {
            tma_load_4d(tile, &in_map, bar, (bx * 8 - 1) * 4, by * 8 - 1, bz * 8 - 1, q);
        } else {
            for (int sub = 0; sub < 8; ++sub)
                tma_load_4d(tile + sub * 216 * 16, &in_map, bar, (bx * 8 + (sub & 1) * 4 - 1) * 4, by * 8 + ((sub >> 1) & 1) * 4 - 1,
                            bz * 8 + (sub >> 2) * 4 - 1, q);
        }
        st_release_shared(issued0 + 4 * (i % NBUF), i);
    };
    // Item i's tile has landed. Consecutive items of a buffer belong to different warps of the team, so a warp first
    // makes sure that its item's copy has been started at all: while the item before it is still on its way, the
    // barrier's parity would say "done" for a phase that has not begun.
    auto wait_tile = [&](int i) {
        unsigned spins = 0;
        while (ld_acquire_shared(issued0 + 4 * (i % NBUF)) != i && ++spins < kSpinLimit) {}
        if (spins >= kSpinLimit || !mbar_wait_bounded(bar0 + 8 * (i % NBUF), (unsigned)(i / NBUF) & 1u, kSpinLimit)) failed = true;
        __syncwarp();
    };
    auto claim = [&]() {  // the next item, for whichever warp is free
        int i = 0;
        if (lane == 0) i = atomicAdd(&claimed[quarter], 1);
        return __shfl_sync(0xffffffffu, i, 0);
    };
    previous_done();
    if (role == 0 && lane == 0)
        for (int i = 0; i < NBUF && i < cnt; ++i) issue(i);
    __syncwarp();
    int i = claim();

    int blk = (int)(n0 / (unsigned)p.Q), q0 = (int)(n0 - (unsigned)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);  // items of this region
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + L.z0) * p.N + (by * 8 + L.y0)) * p.K + bx * 8 + 4 * L.h;  // own patch, native layout
        quad_load_params(p.packed + (size_t)blk * PACK_F, role, lane, tm, [&] {
            if (i0 > 0) {
                tmem_fence_before();
                team_sync<TEAM>(quarter);  // the other warp no longer reads the old region's weights
                tmem_fence_after();
            }
        });
        if (role == 0) quad_load_wsum(p.wsum, blk, lane, tm);
        tmem_wait_st();
        tmem_fence_before();
        team_sync<TEAM>(quarter);
        tmem_fence_after();

        for (int next = 0; i < i0 + here; i = next) {
            const int q = q0 + i - i0;
            const unsigned tile = tiles + (i % NBUF) * G::BUF_BYTES;
            wait_tile(i);

            u64 piv[2], negm[2], inv[2];
            float halo[8], fresh[8];  // per sample: sum, sum of squares, relative to the pivot
            {
                const unsigned t0 = tile + tile_off;
                constexpr int BATCH = SUB == 8 ? 16 : 18;
                auto cell = [&](int k) {
                    int c = first + STRIDE * k;
                    if (SUB == 4 && c >= TILE_CELLS) c -= TILE_CELLS;
                    return t0 + (unsigned)c * 16u;
                };
                auto mine = [&](int k) { return SUB == 4 || first + STRIDE * k < TILE_CELLS; };
                u64 s2[2] = {0, 0}, q2[2] = {0, 0};
#pragma unroll 1
                for (int k0 = 0; k0 < SHARE; k0 += BATCH) {
                    u64 v[BATCH][2];
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) {
                        v[k][0] = v[k][1] = 0;
                        if (mine(k0 + k)) lds128u(cell(k0 + k), v[k][0], v[k][1]);
                    }
#pragma unroll
                    for (int k = 0; k < BATCH; ++k) {
                        s2[0] = fadd2(s2[0], v[k][0]);
                        s2[1] = fadd2(s2[1], v[k][1]);
                    }
                }
                auto spread = [&]() {
                    unpack2(s2[0], halo[0], halo[1]);
                    unpack2(s2[1], halo[2], halo[3]);
                    unpack2(q2[0], halo[4], halo[5]);
                    unpack2(q2[1], halo[6], halo[7]);
                };
                spread();
                quad_tile_sum8<SUB>(halo, lane);  // any pivot near the mean will do
                constexpr float per_cell = 1.0f / TILE_CELLS;
                piv[0] = pack2(halo[0] * per_cell, halo[1] * per_cell);
                piv[1] = pack2(halo[2] * per_cell, halo[3] * per_cell);
                const u64 neg[2] = {fmul2(piv[0], pack2(-1.0f, -1.0f)), fmul2(piv[1], pack2(-1.0f, -1.0f))};
                s2[0] = s2[1] = 0;
#pragma unroll 1
                for (int k0 = 0; k0 < SHARE; k0 += BATCH) {
                    u64 v[BATCH][2];
                    const unsigned in = (unsigned)(inside >> k0);
#pragma unroll
                    for (int k = 0; k < BATCH; ++k)
                        if (mine(k0 + k)) lds128u(cell(k0 + k), v[k][0], v[k][1]);
#pragma unroll
                    for (int k = 0; k < BATCH; ++k)
                        if (mine(k0 + k)) {
                            const float f = in >> k & 1 ? 0.0f : 1.0f;
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                v[k][j] = fadd2(v[k][j], neg[j]);
                                const u64 m = fmul2(v[k][j], pack2(f, f));
                                s2[j] = fadd2(s2[j], m);
                                ffma2(q2[j], m, v[k][j]);
                            }
                            sts128u(cell(k0 + k), v[k][0], v[k][1]);
                        }
                }
                spread();
                quad_tile_sum8<SUB, double>(halo, lane);  // enters every iteration
                __syncwarp();
            }

            const unsigned win = tile + L.cell0 * 16u;  // window cell (0, 0, 0) of this lane
            unsigned rows[4];
#pragma unroll
            for (int ry = 0; ry < 4; ++ry) rows[ry] = win + (unsigned)(ry * L.ysgn * G::ROW * 16);
            const size_t own = ((size_t)q * P + g0) * 4;  // the lane's cells in an IL4 tensor
            const long long zstr = wzs * 4, ystr = wys * 4;
            // The sums over the lane's own cells -> over the tile's interior
            auto sum_fresh = [&](const u64 (&v)[4][4][2], auto add) {
                u64 s2[2] = {0, 0}, q2[2] = {0, 0};
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o)
#pragma unroll
                        for (int k2 = 0; k2 < 2; ++k2) {
                            s2[k2] = fadd2(s2[k2], v[n][o][k2]);
                            ffma2(q2[k2], v[n][o][k2], v[n][o][k2]);
                        }
                unpack2(s2[0], fresh[0], fresh[1]);
                unpack2(s2[1], fresh[2], fresh[3]);
                unpack2(q2[0], fresh[4], fresh[5]);
                unpack2(q2[1], fresh[6], fresh[7]);
                quad_tile_sum8<SUB, decltype(add)>(fresh, lane);
            };
            auto own_cell = [&](int n, int o) {
                return win + (unsigned)((1 + o) * L.xsgn * 16 + (1 + (n & 1)) * L.ysgn * G::ROW * 16) + (1 + (n >> 1)) * G::PLANE * 16u;
            };
            {
                u64 v[4][4][2];
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o) lds128u(own_cell(n, o), v[n][o][0], v[n][o][1]);
                sum_fresh(v, 0.0);  // the step's input: added in double above the lane
            }
            for (int t = 0; t < p.inner; ++t) {
                const bool last = t + 1 == p.inner;
                {
                    constexpr float per_cell = 1.0f / TILE_CELLS;
                    float m[4], sd[4], rs[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        m[s] = (halo[s] + fresh[s]) * per_cell;
                        const float var = fmaxf(fmaf(-m[s], m[s], (halo[4 + s] + fresh[4 + s]) * per_cell), 0.0f);
                        if (SUB == 4) {  // as the kernel that blocks of 4 had before
                            sd[s] = __fsqrt_rn(var);
                            rs[s] = __frcp_rn(sd[s] + p.eps);
                        } else {  // as step_fast.cu: approximate square root and reciprocal, a few ulp
                            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sd[s]) : "f"(var));
                            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rs[s]) : "f"(sd[s] + p.eps));
                        }
                    }
                    negm[0] = pack2(-m[0], -m[1]);
                    negm[1] = pack2(-m[2], -m[3]);
                    inv[0] = pack2(rs[0], rs[1]);
                    inv[1] = pack2(rs[2], rs[3]);
                    if (SAVE && quad_tile_leader<SUB>(lane)) {
                        const size_t ntiles = (size_t)nbx * nby * (p.M >> 3) * (SUB == 8 ? 1 : 8);
                        float4 *to = p.tile_stats + (((size_t)t * p.Q + q) * ntiles + quad_tile_of(L, blk)) * QS_COUNT;
                        float c[4];
                        unpack2(piv[0], c[0], c[1]);
                        unpack2(piv[1], c[2], c[3]);
                        to[QS_MEAN] = make_float4(c[0] + m[0], c[1] + m[1], c[2] + m[2], c[3] + m[3]);
                        to[QS_INV] = make_float4(rs[0], rs[1], rs[2], rs[3]);
                        to[QS_STD] = make_float4(sd[0], sd[1], sd[2], sd[3]);
                        to[QS_STDEPS] = make_float4(sd[0] + p.eps, sd[1] + p.eps, sd[2] + p.eps, sd[3] + p.eps);
                    }
                    __syncwarp();
                }
                u64 acc[4][4][2], hold[2] = {0, 0};
                float *const sh = SAVE ? p.save_h + (size_t)t * p.Q * P * 4 + own : nullptr;
                quad_stencil<G::PLANE, NORMED>(rows, L.xsgn * 16, tm, acc, negm, [&](int n, int o, float scale, float bias, u64 c0, u64 c1) {
                    acc[n][o][0] = ffma2r(acc[n][o][0], inv[0], pack2(bias, bias));
                    acc[n][o][1] = ffma2r(acc[n][o][1], inv[1], pack2(bias, bias));
                    if (SAVE) {  // two neighbours at a time
                        if (o & 1)
                            stg256(sh + (n >> 1) * zstr + (n & 1) * ystr + 8 * ((o >> 1) ^ L.h), L.h ? acc[n][o][0] : hold[0],
                                   L.h ? acc[n][o][1] : hold[1], L.h ? hold[0] : acc[n][o][0], L.h ? hold[1] : acc[n][o][1]);
                        else
                            hold[0] = acc[n][o][0], hold[1] = acc[n][o][1];
                    }
                    acc[n][o][0] = act_residual2<ACT>(acc[n][o][0], scale, c0);
                    acc[n][o][1] = act_residual2<ACT>(acc[n][o][1], scale, c1);
                });
                __syncwarp();  // every lane has read its window
                if (!last) {
#pragma unroll
                    for (int o = 0; o < 4; ++o)
#pragma unroll
                        for (int n = 0; n < 4; ++n) sts128u(own_cell(n, o), acc[n][o][0], acc[n][o][1]);
                    sum_fresh(acc, 0.0f);
                    __syncwarp();
                } else {
                    if (lane == 0 && i + NBUF < cnt) issue(i + NBUF);  // the tile is dead: fetch the next one
                    __syncwarp();
                    next = claim();
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int o = 0; o < 4; ++o)
#pragma unroll
                            for (int k2 = 0; k2 < 2; ++k2) acc[n][o][k2] = fadd2(acc[n][o][k2], piv[k2]);
                    if (p.y) quad_store(p.y + own, zstr, ystr, L.h, acc);
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

// ---- layout conversion at the ends of a loop --------------------------------------------------------------
// IL4 -> [B, P], normalised on the way when statistics are given. grid ceil(B / 4) * parts, one dimension: gridDim.y
// ends at 65535
__global__ void __launch_bounds__(256) from_il4_k(const float4 *il, const float2 *stats, const float *gamma, const float *beta,
                                                  float *y, int B, size_t P, unsigned parts)
{
    const unsigned q = blockIdx.x / parts;
    const size_t c = (size_t)(blockIdx.x - q * parts) * 256 + threadIdx.x;
    previous_done();
    if (c >= P) return;
    const float4 v4 = il[(size_t)q * P + c];
    float v[4] = {v4.x, v4.y, v4.z, v4.w};
    float g = 1.0f, b = 0.0f;
    if (stats) {
        g = gamma[c];
        b = beta[c];
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
        if (4 * q + s < B) {
            if (stats) {
                const float2 mr = stats[4 * q + s];
                v[s] = fmaf((v[s] - mr.x) * mr.y, g, b);
            }
            y[(size_t)(4 * q + s) * P + c] = v[s];
        }
}

// [B, P] -> [Q][P][4]. One cell per thread and step: four coalesced 4-byte reads, one coalesced 16-byte write. Samples
// beyond B: zeros if these are gradients; activations are copies of sample B - 1. Zeros there could end in infinities or NaN where no
// sample does (a constant block or grid and an eps of zero), and zero gradients do not keep those out of the parameters' sums.
__device__ __forceinline__ void to_il4(const float *__restrict__ x, float4 *__restrict__ il, int B, size_t P, int q, size_t part, bool gradient)
{
    const size_t c = part * 256 + threadIdx.x;
    if (c >= P) return;
    float v[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) v[s] = 4 * q + s < B || !gradient ? x[(size_t)min(4 * q + s, B - 1) * P + c] : 0.0f;
    il[(size_t)q * P + c] = make_float4(v[0], v[1], v[2], v[3]);
}

// Parameters in the order of the stencil: vector v of a region is, for every lane, the four x-neighbouring weights of
// one (neuron row, tap), v = 0 .. 107 in the order of the uses in quad_stencil (three x-taps each), then the four rows
// of b, then of s. TRANS: the weights of the backward sum, in which a cell collects from the neurons of its own block
// that read it: the neuron at tap t sees the cell through its tap 26 - t; zero across the block's border. Four CTAs of 256 threads per
// region, so that small grids fill the GPU; reads are 16-byte pieces, writes whole lines.
constexpr int kPackCtas = 4;
template <int SUB, bool TRANS>
__device__ __forceinline__ void quad_pack(const float *__restrict__ w, const float *__restrict__ b, const float *__restrict__ s,
                                          float *__restrict__ packed, size_t tap, int M, int N, int K, int cta)
{
    __shared__ unsigned char uses[36];  // (a * 3 + b) | n << 4
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
    const int nbx = K >> 3, nby = N >> 3, blk = cta / kPackCtas;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t g0 = ((size_t)(bz * 8 + L.z0) * N + (by * 8 + L.y0)) * K + bx * 8 + 4 * L.h;
    const long long zs = (long long)N * K, ys = (long long)L.ysgn * K;
    float4 *out = reinterpret_cast<float4 *>(packed + (size_t)blk * quad::PACK_F) + lane;
#pragma unroll
    for (int i = 0; i < (quad::VECS + 8 * kPackCtas - 1) / (8 * kPackCtas); ++i) {
        const int v = (i * kPackCtas + cta % kPackCtas) * 8 + (threadIdx.x >> 5);
        if (v >= quad::VECS) break;
        int n;
        float4 r;
        if (v < 108) {
            const int u = uses[v / 3], c = v % 3;
            n = u >> 4;
            // the tap as the grid numbers it (gridnet/backend_torch.py:283-298)
            const int ta = (u & 15) / 3, tb = L.ysgn < 0 ? 2 - (u & 15) % 3 : (u & 15) % 3, tc = L.h ? 2 - c : c;
            const int t = ta * 9 + tb * 3 + tc;
            const size_t own = g0 + (n >> 1) * zs + (n & 1) * ys;
            if (!TRANS) {
                const float *src = w + (size_t)t * tap + own;
                if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) r = *reinterpret_cast<const float4 *>(src);
                else r = make_float4(src[0], src[1], src[2], src[3]);
            } else {
                const int lz = L.z0 + (n >> 1) + ta - 1, ly = L.y0 + L.ysgn * (n & 1) + tb - 1;  // source row in the region
                const int mask = ~(SUB - 1);
                const bool row = lz >= 0 && lz < 8 && ly >= 0 && ly < 8 && ((lz ^ (L.z0 + (n >> 1))) & mask & 7) == 0 &&
                                 ((ly ^ (L.y0 + L.ysgn * (n & 1))) & mask & 7) == 0;
                const float *src = w + (size_t)(26 - t) * tap + own + (ta - 1) * zs + (long long)(tb - 1) * K + (tc - 1);
                float f[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int x = 4 * L.h + i, lx = x + tc - 1;
                    f[i] = row && lx >= 0 && lx < 8 && ((lx ^ x) & mask & 7) == 0 ? src[i] : 0.0f;
                }
                r = make_float4(f[0], f[1], f[2], f[3]);
            }
        } else {
            n = v & 3;
            const float *src = (v < 112 ? b : s) + g0 + (n >> 1) * zs + (n & 1) * ys;
            if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) r = *reinterpret_cast<const float4 *>(src);
            else r = make_float4(src[0], src[1], src[2], src[3]);
        }
        out[v * 32] = L.h ? make_float4(r.w, r.z, r.y, r.x) : r;
    }
}

// The same for tap_stencil (step_taps.cu): its order of uses and its lanes, whose rows of four lie along x as they are.
template <int SUB>
__device__ __forceinline__ void tap_pack(const float *__restrict__ w, const float *__restrict__ b, const float *__restrict__ s,
                                         float *__restrict__ packed, size_t tap, int N, int K, int cta)
{
    __shared__ unsigned char uses[36];  // (a * 3 + b) | n << 4
    if (threadIdx.x == 0) {
        int k = 0;
        for (int rz = 0; rz < 6; ++rz)
            for (int bb = 0; bb < 3; ++bb)
                for (int n = 0; n < 4; ++n)
                    if (rz - n >= 0 && rz - n <= 2) uses[k++] = (unsigned char)(((rz - n) * 3 + bb) | n << 4);
    }
    __syncthreads();
    const TapLane L(threadIdx.x & 31);
    const int nbx = K >> 3, nby = N >> 3, blk = cta / kPackCtas;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t g0 = ((size_t)(bz * 8 + 4 * L.zp) * N + (by * 8 + L.y)) * K + bx * 8 + 4 * L.h, zs = (size_t)N * K;
    float4 *out = reinterpret_cast<float4 *>(packed + (size_t)blk * quad::PACK_F) + (threadIdx.x & 31);
#pragma unroll
    for (int i = 0; i < (quad::VECS + 8 * kPackCtas - 1) / (8 * kPackCtas); ++i) {
        const int v = (i * kPackCtas + cta % kPackCtas) * 8 + (threadIdx.x >> 5);
        if (v >= quad::VECS) break;
        const float *src;
        if (v < 108) {
            const int u = uses[v / 3];
            src = w + (size_t)((u & 15) * 3 + v % 3) * tap + g0 + (u >> 4) * zs;
        } else {
            src = (v < 112 ? b : s) + g0 + (v & 3) * zs;
        }
        out[v * 32] = (reinterpret_cast<uintptr_t>(src) & 15) == 0 ? *reinterpret_cast<const float4 *>(src) : make_float4(src[0], src[1], src[2], src[3]);
    }
}

// The sum of every neuron's 27 weights, for per-block normalisation: vector n of a region is, for every lane, its neuron
// row n. One warp per row, two
// regions per CTA.
template <int SUB>
__device__ __forceinline__ void quad_wsum(const float *__restrict__ w, float4 *__restrict__ wsum, int M, int N, int K, int cta)
{
    const int lane = threadIdx.x & 31, n = (threadIdx.x >> 5) & 3;
    const QuadLane<SUB> L(lane);
    const int nbx = K >> 3, nby = N >> 3, blk = 2 * cta + (threadIdx.x >> 7);
    if (blk >= (M >> 3) * nby * nbx) return;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const float *src = w + ((size_t)(bz * 8 + L.z0 + (n >> 1)) * N + (by * 8 + L.y0 + L.ysgn * (n & 1))) * K + bx * 8 + 4 * L.h;
    const bool al = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int t = 0; t < 27; ++t) {
        const float *a = src + (size_t)t * P;
        const float4 v = al ? *reinterpret_cast<const float4 *>(a) : make_float4(a[0], a[1], a[2], a[3]);
        r.x += v.x, r.y += v.y, r.z += v.z, r.w += v.w;
    }
    wsum[(size_t)blk * 128 + (threadIdx.x & 127)] = L.h ? make_float4(r.w, r.z, r.y, r.x) : r;
}

// (gamma, beta) of every tile cell of every region, in the order of the tile buffer
template <int SUB>
__device__ __forceinline__ void quad_table(const float *__restrict__ gamma, const float *__restrict__ beta, float2 *__restrict__ gbt, int M,
                                           int N, int K, int cta)
{
    using G = QuadGeo<SUB>;
    const int nbx = K >> 3, nby = N >> 3, blk = cta;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    for (int c = threadIdx.x; c < G::CELLS; c += 256) {
        int cz, cy, cx;
        G::cell(c, cz, cy, cx);
        const int z = bz * 8 + cz - 1, y = by * 8 + cy - 1, x = bx * 8 + cx - 1;
        float2 gb = make_float2(0.0f, 0.0f);
        if (z >= 0 && z < M && y >= 0 && y < N && x >= 0 && x < K) {
            const size_t i = ((size_t)z * N + y) * K + x;
            gb = make_float2(gamma[i], beta[i]);
        }
        gbt[(size_t)blk * G::CELLS + c] = gb;
    }
}

// Everything that has to be re-ordered before a step or a loop, in one launch (a launch costs the host as much as the
// kernel of a small grid takes): CTAs first .. first + n of job j do that job.
struct PrepareArgs {
    QuadPrepare a;
    int M, N, K;
    unsigned end[5];  // last CTA + 1 of: pack, transposed pack, weight sums, table, conversion
    unsigned parts;   // conversion: CTAs per quad
    unsigned pack;    // packing: CTAs per branch
    int branches;
};
template <int SUB, bool ORDERED>
__global__ void __launch_bounds__(256) quad_prepare_k(const PrepareArgs p)
{
    const unsigned c = blockIdx.x;
    const QuadPrepare &a = p.a;
    const size_t P = (size_t)p.M * p.N * p.K, tap = p.branches * P;
    if (c < p.end[1]) {  // branch k of a gated network: weights [27][2][P], bias [2][P]
        const unsigned j = c < p.end[0] ? c : c - p.end[0], k = j / p.pack;
        const size_t to = (size_t)k * (p.pack / kPackCtas) * quad::PACK_F;
        if (c < p.end[0]) {
            if (ORDERED) tap_pack<SUB>(a.w + k * P, a.b + k * P, a.s, a.packed + to, tap, p.N, p.K, (int)(j % p.pack));
            else quad_pack<SUB, false>(a.w + k * P, a.b + k * P, a.s, a.packed + to, tap, p.M, p.N, p.K, (int)(j % p.pack));
        }
        else quad_pack<SUB, true>(a.w + k * P, a.b_t + k * P, a.s, a.packed_t + to, tap, p.M, p.N, p.K, (int)(j % p.pack));
    }
    else if (c < p.end[2]) quad_wsum<SUB>(a.w, reinterpret_cast<float4 *>(a.wsum), p.M, p.N, p.K, (int)(c - p.end[1]));
    else if (c < p.end[3]) quad_table<SUB>(a.gamma, a.beta, a.gbt, p.M, p.N, p.K, (int)(c - p.end[2]));
    else to_il4(a.x, reinterpret_cast<float4 *>(a.il), a.B, P, (int)((c - p.end[3]) / p.parts), (c - p.end[3]) % p.parts, a.gradient);
}

// ---- host side -----------------------------------------------------------------------------------------------
int quad_tile_cells(int block) { return block == 8 ? QuadGeo<8>::CELLS : QuadGeo<4>::CELLS; }

bool quad_applicable(int M, int N, int K, int block, int inner)
{
    if ((block != 8 && block != 4) || inner < 1 || M % 8 || N % 8 || K % 8) return false;
    if ((long long)M * N * K >= (1LL << 31) / 4) return false;
    return encode_tiled_fn() != nullptr;
}

// tensor map over an IL4 buffer, box = one tile (10^3 or 6^3 cells), or with rows of `row` cells
int quad_make_map(CUtensorMap *map, const float *il, int M, int N, int K, int Q, int block, int row)
{
    const cuuint32_t side = block == 8 ? 10 : 6;
    if (row == 0) row = (int)side;
    MapKey key{il, 4 * row, 0, {M, N, K, Q}};
    (void)cudaGetDevice(&key.dev);
    if (tensor_map_cache_get(key, map)) return GN_OK;
    const cuuint64_t dims[4] = {(cuuint64_t)K * 4, (cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)Q};
    const cuuint64_t strides[3] = {(cuuint64_t)K * 16, (cuuint64_t)N * K * 16, (cuuint64_t)M * N * K * 16};
    const cuuint32_t box[4] = {4 * (cuuint32_t)row, side, side, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(il), dims, strides, box, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        record_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
        return GN_ERR_CUDA;
    }
    tensor_map_cache_put(key, *map);
    return GN_OK;
}

int launch_from_il4(const float *il, const float2 *stats, const float *gamma, const float *beta, float *y, int B, long long P,
                    cudaStream_t st)
{
    const unsigned parts = (unsigned)((P + 255) / 256);
    const unsigned long long n = (unsigned long long)parts * ((B + 3) / 4);
    if (n >= 1ull << 31) return GN_ERR_UNSUPPORTED;
    launch_after(from_il4_k, (unsigned)n, 256, 0, st, reinterpret_cast<const float4 *>(il), stats, gamma, beta, y, B, (size_t)P, parts);
    return check_launch("from_il4");
}

size_t quad_tiles(int M, int N, int K, int block) { return (size_t)(M / block) * (N / block) * (K / block); }
size_t quad_stats_vectors(int M, int N, int K, int Q, int inner, int block) { return (size_t)inner * Q * quad_tiles(M, N, K, block) * QS_COUNT; }
size_t quad_packed_floats(int M, int N, int K) { return (size_t)(M / 8) * (N / 8) * (K / 8) * quad::PACK_F; }

int launch_quad_prepare(const QuadPrepare &a, int M, int N, int K, int block, cudaStream_t st)
{
    const unsigned regions = (unsigned)((M / 8) * (N / 8) * (K / 8));
    PrepareArgs p{a, M, N, K, {}, (unsigned)(((long long)M * N * K + 255) / 256), regions * kPackCtas, a.gated ? 2 : 1};
    const unsigned long long jobs[5] = {a.packed ? p.pack * p.branches : 0u, a.packed_t ? p.pack * p.branches : 0u,
                                        a.wsum ? (regions + 1) / 2 : 0u, a.gbt ? regions : 0u,
                                        a.il ? (unsigned long long)p.parts * ((a.B + 3) / 4) : 0u};
    unsigned long long n = 0;
    for (int j = 0; j < 5; ++j) {
        n += jobs[j];
        if (n >= 1ull << 31) return GN_ERR_UNSUPPORTED;
        p.end[j] = (unsigned)n;
    }
    if (n == 0) return GN_OK;
    if (block == 8 && a.ordered) quad_prepare_k<8, true><<<(unsigned)n, 256, 0, st>>>(p);
    else if (block == 8) quad_prepare_k<8, false><<<(unsigned)n, 256, 0, st>>>(p);
    else if (a.ordered) quad_prepare_k<4, true><<<(unsigned)n, 256, 0, st>>>(p);
    else quad_prepare_k<4, false><<<(unsigned)n, 256, 0, st>>>(p);
    return check_launch("quad_prepare");
}

template <int SUB, int ACT, bool SAVE>
static int launch_quad_one(const CUtensorMap &map, const QuadParams &p, unsigned ctas, cudaStream_t st)
{
    using G = QuadGeo<SUB>;
    auto kern = step_fwd_quad<SUB, ACT, SAVE>;
    constexpr int smem = quad::QUARTERS * G::NBUF * G::BUF_BYTES;
    static_assert(smem <= 232448 - 1024 - 256, "shared memory budget of one SM");
    static unsigned long long attr_set = 0;
    if (first_use_on_device(&attr_set)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            record_cuda_error(e, "cudaFuncSetAttribute(step_fwd_quad)");
            return GN_ERR_CUDA;
        }
    }
    launch_after(kern, ctas, 128 * G::TEAM, smem, st, map, p);
    return check_launch("step_fwd_quad");
}

template <int SUB, int ACT>
static int launch_quad_act(const CUtensorMap &map, const QuadParams &p, unsigned ctas, cudaStream_t st)
{
    return p.save_h ? launch_quad_one<SUB, ACT, true>(map, p, ctas, st) : launch_quad_one<SUB, ACT, false>(map, p, ctas, st);
}

template <int SUB>
static int launch_quad_sub(const CUtensorMap &map, const QuadParams &p, unsigned ctas, int act, cudaStream_t st)
{
    switch (act) {
    case GN_ACT_RELU: return launch_quad_act<SUB, GN_ACT_RELU>(map, p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_quad_act<SUB, GN_ACT_LEAKY_RELU>(map, p, ctas, st);
    case GN_ACT_SILU: return launch_quad_act<SUB, GN_ACT_SILU>(map, p, ctas, st);
    default: return launch_quad_act<SUB, GN_ACT_TANH>(map, p, ctas, st);
    }
}

int launch_step_fwd_quad(const QuadStep &a, int act, cudaStream_t st)
{
    if (!a.wsum) return launch_step_fwd_taps(a, act, st);
    if (a.in_stats || a.out_partials || !a.save_h != !a.tile_stats) return GN_ERR_UNSUPPORTED;
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, a.block);
    if (rc != GN_OK) return rc;
    QuadParams p{};
    p.packed = a.packed;
    p.wsum = a.wsum; p.tile_stats = a.tile_stats; p.eps = a.eps;
    p.y = a.out_il4; p.save_h = a.save_h;
    p.error_flag = a.error_flag ? a.error_flag : device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = (long long)(a.M / 8) * (a.N / 8) * (a.K / 8) * a.Q;
    long long ctas = (p.nitems + quad::QUARTERS - 1) / quad::QUARTERS;
    if (ctas > sm_count()) ctas = sm_count();
    p.unit = quad_split_unit(p.nitems, ctas, p.Q);
    return a.block == 8 ? launch_quad_sub<8>(map, p, (unsigned)ctas, act, st) : launch_quad_sub<4>(map, p, (unsigned)ctas, act, st);
}

}  // namespace gn
