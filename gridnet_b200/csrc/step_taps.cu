// Float forward of the block-local update on the quad layout (block 8 and 4, per-block normalisation off), weights in tensor
// memory and four samples per lane as described in step_quad.cu, every neuron's taps added in the order of their numbers: the same
// bits as the register-patch kernel (step_fast.cu), statistics included. Loops with gradients need that: rounding that
// differs is amplified from step to step (block 4, 8 x 16 iterations, silu: gradients up to 3e-5 apart in the 2-norm), and
// where it carries a pre-activation over the kink of (leaky) relu gradients jump (40 x 56 x 72, 4 x 10 iterations: 1e-4).
//
// What differs from step_quad.cu is the split of a region over the lanes and the layout of the tile (taps_geo.cuh). Fusion as in
// step_fast.cu: FUSE_IN normalises the landed tile in place with the whole-grid statistics of the previous step and a per-region
// (gamma, beta) table; every launch can reduce (sum, sum of squares) per sample and region of what it writes.
// What bounds it: an iteration of an item takes 2820 cycles where two warps share a scheduler (3100 alone), 2270 of them the 864
// packed FMAs, which get their operands from the register file at 2.6 cycles each instead of 2.0, the rest activation functions.
// Around the iterations an item waits for its tile, normalises it and leaves sums and results. For that:
//   - A lane's own cells stay in registers from their normalisation to the last iteration (92 instead of 124 shared loads per
//     iteration). Only the halo's 488 entries of the (gamma, beta) table are in shared memory, a lane's own in tensor memory.
//   - A warp takes the next item of its quarter when it is free (64^3: 1597 -> 1553 us; for its tile it may have to wait for the other
//     warp's buffer), and asks for the first half of the next region's parameters before it waits for the other warp.
//   - The next region's parameters are not prefetched to L2: 256^3 x 32 93.5 -> 88.5 ms, 128^3 x 16 with gradients 9.12 -> 8.85 ms, 40 x 56 x 72
//     290 -> 285 us, at the price of 1554 -> 1565 us at 64^3. Prefetching tiles was slower too (256^3: 99.5 ms).
// Measured before and after: 64^3 x 64, 4 x 12 iterations 1652 -> 1565 us; 40 x 56 x 72 x 37, 3 x 6 315 -> 285 us; 256^3 x 32, 2 x 32 96.5 ->
// 88.5 ms (at 1.77 GHz); 64^3 x 128, block 4, 8 x 16 with gradients 41.3 -> 40.4 ms. Letting one or two warps of a quarter at a time into
// the 27-tap sums, so that the rest of an item overlaps with another's, was slower (1754 and 1721 us).
// Block 8: tiles by bulk tensor copy. Block 4: each warp fetches its own next tile, cell by cell and asynchronously; its
// eight small tiles have to lie an odd number of cells apart, which bulk tensor copies cannot do.
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "taps_geo.cuh"
#include "tmem.cuh"

namespace gn {

namespace {

using namespace quad;
// block 8: halo cells of a tile, whose (gamma, beta) are kept in shared memory; those of a lane's own cells and the places of its
// halo cells are in the columns of tensor memory that parameters leave free
constexpr int HALO8 = 488, COL_GAMMA = 464, COL_BETA = 480, COL_PLACE = 496;

struct TapParams {
    const float *packed;     // [regions][PACK_F], QuadPrepare::ordered
    const float2 *gbt;       // FUSE_IN: (gamma, beta) per tile cell of every region, in the order of QuadGeo
    const float2 *in_stats;  // FUSE_IN: [4 Q] (mean, rstd)
    const float *in;         // block 4: IL4
    double2 *out_partials;   // [4 Q][nparts]: slot `region` of every row is written; nullptr: not wanted
    int nparts;
    float *y;                // IL4; nullptr: not wanted (replay)
    float *save_h;           // SAVE: [inner][Q][P][4]
    int *error_flag;
    int M, N, K, Q, inner;
    int params_old;          // the kernel before this one did not write packed or gbt
    long long nitems;        // regions * Q
    int unit;                // quad_split_unit
};

// 16 bytes to shared memory, asynchronously; zeros where !inside (src is then not read)
__device__ __forceinline__ void cp_async16_or_zero(unsigned dst, const float *src, bool inside)
{
    const int n = inside ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// Block 4: the eight tiles of region (bx, by, bz), quad q. Four lanes per tile: first the 36 rows' inner cells, whole sectors,
// then the two outer cells of two rows at a time.
__device__ __forceinline__ void fetch_tiles4(unsigned tile, const TapParams &p, int bx, int by, int bz, int q, int lane)
{
    using G = TapGeo<4>;
    const int slot = lane >> 2, r = lane & 3;
    const int z0 = bz * 8 + (slot >> 2) * 4 - 1, x0 = bx * 8 + ((slot >> 1) & 1) * 4 - 1, y0 = by * 8 + (slot & 1) * 4 - 1;
    const bool zlo = z0 >= 0, zhi = z0 + 5 < p.M, ylo = y0 >= 0, yhi = y0 + 5 < p.N, xlo = x0 >= 0, xhi = x0 + 5 < p.K;
    const long long zstr = 4ll * p.N * p.K, ystr = 4ll * p.K;
    const float *const corner = p.in + ((long long)q * p.M + z0) * zstr + y0 * ystr + 4ll * x0;  // may lie outside, then not read
    const unsigned to = tile + (unsigned)(slot * G::TILE) * 16u;
    const int rr = r >> 1, side = (r & 1) * 5;
    const bool x_in = side ? xhi : xlo;
#pragma unroll
    for (int cz = 0; cz < 6; ++cz) {
        const bool z_in = cz == 0 ? zlo : (cz == 5 ? zhi : true);
        const float *const plane = corner + cz * zstr;
#pragma unroll
        for (int cy = 0; cy < 6; ++cy) {
            const bool in = z_in && (cy == 0 ? ylo : (cy == 5 ? yhi : true));
            const float *src = plane + cy * ystr + 4 * (1 + r);
            cp_async16_or_zero(to + (unsigned)(cz * G::PLANE + cy * G::ROW + 1 + r) * 16u, in ? src : p.in, in);
        }
#pragma unroll
        for (int c2 = 0; c2 < 6; c2 += 2) {
            const bool in = z_in && x_in && (c2 + rr == 0 ? ylo : (c2 + rr == 5 ? yhi : true));
            const float *src = plane + (c2 + rr) * ystr + 4 * side;
            cp_async16_or_zero(to + (unsigned)(cz * G::PLANE + (c2 + rr) * G::ROW + side) * 16u, in ? src : p.in, in);
        }
    }
}

// Block 8: halo cell j = 0 .. 487 of a tile, as its index among the 10^3 cells: two z faces of 100, then two y faces of 8 x 10,
// then two x faces of 8 x 8
__device__ __forceinline__ int halo_cell(int j)
{
    if (j < 200) return j + (j >= 100 ? 800 : 0);
    if (j < 360) {
        const int e = j - 200, s = e >= 80 ? e - 80 : e;
        return (1 + s / 10) * 100 + (e >= 80 ? 90 : 0) + s % 10;
    }
    const int e = j - 360, s = e & 63;
    return (1 + (s >> 3)) * 100 + (1 + (s & 7)) * 10 + (e >= 64 ? 9 : 0);
}

template <int SUB, int ACT, bool FUSE_IN, bool SAVE>
__global__ void __launch_bounds__(128 * TapGeo<SUB>::TEAM, 1) step_fwd_taps(const __grid_constant__ CUtensorMap in_map, const TapParams p)
{
    using G = TapGeo<SUB>;
    constexpr int TEAM = G::TEAM, NBUF = G::NBUF;
    static_assert(TEAM == 2, "parameters and tables are loaded by two warps");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[QUARTERS * NBUF];
    __shared__ int issued[QUARTERS * NBUF];  // which item's copy into this buffer has been started last
    __shared__ int claimed[QUARTERS];        // items of the team that warps have taken
    __shared__ unsigned tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid == 0) {
        for (int i = 0; i < QUARTERS * NBUF; ++i) {
            mbar_init(smem_u32(&bars[i]), 1);
            issued[i] = -1;
        }
        for (int i = 0; i < QUARTERS; ++i) claimed[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    float2 *const gbs = reinterpret_cast<float2 *>(smem + QUARTERS * NBUF * G::BUF_BYTES) + quarter * HALO8;
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const TapLane L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K;
    const long long worker = (long long)blockIdx.x * QUARTERS + quarter, nworkers = (long long)gridDim.x * QUARTERS;
    const unsigned n0 = (unsigned)(p.nitems / p.unit * worker / nworkers * p.unit);
    const int cnt = (int)(p.nitems / p.unit * (worker + 1) / nworkers * p.unit - n0);
    const unsigned bar0 = smem_u32(&bars[quarter * NBUF]), issued0 = smem_u32(&issued[quarter * NBUF]);
    const unsigned tiles = smem_u32(smem) + quarter * (NBUF * G::BUF_BYTES);
    const long long zstr = 4ll * p.N * p.K;
    bool failed = false;

    // fetch the tile of the team's item i into its buffer: one lane (block 8), the whole warp (block 4)
    auto issue = [&](int i) {
        const unsigned n = n0 + i, blk = n / (unsigned)p.Q, buf = (unsigned)i % NBUF;
        const int q = (int)(n - blk * p.Q);
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const unsigned tile = tiles + buf * G::BUF_BYTES;
        if constexpr (SUB == 8) {
            fence_proxy_async();  // earlier accesses to the buffer precede the bulk copy's writes
            mbar_expect_tx(bar0 + 8 * buf, G::CELLS * 16);
            tma_load_4d(tile, &in_map, bar0 + 8 * buf, (bx * 8 - 1) * 4, by * 8 - 1, bz * 8 - 1, q);
            st_release_shared(issued0 + 4 * buf, i);
        } else {
            fetch_tiles4(tile, p, bx, by, bz, q, lane);
        }
    };
    auto wait_tile = [&](int i) {
        if constexpr (SUB == 8) {  // see step_fwd_quad
            const unsigned buf = (unsigned)i % NBUF;
            unsigned spins = 0;
            while (ld_acquire_shared(issued0 + 4 * buf) != i && ++spins < kSpinLimit) {}
            if (spins >= kSpinLimit || !mbar_wait_bounded(bar0 + 8 * buf, (unsigned)i / NBUF & 1u, kSpinLimit)) failed = true;
        } else {
            cp_async_wait_all();
        }
        __syncwarp();
    };
    // the warp's next item. Block 8: whoever is free takes the next one; with as many buffers as warps its tile has been asked for only
    // if the item two before it is done, else wait_tile waits for the other warp to finish that. Block 4: item i is fetched by the warp
    // that works on it, i mod TEAM.
    auto claim = [&](int last) {
        if constexpr (SUB == 8) {
            int i = 0;
            if (lane == 0) i = atomicAdd(&claimed[quarter], 1);
            return __shfl_sync(0xffffffffu, i, 0);
        } else {
            return last < 0 ? role : last + TEAM;
        }
    };
    auto begin = [&]() {
        previous_done();
        if constexpr (SUB == 8) {
            if (role == 0 && lane == 0)
                for (int i = 0; i < NBUF && i < cnt; ++i) issue(i);
        } else {
            if (role < cnt) issue(role);
        }
        __syncwarp();
    };
    if (FUSE_IN && SUB == 8 && role == 0) {
        float place[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const int l = halo_cell(min(c * 32 + lane, HALO8 - 1));
            place[c] = __int_as_float((l + l / 10) * 16);
        }
        tmem_st16(tm + COL_PLACE, place);
    }
    if (!p.params_old || cnt == 0) begin();  // else the first region's parameters come first

    int blk = (int)(n0 / (unsigned)p.Q), q0 = (int)(n0 - (unsigned)blk * p.Q);
    int i = claim(-1);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);  // items of this region
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + 4 * L.zp) * p.N + (by * 8 + L.y)) * p.K + bx * 8 + 4 * L.h;  // own patch
        quad_load_params(p.packed + (size_t)blk * PACK_F, role, lane, tm, [&] {
            if (i0 > 0) {
                tmem_fence_before();
                team_sync<TEAM>(quarter);  // the other warp no longer reads the old region's weights
                tmem_fence_after();
            }
        });
        if (FUSE_IN && SUB == 8) {
            const float2 *const table = p.gbt + (size_t)blk * QuadGeo<8>::CELLS;
            constexpr int STEPS = (16 + TEAM - 1) / TEAM;
            float2 gh[STEPS], go[8];
            const int n = 2 * role;  // planes whose own cells this warp looks after
#pragma unroll
            for (int c = 0; c < STEPS; ++c) {
                const int j = (c * TEAM + role) * 32 + lane;
                if (j < HALO8) gh[c] = table[halo_cell(j)];
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) go[c] = table[(4 * L.zp + n + (c >> 2) + 1) * 100 + (L.y + 1) * 10 + 4 * L.h + (c & 3) + 1];
#pragma unroll
            for (int c = 0; c < STEPS; ++c) {
                const int j = (c * TEAM + role) * 32 + lane;
                if (j < HALO8) gbs[j] = gh[c];
            }
            __syncwarp();  // tensor memory instructions want the whole warp together
            float ga[8], be[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                ga[c] = go[c].x;
                be[c] = go[c].y;
            }
            tmem_st8(tm + COL_GAMMA + 4 * n, ga);
            tmem_st8(tm + COL_BETA + 4 * n, be);
        }
        tmem_wait_st();
        if (i0 == 0 && p.params_old) begin();
        tmem_fence_before();
        team_sync<TEAM>(quarter);
        tmem_fence_after();

        for (int next; i < i0 + here; i = next) {
            const int q = q0 + i - i0;
            const unsigned tile = tiles + (unsigned)i % NBUF * G::BUF_BYTES;
            const unsigned win = tile + (unsigned)G::corner(L) * 16u;
            const unsigned mine = win + (unsigned)(G::PLANE + G::ROW + 1) * 16u;  // own cell (0, 0)
            u64 own[4][4][2];
            if (FUSE_IN) {
                u64 rs[2], mu[2];  // rstd, -mean
                {
                    float2 mr[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) mr[s] = p.in_stats[4 * q + s];
                    rs[0] = pack2(mr[0].y, mr[1].y);
                    rs[1] = pack2(mr[2].y, mr[3].y);
                    mu[0] = pack2(-mr[0].x, -mr[1].x);
                    mu[1] = pack2(-mr[2].x, -mr[3].x);
                }
                auto normed = [&](u64 v, int k2, float gm, float bt) {
                    return ffma2r(fmul2(fadd2(v, mu[k2]), rs[k2]), pack2(gm, gm), pack2(bt, bt));
                };
                if constexpr (SUB == 8) {
                    float place[16];
                    tmem_ld16(tm + COL_PLACE, place);
                    wait_tile(i);
                    tmem_wait_ld16(place);
#pragma unroll
                    for (int c0 = 0; c0 < 16; c0 += 8) {
                        u64 v[8][2];
                        float2 g2[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            g2[c] = gbs[min((c0 + c) * 32 + lane, HALO8 - 1)];
                            lds128u(tile + __float_as_int(place[c0 + c]), v[c][0], v[c][1]);
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            if (c0 + c < 15 || lane < HALO8 - 15 * 32)
                                sts128u(tile + __float_as_int(place[c0 + c]), normed(v[c][0], 0, g2[c].x, g2[c].y), normed(v[c][1], 1, g2[c].x, g2[c].y));
                    }
#pragma unroll
                    for (int n = 0; n < 4; n += 2) {
                        float gb[16];  // of two planes
                        u64 v[2][4][2];
                        tmem_ld8(tm + COL_GAMMA + 4 * n, gb);
                        tmem_ld8(tm + COL_BETA + 4 * n, gb + 8);
#pragma unroll
                        for (int o = 0; o < 8; ++o) lds128u(mine + (unsigned)((n + (o >> 2)) * G::PLANE + (o & 3)) * 16u, v[o >> 2][o & 3][0], v[o >> 2][o & 3][1]);
                        tmem_wait_ld16(gb);
#pragma unroll
                        for (int o = 0; o < 8; ++o) {
                            const u64 a = normed(v[o >> 2][o & 3][0], 0, gb[o], gb[8 + o]), b = normed(v[o >> 2][o & 3][1], 1, gb[o], gb[8 + o]);
                            sts128u(mine + (unsigned)((n + (o >> 2)) * G::PLANE + (o & 3)) * 16u, a, b);
                            own[n + (o >> 2)][o & 3][0] = a, own[n + (o >> 2)][o & 3][1] = b;
                        }
                    }
                } else {
                    wait_tile(i);
                    // step c: cell 4 c + r of the lane's small tile; the second tile of a pair is walked three cells ahead,
                    // which puts a quarter-warp on eight banks
                    constexpr int STEPS = 54, BATCH = 18;
                    const int slot = lane >> 2, l0 = (lane & 3) + 3 * (slot & 1);
                    const unsigned sub = tile + (unsigned)(slot * G::TILE) * 16u;
                    const float2 *const table = p.gbt + (size_t)blk * QuadGeo<4>::CELLS + ((slot >> 2) * 4 + (slot & 1) * 2 + ((slot >> 1) & 1)) * 216;
                    auto cell = [&](int c) { return l0 + 4 * c >= 216 ? l0 + 4 * c - 216 : l0 + 4 * c; };
#pragma unroll 1
                    for (int c0 = 0; c0 < STEPS; c0 += BATCH) {
                        u64 v[BATCH][2];
                        float2 g2[BATCH];
#pragma unroll
                        for (int c = 0; c < BATCH; ++c) {
                            const int l = cell(c0 + c);
                            g2[c] = table[l];
                            lds128u(sub + (unsigned)l * 16u, v[c][0], v[c][1]);
                        }
#pragma unroll
                        for (int c = 0; c < BATCH; ++c)
                            sts128u(sub + (unsigned)cell(c0 + c) * 16u, normed(v[c][0], 0, g2[c].x, g2[c].y), normed(v[c][1], 1, g2[c].x, g2[c].y));
                    }
                }
                __syncwarp();
            } else {
                wait_tile(i);
            }
            if (!(FUSE_IN && SUB == 8))
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int o = 0; o < 4; ++o) lds128u(mine + (unsigned)(n * G::PLANE + o) * 16u, own[n][o][0], own[n][o][1]);

            const size_t at = ((size_t)q * P + g0) * 4;  // the lane's cells in an IL4 tensor
            for (int t = 0; t < p.inner; ++t) {
                u64 acc[4][4][2], hold[2] = {0, 0};
                float *const sh = SAVE ? p.save_h + (size_t)t * p.Q * P * 4 + at : nullptr;
                tap_stencil<SUB>(win, tm, acc, own, [&](int n, int o, float scale) {
                    if (SAVE) {  // two neighbours at a time
                        if (o & 1) stg256(sh + n * zstr + 8 * (o >> 1), hold[0], hold[1], acc[n][o][0], acc[n][o][1]);
                        else hold[0] = acc[n][o][0], hold[1] = acc[n][o][1];
                    }
                    own[n][o][0] = act_residual2<ACT>(acc[n][o][0], scale, own[n][o][0]);
                    own[n][o][1] = act_residual2<ACT>(acc[n][o][1], scale, own[n][o][1]);
                });
                __syncwarp();  // every lane has read its window
                if (t + 1 < p.inner) {
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int o = 0; o < 4; ++o) sts128u(mine + (unsigned)(n * G::PLANE + o) * 16u, own[n][o][0], own[n][o][1]);
                    __syncwarp();
                } else {
                    // the tile is dead: fetch the next one
                    if (i + NBUF < cnt && (SUB == 4 || lane == 0)) issue(i + NBUF);
                    __syncwarp();
                    next = claim(i);
                    if (p.y)
#pragma unroll
                        for (int n = 0; n < 4; ++n)
#pragma unroll
                            for (int o = 0; o < 4; o += 2)
                                stg256(p.y + at + n * zstr + 4 * o, own[n][o][0], own[n][o][1], own[n][o + 1][0], own[n][o + 1][1]);
                    if (p.out_partials) {
                        const double r = tap_region_sums(own, lane);
                        if ((lane & 20) == 0)
                            reinterpret_cast<double *>(p.out_partials + (size_t)(4 * q + (lane & 2) + (lane >> 3)) * p.nparts + blk)[lane & 1] = r;
                        __syncwarp();
                    }
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

template <int SUB, int ACT, bool FUSE_IN, bool SAVE>
int launch_one(const CUtensorMap &map, const TapParams &p, unsigned ctas, cudaStream_t st)
{
    using G = TapGeo<SUB>;
    auto kern = step_fwd_taps<SUB, ACT, FUSE_IN, SAVE>;
    constexpr int smem = QUARTERS * G::NBUF * G::BUF_BYTES + (SUB == 8 && FUSE_IN ? QUARTERS * HALO8 * 8 : 0);
    static_assert(smem <= 232448 - 1024 - 256, "shared memory budget of one SM");
    static unsigned long long attr_set = 0;
    if (first_use_on_device(&attr_set)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            record_cuda_error(e, "cudaFuncSetAttribute(step_fwd_taps)");
            return GN_ERR_CUDA;
        }
    }
    launch_after(kern, ctas, 128 * G::TEAM, smem, st, map, p);
    return check_launch("step_fwd_taps");
}

template <int SUB, int ACT>
int launch_act(const CUtensorMap &map, const TapParams &p, unsigned ctas, cudaStream_t st)
{
    if (p.save_h) return p.in_stats ? launch_one<SUB, ACT, true, true>(map, p, ctas, st) : launch_one<SUB, ACT, false, true>(map, p, ctas, st);
    return p.in_stats ? launch_one<SUB, ACT, true, false>(map, p, ctas, st) : launch_one<SUB, ACT, false, false>(map, p, ctas, st);
}

template <int SUB>
int launch_sub(const CUtensorMap &map, const TapParams &p, unsigned ctas, int act, cudaStream_t st)
{
    switch (act) {
    case GN_ACT_RELU: return launch_act<SUB, GN_ACT_RELU>(map, p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_act<SUB, GN_ACT_LEAKY_RELU>(map, p, ctas, st);
    case GN_ACT_SILU: return launch_act<SUB, GN_ACT_SILU>(map, p, ctas, st);
    default: return launch_act<SUB, GN_ACT_TANH>(map, p, ctas, st);
    }
}

}  // namespace

int launch_step_fwd_taps(const QuadStep &a, int act, cudaStream_t st)
{
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (a.block == 8) {
        const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, 8, TapGeo<8>::ROW);
        if (rc != GN_OK) return rc;
    }
    TapParams p{};
    p.packed = a.packed; p.params_old = a.params_old;
    p.gbt = a.gbt; p.in_stats = a.in_stats; p.in = a.in_il4;
    p.out_partials = a.out_partials; p.nparts = a.nparts;
    p.y = a.out_il4; p.save_h = a.save_h;
    p.error_flag = a.error_flag ? a.error_flag : device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = (long long)(a.M / 8) * (a.N / 8) * (a.K / 8) * a.Q;
    long long ctas = (p.nitems + QUARTERS - 1) / QUARTERS;
    if (ctas > sm_count()) ctas = sm_count();
    p.unit = quad_split_unit(p.nitems, ctas, p.Q);
    return a.block == 8 ? launch_sub<8>(map, p, (unsigned)ctas, act, st) : launch_sub<4>(map, p, (unsigned)ctas, act, st);
}

}  // namespace gn
