// "Quad" kernels: float forward of the block-local update (block 8 and 4, per-block normalisation off) with the
// weights in tensor memory and four samples per lane.
//
// The register-patch kernel (step_fast.cu) keeps 108 weights per thread in registers and pays 2.25 FMAs per
// shared-memory wavefront; the large-batch kernel (step_pair64.cu) fetches the weights from shared memory and pays
// about 2.9. Here the weights do not touch the shared-memory data pipe at all: a warp handles a whole 8^3 region for
// four samples, a lane owns a 2 x 2 x 4 (z, y, x) patch of neurons, and its 16 x 27 weights, biases and scales are
// 464 of the 512 words that tensor memory has per lane. They are read back in steps of 24 words, a stencil step
// ahead, and each is used for the lane's four samples. A window is 4 x 4 x 6 cells for 16 neurons: 4.5 FMAs per
// wavefront, the most that any split of an 8^3 region over 32 lanes gives.
//
//   * Layout ("IL4"): activations between the steps are interleaved by four samples, [B/4][M][N][K][4], so that a
//     cell of a quad is one 128-bit access and FMAs are packed (fma.rn.f32x2) over sample pairs; a weight is the
//     scalar operand of both.
//   * A warp is on its own: its tile (10 x 10 x 10 cells, rows of 11) is read and written by no other warp, so the
//     inner iterations need no barrier beyond __syncwarp, and new values go back into the tile in place.
//   * Bank conflicts: none, see QuadLane in quad_geo.cuh.
//   * Two warps (w, w + 4) share a quarter of tensor memory and therefore a region: they take its quads in turn. Each
//     such team has its own contiguous range of (region, quad) items, and meets (named barrier) only to exchange the
//     weights at a new region. The two warps sit on the same scheduler, so one's activation functions (MUFU) overlap
//     the other's FMAs.
//   * Tiles arrive by bulk tensor copy (zero fill outside the grid) into three buffers per team (block 4: two), so a
//     tile is under way while the two before it are worked on.
//
// Fusion as in step_fast.cu: FUSE_IN normalises the landed tile in place with the whole-grid statistics of the
// previous step and a per-region (gamma, beta) table; every launch can reduce (sum, sum of squares) per sample and
// region of what it writes. Reference semantics: gridnet/backend_torch.py:61-142; the kernel it stands in for is
// gridnet_cuda_forward_kernel, src/gridnet_cuda_kernels.cu:101-200.
#include <string.h>

#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "quad_geo.cuh"
#include "tmem.cuh"

namespace gn {

struct QuadParams {
    const float *packed;     // [regions][quad::PACK_F]
    const float2 *gbt;       // FUSE_IN: (gamma, beta) per tile cell, [regions][CELLS], zero outside the grid
    const float2 *in_stats;  // FUSE_IN: [4 Q] (mean, rstd)
    double2 *out_partials;   // [4 Q][nparts]: slot `region` of every row is written; nullptr: not wanted
    int nparts;
    float *y;                // IL4; nullptr: not wanted (replay)
    float *save_h;           // SAVE: [inner][Q][P][4]
    int *error_flag;
    int M, N, K, Q, inner;
    long long nitems;        // regions * Q
};

// SAVE: keep every iteration's pre-activations for the backward pass (which gets the activations in between from them and
// the step's input).
template <int SUB, int ACT, bool FUSE_IN, bool SAVE>
__global__ void __launch_bounds__(128 * QuadGeo<SUB>::TEAM, 1)
    step_fwd_quad(const __grid_constant__ CUtensorMap in_map, const QuadParams p)
{
    using namespace quad;
    using G = QuadGeo<SUB>;
    constexpr int TEAM = G::TEAM, NBUF = G::NBUF;
    constexpr bool GB_SMEM = FUSE_IN && SUB == 8;  // the (gamma, beta) table of the team's region is in shared memory
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[QUARTERS * G::NBUF];
    __shared__ int issued[QUARTERS * G::NBUF];  // which item's copy into this buffer has been started last
    __shared__ unsigned tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quarter = warp & 3, role = warp >> 2;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    if (tid == 0) {
        for (int i = 0; i < QUARTERS * G::NBUF; ++i) {
            mbar_init(smem_u32(&bars[i]), 1);
            issued[i] = -1;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    float2 *const gbs = reinterpret_cast<float2 *>(smem + QUARTERS * G::NBUF * G::BUF_BYTES) + quarter * G::CELLS;
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const unsigned tm = tmem_slot + ((unsigned)(quarter * 32) << 16);

    const QuadLane<SUB> L(lane);
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const size_t P = (size_t)p.M * p.N * p.K;
    const long long worker = (long long)blockIdx.x * QUARTERS + quarter, nworkers = (long long)gridDim.x * QUARTERS;
    const long long n0 = p.nitems * worker / nworkers;
    const int cnt = (int)(p.nitems * (worker + 1) / nworkers - n0);
    const unsigned bar0 = smem_u32(&bars[quarter * NBUF]), issued0 = smem_u32(&issued[quarter * NBUF]);
    const unsigned tiles = smem_u32(smem) + quarter * (NBUF * G::BUF_BYTES);
    const long long wzs = (long long)p.N * p.K, wys = (long long)L.ysgn * p.K;
    bool failed = false;

    // one lane: fetch the tile of the team's item i into its buffer
    auto issue = [&](int i) {
        const long long n = n0 + i;
        const int blk = (int)(n / p.Q), q = (int)(n - (long long)blk * p.Q);
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
    if (role == 0 && lane == 0)
        for (int i = 0; i < NBUF && i < cnt; ++i) issue(i);
    __syncwarp();

    int blk = (int)(n0 / p.Q), q0 = (int)(n0 - (long long)blk * p.Q);
    for (int i0 = 0; i0 < cnt;) {
        const int here = min(cnt - i0, p.Q - q0);  // items of this region
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const size_t g0 = ((size_t)(bz * 8 + L.z0) * p.N + (by * 8 + L.y0)) * p.K + bx * 8 + 4 * L.h;  // own patch, native layout
        if (i0 > 0) {
            tmem_fence_before();
            team_sync<TEAM>(quarter);  // the other warps no longer read the old region's weights
            tmem_fence_after();
        }
        if (GB_SMEM) {
            const unsigned char *src = reinterpret_cast<const unsigned char *>(p.gbt + (size_t)blk * G::CELLS);
            const unsigned dst = smem_u32(gbs);
            for (int c = role * 32 + lane; c < G::CELLS / 2; c += 32 * TEAM) cp_async16(dst + c * 16, src + c * 16);
            __syncwarp();  // tensor memory instructions want the whole warp together
        }
        quad_load_params(p.packed + (size_t)blk * PACK_F, role, lane, tm);
        tmem_wait_st();
        if (GB_SMEM) cp_async_wait_all();
        tmem_fence_before();
        team_sync<TEAM>(quarter);
        tmem_fence_after();
        if (i0 + here < cnt) {  // the next region's parameters on their way to L2
            const unsigned char *nx = reinterpret_cast<const unsigned char *>(p.packed + (size_t)(blk + 1) * PACK_F);
            for (int c = role * 32 + lane; c < PACK_F * 4 / 128; c += 32 * TEAM) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c * 128));
            __syncwarp();
        }

        // item i goes to warp i mod TEAM
        for (int k = (role + TEAM - i0 % TEAM) % TEAM; k < here; k += TEAM) {
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
                    nb[0] = pack2(-mr[0].x * mr[0].y, -mr[1].x * mr[1].y);
                    nb[1] = pack2(-mr[2].x * mr[2].y, -mr[3].x * mr[3].y);
                }
                wait_tile(i);
                const float2 *gp = GB_SMEM ? gbs + lane : p.gbt + (size_t)blk * G::CELLS + lane;
                constexpr int STEPS = (G::CELLS + 31) / 32;
                constexpr int BATCH = SUB == 8 ? 16 : 18;  // loads of a batch are in flight together
#pragma unroll 1
                for (int c0 = 0; c0 < STEPS; c0 += BATCH) {
                    const unsigned a = tile + (unsigned)(c0 * 32 + lane) * 16u;
                    u64 v[BATCH][2];
                    float2 g2[BATCH];
#pragma unroll
                    for (int c = 0; c < BATCH; ++c)
                        if ((c0 + c) * 32 + lane < G::CELLS) {
                            g2[c] = gp[(c0 + c) * 32];
                            lds128u(a + c * 512, v[c][0], v[c][1]);
                        }
#pragma unroll
                    for (int c = 0; c < BATCH; ++c)
                        if ((c0 + c) * 32 + lane < G::CELLS) {
                            const u64 gg = pack2(g2[c].x, g2[c].x), bb = pack2(g2[c].y, g2[c].y);
                            sts128u(a + c * 512, ffma2r(ffma2r(v[c][0], na[0], nb[0]), gg, bb), ffma2r(ffma2r(v[c][1], na[1], nb[1]), gg, bb));
                        }
                }
                __syncwarp();
            } else {
                wait_tile(i);
            }

            const unsigned win = tile + L.cell0 * 16u;  // window cell (0, 0, 0) of this lane
            unsigned rows[4];
#pragma unroll
            for (int ry = 0; ry < 4; ++ry) rows[ry] = win + (unsigned)(ry * L.ysgn * G::ROW * 16);
            const size_t own = ((size_t)q * P + g0) * 4;  // the lane's cells in an IL4 tensor
            const long long zstr = wzs * 4, ystr = wys * 4;
            for (int t = 0; t < p.inner; ++t) {
                const bool last = t + 1 == p.inner;
                u64 acc[4][4][2], hold[2] = {0, 0};
                float *const sh = SAVE ? p.save_h + (size_t)t * p.Q * P * 4 + own : nullptr;
                quad_stencil<G::PLANE, true>(rows, L.xsgn * 16, tm, acc, [&](int n, int o, float scale, u64 c0, u64 c1) {
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
                    for (int o = 0; o < 4; ++o) {
                        const unsigned a = win + (unsigned)((1 + o) * L.xsgn * 16) + (unsigned)(L.ysgn * G::ROW * 16) + G::PLANE * 16u;
#pragma unroll
                        for (int n = 0; n < 4; ++n)
                            sts128u(a + (unsigned)((n & 1) * L.ysgn * G::ROW * 16) + (n >> 1) * G::PLANE * 16u, acc[n][o][0], acc[n][o][1]);
                    }
                    __syncwarp();
                } else {
                    if (lane == 0 && i + NBUF < cnt) issue(i + NBUF);  // the tile is dead: fetch the next one
                    __syncwarp();
                    if (p.y) quad_store(p.y + own, zstr, ystr, L.h, acc);
                    if (p.out_partials) {
                        u64 s2[2] = {0, 0}, q2[2] = {0, 0};
#pragma unroll
                        for (int n = 0; n < 4; ++n)
#pragma unroll
                            for (int o = 0; o < 4; ++o)
#pragma unroll
                                for (int k2 = 0; k2 < 2; ++k2) {
                                    s2[k2] = fadd2(s2[k2], acc[n][o][k2]);
                                    ffma2(q2[k2], acc[n][o][k2], acc[n][o][k2]);
                                }
                        float v[8];
                        unpack2(s2[0], v[0], v[1]);
                        unpack2(s2[1], v[2], v[3]);
                        unpack2(q2[0], v[4], v[5]);
                        unpack2(q2[1], v[6], v[7]);
                        const float r = quad_reduce8(v, lane);
                        // lane 4 j holds value j: sums of samples 0..3, then sums of squares
                        if ((lane & 3) == 0)
                            reinterpret_cast<double *>(p.out_partials + (size_t)(4 * q + ((lane >> 2) & 3)) * p.nparts + blk)[lane >> 4] = (double)r;
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

// ---- layout conversion at the ends of a loop --------------------------------------------------------------
// [B, P] -> [Q][P][4]; samples beyond B are zero. One cell per thread and step: four coalesced 4-byte reads, one
// coalesced 16-byte write.
__global__ void __launch_bounds__(256) to_il4_k(const float *__restrict__ x, float4 *__restrict__ il, int B, size_t P)
{
    const size_t c = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= P) return;
    const int q = blockIdx.y;
    float v[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) v[s] = 4 * q + s < B ? x[(size_t)(4 * q + s) * P + c] : 0.0f;
    il[(size_t)q * P + c] = make_float4(v[0], v[1], v[2], v[3]);
}

// IL4 -> [B, P], normalised on the way when statistics are given
__global__ void __launch_bounds__(256) from_il4_k(const float4 *__restrict__ il, const float2 *__restrict__ stats,
                                                  const float *__restrict__ gamma, const float *__restrict__ beta,
                                                  float *__restrict__ y, int B, size_t P)
{
    const size_t c = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= P) return;
    const int q = blockIdx.y;
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

// Parameters in the order of the stencil: vector v of a region is, for every lane, the four x-neighbouring weights of
// one (neuron row, tap), v = 0 .. 107 in the order of the uses in quad_stencil (three x-taps each), then the four rows
// of b, then of s. TRANS: the weights of the backward sum, in which a cell collects from the neurons of its own block
// that read it: the neuron at tap t sees the cell through its tap 26 - t; zero across the block's border. One CTA per
// region; reads are 16-byte pieces, writes whole lines.
template <int SUB, bool TRANS>
__global__ void __launch_bounds__(256) quad_pack_k(const float *__restrict__ w, const float *__restrict__ b, const float *__restrict__ s,
                                                   float *__restrict__ packed, int M, int N, int K)
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
    const int nbx = K >> 3, nby = N >> 3, blk = blockIdx.x;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)M * N * K;
    const size_t g0 = ((size_t)(bz * 8 + L.z0) * N + (by * 8 + L.y0)) * K + bx * 8 + 4 * L.h;
    const long long zs = (long long)N * K, ys = (long long)L.ysgn * K;
    float4 *out = reinterpret_cast<float4 *>(packed + (size_t)blk * quad::PACK_F) + lane;
#pragma unroll 4
    for (int v = threadIdx.x >> 5; v < quad::VECS; v += 8) {
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
                const float *src = w + (size_t)t * P + own;
                if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) r = *reinterpret_cast<const float4 *>(src);
                else r = make_float4(src[0], src[1], src[2], src[3]);
            } else {
                const int lz = L.z0 + (n >> 1) + ta - 1, ly = L.y0 + L.ysgn * (n & 1) + tb - 1;  // source row in the region
                const int mask = ~(SUB - 1);
                const bool row = lz >= 0 && lz < 8 && ly >= 0 && ly < 8 && ((lz ^ (L.z0 + (n >> 1))) & mask & 7) == 0 &&
                                 ((ly ^ (L.y0 + L.ysgn * (n & 1))) & mask & 7) == 0;
                const float *src = w + (size_t)(26 - t) * P + own + (ta - 1) * zs + (long long)(tb - 1) * K + (tc - 1);
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

// (gamma, beta) of every tile cell of every region, in the order of the tile buffer
template <int SUB>
__global__ void __launch_bounds__(256) quad_table_k(const float *__restrict__ gamma, const float *__restrict__ beta,
                                                    float2 *__restrict__ gbt, int M, int N, int K)
{
    using G = QuadGeo<SUB>;
    const int nbx = K >> 3, nby = N >> 3, blk = blockIdx.x;
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

// ---- host side -----------------------------------------------------------------------------------------------
int quad_tile_cells(int block) { return block == 8 ? QuadGeo<8>::CELLS : QuadGeo<4>::CELLS; }

bool quad_applicable(int M, int N, int K, int block, int inner)
{
    if ((block != 8 && block != 4) || inner < 1 || M % 8 || N % 8 || K % 8) return false;
    if ((long long)M * N * K >= (1LL << 31) / 4) return false;
    return encode_tiled_fn() != nullptr;
}

// tensor map over an IL4 buffer, box = one tile (10^3 or 6^3 cells)
int quad_make_map(CUtensorMap *map, const float *il, int M, int N, int K, int Q, int block)
{
    MapKey key{il, block == 8 ? 40 : 24, 0, {M, N, K, Q}};
    (void)cudaGetDevice(&key.dev);
    if (tensor_map_cache_get(key, map)) return GN_OK;
    const cuuint64_t dims[4] = {(cuuint64_t)K * 4, (cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)Q};
    const cuuint64_t strides[3] = {(cuuint64_t)K * 16, (cuuint64_t)N * K * 16, (cuuint64_t)M * N * K * 16};
    const cuuint32_t side = block == 8 ? 10 : 6;
    const cuuint32_t box[4] = {4 * side, side, side, 1};
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

int launch_to_il4(const float *x, float *il, int B, long long P, cudaStream_t st)
{
    dim3 grid((unsigned)((P + 255) / 256), (unsigned)((B + 3) / 4));
    to_il4_k<<<grid, 256, 0, st>>>(x, reinterpret_cast<float4 *>(il), B, (size_t)P);
    return check_launch("to_il4");
}

int launch_from_il4(const float *il, const float2 *stats, const float *gamma, const float *beta, float *y, int B, long long P,
                    cudaStream_t st)
{
    dim3 grid((unsigned)((P + 255) / 256), (unsigned)((B + 3) / 4));
    from_il4_k<<<grid, 256, 0, st>>>(reinterpret_cast<const float4 *>(il), stats, gamma, beta, y, B, (size_t)P);
    return check_launch("from_il4");
}

size_t quad_packed_floats(int M, int N, int K) { return (size_t)(M / 8) * (N / 8) * (K / 8) * quad::PACK_F; }

int launch_quad_pack(const float *w, const float *b, const float *s, float *packed, int M, int N, int K, int block, bool transposed,
                     cudaStream_t st)
{
    const unsigned regions = (unsigned)((M / 8) * (N / 8) * (K / 8));
    if (block == 8 && transposed) quad_pack_k<8, true><<<regions, 256, 0, st>>>(w, b, s, packed, M, N, K);
    else if (block == 8) quad_pack_k<8, false><<<regions, 256, 0, st>>>(w, b, s, packed, M, N, K);
    else if (transposed) quad_pack_k<4, true><<<regions, 256, 0, st>>>(w, b, s, packed, M, N, K);
    else quad_pack_k<4, false><<<regions, 256, 0, st>>>(w, b, s, packed, M, N, K);
    return check_launch("quad_pack");
}

int launch_quad_table(const float *gamma, const float *beta, float2 *gbt, int M, int N, int K, int block, cudaStream_t st)
{
    const unsigned regions = (unsigned)((M / 8) * (N / 8) * (K / 8));
    if (block == 8) quad_table_k<8><<<regions, 256, 0, st>>>(gamma, beta, gbt, M, N, K);
    else quad_table_k<4><<<regions, 256, 0, st>>>(gamma, beta, gbt, M, N, K);
    return check_launch("quad_table");
}

template <int SUB, int ACT, bool FUSE_IN, bool SAVE>
static int launch_quad_one(const CUtensorMap &map, const QuadParams &p, unsigned ctas, cudaStream_t st)
{
    using G = QuadGeo<SUB>;
    auto kern = step_fwd_quad<SUB, ACT, FUSE_IN, SAVE>;
    // tiles; block 8 with normalise-on-load also a (gamma, beta) table per team
    constexpr int smem = quad::QUARTERS * G::NBUF * G::BUF_BYTES + (SUB == 8 && FUSE_IN ? quad::QUARTERS * G::CELLS * 8 : 0);
    static_assert(smem <= 232448 - 1024 - 256, "shared memory budget of one SM");
    static unsigned long long attr_set = 0;
    if (first_use_on_device(&attr_set)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            record_cuda_error(e, "cudaFuncSetAttribute(step_fwd_quad)");
            return GN_ERR_CUDA;
        }
    }
    kern<<<ctas, 128 * G::TEAM, smem, st>>>(map, p);
    return check_launch("step_fwd_quad");
}

template <int SUB, int ACT>
static int launch_quad_act(const CUtensorMap &map, const QuadParams &p, unsigned ctas, cudaStream_t st)
{
    if (p.save_h) return p.in_stats ? launch_quad_one<SUB, ACT, true, true>(map, p, ctas, st) : launch_quad_one<SUB, ACT, false, true>(map, p, ctas, st);
    return p.in_stats ? launch_quad_one<SUB, ACT, true, false>(map, p, ctas, st) : launch_quad_one<SUB, ACT, false, false>(map, p, ctas, st);
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
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    const int rc = quad_make_map(&map, a.in_il4, a.M, a.N, a.K, a.Q, a.block);
    if (rc != GN_OK) return rc;
    QuadParams p{};
    p.packed = a.packed;
    p.gbt = a.gbt; p.in_stats = a.in_stats;
    p.out_partials = a.out_partials; p.nparts = a.nparts;
    p.y = a.out_il4; p.save_h = a.save_h;
    p.error_flag = a.error_flag ? a.error_flag : device_status_ptr();
    p.M = a.M; p.N = a.N; p.K = a.K; p.Q = a.Q; p.inner = a.inner;
    p.nitems = (long long)(a.M / 8) * (a.N / 8) * (a.K / 8) * a.Q;
    long long ctas = (p.nitems + quad::QUARTERS - 1) / quad::QUARTERS;
    if (ctas > sm_count()) ctas = sm_count();
    return a.block == 8 ? launch_quad_sub<8>(map, p, (unsigned)ctas, act, st) : launch_quad_sub<4>(map, p, (unsigned)ctas, act, st);
}

}  // namespace gn
