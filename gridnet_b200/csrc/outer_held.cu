// The whole fused model loop as one persistent kernel, as in outer_small.cu, for grids that have more blocks than that kernel
// can hold weights for in registers: a single sample through 64^3 (512 blocks, 4 x 12 iterations) is 24 launches of 5 to
// 14 us step by step, and every step loads all 30 MB of parameters again.
//
// The weights of 592 blocks fit into the tensor memory of the chip: a CTA per SM holds up to four blocks of one sample (or the
// same samples), each worked on by four warps, one per quarter of tensor memory, where a thread has its 4 x 27 weights, biases,
// scales and norm parameters in 124 of the 512 columns, in the order of their use. The rest is as in outer_small.cu: a thread
// owns a 1 x 2 x 2 patch and keeps it in registers between steps, halo cells and sums go from CTA to CTA in words that
// carry their step, and a further warp per sample publishes the CTA's sums and watches for the others'. A CTA's sums are added up
// before they are published, so that 128 lines are watched at 64^3 instead of 512.
//
// The launch is cooperative and there is one CTA per SM (shared memory is asked for that no second kernel with tensor memory can
// have beside it), so all CTAs are resident, get their tensor memory, and the waits end; should one run out all the same,
// the kernel sets the error flag and the device's status word and goes on.
#include <atomic>

#include "common.cuh"
#include "kernels.h"
#include "outer_words.cuh"
#include "patch_geo.cuh"
#include "tmem.cuh"

namespace gn {

namespace held8 {
constexpr int SLOTS_PER_CTA = 4, COMPUTE = 128, WORKERS = SLOTS_PER_CTA * COMPUTE;
constexpr int MAX_SPC = 2;                     // samples per CTA at most
constexpr int THREADS = WORKERS + 32 * MAX_SPC;
constexpr int WATCHED = WORKERS + 32;          // threads that compute, with the warp that watches a sample
constexpr int HALO = 488, SLOTS = 4;           // halo cells of a tile, per thread
constexpr unsigned kSpinLimit = 1u << 18;      // polls, about a microsecond each
// Inner iterations at most. CTAs wait for each other once a step, those with one block for those with four; an iteration takes up to 0.75 us
// per sample, so nobody waits longer than 6 ms of the 260 that a wait has (at 1.5 million, 8 x 8 x 72, they ran out).
constexpr int MAX_INNER = 4096;
constexpr int B_DONE = 1, B_STATS = 1 + MAX_SPC, B_COMPUTE = 1 + 2 * MAX_SPC;  // named barriers; the last kind one per block
// columns of tensor memory of a block: 9 chunks of 12 weights, then 4 biases, scales, norm weights and norm biases
constexpr int COLS = 128, COL_REST = 108;
constexpr int TS = PatchGeo<8>::TS;
constexpr int TILES = SLOTS_PER_CTA * MAX_SPC * 2 * TS * 4, SMEM = TILES + SLOTS_PER_CTA * HALO * 8;
constexpr int SMEM_ALONE = 120 * 1024;  // more than half of what an SM has
static_assert(SMEM <= SMEM_ALONE, "");
}  // namespace held8

struct OuterHeldParams {
    const float *w, *b, *s, *gamma, *beta, *x;
    float *y;
    unsigned long long *cells;  // [2][B][P] (raw step output, step); zeroed
    unsigned long long *sums;   // [2][B][ctas per sample], a line each: (sum, sum of squares) as doubles, the low 8 bits the step; zeroed
    int *error_flag, *status;   // of the call, and device_status_ptr(): callers seldom hold the workspace that the first one is in
    int nblocks, group;         // group: CTAs that work on the same samples
    int B, M, N, K, inner, outer, spc;
    float eps;
};

template <int ACT>
__global__ void __launch_bounds__(held8::THREADS, 1) outer_held_k(const OuterHeldParams p)
{
    using namespace held8;
    using Geo = PatchGeo<8>;
    constexpr int RS = Geo::RS, PS = Geo::PS;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ float2 mstats[MAX_SPC];
    __shared__ float2 wsum[MAX_SPC][WORKERS / 32];  // per-warp (sum, sum of squares) of the CTA's outputs of this step
    __shared__ unsigned tmem_slot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 0) tmem_alloc_all(&tmem_slot);
    for (int i = tid; i < MAX_SPC * (WORKERS / 32); i += THREADS) wsum[i / (WORKERS / 32)][i % (WORKERS / 32)] = make_float2(0.0f, 0.0f);
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();

    const int member = blockIdx.x % p.group, chunk = blockIdx.x / p.group;
    const int nbx = p.K >> 3, nby = p.N >> 3, K = p.K;
    const size_t P = (size_t)p.M * p.N * K;
    const int s0 = chunk * p.spc, ns = min(p.B - s0, p.spc);
    const int slots = min(SLOTS_PER_CTA, p.nblocks - member * SLOTS_PER_CTA), watched = slots * COMPUTE + 32;
    bool gave_up = false;  // one wait ran out: the results are lost, do not wait again

    if (tid >= WORKERS) {  // ---- the watching warps, one per sample
        const int q = (tid - WORKERS) >> 5;
        if (q < ns) {
            const double per_cell = 1.0 / (double)P;
            for (int o = 1; o <= p.outer; ++o) {
                const unsigned long long tag = (unsigned)o & 0xffu;
                unsigned long long *const sums = p.sums + ((size_t)(o & 1) * p.B + s0 + q) * p.group * kOuterSmallLine;
                bar_sync(B_DONE + q, watched);
                {
                    // in a fixed order; warps without a block have left zeros
                    double sm = lane < WORKERS / 32 ? (double)wsum[q][lane].x : 0.0, sq = lane < WORKERS / 32 ? (double)wsum[q][lane].y : 0.0;
                    sm = warp_sum(sm);
                    sq = warp_sum(sq);
                    if (lane == 0)
                        st_words(sums + kOuterSmallLine * member, ((unsigned long long)__double_as_longlong(sm) & ~0xffull) | tag,
                                 ((unsigned long long)__double_as_longlong(sq) & ~0xffull) | tag);
                }
                __syncwarp();
                const float2 result = watch_sums(sums, p.group, kOuterSmallLine, tag, per_cell, p.eps, lane, kSpinLimit, gave_up);
                if (lane == 0) mstats[q] = result;
                __syncwarp();
                bar_arrive(B_STATS + q, watched);
            }
        }
    } else if (warp >> 2 < slots) {  // ---- a block
        const int slot = warp >> 2, lt = tid & (COMPUTE - 1), blk = member * SLOTS_PER_CTA + slot;
        const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
        const int xp = lt & 3, yp = (lt >> 2) & 3, z = lt >> 4;
        const size_t g00 = ((size_t)(bz * 8 + z) * p.N + (by * 8 + 2 * yp)) * K + (bx * 8 + 2 * xp);
        const long long origin = ((long long)(bz * 8 - 1) * p.N + (by * 8 - 1)) * K + (bx * 8 - 1);
        const unsigned tm = tmem_slot + ((unsigned)((warp & 3) * 32) << 16) + slot * COLS;
        float *const tiles = reinterpret_cast<float *>(smem) + slot * (MAX_SPC * 2 * TS);  // [sample of the CTA][ping-pong]
        float2 *const halo_gb = reinterpret_cast<float2 *>(smem + TILES) + slot * HALO;
        // ---- parameters -> tensor memory. A chunk of 12 weights: two uses (window row r, patch row j), three x-taps, two neurons
#pragma unroll
        for (int c9 = 0; c9 < 9; ++c9) {
            constexpr int R[6] = {0, 1, 1, 2, 2, 3}, J[6] = {0, 0, 1, 0, 1, 1};
            float v[12];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int k = c9 % 3 * 2 + u, j = J[k], tap = c9 / 3 * 9 + (R[k] - j) * 3 + c;
                    const float2 a = *reinterpret_cast<const float2 *>(p.w + (size_t)tap * P + g00 + (size_t)j * K);
                    v[u * 6 + c * 2] = a.x;
                    v[u * 6 + c * 2 + 1] = a.y;
                }
            tmem_st8(tm + c9 * 12, v);
            tmem_st4(tm + c9 * 12 + 8, v + 8);
        }
        {
            const float *const src[4] = {p.b, p.s, p.gamma, p.beta};
            float v[16];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 a = *reinterpret_cast<const float2 *>(src[k] + g00 + (size_t)j * K);
                    v[k * 4 + j * 2] = a.x;
                    v[k * 4 + j * 2 + 1] = a.y;
                }
            tmem_st16(tm + COL_REST, v);
        }
        // halo cells this thread fetches for every sample: tile offset (or -1), offset from the tile's origin (or -1 outside).
        // z faces 2 x 10 x 10, y faces 2 x 8 x 10, x faces 2 x 8 x 8
        int soff[SLOTS], rel[SLOTS];
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            const int i = lt + j * COMPUTE;
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
            soff[j] = rel[j] = -1;
            if (i < HALO) {
                soff[j] = cz * PS + cy * RS + cx;
                const int gz = bz * 8 + cz - 1, gy = by * 8 + cy - 1, gx = bx * 8 + cx - 1;
                float2 gb = make_float2(0.0f, 0.0f);
                if (gz >= 0 && gz < p.M && gy >= 0 && gy < p.N && gx >= 0 && gx < K) {
                    rel[j] = (cz * p.N + cy) * K + cx;
                    gb = make_float2(p.gamma[origin + rel[j]], p.beta[origin + rel[j]]);
                }
                halo_gb[i] = gb;  // read by this thread only
            }
        }
        float own[MAX_SPC][2][2];  // the patch between outer steps: raw outputs
#pragma unroll
        for (int q = 0; q < MAX_SPC; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float *a = p.x + (size_t)(s0 + q) * P + g00 + (size_t)j * K;
                own[q][j][0] = q < ns ? a[0] : 0.0f;
                own[q][j][1] = q < ns ? a[1] : 0.0f;
            }
        const int toff = Geo::window_origin(xp, yp, z);
        const bool surface = z == 0 || z == 7 || yp == 0 || yp == 3 || xp == 0 || xp == 3;  // some cell of the patch is another block's halo
        unsigned long long seen[SLOTS];  // halo cells as last seen
        auto ask = [&](int q, int o) {   // for what the neighbours' step o left (the set of that step)
            const unsigned long long *cells = p.cells + ((size_t)(o & 1) * p.B + s0 + q) * P + origin;
#pragma unroll
            for (int j = 0; j < SLOTS; ++j) seen[j] = rel[j] >= 0 ? ld_word(cells + rel[j]) : (unsigned long long)o << 32;
        };
        __syncwarp();
        tmem_wait_st();
        for (int o = 0; o < p.outer; ++o) {
#pragma unroll
            for (int q = 0; q < MAX_SPC; ++q) {
                if (q >= ns) continue;
                float *const tl0 = tiles + q * (2 * TS);
                {
                    float v[SLOTS], gb[8];
                    if (o == 0) {
                        const float *xs = p.x + (size_t)(s0 + q) * P + origin;
#pragma unroll
                        for (int j = 0; j < SLOTS; ++j) v[j] = rel[j] >= 0 ? xs[rel[j]] : 0.0f;
                    } else {
                        if (ns == 1) ask(q, o);  // else asked for while the other sample was in work
                        for (unsigned spins = 0; !gave_up; ask(q, o)) {
                            bool there = true;
#pragma unroll
                            for (int j = 0; j < SLOTS; ++j) there &= (unsigned)(seen[j] >> 32) == (unsigned)o;
                            if (there) break;
                            gave_up = ++spins > kSpinLimit;
                        }
#pragma unroll
                        for (int j = 0; j < SLOTS; ++j) v[j] = __uint_as_float((unsigned)seen[j]);
                        __syncwarp();
                        bar_sync(B_STATS + q, watched);  // the sample's statistics of that step
                    }
                    __syncwarp();  // tensor memory instructions want the whole warp together
                    tmem_ld8(tm + COL_REST + 8, gb);
                    tmem_wait_ld8(gb);
                    const float2 mr = o > 0 ? mstats[q] : make_float2(0.0f, 1.0f);
                    float *to = tl0 + toff + PS + RS + 1;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            to[j * RS + k] = o > 0 ? fmaf((own[q][j][k] - mr.x) * mr.y, gb[2 * j + k], gb[4 + 2 * j + k]) : own[q][j][k];
#pragma unroll
                    for (int j = 0; j < SLOTS; ++j)
                        if (soff[j] >= 0) {
                            float u = v[j];
                            if (o > 0) {
                                const float2 g2 = halo_gb[lt + j * COMPUTE];
                                u = fmaf((u - mr.x) * mr.y, g2.x, g2.y);
                            }
                            tl0[soff[j]] = u;
                            tl0[TS + soff[j]] = u;
                        }
                }
                bar_sync(B_COMPUTE + slot, COMPUTE);
                if (ns > 1 && (q == 0 ? o > 0 : o + 1 < p.outer)) ask(q ^ 1, o + q);  // what comes next
                for (int it = 0; it < p.inner; ++it) {
                    const int cur = it & 1;
                    const float *tl = tl0 + cur * TS + toff;
                    float bs[8], wb[2][12], acc[2][2], old[2][2];
                    __syncwarp();
                    tmem_ld8(tm + COL_REST, bs);
                    tmem_ld8(tm, wb[0]);
                    tmem_ld4(tm + 8, wb[0] + 8);
                    tmem_wait_ld8(bs);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int k = 0; k < 2; ++k) acc[j][k] = bs[2 * j + k];
                    int use = 0;
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const float2 v01 = *reinterpret_cast<const float2 *>(tl + a * PS + r * RS);
                            const float2 v23 = *reinterpret_cast<const float2 *>(tl + a * PS + r * RS + 2);
                            const float v[4] = {v01.x, v01.y, v23.x, v23.y};
                            if (a == 1 && (r == 1 || r == 2)) {
                                old[r - 1][0] = v[1];
                                old[r - 1][1] = v[2];
                            }
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (r - j < 0 || r - j > 2) continue;
                                float *const wp = wb[use / 2 & 1];
                                if (use % 2 == 0) {
                                    if (use > 0) tmem_wait_ld12(wp);
                                    else tmem_use12(wp);  // the wait for the biases covered it
                                    if (use / 2 + 1 < 9) {
                                        tmem_ld8(tm + (use / 2 + 1) * 12, wb[use / 2 + 1 & 1]);
                                        tmem_ld4(tm + (use / 2 + 1) * 12 + 8, wb[use / 2 + 1 & 1] + 8);
                                    }
                                }
#pragma unroll
                                for (int c = 0; c < 3; ++c) {
                                    acc[j][0] = fmaf(wp[use % 2 * 6 + c * 2], v[c], acc[j][0]);
                                    acc[j][1] = fmaf(wp[use % 2 * 6 + c * 2 + 1], v[c + 1], acc[j][1]);
                                }
                                ++use;
                            }
                        }
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int k = 0; k < 2; ++k) own[q][j][k] = fmaf(Act<ACT, float>::fwd(acc[j][k]), bs[4 + 2 * j + k], old[j][k]);
                    if (it + 1 < p.inner) {
                        float *to = tl0 + (cur ^ 1) * TS + toff + PS + RS + 1;
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            to[j * RS] = own[q][j][0];
                            to[j * RS + 1] = own[q][j][1];
                        }
                        bar_sync(B_COMPUTE + slot, COMPUTE);
                    }
                }
                if (o + 1 < p.outer && surface) {
                    unsigned long long *to = p.cells + ((size_t)((o + 1) & 1) * p.B + s0 + q) * P + g00;
#pragma unroll
                    for (int j = 0; j < 2; ++j) st_words(to + (size_t)j * K, cell_word(own[q][j][0], o + 1), cell_word(own[q][j][1], o + 1));
                }
                // a warp's 128 values in float, doubles above the warp
                float sm = (own[q][0][0] + own[q][0][1]) + (own[q][1][0] + own[q][1][1]);
                float sq = fmaf(own[q][0][0], own[q][0][0], own[q][0][1] * own[q][0][1]) + fmaf(own[q][1][0], own[q][1][0], own[q][1][1] * own[q][1][1]);
                __syncwarp();
                sm = warp_sum(sm);
                sq = warp_sum(sq);
                if (lane == 0) wsum[q][warp] = make_float2(sm, sq);
                __syncwarp();
                bar_arrive(B_DONE + q, watched);
            }
        }
        // ---- the last normalisation
        float gb[8];
        __syncwarp();
        tmem_ld8(tm + COL_REST + 8, gb);
        tmem_wait_ld8(gb);
#pragma unroll
        for (int q = 0; q < MAX_SPC; ++q) {
            if (q >= ns) continue;
            bar_sync(B_STATS + q, watched);
            const float2 mr = mstats[q];
#pragma unroll
            for (int j = 0; j < 2; ++j)
                *reinterpret_cast<float2 *>(p.y + (size_t)(s0 + q) * P + g00 + (size_t)j * K) =
                    make_float2(fmaf((own[q][j][0] - mr.x) * mr.y, gb[2 * j], gb[4 + 2 * j]), fmaf((own[q][j][1] - mr.x) * mr.y, gb[2 * j + 1], gb[5 + 2 * j]));
        }
    }
    if (gave_up) report_wait(p.error_flag, p.status);
    tmem_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free_all(tmem_slot);
}

template <int ACT>
static int launch_one(const OuterHeldParams &p, int ctas, cudaStream_t st)
{
    using namespace held8;
    const void *kern = reinterpret_cast<const void *>(outer_held_k<ACT>);
    static unsigned long long attr_set = 0;
    if (first_use_on_device(&attr_set)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALONE);
        if (e != cudaSuccess) {
            record_cuda_error(e, "cudaFuncSetAttribute(outer_held_k)");
            return GN_ERR_CUDA;
        }
    }
    void *args[] = {const_cast<OuterHeldParams *>(&p)};
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(ctas), dim3(THREADS), args, SMEM_ALONE, st);
    if (e != cudaSuccess) {
        record_cuda_error(e, "cudaLaunchCooperativeKernel(outer_held_k)");
        (void)cudaGetLastError();
        return GN_ERR_CUDA;
    }
    return GN_OK;
}

// CTAs of the kernel that are resident at once, one per SM, 0 where it cannot run; asked once per device
static int usable_sms()
{
    static std::atomic<int> known[64];  // + 1
    int dev = 0, coop = 0, per_sm = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < 64 && known[dev].load(std::memory_order_relaxed)) return known[dev].load(std::memory_order_relaxed) - 1;
    auto kern = outer_held_k<GN_ACT_TANH>;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, held8::SMEM_ALONE) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, held8::THREADS, held8::SMEM_ALONE) == cudaSuccess && per_sm > 0)
        n = sm_count();
    else (void)cudaGetLastError();  // what could not be set or asked is an answer too
    if (dev < 64) known[dev].store(n + 1, std::memory_order_relaxed);
    return n;
}

// Samples per CTA, or 0 if the kernel does not apply: block 8, at least one outer step, at most MAX_INNER inner iterations, all blocks of
// a chunk of samples resident at once, at most MAX_SPC samples per CTA (each takes 10 KB of shared memory per block and registers for its patch). Wherever it
// applies it is ahead of the loop of one launch per step, us, step by step / this kernel: 64^3, 4 x 12, one sample 166 / 80, two 217 / 105;
// 64^3, 1 x 4 54 / 46; 40 x 56 x 72, 3 x 6 87 / 48; 48^3, 4 x 10, four samples 128 / 89; 32^3, 2 x 8, sixteen 101 / 56; 16^3, 2 x 8, 148
// samples 103 / 52, 5 x 16, 120 samples 306 / 140. Where the blocks' weights fit into registers outer_small.cu is: 32^3, 2 x 8, eight samples
// 38 there, 41 here.
int outer_held_spc(int B, int M, int N, int K, int block, int inner, int outer, const void *w, const void *b, const void *s, const void *gamma,
                   const void *beta, const void *x, const void *y)
{
    if (block != 8 || inner < 1 || inner > held8::MAX_INNER || outer < 1 || B < 1 || M % 8 || N % 8 || K % 8) return 0;
    const long long P = (long long)M * N * K;
    if (P >= (1LL << 31) || (long long)B * P > kOuterSmallMaxCells) return 0;
    auto al8 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0; };
    if (!(al8(w) && al8(b) && al8(s) && al8(gamma) && al8(beta) && al8(y)) || (reinterpret_cast<uintptr_t>(x) & 3)) return 0;
    const long long group = ((long long)(M / 8) * (N / 8) * (K / 8) + held8::SLOTS_PER_CTA - 1) / held8::SLOTS_PER_CTA;
    const long long chunks = usable_sms() / group;
    if (chunks < 1) return 0;
    const int spc = (int)((B + chunks - 1) / chunks);
    return spc <= held8::MAX_SPC ? spc : 0;
}

int launch_outer_held(const float *w, const float *b, const float *s, const float *gamma, const float *beta, const float *x, float *y,
                      unsigned long long *cells, unsigned long long *sums, int *error_flag, int B, int M, int N, int K, int inner, int outer,
                      int spc, float eps, int act, cudaStream_t st)
{
    OuterHeldParams p{};
    p.w = w; p.b = b; p.s = s; p.gamma = gamma; p.beta = beta; p.x = x; p.y = y;
    p.cells = cells; p.sums = sums; p.error_flag = error_flag; p.status = device_status_ptr();
    p.nblocks = (M / 8) * (N / 8) * (K / 8);
    p.group = (p.nblocks + held8::SLOTS_PER_CTA - 1) / held8::SLOTS_PER_CTA;
    p.B = B; p.M = M; p.N = N; p.K = K; p.inner = inner; p.outer = outer; p.spc = spc; p.eps = eps;
    const int ctas = p.group * ((B + spc - 1) / spc);
    switch (act) {
    case GN_ACT_RELU: return launch_one<GN_ACT_RELU>(p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_one<GN_ACT_LEAKY_RELU>(p, ctas, st);
    case GN_ACT_SILU: return launch_one<GN_ACT_SILU>(p, ctas, st);
    default: return launch_one<GN_ACT_TANH>(p, ctas, st);
    }
}

}  // namespace gn
