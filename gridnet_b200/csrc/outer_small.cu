// The whole fused model loop as ONE persistent kernel, for problems so small that launches are what they cost
// (the reference's MNIST configuration: 32^3 grid, batch 8, 2 inner x 8 outer iterations is 17 launches of a few
// microseconds each when every outer step is a kernel of its own).
//
//   for o in range(outer): h = layer_norm(gridnet_step(h))          gridnet/scripts/train_mnist.py:62-64
//
// A CTA owns one 8x8x8 block and one or two samples for all outer steps. Four warps compute: they keep their 4 x 27 weights
// per thread in registers from start to end (register-patch mapping of step_fast.cu: a thread owns a 1x2x2 patch,
// the sample's 10^3 tile sits in shared memory with rows of 12 floats, two tiles ping-pong over the inner
// iterations) and their own cells from one outer step to the next; only the halo of 488 cells goes through global memory.
//
// What an outer step costs at this size is the way of its results to the other CTAs, and fences and flags are the longest part
// of it (a fence by the writer is 0.7 us here, an acquire by the reader 2.5). So there are none: every 64-bit word that a CTA
// leaves for another carries the number of the step, a cell as (value, step), a block's sum and sum of squares as doubles
// whose low eight bits hold it (44 bits are left, twenty more than the added values have), and the reader looks at the word
// until the step is right. A further warp per sample publishes
// the block's sums and watches for those of the other blocks of that sample; while it does, the other four warps work on
// the CTA's other sample. All CTAs of a sample add the same sums in the same order, hence get the same bits. The words
// are zeroed before the launch (step numbers start at 1), and steps alternate between two sets of them: a block can be at
// most one step ahead of another, since it needs that one's sums. (With one counter for the whole grid and fences: 50 us at
// 32^3, batch 8, 2 x 8 iterations; now 32. The sums of the blocks lie a line apart: side by side, with several blocks writing
// to a line that all the others read, it was 39 to 50.)
//
// The launch is cooperative, so all CTAs are resident and the waits end; should one run out all the same, the kernel
// sets the error flag and the device's status word and goes on.
#include <atomic>

#include "common.cuh"
#include "kernels.h"
#include "outer_words.cuh"
#include "patch_geo.cuh"

namespace gn {

namespace small8 {
constexpr int COMPUTE = 128, WATCHED = 160;   // threads that compute; with the warp that watches a sample
constexpr int THREADS = 256;                  // two warpgroups, so that registers can be moved from the second to the first
constexpr int REGS_COMPUTE = 208, REGS_WATCH = 40;  // together at most the 2 x 128 of the launch
constexpr int MAX_SPC = 2;                    // samples per CTA at most
constexpr int HALO = 488, SLOTS = 4;          // halo cells of a tile, per thread
constexpr unsigned kSpinLimit = 1u << 18;     // polls of another block's sums, about a microsecond each
// named barriers; the watching warp takes part in the first two kinds
constexpr int B_DONE = 1, B_STATS = 1 + MAX_SPC, B_COMPUTE = 1 + 2 * MAX_SPC;
}  // namespace small8

struct OuterSmallParams {
    const float *w, *b, *s, *gamma, *beta, *x;
    float *y;
    unsigned long long *cells;    // [2][B][P] (raw step output, step); zeroed
    unsigned long long *sums;     // [2][B][nblocks], a line each: (sum, sum of squares) as doubles, the low 8 bits the step; zeroed
    int *error_flag, *status;     // of the call, and device_status_ptr(): callers seldom hold the workspace that the first one is in
    int nblocks;
    int B, M, N, K, inner, outer, spc;
    float eps;
};

template <int ACT>
__global__ void __launch_bounds__(small8::THREADS, 2) outer_small_k(const OuterSmallParams p)
{
    using namespace small8;
    using Geo = PatchGeo<8>;
    constexpr int RS = Geo::RS, PS = Geo::PS, TS = Geo::TS;
    __shared__ __align__(16) float tiles[MAX_SPC][2][TS];  // [sample of the CTA][ping-pong]
    __shared__ float2 halo_gb[HALO];
    __shared__ float2 mstats[MAX_SPC];
    __shared__ float2 wsum[MAX_SPC][4];    // per-warp (sum, sum of squares) of the CTA's outputs of this step

    const int tid = threadIdx.x, lane = tid & 31;
    const int nbx = p.K >> 3, nby = p.N >> 3;
    const int blk = blockIdx.x % p.nblocks, chunk = blockIdx.x / p.nblocks;
    const int bx = blk % nbx, by = (blk / nbx) % nby, bz = blk / nbx / nby;
    const size_t P = (size_t)p.M * p.N * p.K;
    const int K = p.K;
    const int s0 = chunk * p.spc, ns = min(p.B - s0, p.spc);

    if (tid >= COMPUTE) {  // ---- the watching warps, one per sample
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_WATCH));
        const int q = (tid - COMPUTE) >> 5;
        if (q >= ns) return;
        bool gave_up = false;  // one wait ran out: the results are lost, do not wait again
        const double per_cell = 1.0 / (double)P;
        for (int o = 1; o <= p.outer; ++o) {
            const unsigned long long tag = (unsigned)o & 0xffu;
            unsigned long long *const sums = p.sums + ((size_t)(o & 1) * p.B + s0 + q) * p.nblocks * kOuterSmallLine;
            bar_sync(B_DONE + q, WATCHED);
            if (lane == 0) {
                double sm = 0.0, sq = 0.0;
#pragma unroll
                for (int wq = 0; wq < 4; ++wq) {
                    sm += (double)wsum[q][wq].x;
                    sq += (double)wsum[q][wq].y;
                }
                st_words(sums + kOuterSmallLine * blk, ((unsigned long long)__double_as_longlong(sm) & ~0xffull) | tag,
                         ((unsigned long long)__double_as_longlong(sq) & ~0xffull) | tag);
            }
            __syncwarp();
            const float2 result = watch_sums(sums, p.nblocks, kOuterSmallLine, tag, per_cell, p.eps, lane, kSpinLimit, gave_up);
            if (lane == 0) mstats[q] = result;
            __syncwarp();
            bar_arrive(B_STATS + q, WATCHED);
        }
        if (gave_up) report_wait(p.error_flag, p.status);
        return;
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
    const int xp = tid & 3, yp = (tid >> 2) & 3, z = tid >> 4;
    const size_t g00 = ((size_t)(bz * 8 + z) * p.N + (by * 8 + 2 * yp)) * K + (bx * 8 + 2 * xp);
    const long long origin = ((long long)(bz * 8 - 1) * p.N + (by * 8 - 1)) * K + (bx * 8 - 1);
    // halo cells this thread fetches for every sample: tile offset (or -1), offset from the tile's origin (or -1 outside).
    // z faces 2 x 10 x 10, y faces 2 x 8 x 10, x faces 2 x 8 x 8
    int soff[SLOTS], rel[SLOTS];
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        const int i = tid + j * COMPUTE;
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
    float w[27][2][2];
#pragma unroll
    for (int t = 0; t < 27; ++t)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 v = *reinterpret_cast<const float2 *>(p.w + (size_t)t * P + g00 + (size_t)j * K);
            w[t][j][0] = v.x;
            w[t][j][1] = v.y;
        }
    float2 bias[2], scl[2], gm[2], bt[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        bias[j] = *reinterpret_cast<const float2 *>(p.b + g00 + (size_t)j * K);
        scl[j] = *reinterpret_cast<const float2 *>(p.s + g00 + (size_t)j * K);
        gm[j] = *reinterpret_cast<const float2 *>(p.gamma + g00 + (size_t)j * K);
        bt[j] = *reinterpret_cast<const float2 *>(p.beta + g00 + (size_t)j * K);
    }
    const int toff = Geo::window_origin(xp, yp, z);

    const bool surface = z == 0 || z == 7 || yp == 0 || yp == 3 || xp == 0 || xp == 3;  // some cell of the patch is another block's halo
    bool gave_up = false;
    unsigned long long c[SLOTS];  // halo cells as last seen
    auto ask = [&](int q, int o) {  // for what the neighbours' step o left (the set of that step)
        const unsigned long long *cells = p.cells + ((size_t)(o & 1) * p.B + s0 + q) * P + origin;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) c[j] = rel[j] >= 0 ? ld_word(cells + rel[j]) : (unsigned long long)o << 32;
    };
    for (int o = 0; o < p.outer; ++o) {
#pragma unroll
        for (int q = 0; q < MAX_SPC; ++q) {
            if (q >= ns) continue;
            float(*tl2)[TS] = tiles[q];
            {
                float v[SLOTS];
                if (o == 0) {
                    const float *xs = p.x + (size_t)(s0 + q) * P + origin;
#pragma unroll
                    for (int j = 0; j < SLOTS; ++j) v[j] = rel[j] >= 0 ? xs[rel[j]] : 0.0f;
                } else {
                    if (ns == 1) ask(q, o);  // else asked for while the other sample was in work
                    for (unsigned spins = 0; !gave_up; ask(q, o)) {
                        bool there = true;
#pragma unroll
                        for (int j = 0; j < SLOTS; ++j) there &= (unsigned)(c[j] >> 32) == (unsigned)o;
                        if (there) break;
                        gave_up = ++spins > kSpinLimit;
                    }
#pragma unroll
                    for (int j = 0; j < SLOTS; ++j) v[j] = __uint_as_float((unsigned)c[j]);
                    __syncwarp();
                    bar_sync(B_STATS + q, WATCHED);  // the sample's statistics of that step
                }
                const float2 mr = o > 0 ? mstats[q] : make_float2(0.0f, 1.0f);
                float *to = tl2[0] + toff + PS + RS + 1;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float u0 = own[q][j][0], u1 = own[q][j][1];
                    to[j * RS] = o > 0 ? fmaf((u0 - mr.x) * mr.y, gm[j].x, bt[j].x) : u0;
                    to[j * RS + 1] = o > 0 ? fmaf((u1 - mr.x) * mr.y, gm[j].y, bt[j].y) : u1;
                }
#pragma unroll
                for (int j = 0; j < SLOTS; ++j)
                    if (soff[j] >= 0) {
                        float u = v[j];
                        if (o > 0) {
                            const float2 gb = halo_gb[tid + j * COMPUTE];
                            u = fmaf((u - mr.x) * mr.y, gb.x, gb.y);
                        }
                        tl2[0][soff[j]] = u;
                        tl2[1][soff[j]] = u;
                    }
            }
            bar_sync(B_COMPUTE, COMPUTE);
            if (ns > 1 && (q == 0 ? o > 0 : o + 1 < p.outer)) ask(q ^ 1, o + q);  // what comes next
            for (int it = 0; it < p.inner; ++it) {
                const int cur = it & 1;
                const float *tl = tl2[cur] + toff;
                float acc[2][2] = {{bias[0].x, bias[0].y}, {bias[1].x, bias[1].y}};
                float old[2][2];
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
                            const int bb = r - j;
                            if (bb >= 0 && bb <= 2) {
#pragma unroll
                                for (int c = 0; c < 3; ++c) {
                                    acc[j][0] = fmaf(w[a * 9 + bb * 3 + c][j][0], v[c], acc[j][0]);
                                    acc[j][1] = fmaf(w[a * 9 + bb * 3 + c][j][1], v[c + 1], acc[j][1]);
                                }
                            }
                        }
                    }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    own[q][j][0] = fmaf(Act<ACT, float>::fwd(acc[j][0]), scl[j].x, old[j][0]);
                    own[q][j][1] = fmaf(Act<ACT, float>::fwd(acc[j][1]), scl[j].y, old[j][1]);
                }
                if (it + 1 < p.inner) {
                    float *to = tl2[cur ^ 1] + toff + PS + RS + 1;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        to[j * RS] = own[q][j][0];
                        to[j * RS + 1] = own[q][j][1];
                    }
                    bar_sync(B_COMPUTE, COMPUTE);
                }
            }
            if (o + 1 < p.outer && surface) {
                unsigned long long *to = p.cells + ((size_t)((o + 1) & 1) * p.B + s0 + q) * P + g00;
#pragma unroll
                for (int j = 0; j < 2; ++j) st_words(to + (size_t)j * K, cell_word(own[q][j][0], o + 1), cell_word(own[q][j][1], o + 1));
            }
            // a warp's 128 values in float (ten shuffles, not twenty), doubles above the warp
            float sm = (own[q][0][0] + own[q][0][1]) + (own[q][1][0] + own[q][1][1]);
            float sq = fmaf(own[q][0][0], own[q][0][0], own[q][0][1] * own[q][0][1]) + fmaf(own[q][1][0], own[q][1][0], own[q][1][1] * own[q][1][1]);
            sm = warp_sum(sm);
            sq = warp_sum(sq);
            if (lane == 0) wsum[q][tid >> 5] = make_float2(sm, sq);
            __syncwarp();
            bar_arrive(B_DONE + q, WATCHED);
        }
    }

    if (gave_up) report_wait(p.error_flag, p.status);
    // ---- the last normalisation
#pragma unroll
    for (int q = 0; q < MAX_SPC; ++q) {
        if (q >= ns) continue;
        bar_sync(B_STATS + q, WATCHED);
        const float2 mr = mstats[q];
#pragma unroll
        for (int j = 0; j < 2; ++j)
            *reinterpret_cast<float2 *>(p.y + (size_t)(s0 + q) * P + g00 + (size_t)j * K) =
                make_float2(fmaf((own[q][j][0] - mr.x) * mr.y, gm[j].x, bt[j].x), fmaf((own[q][j][1] - mr.x) * mr.y, gm[j].y, bt[j].y));
    }
}

template <int ACT>
static int launch_one(const OuterSmallParams &p, int ctas, cudaStream_t st)
{
    void *args[] = {const_cast<OuterSmallParams *>(&p)};
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(outer_small_k<ACT>), dim3(ctas),
                                                      dim3(small8::THREADS), args, 0, st);
    if (e != cudaSuccess) {
        record_cuda_error(e, "cudaLaunchCooperativeKernel(outer_small_k)");
        (void)cudaGetLastError();
        return GN_ERR_CUDA;
    }
    return GN_OK;
}

// CTAs of the kernel that are resident at once on the current device, 0 where it cannot run. Asked once per device: the
// questions cost the host several microseconds, a tenth of the whole loop at these sizes.
static int resident_ctas()
{
    static std::atomic<int> known[64];  // + 1
    int dev = 0, coop = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < 64 && known[dev].load(std::memory_order_relaxed)) return known[dev].load(std::memory_order_relaxed) - 1;
    int n = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, outer_small_k<GN_ACT_TANH>, small8::THREADS, 0) == cudaSuccess)
        n = per_sm * sm_count();
    if (dev < 64) known[dev].store(n + 1, std::memory_order_relaxed);
    return n;
}

// How many samples per CTA the persistent kernel would use for this problem, or 0 if it does not apply: block 8,
// at least one outer step, all CTAs resident at once, at most MAX_SPC samples per CTA, and little enough work per
// outer step (B * P * inner neuron updates) that launches, not arithmetic, are what the step-by-step loop costs.
int outer_small_spc(int B, int M, int N, int K, int block, int inner, int outer, const void *w, const void *b, const void *s,
                    const void *gamma, const void *beta, const void *x, const void *y)
{
    if (block != 8 || inner < 1 || outer < 1 || B < 1 || M % 8 || N % 8 || K % 8) return 0;
    const long long P = (long long)M * N * K;
    if (P >= (1LL << 31) || (long long)B * P * inner > kOuterSmallMaxCells) return 0;
    auto al8 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0; };
    if (!(al8(w) && al8(b) && al8(s) && al8(gamma) && al8(beta) && al8(y)) || (reinterpret_cast<uintptr_t>(x) & 3)) return 0;
    const long long capacity = resident_ctas();
    if (capacity < 1) return 0;
    const long long nblocks = (long long)(M / 8) * (N / 8) * (K / 8);
    if (nblocks > capacity) return 0;
    long long chunks = capacity / nblocks;
    if (chunks > B) chunks = B;
    const int spc = (int)((B + chunks - 1) / chunks);
    return spc <= small8::MAX_SPC ? spc : 0;
}

int launch_outer_small(const float *w, const float *b, const float *s, const float *gamma, const float *beta, const float *x,
                       float *y, unsigned long long *cells, unsigned long long *sums, int *error_flag, int B, int M, int N, int K,
                       int inner, int outer, int spc, float eps, int act, cudaStream_t st)
{
    OuterSmallParams p{};
    p.w = w; p.b = b; p.s = s; p.gamma = gamma; p.beta = beta; p.x = x; p.y = y;
    p.cells = cells; p.sums = sums; p.error_flag = error_flag; p.status = device_status_ptr();
    p.nblocks = (M / 8) * (N / 8) * (K / 8);
    p.B = B; p.M = M; p.N = N; p.K = K; p.inner = inner; p.outer = outer; p.spc = spc; p.eps = eps;
    const int ctas = p.nblocks * ((B + spc - 1) / spc);
    switch (act) {
    case GN_ACT_RELU: return launch_one<GN_ACT_RELU>(p, ctas, st);
    case GN_ACT_LEAKY_RELU: return launch_one<GN_ACT_LEAKY_RELU>(p, ctas, st);
    case GN_ACT_SILU: return launch_one<GN_ACT_SILU>(p, ctas, st);
    default: return launch_one<GN_ACT_TANH>(p, ctas, st);
    }
}

}  // namespace gn
