// What the loops of quad_loop.cu queue, without a GPU: that file linked with launchers that write down their arguments instead of
// launching. A line per kernel: its name, the buffers that it reads before it has waited for the kernel ahead of it
// (previous_done() in common.cuh), and the buffers that it writes.
//
//   loop_queue gated|plain|residual  sets of parameters  outer steps  sums in the border pass (0, 1)  steps with kept iterations (bits)
//   loop_queue split  regions  CTAs  quads      in which units items are split (quad_split_unit), for every grid and batch up to these
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <initializer_list>
#include <vector>

#include "../gridnet_b200/csrc/common.cuh"
#include "../gridnet_b200/csrc/kernels.h"
#include "../gridnet_b200/csrc/quad_geo.cuh"

static bool g_border_sums;

static int queue(const char *kernel, std::initializer_list<const void *> ahead, std::initializer_list<const void *> writes)
{
    printf("%s;", kernel);
    for (const void *p : ahead)
        if (p) printf("%p ", p);
    printf(";");
    for (const void *p : writes)
        if (p) printf("%p ", p);
    printf("\n");
    return GN_OK;
}

namespace gn {

bool quad_applicable(int, int, int, int, int) { return true; }
size_t quad_packed_floats(int M, int N, int K) { return 29ull * M * N * K; }
int quad_tile_cells(int) { return 1000; }
size_t quad_grad_floats(int M, int N, int K, int, int branches) { return 29ull * branches * M * N * K; }
int quad_norm_parts(long long) { return 4; }
int quad_combine_parts(long long) { return 4; }
bool quad_border_takes_sums(int, int, int, int) { return g_border_sums; }

int launch_quad_prepare(const QuadPrepare &a, int, int, int, int, cudaStream_t) { return queue("prepare", {}, {a.packed, a.packed_t, a.gbt, a.il}); }
int launch_from_il4(const float *, const float2 *, const float *, const float *, float *y, int, long long, cudaStream_t)
{
    return queue("from_il4", {}, {y});
}
int launch_norm_finalize(const double2 *, int, float2 *stats, int, long long, float, cudaStream_t) { return queue("finalize", {}, {stats}); }
int launch_quad_residual_combine(const float *, const float *, const float *, const float *, const float2 *, float *out, double2 *partials, int, long long,
                                 cudaStream_t)
{
    return queue("combine", {}, {out, partials});
}
int launch_step_fwd_quad(const QuadStep &a, int, cudaStream_t)
{
    return queue("step", {a.params_old ? a.packed : nullptr, a.params_old && a.in_stats ? a.gbt : nullptr}, {a.out_il4, a.out_partials, a.save_h});
}
int launch_quad_gated_fwd(const QuadGated &a, int, cudaStream_t)
{
    return queue("gated_step", {a.params_old ? a.packed : nullptr, a.params_old && a.in_stats ? a.gbt : nullptr}, {a.out_il4, a.out_partials, a.hv, a.hg, a.x});
}
int launch_quad_norm_sums(const float *, const float *, const float *, const float *, const float2 *, double2 *partials, float *ggamma, float *gbeta, int,
                          float2 *ac, int, long long, cudaStream_t)
{
    queue("norm_sums", {}, {partials, ggamma, gbeta});
    return queue("norm_ac", {}, {ac});
}
int launch_quad_norm_residual_apply(const float *, const float *, const float *, const float *, const float2 *, const float2 *, float *out, int, long long,
                                    cudaStream_t)
{
    return queue("apply", {}, {out});
}
int launch_quad_reverse(const QuadReverse &a, int, cudaStream_t)
{
    return queue("reverse", {a.params_old ? a.packed_t : nullptr}, {a.delta, a.dsum, a.gx, a.dsq});
}
int launch_quad_gated_reverse(const QuadGatedReverse &a, int, cudaStream_t)
{
    return queue("gated_reverse", {a.packed_t}, {a.delta_v, a.delta_g, a.dsum_v, a.dsum_g, a.gx});
}
int launch_quad_wgrad(const QuadWgrad &a, int, cudaStream_t) { return queue("wgrad", {a.in_stats ? a.gbt : nullptr, a.scale}, {a.gpk}); }
int launch_quad_finish(const float *, float *gw, float *gb, float *gs, const float *, float *x, int, int, int, int, int, int, cudaStream_t)
{
    return queue("finish", {}, {gw, gb, gs, x});
}
int launch_quad_border(const QuadBorder &a, cudaStream_t)
{
    queue("border", {a.w, a.gamma}, {a.gx, a.partials, a.ggamma, a.gbeta});
    return a.gamma ? queue("norm_ac", {}, {a.ac}) : GN_OK;
}

}  // namespace gn

int main(int argc, char **argv)
{
    using namespace gn;
    if (argc == 5 && !strcmp(argv[1], "split")) {
        // every batch of up to the given number of quads, grids of up to the given number of regions
        for (int regions = 1; regions <= atoi(argv[2]); ++regions)
            for (int Q = 1; Q <= atoi(argv[4]); ++Q) {
                const long long items = (long long)regions * Q, need = (items + quad::QUARTERS - 1) / quad::QUARTERS, ctas = need < atoi(argv[3]) ? need : atoi(argv[3]);
                printf("%d %d %lld %d\n", regions, Q, ctas, quad_split_unit(items, ctas, Q));
            }
        return 0;
    }
    if (argc != 6) return 2;
    const bool gated = !strcmp(argv[1], "gated"), residual = !strcmp(argv[1], "residual");
    const int sets = atoi(argv[2]), outer = atoi(argv[3]), B = 4, side = 16, inner = 2;
    g_border_sums = atoi(argv[4]) != 0;
    const unsigned long kept = strtoul(argv[5], nullptr, 0);
    // addresses that nobody looks behind
    size_t next = 1 << 20;
    auto address = [&]() { return reinterpret_cast<float *>(next += 1 << 20); };
    auto addresses = [&](int n) {
        std::vector<float *> v;
        for (int i = 0; i < n; ++i) v.push_back(address());
        return v;
    };
    const auto w = addresses(sets), b = addresses(sets), s = addresses(sets), gw = addresses(sets), gb = addresses(sets), gs = addresses(sets),
               outs = addresses(outer);
    auto stashes = addresses(outer);
    for (int k = 0; k < outer; ++k)
        if (!(kept >> k & 1)) stashes[k] = nullptr;
    float *gamma = address(), *beta = address(), *x = address(), *y = address(), *x_il4 = address(), *stats = address(), *gy = address(), *ggamma = address(),
          *gbeta = address(), *gx = address();
    void *ws = reinterpret_cast<void *>(1ull << 40);
    const size_t room = 1ull << 40;
    int rc = gated ? gn_gated_loop_forward_f32(w[0], b[0], gamma, beta, x, y, x_il4, outs.data(), stats, stashes.data(), B, side, side, side, inner, outer,
                                               1e-5f, GN_ACT_TANH, ws, room, nullptr)
                   : gn_loop_forward_f32(w.data(), b.data(), s.data(), sets, gamma, beta, x, y, x_il4, outs.data(), stats, stashes.data(), B, side, side,
                                         side, inner, outer, 8, 1e-5f, GN_ACT_TANH, residual, ws, room, nullptr);
    if (rc != GN_OK) return 1;
    rc = gated ? gn_gated_loop_backward_f32(w[0], b[0], gamma, beta, x_il4, outs.data(), stats, stashes.data(), gy, gw[0], gb[0], ggamma, gbeta, gx, B, side,
                                            side, side, inner, outer, GN_ACT_TANH, ws, room, nullptr)
               : gn_loop_backward_f32(w.data(), b.data(), s.data(), sets, gamma, beta, x_il4, outs.data(), stats, stashes.data(), gy, gw.data(), gb.data(),
                                      gs.data(), ggamma, gbeta, gx, B, side, side, side, inner, outer, 8, GN_ACT_TANH, residual, ws, room, nullptr);
    return rc == GN_OK ? 0 : 1;
}
