// The model loop with gradients on the quad kernels, as two calls: forward (also without gradients) and backward.
//
//   plain     h = x;  repeat: h = layer_norm(step(h))                gridnet/scripts/train_mnist.py:62-64
//   residual  h = x;  repeat: n = layer_norm(h); h = h + step(n) - n  gridnet/scripts/train_imagenet.py:81-83
//   gated     as plain, with the gated step (gridnet/scripts/train_mnist.py:36-44), block 8, shared parameters
//
// with one set of step parameters for all outer steps or one per step (train_imagenet.py:54-58). Activations stay in the
// IL4 layout from the first step to the last; everything that a step needs is queued from here, so an outer step costs the
// host a few microseconds (as a sequence of library calls and tensor operations from Python it was 30 us forward and
// 150 us backward, which is what small models took).
#include "common.cuh"
#include "kernels.h"

namespace gn {

static size_t up256(size_t v) { return (v + 255) / 256 * 256; }

struct LoopDims {
    int B, M, N, K, Q, inner, outer, block, nparams, residual;
    long long P;
    size_t T4;  // floats of an IL4 tensor
    int regions;
};

static LoopDims loop_dims(int B, int M, int N, int K, int inner, int outer, int block, int nparams, int residual)
{
    LoopDims d;
    d.B = B; d.M = M; d.N = N; d.K = K; d.Q = (B + 3) / 4; d.inner = inner; d.outer = outer; d.block = block;
    d.nparams = nparams; d.residual = residual;
    d.P = (long long)M * N * K;
    d.T4 = (size_t)d.Q * d.P * 4;
    d.regions = (M / 8) * (N / 8) * (K / 8);
    return d;
}

struct LoopWs {
    float *packed, *packed_t, *gpk, *tmp, *g[2], *delta, *dsum, *dsq, *replay;
    float2 *gbt, *ac;
    double2 *partials;
    size_t bytes;
};

// replay: some step has no kept iterations, so the backward pass runs the inner iterations again
static LoopWs carve_loop(void *base, const LoopDims &d, bool backward, bool replay)
{
    LoopWs w{};
    size_t off = 0;
    unsigned char *p = static_cast<unsigned char *>(base);
    auto take = [&](size_t bytes) {
        void *r = p + off;
        off = up256(off + bytes);
        return r;
    };
    const size_t pk = sizeof(float) * quad_packed_floats(d.M, d.N, d.K), t = sizeof(float) * d.T4;
    size_t parts = d.regions;
    if (backward && (size_t)quad_norm_parts(d.P) > parts) parts = quad_norm_parts(d.P);
    if (d.residual && (size_t)quad_combine_parts(d.P) > parts) parts = quad_combine_parts(d.P);
    w.partials = static_cast<double2 *>(take(sizeof(double2) * parts * 4 * d.Q));
    w.gbt = static_cast<float2 *>(take(sizeof(float2) * (size_t)d.regions * quad_tile_cells(d.block)));
    if (!backward || replay) w.packed = static_cast<float *>(take(pk));
    if (!backward && d.residual) w.tmp = static_cast<float *>(take(t));
    if (backward) {
        w.packed_t = static_cast<float *>(take(pk));
        w.gpk = static_cast<float *>(take(sizeof(float) * quad_grad_floats(d.M, d.N, d.K, d.Q, 1)));
        w.ac = static_cast<float2 *>(take(sizeof(float2) * 4 * d.Q));
        for (int i = 0; i < 2; ++i) w.g[i] = static_cast<float *>(take(t));
        w.delta = static_cast<float *>(take(t * d.inner));
        w.dsum = static_cast<float *>(take(t));
        w.dsq = static_cast<float *>(take(t / 4));
        if (replay) w.replay = static_cast<float *>(take(t * d.inner));
    }
    w.bytes = off;
    return w;
}

static int loop_check(int B, int M, int N, int K, int inner, int outer, int block, int act, int nparams)
{
    if (B <= 0 || M <= 0 || N <= 0 || K <= 0 || outer < 1) return GN_ERR_BAD_SHAPE;
    if (block != 4 && block != 8) return GN_ERR_BAD_BLOCK;
    if (inner < 1) return GN_ERR_BAD_INNER;
    if (act < GN_ACT_RELU || act > GN_ACT_TANH) return GN_ERR_BAD_ACTIVATION;
    if (nparams != 1 && nparams != outer) return GN_ERR_BAD_SHAPE;
    if (!quad_applicable(M, N, K, block, inner)) return GN_ERR_UNSUPPORTED;
    return GN_OK;
}

#define TRY_(call)                     \
    do {                               \
        const int rc_ = (call);        \
        if (rc_ != GN_OK) return rc_;  \
    } while (0)

// ---- gated
struct GatedWs {
    float *packed, *packed_t, *gpk, *g[2], *delta, *dsum, *replay;
    float2 *gbt, *ac;
    double2 *partials;
    size_t bytes;
};

static GatedWs carve_gated(void *base, const LoopDims &d, bool backward, bool replay)
{
    GatedWs w{};
    size_t off = 0;
    unsigned char *p = static_cast<unsigned char *>(base);
    auto take = [&](size_t bytes) {
        void *r = p + off;
        off = up256(off + bytes);
        return r;
    };
    const size_t pk = 2 * sizeof(float) * quad_packed_floats(d.M, d.N, d.K), t = sizeof(float) * d.T4;
    size_t parts = 2 * (size_t)d.regions;
    if (backward && (size_t)quad_norm_parts(d.P) > parts) parts = quad_norm_parts(d.P);
    w.partials = static_cast<double2 *>(take(sizeof(double2) * parts * 4 * d.Q));
    w.gbt = static_cast<float2 *>(take(sizeof(float2) * (size_t)d.regions * quad_tile_cells(8)));
    if (!backward || replay) w.packed = static_cast<float *>(take(pk));
    if (backward) {
        w.packed_t = static_cast<float *>(take(pk));
        w.gpk = static_cast<float *>(take(sizeof(float) * quad_grad_floats(d.M, d.N, d.K, d.Q, 2)));
        w.ac = static_cast<float2 *>(take(sizeof(float2) * 4 * d.Q));
        for (int i = 0; i < 2; ++i) w.g[i] = static_cast<float *>(take(t));
        w.delta = static_cast<float *>(take(2 * t * d.inner));
        w.dsum = static_cast<float *>(take(2 * t));
        if (replay) w.replay = static_cast<float *>(take(3 * t * d.inner));
    }
    w.bytes = off;
    return w;
}

// one step; kept: [3][inner] tensors (the two pre-activations, the activations that went in), or nullptr
static int gated_step(const GatedWs &w, const LoopDims &d, const float *in, const float2 *in_stats, float *out, double2 *partials, float *kept,
                      int params_old, int act, cudaStream_t st)
{
    QuadGated a{};
    a.packed = w.packed; a.gbt = w.gbt; a.params_old = params_old; a.in_il4 = in; a.out_il4 = out; a.in_stats = in_stats;
    a.out_partials = partials; a.nparts = 2 * d.regions;
    if (kept) {
        a.hv = kept; a.hg = kept + d.inner * d.T4; a.x = kept + 2 * d.inner * d.T4;
    }
    a.M = d.M; a.N = d.N; a.K = d.K; a.Q = d.Q; a.inner = d.inner;
    return launch_quad_gated_fwd(a, act, st);
}

}  // namespace gn

using namespace gn;

extern "C" {

GN_API int gn_loop_train_supported(int B, int M, int N, int K, int inner, int block)
{
    return loop_check(B, M, N, K, inner, 1, block, GN_ACT_RELU, 1) == GN_OK;
}

GN_API size_t gn_loop_tensor_bytes(int B, int M, int N, int K)
{
    if (B <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
    return (size_t)((B + 3) / 4) * M * N * K * 16;
}

GN_API size_t gn_loop_forward_workspace_bytes(int B, int M, int N, int K, int inner, int outer, int block, int residual)
{
    if (loop_check(B, M, N, K, inner, outer, block, GN_ACT_RELU, 1) != GN_OK) return 0;
    return carve_loop(nullptr, loop_dims(B, M, N, K, inner, outer, block, 1, residual), false, false).bytes;
}

GN_API size_t gn_loop_backward_workspace_bytes(int B, int M, int N, int K, int inner, int outer, int block, int residual, int replay)
{
    if (loop_check(B, M, N, K, inner, outer, block, GN_ACT_RELU, 1) != GN_OK) return 0;
    return carve_loop(nullptr, loop_dims(B, M, N, K, inner, outer, block, 1, residual), true, replay != 0).bytes;
}

GN_API int gn_loop_forward_f32(const float *const *weights, const float *const *biases, const float *const *scales, int nparams,
                               const float *gamma, const float *beta, const float *x, float *y, float *x_il4, float *const *outs,
                               float *stats, float *const *stashes, int B, int M, int N, int K, int inner, int outer, int block,
                               float ln_eps, int act, int residual, void *workspace, size_t workspace_bytes, void *stream)
{
    TRY_(loop_check(B, M, N, K, inner, outer, block, act, nparams));
    if (!weights || !biases || !scales || !gamma || !beta || !x || !y || !x_il4 || !outs || !stats || !workspace) return GN_ERR_NULL_POINTER;
    const LoopDims d = loop_dims(B, M, N, K, inner, outer, block, nparams, residual);
    const LoopWs w = carve_loop(workspace, d, false, false);
    if (workspace_bytes < w.bytes || reinterpret_cast<uintptr_t>(workspace) % 256) return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    float2 *const mr = reinterpret_cast<float2 *>(stats);
    const int S = 4 * d.Q;  // statistics of one step
    {
        QuadPrepare a{};
        a.w = weights[0]; a.b = biases[0]; a.s = scales[0]; a.packed = w.packed; a.ordered = true;
        a.gamma = gamma; a.beta = beta; a.gbt = w.gbt;
        a.x = x; a.il = x_il4; a.B = B;
        TRY_(launch_quad_prepare(a, M, N, K, block, st));
    }
    if (residual) {
        TRY_(launch_quad_residual_combine(x_il4, nullptr, nullptr, nullptr, nullptr, nullptr, w.partials, d.Q, d.P, st));
        TRY_(launch_norm_finalize(w.partials, quad_combine_parts(d.P), mr, S, d.P, ln_eps, st));
    }
    for (int k = 0; k < outer; ++k) {
        if (k > 0 && nparams > 1) {
            QuadPrepare a{};
            a.w = weights[k]; a.b = biases[k]; a.s = scales[k]; a.packed = w.packed; a.ordered = true;
            TRY_(launch_quad_prepare(a, M, N, K, block, st));
        }
        const float *in = k ? outs[k - 1] : x_il4;
        QuadStep a{};
        a.packed = w.packed; a.gbt = w.gbt;
        a.in_il4 = in;
        a.out_il4 = residual ? w.tmp : outs[k];
        a.in_stats = residual ? mr + (size_t)k * S : (k ? mr + (size_t)(k - 1) * S : nullptr);
        a.out_partials = residual ? nullptr : w.partials;
        a.nparts = d.regions;
        a.params_old = k > 0 && nparams == 1;
        if (stashes) a.save_h = stashes[k];
        a.M = M; a.N = N; a.K = K; a.Q = d.Q; a.inner = inner; a.block = block;
        TRY_(launch_step_fwd_quad(a, act, st));
        if (residual) {
            TRY_(launch_quad_residual_combine(in, w.tmp, gamma, beta, mr + (size_t)k * S, outs[k], w.partials, d.Q, d.P, st));
            if (k + 1 < outer) TRY_(launch_norm_finalize(w.partials, quad_combine_parts(d.P), mr + (size_t)(k + 1) * S, S, d.P, ln_eps, st));
        } else {
            TRY_(launch_norm_finalize(w.partials, d.regions, mr + (size_t)k * S, S, d.P, ln_eps, st));
        }
    }
    return launch_from_il4(outs[outer - 1], residual ? nullptr : mr + (size_t)(outer - 1) * S, gamma, beta, y, B, d.P, st);
}

GN_API int gn_loop_backward_f32(const float *const *weights, const float *const *biases, const float *const *scales, int nparams,
                                const float *gamma, const float *beta, const float *x_il4, float *const *outs, const float *stats,
                                float *const *stashes, const float *gy, float *const *gw, float *const *gb, float *const *gs,
                                float *ggamma, float *gbeta, float *gx, int B, int M, int N, int K, int inner, int outer, int block,
                                int act, int residual, void *workspace, size_t workspace_bytes, void *stream)
{
    TRY_(loop_check(B, M, N, K, inner, outer, block, act, nparams));
    if (!weights || !biases || !scales || !gamma || !beta || !x_il4 || !outs || !stats || !gy || !gw || !gb || !gs || !ggamma || !gbeta ||
        !gx || !workspace)
        return GN_ERR_NULL_POINTER;
    const LoopDims d = loop_dims(B, M, N, K, inner, outer, block, nparams, residual);
    bool replay = false;
    for (int k = 0; k < outer; ++k) replay |= !stashes || !stashes[k];
    const LoopWs w = carve_loop(workspace, d, true, replay);
    if (workspace_bytes < w.bytes || reinterpret_cast<uintptr_t>(workspace) % 256) return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const float2 *const mr = reinterpret_cast<const float2 *>(stats);
    const int S = 4 * d.Q;
    const bool with_border = !residual && quad_border_takes_sums(M, N, K, block);
    int cur = 0;
    for (int k = outer - 1; k >= 0; --k) {
        const int kp = nparams > 1 ? k : 0;
        const bool first = k == outer - 1;  // first to be walked back
        const float *in = k ? outs[k - 1] : x_il4;
        const float2 *in_stats = residual ? mr + (size_t)k * S : (k ? mr + (size_t)(k - 1) * S : nullptr);
        const bool kept = stashes && stashes[k];
        bool fresh = false;  // the kernel queued last has re-ordered parameters
        if (first || nparams > 1) {
            QuadPrepare a{};
            a.w = weights[kp]; a.b = biases[kp]; a.s = scales[kp]; a.b_t = gamma; a.packed_t = w.packed_t;
            if (replay) a.packed = w.packed;
            a.ordered = true;
            if (first) {
                a.gamma = gamma; a.beta = beta; a.gbt = w.gbt;
                a.x = gy; a.il = w.g[0]; a.B = B; a.gradient = true;
            }
            TRY_(launch_quad_prepare(a, M, N, K, block, st));
            fresh = true;
        }
        if (!residual && (first || !with_border)) {  // else taken with the border of the step after
            TRY_(launch_quad_norm_sums(outs[k], w.g[cur], nullptr, gamma, mr + (size_t)k * S, w.partials, ggamma, gbeta, !first, w.ac, d.Q, d.P, st));
            fresh = false;
        }
        float *const h = kept ? stashes[k] : w.replay;
        if (!kept) {
            QuadStep a{};
            a.packed = w.packed; a.gbt = w.gbt;
            a.in_il4 = in; a.in_stats = in_stats;
            a.save_h = h;
            a.M = M; a.N = N; a.K = K; a.Q = d.Q; a.inner = inner; a.block = block;
            TRY_(launch_step_fwd_quad(a, act, st));
            fresh = false;
        }
        QuadReverse r{};
        r.packed_t = w.packed_t; r.g = w.g[cur];
        r.params_old = !fresh;
        if (!residual) {
            r.raw = outs[k]; r.stats = mr + (size_t)k * S; r.ac = w.ac;
        }
        r.h = h; r.delta = w.delta; r.dsum = w.dsum; r.gx = w.g[cur ^ 1]; r.dsq = w.dsq;
        r.M = M; r.N = N; r.K = K; r.Q = d.Q; r.inner = inner; r.block = block;
        TRY_(launch_quad_reverse(r, act, st));
        QuadWgrad g{};
        g.in_il4 = in; g.gbt = w.gbt; g.in_stats = in_stats;
        g.delta = w.delta; g.h = h; g.scale = scales[kp]; g.dsq = w.dsq; g.gpk = w.gpk;
        g.accumulate = nparams == 1 && !first;
        g.M = M; g.N = N; g.K = K; g.Q = d.Q; g.inner = inner; g.block = block;
        TRY_(launch_quad_wgrad(g, act, st));
        if (nparams > 1 && k > 0) TRY_(launch_quad_finish(w.gpk, gw[kp], gb[kp], gs[kp], nullptr, nullptr, B, M, N, K, block, 1, st));
        QuadBorder o{};
        o.w = weights[kp]; o.dsum = w.dsum; o.gx = w.g[cur ^ 1];
        if (with_border && k > 0) {  // with the sums of the norm that made this step's input
            o.x_il4 = in; o.stats = in_stats; o.gamma = gamma; o.partials = w.partials; o.ggamma = ggamma; o.gbeta = gbeta; o.ac = w.ac;
            o.accumulate = 1;
        }
        o.M = M; o.N = N; o.K = K; o.Q = d.Q; o.block = block;
        TRY_(launch_quad_border(o, st));
        if (residual) {
            TRY_(launch_quad_norm_sums(in, w.g[cur ^ 1], w.g[cur], gamma, in_stats, w.partials, ggamma, gbeta, !first, w.ac, d.Q, d.P, st));
            TRY_(launch_quad_norm_residual_apply(in, w.g[cur ^ 1], w.g[cur], gamma, in_stats, w.ac, w.g[cur], d.Q, d.P, st));
        } else {
            cur ^= 1;
        }
    }
    return launch_quad_finish(w.gpk, gw[0], gb[0], gs[0], w.g[cur], gx, B, M, N, K, block, 1, st);
}

GN_API size_t gn_gated_loop_workspace_bytes(int B, int M, int N, int K, int inner, int outer, int backward, int replay)
{
    if (loop_check(B, M, N, K, inner, outer, 8, GN_ACT_RELU, 1) != GN_OK) return 0;
    return carve_gated(nullptr, loop_dims(B, M, N, K, inner, outer, 8, 1, 0), backward != 0, replay != 0).bytes;
}

GN_API int gn_gated_loop_forward_f32(const float *weight, const float *bias, const float *gamma, const float *beta, const float *x, float *y,
                                     float *x_il4, float *const *outs, float *stats, float *const *stashes, int B, int M, int N, int K,
                                     int inner, int outer, float ln_eps, int act, void *workspace, size_t workspace_bytes, void *stream)
{
    TRY_(loop_check(B, M, N, K, inner, outer, 8, act, 1));
    if (!weight || !bias || !gamma || !beta || !x || !y || !x_il4 || !outs || !stats || !workspace) return GN_ERR_NULL_POINTER;
    const LoopDims d = loop_dims(B, M, N, K, inner, outer, 8, 1, 0);
    const GatedWs w = carve_gated(workspace, d, false, false);
    if (workspace_bytes < w.bytes || reinterpret_cast<uintptr_t>(workspace) % 256) return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    float2 *const mr = reinterpret_cast<float2 *>(stats);
    const int S = 4 * d.Q;
    QuadPrepare a{};
    a.w = weight; a.b = bias; a.s = weight; a.gated = true; a.packed = w.packed;
    a.gamma = gamma; a.beta = beta; a.gbt = w.gbt;
    a.x = x; a.il = x_il4; a.B = B;
    TRY_(launch_quad_prepare(a, M, N, K, 8, st));
    for (int k = 0; k < outer; ++k) {
        TRY_(gated_step(w, d, k ? outs[k - 1] : x_il4, k ? mr + (size_t)(k - 1) * S : nullptr, outs[k], w.partials, stashes ? stashes[k] : nullptr,
                        k > 0, act, st));
        TRY_(launch_norm_finalize(w.partials, 2 * d.regions, mr + (size_t)k * S, S, d.P, ln_eps, st));
    }
    return launch_from_il4(outs[outer - 1], mr + (size_t)(outer - 1) * S, gamma, beta, y, B, d.P, st);
}

GN_API int gn_gated_loop_backward_f32(const float *weight, const float *bias, const float *gamma, const float *beta, const float *x_il4,
                                      float *const *outs, const float *stats, float *const *stashes, const float *gy, float *gw, float *gb,
                                      float *ggamma, float *gbeta, float *gx, int B, int M, int N, int K, int inner, int outer, int act,
                                      void *workspace, size_t workspace_bytes, void *stream)
{
    TRY_(loop_check(B, M, N, K, inner, outer, 8, act, 1));
    if (!weight || !bias || !gamma || !beta || !x_il4 || !outs || !stats || !gy || !gw || !gb || !ggamma || !gbeta || !gx || !workspace)
        return GN_ERR_NULL_POINTER;
    const LoopDims d = loop_dims(B, M, N, K, inner, outer, 8, 1, 0);
    bool replay = false;
    for (int k = 0; k < outer; ++k) replay |= !stashes || !stashes[k];
    const GatedWs w = carve_gated(workspace, d, true, replay);
    if (workspace_bytes < w.bytes || reinterpret_cast<uintptr_t>(workspace) % 256) return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const float2 *const mr = reinterpret_cast<const float2 *>(stats);
    const int S = 4 * d.Q;
    {
        QuadPrepare a{};
        a.w = weight; a.b = bias; a.s = weight; a.b_t = bias; a.gated = true; a.packed_t = w.packed_t;
        if (replay) a.packed = w.packed;
        a.gamma = gamma; a.beta = beta; a.gbt = w.gbt;
        a.x = gy; a.il = w.g[0]; a.B = B; a.gradient = true;
        TRY_(launch_quad_prepare(a, M, N, K, 8, st));
    }
    const bool with_border = quad_border_takes_sums(M, N, K, 8);
    float *const delta_v = w.delta, *const delta_g = w.delta + inner * d.T4, *const dsum_v = w.dsum, *const dsum_g = w.dsum + d.T4;
    int cur = 0;
    for (int k = outer - 1; k >= 0; --k, cur ^= 1) {
        const bool first = k == outer - 1;
        const float *in = k ? outs[k - 1] : x_il4;
        const float2 *in_stats = k ? mr + (size_t)(k - 1) * S : nullptr;
        if (first || !with_border)  // else taken with the border of the step after
            TRY_(launch_quad_norm_sums(outs[k], w.g[cur], nullptr, gamma, mr + (size_t)k * S, w.partials, ggamma, gbeta, !first, w.ac, d.Q, d.P, st));
        float *kept = stashes ? stashes[k] : nullptr;
        if (!kept) {
            // the step's output is computed once more, into the buffer that receives the gradient afterwards
            kept = w.replay;
            TRY_(gated_step(w, d, in, in_stats, w.g[cur ^ 1], nullptr, kept, 1, act, st));
        }
        QuadGatedReverse r{};
        r.packed_t = w.packed_t; r.gamma = gamma; r.g = w.g[cur]; r.raw = outs[k]; r.stats = mr + (size_t)k * S; r.ac = w.ac;
        r.hv = kept; r.hg = kept + inner * d.T4; r.x = kept + 2 * inner * d.T4;
        r.delta_v = delta_v; r.delta_g = delta_g; r.dsum_v = dsum_v; r.dsum_g = dsum_g; r.gx = w.g[cur ^ 1];
        r.M = M; r.N = N; r.K = K; r.Q = d.Q; r.inner = inner;
        TRY_(launch_quad_gated_reverse(r, act, st));
        QuadWgrad g{};
        g.in_il4 = in; g.gbt = w.gbt; g.in_stats = in_stats;
        g.delta = delta_v; g.delta2 = delta_g; g.h = r.x + d.T4; g.gpk = w.gpk;
        g.accumulate = !first;
        g.M = M; g.N = N; g.K = K; g.Q = d.Q; g.inner = inner; g.block = 8;
        TRY_(launch_quad_wgrad(g, act, st));
        QuadBorder o{};
        o.w = weight; o.dsum = dsum_v; o.dsum2 = dsum_g; o.gx = w.g[cur ^ 1];
        if (with_border && k > 0) {  // with the sums of the norm that made this step's input
            o.x_il4 = in; o.stats = in_stats; o.gamma = gamma; o.partials = w.partials; o.ggamma = ggamma; o.gbeta = gbeta; o.ac = w.ac;
            o.accumulate = 1;
        }
        o.M = M; o.N = N; o.K = K; o.Q = d.Q; o.block = 8;
        TRY_(launch_quad_border(o, st));
    }
    return launch_quad_finish(w.gpk, gw, gb, nullptr, w.g[cur], gx, B, M, N, K, 8, 2, st);
}

}  // extern "C"
