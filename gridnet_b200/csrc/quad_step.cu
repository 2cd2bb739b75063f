// One step of the update on the quad kernels, forward and backward, with or without per-block normalisation.
//
// The tensors of the caller are in the grid's own layout; a step interleaves its input by four samples (IL4), and what
// the backward pass wants from the forward pass stays in that layout. The conversions are 16 bytes per cell and direction,
// less than a tenth of what the step itself moves.
#include "common.cuh"
#include "kernels.h"

namespace gn {

namespace {

struct StepDims {
    int B, M, N, K, Q, inner, block, normalize;
    long long P;
    size_t t;  // bytes of an IL4 tensor
};

StepDims step_dims(int B, int M, int N, int K, int inner, int block, int normalize)
{
    StepDims d;
    d.B = B; d.M = M; d.N = N; d.K = K; d.Q = (B + 3) / 4; d.inner = inner; d.block = block; d.normalize = normalize;
    d.P = (long long)M * N * K;
    d.t = (size_t)d.Q * d.P * 16;
    return d;
}

struct Cut {
    unsigned char *p;
    size_t off = 0;
    explicit Cut(void *base) : p(static_cast<unsigned char *>(base)) {}
    template <typename T>
    void take(T *&r, size_t bytes)
    {
        r = reinterpret_cast<T *>(p + off);
        off += (bytes + 255) / 256 * 256;
    }
};

// What the backward pass needs from the forward pass
struct Kept {
    float *x, *y, *wsum, *h;
    float4 *stats;
    size_t bytes;
};
Kept carve_kept(void *base, const StepDims &d)
{
    Kept k{};
    Cut c(base);
    c.take(k.x, d.t);
    if (d.normalize) {
        c.take(k.y, d.t);
        c.take(k.wsum, sizeof(float) * d.P);
        c.take(k.stats, sizeof(float4) * quad_stats_vectors(d.M, d.N, d.K, d.Q, d.inner, d.block));
    }
    c.take(k.h, d.t * d.inner);
    k.bytes = c.off;
    return k;
}

struct StepWs {
    float *packed, *x, *y, *wsum;                                   // forward
    float *packed_t, *gpk, *gin, *gout, *delta, *dsum, *dsq;  // backward
    float4 *hterm;
    void *kept;
    size_t bytes;
};
// kept: the forward pass keeps (backward: kept) what the backward pass needs
StepWs carve_step(void *base, const StepDims &d, bool backward, bool kept)
{
    StepWs w{};
    Cut c(base);
    const size_t pk = sizeof(float) * quad_packed_floats(d.M, d.N, d.K);
    if (!backward || !kept) c.take(w.packed, pk);
    if (!backward) {
        if (!kept) {
            c.take(w.x, d.t);
            if (d.normalize) c.take(w.wsum, sizeof(float) * d.P);
        }
        if (!kept || !d.normalize) c.take(w.y, d.t);
    } else {
        c.take(w.packed_t, pk);
        c.take(w.gpk, sizeof(float) * quad_grad_floats(d.M, d.N, d.K, d.Q, 1));
        c.take(w.gin, d.t);
        c.take(w.gout, d.t);
        c.take(w.delta, d.t * d.inner);
        c.take(w.dsum, d.t);
        c.take(w.dsq, d.t / 4);
        if (d.normalize) c.take(w.hterm, sizeof(float4) * 2 * d.Q * quad_tiles(d.M, d.N, d.K, d.block));
        if (!kept) c.take(w.kept, carve_kept(nullptr, d).bytes);
    }
    w.bytes = c.off;
    return w;
}

int step_check(int B, int M, int N, int K, int inner, int block, int act)
{
    if (B <= 0 || M <= 0 || N <= 0 || K <= 0) return GN_ERR_BAD_SHAPE;
    if (block != 4 && block != 8) return GN_ERR_BAD_BLOCK;
    if (inner < 1) return GN_ERR_BAD_INNER;
    if (act < GN_ACT_RELU || act > GN_ACT_TANH) return GN_ERR_BAD_ACTIVATION;
    if (!quad_applicable(M, N, K, block, inner)) return GN_ERR_UNSUPPORTED;
    return GN_OK;
}

#define TRY_(call)                     \
    do {                               \
        const int rc_ = (call);        \
        if (rc_ != GN_OK) return rc_;  \
    } while (0)

// the step itself: x -> y (IL4), x_il4; k: keep for the backward pass
int run_forward(const float *w, const float *b, const float *s, float *packed, const float *x, float *x_il4, float *y, float *wsum, const Kept *k,
                float eps, int act, const StepDims &d, cudaStream_t st)
{
    QuadPrepare r{};
    r.w = w; r.b = b; r.s = s; r.packed = packed; r.x = x; r.il = x_il4; r.B = d.B;
    if (d.normalize) r.wsum = wsum;
    r.ordered = !d.normalize;
    TRY_(launch_quad_prepare(r, d.M, d.N, d.K, d.block, st));
    QuadStep a{};
    a.packed = packed; a.in_il4 = x_il4; a.out_il4 = y;
    if (d.normalize) a.wsum = wsum;
    a.eps = eps;
    if (k) {
        a.save_h = k->h;
        a.tile_stats = k->stats;
    }
    a.M = d.M; a.N = d.N; a.K = d.K; a.Q = d.Q; a.inner = d.inner; a.block = d.block;
    return launch_step_fwd_quad(a, act, st);
}

}  // namespace
}  // namespace gn

using namespace gn;

extern "C" {

GN_API size_t gn_step_kept_bytes(int B, int M, int N, int K, int inner, int block, int normalize)
{
    if (step_check(B, M, N, K, inner, block, GN_ACT_RELU) != GN_OK) return 0;
    return carve_kept(nullptr, step_dims(B, M, N, K, inner, block, normalize)).bytes;
}

GN_API size_t gn_step_kept_workspace_bytes(int B, int M, int N, int K, int inner, int block, int normalize, int backward, int kept)
{
    if (step_check(B, M, N, K, inner, block, GN_ACT_RELU) != GN_OK) return 0;
    return carve_step(nullptr, step_dims(B, M, N, K, inner, block, normalize), backward != 0, kept != 0).bytes;
}

GN_API int gn_step_forward_kept_f32(const float *w, const float *b, const float *s, const float *x, float *y, int B, int M, int N, int K,
                                    int inner, int block, float eps, int normalize, int act, void *kept, size_t kept_bytes, void *workspace,
                                    size_t workspace_bytes, void *stream)
{
    TRY_(step_check(B, M, N, K, inner, block, act));
    if (!w || !b || !s || !x || !y || !workspace) return GN_ERR_NULL_POINTER;
    const StepDims d = step_dims(B, M, N, K, inner, block, normalize);
    const StepWs ws = carve_step(workspace, d, false, kept != nullptr);
    const Kept k = carve_kept(kept, d);
    if (workspace_bytes < ws.bytes || (kept && kept_bytes < k.bytes) || reinterpret_cast<uintptr_t>(workspace) % 256 ||
        reinterpret_cast<uintptr_t>(kept) % 256)
        return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    float *const xi = kept ? k.x : ws.x, *const yi = kept && normalize ? k.y : ws.y;
    TRY_(run_forward(w, b, s, ws.packed, x, xi, yi, kept ? k.wsum : ws.wsum, kept ? &k : nullptr, eps, act, d, st));
    return launch_from_il4(yi, nullptr, nullptr, nullptr, y, B, d.P, st);
}

GN_API int gn_step_backward_kept_f32(const float *w, const float *b, const float *s, const float *x, const float *gy, float *gw, float *gb,
                                     float *gs, float *gx, int B, int M, int N, int K, int inner, int block, float eps, int normalize,
                                     int act, void *kept, size_t kept_bytes, void *workspace, size_t workspace_bytes, void *stream)
{
    TRY_(step_check(B, M, N, K, inner, block, act));
    if (!w || !b || !s || (!x && !kept) || !gy || !gw || !gb || !gs || !gx || !workspace) return GN_ERR_NULL_POINTER;
    const StepDims d = step_dims(B, M, N, K, inner, block, normalize);
    const StepWs ws = carve_step(workspace, d, true, kept != nullptr);
    const Kept k = carve_kept(kept ? kept : ws.kept, d);
    if (workspace_bytes < ws.bytes || (kept && kept_bytes < k.bytes) || reinterpret_cast<uintptr_t>(workspace) % 256 ||
        reinterpret_cast<uintptr_t>(kept) % 256)
        return GN_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    if (!kept) TRY_(run_forward(w, b, s, ws.packed, x, k.x, k.y, k.wsum, &k, eps, act, d, st));
    QuadPrepare a{};
    a.w = w; a.b_t = b; a.s = s; a.packed_t = ws.packed_t; a.x = gy; a.il = ws.gin; a.B = B; a.gradient = true;
    TRY_(launch_quad_prepare(a, M, N, K, block, st));
    QuadReverse r{};
    r.packed_t = ws.packed_t; r.g = ws.gin; r.h = k.h;
    if (normalize) {
        r.raw = k.y; r.wsum = k.wsum; r.tile_stats = k.stats; r.hterm = ws.hterm;
    }
    r.delta = ws.delta; r.dsum = ws.dsum; r.gx = ws.gout; r.dsq = ws.dsq;
    r.M = M; r.N = N; r.K = K; r.Q = d.Q; r.inner = inner; r.block = block;
    TRY_(launch_quad_reverse(r, act, st));
    QuadWgrad g{};
    g.in_il4 = k.x; g.delta = ws.delta; g.h = k.h; g.scale = s; g.dsq = ws.dsq; g.gpk = ws.gpk; g.tile_stats = k.stats;
    g.M = M; g.N = N; g.K = K; g.Q = d.Q; g.inner = inner; g.block = block;
    TRY_(launch_quad_wgrad(g, act, st));
    QuadBorder o{};
    o.w = w; o.dsum = ws.dsum; o.gx = ws.gout; o.x_il4 = k.x; o.hterm = ws.hterm;
    o.M = M; o.N = N; o.K = K; o.Q = d.Q; o.block = block;
    TRY_(launch_quad_border(o, st));
    return launch_quad_finish(ws.gpk, gw, gb, gs, ws.gout, gx, B, M, N, K, block, 1, st);
}

}  // extern "C"
