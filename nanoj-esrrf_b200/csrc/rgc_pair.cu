// rgc_pair.cu -- host side of the paired-tap RGC (rgc_pair.cuh) and the kernels that read its two
// planes: the block cumulants of a launch and, for callers that keep a plane per frame (the sweep,
// the adjoint's loss), CGLH over the sum of weights.
#include "fht_fused.cuh"
#include "pair_shape.h"
#include "rgc_pair.cuh"

#include <algorithm>
#include <vector>

namespace esrrf {

cudaError_t fht_rgc_pair_wide(int R, const pair::PairArgs& a, int warps, cudaStream_t stream);

namespace {

using namespace pair;

// Whether the column at position x of a row has a term from a neighbouring strip's sources.
__device__ __forceinline__ bool has_edge(int x, int W, int R) {
    const int pos = x & (kStrip - 1);
    return (pos < R && x >= kStrip) || (pos >= kStrip - 1 - R && (x | (kStrip - 1)) + 1 < W);
}

struct PairCumArgs {
    const float* own;
    const float* edge;
    const float* interp;
    const float* wsum;
    int W, H, F, R, t0;
    float sens;
    int int_weighting;
    BlockState st;
};

// cglh_power with the common whole sensitivities as compile-time constants (SENS 0: any other).
template <int SENS>
__device__ __forceinline__ float power(float c, float s) {
    if (SENS == 0) return dev::cglh_power(c, s);
    return dev::cglh_power(c, (float)SENS);
}

// The launch's frames of one pixel: CGLH over its sum of weights, the sensitivity, the intensity and
// the cumulants, summed in FP64 into the block's accumulators.
template <int SENS>
__global__ void __launch_bounds__(128) pair_cumulants_kernel(PairCumArgs a) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= a.W) return;
    const long wh = (long)a.W * a.H, pix = (long)blockIdx.y * a.W + x;
    const bool e = has_edge(x, a.W, a.R);
    const float ws = a.wsum[pix];
    float prev = a.st.prev[pix];
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    auto frame = [&](int t, float c, float v) {
        const float cg = power<SENS>(c / ws, a.sens);
        const float x = a.int_weighting ? v * cg : cg;
        const double xd = (double)x;
        s0 += xd;
        s1 = fma(xd, xd, s1);
        if (a.t0 + t > 0) s2 = fma(xd, (double)prev, s2);
        s3 += (double)v;
        prev = x;
    };
    // the planes are read once, straight from HBM: a few frames' loads are issued together
    constexpr int kU = 8;
    int t = 0;
    for (; t + kU <= a.F; t += kU) {
        float c[kU], d[kU], v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const long o = (long)(t + u) * wh + pix;
            c[u] = __ldg(a.own + o);
            d[u] = e ? __ldg(a.edge + o) : 0.f;
            v[u] = __ldg(a.interp + o);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) frame(t + u, c[u] + d[u], v[u]);
    }
    for (; t < a.F; ++t) {
        const long o = (long)t * wh + pix;
        frame(t, __ldg(a.own + o) + (e ? __ldg(a.edge + o) : 0.f), __ldg(a.interp + o));
    }
    a.st.acc[pix] += s0;
    a.st.acc[wh + pix] += s1;
    a.st.acc[2 * wh + pix] += s2;
    a.st.acc[3 * wh + pix] += s3;
    a.st.prev[pix] = prev;
}

// cg = (cg + edge) / wsum, one plane per blockIdx.z.
__global__ void __launch_bounds__(128) pair_normalise_kernel(float* cg, const float* __restrict__ edge,
                                                             const float* __restrict__ wsum, int W, int H, int R) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    const long pix = (long)blockIdx.y * W + x, o = (long)blockIdx.z * W * H + pix;
    const float c = cg[o] + (has_edge(x, W, R) ? __ldg(edge + o) : 0.f);
    cg[o] = c / __ldg(wsum + pix);
}

}  // namespace

cudaError_t fht_pair_tables(const FhtGeometry& g, FhtFusedTables& t, cudaStream_t stream) {
    const int R = (g.S - 2) / 2, S = g.S;
    if (!fht_fused_supported(g) || R > kMaxR) return cudaSuccess;
    const int NJ = (R + 3) & ~1;
    std::vector<float2> w((size_t)(R + 2) * NJ, make_float2(0.f, 0.f));
    for (int i = 0; i <= R + 1; ++i) {
        t.pJ[i] = -1;
        t.pfar[i] = 0;
        for (int j = 0; j <= R + 1; ++j) {
            const size_t o = (size_t)(j + R) * S + (i + R);
            w[(size_t)i * NJ + j] = make_float2(g.w[o], g.wd[o]);
            if (g.w[o] == 0.f && g.wd[o] == 0.f && !(i == 0 && j == 0)) continue;
            if (j <= R) t.pJ[i] = (signed char)j;
            else t.pfar[i] = 1;
        }
    }
    t.taps = 0;
    for (int o = 0; o < S * S; ++o) t.taps += g.w[o] != 0.f;
    cudaError_t e = cudaMalloc(&t.ptab, sizeof(float2) * w.size());
    if (e != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(t.ptab, w.data(), sizeof(float2) * w.size(), cudaMemcpyHostToDevice, stream)) != cudaSuccess)
        return e;
    return cudaStreamSynchronize(stream);  // `w` is a host temporary
}

// Whether the paired-tap kernel is the faster one for a launch.  It has half the instructions a tap,
// but a segment's rows follow one another in one warp, so a launch of few strips and frames cuts them
// into short segments that walk more rows around them than their own.  Both kernels' times are
// modelled, each in proportion to its instructions for the box's taps: 0.18 us per row and warp here
// with segments up to 100 rows, 0.13 from 400 rows on (the widest boxes a fifth more), 34.7 us per tile
// and frame for the fused kernel (0.67 of that where every SM has one tile at most; a tenth more
// with several frame groups, which add into the sums with atomics).  Of 521 launches that it gives to this
// kernel, drawn from 4 x 4 to 700 x 700 pixels at M 1 to 13, boxes of 4 to 32 and 1 to 50 frames, four are
// slower by 4 to 10 % (250 to 320 us of one or two frames), the others 0.57 of the fused kernel's time; for one
// frame the fused kernel stays unless the other is ahead by as much (221 x 163 at M4, box 10:
// modelled 49.0 / 49.7 us, measured 5 us behind).
// Paired against fused, one block: 100 frames of 512 x 512 at M4 15.1 / 24.7 ms, 10 of 128 x 128 161 /
// 229 us, one of 256 x 256 103 / 96 us, one of 128 x 128 82 / 39 us.
bool fht_pair_pays(const FhtGeometry& g, const FhtFusedTables& t, const FhtRgcArgs& a) {
    if (!t.ptab || !a.edge || !(a.own || a.cg_out) || a.H > 65535 || a.F > 65535) return false;
    if ((long)(a.W + kStrip - 1) / kStrip * a.F > (1 << 26)) return false;
    const int R = (g.S - 2) / 2;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const int sms = sm_count(dev);
    const PairShape sh = pair_shape((a.W + kStrip - 1) / kStrip * a.F, a.H, R, R <= 12 ? 16 : 12, sms);
    const double row_us = 0.13 + 0.05 * std::min(1.0, std::max(0.0, (400.0 - sh.rows) / 300.0));
    const double pair_us = sh.cost * row_us * (R > 12 ? 1.2 : 1.0) * (2.75 * t.taps + 110) / 808 + 11 +
                           2.5e-6 * a.W * a.H * a.F;
    const int tiles = (a.W + fused::kTX - 1) / fused::kTX * ((a.H + fused::kTH - 1) / fused::kTH);
    const bool emit = a.cg_out != nullptr;
    const int G = emit || a.prev_out ? fused::frame_groups(tiles, a.F, 2 * sms, emit) : 1;
    const long waves = ((long)tiles * G + 2 * sms - 1) / (2 * sms);
    const double fused_us = 10 + waves * ((a.F + G - 1) / G + (G > 1 && !emit ? 1.0 : 0.0) + 0.25) * 34.7 *
                            (6.2 * t.taps + 300) / 1875 * ((long)tiles * G <= sms ? 0.67 : 1.0) *
                                     (G > 1 && !emit ? 1.1 : 1.0);
    return pair_us < (a.F == 1 ? 0.95 : 1.0) * fused_us;
}

cudaError_t fht_rgc_pair(const FhtGeometry& g, const FhtFusedTables& t, const FhtRgcArgs& a,
                         cudaStream_t stream) {
    const int R = (g.S - 2) / 2;
    PairArgs p{};
    p.interp = a.interp;
    p.wt = t.ptab;
    p.own = a.cg_out ? a.cg_out : a.own;
    p.edge = a.edge;
    p.W = a.W;
    p.H = a.H;
    p.F = a.F;
    for (int i = 0; i <= R + 1; ++i) {
        p.J[i] = t.pJ[i];
        p.far[i] = t.pfar[i];
    }
    p.strips = (a.W + kStrip - 1) / kStrip;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const PairShape sh = pair_shape(p.strips * a.F, a.H, R, R <= 12 ? 16 : 12, sm_count(dev));
    p.rows = sh.rows;
    p.segs = sh.segs;
    const int warps = sh.warps;
    e = R <= 8 ? launch_pair_in<1, 8>(R, p, warps, stream)
                           : fht_rgc_pair_wide(R, p, warps, stream);
    if (e != cudaSuccess) return e;
    if (a.cg_out) {
        pair_normalise_kernel<<<dim3((a.W + 127) / 128, a.H, a.F), 128, 0, stream>>>(a.cg_out, a.edge, t.wsum, a.W,
                                                                                     a.H, R);
        return cudaGetLastError();
    }
    PairCumArgs c{};
    c.own = a.own;
    c.edge = a.edge;
    c.interp = a.interp;
    c.wsum = t.wsum;
    c.W = a.W;
    c.H = a.H;
    c.F = a.F;
    c.R = R;
    c.t0 = a.t0;
    c.sens = g.sensitivity;
    c.int_weighting = a.int_weighting;
    c.st = a.st;
    const dim3 grid((a.W + 127) / 128, a.H);
    if (c.sens == 1.f) pair_cumulants_kernel<1><<<grid, 128, 0, stream>>>(c);
    else if (c.sens == 2.f) pair_cumulants_kernel<2><<<grid, 128, 0, stream>>>(c);
    else pair_cumulants_kernel<0><<<grid, 128, 0, stream>>>(c);
    return cudaGetLastError();
}

}  // namespace esrrf
