// bic_pair.cu -- host side of the paired-tap bicubic RGC (bic_pair.cuh), the gradient field it reads
// and the kernel that reads its two planes.
#include "bic_pair.cuh"

#include <math.h>

#include <algorithm>
#include <vector>

#include "device_common.cuh"
#include "pair_shape.h"

namespace esrrf {

namespace {

using namespace bicpair;

// Catmull-Rom sample (sample2d of device_common.cuh, the same arithmetic) of a gradient image at half
// pixel (x + OX / 2, y + OY / 2), away from the border, from its 4 x 4 support g(i, j) (columns x - 1 + i,
// rows y - 1 + j).  On half positions the cubic's weights are 0 1 0 0 or -1/16 9/16 9/16 -1/16, exact both.
// FINITE (whole-number frames): the taps of weight 0 add nothing; else they spread a NaN or an infinity.
template <int OX, int OY, bool FINITE, class G>
__device__ __forceinline__ float half_sample(G g) {
    constexpr float a = -0.0625f, b = 0.5625f;
    constexpr float cx[4] = {OX ? a : 0.f, OX ? b : 1.f, OX ? b : 0.f, OX ? a : 0.f};
    constexpr float cy[4] = {OY ? a : 0.f, OY ? b : 1.f, OY ? b : 0.f, OY ? a : 0.f};
    float q = 0.0f;
#pragma unroll
    for (int j = 0; j <= 3; j++) {
        if (FINITE && cy[j] == 0.f) continue;
        float p = 0.0f;
#pragma unroll
        for (int i = 0; i <= 3; i++)
            if (!(FINITE && cx[i] == 0.f)) p = p + g(i, j) * cx[i];
        q = q + p * cy[j];
    }
    return q;
}

// sample2d's border branch: bilinear with extrapolation.
template <class G>
__device__ __forceinline__ float half_border(int w, int h, int X, int Y, G g) {
    const float x = (float)X / 2.0f, y = (float)Y / 2.0f;
    const int xb = (int)fminf((float)w - 2, fmaxf(x, 0.0f));
    const int yb = (int)fminf((float)h - 2, fmaxf(y, 0.0f));
    const float xf = x - (float)xb, yf = y - (float)yb;
    const float ll = g(xb, yb), lr = g(xb + 1, yb), ur = g(xb + 1, yb + 1), ul = g(xb, yb + 1);
    const float upper = ul + xf * (ur - ul);
    const float lower = ll + xf * (lr - ll);
    return lower + yf * (upper - lower);
}

// Unit gradient at the nodes from the raw frames, in one pass (as separate kernels the gradients,
// their 2x resampling and the normalisation took 3.8 of the 22 ms of a 100-frame block of 512 x 512 at
// M4; 0.6 here).  The tap of node (nx, ny) reads Gx at (ny - 1, nx) and Gy at (ny, nx - 1) of the 2x grid and
// exists for 0 < n < 2 size (liveSRRF.cl:271-292).  A thread has the four nodes 2x + 1, 2x + 2 by
// 2y + 1, 2y + 2, whose samples lie at x, x + 1/2, x + 1 and read one 6 x 6 patch of the frame: one node a
// thread (64 loads each) took 0.46 ms per 32 frames.  Also writes the frame as floats.
template <bool U16>
__global__ void __launch_bounds__(256) bic_nodes_kernel(const void* __restrict__ raw, int w, int h,
                                                        float* __restrict__ fraw, float2* __restrict__ U) {
    const int x = blockIdx.x * 32 + (int)threadIdx.x - 1, y = blockIdx.y * 8 + (int)threadIdx.y - 1;
    const long f = blockIdx.z, base = f * (long)w * h;
    if (x >= w || y >= h) return;
    auto I = [&](int u, int v) { return dev::load_px(raw, U16 ? 1 : 0, base + (long)v * w + u); };
    if (x >= 0 && y >= 0) fraw[base + (long)y * w + x] = I(x, y);
    auto put = [&](int nx, int ny, float Gx, float Gy) {
        if (nx < 0 || ny < 0 || nx >= 2 * w || ny >= 2 * h) return;
        float2 u = make_float2(0.f, 0.f);
        const float n2 = Gx * Gx + Gy * Gy;
        // node 0 takes no tap; no gradient, or one beyond FP32: none
        if (nx > 0 && ny > 0 && n2 > 0.f && n2 <= 3.402823466e38f) {
            const float inv = rsqrtf(n2);
            u = make_float2(Gx * inv, Gy * inv + 0.f);  // + 0: -0 becomes +0
        }
        U[(f * 2 * h + ny) * 2 * w + nx] = u;
    };
    // the samples' supports start at x - 1 .. x (x + 1/2 and x + 1), their gradients one to the left
    if (x >= 2 && x + 1 < w - 2 && y >= 2 && y + 1 < h - 2) {
        float r[6][6];
#pragma unroll
        for (int j = 0; j < 6; ++j)
#pragma unroll
            for (int i = 0; i < 6; ++i) r[j][i] = I(x - 2 + i, y - 2 + j);
        // gradient images at column x - 1 + i, row y - 1 + j
        auto gx = [&](int i, int j) { return r[j + 1][i + 1] - r[j + 1][i]; };
        auto gy = [&](int i, int j) { return r[j + 1][i + 1] - r[j][i + 1]; };
        auto gx_r = [&](int i, int j) { return gx(i + 1, j); };
        auto gy_d = [&](int i, int j) { return gy(i, j + 1); };
        // node (nx, ny): Gx at (nx / 2, (ny - 1) / 2), Gy at ((nx - 1) / 2, ny / 2)
        put(2 * x + 1, 2 * y + 1, half_sample<1, 0, U16>(gx), half_sample<0, 1, U16>(gy));
        put(2 * x + 2, 2 * y + 1, half_sample<0, 0, U16>(gx_r), half_sample<1, 1, U16>(gy));
        put(2 * x + 1, 2 * y + 2, half_sample<1, 1, U16>(gx), half_sample<0, 0, U16>(gy_d));
        put(2 * x + 2, 2 * y + 2, half_sample<0, 1, U16>(gx_r), half_sample<1, 0, U16>(gy_d));
        return;
    }
    auto gxa = [&](int u, int v) { return I(u, v) - I(max(u - 1, 0), v); };
    auto gya = [&](int u, int v) { return I(u, v) - I(u, max(v - 1, 0)); };
    auto at = [&](auto g, int X, int Y) {  // sample2d at (X / 2, Y / 2)
        const int u0 = X >> 1, v0 = Y >> 1;
        if (!(u0 > 0 && u0 < w - 2 && v0 > 0 && v0 < h - 2)) return half_border(w, h, X, Y, g);
        auto s = [&](int i, int j) { return g(u0 - 1 + i, v0 - 1 + j); };
        if (X & 1) return Y & 1 ? half_sample<1, 1, U16>(s) : half_sample<1, 0, U16>(s);
        return Y & 1 ? half_sample<0, 1, U16>(s) : half_sample<0, 0, U16>(s);
    };
    for (int k = 0; k < 4; ++k) {
        const int nx = 2 * x + 1 + (k & 1), ny = 2 * y + 1 + (k >> 1);
        if (nx < 0 || ny < 0 || nx >= 2 * w || ny >= 2 * h) continue;
        if (nx == 0 || ny == 0) put(nx, ny, 0.f, 0.f);
        else put(nx, ny, at(gxa, nx, ny - 1), at(gya, nx - 1, ny));
    }
}

struct BicCumArgs {
    const float* own;
    const float* edge;
    const float* fraw;
    const float* wsum;
    int w, h, F, I, t0;
    float sens;
    int int_weighting;
    BlockState st;
    float* cg_out;  // per-frame mode: own itself
    float* v_out;
};

// The Catmull-Rom weight at distance d (dev::cubic) of the M sub-pixel phases: exact in FP32 for M 2 and 4.
constexpr float cubic_at(float d) {
    const float x = d < 0 ? -d : d;
    return x < 1.0f ? x * x * (x * 1.5f - 2.5f) + 1.0f : x < 2.0f ? -0.5f * x * x * x + 2.5f * x * x - 4.0f * x + 2.0f : 0.0f;
}
template <int M>
struct Vec {
    using T = float4;
};
template <>
struct Vec<2> {
    using T = float2;
};
template <int M>
__device__ __forceinline__ void load_m(float (&d)[M], const float* s) {
    const typename Vec<M>::T v = *reinterpret_cast<const typename Vec<M>::T*>(s);
    d[0] = v.x, d[1] = v.y;
    if constexpr (M == 4) d[2] = v.z, d[3] = v.w;
}

// The same for the two cells at either end of every row, one pixel a thread (16 rows at M 2, 8 at M 4
// a CTA): they are sampled bilinearly at the border, which would hold up the warps of every row.
template <int M, int SENS>
__device__ __noinline__ void ends(const BicCumArgs& a) {
    constexpr int kEnds = 4 * M, kRows = 128 / kEnds;
    const int WM = a.w * M, i = threadIdx.x % kEnds;
    const int x = i < 2 * M ? i : WM - kEnds + i, y = blockIdx.y * kRows + threadIdx.x / kEnds;
    if (y >= a.h * M) return;
    const long wh = (long)WM * a.h * M, pix = (long)y * WM + x, pl = (long)a.w * a.h;
    const bool emit = a.cg_out != nullptr;
    constexpr int SW = 16 * M;
    const int pos = x % SW;
    const bool e = (pos < a.I && x >= SW) || (pos >= SW - a.I && x - pos + SW < WM);
    const dev::Sample2dAt sp = dev::sample2d_at(a.w, a.h, (float)x / (float)M - 0.5f, (float)y / (float)M - 0.5f);
    const float ws = a.wsum[pix];
    float prev = emit ? 0.f : a.st.prev[pix], s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 2
    for (int t = 0; t < a.F; ++t) {
        const long o = (long)t * wh + pix;
        const float g = (a.own[o] + (e ? __ldg(a.edge + o) : 0.f)) / ws;
        const float v = dev::sample2d_apply(a.fraw + t * pl, a.w, sp);
        if (emit) {
            a.cg_out[o] = g;
            a.v_out[o] = v;
            continue;
        }
        const float cg = dev::cglh_power(g, SENS ? (float)SENS : a.sens);
        const float X = a.int_weighting ? v * cg : cg;
        s0 += X;
        s1 = fmaf(X, X, s1);
        if (a.t0 + t > 0) s2 = fmaf(X, prev, s2);
        s3 += v;
        prev = X;
    }
    if (emit) return;
    a.st.acc[pix] += (double)s0;
    a.st.acc[wh + pix] += (double)s1;
    a.st.acc[2 * wh + pix] += (double)s2;
    a.st.acc[3 * wh + pix] += (double)s3;
    a.st.prev[pix] = prev;
}

// sample2d's border branch, for the rows at the top and the bottom (their columns are inside).
__device__ __forceinline__ float row_sample(const float* __restrict__ a, int w, int h, float x, float y) {
    const int xb = (int)x, yb = (int)fminf((float)h - 2, fmaxf(y, 0.0f));
    const float xf = x - (float)xb, yf = y - (float)yb;
    const float* r = a + (long)yb * w + xb;
    const float ll = __ldg(r), lr = __ldg(r + 1), ul = __ldg(r + w), ur = __ldg(r + w + 1);
    const float upper = ul + xf * (ur - ul);
    const float lower = ll + xf * (lr - ll);
    return lower + yf * (upper - lower);
}

// The launch's frames of the M output pixels of a cell's row: CGLH over its sum of weights, the bicubic
// intensity, the sensitivity and the cumulants (FP32 over the launch's frames, folded into the block's
// FP64 accumulators once), or in the per-frame mode the first two.  The M pixels' 4 x 4 supports lie in one 5 x 4 patch (columns q - 2 .. q + 2): 20 loads for M
// samples, the weights of a phase compile-time constants, those of the row the same for a whole CTA.
// One pixel a thread took 1.03 ms per 32 frames of 512 x 512 at M4, this 0.70.
template <int M, int SENS>
__global__ void __launch_bounds__(128, 6) bic_cumulants_kernel(BicCumArgs a) {
    if (blockIdx.x == gridDim.x - 1) {
        ends<M, SENS>(a);
        return;
    }
    const int q = blockIdx.x * blockDim.x + threadIdx.x + 2, y = blockIdx.y;
    if (q >= a.w - 2) return;
    const int WM = a.w * M;
    const long wh = (long)WM * a.h * M, pix = (long)y * WM + q * M, pl = (long)a.w * a.h;
    const bool emit = a.cg_out != nullptr;
    constexpr int SW = 16 * M;
    // which of the pixels have terms in the edge plane (a strip's first and last I columns)
    const int x0 = q * M, pos = x0 % SW;
    const int el = x0 >= SW ? a.I - pos : 0;                       // pixels k < el
    const int er = x0 - pos + SW < WM ? SW - a.I - pos : M;        // pixels k >= er
    const bool any = el > 0 || er < M;
    // sample2d_at of the pixels: columns u0 - 1 .. u0 + 2, u0 = q - 1 (left half of the cell) or q
    const float yc = (float)y / (float)M - 0.5f;
    const int v0 = (int)floorf(yc);
    const bool inner = v0 > 0 && v0 < a.h - 2;  // the columns are: 2 <= q <= w - 3
    float cy[4], ws[M], prev[M];
#pragma unroll
    for (int j = 0; j < 4; ++j) cy[j] = dev::cubic(yc - (float)(v0 - 1 + j));
    load_m<M>(ws, a.wsum + pix);
#pragma unroll
    for (int k = 0; k < M; ++k) prev[k] = emit ? 0.f : a.st.prev[pix + k];
    float s0[M] = {}, s1[M] = {}, s2[M] = {}, s3[M] = {};
    const float* fr = a.fraw + (long)(v0 - 1) * a.w + q - 2;
#pragma unroll 1
    for (int t = 0; t < a.F; ++t, fr += pl) {
        float c[M], v[M];
        const long o = (long)t * wh + pix;
        load_m<M>(c, a.own + o);
        if (any) {
            float d[M];
            load_m<M>(d, a.edge + o);
#pragma unroll
            for (int k = 0; k < M; ++k)
                if (k < el || k >= er) c[k] += d[k];
        }
        if (inner) {
            float r[4][5];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 5; ++i) r[j][i] = __ldg(fr + (long)j * a.w + i);
#pragma unroll
            for (int k = 0; k < M; ++k) {  // sample2d_apply
                constexpr float fM = (float)M;
                float s = 0.0f;
#pragma unroll
                for (int j = 0; j <= 3; j++) {
                    float p = 0.0f;
#pragma unroll
                    for (int i = 0; i <= 3; i++) {
                        const float at = (float)k / fM - 0.5f;  // from q; u0 = -1 or 0
                        p = p + r[j][i + (k < M / 2 ? 0 : 1)] * cubic_at(at - (float)((k < M / 2 ? -2 : -1) + i));
                    }
                    s = s + p * cy[j];
                }
                v[k] = s;
            }
        } else {
#pragma unroll
            for (int k = 0; k < M; ++k)
                v[k] = row_sample(a.fraw + t * pl, a.w, a.h, (float)(x0 + k) / (float)M - 0.5f, yc);
        }
#pragma unroll
        for (int k = 0; k < M; ++k) {
            const float g = c[k] / ws[k];
            if (emit) {
                a.cg_out[o + k] = g;
                a.v_out[o + k] = v[k];
                continue;
            }
            const float cg = dev::cglh_power(g, SENS ? (float)SENS : a.sens);
            const float X = a.int_weighting ? v[k] * cg : cg;
            s0[k] += X;
            s1[k] = fmaf(X, X, s1[k]);
            if (a.t0 + t > 0) s2[k] = fmaf(X, prev[k], s2[k]);
            s3[k] += v[k];
            prev[k] = X;
        }
    }
    if (emit) return;
#pragma unroll
    for (int k = 0; k < M; ++k) {
        a.st.acc[pix + k] += (double)s0[k];
        a.st.acc[wh + pix + k] += (double)s1[k];
        a.st.acc[2 * wh + pix + k] += (double)s2[k];
        a.st.acc[3 * wh + pix + k] += (double)s3[k];
        a.st.prev[pix + k] = prev[k];
    }
}

template <int M>
cudaError_t launch_cumulants(const BicCumArgs& c, cudaStream_t stream) {
    const dim3 grid((c.w - 4 + 127) / 128 + 1, c.h * M);  // cells 2 .. w - 3 and, last, the ends
    if (c.sens == 1.f) bic_cumulants_kernel<M, 1><<<grid, 128, 0, stream>>>(c);
    else if (c.sens == 2.f) bic_cumulants_kernel<M, 2><<<grid, 128, 0, stream>>>(c);
    else bic_cumulants_kernel<M, 0><<<grid, 128, 0, stream>>>(c);
    return cudaGetLastError();
}

}  // namespace

namespace {

// The table's (I + 1) x kNJ entries too, if `tab` is given.
BicPairTables reach(const BicGeometry& g, int M, std::vector<float2>* tab) {
    BicPairTables t;
    if (M != 2 && M != 4) return t;
    // distances of i - 1/2 and j - 1/2 output pixels inside the disc of tSO raw pixels; d, the weight
    // and the cut-off in raw pixels, the reference's floats
    auto weight = [&](int i, int j, float& w, float& wd) {
        w = wd = 0.f;
        const float dx = (float)((i - 0.5) / M), dy = (float)((j - 0.5) / M), d = sqrtf(dx * dx + dy * dy);
        if (!(d <= g.tSO)) return false;
        w = d * expf(-(d * d) / g.tSS);
        w = w * w * w * w;
        wd = (float)((double)w / ((double)d * M));  // the kernel's cross products are in output pixels
        return true;
    };
    float w, wd;
    int I = 0;
    while (I <= kMaxJ && weight(I + 1, 1, w, wd)) ++I;
    if (I < 1 || I > kMaxJ) return t;
    if (tab) tab->assign((size_t)(I + 1) * kNJ, make_float2(0.f, 0.f));
    for (int i = 1; i <= I; ++i)
        for (int j = 1; j < kNJ && weight(i, j, w, wd); ++j) {
            if (tab) (*tab)[(size_t)i * kNJ + j] = make_float2(w, wd);
            t.J[i] = (signed char)j;
            t.taps += 4;  // a quadrant's distance stands for four taps
        }
    t.I = I;
    t.taps = t.taps * 4 / (M * M);  // nodes in an output's disc
    return t;
}

}  // namespace

BicPairTables bic_pair_reach(const BicGeometry& g, int M) { return reach(g, M, nullptr); }

cudaError_t bic_pair_tables(const BicGeometry& g, int M, BicPairTables& t) {
    std::vector<float2> tab;
    t = reach(g, M, &tab);
    if (t.I < 1) return cudaSuccess;
    cudaError_t e = cudaMalloc(&t.wt, sizeof(float2) * tab.size());
    if (e != cudaSuccess) return e;
    return cudaMemcpy(t.wt, tab.data(), sizeof(float2) * tab.size(), cudaMemcpyHostToDevice);
}

void bic_pair_tables_free(BicPairTables& t) {
    cudaFree(t.wt);
    t = BicPairTables();
}

cudaError_t bic_nodes(const void* raw, int is_u16, int w, int h, int F, float* fraw, float2* U, cudaStream_t stream) {
    // threads (x, y) from -1: nodes 0 belong to x = -1 (2x + 2)
    const dim3 grid((w + 32) / 32, (h + 8) / 8, F), block(32, 8);
    if (is_u16) bic_nodes_kernel<true><<<grid, block, 0, stream>>>(raw, w, h, fraw, U);
    else bic_nodes_kernel<false><<<grid, block, 0, stream>>>(raw, w, h, fraw, U);
    return cudaGetLastError();
}

namespace {

BicPairArgs pair_args(const BicPairTables& t, int w, int h, int M) {
    BicPairArgs p{};
    p.W = w * M;
    p.H = h * M;
    p.w2 = 2 * w;
    p.h2 = 2 * h;
    p.strips = (2 * w + 31) / 32;
    p.I = t.I;
    for (int i = 0; i <= t.I; ++i) p.J[i] = t.J[i];
    const int J = t.I, h2 = M / 2;  // the disc is as high as it is wide
    p.CH = 4 * ((J + 3) / 4);
    p.NC = p.CH / 4 + ((kK - 1) * h2 + J - 1) / 4 + 1;
    p.halo = (t.I + h2 - 1) / h2 * h2;
    p.cps = (16 * M + 2 * p.halo) / h2;
    return p;
}

int pair_warps(const BicPairArgs& p, int M) {
    return (int)std::min<size_t>(16, (225 * 1024 - table_bytes(p)) / warp_bytes(p, M / 2)) & ~1;
}

}  // namespace

bool bic_pair_fits(const BicPairTables& t, int w, int h, int M) {
    if (t.I < 1 || (long)h * M > 65535 || 2L * h > 65535 * 8L) return false;
    return pair_warps(pair_args(t, w, h, M), M) >= 4;
}

namespace {

PairShape shape_of(const BicPairArgs& p, int M, int F, int sms) {
    // a segment walks whole blocks of 4 M rows: half of one more on either side, on average
    return pair_shape(p.strips * F, p.H, p.I + 2 * M, pair_warps(p, M), sms);
}

}  // namespace

// Both forms' times modelled as in rgc_pair.cu: 0.20 us per row and warp here with segments up to 100
// rows, 0.13 from 400 on, for 808 instructions a row; the tabulated kernel 6.5 us a CTA and frame with
// four CTAs an SM at 64 taps, and its gradient kernels.  Measured, one launch with its gradients: 25 of
// 512 x 512 at M4 2.1 ms against 5.4, 20 frames of 120 x 100 at M4 141 us / 229, 12 of 90 x 80 at M2 (radius
// 3) 85 / 102, 12 of 37 x 29 at M4 87 / 63, 12 of 60 x 50 at M4 (radius 3) 188 / 128.  Of 251 launches that it
// gives to this form, drawn from 4 x 4 to 700 x 700 pixels, radii 0.5 to 4 and 1 to 32 frames, ten are slower, by
// 3 to 22 % of 40 to 120 us (eight of them at radius 0.5, 24 taps); the others take 0.64 of the tabulated form's time.
bool bic_pair_pays(const BicPairTables& t, int w, int h, int M, int F) {
    if (t.I < 1 || F > 65535 || (2L * w + 31) / 32 * F > (1 << 26)) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const int sms = sm_count(dev);
    const BicPairArgs p = pair_args(t, w, h, M);
    const PairShape sh = shape_of(p, M, F, sms);
    const double per_node = t.taps * M * M / 4.0;  // outputs a node reaches
    const double row = (8 * per_node / 2 * 5.2 + 250 * t.I) / (4 * M);
    const double row_us = 0.13 + 0.07 * std::min(1.0, std::max(0.0, (400.0 - sh.rows) / 300.0));
    const double pair_us = 8 + sh.cost * row_us * row / 808 + (6e-6 + 2.3e-5 / (M * M)) * w * M * h * M * F;
    const long ctas = (long)M * M * ((w + 31) / 32) * ((h + 7) / 8), slots = 4L * sms;
    const double tab_us = 16 + (ctas + slots - 1) / slots * (double)F * 6.5 * (14 * t.taps + 250) / 1146 *
                                   (0.35 + 0.65 * std::min(1.0, (double)ctas / slots)) +
                          1.25e-4 * w * h * F;
    return pair_us < tab_us;
}

bool bic_pair_pays_up_to(const BicPairTables& t, int w, int h, int M, int F) {
    for (int f = F; f >= 1; --f)
        if (bic_pair_pays(t, w, h, M, f)) return true;
    return false;
}

// A frame of the tabulated form holds 19 input planes on the device (the frame and its gradients, the 2x
// gradients and the padded unit-gradient field): launches within 2 GB of them.  The paired form adds its
// two output planes (its nodes share the 2x gradients' memory), 2 M^2 input planes; its launches of few frames run
// shorter segments, so they have the 4 GB of the Fourier path: 100 frames of 1024 x 1024 at M4 36.0
// ms in launches of 9 (2 GB), 33.1 of 17 (4 GB), 32.7 of 25 (5.4 GB).
int bic_launch_cap(const BicGeometry& g, int w, int h, int M, bool plain, int want) {
    const double plane = sizeof(float) * (double)w * h;
    const int f = (int)std::max(1.0, std::min((double)want, 2e9 / (19 * plane)));
    const BicPairTables t = plain ? BicPairTables() : bic_pair_reach(g, M);
    if (!bic_pair_fits(t, w, h, M) || !bic_pair_pays_up_to(t, w, h, M, f)) return f;
    return (int)std::max(1.0, std::min((double)want, 4e9 / ((19 + 2.0 * M * M) * plane)));
}

cudaError_t bic_rgc_pair(const BicPairRun& r, const BicPairTables& t, cudaStream_t stream) {
    BicPairArgs p = pair_args(t, r.w, r.h, r.M);
    p.U = r.U;
    p.wt = reinterpret_cast<const float4*>(t.wt);
    p.own = r.cg_out ? r.cg_out : r.own;
    p.edge = r.edge;
    p.F = r.F;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const PairShape sh = shape_of(p, r.M, r.F, sm_count(dev));
    p.rows = sh.rows;
    p.segs = sh.segs;
    switch (r.M) {
        case 2: e = launch<2>(p, sh.warps, stream); break;
        case 4: e = launch<4>(p, sh.warps, stream); break;
        default: return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    BicCumArgs c{};
    c.own = p.own;
    c.edge = r.edge;
    c.fraw = r.fraw;
    c.wsum = r.wsum;
    c.w = r.w;
    c.h = r.h;
    c.F = r.F;
    c.I = t.I;
    c.t0 = r.t0;
    c.sens = r.sens;
    c.int_weighting = r.int_weighting;
    c.st = r.st;
    c.cg_out = r.cg_out;
    c.v_out = r.v_out;
    return r.M == 2 ? launch_cumulants<2>(c, stream) : launch_cumulants<4>(c, stream);
}

}  // namespace esrrf
