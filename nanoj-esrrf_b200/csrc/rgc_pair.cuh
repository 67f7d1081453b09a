// rgc_pair.cuh -- radial gradient convergence on Fourier-interpolated frames without drift
// (liveSRRF_noInterpolation.cl:245-393), two opposite taps at a time.
//
// A source s with unit gradient g adds w(d) - (w(d) / d) |g x d| to the output s - d for every tap
// d = (i, j) of the disc with g . d < 0.  For the opposite tap -d the weight, the distance and
// |g x d| are the same and g . (-d) has the other sign: the term is computed once and goes to
// exactly one of the outputs s - d and s + d.  One cross product, one weighted difference, one
// comparison and two predicated additions serve two taps (5 issue slots instead of the 8 that two
// independent taps take).  So here threads own sources and scatter into their outputs:
//
//  * A warp owns a strip of 32 source columns, one lane per column, and walks it downwards in
//    blocks of K rows (12 up to radius 8, 8 above) whose unit gradients it holds in registers.
//  * For each column distance i the lane adds its terms to two columns of outputs, at X - i (tile P,
//    taps (i, j)) and X + i (tile M, the opposite taps), held in registers over all K sources x
//    2J + 1 row distances: K + 2J rows each, read from and written back to shared memory once per
//    i, four rows at a time.  The lane's two columns move by one with each i, so lanes pass the
//    columns on through shared memory; tiles P and M are separate, so that both are loaded before
//    the taps and no lane waits for another's half.  The columns of a tile are an odd number of
//    16-byte chunks apart: a warp's 128-bit accesses are free of bank conflicts.
//  * After each block the tiles' first K rows are complete for this strip's sources: they are written out
//    and the other rows move up, in 4-row chunks.
//  * Outputs within R + 1 columns of a strip's edge also receive terms from the neighbouring strip's
//    sources.  Each strip writes its own 32 columns to the plane `own` and the rest to the plane
//    `edge` (every element of it has one writer); the reader adds the two.
// Taps without a partner in the box [-R, R + 1] (column or row R + 1) go through the same code with
// one of the two additions left out.
//
// Bound: instruction issue.  512 x 512 frames at M4, radius 1.5 (254 taps), 34 a launch: 1.176e8 warp
// instructions per frame (the fused tile kernel, fht_fused.cuh: 2.214e8), 0.78 issued per cycle and
// scheduler, 5.02 ms against 8.25; the cumulants (rgc_pair.cu) take 0.35 ms more.  What the split is
// made of, each measured on that launch:
//  * 12 source rows a block up to radius 8 (8: 6 % slower, more loads of the tiles; 16: 10 %, spills);
//    8 above it, where the registers hold no more.
//  * 16 warps a CTA that start each block together: the chords' code (about 60 KB) does not fit the
//    instruction caches, and warps that drift apart in it fetch it one by one (one warp a CTA: 42 %
//    slower; 8: 15 %; together at each column distance instead of each block: 5 %, they then all
//    wait for shared memory at once).  Wide boxes have longer chords and take every third distance.
//  * the next block's source rows prefetched into L1 while a block's taps run (8 %).
// Packing two cross products into one f32x2 instruction makes the code longer, not shorter (register
// pairs for the constants).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "esrrf_internal.h"


namespace esrrf {
namespace pair {

constexpr int kStrip = 32;  // source columns of a strip
constexpr int kMaxR = 15;   // tap boxes up to 32 wide

constexpr int floor4(int x) { return (x >= 0 ? x : x - 3) / 4; }

template <int R>
struct PairLayout {
    static constexpr int K = R <= 8 ? 12 : 8;             // source rows of a block
    static constexpr int CH = 4 * ((R + 1 + 3) / 4);      // rows of the tiles above the block's first row
    static constexpr int HI = 4 * ((K + R + 3) / 4);      // and from it on
    static constexpr int NC = (CH + HI) / 4;              // 4-row chunks of a column
    static constexpr int ST = 4 * (NC | 1);               // floats from one column to the next
    static constexpr int NJ = (R + 3) & ~1;               // weights of one column distance: |j| = 0 .. R + 1
    static constexpr int cols = kStrip + R + 1;           // columns of a tile
    static constexpr size_t warp_bytes = sizeof(float) * 2 * cols * ST, table_bytes = sizeof(float2) * (R + 2) * NJ;
    // warps of a CTA at most: the registers of the taps (128, above radius 12 168 a thread)
    static constexpr int max_warps = R <= 12 ? 16 : 12;
};

struct PairArgs {
    const float* interp;  // [F][H][W]
    const float2* wt;     // [R + 2][NJ] (w, w / d) of tap (i, |j|)
    float* own;           // [F][H][W]
    float* edge;          // [F][H][W]
    int W, H, F;
    int strips;           // strips of a frame
    int rows, segs;       // the first `segs` row segments have `rows` output rows, the last (if any) the rest
    signed char J[kMaxR + 3];     // per column distance: largest |j| <= R of the disc (-1: none)
    unsigned char far[kMaxR + 3]; // per column distance: 1 if row distance R + 1 is in the disc
};

// Inward test of the taps (fi, j) of one source as a threshold in j: g . (fi, j) < 0 is
// j < -fi gx / gy for gy > 0 and the reverse for gy < 0 (approximate reciprocal, whose error moves
// the threshold within rounding of g . d = 0, where the term w - (w / d) |g x d| vanishes).
struct Inward {
    float q;
    bool neg;
    __device__ __forceinline__ Inward(float gx, float gy, float fi) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(gy));
        q = -(gx * r) * fi;
        neg = gy < 0.f;
    }
    __device__ __forceinline__ bool operator()(float j) const { return (j < q) != neg; }
};

__device__ __forceinline__ void load4(float* d, const float* s) {
    const float4 v = *reinterpret_cast<const float4*>(s);
    d[0] = v.x, d[1] = v.y, d[2] = v.z, d[3] = v.w;
}
__device__ __forceinline__ void store4(float* d, const float* s) {
    *reinterpret_cast<float4*>(d) = make_float4(s[0], s[1], s[2], s[3]);
}

// A warp-uniform flag tested once per source without a second copy of the unrolled code around it
// (the compiler would otherwise hoist the test and double the code).
__device__ __forceinline__ bool opaque(bool f) {
    int v = f;
    asm volatile("" : "+r"(v));
    return v != 0;
}

// (w, w / d) of |j| = 0 .. J of one column distance.
template <int J>
__device__ __forceinline__ void load_weights(const float2* __restrict__ wt, float (&w)[J + 2], float (&wd)[J + 2]) {
    const float4* w4 = reinterpret_cast<const float4*>(wt);
#pragma unroll
    for (int q = 0; q < (J + 2) / 2; ++q) {
        const float4 v = w4[q];
        w[2 * q] = v.x, wd[2 * q] = v.y, w[2 * q + 1] = v.z, wd[2 * q + 1] = v.w;
    }
}

// Row distance R + 1 at column distance i, source y of the block: the tap (i, R + 1) into P and
// (-i, R + 1) into M (both: 0 < i <= R), R + 1 rows above the source.  p, m: rows lo .. of the two
// columns, in registers; P, M: their row lo in the tiles.  For y = 0 the output may be the row above.
template <int R>
__device__ __forceinline__ void pair_far(int y, float* __restrict__ P, float* __restrict__ M, float* p, float* m,
                                         float2 wt, float fi, float gx, float gy, bool both) {
    constexpr int j = R + 1, lo = 4 * floor4(-R);
    const float gi = gx * fi, b = gy * fi;
    const float tp = fmaf(-fabsf(fmaf(gx, -(float)j, b)), wt.y, wt.x);
    const float tm = fmaf(-fabsf(fmaf(gx, (float)j, b)), wt.y, wt.x);
    const bool ip = fmaf(gy, (float)j, gi) < 0.f, im = both && fmaf(gy, (float)j, -gi) < 0.f;
    if (y - j < lo) {
        if (ip) P[-1] += tp;
        if (im) M[-1] += tm;
    } else {
        if (ip) p[y - j - lo] += tp;
        if (im) m[y - j - lo] += tm;
    }
}

// Column distance i = fi > 0 whose chord is the rows -J .. J: K sources x (2J + 1) pairs of taps.
// P, M: the lane's output columns at X - i and X + i.  one: the opposite taps lie outside the box
// (i = R + 1), only P is kept.  CHECK: some lane of the warp has a source in the image's columns without
// gradient, whose taps contribute nothing.  (A lane right of the image needs no check: its threshold is NaN, so
// its terms all go to its column of M, right of the image too, which is not written out.  The last strip of
// most frames has such lanes; with the check its warp ran another copy of the code than the rest of its CTA, and
// they waited for each other: 6 frames of 36 x 1576 196 us, 118 without, those of 64 x 1576 114; 34 of
// 1495 x 1015 at radius 10 3.89 ms and 3.77.)  A chunk is loaded one source before the first that reaches
// it and stored after the last.
template <int R, int J, bool CHECK>
__device__ __forceinline__ void pair_column(float* __restrict__ P, float* __restrict__ M,
                                            const float2* __restrict__ wt, float fi, const float (&gx)[PairLayout<R>::K],
                                            const float (&gy)[PairLayout<R>::K], bool one, bool far) {
    using L = PairLayout<R>;
    constexpr int K = L::K, c0 = floor4(-J), c1 = floor4(K - 1 + J), n = c1 - c0 + 1, lo = 4 * c0;
    P += L::CH + lo;  // row lo of the block
    M += L::CH + lo;
    float p[4 * n], m[4 * n], w[J + 2], wd[J + 2];
    constexpr bool FAR = J == R;
    load_weights<J>(wt, w, wd);
#pragma unroll
    for (int y = 0; y < K; ++y) {
#pragma unroll
        for (int c = 0; c < n; ++c) {
            const int first = lo + 4 * c - J - 1;
            if (y == (first > 0 ? first : 0)) {
                load4(p + 4 * c, P + 4 * c);
                load4(m + 4 * c, M + 4 * c);
            }
        }
        if (!(CHECK && gx[y] == 0.f && gy[y] == 0.f)) {
            const float b = gy[y] * fi;
            const Inward in(gx[y], gy[y], fi);
#pragma unroll
            for (int j = -J; j <= J; ++j) {
                const int a = j < 0 ? -j : j;
                const float c = j == 0 ? b : fmaf(gx[y], -(float)j, b);
                const float t = fmaf(-fabsf(c), wd[a], w[a]);
                if (in((float)j))
                    p[y - j - lo] += t;
                else
                    m[y + j - lo] += t;
            }
        }
        if (FAR && opaque(far)) pair_far<R>(y, P, M, p, m, wt[R + 1], fi, gx[y], gy[y], !one);
#pragma unroll
        for (int c = 0; c < n; ++c)
            if (y == min(K - 1, lo + 4 * c + 3 + J + (FAR ? 1 : 0))) {
                store4(P + 4 * c, p + 4 * c);
                if (!one) store4(M + 4 * c, m + 4 * c);
            }
    }
}

template <int R, int J, bool CHECK>
__device__ __forceinline__ void pair_dispatch(int j, float* __restrict__ P, float* __restrict__ M,
                                              const float2* __restrict__ wt, float fi, const float (&gx)[PairLayout<R>::K],
                                              const float (&gy)[PairLayout<R>::K], bool one, bool far) {
    if constexpr (J >= 0) {
        if (j == J) {
            pair_column<R, J, CHECK>(P, M, wt, fi, gx, gy, one, far);
            return;
        }
        pair_dispatch<R, J - 1, CHECK>(j, P, M, wt, fi, gx, gy, one, far);
    }
}

// Column distance 0: the pairs (0, j) and (0, -j), j = 1 .. R, one output column (gy < 0: inward for
// j > 0); the rows of the box are always in the disc (its radius is at least R).
template <int R, bool CHECK>
__device__ __forceinline__ void pair_zero(float* __restrict__ P, const float2* __restrict__ wt,
                                          const float (&gx)[PairLayout<R>::K], const float (&gy)[PairLayout<R>::K],
                                          bool far) {
    using L = PairLayout<R>;
    constexpr int K = L::K, c0 = floor4(-R), c1 = floor4(K - 1 + R), n = c1 - c0 + 1, lo = 4 * c0;
    P += L::CH + lo;
    float p[4 * n], w[R + 2], wd[R + 2];
#pragma unroll
    for (int c = 0; c < n; ++c) load4(p + 4 * c, P + 4 * c);
    load_weights<R>(wt, w, wd);
#pragma unroll
    for (int y = 0; y < K; ++y) {
        const bool neg = gy[y] < 0.f, none = CHECK && gx[y] == 0.f && gy[y] == 0.f;
#pragma unroll
        for (int j = 1; j <= R; ++j) {
            const float t = fmaf(-fabsf(gx[y] * (float)j), wd[j], w[j]);
            if (neg)
                p[y - j - lo] += t;
            else if (!none)
                p[y + j - lo] += t;
        }
        if (opaque(far)) pair_far<R>(y, P, P, p, p, wt[R + 1], 0.f, gx[y], gy[y], false);
    }
#pragma unroll
    for (int c = 0; c < n; ++c) store4(P + 4 * c, p + 4 * c);
}

// The warps of a CTA stay together (once a block; every third column distance in the wide boxes): a
// chord's code is long and straight, and warps at different places of it would each fetch it for
// themselves.
__device__ __forceinline__ void cta_step() { asm volatile("bar.sync 0;" ::: "memory"); }
template <int R>
__device__ __forceinline__ bool together(int i) {
    return R <= 8 ? i == 1 : i % 3 == 1;
}

// All taps of a block of K source rows.
template <int R, bool CHECK>
__device__ __forceinline__ void pair_block(const PairArgs& a, float* __restrict__ sP, float* __restrict__ sM,
                                           const float2* __restrict__ swt, int lane, const float (&gx)[PairLayout<R>::K],
                                           const float (&gy)[PairLayout<R>::K]) {
    using L = PairLayout<R>;
    float* P = sP + (R + 1 + lane) * L::ST;  // tile P starts at column X0 - R - 1, tile M at X0
    float* M = sM + lane * L::ST;
    pair_zero<R, CHECK>(P, swt, gx, gy, a.far[0] != 0);
    __syncwarp();
#pragma unroll 1
    for (int i = 1; i <= R + 1; ++i) {
        const int J = a.J[i];
        if (J < 0) break;
        P -= L::ST;
        M += L::ST;
        if (together<R>(i)) cta_step();
        pair_dispatch<R, R, CHECK>(J, P, M, swt + i * L::NJ, (float)i, gx, gy, i == R + 1, a.far[i] != 0);
        __syncwarp();
    }
}

// The steps of a block without taps.
template <int R>
__device__ __forceinline__ void pair_block_none(const PairArgs& a) {
#pragma unroll 1
    for (int i = 1; i <= R + 1; ++i) {
        if (a.J[i] < 0) break;
        if (together<R>(i)) cta_step();
    }
}

// One warp per (strip, frame) and row segment (blockIdx.y).
template <int R>
__global__ void __launch_bounds__(32 * PairLayout<R>::max_warps, 1) fht_rgc_pair_kernel(const __grid_constant__ PairArgs a) {
    using L = PairLayout<R>;
    extern __shared__ __align__(16) unsigned char smem[];
    float2* swt = reinterpret_cast<float2*>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* sP = reinterpret_cast<float*>(smem + L::table_bytes + warp * L::warp_bytes);
    float* sM = sP + L::cols * L::ST;
    constexpr int K = L::K;
    const int W = a.W, H = a.H;
    const int unit = blockIdx.x * (blockDim.x >> 5) + warp;  // strip fastest
    const bool work = unit < a.strips * a.F;
    const int frame = work ? unit / a.strips : 0;
    const int X0 = (unit - frame * a.strips) * kStrip, X = X0 + lane;
    const int ya = blockIdx.y * a.rows, yb = (int)blockIdx.y < a.segs ? min(H, ya + a.rows) : H;  // output rows
    const size_t plane = (size_t)W * H;
    const float* __restrict__ img = a.interp + frame * plane;
    float* __restrict__ own = a.own + frame * plane;
    float* __restrict__ edge = a.edge + frame * plane;

    for (int q = threadIdx.x; q < (R + 2) * L::NJ; q += blockDim.x) swt[q] = a.wt[q];
    for (int q = lane; q < 2 * L::cols * L::ST / 4; q += 32)
        reinterpret_cast<float4*>(sP)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();

    // columns of the Roberts cross, with the reference's clamps
    const bool in = work && X < W;
    const int xc = min(X, W - 1), xl = max(xc - 1, 0), xr = min(xc + 1, W - 1);
    const bool last = X == W - 1;
    // the halo columns this lane writes: left of the strip from tile P, right of it from tile M
    const bool eleft = lane <= R, eright = lane >= 32 - R;
    const int xe = eleft ? X0 - R - 1 + lane : X0 + R + lane;
    const float* ecol = eleft ? sP + lane * L::ST : sM + (lane + R) * L::ST;
    const bool ein = work && (eleft || eright) && xe >= 0 && xe < W;

    const int ylast = min(H - 1, yb + R);  // last source row that reaches the segment
#pragma unroll 1
    for (int Y0 = max(0, ya - R);; Y0 += K) {
        if (Y0 <= ylast) {
            // unit gradient at each tap source: Gx read at min(X + 1, W - 1), Gy at min(Y + 1, H - 1),
            // Roberts cross with max(. - 1, 0) clamps (liveSRRF_noInterpolation.cl:144-155, 291-292)
            float gx[K], gy[K];
            bool some = false, none = false;
            auto row = [&](int y) { return img + (size_t)min(max(y, 0), H - 1) * W; };
            const float* r = row(Y0 - 1);
            float al = __ldg(r + xl), ac = __ldg(r + xc), ar = __ldg(r + xr);
            r = row(Y0);
            float bl = __ldg(r + xl), bc = __ldg(r + xc), br = __ldg(r + xr);
#pragma unroll
            for (int y = 0; y < K; ++y) {
                const int Y = Y0 + y;
                r = row(Y + 1);
                const float cl = __ldg(r + xl), cc = __ldg(r + xc), cr = __ldg(r + xr);
                // rows Y - 1, Y, Y + 1 in a, b, c; at the last column the cross's left column is xl,
                // at the last row its upper row is Y - 1
                const float Gx = ar - (last ? bl : bc) + br - (last ? al : ac);
                const bool bot = Y == H - 1;
                const float uc = bot ? ac : bc, ul = bot ? al : bl;
                const float Gy = -uc + cl + cc - ul;
                const float n2 = Gx * Gx + Gy * Gy;
                const bool ok = in && Y < H && n2 > 0.f && n2 <= 3.402823466e38f;  // no gradient, or one beyond FP32: none
                const float inv = ok ? rsqrtf(n2) : 0.f;
                gx[y] = ok ? Gx * inv : 0.f;
                gy[y] = ok ? Gy * inv + 0.f : 0.f;  // + 0: -0 becomes +0
                const bool zero = gx[y] == 0.f && gy[y] == 0.f;
                some |= !zero;
                none |= zero && in;  // a lane right of the image: pair_column
                al = bl, ac = bc, ar = br;
                bl = cl, bc = cc, br = cr;
            }
            // the next block's rows into L1 while this block's taps run
            for (int y = Y0 + K + 1; y <= Y0 + 2 * K; ++y) asm volatile("prefetch.global.L1 [%0];" ::"l"(row(y) + xc));
            if (__any_sync(0xffffffffu, none || !work)) {  // a warp without work: none of its sources has a gradient
                if (__any_sync(0xffffffffu, some))
                    pair_block<R, true>(a, sP, sM, swt, lane, gx, gy);
                else
                    pair_block_none<R>(a);
            } else {
                pair_block<R, false>(a, sP, sM, swt, lane, gx, gy);
            }
        }
        // the first K rows (Y0 - CH ..) are complete: write them, move the others up and clear theirs
#pragma unroll
        for (int k = 0; k < K / 4; ++k) {
            const int o = 4 * k, y = Y0 - L::CH + o;
            float vp[4], vm[4], ve[4];
            load4(vp, sP + (R + 1 + lane) * L::ST + o);
            load4(vm, sM + lane * L::ST + o);
            load4(ve, ecol + o);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (y + q >= ya && y + q < yb) {
                    if (in) own[(size_t)(y + q) * W + X] = vp[q] + vm[q];
                    if (ein) edge[(size_t)(y + q) * W + xe] = ve[q];
                }
        }
        __syncwarp();
        for (int q = lane; q < 2 * L::cols; q += 32) {
            float4* col = reinterpret_cast<float4*>(sP + q * L::ST);
#pragma unroll
            for (int k = 0; k < L::NC - K / 4; ++k) col[k] = col[k + K / 4];
#pragma unroll
            for (int k = L::NC - K / 4; k < L::NC; ++k) col[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        if (Y0 - L::CH + K >= yb) break;
    }
}

// Launch of the tap boxes RLO .. RHI; warps of a CTA and row segments by pair_shape.
template <int RLO, int RHI>
cudaError_t launch_pair_in(int R, const PairArgs& a, int warps, cudaStream_t stream) {
    if (R == RLO) {
        using L = PairLayout<RLO>;
        static unsigned long long configured = 0;  // per device: the shared-memory attribute is set
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev >= 64 || !(configured & (1ull << dev))) {
            e = cudaFuncSetAttribute(fht_rgc_pair_kernel<RLO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(L::table_bytes + L::max_warps * L::warp_bytes));
            if (e != cudaSuccess) return e;
            if (dev < 64) configured |= 1ull << dev;
        }
        const dim3 grid((a.strips * a.F + warps - 1) / warps, a.segs + (a.segs * a.rows < a.H ? 1 : 0));
        fht_rgc_pair_kernel<RLO><<<grid, 32 * warps, L::table_bytes + warps * L::warp_bytes, stream>>>(a);
        return cudaGetLastError();
    }
    if constexpr (RLO < RHI) return launch_pair_in<RLO + 1, RHI>(R, a, warps, stream);
    return cudaErrorInvalidValue;
}

}  // namespace pair
}  // namespace esrrf
