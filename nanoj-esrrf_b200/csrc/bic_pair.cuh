// bic_pair.cuh -- radial gradient convergence of the 2-D bicubic path without drift
// (liveSRRF.cl:238-401), two opposite taps at a time.
//
// The taps are nodes of the 2x gradient grid: node n lies at n M / 2 output pixels, output xM at
// xM + 0.5, so a node is a point of symmetry of the output grid and the argument of rgc_pair.cuh
// holds: the term w(d) - (w(d) / d) |g x d| of a node goes to exactly one of the outputs s - d and
// s + d.  A warp owns a strip of 32 node columns, one lane each, walks it in blocks of 8 node rows
// and scatters into its outputs, for every column distance into the columns on both sides.  What
// differs from rgc_pair.cuh:
//  * With M even every node is half an output pixel from the nearest outputs: the distances are half-odd,
//    dx = i - 1/2 and dy = j - 1/2, and no column or row is its own opposite.  (With M odd half-odd and
//    whole distances alternate from node to node; those magnifications keep the tabulated kernel.)
//  * The disc lies inside the reference's box for every radius: there are no taps without a partner.
//  * Nodes are M / 2 output pixels apart, so 8 node rows reach 4 M + 2 J output rows.  Both columns of a
//    distance live in one tile (two would leave too few warps an SM): the left one is held in
//    registers from its load to its store, the right one summed from zero and added to the tile
//    once the left one's chunk is stored, chunk by chunk as the rows go by.
//
// Bound: instruction issue.  512 x 512 at M4, radius 1.5 (64 taps an output, 130 pairs a node): 3.5e7 warp
// instructions a frame, 0.64 issued per cycle and scheduler (the tabulated kernel, one tap at a time
// per output: 1.50e8), 1.62 ms per 32 frames against 5.8.  Stalls: the tile's loads (short scoreboard
// 0.73 per issue), the nodes and the spills of the longest chords (long scoreboard 1.07).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "esrrf_internal.h"

namespace esrrf {
namespace bicpair {

constexpr int kK = 8;      // node rows of a block
constexpr int kMaxJ = 15;  // row and column distances up to 15 output pixels
constexpr int kNJ = 16;    // weights of one column distance: row distances 0 .. 15

__host__ __device__ constexpr int floor4(int x) { return (x >= 0 ? x : x - 3) / 4; }

struct BicPairArgs {
    const float2* U;      // [F][2h][2w] unit gradient at the nodes (node 0: none)
    const float4* wt;     // [I + 1][kNJ / 2] pairs of (w, w / d) of the distances (i - 1/2, j - 1/2)
    float* own;           // [F][H][W] output pixels
    float* edge;          // [F][H][W]
    int W, H, F, w2, h2;  // output size, node grid size
    int strips, rows, segs;  // strips of a frame; `segs` segments of `rows` output rows and the rest
    int I;                // largest column distance (and the halo of a strip)
    int CH, NC;           // rows of the tile above the block's first row; 4-row chunks of a column
    int halo, cps;        // columns left of the strip; columns of a sub-tile
    signed char J[kMaxJ + 1];  // per column distance: largest row distance
};

template <int M>
struct Geo {
    static_assert(M % 2 == 0, "half-odd distances");
    static constexpr int h = M / 2;                   // output pixels from node to node; sub-tiles of a tile
    static constexpr int SW = 16 * M;                 // output columns of a strip
    static constexpr int row(int y) { return y * h; }  // output row of node row y of a block
};

__host__ __device__ inline int tile_stride(const BicPairArgs& a) { return 4 * (a.NC | 1); }
__host__ __device__ inline size_t warp_bytes(const BicPairArgs& a, int h) {
    // the tile and the next block's nodes
    return sizeof(float) * (size_t)h * a.cps * tile_stride(a) + sizeof(float2) * 32 * kK;
}
__host__ __device__ inline size_t table_bytes(const BicPairArgs& a) {
    return sizeof(float4) * (a.I + 1) * (kNJ / 2);
}

__device__ __forceinline__ void load4(float* d, const float* s) {
    const float4 v = *reinterpret_cast<const float4*>(s);
    d[0] = v.x, d[1] = v.y, d[2] = v.z, d[3] = v.w;
}
__device__ __forceinline__ void store4(float* d, const float* s) {
    *reinterpret_cast<float4*>(d) = make_float4(s[0], s[1], s[2], s[3]);
}

// Column distance dx whose chord reaches J rows: 8 nodes x 2J pairs.  P, Q: row 0 of the block in the
// lane's columns left and right of the node.
template <int M, int J>
__device__ __forceinline__ void pass(float* __restrict__ P, float* __restrict__ Q, const float4* __restrict__ wt,
                                     float dx, const float (&gx)[kK], const float (&gy)[kK]) {
    using G = Geo<M>;
    // the rows of a node: o - J .. o + J - 1
    constexpr int c0 = floor4(-J), c1 = floor4(G::row(kK - 1) + J - 1), n = c1 - c0 + 1, lo = 4 * c0;
    P += lo;
    Q += lo;
    float p[4 * n], q[4 * n], w[J + 2], wd[J + 2];
#pragma unroll
    for (int k = 0; k < 4 * n; ++k) q[k] = 0.f;
#pragma unroll
    for (int k = 0; k < (J + 2) / 2; ++k) {
        const float4 v = wt[k];
        w[2 * k] = v.x, wd[2 * k] = v.y, w[2 * k + 1] = v.z, wd[2 * k + 1] = v.w;
    }
#pragma unroll
    for (int y = 0; y < kK; ++y) {
        const int o = G::row(y), next = G::row(y < kK - 1 ? y + 1 : y);
#pragma unroll
        for (int c = 0; c < n; ++c)  // loaded one node row before the first that reaches it
            if (lo + 4 * c < next + J && (y == 0 || lo + 4 * c >= o + J)) load4(p + 4 * c, P + 4 * c);
        if (!(gx[y] == 0.f && gy[y] == 0.f)) {
            const float b = gy[y] * dx;
            float r;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(gy[y]));
            const float thr = -(gx[y] * r) * dx;  // inward: dy < thr for gy > 0, the reverse for gy < 0
            const bool neg = gy[y] < 0.f;
#pragma unroll
            for (int j = 1; j <= J; ++j) {
                const float dy = (float)j - 0.5f;
                const float t = fmaf(-fabsf(fmaf(gx[y], -dy, b)), wd[j], w[j]);
                const float u = fmaf(-fabsf(fmaf(gx[y], dy, b)), wd[j], w[j]);
                const int ra = o - j - lo, rb = o + j - 1 - lo;
                if ((dy < thr) != neg)
                    p[ra] += t;
                else
                    q[rb] += t;
                if ((-dy < thr) != neg)
                    p[rb] += u;
                else
                    q[ra] += u;
            }
        }
#pragma unroll
        for (int c = 0; c < n; ++c) {  // chunks that no later node row reaches
            const int end = lo + 4 * c + 4;
            if ((y == kK - 1 || end <= next - J) && (y == 0 || end > o - J)) {
                store4(P + 4 * c, p + 4 * c);
                __syncwarp();
                float old[4];
                load4(old, Q + 4 * c);
#pragma unroll
                for (int k = 0; k < 4; ++k) old[k] += q[4 * c + k];
                store4(Q + 4 * c, old);
            }
        }
    }
    __syncwarp();
}

template <int M, int J>
__device__ __forceinline__ void dispatch(int j, float* __restrict__ P, float* __restrict__ Q,
                                         const float4* __restrict__ wt, float dx, const float (&gx)[kK],
                                         const float (&gy)[kK]) {
    if constexpr (J >= 1) {
        if (j == J) {
            pass<M, J>(P, Q, wt, dx, gx, gy);
            return;
        }
        dispatch<M, J - 1>(j, P, Q, wt, dx, gx, gy);
    }
}

// One warp per (strip, frame) and row segment (blockIdx.y).
template <int M>
__global__ void __launch_bounds__(512, 1) bic_pair_kernel(const __grid_constant__ BicPairArgs a) {
    using G = Geo<M>;
    constexpr int B = 4 * M;  // output rows of a block
    extern __shared__ __align__(16) unsigned char smem[];
    float4* swt = reinterpret_cast<float4*>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ST = tile_stride(a);
    float* tile = reinterpret_cast<float*>(smem + table_bytes(a) + warp * warp_bytes(a, G::h));
    float2* snode = reinterpret_cast<float2*>(tile + G::h * a.cps * ST) + lane;  // this lane's nodes, 32 apart
    const int unit = blockIdx.x * (blockDim.x >> 5) + warp;  // strip fastest
    const bool work = unit < a.strips * a.F;
    const int frame = work ? unit / a.strips : 0;
    const int strip = work ? unit - frame * a.strips : 0;
    const int n = 32 * strip + lane;   // this lane's node column
    const int X0 = G::SW * strip;      // the strip's first output column
    const int ya = blockIdx.y * a.rows, yb = (int)blockIdx.y < a.segs ? min(a.H, ya + a.rows) : a.H;
    const float2* __restrict__ U = a.U + (size_t)frame * a.w2 * a.h2;
    float* __restrict__ own = a.own + (size_t)frame * a.W * a.H;
    float* __restrict__ edge = a.edge + (size_t)frame * a.W * a.H;

    for (int q = threadIdx.x; q < (a.I + 1) * (kNJ / 2); q += blockDim.x) swt[q] = a.wt[q];
    const int nt = G::h * a.cps * ST / 4;
    for (int q = lane; q < nt; q += 32) reinterpret_cast<float4*>(tile)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // a column of the strip's tile (0: `halo` columns left of the strip), row -CH
    auto column = [&](int c) { return tile + ((c % G::h) * a.cps + c / G::h) * ST; };

    const bool in = work && n < a.w2;
    const int xl = a.halo + lane * G::h;  // the first column right of the node, in the tile
    // the first block whose rows reach the segment, in whole blocks of the frame
    const int first = max(0, (ya - a.I) / B), nlast = min(a.h2 - 1, (yb + a.I) / G::h + 1);
    // a block's nodes are copied to shared memory while the block before runs (each lane its own; rows
    // beyond the grid as zeros): loaded when needed they were the largest stall, and 16 warps' rows do
    // not fit the L1 cache that the tiles leave
    auto fetch = [&](int N0) {
#pragma unroll
        for (int y = 0; y < kK; ++y) {
            const bool ok = in && N0 + y < a.h2;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(snode + 32 * y)),
                         "l"(ok ? U + (size_t)(N0 + y) * a.w2 + n : U), "r"(ok ? 8 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(first * kK);
#pragma unroll 1
    for (int blk = first;; ++blk) {
        const int N0 = blk * kK, Y0 = blk * B;  // first node row and its output row
        if (N0 <= nlast) {
            float gx[kK], gy[kK];
            bool some = false;
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
            for (int y = 0; y < kK; ++y) {
                const float2 g = snode[32 * y];
                gx[y] = g.x;
                gy[y] = g.y;
                some |= g.x != 0.f || g.y != 0.f;
            }
            if (N0 + kK <= nlast) fetch(N0 + kK);
            // the warps of a CTA start a block together: they share the fetches of the long code
            asm volatile("bar.sync 0;" ::: "memory");
            if (__any_sync(0xffffffffu, some)) {
#pragma unroll 1
                for (int i = 1; i <= a.I; ++i)
                    dispatch<M, kMaxJ>(a.J[i], column(xl - i) + a.CH, column(xl + i - 1) + a.CH,
                                       swt + i * (kNJ / 2), (float)i - 0.5f, gx, gy);
            }
        }
        // the first B rows (Y0 - CH ..) are complete: write them, move the others up and clear theirs
        for (int c = lane; c < G::SW + 2 * a.I; c += 32) {
            const float* col = column(c + a.halo - a.I);
            const int x = X0 + c - a.I;
            const bool mine = c >= a.I && c < a.I + G::SW;
            if (!work || x < 0 || x >= a.W) continue;
            float* dst = mine ? own : edge;
#pragma unroll
            for (int k = 0; k < M; ++k) {
                float v[4];
                load4(v, col + 4 * k);
                const int y = Y0 - a.CH + 4 * k;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (y + q >= ya && y + q < yb) dst[(size_t)(y + q) * a.W + x] = v[q];
            }
        }
        __syncwarp();
        for (int q = lane; q < G::h * a.cps; q += 32) {
            float4* col = reinterpret_cast<float4*>(tile + q * ST);
            for (int k = 0; k < a.NC - M; ++k) col[k] = col[k + M];
            for (int k = a.NC - M; k < a.NC; ++k) col[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        if (Y0 - a.CH + B >= yb) break;
    }
}

template <int M>
cudaError_t launch(const BicPairArgs& a, int warps, cudaStream_t stream) {
    const size_t wb = warp_bytes(a, Geo<M>::h), tb = table_bytes(a);
    static unsigned long long configured = 0;  // per device: the shared-memory attribute is set
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(configured & (1ull << dev))) {
        e = cudaFuncSetAttribute(bic_pair_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        if (dev < 64) configured |= 1ull << dev;
    }
    const dim3 grid((a.strips * a.F + warps - 1) / warps, a.segs + (a.segs * a.rows < a.H ? 1 : 0));
    bic_pair_kernel<M><<<grid, 32 * warps, tb + warps * wb, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace bicpair

}  // namespace esrrf
