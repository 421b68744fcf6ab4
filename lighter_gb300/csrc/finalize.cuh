// The finalize step of a lightmap in one pass over its texels: three
// extrapolating dilation sweeps, then the separable Gaussian blur
// (lighter.cpp:880-961), for the bake (bake.cu) and for the entry point on
// caller-owned buffers (noalloc.cu).
//
// As separate kernels (scatter, three mask copies and sweeps, two transposed
// convolutions) the step was bound by launches on one lightmap and by eight
// passes over memory on many. Here a block owns 32 x 32 texels and reads them
// once with a halo of 6 + ext texels (a sweep looks two texels out, the blur
// ext): sweeps and both convolutions run in shared memory, and the tile is
// written once. The halo re-reads 2.1x the texels, from L2. One lightmap is a
// block or two per SM, so a block's own chain of latencies is the time: 512
// threads, five texels per thread read at once (the whole region up to ext = 3), and
// the sweeps go through a list of the uncovered texels, so all lanes have one.
// Measured: 512 x 512 at blur 0.5 11.0 us on the device and 12.4 us a call (13.3 and 16.4
// with every thread looking after its own texels, 30.9 and 53.6 as separate
// kernels), 1024 x 1024 30.8 us (33.8; 90.5); 256 threads 14.1 us at 512 x 512, 384
// 11.7, 1024 11.0 but 32.3 at 1024 x 1024. A bake's stage on four 1024^2 lightmaps took
// 0.34 ms as separate kernels, 0.155 with the first form of this and 0.140 now. The float
// expressions and their order are those of the separate kernels, so the
// results are the same bits.
#pragma once

#include "common.cuh"

namespace lg {

constexpr int kFinTile = 32, kFinThreads = 512;
constexpr int kFinMaxExt = 16;   // largest ceil(blur_size) the tile's shared memory is laid out for

struct FinTaps { float k[2 * kFinMaxExt + 1]; };

// Region side (tile + halo) and shared memory: colours, masks, the rows of the
// first convolution, and the list of uncovered texels.
inline __host__ __device__ int fin_side(int ext) { return kFinTile + 2 * (6 + ext); }
inline size_t fin_smem(int ext)
{
    const size_t s = (size_t) fin_side(ext);
    return s * s * 12 + (s * s + 15) / 16 * 16 + (ext ? (size_t) kFinTile * (kFinTile + 2 * ext) * 12 : 0) + s * s * 2;
}

#ifdef __CUDACC__

// Lets `kernel` be launched with any halo's shared memory. The limit belongs to the kernel,
// not to a launch, so it is always the largest: set to one call's size, it could
// drop between another thread's setting and its launch, which would then be refused.
template <class K>
inline cudaError_t fin_allow_smem(K kernel)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) fin_smem(kFinMaxExt));
}

// One dilation of an unset texel from its set 4-neighbours, each extrapolated
// linearly (2 c1 - c2) when the next texel out is set too; `m` and `col` point
// at the texel in the region, `sweep` counts from 1, and a mask byte holds one
// more than the sweep that set its texel (0: unset, or outside the image).
// Returns whether the texel was set.
__device__ __forceinline__ bool fin_dilate(unsigned char* m, float* col, int side, int sweep)
{
    V3 c = mk(0, 0, 0);
    int cnt = 0;
    auto isset = [&](int o) { const int v = m[o]; return v != 0 && v <= sweep; };
    auto at = [&](int o) { return mk(col[3 * o], col[3 * o + 1], col[3 * o + 2]); };
    const int dir[4] = {-1, 1, -side, side};
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const int o = dir[d];
        if (isset(o)) {
            c += isset(2 * o) ? lerp3(at(2 * o), at(o), 2.0f) : at(o);
            cnt++;
        }
    }
    if (!cnt) return false;
    c = c / (float) cnt;
    col[0] = fmax_(c.x, 0.0f);
    col[1] = fmax_(c.y, 0.0f);
    col[2] = fmax_(c.z, 0.0f);
    m[0] = (unsigned char) (sweep + 1);
    return true;
}

// Tile (bx, by) of a w x h image. load(g, c[3]) returns whether texel g (row
// major) is covered and its colour; out receives the finished texels (row major,
// not read). Every thread of the block calls it.
template <class Load>
__device__ __forceinline__ void fin_tile(int bx, int by, int w, int h, int ext, const FinTaps& taps, Load&& load,
                                         float* __restrict__ out, unsigned char* smem)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kFinThreads / 32;
    const int halo = 6 + ext, side = fin_side(ext);
    float* col = reinterpret_cast<float*>(smem);
    unsigned char* msk = smem + (size_t) side * side * 12;
    float* tmp = reinterpret_cast<float*>(msk + (side * side + 15) / 16 * 16);
    unsigned short* list = reinterpret_cast<unsigned short*>(tmp + (ext ? kFinTile * (kFinTile + 2 * ext) * 3 : 0));
    __shared__ unsigned n_open;
    if (threadIdx.x == 0) n_open = 0;
    __syncthreads();
    const int x0 = bx * kFinTile - halo, y0 = by * kFinTile - halo;   // the region's corner
    const int n = side * side;
    // i / side for i < n: n < 2^13 and side < 2^7, so the rounded-up reciprocal of 20 bits is exact
    const unsigned rcp = (0xfffffu + (unsigned) side) / (unsigned) side;
    constexpr int kBatch = 5;   // up to ext = 3 one batch: one wait for memory
    for (int k0 = 0; k0 * kFinThreads < n; k0 += kBatch) {
        float c[kBatch][3];
        bool set[kBatch], open[kBatch];   // covered; uncovered, and within a sweep's reach
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int i = (int) threadIdx.x + (k0 + k) * kFinThreads;
            const int y = (int) ((unsigned) i * rcp >> 20), gx = x0 + i - y * side, gy = y0 + y;
            c[k][0] = c[k][1] = c[k][2] = 0.0f;
            set[k] = open[k] = false;
            if (i < n && gx >= 0 && gx < w && gy >= 0 && gy < h) {
                set[k] = load((size_t) gy * w + gx, c[k]);
                open[k] = !set[k] && i - y * side >= 2 && i - y * side < side - 2 && y >= 2 && y < side - 2;
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int i = (int) threadIdx.x + (k0 + k) * kFinThreads;
            if (i < n) {
                col[3 * i] = c[k][0]; col[3 * i + 1] = c[k][1]; col[3 * i + 2] = c[k][2];
                msk[i] = set[k] ? 1 : 0;
            }
            const unsigned who = __ballot_sync(0xffffffffu, open[k]);
            unsigned at = 0;
            if (who && lane == 0) at = atomicAdd(&n_open, (unsigned) __popc(who));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (open[k]) list[at + __popc(who & ((1u << lane) - 1u))] = (unsigned short) i;
        }
    }
    __syncthreads();
    const int opened = (int) n_open;   // texels of the image in the region that a sweep may set
    if (opened)
        for (int s = 1; s <= 3; ++s) {
            for (int e = (int) threadIdx.x; e < opened; e += kFinThreads) {
                const int i = list[e], y = (int) ((unsigned) i * rcp >> 20), x = i - y * side;
                if (msk[i] || x < 2 * s || y < 2 * s || x >= side - 2 * s || y >= side - 2 * s) continue;
                fin_dilate(msk + i, col + 3 * i, side, s);
            }
            __syncthreads();
        }
    const int tx = bx * kFinTile + lane;
    float* res = col;   // the finished tile: 32 rows of 96 floats
    int res_stride = 3 * kFinTile;
    if (ext) {
        if (tx < w)
            for (int r = warp; r < kFinTile + 2 * ext; r += kWarps) {   // rows, clamped at the image's edges
                const int gy = by * kFinTile - ext + r;
                if (gy < 0 || gy >= h) continue;
                const float* row = col + 3 * ((gy - y0) * side - x0);
                float s0 = 0, s1 = 0, s2 = 0;
                for (int i = -ext; i <= ext; ++i) {
                    int xx = tx + i;
                    xx = xx < 0 ? 0 : (xx >= w ? w - 1 : xx);
                    const float kq = taps.k[i + ext];
                    s0 += row[3 * xx + 0] * kq;
                    s1 += row[3 * xx + 1] * kq;
                    s2 += row[3 * xx + 2] * kq;
                }
                float* o = tmp + 3 * (r * kFinTile + lane);
                o[0] = s0; o[1] = s1; o[2] = s2;
            }
        __syncthreads();
        if (tx < w)
            for (int r = warp; r < kFinTile; r += kWarps) {   // columns
                const int gy = by * kFinTile + r;
                if (gy >= h) break;
                float s0 = 0, s1 = 0, s2 = 0;
                for (int i = -ext; i <= ext; ++i) {
                    int yy = gy + i;
                    yy = yy < 0 ? 0 : (yy >= h ? h - 1 : yy);
                    const float kq = taps.k[i + ext];
                    const float* q = tmp + 3 * ((yy - (by * kFinTile - ext)) * kFinTile + lane);
                    s0 += q[0] * kq;
                    s1 += q[1] * kq;
                    s2 += q[2] * kq;
                }
                float* o = col + 3 * (r * kFinTile + lane);   // the colours are no longer needed
                o[0] = s0; o[1] = s1; o[2] = s2;
            }
        __syncwarp();   // a warp writes out the rows it summed
    } else {
        res = col + 3 * (6 * side + 6);
        res_stride = 3 * side;
    }
    const int cols = 3 * min(kFinTile, w - bx * kFinTile);
    for (int r = warp; r < kFinTile; r += kWarps) {
        const int gy = by * kFinTile + r;
        if (gy >= h) break;
        float* o = out + 3 * ((size_t) gy * w + (size_t) bx * kFinTile);
        for (int c = lane; c < cols; c += 32) o[c] = res[r * res_stride + c];
    }
}

#endif  // __CUDACC__

}  // namespace lg
