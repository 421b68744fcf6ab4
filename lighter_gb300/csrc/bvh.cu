// GPU build of the flat scene BVH (layout in bvh.cuh).
//
// Replaces the reference's per-instance top-down AABBTree build
// (AABBTree::SetAABBs/_MakeNode, lighter_math.cpp:674-781) and its instance
// tree (lighter.cpp:1060-1069) with one linear BVH over all world-space
// shadow-casting triangles, built in five passes on the GPU:
//   1. 30-bit Morton code of each triangle centroid inside the scene bounds;
//   2. radix sort of (code, triangle) pairs;
//   3. Karras' (HPG 2012) top-down-by-prefix hierarchy, one thread per
//      internal node, ties between equal codes broken by index;
//   4. bottom-up box refit, one thread per leaf, second arrival at a node
//      computes its box (atomic arrival counters);
//   5. packing into 64-byte nodes that hold both child boxes, and
//      triangles reordered into leaf order.
// Pass 3 and 4 serve the radix builder, and a clustering tree too deep for the
// walks; the default hierarchy is locally-ordered clustering (below). Everything
// is queued on one stream without a host wait: what depends on a result (the
// fallback to the radix hierarchy, a failed clustering) is decided on the device.
// Leaves are triangle references: an oversized triangle may be split (on the
// host, bake.cu) into several references with clipped boxes, each holding the
// whole triangle, so every query still tests the original triangle.
#include <cuda_runtime.h>
#include <cub/cub.cuh>
#include <cfloat>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "bvh.cuh"

namespace lg {
namespace {

#define BVH_CHECK(x)                                                                                  \
    do {                                                                                              \
        cudaError_t e_ = (x);                                                                         \
        if (e_ != cudaSuccess) throw std::runtime_error(std::string("bvh: ") + cudaGetErrorString(e_)); \
    } while (0)

__device__ __forceinline__ u32 spread10(u32 v)
{
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__global__ void k_morton(const float* ref_box, int n, float3 mn, float3 inv_ext, u32* codes, u32* ids)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* b = ref_box + 6 * (size_t) i;
    float cx = (b[0] + b[3]) * 0.5f, cy = (b[1] + b[4]) * 0.5f, cz = (b[2] + b[5]) * 0.5f;
    float qx = fminf(fmaxf((cx - mn.x) * inv_ext.x * 1024.0f, 0.0f), 1023.0f);
    float qy = fminf(fmaxf((cy - mn.y) * inv_ext.y * 1024.0f, 0.0f), 1023.0f);
    float qz = fminf(fmaxf((cz - mn.z) * inv_ext.z * 1024.0f, 0.0f), 1023.0f);
    codes[i] = (spread10((u32) qx) << 2) | (spread10((u32) qy) << 1) | spread10((u32) qz);
    ids[i] = (u32) i;
}

__device__ __forceinline__ int prefix(const u32* codes, int n, int i, int j)
{
    if (j < 0 || j >= n) return -1;
    u32 a = codes[i], b = codes[j];
    if (a == b) return 32 + __clz((u32) i ^ (u32) j);
    return __clz(a ^ b);
}

// The walks keep a stack of kStack entries (the 4-wide walk up to 3 per 4-wide
// level): a clustering tree deeper than this is replaced by the radix hierarchy,
// whose depth is bounded by the code and index bits.
constexpr int kPlocMaxDepth = 40;

// status[0]: 1 when the clustering failed; status[1]: depth of the deepest
// internal node of its tree. `status` null: the radix hierarchy is the builder.
__device__ __forceinline__ bool radix_wanted(const int* status)
{
    return !status || (status[0] == 0 && status[1] + 1 > kPlocMaxDepth);   // + 1: the leaves below that node
}

__global__ void k_hierarchy(const int* __restrict__ status, const u32* codes, int n, int* left, int* right,
                            int* parent_int, int* parent_leaf)
{
    if (!radix_wanted(status)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) parent_int[0] = -1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (prefix(codes, n, i, i + 1) - prefix(codes, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = prefix(codes, n, i, i - d);
    int lmax = 2;
    while (prefix(codes, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (prefix(codes, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = prefix(codes, n, i, j);
    int s = 0;
    for (int div = 2;; div <<= 1) {
        int t = (l + div - 1) / div;
        if (prefix(codes, n, i, i + (s + t) * d) > dnode) s += t;
        if (t <= 1) break;
    }
    int gamma = i + s * d + min(d, 0);
    int lc = (min(i, j) == gamma) ? ~gamma : gamma;
    int rc = (max(i, j) == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    left[i] = lc;
    right[i] = rc;
    if (lc < 0) parent_leaf[~lc] = i; else parent_int[lc] = i;
    if (rc < 0) parent_leaf[~rc] = i; else parent_int[rc] = i;
}

// Conservative leaf box: the reference's box widened by a few tens of ulps,
// which absorbs the rounding of the exact hit and distance tests.
__device__ __forceinline__ void leaf_box_of(const float* r, float* b)
{
    float mnx = r[0], mny = r[1], mnz = r[2], mxx = r[3], mxy = r[4], mxz = r[5];
    float m = fmaxf(fmaxf(fmaxf(fabsf(mnx), fabsf(mxx)), fmaxf(fabsf(mny), fabsf(mxy))), fmaxf(fabsf(mnz), fabsf(mxz)));
    float e = m * 2e-5f + 1e-6f;
    b[0] = mnx - e; b[1] = mny - e; b[2] = mnz - e;
    b[3] = mxx + e; b[4] = mxy + e; b[5] = mxz + e;
}

__device__ __forceinline__ void read_box(const float* boxes, int k, float* b)
{
    for (int c = 0; c < 6; ++c) b[c] = __ldcg(boxes + 6 * (size_t) k + c);
}

__global__ void k_refit(const int* __restrict__ status, const float* ref_box, const u32* ids, int n, const int* parent_leaf, const int* parent_int,
                        const int* left, const int* right, float* leaf_box, float* int_box, u32* arrivals)
{
    if (!radix_wanted(status)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float b[6];
    leaf_box_of(ref_box + 6 * (size_t) ids[i], b);
    for (int c = 0; c < 6; ++c) leaf_box[6 * (size_t) i + c] = b[c];
    __threadfence();
    int p = n > 1 ? parent_leaf[i] : -1;
    while (p >= 0) {
        if (atomicAdd(&arrivals[p], 1u) == 0u) return;
        __threadfence();
        float bl[6], br[6];
        int l = left[p], r = right[p];
        if (l < 0) read_box(leaf_box, ~l, bl); else read_box(int_box, l, bl);
        if (r < 0) read_box(leaf_box, ~r, br); else read_box(int_box, r, br);
        for (int c = 0; c < 3; ++c) {
            int_box[6 * (size_t) p + c] = fminf(bl[c], br[c]);
            int_box[6 * (size_t) p + 3 + c] = fmaxf(bl[3 + c], br[3 + c]);
        }
        __threadfence();
        p = parent_int[p];
    }
}

// Binary node i (layout in bvh.cuh) from its children's boxes (min xyz, max xyz) and refs.
__device__ __forceinline__ void put_node(float4* nodes, size_t i, const float* L, int l, const float* R, int r)
{
    float4* o = nodes + 4 * i;
    o[0] = make_float4(L[0], R[0], L[1], R[1]);
    o[1] = make_float4(L[2], R[2], L[3], R[3]);
    o[2] = make_float4(L[4], R[4], L[5], R[5]);
    o[3] = make_float4(__int_as_float(l), __int_as_float(r), 0.0f, 0.0f);
}

// Child s (0 left, 1 right) of binary node i: its box; returns its ref.
__device__ __forceinline__ int get_child(const float4* nodes, size_t i, int s, float* box)
{
    const float* f = reinterpret_cast<const float*>(nodes + 4 * i);
#pragma unroll
    for (int c = 0; c < 6; ++c) box[c] = f[2 * c + s];
    return __float_as_int(f[12 + s]);
}

// Nodes of the radix hierarchy; or, after a failed clustering, nodes whose children are
// both leaf 0, so that kernels queued behind the build end at once: their boxes are
// inside out, which a distance query of finite radius does not enter and a segment
// does (a slab test takes either order of the planes), and then tests that leaf twice. No
// other child may stand there. The failure itself is the status word.
__global__ void k_pack_nodes(const int* __restrict__ status, int n_int, const int* left, const int* right,
                             const float* leaf_box, const float* int_box, float4* nodes)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_int) return;
    if (status && status[0] != 0) {
        const float none[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
        put_node(nodes, i, none, ~0, none, ~0);
        return;
    }
    if (!radix_wanted(status)) return;
    int l = left[i], r = right[i];
    const float* L = l < 0 ? leaf_box + 6 * (size_t) (~l) : int_box + 6 * (size_t) l;
    const float* R = r < 0 ? leaf_box + 6 * (size_t) (~r) : int_box + 6 * (size_t) r;
    put_node(nodes, i, L, l, R, r);
}

// ---- 4-wide nodes: the binary nodes at even depth, with their grandchildren as children

// flag[i] = 1 when internal node i lies at even depth (the root at depth 0).
__global__ void k_even_depth(int n_int, const int* __restrict__ parent_int, int* __restrict__ flag)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n_int) return;
    if (i == n_int) { flag[i] = 0; return; }
    int d = 0;
    for (int p = parent_int[i]; p >= 0 && d < 4096; p = parent_int[p]) ++d;
    flag[i] = (d & 1) == 0;
}

__device__ __forceinline__ void put_slot(float4* o, int k, const float* box, int child)
{
    reinterpret_cast<float*>(&o[0])[k] = box[0];
    reinterpret_cast<float*>(&o[1])[k] = box[3];
    reinterpret_cast<float*>(&o[2])[k] = box[1];
    reinterpret_cast<float*>(&o[3])[k] = box[4];
    reinterpret_cast<float*>(&o[4])[k] = box[2];
    reinterpret_cast<float*>(&o[5])[k] = box[5];
    reinterpret_cast<int*>(&o[6])[k] = child;
}

// Node layout in bvh.cuh (8 float4), from the binary nodes. Child boxes are the
// binary tree's, which are already inflated; a grandchild that is internal is
// referenced by its 4-wide index (it lies at even depth too), a leaf by ~leaf.
__global__ void k_pack4(int n_int, const int* __restrict__ flag, const int* __restrict__ idx4,
                        const float4* __restrict__ nodes, float4* __restrict__ nodes4)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_int || !flag[i]) return;
    float4* o = nodes4 + 8 * (size_t) idx4[i];
    const float empty_box[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
    int k = 0;
    for (int s = 0; s < 2; ++s) {
        float box[6];
        const int c = get_child(nodes, i, s, box);
        if (c < 0) {
            put_slot(o, k++, box, c);
        } else {
            for (int q = 0; q < 2; ++q) {
                const int gc = get_child(nodes, c, q, box);
                put_slot(o, k++, box, gc < 0 ? gc : idx4[gc]);
            }
        }
    }
    for (; k < 4; ++k) put_slot(o, k, empty_box, kNoChild);
    o[7] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Triangle-only terms of the two exact tests per leaf (layout in bvh.cuh),
// computed with the expressions of seg_tri / point_tri_dist in common.cuh.
// And the triangles themselves, in leaf order.
__global__ void k_pack_leaves(int nleaf, const u32* __restrict__ ids, const u32* __restrict__ ref_tri,
                              const float* __restrict__ xyz, const u32* __restrict__ metas,
                              const u32* __restrict__ local, float4* __restrict__ tris, float4* __restrict__ srec,
                              float4* __restrict__ drec)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nleaf) return;
    const u32 src = ref_tri[ids[i]];
    const float* p = xyz + 9 * (size_t) src;
    V3 t0 = mk(p[0], p[1], p[2]), t1 = mk(p[3], p[4], p[5]), t2 = mk(p[6], p[7], p[8]);
    const float meta = __uint_as_float(metas[src]);
    tris[3 * (size_t) i + 0] = make_float4(t0.x, t0.y, t0.z, meta);
    tris[3 * (size_t) i + 1] = make_float4(t1.x, t1.y, t1.z, __uint_as_float(local[src]));
    tris[3 * (size_t) i + 2] = make_float4(t2.x, t2.y, t2.z, __uint_as_float(src));
    V3 u = t1 - t0, v = t2 - t0;
    V3 n = cross(u, v);
    float4* s = srec + 4 * (size_t) i;
    s[0] = make_float4(t0.x, t0.y, t0.z, meta);
    s[1] = make_float4(u.x, u.y, u.z, dot(u, u));
    s[2] = make_float4(v.x, v.y, v.z, dot(u, v));
    s[3] = make_float4(n.x, n.y, n.z, dot(v, v));
    V3 nrm = normalized(cross(t1 - t0, t2 - t0));
    V3 tan0 = normalized(t1 - t0), tan1 = normalized(t2 - t1), tan2 = normalized(t0 - t2);
    V3 en0 = normalized(cross(t1 - t0, nrm)), en1 = normalized(cross(t2 - t1, nrm)), en2 = normalized(cross(t0 - t2, nrm));
    float4* d = drec + 8 * (size_t) i;
    d[0] = make_float4(nrm.x, nrm.y, nrm.z, dot(nrm, t0));
    d[1] = make_float4(tan0.x, tan0.y, tan0.z, dot(tan0, t0));
    d[2] = make_float4(tan1.x, tan1.y, tan1.z, dot(tan1, t1));
    d[3] = make_float4(tan2.x, tan2.y, tan2.z, dot(tan2, t2));
    d[4] = make_float4(dot(tan0, t1), dot(tan1, t2), dot(tan2, t0), meta);
    d[5] = make_float4(en0.x, en0.y, en0.z, dot(en0, t0));
    d[6] = make_float4(en1.x, en1.y, en1.z, dot(en1, t1));
    d[7] = make_float4(en2.x, en2.y, en2.z, dot(en2, t2));
}

// ---- locally-ordered clustering (PLOC; Meister and Bittner, "Parallel
// Locally-Ordered Clustering for Bounding Volume Hierarchy Construction",
// IEEE TVCG 2018). The leaves in Morton order are the first clusters; every
// iteration, each cluster finds within kPlocR positions on either side the one
// whose merged box has the least surface area, mutual nearest pairs merge into
// a new internal node at the lower position, and the list is compacted,
// keeping Morton order. Internal nodes are numbered down from n - 2 in merge
// order (ranks from a scan), so the last merge, the root, is node 0 as in
// Karras' layout. Ties between equal costs go by a key of the pair alone
// (distance in the list, then the lower position's parity, then the lower
// position), so the pairs are totally ordered: the least pair is always mutual
// (every iteration merges), and a run of equal boxes pairs up (0,1), (2,3), ...
// and halves each iteration instead of growing a chain.
//
// All iterations run in one launch: one thread-block cluster, each block owning a
// contiguous run of the list, with two cluster barriers per iteration (merge
// counts, then the compacted list), and one block alone in shared memory once the
// list fits its threads. Bound by the neighbour search of the first iterations
// (about 20 instructions per pair) and by the latency of the later ones, so the
// search is straight-line code over sentinel-padded boxes, and the blocks are as
// many as a cluster takes: 16 where the device can place such a cluster, 8
// otherwise, fewer for short lists (ploc_launch). Measured, whole kernel: 44,652
// references 539 us with 8 blocks and a bounds-checked search -> 264 us, the 1.8k-triangle
// level (22k references) 328 -> 185 us, a 34-triangle room 33 -> 18 us. Launched kernel
// by kernel (as graphs of eight iterations and a read-back of the count) the same
// builds took 2.5 and 1.6 ms.

constexpr int kPlocR = 16;
constexpr int kPlocT = 1024;           // threads per block
constexpr int kPlocMaxCtas = 16;
constexpr int kPlocOwn = kPlocT - 2 * kPlocR;   // most clusters a block merges at a time (its threads' less the halo's)

__device__ __forceinline__ float merged_area(const float* a, const float* b)
{
    float ex = fmaxf(a[3], b[3]) - fminf(a[0], b[0]);
    float ey = fmaxf(a[4], b[4]) - fminf(a[1], b[1]);
    float ez = fmaxf(a[5], b[5]) - fminf(a[2], b[2]);
    return ex * ey + ey * ez + ez * ex;
}

struct PlocArgs {
    int n;
    const float* ref_box;
    const u32* ids;               // references in Morton order
    float4* cl[2];                // clusters, 2 per entry: (mn.xyz, mx.x) (mx.yz, node or ~leaf, height)
    u32* flags;                   // per cluster: partner << 2 | merges (lower half of its pair) << 1 | keeps its place
    unsigned long long* totals;   // [parity][kPlocMaxCtas]: merges << 32 | kept
    float4* nodes;                // bvh.cuh's binary nodes
    int* parent;                  // per internal node (may be null)
    int* status;                  // see radix_wanted
};

// Clusters' boxes in shared memory (16 + 8 bytes, read as two vectors), kPlocR
// slots more on either side. A slot without a cluster holds a box whose merged
// area with any other is infinite.
struct PlocBoxes {
    float4 a[kPlocT + 2 * kPlocR];   // mn.xyz, mx.x
    float2 b[kPlocT + 2 * kPlocR];   // mx.yz
    __device__ __forceinline__ void none(int k)
    {
        a[k] = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, FLT_MAX);
        b[k] = make_float2(FLT_MAX, FLT_MAX);
    }
    __device__ __forceinline__ void get(int k, float* o) const
    {
        const float4 p = a[k];
        const float2 q = b[k];
        o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = p.w; o[4] = q.x; o[5] = q.y;
    }
};

// The nearest neighbour of cluster i (at slot k) as a key that orders its pairs:
// cost (a non-negative float's bits), then list distance, parity of the lower
// position, the lower position (26 bits; bvh_build keeps longer lists away).
// ~0: none (no finite cost).
__device__ __forceinline__ unsigned long long ploc_nearest(const PlocBoxes& s, int k, int i)
{
    float me[6];
    s.get(k, me);
    const u32 same = ((u32) (i & 1) << 26) | (u32) i, flip = same ^ (1u << 26);
    unsigned long long best = ~0ull;
#pragma unroll
    for (int d = -kPlocR; d <= kPlocR; ++d) {
        if (d == 0) continue;
        float o[6];
        s.get(k + d, o);
        const float c = merged_area(me, o);
        // lower position i (d > 0) or i + d, whose parity differs from i's when d is odd
        const u32 tie = d > 0 ? same + ((u32) d << 27) : ((d & 1) ? flip : same) + (u32) d + ((u32) -d << 27);
        const unsigned long long key = ((unsigned long long) __float_as_uint(c) << 32) | tie;
        best = key < best ? key : best;
    }
    return (u32) (best >> 32) <= __float_as_uint(FLT_MAX) ? best : ~0ull;
}

__device__ __forceinline__ int ploc_partner(unsigned long long key, int i)
{
    if (key == ~0ull) return -1;
    const int d = (int) ((u32) key >> 27), mn = (int) (key & 0x3ffffffull);
    return mn == i ? i + d : mn;
}

// Exclusive ranks of two flags over the block's threads, and their totals (kept
// in the low, merged in the high half word).
__device__ __forceinline__ u32 ploc_scan(bool keep, bool merge, u32* wsum, u32& total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 bk = __ballot_sync(0xffffffffu, keep), bm = __ballot_sync(0xffffffffu, merge);
    const u32 below = (1u << lane) - 1u;
    if (lane == 0) wsum[w] = (u32) __popc(bk) | ((u32) __popc(bm) << 16);
    __syncthreads();
    u32 v = wsum[lane];   // 32 warps
    static_assert(kPlocT == 1024, "one warp total per lane");
    u32 inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    total = __shfl_sync(0xffffffffu, inc, 31);
    const u32 before = __shfl_sync(0xffffffffu, inc - v, w);
    __syncthreads();   // wsum may be written again
    return before + ((u32) __popc(bk & below) | ((u32) __popc(bm & below) << 16));
}

// Clusters a (lower) and b become internal node `id`; returns the merged cluster.
__device__ __forceinline__ void ploc_merge(const PlocArgs& p, int id, float4 a0, float4 a1, float4 b0, float4 b1,
                                           float4& o0, float4& o1)
{
    const int ca = __float_as_int(a1.z), cb = __float_as_int(b1.z);
    const float boxa[6] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y}, boxb[6] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y};
    put_node(p.nodes, id, boxa, ca, boxb, cb);
    if (p.parent) {
        if (ca >= 0) p.parent[ca] = id;
        if (cb >= 0) p.parent[cb] = id;
    }
    o0 = make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), fmaxf(a0.w, b0.w));
    o1 = make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), __int_as_float(id),
                     __int_as_float(max(__float_as_int(a1.w), __float_as_int(b1.w)) + 1));
}

__device__ __forceinline__ void ploc_cluster_sync()
{
    __threadfence();
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kPlocT) k_ploc(PlocArgs p)
{
    __shared__ PlocBoxes box;
    __shared__ unsigned long long key[kPlocT];
    __shared__ int2 ref[kPlocT];   // the tail's (node or ~leaf, height)
    __shared__ u32 wsum[32];
    const int tid = threadIdx.x, rank = blockIdx.x, ctas = gridDim.x;
    for (int i = rank * kPlocT + tid; i < p.n; i += ctas * kPlocT) {
        float b[6];
        leaf_box_of(p.ref_box + 6 * (size_t) p.ids[i], b);
        p.cl[0][2 * (size_t) i] = make_float4(b[0], b[1], b[2], b[3]);
        p.cl[0][2 * (size_t) i + 1] = make_float4(b[4], b[5], __int_as_float(~i), __int_as_float(-1));
    }
    ploc_cluster_sync();
    int count = p.n, base = p.n - 1, cur = 0;
    bool ok = true;
    for (int par = 0; ok && count > kPlocT; par ^= 1) {
        const float4* src = cur ? p.cl[1] : p.cl[0];
        float4* dst = cur ? p.cl[0] : p.cl[1];
        // this block's run [r0, r1), in tiles of `own` clusters: thread t stands for
        // cluster start - kPlocR + t, and merges it when it lies in the tile
        const int run = (count + ctas - 1) / ctas, r0 = min(count, rank * run), r1 = min(count, r0 + run);
        const int tiles = (r1 - r0 + kPlocOwn - 1) / kPlocOwn, own = tiles ? (r1 - r0 + tiles - 1) / tiles : 0;
        u32 kept = 0, merged = 0;
        for (int t = 0; t < tiles; ++t) {
            const int start = r0 + t * own, end = min(r1, start + own), i = start - kPlocR + tid;
            {
                const int g0 = i - kPlocR, g1 = g0 + kPlocT;   // slots tid and, for the last ones, tid + kPlocT
                const bool in0 = g0 >= 0 && g0 < count, two = tid < 2 * kPlocR, in1 = two && g1 < count;
                float4 a0, b0, a1, b1;
                if (in0) { a0 = __ldcg(src + 2 * (size_t) g0); b0 = __ldcg(src + 2 * (size_t) g0 + 1); }
                if (in1) { a1 = __ldcg(src + 2 * (size_t) g1); b1 = __ldcg(src + 2 * (size_t) g1 + 1); }
                if (in0) { box.a[tid] = a0; box.b[tid] = make_float2(b0.x, b0.y); } else box.none(tid);
                if (in1) { box.a[tid + kPlocT] = a1; box.b[tid + kPlocT] = make_float2(b1.x, b1.y); }
                else if (two) box.none(tid + kPlocT);
            }
            __syncthreads();
            if (i >= 0 && i < min(count, end + kPlocR)) key[tid] = ploc_nearest(box, tid + kPlocR, i);
            __syncthreads();
            bool keep = false, merge = false;
            if (i >= start && i < end) {
                const int j = ploc_partner(key[tid], i);
                const bool mutual = j >= 0 && ploc_partner(key[tid + j - i], j) == i;
                merge = mutual && i < j;
                keep = !(mutual && i > j);
                p.flags[i] = ((u32) j << 2) | (merge ? 2u : 0u) | (keep ? 1u : 0u);
            }
            kept += (u32) __syncthreads_count(keep);
            merged += (u32) __syncthreads_count(merge);
        }
        if (tid == 0) p.totals[par * kPlocMaxCtas + rank] = ((unsigned long long) merged << 32) | kept;
        ploc_cluster_sync();
        unsigned long long before = 0, total = 0;
        for (int r = 0; r < ctas; ++r) {
            const unsigned long long v = __ldcg(p.totals + par * kPlocMaxCtas + r);
            if (r < rank) before += v;
            total += v;
        }
        u32 pos = (u32) before, mrk = (u32) (before >> 32);
        for (int t = 0; t < tiles; ++t) {
            const int start = r0 + t * own, end = min(r1, start + own), i = start - kPlocR + tid;
            const u32 f = i >= start && i < end ? p.flags[i] : 0u;
            u32 tot;
            const u32 ex = ploc_scan((f & 1u) != 0, (f & 2u) != 0, wsum, tot);
            if (f & 1u) {
                float4 o0 = __ldcg(src + 2 * (size_t) i), o1 = __ldcg(src + 2 * (size_t) i + 1);
                if (f & 2u) {
                    const size_t j = f >> 2;
                    ploc_merge(p, base - 1 - (int) (mrk + (ex >> 16)), o0, o1, __ldcg(src + 2 * j), __ldcg(src + 2 * j + 1),
                               o0, o1);
                }
                float4* o = dst + 2 * (size_t) (pos + (ex & 0xffffu));
                o[0] = o0;
                o[1] = o1;
            }
            pos += tot & 0xffffu;
            mrk += tot >> 16;
        }
        ploc_cluster_sync();
        ok = (total >> 32) != 0;   // the least pair is always mutual: only unordered costs merge nothing
        count = (int) (total & 0xffffffffull);
        base -= (int) (total >> 32);
        cur ^= 1;
    }
    if (rank != 0) return;
    // the list fits this block's threads: one cluster per thread, in shared memory
    // (cluster t at slot t + kPlocR)
    const float4* last = cur ? p.cl[1] : p.cl[0];
    float4 c0 = make_float4(0, 0, 0, 0), c1 = c0;
    if (ok && tid < count) {
        c0 = __ldcg(last + 2 * (size_t) tid);
        c1 = __ldcg(last + 2 * (size_t) tid + 1);
    }
    if (tid < kPlocR) box.none(tid);
    while (ok && count > 1) {
        if (tid < count) {
            box.a[tid + kPlocR] = c0;
            box.b[tid + kPlocR] = make_float2(c1.x, c1.y);
            ref[tid] = make_int2(__float_as_int(c1.z), __float_as_int(c1.w));
        }
        if (tid < kPlocR) box.none(count + kPlocR + tid);
        __syncthreads();
        if (tid < count) key[tid] = ploc_nearest(box, tid + kPlocR, tid);
        __syncthreads();
        bool keep = false, merge = false;
        int j = -1;
        if (tid < count) {
            j = ploc_partner(key[tid], tid);
            const bool mutual = j >= 0 && ploc_partner(key[j], j) == tid;
            merge = mutual && tid < j;
            keep = !(mutual && tid > j);
        }
        u32 tot;
        const u32 ex = ploc_scan(keep, merge, wsum, tot);
        if (merge) {
            const float4 b0 = box.a[j + kPlocR];
            const float2 q = box.b[j + kPlocR];
            const int2 r = ref[j];
            ploc_merge(p, base - 1 - (int) (ex >> 16), c0, c1, b0,
                       make_float4(q.x, q.y, __int_as_float(r.x), __int_as_float(r.y)), c0, c1);
        }
        __syncthreads();   // partners read
        if (keep) {
            const u32 o = ex & 0xffffu;
            box.a[o + kPlocR] = c0;
            box.b[o + kPlocR] = make_float2(c1.x, c1.y);
            ref[o] = make_int2(__float_as_int(c1.z), __float_as_int(c1.w));
        }
        __syncthreads();
        ok = (tot >> 16) != 0;
        count = (int) (tot & 0xffffu);
        base -= (int) (tot >> 16);
        if (tid < count) {
            c0 = box.a[tid + kPlocR];
            const float2 q = box.b[tid + kPlocR];
            const int2 r = ref[tid];
            c1 = make_float4(q.x, q.y, __int_as_float(r.x), __int_as_float(r.y));
        }
        __syncthreads();   // everyone holds its cluster before the boxes are written again
    }
    if (tid == 0) {
        p.status[0] = ok && count == 1 && base == 0 ? 0 : 1;
        p.status[1] = __float_as_int(c1.w);
    }
}

// Blocks of the clustering's cluster for n references: one per full block of
// them (a longer list per block costs more than the wider barrier), up to the
// largest cluster that the current device can place.
cudaError_t ploc_launch(const PlocArgs& pa, cudaStream_t st)
{
    static std::atomic<int> largest[64];   // per device (a property of its SMs), 0 = not asked yet
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.blockDim = dim3(kPlocT);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int most = dev < 64 ? largest[dev].load() : 8;
    if (!most) {
        most = 8;   // the portable limit
        if (cudaFuncSetAttribute(k_ploc, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            int fit = 0;
            at.val.clusterDim.x = kPlocMaxCtas;
            cfg.gridDim = dim3(kPlocMaxCtas);
            if (cudaOccupancyMaxActiveClusters(&fit, k_ploc, &cfg) == cudaSuccess && fit > 0) most = kPlocMaxCtas;
        }
        cudaGetLastError();   // an answer of "no" is not an error of the build
        largest[dev].store(most);
    }
    int ctas = 1;
    while (ctas < most && ctas * kPlocT < pa.n) ctas *= 2;
    // the permission for more than the portable 8 lives in the context, which a device reset
    // replaces: given anew for each such launch
    if (ctas > 8 && cudaFuncSetAttribute(k_ploc, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        ctas = 8;
    }
    at.val.clusterDim.x = (unsigned) ctas;
    cfg.gridDim = dim3((unsigned) ctas);
    return cudaLaunchKernelEx(&cfg, k_ploc, pa);
}

// Parts of one device allocation, 256-byte aligned: a first pass adds up the
// sizes, a second one hands out the addresses.
struct Carve {
    char* base = nullptr;
    size_t at = 0;
    template <class T> T* take(size_t count)
    {
        T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
        at += (count * sizeof(T) + 255) / 256 * 256;
        return p;
    }
};

}  // namespace

void bvh_build(const BvhBuildInput& in, BvhStorage& out, void* stream)
{
    cudaStream_t st = (cudaStream_t) stream;
    const int n = in.n;
    out.n_tris = n;
    out.bytes = 0;
    if (n <= 0) { out.root = 0; return; }
    const int n_int = n - 1;
    out.root = n_int > 0 ? 0 : ~0;
    out.root4 = out.root;   // the root is binary node 0 (both builders), at depth 0: 4-wide node 0
    // list positions take 26 bits of the clustering's keys
    const bool ploc = in.builder != 1 && n_int > 0 && n < (1 << 26);
    const bool wide = n >= kWideTreeMin;

    size_t sort_bytes = 0, scan_bytes = 0;
    BVH_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (u32*) nullptr, (u32*) nullptr, (u32*) nullptr,
                                              (u32*) nullptr, n, 0, 30, st));
    if (wide)
        BVH_CHECK(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (int*) nullptr, (int*) nullptr, n_int + 1, st));

    // what the walks read, in one allocation
    auto layout = [&](Carve& c) {
        out.status = c.take<int>(2);
        out.nodes = c.take<float4>(4 * (size_t) std::max(n_int, 1));
        out.tris = c.take<float4>(3 * (size_t) n);
        out.srec = c.take<float4>(4 * (size_t) n);
        out.drec = c.take<float4>(8 * (size_t) n);
        out.nodes4 = wide ? c.take<float4>(8 * (size_t) n_int) : nullptr;   // at most one per binary node
    };
    Carve size;
    layout(size);
    BVH_CHECK(cudaMallocAsync(&out.mem, size.at, st));
    out.bytes = size.at;
    Carve fill{(char*) out.mem, 0};
    layout(fill);

    // build scratch, in another
    u32 *codes, *codes2, *ids, *ids2, *arrivals, *flags;
    int *left, *right, *parent_int, *parent_leaf, *flag4, *idx4;
    float *leaf_box, *int_box;
    float4* cl[2];
    unsigned long long* totals;
    char *sort_tmp, *scan_tmp;
    auto scratch = [&](Carve& c) {
        codes = c.take<u32>(n); codes2 = c.take<u32>(n); ids = c.take<u32>(n); ids2 = c.take<u32>(n);
        left = c.take<int>(n); right = c.take<int>(n); parent_int = c.take<int>(n); parent_leaf = c.take<int>(n);
        leaf_box = c.take<float>(6 * (size_t) n);
        int_box = c.take<float>(6 * (size_t) n);
        arrivals = c.take<u32>(n);
        sort_tmp = c.take<char>(sort_bytes);
        for (float4*& p : cl) p = c.take<float4>(ploc ? 2 * (size_t) n : 0);
        flags = c.take<u32>(ploc ? n : 0);
        totals = c.take<unsigned long long>(2 * kPlocMaxCtas);
        flag4 = c.take<int>(wide ? n : 0);
        idx4 = c.take<int>(wide ? n : 0);
        scan_tmp = c.take<char>(scan_bytes);
    };
    Carve ssize;
    scratch(ssize);
    void* smem = nullptr;
    BVH_CHECK(cudaMallocAsync(&smem, ssize.at, st));
    struct FreeScratch {
        void* p; cudaStream_t s;
        ~FreeScratch() { cudaFreeAsync(p, s); }
    } free_scratch{smem, st};
    Carve sfill{(char*) smem, 0};
    scratch(sfill);

    const int B = 256;
    float3 mn = make_float3(in.scene_min[0], in.scene_min[1], in.scene_min[2]);
    float ex = in.scene_max[0] - in.scene_min[0], ey = in.scene_max[1] - in.scene_min[1], ez = in.scene_max[2] - in.scene_min[2];
    float3 inv_ext = make_float3(ex > 0 ? 1.0f / ex : 0.0f, ey > 0 ? 1.0f / ey : 0.0f, ez > 0 ? 1.0f / ez : 0.0f);
    k_morton<<<(n + B - 1) / B, B, 0, st>>>(in.ref_box, n, mn, inv_ext, codes, ids); note_launch();
    BVH_CHECK(cudaGetLastError());
    BVH_CHECK(cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, codes, codes2, ids, ids2, n, 0, 30, st));
    BVH_CHECK(cudaMemsetAsync(out.status, 0, 2 * sizeof(int), st));
    if (wide) BVH_CHECK(cudaMemsetAsync(parent_int, 0xff, sizeof(int) * n_int, st));
    if (ploc) {
        PlocArgs pa;
        pa.n = n;
        pa.ref_box = in.ref_box;
        pa.ids = ids2;
        pa.cl[0] = cl[0];
        pa.cl[1] = cl[1];
        pa.flags = flags;
        pa.totals = totals;
        pa.nodes = out.nodes;
        pa.parent = wide ? parent_int : nullptr;
        pa.status = out.status;
        BVH_CHECK(ploc_launch(pa, st)); note_launch();
    }
    if (n_int > 0) {
        const int* status = ploc ? out.status : nullptr;
        BVH_CHECK(cudaMemsetAsync(arrivals, 0, sizeof(u32) * n_int, st));
        k_hierarchy<<<(n_int + B - 1) / B, B, 0, st>>>(status, codes2, n, left, right, parent_int, parent_leaf); note_launch();
        k_refit<<<(n + B - 1) / B, B, 0, st>>>(status, in.ref_box, ids2, n, parent_leaf, parent_int, left, right, leaf_box,
                                                int_box, arrivals); note_launch();
        k_pack_nodes<<<(n_int + B - 1) / B, B, 0, st>>>(status, n_int, left, right, leaf_box, int_box, out.nodes); note_launch();
        BVH_CHECK(cudaGetLastError());
    }
    if (wide) {
        k_even_depth<<<(n_int + 1 + B - 1) / B, B, 0, st>>>(n_int, parent_int, flag4); note_launch();
        BVH_CHECK(cudaGetLastError());
        BVH_CHECK(cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, flag4, idx4, n_int + 1, st));
        k_pack4<<<(n_int + B - 1) / B, B, 0, st>>>(n_int, flag4, idx4, out.nodes, out.nodes4); note_launch();
        BVH_CHECK(cudaGetLastError());
    }
    k_pack_leaves<<<(n + B - 1) / B, B, 0, st>>>(n, ids2, in.ref_tri, in.tri_xyz, in.tri_meta, in.tri_local, out.tris,
                                                  out.srec, out.drec); note_launch();
    BVH_CHECK(cudaGetLastError());
}

void bvh_check_status(int status)
{
    if (status) throw std::runtime_error("bvh: clustering step inconsistent");
}

// Copies the topology back and checks that a walk from the root reaches every
// internal node and every leaf exactly once; returns an empty string when the
// tree is sound. Used by the LTRG_VALIDATE=1 debug mode of the bake.
std::string bvh_validate(const BvhStorage& s, void* stream)
{
    if (s.n_tris <= 1) return "";
    const int n = s.n_tris, n_int = n - 1;
    std::vector<float4> nodes(4 * (size_t) n_int);
    BVH_CHECK(cudaMemcpyAsync(nodes.data(), s.nodes, nodes.size() * sizeof(float4), cudaMemcpyDeviceToHost,
                              (cudaStream_t) stream));
    BVH_CHECK(cudaStreamSynchronize((cudaStream_t) stream));
    std::vector<int> seen_int(n_int, 0), seen_leaf(n, 0);
    std::vector<int> stack(1, s.root);
    while (!stack.empty()) {
        int c = stack.back();
        stack.pop_back();
        if (c < 0) {
            if (~c >= n) return "leaf index out of range: " + std::to_string(~c);
            if (seen_leaf[~c]++) return "leaf reached twice: " + std::to_string(~c);
            continue;
        }
        if (c >= n_int) return "node index out of range: " + std::to_string(c);
        if (seen_int[c]++) return "node reached twice: " + std::to_string(c);
        float4 n3 = nodes[4 * (size_t) c + 3];
        int l, r;
        memcpy(&l, &n3.x, 4);
        memcpy(&r, &n3.y, 4);
        stack.push_back(l);
        stack.push_back(r);
    }
    for (int i = 0; i < n_int; ++i)
        if (!seen_int[i]) return "node unreachable: " + std::to_string(i);
    for (int i = 0; i < n; ++i)
        if (!seen_leaf[i]) return "leaf unreachable: " + std::to_string(i);
    return "";
}

void bvh_free(BvhStorage& s, void* stream)
{
    if (s.mem) cudaFreeAsync(s.mem, (cudaStream_t) stream);
    s = BvhStorage();
}

}  // namespace lg
