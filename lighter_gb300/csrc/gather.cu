// Multi-right-hand-side radiosity gather on dense form factors.
//
// The reference's bounce (Int_RDBounce, lighter.cpp:767-797) is one sweep of
// B <- E + K B over sparse links, K_ij = f_ij area_j diffuse_j, for one light
// configuration. For R right-hand sides (RGB x light configurations) the sweep
// is the contraction
//     B_k = E + G X_{k-1},   G_ij = f_ij area_j,   X_j(r) = albedo_j(r mod 3) B_j(r)
// whose left operand G (N x N) streams from HBM once per bounce while X
// (N x R) stays in L2.
//
//   FP32        G in FP32, SIMT stream-K GEMM                       k_sgemm_bounce
//   FP16/BF16   G in 16 bits on the tcgen05 tensor cores            k_umma_gather
//               (FP32 accumulation in TMEM), with optional head/tail
//               splits of X and of G (LTRG_REFINE_*) whose extra products
//               accumulate into the same FP32 accumulator
//
// k_umma_gather is a persistent stream-K kernel: the (256-row block, 64-wide
// k block) units of the whole product are cut into one contiguous range per
// CTA, so every SM gets the same number of units whatever N is. Per CTA:
//   warp 0      TMA producer: 256 x 64 tile of G (+ residual), BN x 64 tiles of
//               X^T (head, tail), 128-byte swizzle, into an S-stage ring
//   warp 1      allocates 512 TMEM columns; one thread issues
//               tcgen05.mma.cta_group::1.kind::f16 (M=128, N=BN, K=16) for both
//               128-row halves into two FP32 accumulators (columns 0 and 256)
//   warps 2-5   epilogue: tcgen05.ld of the accumulators, partial sums of each
//               row block written to a workspace slot
// Wide split right-hand sides run on pairs of CTAs instead (cta_group::2, M=256).
// k_combine then adds E and the slots of every row block in a fixed order
// (deterministic) and writes B and the next bounce's X^T. Every mbarrier wait
// is bounded: on expiry the kernel sets a bit of the error word, stops its
// loops, waits (bounded) for its own copies and products and frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "../../include/lighter_gb300.h"
#include "bvh.cuh"
#include "async.cuh"
#include "radiosity.cuh"

namespace lg {
void keep_pool_memory(int device);   // bake.cu

namespace {

void gck(cudaError_t e, const char* what, int line)
{
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e) + " at gather.cu:" +
                                 std::to_string(line) + " (" + what + ")");
}
#define GCK(x) gck((x), #x, __LINE__)

constexpr int BM = 128;                  // rows per tcgen05.mma (M)
constexpr int ROWS = 2 * BM;             // rows of G per work unit
constexpr int BK = 64;                   // k per work unit (and the padding of a row of G)
constexpr int UK = 16;                   // k per tcgen05.mma (kind::f16)
constexpr int MAX_BN = 256;
constexpr int TMEM_COLS = 512;           // two accumulators of up to 256 columns
constexpr int kThreads = 192;
constexpr int kMaxStages = 8;
constexpr int kSmemLimit = 232448;       // opt-in dynamic shared memory per block
constexpr int kSmemExtra = 1024 + 256;   // alignment slack + barriers
constexpr unsigned long long kWaitCycles = 4000000000ull;   // about 2 s at 2 GHz

// error word bits
constexpr u32 kErrProducer = 1u, kErrMma = 2u, kErrEpilogue = 4u, kErrDrain = 8u;

// ----------------------------------------------------------------------------- PTX helpers

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            saddr(dst)),
        "l"(map), "r"(saddr(bar)), "r"(x), "r"(y)
        : "memory");
}

// The same into this CTA of a pair, completing on the barrier in its even CTA (an
// address from mapa).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t even_bar, int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];" ::"r"(
            saddr(dst)),
        "l"(map), "r"(even_bar), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ uint32_t even_cta_addr(const void* p)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(saddr(p)));
    return a;
}

// Matrix descriptor of a K-major operand tile written by TMA with the swizzle
// of its row length KB x 2 bytes: 128-byte rows (KB = 64, 128-byte swizzle) or
// 64-byte rows (KB = 32, 64-byte swizzle), groups of 8 rows 8 x row bytes
// apart. Advancing K by 16 elements inside a row adds 32 bytes to the start.
// Only the low word depends on the address, and no offset inside shared memory
// (below 256 KB) carries out of its 14 bits: a tile's descriptors are its low word
// plus constants.
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t addr)
{
    return ((addr >> 4) & 0x3FFFu) | 1u << 16;   // start address >> 4; leading byte offset (unused for swizzled K-major)
}
template <int KB>
__device__ __forceinline__ uint64_t sdesc(uint32_t lo)
{
    static_assert(KB == 64 || KB == 32, "stage k must be 64 or 32");
    const uint32_t hi = ((8u * KB * 2) >> 4)          // stride byte offset: 8 rows
                        | 1u << 14                    // descriptor version
                        | (KB == 64 ? 2u : 4u) << 29; // 128-byte or 64-byte swizzle
    return (uint64_t) hi << 32 | lo;
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), A and
// B of format `fmt` (0 FP16, 1 BF16; bits 7-9 and 10-12), both K-major
// (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
uint32_t idesc_f16(uint32_t fmt, uint32_t m, uint32_t bn)
{
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((bn >> 3) << 17) | ((m >> 4) << 24);
}

// CTAS = 2: one product over the CTA pair, issued by its even CTA (see k_umma_gather).
template <int CTAS>
__device__ __forceinline__ void umma(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc)
{
    if (CTAS == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
}

// Arrives on `bar` (CTAS = 2: in the CTAs of `mask`) once every tcgen05.mma issued so far by
// this thread completes.
template <int CTAS>
__device__ __forceinline__ void umma_commit(uint64_t* bar, uint16_t mask = 3)
{
    if (CTAS == 2)
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                saddr(bar)),
            "h"(mask)
            : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
                     : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// All threads of the block, or of the pair.
template <int CTAS>
__device__ __forceinline__ void group_sync()
{
    if (CTAS == 2) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    } else __syncthreads();
}

// ----------------------------------------------------------------------------- tcgen05 gather

struct UmmaArgs {
    u32 nkb;              // k blocks (ld / 64)
    u32 n_rp;             // 256-row blocks
    u32 R, BN;            // right-hand sides, MMA N (multiple of 32, >= R)
    u32 stages, stage_bytes;
    u32 idesc;
    u32 max_slots;
    u32 kchunk;           // k blocks accumulated in TMEM before moving to the FP32 workspace (0: no limit)
    const u32* rp_first;  // first range (CTA or pair) that touches each row block
    float* partial;       // [rp][slot][R][256]
    u32* err;
    unsigned long long wait_cycles;   // limit of every mbarrier wait (kWaitCycles)
    u32 issue;            // 0: the producer issues no copies (ltrdbg_GatherStallNextSolve), else 1
};

// KB: k per pipeline stage (a 64-wide work unit takes 64 / KB stages).
//
// CTAS = 2: a pair of CTAs (a cluster, on one pair of SMs) takes units of two row
// blocks. Each holds the G tile of its own row block and half of the rows of the
// X tile; the even CTA issues products with M = 256 (cta_group::2) that read both
// CTAs' tiles and leave each CTA its own 128 rows x BN in its own tensor memory.
// X, which every row block reads again, costs half the L2 reads and half the shared
// memory, so the ring has twice the stages (figures at gather_plan).
// Both CTAs' copies complete on the even CTA's `full`; commits arrive in both CTAs;
// both epilogues arrive on the even CTA's `acce`.
template <int KB, int CTAS, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    k_umma_gather(const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmGl,
                  const __grid_constant__ CUtensorMap tmXh, const __grid_constant__ CUtensorMap tmXl, UmmaArgs a)
{
    constexpr int SPU = BK / KB;                 // stages per work unit
    constexpr u32 A_BYTES = ROWS * KB * 2;       // one 256-row tile of G per stage
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*) ((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + (size_t) a.stages * a.stage_bytes);
    uint64_t* full = bars;
    uint64_t* empty = bars + kMaxStages;
    uint64_t* accf = bars + 2 * kMaxStages;       // accumulators ready for the epilogue
    uint64_t* acce = accf + 1;                    // accumulators drained
    uint64_t* done = accf + 2;                    // all products of this CTA complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accf + 3);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 rank = CTAS == 2 ? blockIdx.x & 1u : 0u, range = blockIdx.x / CTAS;   // clusters are consecutive blocks
    const uint64_t total = (uint64_t) ((a.n_rp + CTAS - 1) / CTAS) * a.nkb;   // a unit: CTAS row blocks x one k block
    const uint64_t lo = (uint64_t) range * total / (gridDim.x / CTAS);
    const uint64_t hi = (uint64_t) (range + 1) * total / (gridDim.x / CTAS);
    const u32 n_units = (u32) (hi - lo);   // below 2^32: at most 8,192 row blocks x 32,768 k blocks
    const u32 b_bytes = a.BN / CTAS * KB * 2;
    constexpr u32 off_gl = A_BYTES;
    constexpr u32 off_xh = MODE == LTRG_REFINE_FULL ? 2 * A_BYTES : A_BYTES;
    const u32 off_xl = off_xh + b_bytes;
    const u32 tx_bytes = (MODE == LTRG_REFINE_FULL ? 2 : 1) * A_BYTES + (MODE >= LTRG_REFINE_RHS ? 2 : 1) * b_bytes;

    if (threadIdx.x == 0) {
        for (u32 s = 0; s < a.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(accf, 1);
        mbar_init(acce, 4 * CTAS);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (CTAS == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    group_sync<CTAS>();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // producer: stage s, whose use number has parity ph
            u32 s = 0, ph = 0, used = 0, ru = (u32) (lo / a.nkb), kb = (u32) (lo % a.nkb);
            const int rx = (int) (rank * a.BN / CTAS);   // this CTA's rows of X
            const uint32_t full_even = CTAS == 2 ? even_cta_addr(full) : 0u;
            bool ok = true;
            for (u32 left = a.issue ? n_units : 0; left && ok; --left) {
                for (int q = 0; q < SPU; ++q) {
                    if (used == a.stages) {
                        if (!mbar_wait(&empty[s], ph ^ 1u, a.err, kErrProducer, a.wait_cycles)) {
                            ok = false;
                            break;
                        }
                    } else ++used;
                    const int kx = (int) (kb * BK + q * KB), ry = (int) ((ru * CTAS + rank) * ROWS);
                    unsigned char* st = base + (size_t) s * a.stage_bytes;
                    // the even CTA's barrier counts both CTAs' bytes; the odd CTA's copies cannot
                    // run ahead into its next phase, since they wait for this one's products
                    if (rank == 0) mbar_expect_tx(&full[s], CTAS * tx_bytes);
                    auto load = [&](uint32_t off, const CUtensorMap* m, int x, int y) {
                        if (CTAS == 2) tma_load_2d_pair(st + off, m, full_even + 8 * s, x, y);
                        else tma_load_2d(st + off, m, &full[s], x, y);
                    };
                    load(0, &tmG, kx, ry);
                    if (MODE == LTRG_REFINE_FULL) load(off_gl, &tmGl, kx, ry);
                    load(off_xh, &tmXh, kx, rx);
                    if (MODE >= LTRG_REFINE_RHS) load(off_xl, &tmXl, kx, rx);
                    if (++s == a.stages) { s = 0; ph ^= 1u; }
                }
                if (++kb == a.nkb) { kb = 0; ++ru; }
            }
            // wait for the copies still in flight (complete already unless a wait above expired)
            // the last `used` stages issued end at stage s, so stage t was last used in
            // this round of the ring (t < s) or the one before
            for (u32 t = 0; rank == 0 && t < used; ++t)
                if (!mbar_wait(&full[t], t < s ? ph : ph ^ 1u, a.err, kErrDrain, a.wait_cycles)) break;
            // in a pair, also for the issuer's last commits into this CTA; where they do not
            // come, the odd CTA gives its own copies (microseconds at most) a millisecond or so
            if (CTAS == 2)
                for (u32 t = 0; t < used; ++t)
                    if (!mbar_wait(&empty[t], t < s ? ph : ph ^ 1u, a.err, kErrDrain, a.wait_cycles)) {
                        for (const long long t0 = clock64(); clock64() - t0 < 2000000;) {}
                        break;
                    }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // MMA issuer. One thread issues everything, so its own instructions count: no
            // divisions, descriptors by adding constants (with a 64-bit remainder per unit and
            // stage and descriptors built from addresses, a product of any width took 155
            // cycles: 32,768 patches, 0.56 ms per sweep even for R = 3)
            u32 s = 0, ph = 0, seg = 0, kb = (u32) (lo % a.nkb), kc = a.kchunk ? kb % a.kchunk : 0;
            bool ok = true, first = true;
            for (u32 left = n_units; left && ok; --left) {
                const bool last = left == 1 || kb + 1 == a.nkb || (a.kchunk && kc + 1 == a.kchunk);
                if (first && seg > 0 && !mbar_wait<CTAS == 2>(acce, (seg - 1) & 1u, a.err, kErrMma, a.wait_cycles)) break;
                for (int q = 0; q < SPU; ++q) {
                    if (!mbar_wait(&full[s], ph, a.err, kErrMma, a.wait_cycles)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t lg = sdesc_lo(saddr(base) + s * a.stage_bytes), lh = lg + (off_xh >> 4), ll = lg + (off_xl >> 4);
                    uint32_t acc = first && q == 0 ? 0u : 1u;
#pragma unroll
                    for (int k = 0; k < KB / UK; ++k) {
                        const uint64_t bh = sdesc<KB>(lh + k * (UK * 2 / 16)), bl = sdesc<KB>(ll + k * (UK * 2 / 16));
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t d = tmem + h * 256, ao = lg + h * (BM * KB * 2 / 16) + k * (UK * 2 / 16);
                            umma<CTAS>(d, sdesc<KB>(ao), bh, a.idesc, acc);
                            if (MODE >= LTRG_REFINE_RHS) umma<CTAS>(d, sdesc<KB>(ao), bl, a.idesc, 1u);
                            if (MODE == LTRG_REFINE_FULL) umma<CTAS>(d, sdesc<KB>(ao + A_BYTES / 16), bh, a.idesc, 1u);
                        }
                        acc = 1u;
                    }
                    umma_commit<CTAS>(&empty[s]);
                    if (++s == a.stages) { s = 0; ph ^= 1u; }
                }
                if (ok && last) { umma_commit<CTAS>(accf); ++seg; }
                first = last;
                if (++kc == a.kchunk) kc = 0;
                if (++kb == a.nkb) kb = kc = 0;
            }
            umma_commit<CTAS>(done, 1);
            mbar_wait(done, 0, a.err, kErrDrain, a.wait_cycles);
        }
    } else {
        // epilogue: TMEM lanes of quadrant q = rows 32q .. 32q+31 of each 128-row half
        const int q = warp & 3;
        // Segments (the MMA issuer's accumulations) in the same order: maximal runs of
        // units within one row block and, when kchunk > 0, within one k chunk. The
        // first segment of a row block writes its workspace slot, later ones add to it.
        uint64_t u = lo;
        for (u32 seg = 0; u < hi; ++seg) {
            const u32 ru = (u32) (u / a.nkb), rp = ru * CTAS + rank, kb = (u32) (u % a.nkb);
            const u32 kend = a.kchunk ? min(a.nkb, (kb / a.kchunk + 1) * a.kchunk) : a.nkb;
            const bool fresh = u == lo || kb == 0;
            u = min(hi, (uint64_t) ru * a.nkb + kend);
            // every lane waits; the warp goes on only if all of them saw the phase, so the
            // .sync.aligned loads below always run converged
            const bool ok = mbar_wait(accf, seg & 1u, a.err, kErrEpilogue, a.wait_cycles);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const bool real = rp < a.n_rp;   // the odd row block of the last pair may not be one
            const u32 slot = real ? range - __ldg(&a.rp_first[rp]) : 0u;
            float* P = a.partial + ((size_t) rp * a.max_slots + slot) * a.R * ROWS;
            for (int h = 0; h < 2 && real; ++h) {
                const u32 row = h * BM + q * 32 + lane;
                for (u32 c0 = 0; c0 < a.BN; c0 += 32) {
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t) (q * 32) << 16) + h * 256 + c0, v);
                    float* d = P + (size_t) c0 * ROWS + row;
                    if (!fresh) {   // all loads first, then all stores: one round trip per 32 columns
                        float prev[32];
#pragma unroll
                        for (int c = 0; c < 32; ++c) prev[c] = c0 + c < a.R ? d[(size_t) c * ROWS] : 0.0f;
#pragma unroll
                        for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + prev[c]);
                    }
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (c0 + c < a.R) d[(size_t) c * ROWS] = __uint_as_float(v[c]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(acce);
                else mbar_arrive_rank(acce, 0);
            }
        }
    }
    // nothing of the pair is in flight beyond this point: every copy and product was
    // waited for (within the limit) by the CTA that issued it
    tc_fence_before();
    group_sync<CTAS>();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        if (CTAS == 2)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ----------------------------------------------------------------------------- combine

template <class T> __device__ __forceinline__ T to16(float f);
template <> __device__ __forceinline__ __half to16<__half>(float f) { return __float2half_rn(f); }
template <> __device__ __forceinline__ __nv_bfloat16 to16<__nv_bfloat16>(float f) { return __float2bfloat16_rn(f); }
__device__ __forceinline__ float from16(__half h) { return __half2float(h); }
__device__ __forceinline__ float from16(__nv_bfloat16 h) { return __bfloat162float(h); }

// Exponent of the power-of-two scale of X: the largest emission maps below
// 2^9, which leaves room for the bounced light to grow 100x and keeps small
// values out of the FP16 subnormal range.
__device__ __forceinline__ int x_scale_exp(const u32* emax_bits)
{
    const float emax = __uint_as_float(*emax_bits);
    if (!(emax > 0.0f) || !(emax < 3.0e38f)) return 0;
    int p;
    frexpf(emax, &p);
    return 9 - p;
}

// One 32 (patches) x 32 (right-hand sides) tile:
//   B[j][r] = E[j][r] + 2^-(g_exp + x_exp) * sum over the row block's slots of
//             the partials (slot order)
//   X^T[r][j] = head (+ tail) of 2^x_exp * albedo_j(r mod 3) * B[j][r], zero for
//             j >= n or r >= R
// The G operand holds 2^g_exp G, the X operand 2^x_exp X (exact scalings).
// B_out and xh may be null (not wanted); partial null means B = E.
//
// With few row blocks (small n) a row block has a dozen slots, and their sum is a
// chain of loads: SLOTS of them are in flight at a time, for PER elements per thread.
// err: the products' error word; after a failed product B_out is left alone. err_host:
// null, or host memory that the last call copies it to.
template <class T, int PER, int SLOTS>
__global__ void __launch_bounds__(1024 / PER) k_combine(u32 n, u32 ld, u32 R, u32 Rpad, const float* __restrict__ partial,
                                                        u32 max_slots, const u32* __restrict__ rp_cnt,
                                                        const float* __restrict__ E, const float* __restrict__ albedo,
                                                        float* __restrict__ B_out, T* __restrict__ xh, T* __restrict__ xl,
                                                        int g_exp, const u32* __restrict__ emax_bits, const u32* __restrict__ err,
                                                        u32* __restrict__ err_host)
{
    constexpr int ROWSTEP = 32 / PER;
    __shared__ float tile[32][33];
    const u32 j0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x_exp = x_scale_exp(emax_bits);
    const float unscale = ldexpf(1.0f, -(g_exp + x_exp)), xscale = ldexpf(1.0f, x_exp);
    const u32 failed = *err;
    const bool store = B_out && failed == 0u;
    if (err_host && blockIdx.x == 0 && blockIdx.y == 0 && tx == 0 && ty == 0) *err_host = failed;
    // the loads of the second phase (E, albedo) go out together with those of the first,
    // so a block waits for about one memory round trip instead of three
    float e[PER], al[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {   // tx along r
        const u32 j = j0 + ty + ROWSTEP * i, r = r0 + tx;
        const bool in = j < n && r < R;
        e[i] = in ? __ldg(&E[(size_t) j * R + r]) : 0.0f;
        al[i] = in ? __ldg(&albedo[3 * j + r % 3]) : 0.0f;
    }
    // the 32 patches of a tile lie in one 256-row block (j0 is a multiple of 32)
    const u32 rp = j0 / ROWS, cnt = (partial && j0 < n) ? __ldg(&rp_cnt[rp]) : 0u;
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = 0.0f;
    const size_t step = (size_t) R * ROWS;
    const float* P = partial + ((size_t) rp * max_slots * R + r0 + ty) * ROWS + (j0 + tx) % ROWS;   // tx along j
    for (u32 s = 0; s < cnt; s += SLOTS) {
        float q[SLOTS][PER];
#pragma unroll
        for (u32 u = 0; u < SLOTS; ++u)
#pragma unroll
            for (int i = 0; i < PER; ++i)
                q[u][i] = s + u < cnt && r0 + ty + ROWSTEP * i < R && j0 + tx < n
                              ? __ldg(P + (s + u) * step + ROWSTEP * i * ROWS) : 0.0f;
#pragma unroll
        for (u32 u = 0; u < SLOTS; ++u)
#pragma unroll
            for (int i = 0; i < PER; ++i)
                if (s + u < cnt) v[i] += q[u][i];
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) tile[ty + ROWSTEP * i][tx] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i) {   // tx along r
        const int k = ty + ROWSTEP * i;
        const u32 j = j0 + k, r = r0 + tx;
        float x = 0.0f;
        if (j < n && r < R) {
            const float b = e[i] + tile[tx][k] * unscale;
            if (store) B_out[(size_t) j * R + r] = b;
            x = al[i] * b * xscale;
        }
        tile[tx][k] = x;   // the element that this thread read
    }
    if (!xh) return;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i) {   // tx along j
        const int k = ty + ROWSTEP * i;
        const u32 r = r0 + k, j = j0 + tx;
        if (r < Rpad && j < ld) {
            const float w = tile[k][tx];
            const T h = to16<T>(w);
            xh[(size_t) r * ld + j] = h;
            if (xl) xl[(size_t) r * ld + j] = to16<T>(w - from16(h));
        }
    }
}

// ----------------------------------------------------------------------------- FP32 SIMT gather

// Partial sums of G X for FP32 (G n x n, row stride ldg a multiple of 4; X rows of ldr
// floats, zero past n and past R). Bound by the FP32 pipes (G streams at a fifth of
// HBM's rate), so the shape serves the multiply-adds:
//  * G lies k-contiguous in shared memory, X as it is, k by k (no transposition on the
//    way in); a thread owns 16 rows ty + 8 i and TN columns, four neighbours 4 tx .. of
//    each 64 and two of the last 32, and reads four k at a time, 16 + 8 loads of up to 16
//    bytes for 384 multiply-adds (TN = 6). A warp spans 4 x 8 threads, so with G's
//    rows padded to 36 floats its loads touch 4 rows on different banks, and 128
//    contiguous bytes of X. Neighbouring columns also keep an X value's register
//    bank the same for every k, so accumulators can sit in the other: with X
//    k-contiguous too, half the issue slots lost were register conflicts
//    (dispatch stalls 0.48 per instruction against 0.21, issue 73% against 79%).
//  * 128 x (16 TN) tiles, k blocks of 32 in three cp.async stages, 128 threads, two
//    blocks per SM.
//  * the (tile, k block) units are cut into equal contiguous ranges, one per
//    resident block, so the SMs stay filled whatever n and R are; a block writes the
//    sums of each tile it touches into its slot of that tile and k_combine32 adds
//    the slots in order (deterministic, and shorter sums than one range of n).
// TN by R (sgemm_tn): the least padding wins, with a charge per tile for G's re-read.
// Measured, n = 8192: R = 96 1541 -> 254 us a bounce with both operands k-contiguous and
// 241 now (54 TFLOP/s; the 128 x 192 tile on 64 blocks at first), R = 192 515 -> 472.
// Tried: fma.rn.f32x2 on column pairs 252 and 496 (its 64-bit operands cost the
// register ports what it saves in issue slots), on k pairs 46 TFLOP/s; 8 x 6 and 8 x 12
// per thread 47 and 49.
constexpr int SGM = 128, SGK = 32, SGS = SGK + 4, SGStages = 3, SGThreads = 128, SGBlocksPerSM = 2;

struct SgemmArgs {
    u32 n, ldg, ldr, nkb;     // rows, strides of G and X, k blocks
    u32 tiles_n, max_slots;
    uint64_t total;           // (tile, k block) units
    const float* G;
    const float* X;           // [k][ldr], zero rows up to nkb SGK
    float* partial;           // [tile][slot][SGM][16 TN]
};

// Which of `n_cta` equal ranges of `total` units holds unit u.
__host__ __device__ __forceinline__ u32 range_of(uint64_t u, uint64_t total, u32 n_cta)
{
    return (u32) (((u + 1) * n_cta + total - 1) / total - 1);
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

__device__ __forceinline__ float f4at(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// FEW: fewer patches than a tile has rows; those past n are not written (8 patches, 100,000
// right-hand sides, three bounces: 0.181 -> 0.144 ms; the test costs a full tile 1%).
template <int TN, bool FEW>
__global__ void __launch_bounds__(SGThreads, SGBlocksPerSM) k_sgemm_bounce(SgemmArgs a)
{
    constexpr int BN = 16 * TN, TM = SGM / 8, STAGE = SGM * SGS + SGK * BN, CG = SGM / 16;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int ty = (w >> 1) * 4 + (lane >> 3), tx = (w & 1) * 8 + (lane & 7);
    const uint64_t lo = (uint64_t) blockIdx.x * a.total / gridDim.x, hi = (uint64_t) (blockIdx.x + 1) * a.total / gridDim.x;
    // copies: 8 chunks of 16 bytes per row of a stage; this thread's are rows tid / 8 + 16 t
    const int cr = tid >> 3, cc = (tid & 7) * 4;
    u32 ft = (u32) (lo / a.nkb), fk = (u32) (lo % a.nkb);   // the next unit to fetch
    const float* gp[CG];
    bool gin[CG];
    const float* xp;
    // X rows of BN floats: chunks tid + 128 t of the stage's SGK x BN / 4
    u32 xoff[TN];
#pragma unroll
    for (int t = 0; t < TN; ++t) {
        const u32 c = tid + SGThreads * t;
        xoff[t] = c / (BN / 4) * a.ldr + c % (BN / 4) * 4;
    }
    auto seek = [&]() {
        const u32 m0 = ft / a.tiles_n * SGM, n0 = ft % a.tiles_n * BN;
#pragma unroll
        for (int t = 0; t < CG; ++t) {
            const u32 m = m0 + cr + 16 * t;
            gin[t] = m < a.n;
            gp[t] = a.G + (gin[t] ? (size_t) m * a.ldg : 0) + fk * SGK + cc;
        }
        xp = a.X + (size_t) fk * SGK * a.ldr + n0;
    };
    seek();
    auto fetch = [&](int stage) {
        float* S = sm + stage * STAGE + cr * SGS + cc;
        float* SX = sm + stage * STAGE + SGM * SGS + 4 * tid;
        const bool kin = fk * SGK + cc < a.ldg;
#pragma unroll
        for (int t = 0; t < CG; ++t) {
            cp16(S + 16 * t * SGS, gin[t] && kin ? gp[t] : a.G, gin[t] && kin);
            gp[t] += SGK;
        }
#pragma unroll
        for (int t = 0; t < TN; ++t) cp16(SX + 4 * SGThreads * t, xp + xoff[t], true);
        xp += (size_t) SGK * a.ldr;
        if (++fk == a.nkb) {
            fk = 0;
            ++ft;
            seek();
        }
    };
    // this thread's column j of the tile: four and two neighbouring ones
    auto col = [&](int j) { return j < (TN & ~3) ? 16 * (j & ~3) + 4 * tx + (j & 3) : 16 * (TN & ~3) + 2 * tx + (j & 1); };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
#pragma unroll
    for (int q = 0; q < SGStages - 1; ++q) {
        if (lo + q < hi) fetch(q);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    u32 ct = (u32) (lo / a.nkb), ck = (u32) (lo % a.nkb);   // the unit being summed
    for (uint64_t u = lo; u < hi; ++u) {
        asm volatile("cp.async.wait_group %0;" ::"n"(SGStages - 2) : "memory");
        __syncthreads();   // stage `stage` has landed, and everyone is done with the one refilled here
        if (u + SGStages - 1 < hi) fetch(stage == 0 ? SGStages - 1 : stage - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* As = sm + stage * STAGE + ty * SGS;
        const float* Bs = sm + stage * STAGE + SGM * SGS;
#pragma unroll 4
        for (int k = 0; k < SGK; k += 4) {
            float b[4][TN];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
#pragma unroll
                for (int j = 0; j + 4 <= TN; j += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(Bs + (k + h) * BN + 16 * j + 4 * tx);
                    b[h][j] = v.x; b[h][j + 1] = v.y; b[h][j + 2] = v.z; b[h][j + 3] = v.w;
                }
                if (TN % 4) {
                    const float2 v = *reinterpret_cast<const float2*>(Bs + (k + h) * BN + 16 * (TN & ~3) + 2 * tx);
                    b[h][TN - 2] = v.x; b[h][TN - 1] = v.y;
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 av = *reinterpret_cast<const float4*>(As + 8 * i * SGS + k);
#pragma unroll
                for (int h = 0; h < 4; ++h)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = __fmaf_rn(f4at(av, h), b[h][j], acc[i][j]);
            }
        }
        stage = stage + 1 == SGStages ? 0 : stage + 1;
        ++ck;
        if (u + 1 == hi || ck == a.nkb) {   // the end of this block's part of the tile
            const u32 slot = blockIdx.x - range_of((uint64_t) ct * a.nkb, a.total, gridDim.x);
            float* P = a.partial + ((size_t) ct * a.max_slots + slot) * (SGM * BN);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    if (!FEW || ty + 8 * i < a.n) P[(ty + 8 * i) * BN + col(j)] = acc[i][j];
                    acc[i][j] = 0.0f;
                }
            ck = 0;
            ++ct;
        }
    }
}

// A bounce's sums: B = E + the tile's slots in order (no slots: B = E), and the next
// X[j][r] = albedo_j(r mod 3) B (rows of ldr), zero for j >= n or r >= R. B_out and x
// may be null (not wanted); E and B_out have rows of ldb floats. 32 right-hand sides (along the grid's x,
// which has room for any number) x 8 patches (y: as many as a matrix in device memory has) per block.
__global__ void __launch_bounds__(256) k_combine32(u32 n, u32 ldx, u32 ldr, u32 ldb, u32 R, u32 BN, u32 tiles_n, u32 nkb, uint64_t total,
                                                   u32 n_cta, u32 max_slots, const float* __restrict__ partial,
                                                   const float* __restrict__ E, const float* __restrict__ albedo,
                                                   float* __restrict__ B_out, float* __restrict__ x_out)
{
    const u32 j = blockIdx.y * 8 + threadIdx.y, r0 = blockIdx.x * 32, r = r0 + threadIdx.x;
    float x = 0.0f;
    if (j < n && r < R) {
        const float e = __ldg(&E[(size_t) j * ldb + r]), al = __ldg(&albedo[3 * j + r % 3]);
        float v = 0.0f;
        if (partial) {
            // 8 divides the tile's rows and 32 its BN columns: one product tile for the block
            const u32 t = j / SGM * tiles_n + r0 / BN;
            const u32 cnt = range_of((uint64_t) (t + 1) * nkb - 1, total, n_cta) - range_of((uint64_t) t * nkb, total, n_cta) + 1;
            const float* P = partial + (size_t) t * max_slots * (SGM * BN) + (size_t) (j % SGM) * BN + r % BN;
            for (u32 s = 0; s < cnt; s += 4) {   // four slots in flight
                float q[4];
#pragma unroll
                for (u32 u = 0; u < 4; ++u) q[u] = s + u < cnt ? __ldg(&P[(size_t) (s + u) * (SGM * BN)]) : 0.0f;
#pragma unroll
                for (u32 u = 0; u < 4; ++u)
                    if (s + u < cnt) v += q[u];
            }
        }
        const float b = e + v;
        if (B_out) B_out[(size_t) j * ldb + r] = b;
        x = al * b;
    }
    if (x_out && j < ldx) x_out[(size_t) j * ldr + r] = x;
}

// Column groups of 16 per tile (TN of k_sgemm_bounce) for R right-hand sides: the
// least ceil(R / BN) (BN + 24). The 24 columns per tile stand for reading G once more.
int sgemm_tn(u32 R)
{
    int best = 6;
    u32 cost = UINT32_MAX;
    for (int tn : {6, 4, 2}) {
        const u32 bn = 16 * (u32) tn, c = (R + bn - 1) / bn * (bn + 24);
        if (c < cost) { cost = c; best = tn; }
    }
    return best;
}

// Right-hand sides solved at a time: the most whose slots (two per tile where there are
// many) and X take 1 GiB, so that a solve of any width needs little beside its own arrays.
// A multiple of 96, which keeps the columns' albedo channels (r mod 3) and whole tiles.
u32 sgemm_columns(u32 tiles_m, u32 ldx)
{
    const uint64_t per96 = (2ull * tiles_m * SGM + ldx) * 96 * 4;
    return 96 * (u32) std::max<uint64_t>(1, std::min<uint64_t>((1ull << 30) / per96, 40000000));
}

// ----------------------------------------------------------------------------- G preparation

// G_ij = F_ij * area_j, in place, and *out = max G_ij as float bits (non-negative
// floats order like their bits; *out starts at 0). Rows of ldg floats, a multiple of
// 4; the padding columns stay 0. One pass over G, 16 bytes at a time (as two passes
// of single floats with a 64-bit remainder each, 4,096 patches took 81 us).
__global__ void __launch_bounds__(256) k_scale_cols(u32 n, u32 ldg, float* __restrict__ G, const float* __restrict__ area, u32* out)
{
    float m = 0.0f;
    for (u32 i = blockIdx.x; i < n; i += gridDim.x) {
        float4* row = reinterpret_cast<float4*>(G + (size_t) i * ldg);
        for (u32 c = threadIdx.x; c < ldg / 4; c += 256) {
            float4 g = row[c];
            const u32 j = 4 * c;
            g.x *= __ldg(&area[j]);   // j < n: the padding is less than four columns
            if (j + 1 < n) g.y *= __ldg(&area[j + 1]);
            if (j + 2 < n) g.z *= __ldg(&area[j + 2]);
            if (j + 3 < n) g.w *= __ldg(&area[j + 3]);
            row[c] = g;
            m = fmaxf(m, fmaxf(fmaxf(fabsf(g.x), fabsf(g.y)), fmaxf(fabsf(g.z), fabsf(g.w))));
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(out, __float_as_uint(m));
}

// The right-hand sides on their way in: *out = max |x| as float bits (*out starts at
// 0) and, with copy, copy = x; with alb, alb_copy = alb (na floats). x and alb are
// then the caller's host arrays where kernels can address pageable host memory
// (cudaDevAttrPageableMemoryAccess, e.g. Grace systems: the GPU walks the host page
// tables over the CPU-GPU link). 16-byte vectors when both sides are aligned.
__device__ __forceinline__ float copy_max(const float* __restrict__ x, float* __restrict__ copy, size_t count)
{
    float m = 0.0f;
    const size_t stride = (size_t) gridDim.x * blockDim.x, t0 = blockIdx.x * (size_t) blockDim.x + threadIdx.x;
    size_t t = t0;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(copy)) & 15u) == 0) {
        for (size_t k = t0; k < count / 4; k += stride) {
            const float4 v = reinterpret_cast<const float4*>(x)[k];
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
            if (copy) reinterpret_cast<float4*>(copy)[k] = v;
        }
        t = count / 4 * 4 + t0;
    }
    for (; t < count; t += stride) {
        const float v = x[t];
        m = fmaxf(m, fabsf(v));
        if (copy) copy[t] = v;
    }
    return m;
}

__global__ void __launch_bounds__(256) k_take_in(const float* __restrict__ x, float* __restrict__ copy, size_t count,
                                                 const float* __restrict__ alb, float* __restrict__ alb_copy, size_t na,
                                                 u32* out)
{
    if (alb) copy_max(alb, alb_copy, na);
    float m = copy_max(x, copy, count);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(out, __float_as_uint(m));
}

// hi = 16-bit 2^g_exp G (row stride ld, zero columns j >= n); lo = 16-bit residual when requested.
// Four columns per thread: 16 bytes in, 8 out.
template <class T>
__global__ void __launch_bounds__(256) k_g_to_16(u32 n, u32 ld, u32 ldg, const float* __restrict__ G, T* __restrict__ hi,
                                                 T* __restrict__ lo, float gscale)
{
    for (u32 i = blockIdx.x; i < n; i += gridDim.x) {
        const float4* row = reinterpret_cast<const float4*>(G + (size_t) i * ldg);
        for (u32 c = threadIdx.x; c < ld / 4; c += 256) {
            const float4 g = 4 * c < ldg ? __ldcs(&row[c]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float v[4] = {g.x * gscale, g.y * gscale, g.z * gscale, g.w * gscale};
            alignas(8) T h[4], l[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                h[k] = to16<T>(v[k]);
                l[k] = to16<T>(v[k] - from16(h[k]));
            }
            reinterpret_cast<uint2*>(hi + (size_t) i * ld)[c] = *reinterpret_cast<const uint2*>(h);
            if (lo) reinterpret_cast<uint2*>(lo + (size_t) i * ld)[c] = *reinterpret_cast<const uint2*>(l);
        }
    }
}

// ----------------------------------------------------------------------------- host helpers

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000) p;
    });
    if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// 2-D map over `rows` rows of `ld` 16-bit elements (row stride ld * 2 bytes,
// a multiple of 128), box of 64 elements (128 bytes) x box_rows, 128-byte
// swizzle; rows past the end read as zero.
CUtensorMap make_map(const void* ptr, CUtensorMapDataType dt, u32 ld, u32 rows, u32 box_rows, u32 box_k)
{
    if ((reinterpret_cast<uintptr_t>(ptr) & 127) || (ld % BK) || box_rows == 0 || box_rows > 256 ||
        (box_k != 64 && box_k != 32))
        throw std::runtime_error("tensor map: misaligned base, row length or box");
    CUtensorMap m;
    cuuint64_t dims[2] = {ld, rows};
    cuuint64_t strides[1] = {(cuuint64_t) ld * 2};
    cuuint32_t box[2] = {(cuuint32_t) box_k, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             box_k == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed with " + std::to_string((int) r));
    return m;
}

// How a product runs, from the refine level and the MMA N (measured on GB300, us per
// product of 32,768 patches unless noted).
//
// k per stage: 64 for one and two products on single CTAs (R = 192: 360 and 538 against
// 363 and 462 with 32, R = 3: 320 and 328 against 315 and 353; where 64 leaves two
// stages, pairs are taken instead, below); 32 for three products, whose stages hold
// two G tiles and two X tiles (R = 192: 691 against 746; it also lets that mode take
// R = 256).
//
// Pairs of CTAs with split right-hand sides, where a single CTA has room for two stages
// only (N > 160), from 16 units per SM on: R = 192, one CTA / pair: 538 / 430, 8,192
// patches 46.0 / 41.9, 6,000 30.6 / 30.5, 4,096 20.8 / 22.8; R = 256: 675 / 547, 4,096
// patches 25.5 / 27.2. With three stages or more both are the same at large sizes
// (R = 144: 386 / 390) and a pair's start and end cost a microsecond or two at small
// ones. A pair's stages are 32 wide (R = 192, 256: 430, 547; 64 wide 438, 565).
struct GatherPlan {
    bool pair;
    u32 kb, stages, stage_bytes;
};
GatherPlan gather_plan(int refine, u32 bn, uint64_t units, int sm_count)
{
    auto stage = [&](u32 kb, u32 ctas) {
        return (refine == LTRG_REFINE_FULL ? 2u : 1u) * ROWS * kb * 2 + (refine >= LTRG_REFINE_RHS ? 2u : 1u) * (bn / ctas) * kb * 2;
    };
    GatherPlan p;
    p.kb = refine == LTRG_REFINE_FULL ? 32u : 64u;
    p.pair = refine == LTRG_REFINE_RHS && 3 * stage(p.kb, 1) + kSmemExtra > (u32) kSmemLimit && units >= 16ull * (u32) sm_count;
    if (p.pair) p.kb = 32;
    p.stage_bytes = stage(p.kb, p.pair ? 2 : 1);
    p.stages = std::min<u32>(kMaxStages, (kSmemLimit - kSmemExtra) / p.stage_bytes);
    return p;
}

// Device buffer from the device's memory pool (which the bakes keep filled between
// objects, see keep_pool_memory: mapping and unmapping a gather's matrices took
// most of a millisecond), allocated and freed on the gather's stream.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    bool ensure(size_t b, cudaStream_t st)   // whether it was allocated anew
    {
        if (b <= bytes) return false;
        release(st);
        GCK(cudaMallocAsync(&p, b, st));
        bytes = b;
        return true;
    }
    void release(cudaStream_t st)
    {
        if (p) cudaFreeAsync(p, st);
        p = nullptr;
        bytes = 0;
    }
    template <class T> T* as() const { return reinterpret_cast<T*>(p); }
};

// Page-locked host buffer kept by a gather (grown, never shrunk).
struct PinBuf {
    void* p = nullptr;
    size_t bytes = 0;
    void ensure(size_t b)
    {
        if (b <= bytes) return;
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
        GCK(cudaHostAlloc(&p, b, cudaHostAllocPortable));
        bytes = b;
    }
    void release()
    {
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
    }
};

// Whether kernels on `device` may address pageable host memory (queried once).
bool pageable_access(int device)
{
    static std::mutex mu;
    static int known[64] = {};   // 0 unknown, 1 no, 2 yes
    if (device < 0 || device >= 64) return false;
    std::lock_guard<std::mutex> lk(mu);
    if (!known[device]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccess, device) != cudaSuccess) v = 0;
        known[device] = v ? 2 : 1;
    }
    return known[device] == 2;
}

// Host threads kept by a gather for its host-buffer copies: run(k, f) calls
// f(0 .. k-1) on the workers (and the caller) and returns when all are done.
struct StagePool {
    std::vector<std::thread> th;
    std::mutex mu;
    std::condition_variable cv_go, cv_done;
    std::function<void(int)> job;
    int n_job = 0, next = 0, done = 0;
    unsigned long long gen = 0;
    bool quit = false;

    void start(int workers)
    {
        for (int w = 0; w < workers; ++w)
            th.emplace_back([this]() {
                unsigned long long seen = 0;
                std::unique_lock<std::mutex> lk(mu);
                for (;;) {
                    cv_go.wait(lk, [&] { return quit || gen != seen; });
                    if (quit) return;
                    seen = gen;
                    drain(lk);
                }
            });
    }
    // takes items until none are left; called with the lock held
    void drain(std::unique_lock<std::mutex>& lk)
    {
        while (next < n_job) {
            const int t = next++;
            lk.unlock();
            job(t);
            lk.lock();
            if (++done == n_job) cv_done.notify_all();
        }
    }
    void run(int k, std::function<void(int)> f)
    {
        std::unique_lock<std::mutex> lk(mu);
        job = std::move(f);
        n_job = k;
        next = done = 0;
        ++gen;
        cv_go.notify_all();
        drain(lk);
        cv_done.wait(lk, [&] { return done == n_job; });
    }
    ~StagePool()
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            quit = true;
        }
        cv_go.notify_all();
        for (auto& t : th) t.join();
    }
};

// Host <-> device copies of the host-buffer entry point through kept
// page-locked buffers. A copy straight from the caller's pageable memory runs
// at about 10 GB/s; here the bytes are cut into slices, the pool's threads
// copy the slices into the page-locked buffer and each queues its slice's
// DMA at once, so the DMA of early slices overlaps the host copies of later
// ones (and the reverse for the result: each slice's DMA is followed by an
// event its thread waits on before copying the slice out).
constexpr size_t kStageMinSlice = 1 << 20;

int stage_slices(size_t bytes, int threads)
{
    return (int) std::max<size_t>(1, std::min<size_t>((size_t) threads, bytes / kStageMinSlice));
}

void stage_h2d(void* dev, const void* host, size_t bytes, PinBuf& pin, cudaStream_t s, StagePool& pool, int threads)
{
    if (!bytes) return;
    pin.ensure(bytes);
    const int k = stage_slices(bytes, threads);
    const size_t step = (bytes / k + 255) / 256 * 256;
    std::vector<cudaError_t> rc(k, cudaSuccess);
    pool.run(k, [&](int t) {
        const size_t a = std::min(bytes, t * step), b = std::min(bytes, a + step);
        if (a >= b) return;
        memcpy((char*) pin.p + a, (const char*) host + a, b - a);
        rc[t] = cudaMemcpyAsync((char*) dev + a, (char*) pin.p + a, b - a, cudaMemcpyHostToDevice, s);
    });
    for (cudaError_t e : rc) GCK(e);
}

void stage_d2h(void* host, const void* dev, size_t bytes, PinBuf& pin, cudaStream_t s, StagePool& pool, int threads)
{
    if (!bytes) return;
    pin.ensure(bytes);
    const int k = stage_slices(bytes, threads);
    const size_t step = (bytes / k + 255) / 256 * 256;
    std::vector<cudaEvent_t> ev(k, nullptr);
    for (int t = 0; t < k; ++t) {
        const size_t a = std::min(bytes, t * step), b = std::min(bytes, a + step);
        GCK(cudaEventCreateWithFlags(&ev[t], cudaEventDisableTiming));
        if (a < b) GCK(cudaMemcpyAsync((char*) pin.p + a, (const char*) dev + a, b - a, cudaMemcpyDeviceToHost, s));
        GCK(cudaEventRecord(ev[t], s));
    }
    std::vector<cudaError_t> rc(k, cudaSuccess);
    pool.run(k, [&](int t) {
        const size_t a = std::min(bytes, t * step), b = std::min(bytes, a + step);
        rc[t] = cudaEventSynchronize(ev[t]);
        if (rc[t] == cudaSuccess && a < b) memcpy((char*) host + a, (const char*) pin.p + a, b - a);
    });
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
    for (cudaError_t e : rc) GCK(e);
}

}  // namespace
}  // namespace lg

using namespace lg;

struct ltrg_Gather {
    int device = 0;
    int sm_count = 0;
    cudaStream_t st = nullptr;
    u32 n = 0, ld = 0;
    u32 ldg = 0;                  // row stride of G32: n rounded up to 4 floats (16-byte rows), zeros past n
    DevBuf G32;                   // n x ldg FP32
    DevBuf G16, G16lo;            // n x ld 16-bit head and residual
    int g16_kind = -1;            // precision held in G16 (-1: none)
    int g_exp = 0;                // G16 holds 2^g_exp G: max |G| maps below 2^14
    bool g16_has_lo = false;
    // stream-K schedule of the tcgen05 kernel (fixed by n and the SM count)
    u32 n_rp = 0, nkb = 0;
    u32 n_ranges[2] = {}, max_slots[2] = {};   // stream-K ranges and most slots of a row block: single CTAs, pairs
    u32 kchunk = 0;               // k blocks per TMEM accumulation (0: whole range of a CTA)
    DevBuf rp_tab;                // rp_first[n_rp], rp_cnt[n_rp] of single CTAs, then of pairs
    // solve scratch
    DevBuf partial, xh, xl, x32;
    DevBuf words;                 // [0] error word of the products, [1] largest emission
    DevBuf h_alb, h_E, h_out;     // device copies for the host-buffer entry point
    PinBuf pin_in, pin_out;       // its page-locked staging
    u32 h_err = 0;                // the error word as read back
    std::vector<cudaEvent_t> events;   // of a solve's timings, used again by the next
    bool grown = false;           // a buffer was allocated since the last wait for `st`
    std::unique_ptr<StagePool> pool;   // its host copy threads (started by the first host-buffer solve)
    int pool_threads = 0;
    uint64_t links = 0, vis_rays = 0, pairs = 0;
    double ms_build = 0;
    u32 stall_us = 0;             // ltrdbg_GatherStallNextSolve
    int host_path = 0;            // ltrdbg_GatherHostPath: 0 by device, 1 staged, 2 direct
    std::string error;
    std::mutex mu;

    ~ltrg_Gather()
    {
        if (!st) return;
        cudaSetDevice(device);
        cudaStreamSynchronize(st);
        DevBuf* all[] = {&G32, &G16, &G16lo, &rp_tab, &partial, &xh, &xl, &x32, &words, &h_alb, &h_E, &h_out};
        for (DevBuf* b : all) b->release(st);
        for (cudaEvent_t e : events) cudaEventDestroy(e);
        pin_in.release();
        pin_out.release();
        cudaStreamSynchronize(st);
        // as a destroyed scene does: the pool gives back what it holds beyond 8 GiB
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, device) != cudaSuccess || cudaMemPoolTrimTo(pool, 8ull << 30) != cudaSuccess)
            (void) cudaGetLastError();
        cudaStreamDestroy(st);
    }

    void need(DevBuf& b, size_t bytes)
    {
        if (b.ensure(bytes, st)) grown = true;
    }

    void schedule()
    {
        n_rp = (n + ROWS - 1) / ROWS;
        nkb = ld / BK;
        std::vector<u32> tab;
        for (u32 ctas = 1; ctas <= 2; ++ctas) {
            const uint64_t total = (uint64_t) ((n_rp + ctas - 1) / ctas) * nkb;
            const u32 ranges = (u32) std::min<uint64_t>((uint64_t) sm_count / ctas, total);
            std::vector<u32> first(n_rp, UINT32_MAX), cnt(n_rp, 0);
            u32 most = 0;
            for (u32 c = 0; c < ranges; ++c) {
                const uint64_t lo = (uint64_t) c * total / ranges, hi = (uint64_t) (c + 1) * total / ranges;
                if (hi <= lo) continue;
                for (uint64_t ru = lo / nkb; ru <= (hi - 1) / nkb; ++ru)
                    for (u32 rp = (u32) ru * ctas; rp < std::min<u32>(n_rp, ((u32) ru + 1) * ctas); ++rp) {
                        if (first[rp] == UINT32_MAX) first[rp] = c;
                        cnt[rp] = c - first[rp] + 1;
                        most = std::max(most, cnt[rp]);
                    }
            }
            n_ranges[ctas - 1] = ranges;
            max_slots[ctas - 1] = most;
            tab.insert(tab.end(), first.begin(), first.end());
            tab.insert(tab.end(), cnt.begin(), cnt.end());
        }
        need(rp_tab, tab.size() * 4);
        GCK(cudaMemcpyAsync(rp_tab.p, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice, st));
        GCK(cudaStreamSynchronize(st));
    }

    // B for R right-hand sides, enqueued on `s`; all pointers are addressable by this
    // device's kernels. alb_host/E_host (or null): host arrays to be copied to alb
    // and E first, by kernels; `out` may then be a host array too.
    void solve(float* alb, float* E, u32 R, int bounces, int precision, int refine, float* out, ltrg_GatherStats* stats,
               cudaStream_t s, const float* alb_host = nullptr, const float* E_host = nullptr);
};

void ltrg_Gather::solve(float* alb, float* E, u32 R, int bounces, int precision, int refine, float* out,
                        ltrg_GatherStats* stats, cudaStream_t s, const float* alb_host, const float* E_host)
{
    const bool tc = precision != LTRG_F_FP32;
    if (tc && R > (u32) MAX_BN) throw std::runtime_error("tensor-core gather takes at most 256 right-hand sides");
    if (refine < LTRG_REFINE_NONE || refine > LTRG_REFINE_FULL) throw std::runtime_error("invalid refine level");
    need(words, 8);
    u32* d_err = words.as<u32>();
    u32* d_emax = words.as<u32>() + 1;
    size_t ev_used = 0;
    auto event = [&]() {
        if (ev_used == events.size()) {
            cudaEvent_t e;
            GCK(cudaEventCreate(&e));
            events.push_back(e);
        }
        GCK(cudaEventRecord(events[ev_used], s));
        return events[ev_used++];
    };
    // buffers allocated on the gather's stream are used on `s`
    auto begin = [&]() {
        if (grown) {
            GCK(cudaStreamSynchronize(st));
            grown = false;
        }
        GCK(cudaMemsetAsync(words.p, 0, 8, s));
        if (tc || E_host) {
            const size_t count = (size_t) n * R;
            k_take_in<<<(unsigned) std::min<size_t>((size_t) sm_count * 8, (count + 1023) / 1024), 256, 0, s>>>(
                E_host ? E_host : E, E_host ? E : nullptr, count, alb_host, alb, (size_t) n * 3, d_emax); note_launch();
            GCK(cudaGetLastError());
        }
    };
    // nothing of a solve that ends by an exception runs on after it
    struct Wait {
        cudaStream_t s;
        bool on;
        ~Wait() { if (on) cudaStreamSynchronize(s); }
    } wait{s, true};
    // the end of a solve: one wait, after which the products' error word is on the host
    // (the last slot sum wrote it there where the device can)
    const bool err_direct = tc && pageable_access(device);
    auto finish = [&]() {
        if (tc && !err_direct) GCK(cudaMemcpyAsync(&h_err, d_err, 4, cudaMemcpyDeviceToHost, s));
        GCK(cudaStreamSynchronize(s));
        wait.on = false;
        if (tc && h_err)
            throw std::runtime_error("tensor-core gather: a pipeline wait expired (error word " + std::to_string(h_err) + ")");
    };
    double ms_convert = 0, ms_gemm = 0, ms_bounces = 0;
    int stages = 0, products = 1;
    int32_t ctas_run = 0;
    uint64_t bytes_bounce = 0;

    if (!tc) {
        const u32 tiles_m = (n + SGM - 1) / SGM, skb = (ldg + SGK - 1) / SGK, ldx = skb * SGK;
        const u32 wide = sgemm_columns(tiles_m, ldx);
        struct Run {   // the solve of `w` right-hand sides
            u32 w;
            int tn;
            u32 bn, tiles_n, sg_cta, slots;
            uint64_t total;
        };
        auto run_of = [&](u32 w) {
            Run q;
            q.w = w;
            q.tn = sgemm_tn(w);
            q.bn = 16 * (u32) q.tn;
            q.tiles_n = (w + q.bn - 1) / q.bn;
            q.total = (uint64_t) tiles_m * q.tiles_n * skb;
            q.sg_cta = (u32) std::min<uint64_t>((uint64_t) sm_count * SGBlocksPerSM, q.total);
            // slots: the most ranges that one tile's units can fall into
            q.slots = (u32) std::min<uint64_t>(q.sg_cta, ((uint64_t) skb * q.sg_cta + q.total - 1) / q.total + 1);
            return q;
        };
        for (const Run& q : {run_of(std::min(R, wide)), run_of(R > wide && R % wide ? R % wide : std::min(R, wide))}) {
            need(partial, (size_t) tiles_m * q.tiles_n * q.slots * SGM * q.bn * 4);
            need(x32, (size_t) q.tiles_n * q.bn * ldx * 4);
        }
        begin();
        cudaEvent_t e0 = event();
        std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ge;
        for (u32 c = 0; c < R; c += std::min(R - c, wide)) {
            const Run q = run_of(std::min(R - c, wide));
            const u32 ldr = q.tiles_n * q.bn;
            auto combine = [&](bool with_partial, bool last) {
                const u32 rows = with_partial ? n : ldx;   // X's rows past n are zero from the first call on
                const dim3 grid(ldr / 32, (rows + 7) / 8), block(32, 8);
                k_combine32<<<grid, block, 0, s>>>(n, rows, ldr, R, q.w, q.bn, q.tiles_n, skb, q.total, q.sg_cta, q.slots,
                                                   with_partial ? partial.as<float>() : nullptr, E + c, alb,
                                                   last ? out + c : nullptr, last ? nullptr : x32.as<float>()); note_launch();
                GCK(cudaGetLastError());
            };
            const SgemmArgs sa{n, ldg, ldr, skb, q.tiles_n, q.slots, q.total, G32.as<float>(), x32.as<float>(), partial.as<float>()};
            auto kern = n < SGM ? (q.tn == 6 ? k_sgemm_bounce<6, true> : q.tn == 4 ? k_sgemm_bounce<4, true> : k_sgemm_bounce<2, true>)
                                : (q.tn == 6 ? k_sgemm_bounce<6, false> : q.tn == 4 ? k_sgemm_bounce<4, false> : k_sgemm_bounce<2, false>);
            const size_t sg_smem = (size_t) SGStages * (SGM * SGS + SGK * q.bn) * 4;
            GCK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sg_smem));
            ctas_run = (int32_t) q.sg_cta;
            combine(false, bounces == 0);
            for (int b = 0; b < bounces; ++b) {
                cudaEvent_t g0 = event();
                kern<<<q.sg_cta, SGThreads, sg_smem, s>>>(sa); note_launch();
                cudaEvent_t g1 = event();
                ge.push_back({g0, g1});
                GCK(cudaGetLastError());
                combine(true, b + 1 == bounces);
            }
        }
        cudaEvent_t e1 = event();
        finish();
        float m = 0;
        cudaEventElapsedTime(&m, e0, e1);
        ms_bounces = m;
        for (auto& p : ge) { cudaEventElapsedTime(&m, p.first, p.second); ms_gemm += m; }
        bytes_bounce = (uint64_t) n * n * 4;
    } else {
        const bool need_lo = refine == LTRG_REFINE_FULL;
        const u32 BN = std::max<u32>(32, (R + 31) / 32 * 32);
        const GatherPlan plan = gather_plan(refine, BN, (uint64_t) n_rp * nkb, sm_count);
        const bool pair = plan.pair;
        const u32 KB = plan.kb, ctas = pair ? 2 : 1, slots_max = max_slots[pair];
        const u32 stage_bytes = plan.stage_bytes;
        stages = (int) plan.stages;
        if (stages < 2) throw std::runtime_error("tensor-core gather: stage does not fit in shared memory");
        const size_t smem = (size_t) stages * stage_bytes + kSmemExtra;
        products = 1 + (refine >= LTRG_REFINE_RHS) + (refine == LTRG_REFINE_FULL);
        // every element of X^T (padding included) is written by the first k_combine
        need(G16, (size_t) n * ld * 2);
        if (need_lo) need(G16lo, (size_t) n * ld * 2);
        need(xh, (size_t) BN * ld * 2);
        need(xl, (size_t) BN * ld * 2);
        need(partial, (size_t) n_rp * slots_max * R * ROWS * 4);
        begin();
        cudaEvent_t c0 = nullptr, c1 = nullptr;
        if (g16_kind != precision || (need_lo && !g16_has_lo)) {
            c0 = event();
            const unsigned grid = (unsigned) std::min<u32>(n, (u32) sm_count * 8);
            const float gscale = ldexpf(1.0f, g_exp);
            if (precision == LTRG_F_FP16)
                k_g_to_16<__half><<<grid, 256, 0, s>>>(n, ld, ldg, G32.as<float>(), G16.as<__half>(),
                                                       need_lo ? G16lo.as<__half>() : nullptr, gscale);
            else
                k_g_to_16<__nv_bfloat16><<<grid, 256, 0, s>>>(n, ld, ldg, G32.as<float>(), G16.as<__nv_bfloat16>(),
                                                              need_lo ? G16lo.as<__nv_bfloat16>() : nullptr, gscale);
            note_launch();
            GCK(cudaGetLastError());
            c1 = event();
            g16_kind = -1;   // until the conversion is known to be done
        }
        const CUtensorMapDataType dt =
            precision == LTRG_F_FP16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const CUtensorMap mG = make_map(G16.p, dt, ld, n, ROWS, KB);
        const CUtensorMap mGl = make_map(need_lo ? G16lo.p : G16.p, dt, ld, n, ROWS, KB);
        const CUtensorMap mXh = make_map(xh.p, dt, ld, BN, BN / ctas, KB);
        const CUtensorMap mXl = make_map(xl.p, dt, ld, BN, BN / ctas, KB);
        auto kern = refine == LTRG_REFINE_NONE   ? k_umma_gather<64, 1, LTRG_REFINE_NONE>
                    : refine == LTRG_REFINE_FULL ? k_umma_gather<32, 1, LTRG_REFINE_FULL>
                    : pair                       ? k_umma_gather<32, 2, LTRG_REFINE_RHS>
                                                 : k_umma_gather<64, 1, LTRG_REFINE_RHS>;
        // the limit is the kernel's, and other gathers' threads set it too: always the same value
        GCK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
        UmmaArgs ua;
        ua.nkb = nkb; ua.n_rp = n_rp; ua.R = R; ua.BN = BN;
        ua.stages = (u32) stages; ua.stage_bytes = stage_bytes;
        ua.idesc = idesc_f16(precision == LTRG_F_BF16 ? 1u : 0u, BM * ctas, BN);
        ua.max_slots = slots_max;
        ua.kchunk = kchunk;
        ua.rp_first = rp_tab.as<u32>() + (pair ? 2 * n_rp : 0);
        ua.partial = partial.as<float>();
        ua.err = d_err;
        ua.wait_cycles = kWaitCycles;
        ua.issue = 1;
        if (stall_us) {   // test hook: copies never issued, waits cut short
            ua.issue = 0;
            ua.wait_cycles = (unsigned long long) stall_us * 2000ull;
            stall_us = 0;
        }
        const u32* rp_cnt = ua.rp_first + n_rp;
        cudaLaunchConfig_t lc = {};
        cudaLaunchAttribute la[1];
        la[0].id = cudaLaunchAttributeClusterDimension;
        la[0].val.clusterDim.x = ctas;
        la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
        lc.gridDim = dim3(n_ranges[pair] * ctas);
        lc.blockDim = dim3(kThreads);
        lc.dynamicSmemBytes = smem;
        lc.stream = s;
        lc.attrs = la;
        lc.numAttrs = 1;
        ctas_run = (int32_t) lc.gridDim.x;
        // Up to one tile per SM, a block's own chain of slots is the time: one element per
        // thread, eight slots in flight (1,500 patches, R = 45, 26 slots: 7.8 us; four
        // elements and one slot 11.0, four and four 9.5). While the blocks of all tiles are
        // resident at once, four elements and four slots (3,000 patches, R = 45: 7.9 us;
        // one at a time 9.3). Beyond, the blocks that wait their turn cover the loads and
        // more registers only cost occupancy (16,384 patches, R = 192: 15.6 us with one slot
        // at a time, 16.8 with four, 28.2 with one element per thread).
        const dim3 cg((ld + 31) / 32, (BN + 31) / 32);
        const u32 tiles = cg.x * cg.y, per = tiles <= (u32) sm_count ? 1 : 4, slots = tiles <= 8u * (u32) sm_count ? 4 : 1;
        auto combine_as = [&](auto type, bool with_partial, bool last) {
            using T = decltype(type);
            (per == 1 ? k_combine<T, 1, 8> : slots == 4 ? k_combine<T, 4, 4> : k_combine<T, 4, 1>)<<<cg, dim3(32, 32 / per), 0, s>>>(
                n, ld, R, BN, with_partial ? partial.as<float>() : nullptr, slots_max, rp_cnt, E, alb, last ? out : nullptr,
                last ? nullptr : xh.as<T>(), (last || refine == LTRG_REFINE_NONE) ? nullptr : xl.as<T>(), g_exp, d_emax,
                d_err, last && err_direct ? &h_err : nullptr);
            note_launch();
        };
        auto combine = [&](bool with_partial, bool last) {
            if (precision == LTRG_F_FP16) combine_as(__half(), with_partial, last);
            else combine_as(__nv_bfloat16(), with_partial, last);
        };
        cudaEvent_t e0 = event();
        combine(false, bounces == 0);
        std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ge;
        for (int b = 0; b < bounces; ++b) {
            cudaEvent_t g0 = event();
            GCK(cudaLaunchKernelEx(&lc, kern, mG, mGl, mXh, mXl, ua)); note_launch();
            cudaEvent_t g1 = event();
            ge.push_back({g0, g1});
            GCK(cudaGetLastError());
            combine(true, b + 1 == bounces);
        }
        cudaEvent_t e1 = event();
        finish();
        float m = 0;
        if (c0) {
            g16_kind = precision;
            g16_has_lo = need_lo;
            cudaEventElapsedTime(&m, c0, c1);
            ms_convert = m;
        }
        cudaEventElapsedTime(&m, e0, e1);
        ms_bounces = m;
        for (auto& p : ge) { cudaEventElapsedTime(&m, p.first, p.second); ms_gemm += m; }
        bytes_bounce = (uint64_t) n * ld * 2 * (need_lo ? 2 : 1);
    }
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->ms_build = ms_build;
        stats->ms_convert = ms_convert;
        stats->ms_bounces = ms_bounces;
        stats->ms_per_bounce = bounces ? ms_bounces / bounces : 0;
        stats->ms_gemm = ms_gemm;
        stats->flops_per_bounce = 2.0 * n * (double) n * R * products;
        stats->bytes_per_bounce = bytes_bounce;
        stats->links = links;
        stats->vis_rays = vis_rays;
        stats->pairs = pairs;
        stats->tensor_cores = tc ? 1 : 0;
        stats->stages = stages;
        stats->ctas = ctas_run;
        stats->products = tc ? products : 1;
    }
}

extern "C" {

LTRAPI ltrg_Gather* ltrg_GatherCreate(const float* tri_xyz, u32 n_tris, const float* pos3, const float* nrm3,
                                      const float* area, u32 n, int links, int device)
{
    ltrg_Gather* g = new ltrg_Gather;
    try {
        if (!pos3 || !nrm3 || !area || n == 0 || (n_tris && !tri_xyz)) throw std::runtime_error("invalid arguments");
        if (links != LTRG_LINKS_REFERENCE && links != LTRG_LINKS_VISIBLE) throw std::runtime_error("invalid link predicate");
        if (n > 65535u * 32u) throw std::runtime_error("too many patches");
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) throw std::runtime_error("no CUDA device available");
        if (device < 0 || device >= ndev) throw std::runtime_error("device out of range");
        g->device = device;
        GCK(cudaSetDevice(device));
        keep_pool_memory(device);
        GCK(cudaDeviceGetAttribute(&g->sm_count, cudaDevAttrMultiProcessorCount, device));
        GCK(cudaStreamCreateWithFlags(&g->st, cudaStreamNonBlocking));
        g->n = n;
        g->ld = (n + BK - 1) / BK * BK;
        g->ldg = (n + 3) / 4 * 4;
        cudaStream_t st = g->st;

        // occluder BVH (one instance, every triangle casts shadows)
        std::vector<float> xyz(tri_xyz, tri_xyz + 9 * (size_t) n_tris);
        std::vector<u32> meta(n_tris, kOccluderBit), local(n_tris);
        for (u32 i = 0; i < n_tris; ++i) local[i] = i;
        std::vector<u32> ref_tri;
        std::vector<float> ref_box;
        float cmin[3], cmax[3];
        build_refs_host(xyz, ref_tri, ref_box, cmin, cmax);
        std::vector<float4> hp(n), hn(n);   // patches: position, unit normal
        std::vector<void*> tmp;
        struct TmpGuard {   // waits for the copies before the vectors above go
            std::vector<void*>& v; cudaStream_t s;
            ~TmpGuard() { for (void* p : v) cudaFreeAsync(p, s); cudaStreamSynchronize(s); }
        } tg{tmp, st};
        auto up = [&](const void* h, size_t b) {
            void* d = nullptr;
            GCK(cudaMallocAsync(&d, b ? b : 16, st));
            tmp.push_back(d);
            if (b) GCK(cudaMemcpyAsync(d, h, b, cudaMemcpyHostToDevice, st));
            return d;
        };
        BvhBuildInput bin;
        bin.tri_xyz = (const float*) up(xyz.data(), xyz.size() * 4);
        bin.tri_meta = (const u32*) up(meta.data(), meta.size() * 4);
        bin.tri_local = (const u32*) up(local.data(), local.size() * 4);
        bin.ref_tri = (const u32*) up(ref_tri.data(), ref_tri.size() * 4);
        bin.ref_box = (const float*) up(ref_box.data(), ref_box.size() * 4);
        bin.n = (int) ref_tri.size();
        for (int c = 0; c < 3; ++c) {
            bin.scene_min[c] = bin.n ? cmin[c] : 0;
            bin.scene_max[c] = bin.n ? cmax[c] : 0;
        }
        BvhStorage bvh;
        if (bin.n) bvh_build(bin, bvh, st);
        struct BvhGuard {
            BvhStorage& b; cudaStream_t s; bool on;
            ~BvhGuard() { if (on) bvh_free(b, s); }
        } bg{bvh, st, bin.n > 0};

        // (normalised as the reference's samples are)
        for (u32 i = 0; i < n; ++i) {
            hp[i] = make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], 0.0f);
            V3 nn = normalized(mk(nrm3[3 * i], nrm3[3 * i + 1], nrm3[3 * i + 2]));
            hn[i] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        }
        const float4* dp = (const float4*) up(hp.data(), n * sizeof(float4));
        const float4* dn = (const float4*) up(hn.data(), n * sizeof(float4));
        const float* da = (const float*) up(area, n * sizeof(float));
        u32* derr = (u32*) up(nullptr, 0);
        GCK(cudaMemsetAsync(derr, 0, 4, st));
        g->need(g->G32, (size_t) n * g->ldg * 4);

        cudaEvent_t e0, e1;
        GCK(cudaEventCreate(&e0));
        GCK(cudaEventCreate(&e1));
        GCK(cudaEventRecord(e0, st));
        BvhView view = bin.n ? bvh.view() : BvhView{nullptr, nullptr, nullptr, nullptr, 0, 0};
        RadFormFactors ff = radiosity_form_factors_f32(n, g->ldg, dp, dn, view, ErrFlag{derr}, links, g->G32.as<float>(), st);
        u32* dgmax = (u32*) up(nullptr, 0);
        GCK(cudaMemsetAsync(dgmax, 0, 4, st));
        k_scale_cols<<<std::min<u32>(n, (u32) g->sm_count * 8), 256, 0, st>>>(n, g->ldg, g->G32.as<float>(), da, dgmax); note_launch();
        GCK(cudaGetLastError());
        GCK(cudaEventRecord(e1, st));
        u32 herr = 0, hgmax = 0;
        int hbvh = 0;
        if (bin.n) GCK(cudaMemcpyAsync(&hbvh, bvh.status, sizeof(int), cudaMemcpyDeviceToHost, st));
        GCK(cudaMemcpyAsync(&hgmax, dgmax, 4, cudaMemcpyDeviceToHost, st));
        GCK(cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st));
        GCK(cudaStreamSynchronize(st));
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        bvh_check_status(hbvh);
        if (herr) throw std::runtime_error("form-factor traversal error word " + std::to_string(herr));
        float gmax;
        memcpy(&gmax, &hgmax, 4);
        if (gmax > 0.0f && gmax < 3.0e38f) {
            int p;
            frexpf(gmax, &p);
            g->g_exp = 14 - p;
        }
        g->ms_build = ms;
        g->links = ff.links;
        g->vis_rays = ff.vis_rays;
        g->pairs = (uint64_t) n * (n - 1) / 2;
        g->schedule();
    } catch (const std::exception& e) {
        fprintf(stderr, "ltrg_GatherCreate: %s\n", e.what());
        delete g;
        return nullptr;
    }
    return g;
}

LTRAPI void ltrg_GatherDestroy(ltrg_Gather* g) { delete g; }

LTRAPI LTRBOOL ltrg_GatherSetChunk(ltrg_Gather* g, u32 k_blocks)
{
    if (!g) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    g->kchunk = k_blocks;
    return 1;
}

LTRAPI u32 ltrg_GatherSize(ltrg_Gather* g) { return g ? g->n : 0; }

LTRAPI LTRBOOL ltrg_GatherGetG(ltrg_Gather* g, float* out)
{
    if (!g || !out) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    if (cudaSetDevice(g->device) != cudaSuccess) return 0;
    if (cudaStreamSynchronize(g->st) != cudaSuccess) return 0;
    if (cudaMemcpy2D(out, (size_t) g->n * 4, g->G32.p, (size_t) g->ldg * 4, (size_t) g->n * 4, g->n, cudaMemcpyDeviceToHost) !=
        cudaSuccess)
        return 0;
    return 1;
}

LTRAPI const char* ltrg_GatherLastError(ltrg_Gather* g) { return g && !g->error.empty() ? g->error.c_str() : nullptr; }

LTRAPI LTRBOOL ltrdbg_GatherStallNextSolve(ltrg_Gather* g, u32 wait_us)
{
    if (!g || wait_us == 0 || wait_us > 2000000u) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    g->stall_us = wait_us;
    return 1;
}

LTRAPI LTRBOOL ltrdbg_GatherHostPath(ltrg_Gather* g, int mode)
{
    if (!g || mode < 0 || mode > 2) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    if (mode == 2 && !pageable_access(g->device)) return 0;
    g->host_path = mode;
    return 1;
}

LTRAPI int ltrdbg_GatherHostPathUsed(ltrg_Gather* g)
{
    if (!g) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    return g->host_path ? g->host_path : (pageable_access(g->device) ? 2 : 1);
}

LTRAPI LTRBOOL ltrg_GatherSolveDevice(ltrg_Gather* g, const float* albedo_rgb, const float* emission, u32 R,
                                      int bounces, int precision, int refine, float* out, ltrg_GatherStats* stats,
                                      void* stream)
{
    if (!g) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    g->error.clear();
    try {
        if (!albedo_rgb || !emission || !out || R == 0 || bounces < 0 || precision < LTRG_F_FP32 ||
            precision > LTRG_F_BF16)
            throw std::runtime_error("invalid arguments");
        GCK(cudaSetDevice(g->device));
        g->solve(const_cast<float*>(albedo_rgb), const_cast<float*>(emission), R, bounces, precision, refine, out, stats,
                 stream ? (cudaStream_t) stream : g->st);   // (without host arrays, alb and E are only read)
    } catch (const std::exception& e) {
        g->error = e.what();
        cudaGetLastError();   // the error is reported here; none is left for the caller's next CUDA call
        return 0;
    }
    return 1;
}

LTRAPI LTRBOOL ltrg_GatherSolve(ltrg_Gather* g, const float* albedo_rgb, const float* emission, u32 R, int bounces,
                                int precision, int refine, float* out, ltrg_GatherStats* stats)
{
    if (!g) return 0;
    std::lock_guard<std::mutex> lk(g->mu);
    g->error.clear();
    try {
        if (!albedo_rgb || !emission || !out || R == 0 || bounces < 0 || precision < LTRG_F_FP32 ||
            precision > LTRG_F_BF16)
            throw std::runtime_error("invalid arguments");
        GCK(cudaSetDevice(g->device));
        const u32 n = g->n;
        cudaStream_t s = g->st;
        g->need(g->h_alb, (size_t) n * 3 * 4);
        g->need(g->h_E, (size_t) n * R * 4);
        const bool direct = g->host_path ? g->host_path == 2 : pageable_access(g->device);
        note_h2d((size_t) n * (3 + R) * 4);
        if (direct) {
            // the GPU reads and writes the caller's arrays over the CPU-GPU link: no host
            // copies; the emission's maximum is taken on its way in, and the last bounce
            // writes its result where it belongs
            g->solve(g->h_alb.as<float>(), g->h_E.as<float>(), R, bounces, precision, refine, out, stats, s, albedo_rgb,
                     emission);
            note_d2h((size_t) n * R * 4);
            return 1;
        }
        g->need(g->h_out, (size_t) n * R * 4);
        GCK(cudaMemcpyAsync(g->h_alb.p, albedo_rgb, (size_t) n * 3 * 4, cudaMemcpyHostToDevice, s));
        if (!g->pool) {
            g->pool_threads = std::max(1, std::min(16, (int) std::thread::hardware_concurrency()));
            g->pool.reset(new StagePool);
            g->pool->start(g->pool_threads - 1);   // the calling thread works too
        }
        stage_h2d(g->h_E.p, emission, (size_t) n * R * 4, g->pin_in, s, *g->pool, g->pool_threads);
        g->solve(g->h_alb.as<float>(), g->h_E.as<float>(), R, bounces, precision, refine, g->h_out.as<float>(), stats, s);
        stage_d2h(out, g->h_out.p, (size_t) n * R * 4, g->pin_out, s, *g->pool, g->pool_threads);
        note_d2h((size_t) n * R * 4);
        GCK(cudaStreamSynchronize(s));
    } catch (const std::exception& e) {
        g->error = e.what();
        cudaGetLastError();   // the error is reported here; none is left for the caller's next CUDA call
        return 0;
    }
    return 1;
}

}  // extern "C"
