// Finishing one lightmap without allocating device memory.
//
// Some callers of this library cannot call cudaMalloc at the point where they
// finish a lightmap: code that runs while its stream is being captured into a
// CUDA graph (allocation is not a capturable operation), engine or editor
// plugins whose host application owns all device memory through its own
// allocator, and per-frame callbacks that must not stall the device (cudaFree
// synchronises). ltrg_FinalizeLightmapNoAlloc gives them the finalize step of
// the bake -- three extrapolating dilation sweeps followed by the separable
// Gaussian blur (lighter.cpp:880-961) -- on device buffers they own. The step
// is one kernel that works in shared memory (finalize.cuh); a call whose input
// and output share memory first copies its input to one fixed scratch array
// compiled into the library.
//
// The scratch array is a file-scope __device__ variable, so every GPU that
// loads this library holds it (LTRG_NOALLOC_SCRATCH_BYTES, 14 MiB) until the
// process exits. Host code cannot use the array's name as a device address: a
// call whose stream is not being captured looks the address up with
// cudaGetSymbolAddress, with the caller's device current, and remembers it for
// that device and CUDA context; a call on a stream under capture uses the
// remembered address (looking it up only if there is none yet). So the first
// call in each context -- on each device, and again after a cudaDeviceReset,
// which destroys the context that held the array -- should come before any
// stream capture.
//
// Calls that work in place share the one array: when their work overlaps on
// the GPU (two streams, or two host threads on one device) they race on it and
// must be serialised by the caller.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <mutex>

#include "../../include/lighter_gb300.h"
#include "common.cuh"
#include "finalize.cuh"

namespace lg {
namespace {

constexpr unsigned kNaMaxTexels = LTRG_NOALLOC_MAX_TEXELS;
constexpr int kNaMaxExt = kFinMaxExt;
constexpr size_t kMaskBytes = kNaMaxTexels;                        // one u8 mask
constexpr size_t kImageOffset = 2 * kMaskBytes;                    // after two masks (256-byte aligned)
constexpr size_t kScratchBytes = kImageOffset + (size_t) kNaMaxTexels * 3 * sizeof(float);
static_assert(kScratchBytes == LTRG_NOALLOC_SCRATCH_BYTES, "scratch size mismatch with the header");

__device__ __align__(256) unsigned char g_na_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_na_mutex;
void* g_na_addr[kMaxDevices] = {};
CUcontext g_na_ctx[kMaxDevices] = {};

// The calling thread's current CUDA context (driver entry point, so the
// library needs no link-time dependency on the driver library).
CUcontext current_context()
{
    static PFN_cuCtxGetCurrent_v4000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuCtxGetCurrent_v4000) p;
    });
    CUcontext c = nullptr;
    if (fn) fn(&c);
    return c;
}

// Device address of the scratch array for the current device and context:
// looked up afresh unless `capturing`, in which case the address remembered
// for this device and context is used; nullptr on failure.
void* scratch_address(bool capturing, cudaError_t* err)
{
    int dev = -1;
    *err = cudaGetDevice(&dev);
    if (*err != cudaSuccess) return nullptr;
    if (dev < 0 || dev >= kMaxDevices) { *err = cudaErrorInvalidDevice; return nullptr; }
    const CUcontext ctx = current_context();
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!capturing || !g_na_addr[dev] || g_na_ctx[dev] != ctx) {
        void* p = nullptr;
        *err = cudaGetSymbolAddress(&p, g_na_scratch);
        if (*err != cudaSuccess) return nullptr;
        g_na_addr[dev] = p;
        g_na_ctx[dev] = ctx;
    }
    return g_na_addr[dev];
}

// The whole step (finalize.cuh), one block per tile: one launch instead of nine.
__global__ void __launch_bounds__(kFinThreads) k_na_finalize(unsigned w, unsigned h, unsigned tiles_x, int ext, FinTaps taps,
                                                             const float* __restrict__ rgb,
                                                             const unsigned char* __restrict__ mask, float* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem[];
    fin_tile((int) (blockIdx.x % tiles_x), (int) (blockIdx.x / tiles_x), (int) w, (int) h, ext, taps,
             [&](size_t g, float* c) {
                 c[0] = rgb[3 * g]; c[1] = rgb[3 * g + 1]; c[2] = rgb[3 * g + 2];
                 return mask[g] != 0;
             },
             out, smem);
}

__global__ void k_na_copy(unsigned n, const float* __restrict__ src, float* __restrict__ dst)
{
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) dst[g] = src[g];
}

}  // namespace
}  // namespace lg

using namespace lg;

extern "C" LTRAPI int ltrg_FinalizeLightmapNoAlloc(const float* rgb, const unsigned char* mask, float* out,
                                                    u32 width, u32 height, float blur_size, void* stream)
{
    if (!rgb || !mask || !out || width == 0 || height == 0) return LTRG_NOALLOC_EINVAL;
    if ((unsigned long long) width * height > kNaMaxTexels) return LTRG_NOALLOC_ETOOBIG;
    if (!(blur_size >= 0.0f) || std::ceil(blur_size) > (float) kNaMaxExt) return LTRG_NOALLOC_EINVAL;
    cudaStream_t st = (cudaStream_t) stream;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
    cudaError_t e;
    unsigned char* base = (unsigned char*) scratch_address(capturing, &e);
    if (!base) return LTRG_NOALLOC_ECUDA;
    float* tmp = (float*) (base + kImageOffset);
    const unsigned n = width * height;
    int ext = 0;
    FinTaps taps = {};
    if (blur_size != 0.0f) {
        // Gaussian taps on the host with the reference's formula
        // (Generate_Gaussian_Kernel, lighter_math.cpp:357-365)
        ext = (int) std::ceil(blur_size);
        float sum = 0.0f;
        float mc = 1.0f / sqrtf(2.0f * 3.14159265358979323846f * blur_size * blur_size);
        for (int i = -ext; i <= ext; ++i) sum += taps.k[i + ext] = expf(-0.5f * powf((float) i / blur_size, 2.0f)) * mc;
        for (int i = -ext; i <= ext; ++i) taps.k[i + ext] /= sum;
    }
    // a tile's halo is read while its neighbours are written: input and output
    // that share memory go through the scratch image
    const uintptr_t ri = (uintptr_t) rgb, ro = (uintptr_t) out, bytes = (uintptr_t) n * 12;
    if (ri < ro + bytes && ro < ri + bytes) {
        k_na_copy<<<(3 * n + 1023) / 1024, 256, 0, st>>>(3 * n, rgb, tmp);
        rgb = tmp;
    }
    const unsigned tx = (width + kFinTile - 1) / kFinTile, ty = (height + kFinTile - 1) / kFinTile;
    const size_t smem = fin_smem(ext);
    if (smem > 48 * 1024 && fin_allow_smem(k_na_finalize) != cudaSuccess) return LTRG_NOALLOC_ECUDA;
    k_na_finalize<<<tx * ty, kFinThreads, smem, st>>>(width, height, tx, ext, taps, rgb, mask, out);
    e = cudaGetLastError();
    return e == cudaSuccess ? LTRG_NOALLOC_OK : LTRG_NOALLOC_ECUDA;
}
