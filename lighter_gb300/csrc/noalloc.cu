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
// is one kernel that works in shared memory (finalize.cuh), or a few passes over
// a thin image; the passes' masks and middle image, and the input of a call
// whose input and output share memory, go to one fixed scratch array compiled into the library.
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
// Calls share the one array: when their work overlaps on the GPU (two streams,
// or two host threads on one device) they may race on it and must be serialised by
// the caller.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <utility>

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

// The same step pass by pass, for thin images (finish_in_passes): out = rgb and the input mask ...
__global__ void k_na_init(unsigned n, const float* rgb, const unsigned char* __restrict__ mask, float* out,
                          unsigned char* __restrict__ set)
{
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        for (int c = 0; c < 3; ++c) out[3 * g + c] = rgb[3 * g + c];
        set[g] = mask[g] ? 1 : 0;
    }
}

// ... one sweep (fin_dilate; texels set in `old` are not written, so reading them is race-free) ...
__global__ void k_na_dilate(unsigned w, unsigned h, const unsigned char* __restrict__ old, unsigned char* __restrict__ next,
                            float* img)
{
    const unsigned n = w * h;
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        unsigned char set = old[g];
        if (!set) {
            const unsigned x = g % w, y = g / w;
            auto isset = [&](unsigned xx, unsigned yy) { return xx < w && yy < h && old[xx + yy * w]; };
            auto col = [&](unsigned xx, unsigned yy) { const float* p = img + 3 * (xx + yy * w); return mk(p[0], p[1], p[2]); };
            V3 c = mk(0, 0, 0);
            int cnt = 0;
            if (isset(x - 1, y)) { c += isset(x - 2, y) ? lerp3(col(x - 2, y), col(x - 1, y), 2.0f) : col(x - 1, y); cnt++; }
            if (isset(x + 1, y)) { c += isset(x + 2, y) ? lerp3(col(x + 2, y), col(x + 1, y), 2.0f) : col(x + 1, y); cnt++; }
            if (isset(x, y - 1)) { c += isset(x, y - 2) ? lerp3(col(x, y - 2), col(x, y - 1), 2.0f) : col(x, y - 1); cnt++; }
            if (isset(x, y + 1)) { c += isset(x, y + 2) ? lerp3(col(x, y + 2), col(x, y + 1), 2.0f) : col(x, y + 1); cnt++; }
            if (cnt) {
                c = c / (float) cnt;
                float* p = img + 3 * g;
                p[0] = fmax_(c.x, 0.0f);
                p[1] = fmax_(c.y, 0.0f);
                p[2] = fmax_(c.z, 0.0f);
                set = 1;
            }
        }
        next[g] = set;
    }
}

// ... and a clamp-to-edge row convolution written transposed (lighter_math.cpp:367-398):
// src is W x H, dst is H x W.
__global__ void k_na_conv_t(unsigned W, unsigned H, int ext, FinTaps taps, const float* __restrict__ src, float* __restrict__ dst)
{
    const unsigned n = W * H;
    for (unsigned g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const unsigned x = g % W, y = g / W;
        const float* row = src + 3 * (size_t) y * W;
        float s0 = 0, s1 = 0, s2 = 0;
        for (int i = -ext; i <= ext; ++i) {
            int xx = (int) x + i;
            xx = xx < 0 ? 0 : (xx >= (int) W ? (int) W - 1 : xx);
            const float kq = taps.k[i + ext];
            s0 += row[3 * xx + 0] * kq;
            s1 += row[3 * xx + 1] * kq;
            s2 += row[3 * xx + 2] * kq;
        }
        float* o = dst + 3 * ((size_t) y + (size_t) H * x);
        o[0] = s0; o[1] = s1; o[2] = s2;
    }
}

// Whether the passes beat the tiles: a tile works on its region of side x side texels
// whatever it holds of the image, so images a few texels wide are nearly all halo. The
// passes' launches take as long as about 4M texels of regions, and their own work per
// texel is that of 8 texels of regions. Tiles / passes, us: 1 x 2^20 blur 0 322 / 40,
// blur 0.5 505 / 56, blur 16 2,410 / 94; 4 x 2^18 blur 0.5 138 / 62; 8 x 2^17 blur 0.5 76 / 68,
// blur 16 318 / 97; 16 x 2^16 blur 16 175 / 107; and with the masks copied between the sweeps (13 us
// more) 16 x 2^16 blur 0.5 46 / 88, 1,024 x 1,024 blur 16 119 / 145.
bool finish_in_passes(unsigned n, unsigned tiles, int ext)
{
    const unsigned long long side = (unsigned long long) fin_side(ext), regions = tiles * side * side;
    return regions > (4ull << 20) && regions > 8ull * n;
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
    const unsigned tx = (width + kFinTile - 1) / kFinTile, ty = (height + kFinTile - 1) / kFinTile;
    const uintptr_t ri = (uintptr_t) rgb, ro = (uintptr_t) out, bytes = (uintptr_t) n * 12;
    const bool overlap = ri < ro + bytes && ro < ri + bytes;
    if (finish_in_passes(n, tx * ty, ext) && (!overlap || ri == ro)) {
        const unsigned threads = 256, blocks = std::min((n + threads - 1) / threads, 4864u);
        unsigned char *set = base, *next = base + kMaskBytes;
        k_na_init<<<blocks, threads, 0, st>>>(n, rgb, mask, out, set);
        for (int it = 0; it < 3; ++it) {
            k_na_dilate<<<blocks, threads, 0, st>>>(width, height, set, next, out);
            std::swap(set, next);
        }
        if (ext) {
            k_na_conv_t<<<blocks, threads, 0, st>>>(width, height, ext, taps, out, tmp);
            k_na_conv_t<<<blocks, threads, 0, st>>>(height, width, ext, taps, tmp, out);
        }
        e = cudaGetLastError();
        return e == cudaSuccess ? LTRG_NOALLOC_OK : LTRG_NOALLOC_ECUDA;
    }
    // a tile's halo is read while its neighbours are written: input and output
    // that share memory go through the scratch image
    if (overlap) {
        k_na_copy<<<(3 * n + 1023) / 1024, 256, 0, st>>>(3 * n, rgb, tmp);
        rgb = tmp;
    }
    const size_t smem = fin_smem(ext);
    if (smem > 48 * 1024 && fin_allow_smem(k_na_finalize) != cudaSuccess) return LTRG_NOALLOC_ECUDA;
    k_na_finalize<<<tx * ty, kFinThreads, smem, st>>>(width, height, tx, ext, taps, rgb, mask, out);
    e = cudaGetLastError();
    return e == cudaSuccess ? LTRG_NOALLOC_OK : LTRG_NOALLOC_ECUDA;
}
