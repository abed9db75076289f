/*
 * quantize.cu - the format's quantizer on the GPU: FP32 [N][K] in device memory -> packed nibbles
 * [N][K/2] and BF16 scales [N][K/128], byte-identical to the reference's CPU quantizer
 * (linear_quantize_int4, csrc/linear_weight.cpp:108-176), which its offline converter calls once per
 * tensor through a subprocess (scripts/quantize_weights.py:136-156).
 *
 * Arithmetic, in the reference's order and with IEEE operations (no fast-math, denormals kept):
 *   max_abs over the 128-group; scale = BF16_RNE(max_abs / 7), the all-zero group's scale = 1;
 *   q = clip(nearbyintf(w / scale), -7, 7) against the ROUNDED scale; low K index in the low nibble.
 * Refusals, also the reference's: a non-finite element; a group whose scale does not round to a
 * positive finite BF16 (e.g. a group of 1e-40).  The reference validates everything before it
 * writes anything; so does this file (one checking pass, then the writing pass).
 *
 * HBM bound: the FP32 input is read once.  The checking pass quantizes into scratch as it goes, and a second
 * launch moves the bytes to the caller once nothing was refused - it looks at the verdict itself and tells the host, which
 * waits once, at the end.  5120 x 17408: 221 us with a checking and a writing pass over the input, a wait
 * between them and cudaMalloc / cudaFree around them; 111 with the verdict cleared and copied by operations of
 * their own, 104 now (1024 x 2560: 46 -> 38 as the caller sees it).  Where the bytes exceed the scratch that
 * the library keeps (kScratchMost), or there is no memory for them, the second launch quantizes again instead.
 *
 * Eight lanes per group: a lane holds sixteen elements in four 16-byte loads (128 contiguous bytes of a group
 * each), so the group's division, reciprocal and reduction are paid once per sixteen elements: instructions, not
 * bytes, are what is left (142 us with a warp per group and four elements a lane).
 */
#include <mutex>

#include "common.cuh"
#include "kernels.h"

namespace ffn {

/* BF16 round-to-nearest-even by the reference's bit formula (csrc/linear_weight.cpp:34-45); the
 * inputs here are finite. */
__device__ __forceinline__ uint16_t bf16_rne_bits(float v) {
    uint32_t bits = __float_as_uint(v);
    bits += 0x7FFFu + ((bits >> 16) & 1u);
    return (uint16_t)(bits >> 16);
}

struct QuantStatus {
    unsigned long long bad_element; /* 1 + index of a non-finite element, 0 = none */
    unsigned long long bad_group;   /* 1 + (row * groups + group) of an unrepresentable scale, 0 = none */
};

/* The verdict of a call.  Every launch of a call is handed all of it: the checking pass marks what it finds in `here`
 * (none at the start of the call) and leaves `next`, the words of the call after, clear; the last launch tells the host.
 * So a call needs no clearing and no copy of its own. */
struct QuantVerdict {
    QuantStatus *here, *next; /* device memory; next may be null */
    QuantStatus *host;        /* mapped host memory; may be null */
};
__device__ __forceinline__ void quant_clear_next(const QuantVerdict &v) {
    if (v.next && blockIdx.x == 0 && threadIdx.x == 0) { v.next->bad_element = ~0ull; v.next->bad_group = ~0ull; }
}
__device__ __forceinline__ void quant_tell(const QuantVerdict &v) {
    if (v.host && blockIdx.x == 0 && threadIdx.x == 0) *v.host = *v.here;
}

constexpr int kGroupsInFlight = 4;
constexpr int kQuantThreads = 256;
constexpr size_t kScratchMost = 56ull << 20; /* of the 64 MiB that the library's pool keeps between calls */

/* CHECK: looks for what the format cannot hold (and writes the bytes where `packed` is given); else nothing is
 * written when a check before this launch found something. */
template <bool CHECK>
__global__ void __launch_bounds__(kQuantThreads) quantize_int4_kernel(const float *__restrict__ w, uint8_t *__restrict__ packed,
                                                                     uint16_t *__restrict__ scales, long long groups_total,
                                                                     const QuantVerdict verdict) {
    QuantStatus *const status = verdict.here;
    if (CHECK) quant_clear_next(verdict);
    else quant_tell(verdict);
    if (!CHECK && (status->bad_element != ~0ull || status->bad_group != ~0ull)) return;
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long first = warp * kGroupsInFlight; first < groups_total; first += nwarps * kGroupsInFlight) {
        const long long grp = first + (lane >> 3);
        const bool live = grp < groups_total; /* the lanes of a group agree */
        const long long base = grp * FFN_INT4_GROUP + sub * 4;
        float e[16]; /* elements base + 32 * j + i */
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = live ? __ldcs((const float4 *)(w + base + 32 * j)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            e[4 * j] = v.x; e[4 * j + 1] = v.y; e[4 * j + 2] = v.z; e[4 * j + 3] = v.w;
        }
        /* magnitudes compare like their bits, with Inf and NaN above every finite one */
        unsigned top = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) top = max(top, __float_as_uint(e[i]) & 0x7FFFFFFFu);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
        if (top >= 0x7F800000u) { /* a group with an Inf or a NaN */
            if (CHECK) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (!isfinite(e[i])) atomicMin(&status->bad_element, (unsigned long long)(base + 32 * (i >> 2) + (i & 3)) + 1ull);
            }
            continue;
        }
        if (!live) continue;
        const uint16_t scale_bits = top == 0u ? (uint16_t)0x3F80u : bf16_rne_bits(__fdiv_rn(__uint_as_float(top), 7.0f));
        const float scale = bf16_bits_to_f32(scale_bits);
        if (CHECK && sub == 0 && (!(scale > 0.0f) || !isfinite(scale))) atomicMin(&status->bad_group, (unsigned long long)grp + 1ull);
        if (CHECK && !packed) continue;
        if (sub == 0) scales[grp] = scale_bits;
        /* The code is rint(e / scale), nearest even, of the correctly rounded quotient.  The product with the
         * reciprocal is within 2e-6 of it (|quotient| < 7.1, three roundings), so the two agree unless the product
         * lies that close to a half; those, and groups whose scale is too small for the bound, divide.
         * Adding 1.5 * 2^23 leaves the rounded integer in the low bits, in two's complement. */
        uint32_t nib[16];
        const float recip = __frcp_rn(scale);
        float off = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float t = e[i] * recip, m = t + 12582912.0f;
            off = fmaxf(off, fabsf(t - (m - 12582912.0f)));
            nib[i] = __float_as_uint(m) & 0xFu;
        }
        if (!(off < 0.49999f) || scale < 7.8886091e-31f /* 2^-100 */) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float q = fminf(fmaxf(rintf(__fdiv_rn(e[i], scale)), -7.0f), 7.0f);
                nib[i] = (uint32_t)((int)q) & 0xFu;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *(uint16_t *)(packed + base / 2 + 16 * j) = (uint16_t)(nib[4 * j] | (nib[4 * j + 1] << 4) | (nib[4 * j + 2] << 8) | (nib[4 * j + 3] << 12));
    }
}

/* The quantized bytes from scratch to the caller, unless something was refused.  Both counts are in units of
 * T: 16 bytes where the caller's pointers allow it, else 2. */
template <typename T>
__global__ void __launch_bounds__(kQuantThreads) quantize_deliver_kernel(T *__restrict__ packed, const T *__restrict__ from_packed, long long np,
                                                                        T *__restrict__ scales, const T *__restrict__ from_scales, long long ns,
                                                                        const QuantVerdict verdict) {
    const QuantStatus *const status = verdict.here;
    quant_tell(verdict);
    if (status->bad_element != ~0ull || status->bad_group != ~0ull) return;
    const long long step = (long long)gridDim.x * kQuantThreads, at = (long long)blockIdx.x * kQuantThreads + threadIdx.x;
    for (long long i = at; i < np; i += step) packed[i] = from_packed[i];
    for (long long i = at; i < ns; i += step) scales[i] = from_scales[i];
}

/* The words of calls in flight: per device eight at most, kept until the process ends, each one call's at a time - a
 * call ends when the stream has been waited for.  Calls beyond those clear and copy words of their own. */
struct QuantWords {
    QuantStatus *device = nullptr, *host = nullptr, *host_mapped = nullptr;
    int turn = 0;
    bool busy = false;
};
constexpr int kQuantWords = 8;
static QuantWords g_quant_words[64][kQuantWords];
static std::mutex g_quant_mutex;

static QuantWords *quant_words_take() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return nullptr; }
    std::lock_guard<std::mutex> lock(g_quant_mutex);
    for (QuantWords &w : g_quant_words[dev]) {
        if (w.busy) continue;
        if (!w.device) {
            QuantStatus *device = nullptr, *host = nullptr, *mapped = nullptr;
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed; /* another thread's capture in global mode goes on */
            (void)cudaThreadExchangeStreamCaptureMode(&mode);
            const bool failed = cudaMalloc(&device, 2 * sizeof(QuantStatus)) != cudaSuccess || cudaHostAlloc(&host, sizeof(QuantStatus), cudaHostAllocMapped) != cudaSuccess ||
                cudaHostGetDevicePointer(&mapped, host, 0) != cudaSuccess ||
                cudaMemsetAsync(device, 0xFF, 2 * sizeof(QuantStatus), cudaStreamPerThread) != cudaSuccess || cudaStreamSynchronize(cudaStreamPerThread) != cudaSuccess;
            (void)cudaThreadExchangeStreamCaptureMode(&mode);
            if (failed) {
                (void)cudaGetLastError();
                if (device) cudaFree(device);
                if (host) cudaFreeHost(host);
                return nullptr;
            }
            w.device = device; w.host = host; w.host_mapped = mapped;
        }
        w.busy = true;
        return &w;
    }
    return nullptr;
}
static void quant_words_return(QuantWords *w, bool sound) {
    if (!w) return;
    std::lock_guard<std::mutex> lock(g_quant_mutex);
    w->turn ^= 1;
    w->busy = !sound; /* words that a failed launch may have left anyhow are not used again */
}

}  // namespace ffn

using namespace ffn;

extern "C" int ffn_quantize_int4(const void *weights, void *packed, void *scales, long long n, long long k, void *stream_) {
    clear_error();
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!weights || !packed || !scales) return fail(FFN_ERR_CONFIG, "ffn_quantize_int4: null argument");
    if (n <= 0 || k <= 0) return fail(FFN_ERR_CONFIG, "ffn_quantize_int4: [%lld, %lld] is not a weight shape", n, k);
    if (k % FFN_INT4_GROUP) return fail(FFN_ERR_CONFIG, "ffn_quantize_int4: K = %lld is not a whole number of %d-wide groups", k, FFN_INT4_GROUP);
    if (n % 8) return fail(FFN_ERR_CONFIG, "ffn_quantize_int4: N = %lld is not a multiple of the 8-row tile", n);
    if (((uintptr_t)weights & 15) || ((uintptr_t)packed & 1) || ((uintptr_t)scales & 1))
        return fail(FFN_ERR_CONFIG, "ffn_quantize_int4: weights must be 16-byte aligned, outputs 2-byte aligned");
    const long long groups = n * (k / FFN_INT4_GROUP);
    const long long packed_bytes = n * k / 2, scale_bytes = groups * 2;
    bool keep = (size_t)(packed_bytes + scale_bytes) <= kScratchMost;
    QuantWords *const words = quant_words_take();
    const size_t scales_at = 256 + ((size_t)packed_bytes + 255) / 256 * 256;
    uint8_t *scratch = nullptr;
    const bool pooled = scratch_alloc((void **)&scratch, keep ? scales_at + (size_t)scale_bytes : 256, stream) == FFN_OK;
    if (!pooled) {
        /* no room for the bytes (the call is made while weights fill the device): two passes and the status words */
        keep = false;
        if (!words && cudaMalloc(&scratch, sizeof(QuantStatus)) != cudaSuccess) { (void)cudaGetLastError(); return fail(FFN_ERR_ALLOC, "ffn_quantize_int4: cannot allocate the status words"); }
    }
    int rc = FFN_OK;
    bool sound = true;
    QuantStatus host;
    QuantVerdict status = {(QuantStatus *)scratch, nullptr, nullptr};
    if (words) status = {words->device + words->turn, words->device + (words->turn ^ 1), words->host_mapped};
    const long long turns = (groups + kGroupsInFlight * 8 - 1) / (kGroupsInFlight * 8);
    const unsigned grid = (unsigned)(turns < 148ll * 16 ? turns : 148ll * 16);
    do {
        if (!words && cudaMemsetAsync(status.here, 0xFF, sizeof(QuantStatus), stream) != cudaSuccess) { rc = fail(FFN_ERR_CUDA, "ffn_quantize_int4: memset failed"); break; }
        quantize_int4_kernel<true><<<grid, kQuantThreads, 0, stream>>>((const float *)weights, keep ? scratch + 256 : nullptr,
                                                                       keep ? (uint16_t *)(scratch + scales_at) : nullptr, groups, status);
        if (!keep) {
            quantize_int4_kernel<false><<<grid, kQuantThreads, 0, stream>>>((const float *)weights, (uint8_t *)packed, (uint16_t *)scales, groups, status);
        } else if (!(((uintptr_t)packed | (uintptr_t)scales) & 15)) { /* both counts are multiples of 16: n % 8 == 0, k % 128 == 0 */
            quantize_deliver_kernel<uint4><<<148 * 8, kQuantThreads, 0, stream>>>((uint4 *)packed, (const uint4 *)(scratch + 256), packed_bytes / 16, (uint4 *)scales,
                                                                                  (const uint4 *)(scratch + scales_at), scale_bytes / 16, status);
        } else {
            quantize_deliver_kernel<uint16_t><<<148 * 8, kQuantThreads, 0, stream>>>((uint16_t *)packed, (const uint16_t *)(scratch + 256), packed_bytes / 2,
                                                                                     (uint16_t *)scales, (const uint16_t *)(scratch + scales_at), scale_bytes / 2, status);
        }
        if (cudaGetLastError() != cudaSuccess || (!words && cudaMemcpyAsync(&host, status.here, sizeof(host), cudaMemcpyDeviceToHost, stream) != cudaSuccess) ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            rc = fail(FFN_ERR_CUDA, "ffn_quantize_int4: quantizing failed: %s", cudaGetErrorString(cudaGetLastError()));
            sound = false;
            break;
        }
        if (words) host = *words->host;
        if (host.bad_element != ~0ull) {
            rc = fail(FFN_ERR_WEIGHTS, "ffn_quantize_int4: element %llu is not finite; a quantizer cannot invent a scale for it",
                      host.bad_element - 1ull);
            break;
        }
        if (host.bad_group != ~0ull) {
            const unsigned long long g = host.bad_group - 1ull, per_row = (unsigned long long)(k / FFN_INT4_GROUP);
            rc = fail(FFN_ERR_WEIGHTS, "ffn_quantize_int4: row %llu group %llu rounds to a scale that is not positive and finite; "
                      "the format cannot represent it", g / per_row, g % per_row);
            break;
        }
    } while (0);
    quant_words_return(words, sound);
    if (pooled) (void)cudaFreeAsync(scratch, stream);
    else if (scratch) cudaFree(scratch);
    return rc;
}
