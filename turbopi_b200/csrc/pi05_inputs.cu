// The pipeline's inputs in one launch each: camera images to bf16 patch rows, prompt tokens to scaled embedding rows
// (openpi/src/openpi/models_pytorch/pi0_pytorch.py:215-345).  Each stood for four or five elementwise launches of 2-3 us without
// programmatic dependent launch in front of the first GEMM; the work itself is 0.6 MB of reads and 1.4 MB of writes.
#include "common.cuh"

namespace tpb {
namespace {

// one CTA per patch; values in (channel, row, column) order, x * (1 / 127.5) - 1 in fp32, rounded to bf16 once
__global__ void __launch_bounds__(256) pi05_patches_kernel(const uint8_t* images, __nv_bfloat16* out, int size, int patch, int pitch) {
    pdl_launch_dependents();
    pdl_wait_prior_grids();
    const int n = size / patch, t = blockIdx.x, im = t / (n * n), py = t / n % n, px = t % n;
    const uint8_t* src = images + (static_cast<size_t>(im) * size + py * patch) * size * 3 + px * patch * 3;
    const int area = patch * patch;
    for (int e = threadIdx.x; e < 3 * area; e += blockDim.x) {
        const int c = e / area, i = e % area / patch, j = e % patch;
        const float v = static_cast<float>(src[(static_cast<size_t>(i) * size + j) * 3 + c]);
        out[static_cast<size_t>(t) * pitch + e] = __float2bfloat16_rn(__fsub_rn(__fmul_rn(v, 1.0f / 127.5f), 1.0f));   // as torch divides by a scalar
    }
}

// one CTA per token; a negative index counts from the end.  One outside the table gives zeros, or with `strict` NaN and an
// error: masked or not, a prompt row of NaN reaches every action through the attention
__global__ void __launch_bounds__(256) pi05_embed_kernel(const long long* tokens, const __nv_bfloat16* table, __nv_bfloat16* out,
                                                         long long vocab, int width, float scale, bool strict) {
    pdl_launch_dependents();
    pdl_wait_prior_grids();
    long long t = tokens[blockIdx.x];
    if (t < 0) t += vocab;
    const bool in = t >= 0 && t < vocab;
    const float outside = strict ? __int_as_float(0x7fffffff) : 0.0f;
    if (!in && strict && threadIdx.x == 0) record_error(kErrTokenOutOfRange);
    for (int e = threadIdx.x * 2; e < width; e += 2 * blockDim.x) {
        __nv_bfloat162 v = __floats2bfloat162_rn(outside, outside);
        if (in) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(table + t * width + e));
            v = __floats2bfloat162_rn(f.x * scale, f.y * scale);
        }
        *reinterpret_cast<__nv_bfloat162*>(out + static_cast<size_t>(blockIdx.x) * width + e) = v;
    }
}

cudaLaunchConfig_t config(int blocks, int flags, cudaLaunchAttribute* attr, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (flags & TPB200_FLAG_PDL) ? 1 : 0;
    return cfg;
}

}  // namespace

int device_error_pi05_inputs(int clear) { return read_device_error(clear); }

}  // namespace tpb

extern "C" int tpb200_pi05_patches(const void* images_u8, void* patches, int num_images, int size, int patch, int pitch, int flags,
                                   tpb200_stream_t stream) {
    TPB_REQUIRE(images_u8 != nullptr && patches != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE((flags & ~TPB200_FLAG_PDL) == 0, TPB200_ERR_ENUM);
    TPB_REQUIRE(num_images >= 1 && patch >= 1 && size >= patch && size % patch == 0 && pitch >= 3 * patch * patch, TPB200_ERR_SHAPE);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = tpb::config(num_images * (size / patch) * (size / patch), flags, &attr,
                                               reinterpret_cast<cudaStream_t>(stream));
    return cudaLaunchKernelEx(&cfg, tpb::pi05_patches_kernel, static_cast<const uint8_t*>(images_u8), static_cast<__nv_bfloat16*>(patches),
                              size, patch, pitch) == cudaSuccess ? TPB200_OK : TPB200_ERR_CUDA;
}

extern "C" int tpb200_pi05_embed(const long long* tokens, const void* table, void* out, int num_tokens, long long vocab, int width,
                                 float scale, int flags, tpb200_stream_t stream) {
    TPB_REQUIRE(tokens != nullptr && table != nullptr && out != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE((flags & ~(TPB200_FLAG_PDL | TPB200_FLAG_STRICT_TOKENS)) == 0, TPB200_ERR_ENUM);
    TPB_REQUIRE(num_tokens >= 1 && vocab >= 1 && width >= 2 && width % 2 == 0, TPB200_ERR_SHAPE);
    TPB_REQUIRE(((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) & 3) == 0, TPB200_ERR_ALIGN);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = tpb::config(num_tokens, flags, &attr, reinterpret_cast<cudaStream_t>(stream));
    return cudaLaunchKernelEx(&cfg, tpb::pi05_embed_kernel, tokens, static_cast<const __nv_bfloat16*>(table),
                              static_cast<__nv_bfloat16*>(out), vocab, width, scale, (flags & TPB200_FLAG_STRICT_TOKENS) != 0) == cudaSuccess ? TPB200_OK : TPB200_ERR_CUDA;
}
