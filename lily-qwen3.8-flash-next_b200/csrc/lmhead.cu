// The LM head's translation unit: its instantiations and their launches.
#include <atomic>

#include "lmhead_kernel.cuh"

namespace lily_head {

Prepared prepared_at(void *base, uint32_t padded) {
    Prepared p;
    uint8_t *at = static_cast<uint8_t *>(base);
    for (int i = 0; i < 2; ++i) {
        p.image[i] = reinterpret_cast<uint4 *>(at);
        at += (size_t)padded * CHUNK_K * 2u;
    }
    for (int i = 0; i < 2; ++i) {
        p.sums[i] = reinterpret_cast<float *>(at);
        at += (size_t)padded * (CHUNK_K / GROUP_K) * 4u;
    }
    p.unscale = reinterpret_cast<float *>(at);
    p.inexact = reinterpret_cast<uint32_t *>(at + TOK * 4u);
    return p;
}

cudaError_t launch_prepare(const Prepared &p, const void *hidden, uint64_t hidden_ld, uint32_t tokens, uint32_t groups,
                           Format format, uint32_t *flags, uint32_t sms, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(padded_tokens(tokens), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, prepare_hidden_kernel, p, static_cast<const __nv_bfloat16 *>(hidden), hidden_ld, tokens,
                              groups, format == FMT_U4 ? 1 : 0, flags, sms * EPILOGUE_WARPS);
}

namespace {

template <uint32_t N, int FMT>
cudaError_t launch_one(const Args &a, uint32_t sms, cudaStream_t stream) {
    auto kernel = lmhead_kernel<N, FMT>;
    using S = Shape<N, FMT>;
    static std::atomic<uint64_t> ready{0};  // (bit d: device d has seen the set-up below)
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        return e;
    }
    const uint64_t bit = 1ull << (device & 63);
    if (!(ready.load(std::memory_order_relaxed) & bit)) {
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess ||
            (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::BYTES)) != cudaSuccess) {
            return e;
        }
        if (fa.numRegs != (int)S::REGS) {
            return cudaErrorInvalidKernelImage;  // the roles would wait for registers the block does not have
        }
        ready.fetch_or(bit, std::memory_order_relaxed);
    }
    const uint32_t tiles = (a.rows + TILE_ROWS - 1u) / TILE_ROWS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles < sms ? tiles : sms, 1, 1);
    cfg.blockDim = dim3(S::THREADS, 1, 1);
    cfg.dynamicSmemBytes = S::BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <uint32_t N>
cudaError_t launch_for(const Args &a, Format format, uint32_t sms, cudaStream_t stream) {
    return format == FMT_S8   ? launch_one<N, FMT_S8>(a, sms, stream)
           : format == FMT_U8 ? launch_one<N, FMT_U8>(a, sms, stream)
                              : launch_one<N, FMT_U4>(a, sms, stream);
}

}  // namespace

// The token count is padded to 16, 32 or 64: the multiplies, the read-back of the sums and
// their scaling all go with it. Measured per call, both launches, back to back (before:
// 64 always, one pipeline for both halves of a tile, bf16 only, the affine term in a kernel
// of its own, whole tiles only):
//   262144 x 4096, symmetric:     64 tokens 325 -> 240 us, 32 tokens 193, 16 tokens 179
//   248320 x 4096, affine 8 bits: 64 tokens 430 -> 280 us,  4 tokens 435 -> 170
//   151936 x 2048, affine 4 bits: 64 tokens 89 us, 32 tokens 160 -> 57, 4 tokens 48
// (4 bits, 32 tokens, step by step: 80; two groups per hand-over and fewer stages 70; codes
// as subnormals 61; sums of shared tiles handed on through the logits' place instead of a
// workspace: + 0.6 to 1.2 at 4 bits, nothing elsewhere; scales through shared memory 58.4; a warp's waits as one
// 57.3.) At 16 tokens the weights' stream bounds bytes (5.9 TB/s of 6.6
// measured for a copy); the rest is bound by what its warps issue (slots 58 to 63 % busy; 4 % more
// instructions take 3.6 % longer): widening a weight, one FMA per logit and group, and the waits. In calls
// that go on for a tenth of a second the power limit lowers the clock: 64 tokens 240 -> 275 us.
cudaError_t launch_head(const Args &a, Format format, uint32_t sms, cudaStream_t stream) {
    switch (padded_tokens(a.tokens)) {
        case 16: return launch_for<16>(a, format, sms, stream);
        case 32: return launch_for<32>(a, format, sms, stream);
        default: return launch_for<64>(a, format, sms, stream);
    }
}

}  // namespace lily_head
