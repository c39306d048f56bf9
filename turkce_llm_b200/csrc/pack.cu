// float32 -> bf16 operand packing for callers that keep their matrices in float32, as the
// reference does (its kernels convert while staging tiles: cuda/train_kernels.cu:256-263).
// Rounding is round-to-nearest-even, the same as the reference's f32_to_bf16
// (cuda/train_kernels.cu:207-212) on every finite input.
//
// The packed copy gets a leading dimension that is a multiple of 8 elements so that TMA can
// address it whatever the source's leading dimension was (the 31,769-column logits included).
#include "common.h"

#include <algorithm>

namespace tb {

// The three conversions of a float32 matrix into an operand: bf16, a float32 copy with another leading dimension, and the
// tf32-exact pieces of the 3xTF32 product.  In the last, hi keeps the 19 bits a tf32 operand has (sign, 8 exponent, 10
// mantissa); lo = x - hi is exact in float32 and itself enters the tensor core truncated to tf32, which loses about 2^-21 of x.
//
// The kernels are bound by memory for large matrices and by launch and division latency for the layer-sized ones (1024 x 384
// took 5 us): both operands of a product are converted by ONE launch, each by its own share of the blocks; indices are
// 32-bit (a 64-bit division per element cost more than the element's bytes); the launch carries the programmatic attribute,
// since what follows is always the GEMM that waits for it.
enum { CONV_BF16 = 0, CONV_COPY = 1, CONV_SPLIT3 = 2 };

template <int MODE>
__device__ __forceinline__ void convert_quad(const ConvSide& c, void* dst, unsigned r, unsigned col, const float (&x)[4], int n) {
    if (MODE == CONV_BF16) {
        bf16* d = static_cast<bf16*>(dst) + (long long)r * c.ld_dst + col;
        if (n == 4) {
            __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
            *reinterpret_cast<uint2*>(d) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
        } else {
            *d = __float2bfloat16_rn(x[0]);
        }
        return;
    }
    auto put = [&](float* d, const float (&v)[4]) {
        if (n == 4) *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
        else *d = v[0];
    };
    float* d = static_cast<float*>(dst) + (long long)r * c.ld_dst + col;
    if (MODE == CONV_COPY) { put(d, x); return; }
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        hi[e] = __uint_as_float(__float_as_uint(x[e]) & 0xFFFFE000u);
        lo[e] = x[e] - hi[e];
    }
    const long long step = c.along_cols ? (long long)c.cols : (long long)c.rows * c.ld_dst;      // from piece to piece
    put(d, hi);
    if (c.pattern == 0) { put(d + step, hi); put(d + 2 * step, lo); }
    else { put(d + step, lo); put(d + 2 * step, hi); }
}

template <int MODE, typename Index>
__device__ __forceinline__ void convert_side(const ConvSide& c, int block) {
    const float* s = c.src + (long long)blockIdx.z * c.stride_src;
    void* d = MODE == CONV_BF16 ? static_cast<void*>(static_cast<bf16*>(c.dst) + (long long)blockIdx.z * c.stride_dst)
                                : static_cast<void*>(static_cast<float*>(c.dst) + (long long)blockIdx.z * c.stride_dst);
    const unsigned w = c.vec ? 4u : 1u;
    const Index per_row = (Index)((unsigned)c.cols / w);
    const Index total = (Index)c.rows * per_row;
    for (Index i = (Index)block * blockDim.x + threadIdx.x; i < total; i += (Index)c.blocks * blockDim.x) {
        const unsigned r = (unsigned)(i / per_row), col = (unsigned)(i - (Index)r * per_row) * w;
        const float* p = s + (long long)r * c.ld_src + col;
        float x[4];
        if (c.vec) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else {
            x[0] = *p; x[1] = x[2] = x[3] = 0.0f;
        }
        convert_quad<MODE>(c, d, r, col, x, c.vec ? 4 : 1);
    }
}

template <int MODE>
__global__ void convert_kernel(const ConvSide a, const ConvSide b) {
    pdl_wait();
    pdl_launch_dependents();
    const bool first = (int)blockIdx.x < a.blocks;
    const ConvSide& c = first ? a : b;
    const int block = first ? (int)blockIdx.x : (int)blockIdx.x - a.blocks;
    // (the last index plus one grid's stride has to stay below 2^32)
    if ((long long)c.rows * c.cols < (1LL << 31)) convert_side<MODE, unsigned>(c, block);
    else convert_side<MODE, unsigned long long>(c, block);
}

static int launch_convert(DeviceCtx* ctx, int mode, ConvSide* sides, int count, int batch, cudaStream_t stream) {
    static const char* const tag[3] = {"pack_bf16", "copy_f32", "split3_f32"};
    static const double bytes_per[3] = {6.0, 8.0, 16.0};
    double bytes = 0.0;
    int blocks = 0;
    for (int k = 0; k < 2; ++k) {
        ConvSide& c = sides[k];
        c.blocks = 0;
        if (k >= count) continue;
        TB_CHECK(c.rows > 0 && c.cols > 0 && batch > 0, "%s: empty matrix", tag[mode]);
        const unsigned dst_align = mode == CONV_BF16 ? 8 : 16;
        c.vec = c.cols % 4 == 0 && c.ld_src % 4 == 0 && c.ld_dst % 4 == 0 && c.stride_src % 4 == 0 && c.stride_dst % 4 == 0 &&
                reinterpret_cast<uintptr_t>(c.src) % 16 == 0 && reinterpret_cast<uintptr_t>(c.dst) % dst_align == 0;
        const long long work = (long long)c.rows * (c.vec ? c.cols / 4 : c.cols);
        c.blocks = (int)std::max<long long>(1, std::min<long long>((work + 255) / 256, 8LL * ctx->sm_count));
        blocks += c.blocks;
        bytes += (double)c.rows * c.cols * batch * bytes_per[mode];
    }
    prof_mark(ctx, tag[mode], 0.0, bytes, stream);
    void (*kernel)(const ConvSide, const ConvSide) =
        mode == CONV_BF16 ? convert_kernel<CONV_BF16> : mode == CONV_COPY ? convert_kernel<CONV_COPY> : convert_kernel<CONV_SPLIT3>;
    TB_CUDA(launch_kernel_early(kernel, dim3((unsigned)blocks, 1, (unsigned)batch), dim3(256), 0, stream, sides[0], sides[1]));
    ctx->launches++;
    prof_close(ctx, stream);
    return 0;
}

int launch_pack_bf16(DeviceCtx* ctx, const float* src, bf16* dst, int rows, int cols, long long ld_src,
                     long long ld_dst, int batch, long long stride_src, long long stride_dst, cudaStream_t stream) {
    ConvSide sides[2] = {{src, dst, rows, cols, ld_src, ld_dst, stride_src, stride_dst}, {}};
    return launch_convert(ctx, CONV_BF16, sides, 1, batch, stream);
}
int launch_pack_operands(DeviceCtx* ctx, ConvSide* sides, int count, int batch, cudaStream_t stream) {
    return launch_convert(ctx, CONV_BF16, sides, count, batch, stream);
}
int launch_copy_operands(DeviceCtx* ctx, ConvSide* sides, int count, int batch, cudaStream_t stream) {
    return launch_convert(ctx, CONV_COPY, sides, count, batch, stream);
}
int launch_split3_operands(DeviceCtx* ctx, ConvSide* sides, int count, int batch, cudaStream_t stream) {
    return launch_convert(ctx, CONV_SPLIT3, sides, count, batch, stream);
}

// bf16 -> float32 (exact): the TF32 mode of the trainer widens the outputs of the attention kernels, which
// stay bf16, before they enter a float32-operand GEMM.  n must be a multiple of 4, pointers 16-byte aligned.
__global__ void widen_bf16_kernel(const uint2* __restrict__ src, float4* __restrict__ dst, long long n4) {
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const uint2 v = src[i];
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&v.x);
        const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
        dst[i] = make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
    }
}

int launch_widen_bf16(DeviceCtx* ctx, const bf16* src, float* dst, long long n, cudaStream_t stream) {
    TB_CHECK(n > 0 && n % 4 == 0, "widen: element count must be a positive multiple of 4");
    long long blocks = (n / 4 + 255) / 256;
    if (blocks > 8LL * ctx->sm_count) blocks = 8LL * ctx->sm_count;
    prof_mark(ctx, "widen_bf16", 0.0, (double)n * 6.0, stream);
    TB_CUDA(launch_kernel(widen_bf16_kernel, dim3((unsigned)blocks), dim3(256), 0, stream,
                          reinterpret_cast<const uint2*>(src), reinterpret_cast<float4*>(dst), n / 4));
    TB_CUDA(cudaGetLastError());
    ctx->launches++;
    prof_close(ctx, stream);
    return 0;
}

}  // namespace tb
