// Kernels of the warm-start network: a convolutional encoder-decoder that
// maps a target image and the site layout to initial dual weights.  BF16
// operands, FP32 accumulation.  3x3 convolutions run as im2col + a tensor-core
// GEMM (tcgen05 through the CUTLASS sm100 collective templates); everything
// around them (im2col / col2im, bias + ReLU, pooling, upsampling, concat,
// loss, optimizer) is written here.  Activations are NHWC; a layer's weights
// are [Cout][9*Cin] (tap-major, channel-minor), the matrix B of the GEMM
// D[M, Cout] = cols[M, 9*Cin] * W^T.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cutlass/cutlass.h>
#include <cute/tensor.hpp>
#include <cutlass/gemm/device/gemm_universal_adapter.h>
#include <cutlass/gemm/kernel/gemm_universal.hpp>
#include <cutlass/gemm/collective/collective_builder.hpp>
#include <cutlass/epilogue/collective/collective_builder.hpp>
#include <cutlass/epilogue/fusion/operations.hpp>
#include <cutlass/util/packed_stride.hpp>

#include <algorithm>
#include <initializer_list>

#include "../../include/causticws.h"

namespace {

using bf16 = __nv_bfloat16;

// ---------------------------------------------------------------------------
// GEMM: D[M,N] (fp32, row-major) = alpha * A[M,K] * B[K,N] + beta * D
// ---------------------------------------------------------------------------
// One GEMM configuration per operand layout: MT x NT x 64 tiles on one SM,
// fp32 accumulators in tensor memory, fp32 output.
#define WS_GEMM_CONFIG(NAME, LA, LB, MT, NT)                                                                        \
    namespace NAME {                                                                                                \
    using ElemAB = cutlass::bfloat16_t;                                                                            \
    using Tile = cute::Shape<cute::Int<MT>, cute::Int<NT>, cute::_64>;                                             \
    using Cluster = cute::Shape<cute::_1, cute::_1, cute::_1>;                                                     \
    using Epilogue = cutlass::epilogue::collective::CollectiveBuilder<                                             \
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, Tile, Cluster,                                       \
        cutlass::epilogue::collective::EpilogueTileAuto, float, float, float, cutlass::layout::RowMajor, 4, float,  \
        cutlass::layout::RowMajor, 4, cutlass::epilogue::collective::EpilogueScheduleAuto>::CollectiveOp;          \
    using Mainloop = cutlass::gemm::collective::CollectiveBuilder<                                                 \
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, ElemAB, LA, 8, ElemAB, LB, 8, float, Tile, Cluster,  \
        cutlass::gemm::collective::StageCountAutoCarveout<static_cast<int>(sizeof(Epilogue::SharedStorage))>,      \
        cutlass::gemm::collective::KernelScheduleAuto>::CollectiveOp;                                              \
    using Kernel = cutlass::gemm::kernel::GemmUniversal<cute::Shape<int, int, int, int>, Mainloop, Epilogue, void>; \
    using Gemm = cutlass::gemm::device::GemmUniversalAdapter<Kernel>;                                              \
    inline Gemm::Arguments args(int M, int N, int K, const void *A, const void *B, float *D, float alpha,          \
                                float beta)                                                                         \
    {                                                                                                              \
        auto sa = cutlass::make_cute_packed_stride(Kernel::StrideA{}, cute::make_shape(M, K, 1));                  \
        auto sb = cutlass::make_cute_packed_stride(Kernel::StrideB{}, cute::make_shape(N, K, 1));                  \
        auto sd = cutlass::make_cute_packed_stride(Kernel::StrideD{}, cute::make_shape(M, N, 1));                  \
        return Gemm::Arguments{cutlass::gemm::GemmUniversalMode::kGemm,                                            \
                               {M, N, K, 1},                                                                        \
                               {static_cast<const ElemAB *>(A), sa, static_cast<const ElemAB *>(B), sb},            \
                               {{alpha, beta}, D, sd, D, sd}};                                                      \
    }                                                                                                              \
    inline int run(int M, int N, int K, const void *A, const void *B, float *D, float alpha, float beta, void *ws, \
                   size_t ws_bytes, cudaStream_t s)                                                                \
    {                                                                                                              \
        auto a = args(M, N, K, A, B, D, alpha, beta);                                                              \
        Gemm g;                                                                                                    \
        if (g.can_implement(a) != cutlass::Status::kSuccess) return WS_EINVAL;                                    \
        if (Gemm::get_workspace_size(a) > ws_bytes) return WS_ECAPACITY;                                          \
        if (g.initialize(a, ws, s) != cutlass::Status::kSuccess) return WS_ECUDA;                                 \
        return g.run(s) == cutlass::Status::kSuccess ? WS_OK : WS_ECUDA;                                          \
    }                                                                                                              \
    inline size_t workspace(int M, int N, int K)                                                                   \
    {                                                                                                              \
        return Gemm::get_workspace_size(args(M, N, K, nullptr, nullptr, nullptr, 1.f, 0.f));                       \
    }                                                                                                              \
    }

// A[M,K] K-contiguous, B stored [N][K]  (forward: D = cols W^T)
WS_GEMM_CONFIG(GemmRC, cutlass::layout::RowMajor, cutlass::layout::ColumnMajor, 128, 128)
// A stored [K][M], B[K,N] N-contiguous   (weight gradient: dW = dZ^T cols)
WS_GEMM_CONFIG(GemmCR, cutlass::layout::ColumnMajor, cutlass::layout::RowMajor, 128, 128)
// the same with narrow tiles: a weight gradient has few of them and thousands
// of rows to add up.  Its rows are one chain of sums in the tensor memory, in
// order (sharing them out would round elsewhere), so more and lighter tiles
// are what shortens it.
WS_GEMM_CONFIG(GemmCR64, cutlass::layout::ColumnMajor, cutlass::layout::RowMajor, 64, 64)
// A[M,K], B[K,N] both row-major         (input gradient: dcols = dZ W)
WS_GEMM_CONFIG(GemmRR, cutlass::layout::RowMajor, cutlass::layout::RowMajor, 128, 128)

// max(v, 0) as k_bias_act takes it: a NaN becomes 0 (CUTLASS's ReLu keeps it).
// A positive value that bf16 rounds to 0 (at most half its smallest, 2^-133)
// becomes -0: the backward pass reads the ReLU's mask from the output, and such
// a value passes its gradient on.
__host__ __device__ __forceinline__ float relu_marked(float v)
{
    return v > 0.f ? (v > 0x1p-134f ? v : -0.f) : 0.f;
}
template <class V>
struct ReluMax {
    CUTLASS_HOST_DEVICE V operator()(V v) const { return relu_marked(v); }
};
template <class V, int N>
struct ReluMax<cutlass::Array<V, N>> {
    CUTLASS_HOST_DEVICE cutlass::Array<V, N> operator()(cutlass::Array<V, N> const &v) const
    {
        cutlass::Array<V, N> r;
        CUTLASS_PRAGMA_UNROLL
        for (int i = 0; i < N; i++) r[i] = relu_marked(v[i]);
        return r;
    }
};

// The forward layer: y[M,N] (bf16) = relu(A[M,K] W[N,K]^T + bias), the sums of
// GemmRC (same K blocks, same order) with the bias, the ReLU and the rounding
// in the epilogue, so the fp32 result is never written.  NT columns a tile: as
// wide as the layer where that still gives every SM a tile, else narrower.
template <int NT>
struct GemmAct {
    using ElemAB = cutlass::bfloat16_t;
    using Tile = cute::Shape<cute::_128, cute::Int<NT>, cute::_64>;
    using Cluster = cute::Shape<cute::_1, cute::_1, cute::_1>;
    using Fusion = cutlass::epilogue::fusion::LinCombPerColBiasEltAct<ReluMax, ElemAB, float, float, void>;
    using Epilogue = typename cutlass::epilogue::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, Tile, Cluster,
        cutlass::epilogue::collective::EpilogueTileAuto, float, float, void, cutlass::layout::RowMajor, 8, ElemAB,
        cutlass::layout::RowMajor, 8, cutlass::epilogue::collective::EpilogueScheduleAuto, Fusion>::CollectiveOp;
    using Mainloop = typename cutlass::gemm::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, ElemAB, cutlass::layout::RowMajor, 8, ElemAB,
        cutlass::layout::ColumnMajor, 8, float, Tile, Cluster,
        cutlass::gemm::collective::StageCountAutoCarveout<static_cast<int>(sizeof(typename Epilogue::SharedStorage))>,
        cutlass::gemm::collective::KernelScheduleAuto>::CollectiveOp;
    using Kernel = cutlass::gemm::kernel::GemmUniversal<cute::Shape<int, int, int, int>, Mainloop, Epilogue, void>;
    using Gemm = cutlass::gemm::device::GemmUniversalAdapter<Kernel>;
    static typename Gemm::Arguments args(int M, int N, int K, const void *A, const void *B, const float *bias, void *D)
    {
        auto sa = cutlass::make_cute_packed_stride(typename Kernel::StrideA{}, cute::make_shape(M, K, 1));
        auto sb = cutlass::make_cute_packed_stride(typename Kernel::StrideB{}, cute::make_shape(N, K, 1));
        auto sd = cutlass::make_cute_packed_stride(typename Kernel::StrideD{}, cute::make_shape(M, N, 1));
        typename Gemm::Arguments a{cutlass::gemm::GemmUniversalMode::kGemm,
                                   {M, N, K, 1},
                                   {static_cast<const ElemAB *>(A), sa, static_cast<const ElemAB *>(B), sb},
                                   {{}, nullptr, {}, static_cast<ElemAB *>(D), sd}};
        a.epilogue.thread.alpha = 1.f;
        a.epilogue.thread.beta = 0.f;
        a.epilogue.thread.bias_ptr = bias;
        return a;
    }
    static int run(int M, int N, int K, const void *A, const void *B, const float *bias, void *D, cudaStream_t s)
    {
        auto a = args(M, N, K, A, B, bias, D);
        Gemm g;
        if (g.can_implement(a) != cutlass::Status::kSuccess || Gemm::get_workspace_size(a) > 0) return WS_EINVAL;
        if (g.initialize(a, nullptr, s) != cutlass::Status::kSuccess) return WS_ECUDA;
        return g.run(s) == cutlass::Status::kSuccess ? WS_OK : WS_ECUDA;
    }
};

constexpr int T = 256;
constexpr int kSms = 148;

// n / d for n < 2^31 by a multiplication (Granlund and Montgomery 1994).
struct FastDiv {
    unsigned d, mul, shift;
    explicit FastDiv(unsigned div) : d(div)
    {
        shift = 0;
        while ((1ull << shift) < d) shift++;
        mul = (unsigned)(((1ull << 32) * ((1ull << shift) - d)) / d + 1);
    }
    __device__ __forceinline__ unsigned div(unsigned n) const { return (__umulhi(n, mul) + n) >> shift; }
    __device__ __forceinline__ void divmod(unsigned n, unsigned &q, unsigned &r) const
    {
        q = div(n);
        r = n - q * d;
    }
};

// The layers around the GEMMs move 16 bytes a thread (8 bf16 or 4 fp32
// channels, which the GEMMs' 16-byte rows guarantee); what does not fit that
// (channel counts or addresses that are no multiple, 2^31 pieces) takes the
// element-wise kernels further down.  One thread an element with 64-bit
// divisions ran at 1/12 of the memory's rate (im2col of 16 x 128^2 x 96: 1.2
// ms against 0.1 now).
inline bool wide(int C, int per, long long pieces, std::initializer_list<const void *> ps)
{
    if (C % per || pieces >= (1ll << 31)) return false;
    for (const void *p : ps)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

// im2col of one or two sources: channels [0, C0) from in0 (half the
// resolution where UP: a nearest 2x upsampling read in place), the rest from
// in1 (a skip connection), as the concatenated tensor would give.  dh: the
// rows of an image that this launch takes, from y0 on.
template <bool UP>
__global__ void __launch_bounds__(T) k_im2col16(unsigned total, int H, int W, int y0, int c0, int c1, FastDiv dk, FastDiv dc,
                                                FastDiv dw, FastDiv dh, const uint4 *__restrict__ in0,
                                                const uint4 *__restrict__ in1, uint4 *__restrict__ cols)
{
    for (unsigned q = blockIdx.x * T + threadIdx.x; q < total; q += gridDim.x * T) {
        unsigned row, k, tap, c, x, y, b, t;
        dk.divmod(q, row, k);
        dc.divmod(k, tap, c);
        dw.divmod(row, t, x);
        dh.divmod(t, b, y);
        y += y0;
        const int dy = (int)(tap * 11u >> 5), dx = (int)tap - 3 * dy;  // tap / 3, tap % 3 for tap < 9
        const int yy = (int)y + dy - 1, xx = (int)x + dx - 1;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) {
            if ((int)c >= c0) v = in1[(((size_t)b * H + yy) * W + xx) * c1 + c - c0];
            else if (UP) v = in0[(((size_t)b * (H / 2) + yy / 2) * (W / 2) + xx / 2) * c0 + c];
            else v = in0[(((size_t)b * H + yy) * W + xx) * c0 + c];
        }
        cols[q] = v;
    }
}

// col2im, 4 channels a thread: the taps in k_col2im's order.
__global__ void __launch_bounds__(T) k_col2im4(unsigned total, int H, int W, int c4, FastDiv dc, FastDiv dw, FastDiv dh,
                                               const float4 *__restrict__ dcols, float4 *__restrict__ dx)
{
    for (unsigned q = blockIdx.x * T + threadIdx.x; q < total; q += gridDim.x * T) {
        unsigned pix, c, x, y, b, t;
        dc.divmod(q, pix, c);
        dw.divmod(pix, t, x);
        dh.divmod(t, b, y);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int tap = 0; tap < 9; tap++) {
            const int oy = (int)y - (tap / 3 - 1), ox = (int)x - (tap % 3 - 1);
            if (oy < 0 || oy >= H || ox < 0 || ox >= W) continue;
            const float4 v = __ldcs(dcols + ((((size_t)b * H + oy) * W + ox) * 9 + tap) * c4 + c);
            acc.x += v.x;
            acc.y += v.y;
            acc.z += v.z;
            acc.w += v.w;
        }
        dx[q] = acc;
    }
}

__device__ __forceinline__ uint2 pack4(float4 v)
{
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    return make_uint2(reinterpret_cast<const unsigned &>(a), reinterpret_cast<const unsigned &>(b));
}
__device__ __forceinline__ float4 unpack4(uint2 v)
{
    const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(v.x));
    const float2 b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// dz = dy where the layer's output y is positive or -0 (relu_marked; y null:
// everywhere; bf16, for the GEMMs), and the column sums of that: a block's rows
// in a fixed order into part[block][C].
// A thread takes 4 channels of every T / w-th row, w pieces of 4 channels a
// block: all C / 4, or T of them from the block's y on.
__global__ void __launch_bounds__(T) k_act_back_sum(long long M, int Cn, int rows_per, const float4 *__restrict__ dy,
                                                    const uint2 *__restrict__ y, uint2 *__restrict__ dz,
                                                    float4 *__restrict__ part)
{
    extern __shared__ float4 sh[];
    const int c4 = Cn / 4, w0 = blockIdx.y * T, w = min(c4 - w0, T), lanes = T / w;
    const int at = threadIdx.x % w, c = w0 + at, lane = threadIdx.x / w;
    const long long r0 = (long long)blockIdx.x * rows_per, r1 = min(M, r0 + rows_per);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane < lanes) {
        for (long long r = r0 + lane; r < r1; r += lanes) {
            float4 g = dy[r * c4 + c];
            if (y != nullptr) {
                const float4 v = unpack4(y[r * c4 + c]);
                // (the bits less one: below the sign bit for these alone)
                const auto on = [](float u) { return (int)(__float_as_uint(u) - 1u) >= 0; };
                g.x = on(v.x) ? g.x : 0.f;
                g.y = on(v.y) ? g.y : 0.f;
                g.z = on(v.z) ? g.z : 0.f;
                g.w = on(v.w) ? g.w : 0.f;
            }
            dz[r * c4 + c] = pack4(g);
            acc.x += g.x;
            acc.y += g.y;
            acc.z += g.z;
            acc.w += g.w;
        }
        sh[threadIdx.x] = acc;
    }
    __syncthreads();
    if (lane == 0) {
        for (int l = 1; l < lanes; l++) {
            const float4 v = sh[l * w + at];
            acc.x += v.x;
            acc.y += v.y;
            acc.z += v.z;
            acc.w += v.w;
        }
        part[(size_t)blockIdx.x * c4 + c] = acc;
    }
}

// out[i] += the sum of `count` slices part[s][i] in a fixed order: 8 strands
// of slices, then the strands.
__global__ void __launch_bounds__(256) k_sum_slices(int n, int count, const float *__restrict__ part,
                                                    float *__restrict__ out)
{
    __shared__ float sh[8][33];
    const int i = blockIdx.x * 32 + threadIdx.x;
    float acc = 0.f;
    if (i < n)
        for (int s = threadIdx.y; s < count; s += 8) acc += part[(size_t)s * n + i];
    sh[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && i < n) {
        for (int k = 1; k < 8; k++) acc += sh[k][threadIdx.x];
        out[i] += acc;
    }
}

// 2x2 average pooling, 8 channels a thread (k_pool2's sums).
__global__ void __launch_bounds__(T) k_pool16(unsigned total, int W, int c8, FastDiv dc, FastDiv dw, FastDiv dh,
                                              const uint4 *__restrict__ in, uint4 *__restrict__ out)
{
    for (unsigned q = blockIdx.x * T + threadIdx.x; q < total; q += gridDim.x * T) {
        unsigned p, c, x, y, b, t;
        dc.divmod(q, p, c);
        dw.divmod(p, t, x);
        dh.divmod(t, b, y);
        const uint4 *src = in + (((size_t)b * 2 * dh.d + 2 * y) * W + 2 * x) * c8 + c;
        const uint4 v0 = src[0], v1 = src[c8], v2 = src[(size_t)W * c8], v3 = src[(size_t)(W + 1) * c8];
        uint4 r;
        const auto avg = [](unsigned a, unsigned b2, unsigned c2, unsigned d) {
            const float2 fa = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(a));
            const float2 fb = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(b2));
            const float2 fc = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(c2));
            const float2 fd = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 &>(d));
            const __nv_bfloat162 m = __floats2bfloat162_rn(0.25f * (fa.x + fb.x + fc.x + fd.x),
                                                           0.25f * (fa.y + fb.y + fc.y + fd.y));
            return reinterpret_cast<const unsigned &>(m);
        };
        r.x = avg(v0.x, v1.x, v2.x, v3.x);
        r.y = avg(v0.y, v1.y, v2.y, v3.y);
        r.z = avg(v0.z, v1.z, v2.z, v3.z);
        r.w = avg(v0.w, v1.w, v2.w, v3.w);
        out[q] = r;
    }
}

// The adjoint of the pooling with the skip connection's gradient added:
// din = dout / 4 + dskip, dskip being channels c0.. of rows of ct channels.
__global__ void __launch_bounds__(T) k_pool_back_skip(unsigned total, int W, int c4, int ct4, int c04, FastDiv dc,
                                                      FastDiv dw, FastDiv dh, const float4 *__restrict__ dout,
                                                      const float4 *__restrict__ skip, float4 *__restrict__ din)
{
    for (unsigned q = blockIdx.x * T + threadIdx.x; q < total; q += gridDim.x * T) {
        unsigned p, c, x, y, b, t;
        dc.divmod(q, p, c);
        dw.divmod(p, t, x);
        dh.divmod(t, b, y);
        const float4 d = dout[(((size_t)b * (dh.d / 2) + y / 2) * (W / 2) + x / 2) * c4 + c];
        const float4 s = skip[(size_t)p * ct4 + c04 + c];
        din[q] = make_float4(0.25f * d.x + s.x, 0.25f * d.y + s.y, 0.25f * d.z + s.z, 0.25f * d.w + s.w);
    }
}

// The adjoint of the upsampling, 4 channels a thread (k_up2_back's sums).
__global__ void __launch_bounds__(T) k_up_back4(unsigned total, int W, int c4, int ct4, FastDiv dc, FastDiv dw, FastDiv dh,
                                                const float4 *__restrict__ dout, float4 *__restrict__ din)
{
    for (unsigned q = blockIdx.x * T + threadIdx.x; q < total; q += gridDim.x * T) {
        unsigned p, c, x, y, b, t;
        dc.divmod(q, p, c);
        dw.divmod(p, t, x);
        dh.divmod(t, b, y);
        const float4 *src = dout + (((size_t)b * 2 * dh.d + 2 * y) * 2 * W + 2 * x) * ct4 + c;
        const float4 v0 = src[0], v1 = src[ct4], v2 = src[(size_t)2 * W * ct4], v3 = src[(size_t)(2 * W + 1) * ct4];
        din[q] = make_float4(v0.x + v1.x + v2.x + v3.x, v0.y + v1.y + v2.y + v3.y, v0.z + v1.z + v2.z + v3.z,
                             v0.w + v1.w + v2.w + v3.w);
    }
}

// ---------------------------------------------------------------------------
// im2col / col2im for 3x3, stride 1, zero padding 1, NHWC
// ---------------------------------------------------------------------------
// cols[(b*H + y)*W + x][tap*C + c] = in[b][y+dy][x+dx][c], tap = (dy+1)*3 + (dx+1)
__global__ void k_im2col(int B, int H, int W, int Cn, const bf16 *__restrict__ in, bf16 *__restrict__ cols)
{
    const long long K = 9LL * Cn;
    const long long total = (long long)B * H * W * K;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const long long row = q / K;
        const int k = (int)(q - row * K);
        const int tap = k / Cn, c = k - tap * Cn;
        const int x = (int)(row % W), y = (int)((row / W) % H), b = (int)(row / ((long long)W * H));
        const int yy = y + tap / 3 - 1, xx = x + tap % 3 - 1;
        bf16 v = __float2bfloat16(0.f);
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) v = in[(((long long)b * H + yy) * W + xx) * Cn + c];
        cols[q] = v;
    }
}

// dx[b][y][x][c] = sum over the (up to 9) output pixels that read it: a
// gather, so the sum order is fixed and no atomics are needed.
__global__ void k_col2im(int B, int H, int W, int Cn, const float *__restrict__ dcols, float *__restrict__ dx)
{
    const long long K = 9LL * Cn;
    const long long total = (long long)B * H * W * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % Cn);
        const long long pix = q / Cn;
        const int x = (int)(pix % W), y = (int)((pix / W) % H), b = (int)(pix / ((long long)W * H));
        float acc = 0.f;
        for (int tap = 0; tap < 9; tap++) {
            // output pixel (y - dy, x - dx) read this input through tap (dy, dx)
            const int oy = y - (tap / 3 - 1), ox = x - (tap % 3 - 1);
            if (oy < 0 || oy >= H || ox < 0 || ox >= W) continue;
            acc += dcols[(((long long)b * H + oy) * W + ox) * K + tap * Cn + c];
        }
        dx[q] = acc;
    }
}

// y = relu(d + bias) (bf16), pre = d + bias kept for the backward pass
__global__ void k_bias_act(long long M, int Cn, const float *__restrict__ d, const float *__restrict__ bias,
                           int relu, bf16 *__restrict__ y, float *__restrict__ pre)
{
    const long long total = M * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const float v = d[q] + bias[q % Cn];
        if (pre) pre[q] = v;
        y[q] = __float2bfloat16(relu ? fmaxf(v, 0.f) : v);
    }
}

// dz = dy * relu'(pre) in bf16 for the GEMMs
__global__ void k_act_back(long long n, int relu, const float *__restrict__ dy, const float *__restrict__ pre,
                           bf16 *__restrict__ dz, float *__restrict__ dz32)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const float g = (!relu || pre[q] > 0.f) ? dy[q] : 0.f;
        dz[q] = __float2bfloat16(g);
        if (dz32) dz32[q] = g;
    }
}

// db[c] = sum_m dz[m][c], one block per channel, fixed order
__global__ void k_colsum(long long M, int Cn, const float *__restrict__ dz, float *__restrict__ db)
{
    __shared__ float sh[T];
    const int c = blockIdx.x;
    float acc = 0.f;
    for (long long m = threadIdx.x; m < M; m += blockDim.x) acc += dz[m * Cn + c];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) db[c] = sh[0];
}

// 2x2 average pooling (H, W even) and its adjoint
__global__ void k_pool2(int B, int H, int W, int Cn, const bf16 *__restrict__ in, bf16 *__restrict__ out)
{
    const int Ho = H / 2, Wo = W / 2;
    const long long total = (long long)B * Ho * Wo * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % Cn);
        const long long p = q / Cn;
        const int x = (int)(p % Wo), y = (int)((p / Wo) % Ho), b = (int)(p / ((long long)Wo * Ho));
        const bf16 *src = in + (((long long)b * H + 2 * y) * W + 2 * x) * Cn + c;
        const float s = __bfloat162float(src[0]) + __bfloat162float(src[Cn]) + __bfloat162float(src[(long long)W * Cn]) +
                        __bfloat162float(src[(long long)W * Cn + Cn]);
        out[q] = __float2bfloat16(0.25f * s);
    }
}

__global__ void k_pool2_back(int B, int H, int W, int Cn, const float *__restrict__ dout, float *__restrict__ din)
{
    const long long total = (long long)B * H * W * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % Cn);
        const long long p = q / Cn;
        const int x = (int)(p % W), y = (int)((p / W) % H), b = (int)(p / ((long long)W * H));
        din[q] = 0.25f * dout[(((long long)b * (H / 2) + y / 2) * (W / 2) + x / 2) * Cn + c];
    }
}

// nearest 2x upsampling into channels [c0, c0 + Cn) of an output with Ct channels
__global__ void k_up2(int B, int H, int W, int Cn, const bf16 *__restrict__ in, int Ct, int c0, bf16 *__restrict__ out)
{
    const long long total = (long long)B * (2 * H) * (2 * W) * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % Cn);
        const long long p = q / Cn;
        const int x = (int)(p % (2 * W)), y = (int)((p / (2 * W)) % (2 * H)), b = (int)(p / (4LL * W * H));
        out[p * Ct + c0 + c] = in[(((long long)b * H + y / 2) * W + x / 2) * Cn + c];
    }
}

__global__ void k_up2_back(int B, int H, int W, int Cn, const float *__restrict__ dout, int Ct, int c0,
                           float *__restrict__ din)
{
    const long long total = (long long)B * H * W * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(q % Cn);
        const long long p = q / Cn;
        const int x = (int)(p % W), y = (int)((p / W) % H), b = (int)(p / ((long long)W * H));
        float s = 0.f;
        for (int dy = 0; dy < 2; dy++)
            for (int dx = 0; dx < 2; dx++)
                s += dout[(((long long)b * 2 * H + 2 * y + dy) * 2 * W + 2 * x + dx) * Ct + c0 + c];
        din[q] = s;
    }
}

// copy channels: out[p][c0 + c] = in[p][c] (a skip connection into a concat
// buffer) and the backward split din[p][c] = dout[p][c0 + c]
__global__ void k_put_channels(long long P, int Cn, const bf16 *__restrict__ in, int Ct, int c0, bf16 *__restrict__ out)
{
    const long long total = P * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x)
        out[(q / Cn) * Ct + c0 + q % Cn] = in[q];
}

__global__ void k_take_channels(long long P, int Cn, const float *__restrict__ dout, int Ct, int c0, float add,
                                float *__restrict__ din)
{
    const long long total = P * Cn;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const float v = dout[(q / Cn) * Ct + c0 + q % Cn];
        din[q] = add != 0.f ? din[q] + v : v;
    }
}

// Mean-free error per sample on a gy x gx grid: the weights are defined up
// to a constant, so prediction and target are compared after removing each
// one's mean.  With e = pred - target - mean:
//   loss_b = [ sum_i e_i^2 + lambda * sum (forward differences of e)^2 ] / (n B)
// (the second term weighs the local differences that set the cells' masses)
// and grad = d(sum_b loss_b) / d pred.
__global__ void k_mse_centered(int B, int gy, int gx, float lambda, const float *__restrict__ p,
                               const float *__restrict__ t, float *__restrict__ grad, float *__restrict__ loss_b)
{
    __shared__ float sh[T];
    const int n = gy * gx;
    const int b = blockIdx.x;
    const float *pb = p + (long long)b * n;
    const float *tb = t + (long long)b * n;
    float acc = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += pb[i] - tb[i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    const float mean = sh[0] / n;
    __syncthreads();
    const float sc = 1.f / ((float)n * B);
    float l = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int x = i % gx, y = i / gx;
        const float e = pb[i] - tb[i] - mean;
        float g = 2.f * e;
        l += e * e;
        if (lambda != 0.f) {
            // differences to the right / upper neighbour (counted once) and
            // the gradient of every difference this site is part of
            if (x + 1 < gx) {
                const float d = (pb[i + 1] - tb[i + 1] - mean) - e;
                l += lambda * d * d;
                g -= 2.f * lambda * d;
            }
            if (x > 0) g += 2.f * lambda * (e - (pb[i - 1] - tb[i - 1] - mean));
            if (y + 1 < gy) {
                const float d = (pb[i + gx] - tb[i + gx] - mean) - e;
                l += lambda * d * d;
                g -= 2.f * lambda * d;
            }
            if (y > 0) g += 2.f * lambda * (e - (pb[i - gx] - tb[i - gx] - mean));
        }
        grad[(long long)b * n + i] = g * sc;
    }
    sh[threadIdx.x] = l;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss_b[b] = sh[0] * sc;
}

// Adam on fp32 master weights, with the bf16 copy the GEMMs read
__global__ void k_adam(long long n, float *__restrict__ w, bf16 *__restrict__ w16, const float *__restrict__ g,
                       float *__restrict__ m, float *__restrict__ v, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const float gq = g[q];
        const float mq = b1 * m[q] + (1.f - b1) * gq;
        const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        const float wq = w[q] - lr * (mq / c1) / (sqrtf(vq / c2) + eps);
        w[q] = wq;
        if (w16) w16[q] = __float2bfloat16(wq);
    }
}

__global__ void k_to_bf16(long long n, const float *__restrict__ x, bf16 *__restrict__ y)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x)
        y[q] = __float2bfloat16(x[q]);
}

inline int grid16(unsigned total)
{
    return (int)std::min<unsigned>((total + T - 1) / T, kSms * 16u);
}

inline bool narrow_cr(int M, int N) { return ((M + 127) / 128) * ((N + 127) / 128) < kSms; }

inline int grid_for(long long n)
{
    const long long b = (n + T - 1) / T;
    return (int)(b < 148LL * 32 ? b : 148LL * 32);
}

inline int last_error()
{
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ECUDA;
}

}  // namespace

extern "C" {

WS_API int ws_gemm(int layout, int M, int N, int K, const void *A, const void *B, float *D, float alpha, float beta,
                   void *workspace, size_t workspace_bytes, void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !D) return WS_EINVAL;
    if (K % 8 != 0) return WS_EINVAL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (layout) {
    case WS_GEMM_RC: return GemmRC::run(M, N, K, A, B, D, alpha, beta, workspace, workspace_bytes, s);
    case WS_GEMM_CR:
        if (M % 8 != 0 || N % 8 != 0) return WS_EINVAL;
        if (narrow_cr(M, N)) return GemmCR64::run(M, N, K, A, B, D, alpha, beta, workspace, workspace_bytes, s);
        return GemmCR::run(M, N, K, A, B, D, alpha, beta, workspace, workspace_bytes, s);
    case WS_GEMM_RR:
        if (N % 8 != 0) return WS_EINVAL;
        return GemmRR::run(M, N, K, A, B, D, alpha, beta, workspace, workspace_bytes, s);
    default: return WS_EINVAL;
    }
}

WS_API size_t ws_gemm_workspace(int layout, int M, int N, int K)
{
    switch (layout) {
    case WS_GEMM_RC: return GemmRC::workspace(M, N, K);
    case WS_GEMM_CR: return narrow_cr(M, N) ? GemmCR64::workspace(M, N, K) : GemmCR::workspace(M, N, K);
    case WS_GEMM_RR: return GemmRR::workspace(M, N, K);
    default: return 0;
    }
}

WS_API int ws_im2col(int B, int H, int W, int C, const void *in, void *cols, void *stream)
{
    const long long n = (long long)B * H * W * 9 * C;
    if (n > 0 && wide(C, 8, n / 8, {in, cols})) {
        const unsigned c8 = C / 8, total = (unsigned)(n / 8);
        k_im2col16<false><<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
            total, H, W, 0, (int)c8, 0, FastDiv(9 * c8), FastDiv(c8), FastDiv(W), FastDiv(H),
            static_cast<const uint4 *>(in), nullptr, static_cast<uint4 *>(cols));
        return last_error();
    }
    k_im2col<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, static_cast<const bf16 *>(in),
                                                                        static_cast<bf16 *>(cols));
    return last_error();
}

WS_API int ws_im2col_up(int B, int H, int W, int C0, const void *up, int C1, const void *skip, void *cols, void *stream)
{
    if (B <= 0 || H <= 0 || W <= 0 || H % 2 || W % 2 || C0 <= 0 || C0 % 8 || C1 <= 0 || !wide(C1, 8, 0, {up, skip, cols}))
        return WS_EINVAL;
    // launches of at most 2^30 pieces: all images, a few, or bands of one's rows
    const unsigned c0 = C0 / 8, c1 = C1 / 8, c8 = c0 + c1;
    const long long row = (long long)W * 9 * c8, most = 1ll << 30;
    if (row > most) return WS_EINVAL;
    const int band = (int)std::min<long long>(H, most / row);
    const int images = band < H ? 1 : (int)std::min<long long>(B, most / (row * H));
    for (int b = 0; b < B; b += images)
        for (int y = 0; y < H; y += band) {
            const int ni = std::min(images, B - b), ny = std::min(band, H - y);
            const unsigned total = (unsigned)(row * ny * ni);
            k_im2col16<true><<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
                total, H, W, y, c0, c1, FastDiv(9 * c8), FastDiv(c8), FastDiv(W), FastDiv(ny),
                static_cast<const uint4 *>(up) + (size_t)b * (H / 2) * (W / 2) * c0,
                static_cast<const uint4 *>(skip) + (size_t)b * H * W * c1,
                static_cast<uint4 *>(cols) + ((size_t)b * H + y) * row);
        }
    return last_error();
}

WS_API int ws_layer(int M, int N, int K, const void *A, const void *Wt, const float *bias, void *y, void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0 || !A || !Wt || !bias || !y || K % 8 || !wide(N, 8, 0, {A, Wt, bias, y}))
        return WS_EINVAL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int rows = (M + 127) / 128;
    if (N > 64 && rows * ((N + 127) / 128) >= kSms) return GemmAct<128>::run(M, N, K, A, Wt, bias, y, s);
    if (N > 32 && rows * ((N + 63) / 64) >= kSms) return GemmAct<64>::run(M, N, K, A, Wt, bias, y, s);
    return GemmAct<32>::run(M, N, K, A, Wt, bias, y, s);
}

WS_API size_t ws_act_back_sum_workspace(int C) { return (size_t)kSms * 4 * C * sizeof(float); }

WS_API int ws_act_back_sum(long long M, int C, const float *dy, const void *y, void *dz, float *gb, void *workspace,
                           size_t workspace_bytes, void *stream)
{
    if (M <= 0 || C <= 0 || !dy || !dz || !workspace || C % 8) return WS_EINVAL;
    if (!wide(C, 4, M * (C / 4), {dy, y, dz, workspace}) || workspace_bytes < ws_act_back_sum_workspace(C))
        return WS_EINVAL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *part = static_cast<float *>(workspace);
    const int rows_per = (int)std::max<long long>((M + 4 * kSms - 1) / (4 * kSms), 32);
    const int blocks = (int)((M + rows_per - 1) / rows_per);
    const dim3 grid((unsigned)blocks, (unsigned)((C / 4 + T - 1) / T));
    k_act_back_sum<<<grid, T, T * sizeof(float4), s>>>(M, C, rows_per, reinterpret_cast<const float4 *>(dy),
                                                         static_cast<const uint2 *>(y), static_cast<uint2 *>(dz),
                                                         reinterpret_cast<float4 *>(part));
    if (gb) k_sum_slices<<<(C + 31) / 32, dim3(32, 8), 0, s>>>(C, blocks, part, gb);
    return last_error();
}

WS_API int ws_pool2_back_skip(int B, int H, int W, int C, const float *dout, const float *dskip, int Ct, int c0, float *din,
                              void *stream)
{
    const long long n = (long long)B * H * W * C;
    if (n <= 0 || H % 2 || W % 2 || Ct % 4 || c0 % 4 || !wide(C, 4, n / 4, {dout, dskip, din})) return WS_EINVAL;
    const unsigned total = (unsigned)(n / 4);
    k_pool_back_skip<<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
        total, W, C / 4, Ct / 4, c0 / 4, FastDiv(C / 4), FastDiv(W), FastDiv(H), reinterpret_cast<const float4 *>(dout),
        reinterpret_cast<const float4 *>(dskip), reinterpret_cast<float4 *>(din));
    return last_error();
}

WS_API int ws_col2im(int B, int H, int W, int C, const float *dcols, float *dx, void *stream)
{
    const long long n = (long long)B * H * W * C;
    if (n > 0 && wide(C, 4, n * 9 / 4, {dcols, dx})) {
        const unsigned total = (unsigned)(n / 4);
        k_col2im4<<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
            total, H, W, C / 4, FastDiv(C / 4), FastDiv(W), FastDiv(H), reinterpret_cast<const float4 *>(dcols),
            reinterpret_cast<float4 *>(dx));
        return last_error();
    }
    k_col2im<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, dcols, dx);
    return last_error();
}

WS_API int ws_bias_act(long long M, int C, const float *d, const float *bias, int relu, void *y, float *pre,
                       void *stream)
{
    k_bias_act<<<grid_for(M * C), T, 0, static_cast<cudaStream_t>(stream)>>>(M, C, d, bias, relu,
                                                                              static_cast<bf16 *>(y), pre);
    return last_error();
}

WS_API int ws_act_back(long long n, int relu, const float *dy, const float *pre, void *dz, float *dz32, void *stream)
{
    k_act_back<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(n, relu, dy, pre, static_cast<bf16 *>(dz),
                                                                          dz32);
    return last_error();
}

WS_API int ws_colsum(long long M, int C, const float *dz, float *db, void *stream)
{
    k_colsum<<<C, T, 0, static_cast<cudaStream_t>(stream)>>>(M, C, dz, db);
    return last_error();
}

WS_API int ws_pool2(int B, int H, int W, int C, const void *in, void *out, void *stream)
{
    if (H % 2 || W % 2) return WS_EINVAL;
    const long long n = (long long)B * (H / 2) * (W / 2) * C;
    if (n > 0 && wide(C, 8, n / 2, {in, out})) {
        const unsigned total = (unsigned)(n / 8);
        k_pool16<<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
            total, W, C / 8, FastDiv(C / 8), FastDiv(W / 2), FastDiv(H / 2), static_cast<const uint4 *>(in),
            static_cast<uint4 *>(out));
        return last_error();
    }
    k_pool2<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, static_cast<const bf16 *>(in),
                                                                        static_cast<bf16 *>(out));
    return last_error();
}

WS_API int ws_pool2_back(int B, int H, int W, int C, const float *dout, float *din, void *stream)
{
    if (H % 2 || W % 2) return WS_EINVAL;
    const long long n = (long long)B * H * W * C;
    k_pool2_back<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, dout, din);
    return last_error();
}

WS_API int ws_up2(int B, int H, int W, int C, const void *in, int Ct, int c0, void *out, void *stream)
{
    const long long n = (long long)B * 4 * H * W * C;
    k_up2<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, static_cast<const bf16 *>(in), Ct, c0,
                                                                      static_cast<bf16 *>(out));
    return last_error();
}

WS_API int ws_up2_back(int B, int H, int W, int C, const float *dout, int Ct, int c0, float *din, void *stream)
{
    const long long n = (long long)B * H * W * C;
    if (n > 0 && Ct % 4 == 0 && c0 % 4 == 0 && wide(C, 4, (long long)B * H * W * Ct, {dout, din})) {
        const unsigned total = (unsigned)(n / 4);
        k_up_back4<<<grid16(total), T, 0, static_cast<cudaStream_t>(stream)>>>(
            total, W, C / 4, Ct / 4, FastDiv(C / 4), FastDiv(W), FastDiv(H),
            reinterpret_cast<const float4 *>(dout) + c0 / 4, reinterpret_cast<float4 *>(din));
        return last_error();
    }
    k_up2_back<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(B, H, W, C, dout, Ct, c0, din);
    return last_error();
}

WS_API int ws_put_channels(long long P, int C, const void *in, int Ct, int c0, void *out, void *stream)
{
    k_put_channels<<<grid_for(P * C), T, 0, static_cast<cudaStream_t>(stream)>>>(
        P, C, static_cast<const bf16 *>(in), Ct, c0, static_cast<bf16 *>(out));
    return last_error();
}

WS_API int ws_take_channels(long long P, int C, const float *dout, int Ct, int c0, int add, float *din, void *stream)
{
    k_take_channels<<<grid_for(P * C), T, 0, static_cast<cudaStream_t>(stream)>>>(P, C, dout, Ct, c0,
                                                                                   add ? 1.f : 0.f, din);
    return last_error();
}

WS_API int ws_mse_centered(int B, int gy, int gx, float lambda, const float *pred, const float *target, float *grad,
                           float *loss_b, void *stream)
{
    if (B <= 0 || gy <= 0 || gx <= 0) return WS_EINVAL;
    k_mse_centered<<<B, T, 0, static_cast<cudaStream_t>(stream)>>>(B, gy, gx, lambda, pred, target, grad, loss_b);
    return last_error();
}

WS_API int ws_adam(long long n, float *w, void *w16, const float *g, float *m, float *v, float lr, float b1, float b2,
                   float eps, int step, void *stream)
{
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(n, w, static_cast<bf16 *>(w16), g, m, v, lr, b1,
                                                                      b2, eps, c1, c2);
    return last_error();
}

WS_API int ws_to_bf16(long long n, const float *x, void *y, void *stream)
{
    k_to_bf16<<<grid_for(n), T, 0, static_cast<cudaStream_t>(stream)>>>(n, x, static_cast<bf16 *>(y));
    return last_error();
}

}  // extern "C"
