// Column sums of bf16 matrices (bias gradients), the backward of the gated residual, and scaling in place.  All are bound by HBM.
#include "common.cuh"

namespace {

constexpr int kWarps = 8, kCols = 256;      // a warp reads 256 columns of a row (16 bytes a lane), a block 8 rows at a time

// partial[b][split][c] = sum over the rows of batch b that the split walks of x[r][c] (times y[r][c] if GATED, which also writes
// out = x * gate[b]).  Blocks: (batch and column group, row split); the warps of a block take every 8th row, four rows in flight each,
// and meet in shared memory.  Rows are split so that the grid fills the SMs whatever the width is: 8192 x 3840 -> 15 x 40 blocks.
template <bool GATED>
__global__ void __launch_bounds__(kWarps * 32) column_sum_kernel(const bf16* __restrict__ x, const bf16* __restrict__ y,
                                                                const bf16* __restrict__ gate, bf16* __restrict__ out,
                                                                float* __restrict__ partial, int rows, int cols, long long ldx) {
    __shared__ float tile[kWarps][kCols + 4];
    const int groups = (cols + kCols - 1) / kCols, b = blockIdx.x / groups, c0 = (blockIdx.x - b * groups) * kCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = c0 + lane * 8;
    const int split = blockIdx.y, splits = gridDim.y;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c < cols) {
        const bf16* xb = x + (size_t)b * rows * ldx + c;
        float g[8];
        if constexpr (GATED) unpack8(*reinterpret_cast<const Vec8*>(gate + (size_t)b * cols + c), g);
#pragma unroll 4
        for (int r = split * kWarps + warp; r < rows; r += splits * kWarps) {
            float f[8];
            unpack8(*reinterpret_cast<const Vec8*>(xb + (size_t)r * ldx), f);
            if constexpr (GATED) {
                const size_t at = ((size_t)b * rows + r) * cols + c;
                float h[8];
                unpack8(*reinterpret_cast<const Vec8*>(y + at), h);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    acc[k] += f[k] * h[k];
                    f[k] *= g[k];
                }
                *reinterpret_cast<Vec8*>(out + at) = pack8(f);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[k] += f[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) tile[warp][lane * 8 + k] = acc[k];
    __syncthreads();
    const int col = c0 + threadIdx.x;
    if (col < cols) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s += tile[w][threadIdx.x];
        partial[((size_t)b * splits + split) * cols + col] = s;
    }
}

// sums[b][c] = sum over the splits, in their order
__global__ void __launch_bounds__(256) fold_splits_kernel(const float* __restrict__ partial, bf16* __restrict__ sums, int splits, int cols) {
    __shared__ float tile[8][33];
    const int groups = (cols + 31) / 32, b = blockIdx.x / groups, c = (blockIdx.x - b * groups) * 32 + threadIdx.x;
    float s = 0.f;
    if (c < cols)
#pragma unroll 4
        for (int p = threadIdx.y; p < splits; p += 8) s += partial[((size_t)b * splits + p) * cols + c];
    tile[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && c < cols) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += tile[k][threadIdx.x];
        sums[(size_t)b * cols + c] = __float2bfloat16(t);
    }
}

// x *= *scale in place; nothing is read when the scale is one
__global__ void __launch_bounds__(256) scale_kernel(bf16* __restrict__ x, long long n, const float* __restrict__ scale) {
    const float s = *scale;
    if (s == 1.f) return;
    const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long i = first; i < n >> 4; i += stride) {
        Vec16 v = ld_v16(x + i * 16);
        float f[16];
        unpack16(v, f);
#pragma unroll
        for (int k = 0; k < 16; ++k) f[k] *= s;
        st_v16(x + i * 16, pack16(f));
    }
    for (long long i = (n & ~15LL) + first; i < n; i += stride) x[i] = __float2bfloat16(__bfloat162float(x[i]) * s);
}

int splits_of(int rows, int cols, int batches) {
    if (rows < 1 || cols < 1 || batches < 1) return 1;
    const long long groups = (long long)((cols + kCols - 1) / kCols) * batches;
    long long s = (148 * 4 + groups - 1) / groups;                   // four blocks an SM
    const long long most = (rows + kWarps * 4 - 1) / (kWarps * 4);     // at least four rows a warp
    s = s < most ? s : most;
    return (int)(s < 1 ? 1 : s);
}

}  // namespace

// Row splits, i.e. scratch of batches * splits * cols floats for the two entries below.
MM_API int mm_column_splits(int rows, int cols, int batches) { return splits_of(rows, cols, batches); }

// sums[c] (bf16) = sum over r of x[r, c], fp32 inside.  x: [rows, cols] bf16 with ldx elements between rows; cols and ldx multiples
// of 8, 16-byte aligned.  8192 x (3840 + 1280 + 6912 + 1280): see native.py.
MM_API int mm_column_sum(const void* x, void* sums, float* partial, int rows, int cols, long long ldx, cudaStream_t st) {
    if (cols % 8 || ldx % 8 || ((uintptr_t)x & 15)) return -1;
    if (rows < 1 || cols < 1) return -2;
    const int splits = splits_of(rows, cols, 1);
    column_sum_kernel<false><<<dim3((cols + kCols - 1) / kCols, splits), kWarps * 32, 0, st>>>((const bf16*)x, nullptr, nullptr, nullptr,
                                                                                                  partial, rows, cols, ldx);
    fold_splits_kernel<<<(cols + 31) / 32, dim3(32, 8), 0, st>>>(partial, (bf16*)sums, splits, cols);
    return (int)cudaGetLastError();
}

// Backward of x + gate[b] * y: dy = dout * gate[b], dgate[b, c] = sum over the rows of dout * y (fp32 inside).  dout, y, dy: dense
// [batches, rows, cols]; one pass over dout and y.  Nothing to sum over (rows == 0): zeros.
MM_API int mm_gated_residual_bwd(const void* dout, const void* y, const void* gate, void* dy, void* dgate, float* partial, int batches,
                                 int rows, int cols, cudaStream_t st) {
    if (cols % 8 || ((uintptr_t)dout | (uintptr_t)y | (uintptr_t)gate | (uintptr_t)dy) & 15) return -1;
    if (rows < 0 || cols < 0 || batches < 0) return -2;
    if (!batches || !cols) return 0;
    if (!rows) return (int)cudaMemsetAsync(dgate, 0, (size_t)batches * cols * sizeof(bf16), st);
    const long long blocks = (long long)batches * ((cols + 31) / 32);       // a gate per token is as many batches as there are tokens
    if (blocks > 0x7fffffffLL) return -2;
    const int splits = splits_of(rows, cols, batches);
    column_sum_kernel<true><<<dim3(batches * ((cols + kCols - 1) / kCols), splits), kWarps * 32, 0, st>>>(
        (const bf16*)dout, (const bf16*)y, (const bf16*)gate, (bf16*)dy, partial, rows, cols, cols);
    fold_splits_kernel<<<(int)blocks, dim3(32, 8), 0, st>>>(partial, (bf16*)dgate, splits, cols);
    return (int)cudaGetLastError();
}

// x: n bf16, 32-byte aligned; scale: one fp32 on the device.
MM_API int mm_scale_bf16(void* x, long long n, const float* scale, cudaStream_t st) {
    if ((uintptr_t)x & 31) return -1;
    if (n < 1) return 0;
    const long long blocks = (n / 16 + 255) / 256;
    scale_kernel<<<(int)(blocks < 1 ? 1 : blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, st>>>((bf16*)x, n, scale);
    return (int)cudaGetLastError();
}
