// Column sums of bf16 matrices (bias gradients), the backward of the gated residual, and scaling in place.  All are bound by HBM.
#include "common.cuh"

namespace {

constexpr int kWarps = 8, kCols = 256;      // a warp reads 256 columns of a row (16 bytes a lane), or several rows of a narrower matrix
constexpr int kFlight = 8;                  // rows that a lane has in flight

// Lanes of a warp that share a row: a power of two, 32 from 256 columns on.
__host__ __device__ __forceinline__ int lanes_per_row(int cols) {
    int n = 1;
    while (n < 32 && n * 8 < cols) n *= 2;
    return n;
}

// partial[b][split][c] = sum over the rows of batch b that the split walks of x[r][c] (times y[r][c] if GATED, which also writes
// out = x * gate[b]).  Blocks: (batch and column group, row split); the warps of a block take every 8th row (or group of rows of a
// narrow matrix) and meet in shared memory.  Rows are split so that the grid fills the SMs whatever the width is (see splits_of).
// Bound by HBM.  Plain sums have eight rows a lane in flight, asked for before the first is added: 75600 x 13824 347 us, 75600 x 5120
// 146, 300000 x 8 15; 476, 187 and 46 in a loop unrolled four times with a row per warp whatever its width, 370, 182 and 20 as
// torch.sum.  With a gate, which reads two rows and writes one, that loop stays: 1 x 32760 x 5120 183 us, 228 with eight in flight.
template <bool GATED>
__global__ void __launch_bounds__(kWarps * 32) column_sum_kernel(const bf16* __restrict__ x, const bf16* __restrict__ y,
                                                                const bf16* __restrict__ gate, bf16* __restrict__ out,
                                                                float* __restrict__ partial, int rows, int cols, long long ldx) {
    let_successor_start();
    __shared__ float tile[kWarps][kCols + 4];
    const int groups = (cols + kCols - 1) / kCols, b = blockIdx.x / groups, c0 = (blockIdx.x - b * groups) * kCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per_row = lanes_per_row(cols), sub = lane / per_row, at_once = 32 / per_row;
    const int c = c0 + (lane - sub * per_row) * 8, split = blockIdx.y, splits = gridDim.y;
    const long long step = (long long)splits * kWarps * at_once;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c < cols) {
        const bf16* xb = x + (size_t)b * rows * ldx + c;
        float g[8];
        if constexpr (GATED) unpack8(*reinterpret_cast<const Vec8*>(gate + (size_t)b * cols + c), g);
        long long r = (long long)(split * kWarps + warp) * at_once + sub;
        if constexpr (GATED) {
#pragma unroll 4
            for (; r < rows; r += step) {
                const size_t at = ((size_t)b * rows + r) * cols + c;
                float f[8], h[8];
                unpack8(*reinterpret_cast<const Vec8*>(xb + r * ldx), f);
                unpack8(*reinterpret_cast<const Vec8*>(y + at), h);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    acc[k] += f[k] * h[k];
                    f[k] *= g[k];
                }
                *reinterpret_cast<Vec8*>(out + at) = pack8(f);
            }
        } else {
            for (; r < rows; r += kFlight * step) {
                Vec8 v[kFlight];
#pragma unroll
                for (int j = 0; j < kFlight; ++j)
                    if (r + j * step < rows) v[j] = *reinterpret_cast<const Vec8*>(xb + (r + j * step) * ldx);
#pragma unroll
                for (int j = 0; j < kFlight; ++j) {
                    if (r + j * step >= rows) break;
                    float f[8];
                    unpack8(v[j], f);
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[k] += f[k];
                }
            }
        }
    }
    for (int o = per_row; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (sub == 0)
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

// Batches of fewer rows than a block has warps (a gate per token, or per few): a thread walks the rows of 8 columns of a batch itself.
// dy = dout * gate[b], dgate[b][c] = sum over the rows of dout * y.  70000 x 1 x 512 75 us, 4096 x 1 x 3072 33; 1218 and 419 with a block
// for each batch and column group, 431 and 153 in PyTorch.
__global__ void __launch_bounds__(256) gated_short_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ y, const bf16* __restrict__ gate,
                                                          bf16* __restrict__ dy, bf16* __restrict__ dgate, int batches, int rows, int cols) {
    let_successor_start();
    const int vecs = cols >> 3;
    const long long total = (long long)batches * vecs;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const long long b = i / vecs;
        const int c = (int)(i - b * vecs) * 8;
        float g[8], acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        unpack8(*reinterpret_cast<const Vec8*>(gate + b * cols + c), g);
        for (int r = 0; r < rows; ++r) {
            const size_t at = (size_t)(b * rows + r) * cols + c;
            float f[8], h[8];
            unpack8(*reinterpret_cast<const Vec8*>(dout + at), f);
            unpack8(*reinterpret_cast<const Vec8*>(y + at), h);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                acc[k] += f[k] * h[k];
                f[k] *= g[k];
            }
            *reinterpret_cast<Vec8*>(dy + at) = pack8(f);
        }
        *reinterpret_cast<Vec8*>(dgate + b * cols + c) = pack8(acc);
    }
}

// sums[b][c] = sum over the splits, in their order
__global__ void __launch_bounds__(256) fold_splits_kernel(const float* __restrict__ partial, bf16* __restrict__ sums, int splits, int cols) {
    let_successor_start();
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
    let_successor_start();
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

int splits_of(int rows, int cols, int batches, bool gated) {
    if (rows < 1 || cols < 1 || batches < 1) return 1;
    const long long groups = (long long)((cols + kCols - 1) / kCols) * batches, at_once = 32 / lanes_per_row(cols) * kWarps;
    long long s = (148 * (gated ? 4 : 8) + groups - 1) / groups;     // blocks an SM: 8 for plain sums (4: 75600 x 13824 392 us, 8: 347)
    const long long most = (rows + at_once * 4 - 1) / (at_once * 4);   // at least four rows a lane
    s = s < most ? s : most;
    return (int)(s < 1 ? 1 : s);
}

}  // namespace

// Row splits, i.e. scratch of batches * splits * cols floats for the two entries below.
MM_API int mm_column_splits(int rows, int cols, int batches, int gated) { return splits_of(rows, cols, batches, gated != 0); }

// sums[c] (bf16) = sum over r of x[r, c], fp32 inside.  x: [rows, cols] bf16 with ldx elements between rows; cols and ldx multiples
// of 8, 16-byte aligned.  8192 x (3840 + 1280 + 6912 + 1280): see native.py.
MM_API int mm_column_sum(const void* x, void* sums, float* partial, int rows, int cols, long long ldx, cudaStream_t st) {
    if (cols % 8 || ldx % 8 || ((uintptr_t)x & 15)) return -1;
    if (rows < 1 || cols < 1) return -2;
    const int splits = splits_of(rows, cols, 1, false);
    column_sum_kernel<false><<<dim3((cols + kCols - 1) / kCols, splits), kWarps * 32, 0, st>>>((const bf16*)x, nullptr, nullptr, nullptr,
                                                                                                  partial, rows, cols, ldx);
    fold_splits_kernel<<<(cols + 31) / 32, dim3(32, 8), 0, st>>>(partial, (bf16*)sums, splits, cols);
    return (int)cudaGetLastError();
}

// Backward of x + gate[b] * y: dy = dout * gate[b], dgate[b, c] = sum over the rows of dout * y (fp32 inside).  dout, y, dy: dense
// [batches, rows, cols]; one pass over dout and y.  Nothing to sum over (rows == 0): zeros.
MM_API int mm_gated_residual_bwd(const void* dout, const void* y, const void* gate, void* dy, void* dgate, float* partial, int batches,
                                 int rows, int cols, cudaStream_t st) {
    if (cols % 8 || ((uintptr_t)dout | (uintptr_t)y | (uintptr_t)gate | (uintptr_t)dy | (uintptr_t)dgate) & 15) return -1;
    if (rows < 0 || cols < 0 || batches < 0) return -2;
    if (!batches || !cols) return 0;
    if (!rows) return (int)cudaMemsetAsync(dgate, 0, (size_t)batches * cols * sizeof(bf16), st);
    if (rows < kWarps) {
        const long long most = ((long long)batches * (cols / 8) + 255) / 256;
        gated_short_kernel<<<(int)(most < 148 * 32 ? most : 148 * 32), 256, 0, st>>>((const bf16*)dout, (const bf16*)y, (const bf16*)gate, (bf16*)dy,
                                                                                (bf16*)dgate, batches, rows, cols);
        return (int)cudaGetLastError();
    }
    const long long blocks = (long long)batches * ((cols + 31) / 32);
    if (blocks > 0x7fffffffLL) return -2;
    const int splits = splits_of(rows, cols, batches, true);
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
