// Column sums of a matrix: the bias gradients of a layer's projections.
//
// torch forms grad_bias of a linear layer with its general reduction, which for the shapes of
// an encoder layer (43 008 rows of 96 to 256 bf16 columns) takes 58 us where reading the matrix
// takes 4: four of them were 230 of a layer's 840 us of forward + backward.  Here every CTA sums a
// stretch of rows with 16-byte loads, float32 accumulation in registers, and a second kernel adds
// the CTAs' sums: 6 to 9 us together.  No atomics: the result is the same on every run.
#include <algorithm>

#include "../../include/msda_b200.h"
#include "msda_common.cuh"

namespace msda_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 4;           // rows a thread has in flight (8: no difference)

// partial[blockIdx.y][column]: CTA (x, y) takes 32 lanes of VEC columns and the rows y, y + grid.y, ...
// of kThreads / 32 at a time
template <typename T, int VEC>
__global__ void __launch_bounds__(kThreads) column_partials_kernel(const T *__restrict__ x,
                                                                   float *__restrict__ partial,
                                                                   int64_t rows, int cols) {
    struct alignas(sizeof(T) * VEC) Vec {
        T v[VEC];
    };
    constexpr int kRows = kThreads / 32;
    __shared__ float sums[kRows][32 * VEC];
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int col = ((int)blockIdx.x * 32 + lane) * VEC;
    float acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
    if (col < cols) {
        const int64_t step = (int64_t)gridDim.y * kRows;
        int64_t r = (int64_t)blockIdx.y * kRows + row;
        for (; r + (kUnroll - 1) * step < rows; r += kUnroll * step) {
            Vec in[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                in[u] = *reinterpret_cast<const Vec *>(x + (r + u * step) * cols + col);
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
#pragma unroll
                for (int i = 0; i < VEC; ++i) acc[i] += VecTraits<T>::to_float(in[u].v[i]);
        }
        for (; r < rows; r += step) {
            const Vec in = *reinterpret_cast<const Vec *>(x + r * cols + col);
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc[i] += VecTraits<T>::to_float(in.v[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) sums[row][lane * VEC + i] = acc[i];
    __syncthreads();
    for (int k = threadIdx.x; k < 32 * VEC; k += kThreads) {
        const int c = (int)blockIdx.x * 32 * VEC + k;
        if (c >= cols) continue;
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < kRows; ++i) s += sums[i][k];
        partial[(int64_t)blockIdx.y * cols + c] = s;
    }
}

// Bound by latency: every thread has all its parts in flight (at most 296 over 32 rows of threads; 4.5 us
// -> 3.4 against 8 rows and five round trips), and the kernel is launched while the sums are formed.  Small
// matrices too: that launch costs the host no more than another (both sums, us a call, called in a row: 300 x 256
// 8.2 -> 5.6, 3 600 x 256 8.2 -> 6.1, 43 008 x 256 10.3 -> 8.2; host 6.5 .. 6.9 -> 5.5 .. 6.0).
constexpr int kFinishRows = 32;
template <typename T>
__global__ void __launch_bounds__(kFinishRows * 32) column_finish_kernel(const float *__restrict__ partial,
                                                                         T *__restrict__ out, int parts, int cols) {
    __shared__ float sums[kFinishRows][33];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int col = (int)blockIdx.x * 32 + lane;
    grid_dependency_wait();
    float s = 0.f;
    if (col < cols) {
        // (plain loads: what the kernel before wrote)
        for (int i = row; i < parts; i += kFinishRows * 10) {
            float v[10];
#pragma unroll
            for (int u = 0; u < 10; ++u)
                v[u] = i + u * kFinishRows < parts ? __ldcg(partial + (int64_t)(i + u * kFinishRows) * cols + col) : 0.f;
#pragma unroll
            for (int u = 0; u < 10; ++u) s += v[u];
        }
    }
    sums[row][lane] = s;
    __syncthreads();
    // column `row`, summed over the lanes
    s = sums[lane][row];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0 && (int)blockIdx.x * 32 + row < cols) out[(int)blockIdx.x * 32 + row] = VecTraits<T>::from_float(s);
}

// CTAs over the rows: two per SM over all column blocks, each with at least some rows to sum
int row_parts(int64_t rows, int column_blocks) {
    const int64_t wanted = std::max(1, 148 * 2 / column_blocks);
    return (int)std::max<int64_t>(1, std::min(wanted, rows / (kThreads / 32 * kUnroll)));
}

template <typename T, int VEC>
cudaError_t launch(const void *x, void *out, float *partial, int64_t rows, int cols, cudaStream_t stream) {
    const int blocks = (cols + 32 * VEC - 1) / (32 * VEC);
    const int parts = row_parts(rows, blocks);
    column_partials_kernel<T, VEC><<<dim3(blocks, parts), kThreads, 0, stream>>>(
        static_cast<const T *>(x), partial, rows, cols);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((cols + 31) / 32, 1, 1);
    cfg.blockDim = dim3(kFinishRows * 32, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, column_finish_kernel<T>, static_cast<const float *>(partial), static_cast<T *>(out),
                              parts, cols);
}

template <typename T>
cudaError_t launch_typed(const void *x, void *out, float *partial, int64_t rows, int cols, cudaStream_t stream) {
    // the widest load that every row of the matrix is aligned for
    constexpr int kWide = 16 / sizeof(T);
    const uintptr_t at = reinterpret_cast<uintptr_t>(x);
    if (cols % kWide == 0 && at % 16 == 0) return launch<T, kWide>(x, out, partial, rows, cols, stream);
    if (cols % 2 == 0 && at % (2 * sizeof(T)) == 0) return launch<T, 2>(x, out, partial, rows, cols, stream);
    return launch<T, 1>(x, out, partial, rows, cols, stream);
}

}  // namespace

}  // namespace msda_b200

extern "C" {

int64_t msda_b200_column_sums_scratch_bytes(int64_t rows, int64_t cols) {
    // (a column block is at least 32 columns wide)
    (void)rows;
    return 4 * cols * 148 * 2;
}

int msda_b200_column_sums(const void *x, void *out, void *scratch, int64_t rows, int64_t cols, int dtype,
                          void *stream) {
    using namespace msda_b200;
    if (rows < 0 || cols <= 0 || cols > 0x7fffffff / 2)
        return set_last_error(MSDA_B200_INVALID_ARGUMENT, "column_sums: sizes out of range");
    if (!x || !out || !scratch)
        return set_last_error(MSDA_B200_INVALID_ARGUMENT, "column_sums: null pointer argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *partial = static_cast<float *>(scratch);
    cudaError_t e;
    switch (dtype) {
        case MSDA_B200_F32: e = launch_typed<float>(x, out, partial, rows, (int)cols, s); break;
        case MSDA_B200_F16: e = launch_typed<__half>(x, out, partial, rows, (int)cols, s); break;
        case MSDA_B200_BF16: e = launch_typed<__nv_bfloat16>(x, out, partial, rows, (int)cols, s); break;
        default: return set_last_error(MSDA_B200_INVALID_ARGUMENT, "column_sums: dtype is not f32, f16 or bf16");
    }
    if (e != cudaSuccess) return set_last_error(MSDA_B200_CUDA_ERROR, cudaGetErrorString(e));
    count_launches(2, 0);
    return MSDA_B200_OK;
}

}  // extern "C"
