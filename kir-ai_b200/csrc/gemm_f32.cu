// 32-bit matrix product C[M, N] = A[M, K] * W[N, K]^T for few rows of A (decode steps of the true 32-bit path).
//
// Up to 8 rows the product is a read of W: 4 bytes a weight against 2 M flops.  A block streams rows of W with 16-byte
// loads, every warp R rows over its share of K (the warps of a row group take adjacent 512-byte pieces), with the next
// pieces in flight while the present ones are multiplied; A comes from the cache, and R rows of W share each of its
// values.  Every value of W is multiplied with all M rows in registers by 32-bit FMAs; the M x R sums of a lane meet in a
// butterfly that halves what each lane still holds at every step, and the warps of a row group meet in shared memory, in
// order.  A row of C depends on K and on how many rows there are, not on the other rows' values.
// Bound by HBM.  Measured (inputs beyond L2): 19,456 x 2,560 at 1 / 4 rows 31 / 37 us (6.4 / 5.3 TB/s), 151,936 x 2,560
// 214 / 240 us (7.3 / 6.5 TB/s), 2,560 x 9,728 18.5 / 20.5 us, where the plain kernel (64 x 64 tiles, a k axis walked 16
// at a time with nothing in flight) took 513 us on average over the products of a step of 4 rows of such sizes.
#include "common.cuh"

namespace {

constexpr int ROWS_WARPS = 8;

// Adds every one of V values (a power of two up to 32) over the 32 lanes: at each step a lane hands half of what it holds to the lane `o` away
// and keeps the other half.  Afterwards lane l holds the total of value `first` (returned) in v[0].
template <int V>
__device__ __forceinline__ int butterfly_sums(float (&v)[V], int lane) {
    int first = 0, held = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (held > 1) {
            held >>= 1;
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                if (i >= held) break;
                const float give = upper ? v[i] : v[i + held];
                const float keep = upper ? v[i + held] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
            first += upper ? held : 0;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return first;
}

// M rows of A, R rows of W a warp, the K axis over WK warps.  K, the row strides and the pointers allow 16-byte loads
// (the launcher checks).
template <int M, int R, int WK>
__global__ void __launch_bounds__(ROWS_WARPS * 32)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int N, int K,
                     long lda, long ldc, int constant) {
    constexpr int GROUPS = ROWS_WARPS / WK;  // row groups of a block
    constexpr int SUMS = M * R <= 4 ? 4 : (M * R <= 8 ? 8 : (M * R <= 16 ? 16 : 32));  // M R and padding up to a power of two
    __shared__ float part_s[ROWS_WARPS][SUMS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slice = warp % WK, group = warp / WK;
    const int n0 = (blockIdx.x * GROUPS + group) * R;
    const int pieces = K >> 2;
    pdl_launch_dependents();

    const float4* w_row[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w_row[r] = reinterpret_cast<const float4*>(W + (size_t)min(n0 + r, N - 1) * K);
    float4 w[R];
    int at = slice * 32 + lane;
    if (!constant) pdl_wait();
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = at < pieces ? __ldcs(w_row[r] + at) : zero;
    pdl_wait();  // constant weights do not depend on the kernel before this one, A does

    float acc[SUMS];
#pragma unroll
    for (int i = 0; i < SUMS; ++i) acc[i] = 0.0f;
    const int steps = (pieces + 32 * WK - 1) / (32 * WK);
    for (int step = 0; step < steps; ++step, at += 32 * WK) {
        float4 next[R];
        const bool more = at + 32 * WK < pieces;
#pragma unroll
        for (int r = 0; r < R; ++r) next[r] = more ? __ldcs(w_row[r] + at + 32 * WK) : zero;
        if (at < pieces) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(A + (size_t)m * lda) + at);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float s = acc[m * R + r];
                    s = fmaf(a.x, w[r].x, s);
                    s = fmaf(a.y, w[r].y, s);
                    s = fmaf(a.z, w[r].z, s);
                    acc[m * R + r] = fmaf(a.w, w[r].w, s);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = next[r];
    }

    const int first = butterfly_sums<SUMS>(acc, lane);
    if (lane % (32 / SUMS) == 0) part_s[warp][first] = acc[0];  // (fewer than 32 sums: several lanes hold the same one)
    __syncthreads();
    for (int i = threadIdx.x; i < GROUPS * M * R; i += ROWS_WARPS * 32) {
        const int g = i / (M * R), m = (i / R) % M, r = i % R;
        const int n = (blockIdx.x * GROUPS + g) * R + r;
        if (n >= N) continue;
        float sum = 0.0f;
#pragma unroll
        for (int q = 0; q < WK; ++q) sum += part_s[g * WK + q][m * R + r];
        C[(size_t)m * ldc + n] = sum;
    }
}

template <int M>
int launch_rows(const float* A, const float* W, float* C, int N, int K, long lda, long ldc, int constant, cudaStream_t stream) {
    // Four rows of W a warp: eight took 4 to 40 % longer at every size tried (fewer blocks on a processor).  A K axis of
    // at most four pieces a lane is not cut.
    constexpr int R = 4;
    if (K <= 512) {
        const unsigned blocks = (unsigned)((N + ROWS_WARPS * R - 1) / (ROWS_WARPS * R));
        return launch_pdl(gemm_f32_rows_kernel<M, R, 1>, dim3(blocks), dim3(ROWS_WARPS * 32), 0, stream, 1u, A, W, C, N, K, lda, ldc, constant);
    }
    const unsigned blocks = (unsigned)((N + 2 * R - 1) / (2 * R));
    return launch_pdl(gemm_f32_rows_kernel<M, R, 4>, dim3(blocks), dim3(ROWS_WARPS * 32), 0, stream, 1u, A, W, C, N, K, lda, ldc, constant);
}

}  // namespace

// Up to 8 rows; K and the row stride of A multiples of 4, A and W on 16-byte boundaries.  constant: W is not written by the
// kernel ahead in the stream (weights of a loaded model), and is fetched before that has finished.
KIRAI_EXPORT int kirai_gemm_f32_rows(const void* A_, const void* W_, void* C_, int M, int N, int K, long lda, long ldc,
                                     int constant, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 8 || K <= 0) return KIRAI_ERR_BAD_SIZE;
    if (K % 4 != 0 || lda % 4 != 0 || (((uintptr_t)A_ | (uintptr_t)W_) & 15) != 0) return KIRAI_ERR_BAD_ALIGN;
    const float *A = (const float*)A_, *W = (const float*)W_;
    float* C = (float*)C_;
    switch (M) {
        case 1: return launch_rows<1>(A, W, C, N, K, lda, ldc, constant, stream);
        case 2: return launch_rows<2>(A, W, C, N, K, lda, ldc, constant, stream);
        case 3: return launch_rows<3>(A, W, C, N, K, lda, ldc, constant, stream);
        case 4: return launch_rows<4>(A, W, C, N, K, lda, ldc, constant, stream);
        case 5: return launch_rows<5>(A, W, C, N, K, lda, ldc, constant, stream);
        case 6: return launch_rows<6>(A, W, C, N, K, lda, ldc, constant, stream);
        case 7: return launch_rows<7>(A, W, C, N, K, lda, ldc, constant, stream);
        default: return launch_rows<8>(A, W, C, N, K, lda, ldc, constant, stream);
    }
}
