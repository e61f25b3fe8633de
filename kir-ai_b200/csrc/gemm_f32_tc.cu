// 32-bit matrix product C[M, N] = A[M, K] * W[N, K]^T for many rows of A on the fifth-generation tensor cores.
//
// A float has 24 significant bits and a bf16 eight: every float (from 2^-110 on) is the sum of three bf16 values exactly, the
// nearest one, the nearest to what is left, and the rest.  With both operands cut that way the product of two floats is the
// sum of nine products of bf16 values, which the tensor cores form exactly.  To nearest, a second cut is at most 2^-8 and a
// third 2^-17 of the value, of either sign: the three smallest products are at most 2^-24 of the whole together (0.87 x 2^-24 of
// 4 million pairs, 0 on average; cuts that drop bits leave out up to 7.8 x 2^-24, always of the product's sign).  They are
// left out and six are summed: lo hi, mid mid, hi lo, mid hi, hi mid, hi hi, in
// this order.  The tensor cores' own additions drop low bits instead of rounding, so they only sum over 32 values of K;
// every such block of partial sums is then added to the tile's sums in registers by ordinary 32-bit additions.  From 32 values
// of K on the result is nearer to the exact one than a chain of 32-bit FMAs, where no single product outweighs the others
// (measured: see the launcher).  A row of C depends on how the product was cut, and that on the number of rows.
//
// A CTA computes 128 columns of C (128 rows of W fill the MMA) for BN rows of A.  Three planes of A are made by a kernel
// of their own, once per product (A is small beside W), and come in by TMA as the K-major B operand.  W comes in as it
// is, 128 rows x 32 columns of floats at a time; eight warps, whose threads own a row each, cut it and put the planes into
// tensor memory, where the MMA takes its A operand from: neither memory nor shared memory ever holds the planes of W.
// Warp roles: 0-7 cut W and add up partial sums, 8 loads W, 9 loads A's planes, 10 issues the MMAs.  Planes and partial
// sums are both double: while the tensor cores multiply block i, the warps add up block i - 1 and cut block i + 1.
// Split along K: the CTAs of a cluster leave their sums in shared memory and each adds up and stores a share of the rows.
//
// Values that are not finite: the cuts of an infinity are not numbers, so a sum that is not finite is worked out again by
// its thread as the chain of FMAs that the plain kernel computes.
#include <algorithm>

#include "sm100.cuh"
#include "tensor_map.cuh"

using namespace sm100;

namespace {

constexpr int TILE_N = 128;   // rows of W
constexpr int BLOCK_K = 32;
constexpr int WORKERS = 8;
constexpr int THREADS = (WORKERS + 3) * 32;
constexpr int W_STAGE = TILE_N * BLOCK_K * 4;

// BN up to 64 (few rows: the reading of W is what takes the time): two CTAs on an SM, so that one loads and cuts while
// the other waits for its MMAs.  Else one CTA with as deep a ring as fits.
template <int BN>
struct Shape {
    static constexpr int a_stage = 3 * BN * BLOCK_K * 2;
    static constexpr int ctas = BN <= 64 ? 2 : 1;
    static constexpr int w_stages = BN <= 64 ? 4 : (BN <= 128 ? 5 : 4);
    static constexpr int a_stages = BN <= 64 ? 3 : (BN <= 128 ? 5 : 4);
    static constexpr int ring = w_stages * W_STAGE + a_stages * a_stage;
    static constexpr int total = ring + 256 + 1024;  // barriers, slack to align the base
    static constexpr int columns = BN <= 64 ? 256 : 512;
    static_assert(ring >= BN * TILE_N * 4, "the ring takes a tile's sums");
    static_assert(2 * BN + 2 * 48 <= columns, "tensor memory: two blocks of partial sums and of planes");
    static_assert(total * ctas <= 227 * 1024, "shared memory of an SM");
    static_assert(alone_with_all_columns(total), "a CTA with all of the tensor memory shares no SM with this one");
    static_assert(columns < 512 || total >= ALL_COLUMNS_SHARED, "all columns");
};

__device__ __forceinline__ void tmem_store_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// K-major tile with rows of 64 bytes (32 bf16) under the 64-byte swizzle: 8-row groups 512 bytes apart, layout type 4.
__device__ __forceinline__ uint64_t smem_desc_k_major_sw64(uint32_t addr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((addr & 0x3FFFF) >> 4);
    desc |= (uint64_t)1 << 16;
    desc |= (uint64_t)(512 >> 4) << 32;
    desc |= (uint64_t)1 << 46;
    desc |= (uint64_t)4 << 61;
    return desc;
}

// Two floats cut into three pairs of bf16 (the first in the lower half), each cut the nearest bf16 to what is left: the
// subtractions are exact, and what the second leaves has at most eight bits, so that the third takes all of it (above 2^-110:
// bits of a value below 2^-133 have no place in a bf16).
__device__ __forceinline__ void cut_pair(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto nearest = [](float a, float b) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&v);
    };
    hi = nearest(x, y);
    const float xr = x - __uint_as_float(hi << 16), yr = y - __uint_as_float(hi & 0xffff0000u);
    mid = nearest(xr, yr);
    lo = nearest(xr - __uint_as_float(mid << 16), yr - __uint_as_float(mid & 0xffff0000u));
}

// planes[3][M][pitch] of A[M, K]; K a multiple of 4, a thread four columns of a row.
__global__ void __launch_bounds__(256)
f32_planes_kernel(const float* __restrict__ A, bf16* __restrict__ planes, int M, int K, long lda, int pitch) {
    pdl_launch_dependents();
    pdl_wait();
    const int quads = K >> 2;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long)M * quads) return;
    const int m = (int)(i / quads), q = (int)(i - (long)m * quads);
    const float4 v = *reinterpret_cast<const float4*>(A + (size_t)m * lda + 4 * q);
    uint2 hi, mid, lo;
    cut_pair(v.x, v.y, hi.x, mid.x, lo.x);
    cut_pair(v.z, v.w, hi.y, mid.y, lo.y);
    bf16* to = planes + (size_t)m * pitch + 4 * q;
    const size_t plane = (size_t)M * pitch;
    *reinterpret_cast<uint2*>(to) = hi;
    *reinterpret_cast<uint2*>(to + plane) = mid;
    *reinterpret_cast<uint2*>(to + 2 * plane) = lo;
}

__device__ __noinline__ float chain_of_fmas(const float* a, const float* w, int K) {
    float sum = 0.0f;
    for (int k = 0; k < K; ++k) sum = fmaf(a[k], w[k], sum);
    return sum;
}

template <int BN>
__global__ void __launch_bounds__(THREADS, Shape<BN>::ctas)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A,
                   const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, long lda, long ldc, int blocks_per_split,
                   int constant, int* __restrict__ error_flag) {
    using S = Shape<BN>;
    constexpr int WS = S::w_stages, AS = S::a_stages, HALF = BN / 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t w_ring = smem_addr(smem), a_ring = w_ring + WS * W_STAGE;
    uint64_t* bars = (uint64_t*)(smem + S::ring);
    uint64_t *w_full = bars, *w_empty = w_full + WS, *a_full = w_empty + WS, *a_empty = a_full + AS;
    uint64_t *planes_full = a_empty + AS, *block_done = planes_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(block_done + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * TILE_N, m0 = blockIdx.y * BN;
    const int total_blocks = (K + BLOCK_K - 1) / BLOCK_K;
    const int first_block = blockIdx.z * blocks_per_split;
    const int blocks = max(0, min(total_blocks - first_block, blocks_per_split));
    const int splits = gridDim.z;

    if (threadIdx.x == 0) {
        tma_prefetch_descriptor(&map_w);
        tma_prefetch_descriptor(&map_a);
        for (int s = 0; s < WS; ++s) {
            mbar_init(smem_addr(&w_full[s]), 1);
            mbar_init(smem_addr(&w_empty[s]), WORKERS);
        }
        for (int s = 0; s < AS; ++s) {
            mbar_init(smem_addr(&a_full[s]), 1);
            mbar_init(smem_addr(&a_empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_addr(&planes_full[s]), WORKERS);
            mbar_init(smem_addr(&block_done[s]), 1);
        }
        mbar_fence_init();
    }
    if (warp == WORKERS + 2) {
        tmem_alloc(smem_addr(tmem_slot), S::columns);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();  // only now: a CTA of the next kernel that shares the SM must find its tensor memory after this one
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_planes = tmem + 2 * BN;  // [2][3][16 columns]
    bool ok = true;

    if (warp < WORKERS) {
        pdl_wait();  // C may still be read by the kernel before this one
        const int quadrant = warp & 3, half = warp >> 2;  // the warp's lanes of tensor memory; its half of a block's k and of the sums' columns
        const uint32_t lanes = (uint32_t)(quadrant * 32) << 16;
        const int row = quadrant * 32 + lane;
        float sum[HALF];
#pragma unroll
        for (int j = 0; j < HALF; ++j) sum[j] = 0.0f;

        auto add_block = [&](int i) {
            if (!mbar_wait_hot(smem_addr(&block_done[i & 1]), (uint32_t)(i >> 1) & 1u)) { ok = false; return; }
            tc_fence_after();
            const uint32_t from = tmem + lanes + (uint32_t)((i & 1) * BN + half * HALF);
            if constexpr (HALF % 32 == 0) {
#pragma unroll
                for (int c = 0; c < HALF; c += 32) {
                    uint32_t r[32];
                    tmem_load_32x32(from + (uint32_t)c, r);
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[c + j] += __uint_as_float(r[j]);
                }
            } else {
                uint32_t r[16];
                tmem_load_32x16(from, r);
                tmem_load_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[j] += __uint_as_float(r[j]);
            }
            tc_fence_before();
        };

        for (int i = 0; i < blocks && ok; ++i) {
            const int s = i % WS;
            if (!mbar_wait_hot(smem_addr(&w_full[s]), (uint32_t)(i / WS) & 1u)) { ok = false; break; }
            const uint8_t* tile = smem + s * W_STAGE + row * 128;
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const float4*>(tile + (((half * 4 + j) ^ (row & 7)) << 4));
            uint32_t hi[8], mid[8], lo[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                cut_pair(v[j].x, v[j].y, hi[2 * j], mid[2 * j], lo[2 * j]);
                cut_pair(v[j].z, v[j].w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&w_empty[s]));
            // (block i - 2, whose planes these replace, was added up one turn ago: its MMAs are done)
            const uint32_t to = tmem_planes + lanes + (uint32_t)((i & 1) * 48 + half * 8);
            tmem_store_32x8(to, hi);
            tmem_store_32x8(to + 16, mid);
            tmem_store_32x8(to + 32, lo);
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&planes_full[i & 1]));
            if (i > 0) add_block(i - 1);
        }
        if (blocks > 0 && ok) add_block(blocks - 1);

        const int n = n0 + row;
        if (splits == 1) {
            if (n < N) {
#pragma unroll
                for (int j = 0; j < HALF; ++j) {
                    const int m = m0 + half * HALF + j;
                    if (m >= M) continue;
                    float value = sum[j];
                    if (!isfinite(value)) value = chain_of_fmas(A + (size_t)m * lda, W + (size_t)n * K, K);
                    C[(size_t)m * ldc + n] = value;
                }
            }
        } else {
            // (every load has been consumed and every MMA is done: the ring is free; [BN][128], lanes side by side)
            float* mine = reinterpret_cast<float*>(smem);
#pragma unroll
            for (int j = 0; j < HALF; ++j) mine[(half * HALF + j) * TILE_N + row] = sum[j];
        }
    } else if (warp == WORKERS) {
        if (elect_one()) {
            if (!constant) pdl_wait();  // constant weights do not depend on the kernel before this one, nor on the one before that
            int i = 0;
            for (; i < blocks; ++i) {
                const int s = i % WS;
                if (!mbar_wait(smem_addr(&w_empty[s]), ((uint32_t)(i / WS) & 1u) ^ 1u)) { ok = false; break; }
                mbar_expect_tx(smem_addr(&w_full[s]), W_STAGE);
                tma_load_2d(w_ring + s * W_STAGE, &map_w, smem_addr(&w_full[s]), (first_block + i) * BLOCK_K, n0);
            }
            for (int j = max(0, i - WS); j < i; ++j) ok &= mbar_wait(smem_addr(&w_full[j % WS]), (uint32_t)(j / WS) & 1u);  // none in flight at the end
        }
    } else if (warp == WORKERS + 1) {
        if (elect_one()) {
            pdl_wait();
            int i = 0;
            for (; i < blocks; ++i) {
                const int s = i % AS;
                if (!mbar_wait(smem_addr(&a_empty[s]), ((uint32_t)(i / AS) & 1u) ^ 1u)) { ok = false; break; }
                mbar_expect_tx(smem_addr(&a_full[s]), S::a_stage);
#pragma unroll
                for (int p = 0; p < 3; ++p)  // (rows beyond M are another plane's or zero: they end in columns that are not stored)
                    tma_load_2d(a_ring + s * S::a_stage + p * (BN * BLOCK_K * 2), &map_a, smem_addr(&a_full[s]), (first_block + i) * BLOCK_K, p * M + m0);
            }
            for (int j = max(0, i - AS); j < i; ++j) ok &= mbar_wait(smem_addr(&a_full[j % AS]), (uint32_t)(j / AS) & 1u);
        }
    } else {
        if (elect_one()) {
            constexpr uint32_t idesc = instr_desc_bf16(TILE_N, BN);
            int i = 0;
            for (; i < blocks; ++i) {
                const int s = i % AS;
                if (!mbar_wait_hot(smem_addr(&a_full[s]), (uint32_t)(i / AS) & 1u) ||
                    !mbar_wait_hot(smem_addr(&planes_full[i & 1]), (uint32_t)(i >> 1) & 1u)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_addr = a_ring + s * S::a_stage;
                const uint32_t planes = tmem_planes + (uint32_t)((i & 1) * 48), into = tmem + (uint32_t)((i & 1) * BN);
                // (plane of W, plane of A), the smallest products first
                constexpr int of_w[6] = {2, 1, 0, 1, 0, 0}, of_a[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
                for (int t = 0; t < 6; ++t) {
                    const uint64_t desc = smem_desc_k_major_sw64(a_addr + of_a[t] * (BN * BLOCK_K * 2));
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        mma_bf16_ts(into, planes + (uint32_t)(of_w[t] * 16 + k * 8), desc + (uint64_t)(2 * k), idesc, (t > 0 || k > 0) ? 1u : 0u);
                }
                mma_commit(smem_addr(&a_empty[s]));
                mma_commit(smem_addr(&block_done[i & 1]));
            }
            if (i > 0) ok &= mbar_wait(smem_addr(&block_done[(i - 1) & 1]), (uint32_t)((i - 1) >> 1) & 1u);  // none in flight at the end
        }
    }
    __syncwarp();
    if (splits > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        // this CTA's share of the tile's rows of A: 128 columns of C each, the CTAs' sums added in rank order
        const int share = (BN + splits - 1) / splits, from = blockIdx.z * share, to = min(BN, from + share);
        if (warp < WORKERS) {
            const int row = threadIdx.x & (TILE_N - 1), n = n0 + row;
            for (int j = from + (int)(threadIdx.x >> 7); j < to; j += 2) {
                const int m = m0 + j;
                if (m >= M) break;
                float value = 0.0f;
                for (int q = 0; q < splits; ++q) {
                    uint32_t remote;
                    float part;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(smem) + (uint32_t)((j * TILE_N + row) * 4)), "r"(q));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(remote) : "memory");
                    value += part;
                }
                if (n < N) {
                    if (!isfinite(value)) value = chain_of_fmas(A + (size_t)m * lda, W + (size_t)n * K, K);
                    C[(size_t)m * ldc + n] = value;
                }
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (!ok) atomicExch(error_flag, KIRAI_FLAG_WAIT_RAN_OUT);
    tc_fence_before();
    __syncthreads();
    if (warp == WORKERS + 2) {
        tc_fence_after();
        tmem_dealloc(tmem, S::columns);
    }
}

template <int BN>
int launch_tc(const float* A, const float* W, const bf16* planes, float* C, int M, int N, int K, long lda, long ldc, int pitch, int splits,
              int constant, int* error_flag, cudaStream_t stream) {
    using S = Shape<BN>;
    CUtensorMap map_w, map_a;
    if (!tmap::matrix_boxes<0>(&map_w, W, (uint64_t)N, (uint64_t)K, (uint64_t)K, TILE_N)) return KIRAI_ERR_BAD_ALIGN;
    if (!tmap::matrix_boxes<1>(&map_a, planes, (uint64_t)3 * M, (uint64_t)K, (uint64_t)pitch, BN)) return KIRAI_ERR_BAD_ALIGN;
    auto kernel = gemm_f32_tc_kernel<BN>;
    const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::total);
    if (set != cudaSuccess) return (int)set;
    const int blocks = (K + BLOCK_K - 1) / BLOCK_K;
    const dim3 grid((unsigned)((N + TILE_N - 1) / TILE_N), (unsigned)((M + BN - 1) / BN), (unsigned)splits);
    return launch_pdl(kernel, grid, dim3(THREADS), (size_t)S::total, stream, (unsigned)splits, map_w, map_a, A, W, C, M, N, K, lda, ldc,
                      (blocks + splits - 1) / splits, constant, error_flag);
}

}  // namespace

// How a product is cut into CTAs: the tile's rows of A and the split of K that the times below make the shortest.  A
// round of CTAs takes 8 us and, per 32 values of K, 0.66 us (32 rows, two CTAs on an SM or one), 0.58 or 0.90 us (64 rows,
// one or two), 0.70 us (128 rows) or 0.88 us (192 rows); fewer CTAs run at once where they come in clusters of 3, 4 or 8.
// A split has to save a twentieth.  (Of all cuts, swept over 4 weight sizes and 9 to 800 rows, this takes the fastest.)
// The times and the clusters that run at once are those of 148 SMs; with another number a round is as many CTAs as that holds.
static int sm_count() {
    static const int count = [] {
        int device = 0, value = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 148;
        return value;
    }();
    return count;
}
struct Cut {
    int bn, splits;
    float us;  // by the times above
};
static constexpr int cut_rows[4] = {32, 64, 128, 192};
static constexpr float cut_block_us[4] = {0.66f, 0.58f, 0.70f, 0.88f};
static Cut choose_cut(int M, int N, int K, int sms) {
    constexpr int cuts[5] = {1, 2, 3, 4, 8}, at_once[5] = {148, 148, 120, 132, 112};
    constexpr const int* bns = cut_rows;
    constexpr const float* block_us = cut_block_us;
    const int blocks = (K + BLOCK_K - 1) / BLOCK_K;
    const long columns = (N + TILE_N - 1) / TILE_N;
    Cut best{192, 1, 0.0f};
    float least = 0.0f;
    for (int b = 0; b < 4; ++b) {
        if (b > 0 && bns[b - 1] >= M) break;  // one tile already takes every row
        const long tiles = columns * ((M + bns[b] - 1) / bns[b]);
        if (tiles / columns > 65535) continue;
        for (int c = 0; c < 5; ++c) {
            const int s = cuts[c];
            if (s > 1 && blocks / s < 4) break;
            const long ctas = tiles * s, fit = std::max(1L, (long)at_once[c] * sms / 148), room = bns[b] <= 64 ? 2 * fit : fit;
            const long rounds = (ctas + room - 1) / room;
            const float us = bns[b] == 64 && ctas > 128 ? 0.90f : block_us[b];
            const float total = (float)rounds * (8.0f + us * (float)((blocks + s - 1) / s)) * (s > 1 ? 1.05f : 1.0f);
            if (least == 0.0f || total < least) {
                least = total;
                best = Cut{bns[b], s, total};
            }
        }
    }
    return best;
}

// Where a product's tiles fill a few rounds and a little of one more (456 CTAs of 192 rows on 148 SMs: four rounds, the last with
// 12), the columns of the whole rounds are one launch and the rest a second one with a cut of its own, finer along K, which
// starts as the first one's CTAs end.  How many columns (a multiple of TILE_N) the first launch takes and its rows a tile;
// 0 where one launch is as good to a twentieth.  A single launch of several rounds of 128 rows counts 0.63 us a block here (measured: 640 rows of 6,144 x
// 2,560 111 us, counted 128 by the time above, and 119 as two launches; of 19,456 x 2,560 360 us, counted 384, and 379 as two).
static int whole_rounds(int M, int N, int K, int sms, const Cut& single, int* bn) {
    const int blocks = (K + BLOCK_K - 1) / BLOCK_K;
    const long columns = (N + TILE_N - 1) / TILE_N;
    const bool counted_high = single.bn == 128 && single.splits == 1;
    float least = 0.95f * single.us * (counted_high ? (8.0f + 0.63f * (float)blocks) / (8.0f + cut_block_us[2] * (float)blocks) : 1.0f);
    int taken = 0;
    for (int b = 0; b < 4; ++b) {
        if (b > 0 && cut_rows[b - 1] >= M) break;
        const long row_tiles = (M + cut_rows[b] - 1) / cut_rows[b], room = cut_rows[b] <= 64 ? 2L * sms : sms;
        const long rounds = columns * row_tiles / room, first = rounds * room / row_tiles;
        if (rounds < 1 || first < 1 || first >= columns || row_tiles > 65535) continue;
        const float us = (cut_rows[b] == 64 ? 0.90f : cut_block_us[b]) * (float)blocks;
        const float total = (float)rounds * (8.0f + us) + choose_cut(M, (int)(N - first * TILE_N), K, sms).us;
        if (total < least) least = total, taken = (int)first * TILE_N, *bn = cut_rows[b];
    }
    return taken;
}
// The same for a device of `sms` SMs: the columns of the first launch (0: one launch takes them all), `rows` its rows a tile.
KIRAI_EXPORT int kirai_gemm_f32_tc_first_columns(int M, int N, int K, int sms, int* rows) {
    return whole_rounds(M, N, K, sms, choose_cut(M, N, K, sms), rows);
}

static int launch_cut(const Cut& cut, const float* A, const float* W, bf16* planes, float* C, int M, int N, int K, long lda, long ldc, int pitch,
                      int constant, int* error_flag, cudaStream_t stream) {
    switch (cut.bn) {
        case 32: return launch_tc<32>(A, W, planes, C, M, N, K, lda, ldc, pitch, cut.splits, constant, error_flag, stream);
        case 64: return launch_tc<64>(A, W, planes, C, M, N, K, lda, ldc, pitch, cut.splits, constant, error_flag, stream);
        case 128: return launch_tc<128>(A, W, planes, C, M, N, K, lda, ldc, pitch, cut.splits, constant, error_flag, stream);
        case 192: return launch_tc<192>(A, W, planes, C, M, N, K, lda, ldc, pitch, cut.splits, constant, error_flag, stream);
    }
    return KIRAI_ERR_BAD_SIZE;
}

// planes: 3 M pitch bf16 of scratch, pitch = K rounded up to a multiple of 8.  K and the row stride of A multiples of 4, A, W
// and planes on 16-byte boundaries.  bn 0: the cut is chosen here; else 32, 64, 128 or 192 rows of A to a tile and K over
// `splits` CTAs (1 to 8).  constant: W is not written by the kernel ahead in the stream (weights of a loaded model), and is fetched
// before that has finished.
// Measured at 515 rows of the 4B shape's products (6,144 x 2,560, 2,560 x 4,096, 19,456 x 2,560, 2,560 x 9,728): 81, 71,
// 298 and 147 us as one launch each (201, 152, 172 and 174 TFLOP/s of 32-bit arithmetic, six times that in the tensor cores; the third
// is two launches now, and six layers' products take 3.34 ms in place of 3.86), where the plain
// kernel took 5.3 ms together (20 TFLOP/s).  2-norm of the error over that of the result, in 2^-24, here and in the plain kernel:
// normal values 0.79 and 0.68 at K = 4, 0.80 and 1.24 at 16, 0.96 and 1.7 at 32, 1.7 and 15 at 2,560, 2.4 and 29 at 9,728; values of one
// sign 0.90 and 0.60, 1.0 and 1.06, 1.0 and 1.4, 1.3 and 13, 1.3 and 26.
KIRAI_EXPORT int kirai_gemm_f32_tc(const void* A_, const void* W_, void* planes_, void* C_, int M, int N, int K, long lda, long ldc,
                                   int bn, int splits, int constant, int* error_flag, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || (long)3 * M > 0x7fffffffL || splits < 0 || splits > 8) return KIRAI_ERR_BAD_SIZE;
    if (K % 4 != 0 || lda % 4 != 0 || (((uintptr_t)A_ | (uintptr_t)W_ | (uintptr_t)planes_) & 15) != 0) return KIRAI_ERR_BAD_ALIGN;
    const int sms = sm_count();
    const Cut cut = bn == 0 ? choose_cut(M, N, K, sms) : Cut{bn, splits > 0 ? splits : 1, 0.0f};
    int first_bn = 0;
    const int first = bn == 0 && splits == 0 ? whole_rounds(M, N, K, sms, cut, &first_bn) : 0;
    const int pitch = (K + 7) / 8 * 8;
    const long quads = (long)M * (K / 4);
    const long cut_blocks = (quads + 255) / 256;
    if (cut_blocks > 0x7fffffffL || (M + cut.bn - 1) / cut.bn > 65535) return KIRAI_ERR_BAD_SIZE;
    const float *A = (const float*)A_, *W = (const float*)W_;
    bf16* planes = (bf16*)planes_;
    const int status = launch_pdl(f32_planes_kernel, dim3((unsigned)cut_blocks), dim3(256), 0, stream, 1u, A, planes, M, K, lda, pitch);
    if (status != 0) return status;
    float* C = (float*)C_;
    if (first > 0) {
        const int done = launch_cut(Cut{first_bn, 1, 0.0f}, A, W, planes, C, M, first, K, lda, ldc, pitch, constant, error_flag, stream);
        if (done != 0) return done;
        return launch_cut(choose_cut(M, N - first, K, sms), A, W + (size_t)first * K, planes, C + first, M, N - first, K, lda, ldc, pitch, constant,
                          error_flag, stream);
    }
    return launch_cut(cut, A, W, planes, C, M, N, K, lda, ldc, pitch, constant, error_flag, stream);
}
