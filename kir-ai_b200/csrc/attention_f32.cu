// Causal grouped-query attention of the true 32-bit path over the paged cache, for heads of up to 128 columns in fours.
// Scores, softmax and weighted sums are 32-bit throughout, as in attention_plain.cu (which takes every other size); masks,
// soft caps and sinks are the ones of that file.  What differs is how the keys are read: there a block serves one (token,
// query head) and every warp of it walks a chain of load, sum over the warp, exponential; here a key row is read once for
// many query rows.
//
// Prompt kernel: a CTA takes 64 query rows of one kv head's group (64 / group tokens, all heads of the group) over tiles of 64
// keys.  256 threads hold 4 x 4 scores and 4 x (head columns / 16) results each (with 128 threads and 8 x 4 an SM had eight
// warps, too few to hide the barriers of a tile); the operands of four columns come from
// shared memory as 16-byte loads (12 wavefronts for 64 FMAs a lane, so that the FMA pipe and not shared memory sets the
// pace), and `fma.rn.f32x2` halves the instructions.  Bound by the FMA pipe: the 4B shape's layer (32 heads of 128, 8 kv
// heads) at 515 tokens is 2.2 GFLOP, 30 us at 72 TFLOP/s; measured 116 us inside a prompt (152 with four warps a CTA and the
// longest rows of the rest beside the longest; plain kernel: 1,139), the heaviest row tile's nine key tiles one after another setting
// the end.  Weights overlay the key tile, so that a CTA takes 101 KB and
// two fit an SM; the value tile is fetched while the scores are made, and a key tile's fetch hides behind the other CTA.
//
// Decode kernel (one token per request): a CTA takes a (request, kv head) and up to eight query heads of its group; each
// warp takes eight keys at a time (four for more than four heads), all their rows in flight together, a lane holding four
// columns.  The warp's sums for all (head, key) pairs are made by one transposing butterfly, 31 shuffles for 32 sums, after
// which a lane owns one score; weights go back by shuffles.  Bound by the latency of the loads (4 requests of about 106 tokens:
// 6.4 us a layer, plain kernel 23); long contexts are cut over
// a cluster of CTAs that merge through distributed shared memory, one CTA per 128 keys and at most eight, and as many as run
// at once: the order of a request's sums, and so its last bits, follow the number of requests and the longest of them.
#include "common.cuh"

#define AF_ROWS 64
#define AF_KEYS 64
#define AF_THREADS 256
#define AF_TY (AF_THREADS / 16)   // threads along the query rows (sixteen stand along the keys and the columns)
#define AF_R (AF_ROWS / AF_TY)    // query rows of a thread
#define AF_PSTRIDE (AF_KEYS + 4)

__device__ __forceinline__ void copy_16(float* dst, const float* src, bool present) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(present ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Where key `j` of kv head `kv_head` begins in the cache, or -1 without a page (the error word is then set).
__device__ __forceinline__ long key_row(const int* table, int j, int page_size, int table_width, int num_pages, int kv_heads,
                                        int kv_head, int head_dim, int* error_flag) {
    const int logical = j / page_size;
    const int page = logical < table_width ? table[logical] : -1;
    if (page < 0 || page >= num_pages) {
        atomicExch(error_flag, KIRAI_FLAG_NO_PAGE_READ);
        return -1;
    }
    return ((((long)page * 2) * kv_heads + kv_head) * page_size + (j - logical * page_size)) * (long)head_dim;
}

// ---------------------------------------------------------------------------------------------------- prompt portions
// The weighted sum of one tile.  EDGE: some row of the CTA does not see some key of the tile; such a key's value is then
// not multiplied at all (a weight of 0 would still make NaN of an infinite value that the row may not see).
template <int DP, bool EDGE>
__device__ __forceinline__ void weighted_sum(f32x2 (&o)[AF_R][DP / 32], const float* __restrict__ p_s, const float* __restrict__ v_s,
                                             const long* __restrict__ base_s, int key0, const int (&pos)[AF_R], int window, int keep,
                                             int ty, int tx) {
#pragma unroll 2
    for (int k = 0; k < AF_KEYS; k += 4) {
        float4 p[AF_R];
#pragma unroll
        for (int i = 0; i < AF_R; ++i) p[i] = *reinterpret_cast<const float4*>(p_s + (ty + AF_TY * i) * AF_PSTRIDE + k);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            f32x2 v[DP / 32];
#pragma unroll
            for (int c = 0; c < DP / 64; ++c) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(v_s + (k + u) * DP + 64 * c + 4 * tx);
                v[2 * c] = w.x, v[2 * c + 1] = w.y;
            }
            const int j = key0 + k + u;
            const bool present = EDGE ? base_s[k + u] >= 0 : true;
#pragma unroll
            for (int i = 0; i < AF_R; ++i) {
                if (EDGE && !(present && j <= pos[i] && (j >= first_visible_key(pos[i], window) || j < keep))) continue;
                const float w = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                const f32x2 ww = pair(w, w);
#pragma unroll
                for (int c = 0; c < DP / 32; ++c) fma2(o[i][c], ww, v[c]);
            }
        }
    }
}

template <int DP>
__global__ void __launch_bounds__(AF_THREADS, 2)
attention_f32_prefill_kernel(const float* __restrict__ q, const float* __restrict__ cache, float* __restrict__ out,
                             const int* __restrict__ block_table, const int* __restrict__ query_start,
                             const int* __restrict__ context_len, int q_heads, int kv_heads, int head_dim, long q_row_stride,
                             int page_size, int table_width, int num_pages, int mask, float scale, float softcap,
                             const float* __restrict__ sinks, int first_tiles, int* __restrict__ error_flag) {
    extern __shared__ float4 smem4[];
    float* q_s = reinterpret_cast<float*>(smem4);        // [AF_ROWS][DP + 4]
    float* k_s = q_s + AF_ROWS * (DP + 4);               // [AF_KEYS][DP + 4], then the weights [AF_ROWS][AF_PSTRIDE]
    float* p_s = k_s;
    float* v_s = k_s + (DP >= 64 ? AF_KEYS * (DP + 4) : 0);  // [AF_KEYS][DP]
    __shared__ long base_s[2][AF_KEYS];                  // where the tile's key rows begin (-1: not to be read)

    pdl_launch_dependents();
    pdl_wait();
    const int request = blockIdx.z, kv_head = blockIdx.x;
    const int group = q_heads / kv_heads;
    const int tokens_per_tile = AF_ROWS / group;
    const int row0 = query_start[request], run = query_start[request + 1] - row0;
    const int row_tiles = (run + tokens_per_tile - 1) / tokens_per_tile;
    // the longest rows of keys are handed out first; where all CTAs start at once, two to an SM (`first_tiles` > 0), the second
    // ones, from row tile `first_tiles` of the order on, come shortest first, so that an SM's two add up alike
    const int place = blockIdx.y;
    const int row_tile = first_tiles > 0 && row_tiles == (int)gridDim.y && place >= first_tiles ? place - first_tiles : row_tiles - 1 - place;
    if (row_tile < 0) return;
    const int token0 = row_tile * tokens_per_tile;
    const int first_pos = context_len[request] - run;
    const int last_pos = first_pos + min(token0 + tokens_per_tile, run) - 1;
    const int window = mask_window(mask), keep = mask_keep(mask);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int* table = block_table + (long)request * table_width;
    const int columns4 = head_dim >> 2;

    int pos[AF_R];
#pragma unroll
    for (int i = 0; i < AF_R; ++i) pos[i] = min(first_pos + token0 + (ty + AF_TY * i) / group, last_pos);
    const int tile_first_pos = first_pos + token0;
    const int lo_first = first_visible_key(tile_first_pos, window);
    const int lo_last = first_visible_key(last_pos, window);
    const TileRuns runs = tile_runs(lo_first, keep, AF_KEYS);
    const int last_tile = last_pos / AF_KEYS;
    const int tiles = runs.kept + last_tile - runs.first + 1;

    auto find_rows = [&](int it) {
        if (tid < AF_KEYS) {
            const int j = runs.tile(it) * AF_KEYS + tid;
            long base = -1;
            if (j <= last_pos && (j >= lo_first || j < keep))
                base = key_row(table, j, page_size, table_width, num_pages, kv_heads, kv_head, head_dim, error_flag);
            base_s[it & 1][tid] = base;
        }
    };
    auto fetch = [&](float* dst, int stride, long offset, int it) {
        for (int n = tid; n < AF_KEYS * (DP / 4); n += AF_THREADS) {
            const int key = n / (DP / 4), c = n % (DP / 4);
            if (c >= columns4) continue;
            const long base = base_s[it & 1][key];
            copy_16(dst + key * stride + 4 * c, cache + (base < 0 ? 0 : base + offset + 4 * c), base >= 0);
        }
    };
    const long v_offset = (long)kv_heads * page_size * head_dim;

    for (int n = tid; n < AF_ROWS * (DP / 4); n += AF_THREADS) {
        const int r = n / (DP / 4), c = n % (DP / 4), token = token0 + r / group;
        if (c >= columns4) continue;
        const bool present = r < tokens_per_tile * group && token < run;
        const float* src = q + (present ? (size_t)(row0 + token) * q_row_stride + (size_t)(kv_head * group + r % group) * head_dim + 4 * c : 0);
        copy_16(q_s + r * (DP + 4) + 4 * c, src, present);
    }
    find_rows(0);
    __syncthreads();
    fetch(k_s, DP + 4, 0, 0);
    copy_commit();

    f32x2 o[AF_R][DP / 32];
    float m[AF_R], l[AF_R];
#pragma unroll
    for (int i = 0; i < AF_R; ++i) {
        m[i] = -INFINITY, l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < DP / 32; ++c) o[i][c] = 0ull;
    }

    for (int it = 0; it < tiles; ++it) {
        const int key0 = runs.tile(it) * AF_KEYS;
        const long* base = base_s[it & 1];
        copy_wait<0>();
        // (also the barrier behind the tile before it: its values may be overwritten)
        const bool lost = __syncthreads_or(tid < AF_KEYS && base[tid] < 0);
        const bool edge = lost || key0 + AF_KEYS - 1 > tile_first_pos || (key0 < lo_last && key0 + AF_KEYS > keep);
        fetch(v_s, DP, v_offset, it);
        copy_commit();
        if (it + 1 < tiles) find_rows(it + 1);

        f32x2 s2[AF_R][4];
#pragma unroll
        for (int i = 0; i < AF_R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 2
        for (int c = 0; c < head_dim; c += 4) {
            ulonglong2 a[AF_R], b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(k_s + (tx + 16 * j) * (DP + 4) + c);
#pragma unroll
            for (int i = 0; i < AF_R; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(q_s + (ty + AF_TY * i) * (DP + 4) + c);
#pragma unroll
            for (int i = 0; i < AF_R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fma2(s2[i][j], a[i].x, b[j].x);
                    fma2(s2[i][j], a[i].y, b[j].y);
                }
        }
        __syncthreads();  // the keys have been read: the weights take their place
#pragma unroll
        for (int i = 0; i < AF_R; ++i) {
            float s[4];
            bool seen[4];
            float top = m[i];
            const int lo = first_visible_key(pos[i], window);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float even, odd;
                unpair(s2[i][j], even, odd);
                s[j] = (even + odd) * scale;
                if (softcap > 0.0f) s[j] = softcap * tanhf(s[j] / softcap);
                const int key = key0 + tx + 16 * j;
                seen[j] = !edge || (base[tx + 16 * j] >= 0 && key <= pos[i] && (key >= lo || key < keep));
                if (seen[j]) top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int offset = 8; offset > 0; offset >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
            const float corr = m[i] == -INFINITY ? 0.0f : expf(m[i] - top);
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float w = seen[j] ? expf(s[j] - top) : 0.0f;
                sum += w;
                p_s[(ty + AF_TY * i) * AF_PSTRIDE + tx + 16 * j] = w;
            }
            l[i] = l[i] * corr + sum;  // this thread's keys only; the sixteen threads of a row meet at the end
            m[i] = top;
            const f32x2 cc = pair(corr, corr);
#pragma unroll
            for (int c = 0; c < DP / 32; ++c) o[i][c] = mul2(o[i][c], cc);
        }
        copy_wait<0>();
        __syncthreads();
        if (edge) weighted_sum<DP, true>(o, p_s, v_s, base, key0, pos, window, keep, ty, tx);
        else weighted_sum<DP, false>(o, p_s, v_s, base, key0, pos, window, keep, ty, tx);
        if (it + 1 < tiles) {
            __syncthreads();  // the weights have been read: the next keys take their place
            fetch(k_s, DP + 4, 0, it + 1);
            copy_commit();
        }
    }
#pragma unroll
    for (int i = 0; i < AF_R; ++i) {
        float sum = l[i];
#pragma unroll
        for (int offset = 8; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
        const int r = ty + AF_TY * i, token = token0 + r / group;
        if (r >= tokens_per_tile * group || token >= run) continue;
        const int head = kv_head * group + r % group;
        float* row = out + ((size_t)(row0 + token) * q_heads + head) * head_dim;
        const float inverse = sinks ? softmax_inverse(m[i] * 1.4426950408889634f, sum, sinks, head) : 0.0f;
#pragma unroll
        for (int c = 0; c < DP / 64; ++c) {
            float4 v;
            unpair(o[i][2 * c], v.x, v.y);
            unpair(o[i][2 * c + 1], v.z, v.w);
            if (sinks) v.x *= inverse, v.y *= inverse, v.z *= inverse, v.w *= inverse;
            else if (sum > 0.0f) v.x /= sum, v.y /= sum, v.z /= sum, v.w /= sum;
            else v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (64 * c + 4 * tx < head_dim) *reinterpret_cast<float4*>(row + 64 * c + 4 * tx) = v;
        }
    }
}

// --------------------------------------------------------------------------------------------- one token per request
#define AD_WARPS 8
#define AD_MAX_CLUSTER 8

// Sums `v[i]` over the warp for all COUNT values (a power of two up to 32) at once: afterwards lane L holds the sum of
// value L / (32 / COUNT).
template <int COUNT>
__device__ __forceinline__ float transposed_sum(float (&v)[COUNT]) {
    const int lane = threadIdx.x & 31;
    int offset = 16;
#pragma unroll
    for (int half = COUNT / 2; half > 0; half /= 2) {
        const bool upper = lane & offset;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float mine = upper ? v[i + half] : v[i], other = upper ? v[i] : v[i + half];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, other, offset);
        }
        offset >>= 1;
    }
    float sum = v[0];
    for (; offset > 0; offset >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, offset);
    return sum;
}

__device__ __forceinline__ float peer_value(const float* local, uint32_t rank) {
    uint32_t remote;
    float value;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(value) : "r"(remote) : "memory");
    return value;
}
__device__ __forceinline__ void meet_cluster() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// G: query heads of this CTA (the group's, rounded up to a power of two; at most eight), KEYS: keys a warp takes at a time.
template <int G, int KEYS>
__global__ void __launch_bounds__(AD_WARPS * 32)
attention_f32_decode_kernel(const float* __restrict__ q, const float* __restrict__ cache, float* __restrict__ out,
                            const int* __restrict__ block_table, const int* __restrict__ context_len, int q_heads, int kv_heads,
                            int head_dim, long q_row_stride, int page_size, int table_width, int num_pages, int mask, float scale,
                            float softcap, const float* __restrict__ sinks, int cluster, int* __restrict__ error_flag) {
    constexpr int PAIRS = G * KEYS, SPREAD = 32 / PAIRS;  // SPREAD lanes hold the same (head, key) pair
    __shared__ float o_s[AD_WARPS][G][128];
    __shared__ float m_s[AD_WARPS][G], l_s[AD_WARPS][G];
    __shared__ float o_c[G][128], m_c[G], l_c[G];  // this CTA's result, for the cluster

    pdl_launch_dependents();
    pdl_wait();
    const int request = blockIdx.z, rank = blockIdx.x;
    const int group = q_heads / kv_heads, chunks = (group + G - 1) / G;
    const int kv_head = blockIdx.y / chunks, head0 = kv_head * group + (blockIdx.y % chunks) * G;
    const int heads = min(G, (kv_head + 1) * group - head0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pos = context_len[request] - 1;
    const int* table = block_table + (long)request * table_width;
    const int window = mask_window(mask), keep = mask_keep(mask);
    const int lo = first_visible_key(pos, window);
    const int kept = min(keep, lo);  // kept first keys that the window no longer covers
    const int visible = kept + pos - lo + 1;
    const int begin = (int)((long)visible * rank / cluster), end = (int)((long)visible * (rank + 1) / cluster);
    const bool mine = 4 * lane < head_dim;
    const long v_offset = (long)kv_heads * page_size * head_dim;

    float4 query[G];
#pragma unroll
    for (int h = 0; h < G; ++h)
        query[h] = mine && h < heads ? *reinterpret_cast<const float4*>(q + (size_t)request * q_row_stride + (size_t)(head0 + h) * head_dim + 4 * lane)
                                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 o[G];
#pragma unroll
    for (int h = 0; h < G; ++h) o[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float m = -INFINITY, l = 0.0f;  // of this lane's head; `l` of this lane's keys only
    const int my_key = (lane / SPREAD) % KEYS;

    for (int at = begin + warp * KEYS; at < end; at += AD_WARPS * KEYS) {
        long base = -1;
        if (lane < KEYS && at + lane < end) {
            const int j = at + lane < kept ? at + lane : lo + at + lane - kept;
            base = key_row(table, j, page_size, table_width, num_pages, kv_heads, kv_head, head_dim, error_flag);
        }
        float4 k[KEYS], v[KEYS];
#pragma unroll
        for (int n = 0; n < KEYS; ++n) {
            const long b = __shfl_sync(0xffffffffu, base, n);
            k[n] = v[n] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (b >= 0 && mine) {
                k[n] = *reinterpret_cast<const float4*>(cache + b + 4 * lane);
                v[n] = *reinterpret_cast<const float4*>(cache + b + v_offset + 4 * lane);
            }
        }
        float dots[PAIRS];
#pragma unroll
        for (int h = 0; h < G; ++h)
#pragma unroll
            for (int n = 0; n < KEYS; ++n)
                dots[h * KEYS + n] = fmaf(query[h].x, k[n].x, fmaf(query[h].y, k[n].y, fmaf(query[h].z, k[n].z, query[h].w * k[n].w)));
        float score = transposed_sum<PAIRS>(dots) * scale;
        if (softcap > 0.0f) score = softcap * tanhf(score / softcap);
        const bool seen = __shfl_sync(0xffffffffu, base, my_key) >= 0;
        float top = seen ? fmaxf(m, score) : m;
#pragma unroll
        for (int offset = SPREAD; offset < SPREAD * KEYS; offset <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
        const float corr = m == -INFINITY ? 0.0f : expf(m - top);
        const float weight = seen ? expf(score - top) : 0.0f;
        l = l * corr + weight;
        m = top;
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float c = __shfl_sync(0xffffffffu, corr, h * KEYS * SPREAD);
            o[h].x *= c, o[h].y *= c, o[h].z *= c, o[h].w *= c;
#pragma unroll
            for (int n = 0; n < KEYS; ++n) {
                const float w = __shfl_sync(0xffffffffu, weight, (h * KEYS + n) * SPREAD);
                o[h].x = fmaf(w, v[n].x, o[h].x), o[h].y = fmaf(w, v[n].y, o[h].y);
                o[h].z = fmaf(w, v[n].z, o[h].z), o[h].w = fmaf(w, v[n].w, o[h].w);
            }
        }
    }
#pragma unroll
    for (int offset = SPREAD; offset < SPREAD * KEYS; offset <<= 1) l += __shfl_xor_sync(0xffffffffu, l, offset);
    if (lane % (KEYS * SPREAD) == 0) m_s[warp][lane / (KEYS * SPREAD)] = m, l_s[warp][lane / (KEYS * SPREAD)] = l;
#pragma unroll
    for (int h = 0; h < G; ++h) *reinterpret_cast<float4*>(&o_s[warp][h][4 * lane]) = o[h];
    __syncthreads();
    // the warps' results added up: a thread takes one column of every (256 / 128)-th head
    for (int n = threadIdx.x; n < G * 128; n += AD_WARPS * 32) {
        const int h = n >> 7, column = n & 127;
        float top = -INFINITY, sum = 0.0f, acc = 0.0f;
#pragma unroll
        for (int w = 0; w < AD_WARPS; ++w) top = fmaxf(top, m_s[w][h]);
#pragma unroll
        for (int w = 0; w < AD_WARPS; ++w) {
            const float weight = m_s[w][h] == -INFINITY ? 0.0f : expf(m_s[w][h] - top);
            sum += l_s[w][h] * weight;
            acc += o_s[w][h][column] * weight;
        }
        o_c[h][column] = acc;
        if (column == 0) m_c[h] = top, l_c[h] = sum;
    }
    if (cluster > 1) meet_cluster();
    else __syncthreads();
    // every CTA of the cluster stores a share of the columns
    for (int n = rank * AD_WARPS * 32 + threadIdx.x; n < heads * 128; n += cluster * AD_WARPS * 32) {
        const int h = n >> 7, column = n & 127;
        if (column >= head_dim) continue;
        float top = m_c[h], sum = l_c[h], acc = o_c[h][column];
        if (cluster > 1) {
            float tops[AD_MAX_CLUSTER];
            top = -INFINITY;
            for (int c = 0; c < cluster; ++c) top = fmaxf(top, tops[c] = peer_value(&m_c[h], c));
            sum = acc = 0.0f;
            for (int c = 0; c < cluster; ++c) {
                const float part = peer_value(&l_c[h], c);
                const float weight = tops[c] == -INFINITY ? 0.0f : expf(tops[c] - top);
                sum += part * weight;
                acc += peer_value(&o_c[h][column], c) * weight;
            }
        }
        const float inverse = sinks ? softmax_inverse(top * 1.4426950408889634f, sum, sinks, head0 + h) : 0.0f;
        out[((size_t)request * q_heads + head0 + h) * head_dim + column] = sinks ? acc * inverse : sum > 0.0f ? acc / sum : 0.0f;
    }
    if (cluster > 1) meet_cluster();  // nobody leaves while its result may still be read
}

static int attention_f32_refusal(const void* q, const void* cache, const void* out, int q_heads, int kv_heads, int head_dim,
                                 long q_row_stride, int page_size) {
    if (kv_heads <= 0 || q_heads <= 0 || q_heads % kv_heads != 0 || q_heads / kv_heads > AF_ROWS || page_size <= 0) return KIRAI_ERR_BAD_SIZE;
    if (head_dim <= 0 || head_dim > 128 || head_dim % 4 != 0) return KIRAI_ERR_BAD_SIZE;
    if (q_row_stride % 4 != 0 || ((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) % 16 != 0) return KIRAI_ERR_BAD_ALIGN;
    return 0;
}

template <int DP>
static int attention_f32_prefill_launch(dim3 grid, cudaStream_t stream, const float* q, const float* cache, float* out,
                                        const int* block_table, const int* query_start, const int* context_len, int q_heads,
                                        int kv_heads, int head_dim, long q_row_stride, int page_size, int table_width,
                                        int num_pages, int mask, float scale, float softcap, const float* sinks, int* error_flag) {
    const size_t smem = (size_t)(AF_ROWS * (DP + 4) + AF_KEYS * (DP + 4) + AF_KEYS * DP) * sizeof(float);
    const cudaError_t err = cudaFuncSetAttribute(attention_f32_prefill_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    static const int sms = [] {
        int device = 0, value = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
        return value;
    }();
    const long ctas = (long)grid.x * grid.y;
    const int first_tiles = grid.z == 1 && ctas > sms && ctas <= 2L * sms ? sms / (int)grid.x : 0;
    return launch_pdl(attention_f32_prefill_kernel<DP>, grid, dim3(AF_THREADS), smem, stream, 1u, q, cache, out, block_table,
                      query_start, context_len, q_heads, kv_heads, head_dim, q_row_stride, page_size, table_width, num_pages,
                      mask, scale, softcap, sinks, first_tiles, error_flag);
}

// Runs of new tokens: query_start [requests + 1] rows of q and out, context_len [requests] tokens in the cache after the step.
KIRAI_EXPORT int kirai_attention_f32_prefill(const float* q, const float* cache, float* out, const int* block_table,
                                             const int* query_start, const int* context_len, int requests, int max_query_len,
                                             int q_heads, int kv_heads, int head_dim, long q_row_stride, int page_size,
                                             int table_width, int num_pages, int mask, float scale, float softcap,
                                             const float* sinks, int* error_flag, cudaStream_t stream) {
    if (requests <= 0 || max_query_len <= 0) return 0;
    const int refusal = attention_f32_refusal(q, cache, out, q_heads, kv_heads, head_dim, q_row_stride, page_size);
    if (refusal) return refusal;
    const int tokens_per_tile = AF_ROWS / (q_heads / kv_heads);
    const int row_tiles = (max_query_len + tokens_per_tile - 1) / tokens_per_tile;
    if (row_tiles > 65535 || requests > 65535) return KIRAI_ERR_BAD_SIZE;
    const dim3 grid(kv_heads, row_tiles, requests);
    if (head_dim <= 64)
        return attention_f32_prefill_launch<64>(grid, stream, q, cache, out, block_table, query_start, context_len, q_heads, kv_heads, head_dim,
                                                q_row_stride, page_size, table_width, num_pages, mask, scale, softcap, sinks, error_flag);
    return attention_f32_prefill_launch<128>(grid, stream, q, cache, out, block_table, query_start, context_len, q_heads, kv_heads, head_dim,
                                             q_row_stride, page_size, table_width, num_pages, mask, scale, softcap, sinks, error_flag);
}

// One token per request.  `longest`: the most keys that a token may see, by which the launch is cut.
KIRAI_EXPORT int kirai_attention_f32_decode(const float* q, const float* cache, float* out, const int* block_table,
                                            const int* context_len, int requests, int q_heads, int kv_heads, int head_dim,
                                            long q_row_stride, int page_size, int table_width, int num_pages, int mask, float scale,
                                            float softcap, const float* sinks, int longest, int sms, int* error_flag,
                                            cudaStream_t stream) {
    if (requests <= 0) return 0;
    const int refusal = attention_f32_refusal(q, cache, out, q_heads, kv_heads, head_dim, q_row_stride, page_size);
    if (refusal) return refusal;
    const int group = q_heads / kv_heads;
    const int G = group <= 1 ? 1 : group <= 2 ? 2 : group <= 4 ? 4 : 8;
    const long blocks = (long)kv_heads * ((group + G - 1) / G);
    if (blocks > 65535 || requests > 65535) return KIRAI_ERR_BAD_SIZE;
    // a CTA more for every 128 keys (two rounds of the CTA's warps), as long as all CTAs run at once, two to an SM
    int cluster = 1;
    while (cluster < AD_MAX_CLUSTER && longest > 128 * cluster && blocks * requests * cluster * 2 <= 2L * sms) cluster *= 2;
    const dim3 grid(cluster, (unsigned)blocks, requests);
    auto launch = [&](auto kernel) {
        return launch_pdl_clusters(kernel, grid, dim3(AD_WARPS * 32), 0, stream, dim3(cluster, 1, 1), q, cache, out, block_table, context_len,
                                   q_heads, kv_heads, head_dim, q_row_stride, page_size, table_width, num_pages, mask, scale, softcap,
                                   sinks, cluster, error_flag);
    };
    if (G == 1) return launch(attention_f32_decode_kernel<1, 8>);
    if (G == 2) return launch(attention_f32_decode_kernel<2, 8>);
    if (G == 4) return launch(attention_f32_decode_kernel<4, 8>);
    return launch(attention_f32_decode_kernel<8, 4>);
}
