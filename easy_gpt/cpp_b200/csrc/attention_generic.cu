// Attention over the paged cache, for any mix of prompt portions and decoded
// tokens: a CTA per (token, KV head), or per eight of the query heads that share it.
//
// The token at absolute position p of its request sees the keys at positions
// first..p of that request, first = 0 or p - window + 1 with a sliding window.
// Keys are found through the request's row of the block table:
//   page = table[seq, pos / page_size], offset = pos % page_size.
// Query head h reads KV head h / (num_heads / num_kv_heads)
// (src/cuda/ops/self_attn_detail.cuh:667-669).
//
// score = (q . k) * scale (scaled after the dot product like the reference,
// src/models/self_attn.cpp:251-253), then a running softmax in float32 over
// chunks of 32 keys (one key per lane): m, l, acc as in
// src/cuda/ops/self_attn_detail.cuh:325-382, with expf, not the fast
// approximation.  Warp w takes the chunks w, w + warps, ... from `first` on, and
// the warps' results are merged in their order: the order of the sums depends only
// on the token's own position, the window and the head size, not on how the request
// was cut into steps, on the batch, or on the page ids.
//
// What bounds it is latency: a decode step has a handful of CTAs.  So a chunk's keys
// come to shared memory in one batch of coalesced loads and serve all query heads
// of the group, values are loaded for eight keys at a time, and a token's chunks
// run on eight warps at once.  (Measured on B200, 4 tokens at 100 keys, 14 heads of
// 64 on 2 KV heads, float32: a warp per (token, head), its lanes each walking a key's
// row, took 76 us; this takes 17.)
//
// This is the kernel of the 32-bit path and the fallback of the bfloat16 path
// for sizes the tensor-core kernels refuse.
#include "common.cuh"

namespace {
constexpr int MAX_DIMS_PER_LANE = 8;      // head_dim <= 256
constexpr int MAX_HEADS = 8;              // query heads of a CTA

// a chunk's rows of keys are this far apart (floats): 16-byte loads by lanes of eight rows meet no bank twice
__host__ __device__ constexpr int row_floats(int head_dim) { return (head_dim + 3) / 4 * 4 + 4; }
constexpr int warps_for(int head_dim) { return head_dim <= 64 ? 8 : 4; }
// of a warp: the chunk's keys, the weights [heads][32] and where its 32 rows start
__host__ __device__ constexpr int warp_floats(int head_dim) { return 32 * row_floats(head_dim) + MAX_HEADS * 32 + 64; }
}  // namespace

// HG: query heads a CTA has room for; DPL: dimensions a lane accumulates (head_dim <= 32 * DPL); VEC: rows come in pieces of four
template <typename T, int HG, int DPL, bool VEC>
__global__ void __launch_bounds__(256)
attention_generic_kernel(const T* __restrict__ q, int ldq, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                         const int* __restrict__ block_table, int table_stride, const int* __restrict__ token_seq,
                         const int* __restrict__ positions, T* __restrict__ out, int ldo, int num_heads, int num_kv_heads,
                         int head_dim, int page_size, long long page_stride, long long head_stride, int num_pages,
                         int window, float scale, int* status) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int t = blockIdx.x, kvh = blockIdx.y, group = num_heads / num_kv_heads;
    const int h0 = kvh * group + blockIdx.z * HG, heads = min(HG, group - (int)blockIdx.z * HG);
    const int pos = positions[t], row = row_floats(head_dim), quads = row / 4 - 1;
    const int rows_on = 32 / quads, quads_on = 32 % quads;        // from a lane's piece of the keys to its next
    const int* table = block_table + (size_t)token_seq[t] * table_stride;
    float* qs = smem;                                             // [HG][row], behind them a region per warp
    float* keys = smem + HG * row + warp * warp_floats(head_dim);
    float* weights = keys + 32 * row;
    long long* starts = reinterpret_cast<long long*>(weights + MAX_HEADS * 32);
    for (int e = threadIdx.x; e < HG * row; e += blockDim.x) {
        const int h = e / row, d = e % row;
        qs[e] = h < heads && d < head_dim ? to_f32<T>(q[(size_t)t * ldq + (h0 + h) * head_dim + d]) : 0.f;
    }
    __syncthreads();

    const int first = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    float m[HG], l[HG], acc[HG][DPL];
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[h][i] = 0.f;
    }

    for (int base = first + warp * 32; base <= pos; base += warps * 32) {
        const int kpos = base + lane;
        long long row_off = -1;
        if (kpos <= pos) {
            const int page = table[kpos / page_size];
            if (page < 0 || page >= num_pages) {
                atomicOr(status, EG_STATUS_BAD_PAGE);
            } else {
                row_off = (long long)page * page_stride + kvh * head_stride + (long long)(kpos % page_size) * head_dim;
            }
        }
        __syncwarp();                                             // the chunk in front has been read
        starts[lane] = row_off;
        __syncwarp();
        // the keys, as float32; rows that cannot be read and what pads a row are zeros
        if (VEC) {
#pragma unroll 8
            for (int e = lane, j = lane / quads, c = lane % quads; e < 32 * quads; e += 32, j += rows_on, c += quads_on) {
                if (c >= quads) { c -= quads; ++j; }
                const long long at = starts[j];
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (at >= 0) {
                    if (sizeof(T) == 4) {
                        v = *reinterpret_cast<const float4*>(k_cache + at + c * 4);
                    } else {
                        const uint2 raw = *reinterpret_cast<const uint2*>(k_cache + at + c * 4);
                        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
                        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
                        v = make_float4(lo.x, lo.y, hi.x, hi.y);
                    }
                }
                *reinterpret_cast<float4*>(keys + j * row + c * 4) = v;
            }
        } else {
            for (int j = 0; j < 32; ++j) {
                const long long at = starts[j];
                for (int d = lane; d < quads * 4; d += 32) keys[j * row + d] = at >= 0 && d < head_dim ? to_f32<T>(k_cache[at + d]) : 0.f;
            }
        }
        __syncwarp();
        float s[HG];
#pragma unroll
        for (int h = 0; h < HG; ++h) s[h] = 0.f;
#pragma unroll 4
        for (int c = 0; c < quads; ++c) {
            const float4 k = *reinterpret_cast<const float4*>(keys + lane * row + c * 4);
#pragma unroll
            for (int h = 0; h < HG; ++h) {
                const float4 x = *reinterpret_cast<const float4*>(qs + h * row + c * 4);
                s[h] = fmaf(x.w, k.w, fmaf(x.z, k.z, fmaf(x.y, k.y, fmaf(x.x, k.x, s[h]))));
            }
        }
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            const float score = row_off >= 0 ? s[h] * scale : -INFINITY;
            const float m_new = fmaxf(m[h], warp_max(score));
            // (-inf: nothing readable so far, bad pages only)
            const float p = row_off >= 0 && m_new != -INFINITY ? expf(score - m_new) : 0.f;
            const float corr = m_new == -INFINITY ? 1.f : expf(m[h] - m_new);      // m = -inf -> 0
            l[h] = l[h] * corr + warp_sum(p);
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[h][i] *= corr;
            m[h] = m_new;
            weights[h * 32 + lane] = p;
        }
        __syncwarp();
        const int nkeys = min(32, pos - base + 1);
        for (int j0 = 0; j0 < nkeys; j0 += 8) {
            float v[8][DPL];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const long long at = starts[j0 + j];
#pragma unroll
                for (int i = 0; i < DPL; ++i) {
                    const int d = lane + 32 * i;
                    v[j][i] = at >= 0 && d < head_dim ? to_f32<T>(v_cache[at + d]) : 0.f;
                }
            }
#pragma unroll
            for (int h = 0; h < HG; ++h) {
                const float4 p0 = *reinterpret_cast<const float4*>(weights + h * 32 + j0), p1 = *reinterpret_cast<const float4*>(weights + h * 32 + j0 + 4);
                const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int i = 0; i < DPL; ++i) acc[h][i] = fmaf(p[j], v[j][i], acc[h][i]);
            }
        }
    }

    // ---- the warps' results, merged in their order: [warp][head][32 * DPL] sums, then m and l
    __syncthreads();                                              // queries and keys are dead
    float* sums = smem;
    float* ml = smem + warps * HG * 32 * DPL;                     // [warp][head][2]
#pragma unroll
    for (int h = 0; h < HG; ++h) {
#pragma unroll
        for (int i = 0; i < DPL; ++i) sums[((warp * HG + h) * DPL + i) * 32 + lane] = acc[h][i];
        if (lane == 0) {
            ml[(warp * HG + h) * 2] = m[h];
            ml[(warp * HG + h) * 2 + 1] = l[h];
        }
    }
    __syncthreads();
    const int used = min(warps, (pos - first) / 32 + 1);
    for (int e = threadIdx.x; e < heads * 32 * DPL; e += blockDim.x) {
        const int h = e / (32 * DPL), d = e % (32 * DPL);
        if (d >= head_dim) continue;
        float top = -INFINITY;
        for (int w = 0; w < used; ++w) top = fmaxf(top, ml[(w * HG + h) * 2]);
        float sum = 0.f, total = 0.f;
        if (top > -INFINITY)
            for (int w = 0; w < used; ++w) {
                const float f = expf(ml[(w * HG + h) * 2] - top);
                total = fmaf(ml[(w * HG + h) * 2 + 1], f, total);
                sum = fmaf(sums[(w * HG + h) * 32 * DPL + d], f, sum);
            }
        out[(size_t)t * ldo + (h0 + h) * head_dim + d] = from_f32<T>(total > 0.0f ? sum * (1.0f / total) : 0.f);
    }
}

namespace {
template <typename T, int HG, int DPL, bool VEC>
int launch_generic(cudaStream_t stream, const T* q, int ldq, const T* k, const T* v, const int* table, int table_stride, const int* token_seq, const int* positions,
                   T* out, int ldo, int tokens, int num_heads, int num_kv_heads, int head_dim, int page_size, long long page_stride, long long head_stride,
                   int num_pages, int window, float scale, int* status) {
    const int warps = warps_for(head_dim);
    const size_t walk = (size_t)HG * row_floats(head_dim) + (size_t)warps * warp_floats(head_dim), merge = (size_t)warps * HG * (32 * DPL + 2);
    const size_t bytes = (walk > merge ? walk : merge) * sizeof(float);
    auto kernel = attention_generic_kernel<T, HG, DPL, VEC>;
    static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (configured != cudaSuccess) return (int)configured;
    const dim3 grid(tokens, num_kv_heads, (num_heads / num_kv_heads + HG - 1) / HG);
    kernel<<<grid, warps * 32, bytes, stream>>>(q, ldq, k, v, table, table_stride, token_seq, positions, out, ldo, num_heads, num_kv_heads, head_dim, page_size,
                                                page_stride, head_stride, num_pages, window, scale, status);
    return eg_launch_status();
}

template <typename T, class... Args>
int launch_for(bool vec, int group, int head_dim, Args... args) {
#define EG_GENERIC(HG, DPL) return vec ? launch_generic<T, HG, DPL, true>(args...) : launch_generic<T, HG, DPL, false>(args...)
    if (group == 1) {
        if (head_dim <= 64) EG_GENERIC(1, 2);
        if (head_dim <= 128) EG_GENERIC(1, 4);
        EG_GENERIC(1, 8);
    }
    if (group <= 4) {
        if (head_dim <= 64) EG_GENERIC(4, 2);
        if (head_dim <= 128) EG_GENERIC(4, 4);
        EG_GENERIC(4, 8);
    }
    if (head_dim <= 64) EG_GENERIC(8, 2);
    if (head_dim <= 128) EG_GENERIC(8, 4);
    EG_GENERIC(4, 8);
#undef EG_GENERIC
}
}  // namespace

// Returns cudaErrorInvalidValue for sizes this kernel does not take.
EG_API int eg_attention_generic(cudaStream_t stream, int dtype, const void* q, int ldq, const void* k_cache,
                                const void* v_cache, const int* block_table, int table_stride, const int* token_seq,
                                const int* positions, void* out, int ldo, int tokens, int num_heads, int num_kv_heads,
                                int head_dim, int page_size, long long page_stride, long long head_stride, int num_pages,
                                int window, float scale, int* status) {
    if (tokens <= 0) return 0;
    if (head_dim > 32 * MAX_DIMS_PER_LANE || head_dim <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads)
        return (int)cudaErrorInvalidValue;
    if (num_kv_heads > 65535) return (int)cudaErrorInvalidValue;
    const int group = num_heads / num_kv_heads, piece = dtype == EG_BF16 ? 8 : 16;          // bytes of four values
    const bool vec = head_dim % 4 == 0 && page_stride % 4 == 0 && head_stride % 4 == 0 && (uintptr_t)k_cache % piece == 0;
    if (dtype == EG_BF16)
        return launch_for<bf16>(vec, group, head_dim, stream, (const bf16*)q, ldq, (const bf16*)k_cache, (const bf16*)v_cache, block_table, table_stride, token_seq,
                                positions, (bf16*)out, ldo, tokens, num_heads, num_kv_heads, head_dim, page_size, page_stride, head_stride, num_pages, window, scale,
                                status);
    return launch_for<float>(vec, group, head_dim, stream, (const float*)q, ldq, (const float*)k_cache, (const float*)v_cache, block_table, table_stride, token_seq,
                             positions, (float*)out, ldo, tokens, num_heads, num_kv_heads, head_dim, page_size, page_stride, head_stride, num_pages, window, scale,
                             status);
}
