// True float32 matrix product for the 32-bit path:  C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
// FFMA on the CUDA cores: no tensor cores, no TF32.  (The reference's Linear is the same contraction with float32
// accumulation, src/ops.cpp:79-121.)
//
// The order of a sum depends on N and K alone, never on M, i.e. never on how tokens were batched: K is cut into
// groups of PARTS parts of `part_len` terms (f32_cut below); a part is one thread's chain of fused multiply-adds over
// ascending k, a group is the sum of its parts in their order, an element the sum of its groups in their order.  Both
// kernels compute exactly that:
//
//   f32_rows_kernel   up to 32 tokens: bound by the stream of the weights.  A CTA has 64 rows of W and one group of K,
//                     a warp one part, a lane two rows; a warp copies its rows ahead in pieces of 32 terms (asynchronous
//                     copies, two stages, two CTAs an SM: about 64 KB on their way per SM) and the parts meet in shared
//                     memory, the groups (a cluster of up to 8 CTAs) through distributed shared memory.
//   f32_tile_kernel   more tokens: tiles of 64 or 128 tokens by 128 rows, 8 rows a thread, packed pairs of tokens
//                     (fma.rn.f32x2 rounds like two fmaf).  Where the tiles alone do not fill the SMs the groups of K
//                     are a cluster here too.
//
// Measured on B200 (weights not in the L2), against one 64 x 64 tile kernel for every size, whose few CTAs walked K alone:
//     4 tokens    [896 x 4864] 518 -> 10.4 us    [9728 x 896] 122 -> 12.7 us    [151936 x 896] 786 -> 94 us (5.8 TB/s)
//   300 tokens    [896 x 4864] 457 -> 121 us     [9728 x 896] 291 -> 162 us     [1152 x 896] 85 -> 32 us
// and the error of the 0.5B logits against 64 bits fell from 3.4e-6 to 1.1e-6 (shorter chains).
#include <cooperative_groups.h>

#include "common.cuh"

namespace {
namespace cg = cooperative_groups;

constexpr int PARTS = 4;             // parts of a group
constexpr int MAX_GROUPS = 8;        // the portable cluster size
constexpr int ROWS = 64;             // rows of W a CTA of the streaming kernel has
constexpr int ROWS_MAX_TOKENS = 32;
constexpr int CHUNK = 32;            // terms a warp copies at once
constexpr int W_STRIDE = CHUNK + 4;  // eight rows' 16-byte pieces fall into different banks
constexpr int BN = 128, BK = 16;

struct Cut {
    int groups, part_len;
};
// As many groups as give every SM a CTA of the streaming kernel, at least 128 terms each; a constant number of SMs, so
// that results do not hang off the GPU.  Parts are whole pieces of 32 terms.
Cut f32_cut(int N, int K) {
    const long long tiles = (N + ROWS - 1) / ROWS;
    int groups = 1;
    while (groups < MAX_GROUPS && tiles * groups < 148 && K > 128 * groups) groups *= 2;
    int part_len = (K + PARTS * groups - 1) / (PARTS * groups);
    part_len = (part_len + CHUNK - 1) / CHUNK * CHUNK;
    if (part_len == 0) part_len = CHUNK;
    groups = (K + PARTS * part_len - 1) / (PARTS * part_len);
    return {groups < 1 ? 1 : groups, part_len};
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint32_t shared_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// copies `valid` of 16 (of 4) bytes and fills the rest with zeros; with valid 0 the source is not read
__device__ __forceinline__ void copy16(void* to, const void* from, int valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(shared_at(to)), "l"(from), "r"(valid) : "memory");
}
__device__ __forceinline__ void copy4(void* to, const void* from, int valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(shared_at(to)), "l"(from), "r"(valid) : "memory");
}
}  // namespace

// Shared memory of a warp: two stages of [64 rows][W_STRIDE] weights and [CHUNK][BM] inputs.  The parts' sums
// [PARTS][ROWS * BM] take the same room behind the last piece, the group's sums [ROWS * BM] lie behind it.
template <int BM> struct RowsMemory {
    static constexpr int STAGE = ROWS * W_STRIDE + CHUNK * BM;      // floats
    static constexpr int BYTES = (PARTS * 2 * STAGE + ROWS * BM) * 4;
};

template <int BM, bool VEC>
__global__ void __launch_bounds__(PARTS * 32)
f32_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias, float* __restrict__ C, int ldc,
                int M, int N, int K, int part_len, int groups) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = blockIdx.x % groups, n0 = blockIdx.x / groups * ROWS;
    const int first = min(K, (group * PARTS + warp) * part_len), last = min(K, first + part_len);
    float* stages = smem + warp * 2 * RowsMemory<BM>::STAGE;
    const int chunks = (last - first + CHUNK - 1) / CHUNK;

    auto stage = [&](int c) {
        float* ws = stages + (c & 1) * RowsMemory<BM>::STAGE;
        float* xs = ws + ROWS * W_STRIDE;
        const int k0 = first + c * CHUNK;
        if (VEC) {
#pragma unroll
            for (int i = 0; i < ROWS / 4; ++i) {
                const int row = i * 4 + lane / 8, k = k0 + lane % 8 * 4;
                const bool in = n0 + row < N && k < last;
                copy16(ws + row * W_STRIDE + lane % 8 * 4, in ? W + (size_t)(n0 + row) * ldw + k : W, in ? min(16, (last - k) * 4) : 0);
            }
        } else {
            for (int row = 0; row < ROWS; ++row) {
                const bool in = n0 + row < N && k0 + lane < last;
                copy4(ws + row * W_STRIDE + lane, in ? W + (size_t)(n0 + row) * ldw + k0 + lane : W, in ? 4 : 0);
            }
        }
#pragma unroll
        for (int m = 0; m < BM; ++m) {
            const bool in = m < M && k0 + lane < last;
            copy4(xs + lane * BM + m, in ? A + (size_t)m * lda + k0 + lane : A, in ? 4 : 0);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    f32x2 acc[2][BM / 2];
#pragma unroll
    for (int m = 0; m < BM / 2; ++m) acc[0][m] = acc[1][m] = 0ull;
    if (chunks > 0) stage(0);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            stage(c + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncwarp();
        const float* ws = stages + (c & 1) * RowsMemory<BM>::STAGE;
        const float* xs = ws + ROWS * W_STRIDE;
#pragma unroll 2
        for (int k = 0; k < CHUNK; k += 4) {
            const float4 wa = *reinterpret_cast<const float4*>(ws + lane * W_STRIDE + k);
            const float4 wb = *reinterpret_cast<const float4*>(ws + (lane + 32) * W_STRIDE + k);
            const float a4[4] = {wa.x, wa.y, wa.z, wa.w}, b4[4] = {wb.x, wb.y, wb.z, wb.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const f32x2 a = pack2(a4[j], a4[j]), b = pack2(b4[j], b4[j]);
#pragma unroll
                for (int m = 0; m < BM / 4; ++m) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xs + (k + j) * BM + m * 4);
                    acc[0][2 * m] = fma2(x.x, a, acc[0][2 * m]);
                    acc[0][2 * m + 1] = fma2(x.y, a, acc[0][2 * m + 1]);
                    acc[1][2 * m] = fma2(x.x, b, acc[1][2 * m]);
                    acc[1][2 * m + 1] = fma2(x.y, b, acc[1][2 * m + 1]);
                }
            }
        }
        __syncwarp();                 // the stage may be overwritten
    }

    // the parts meet: [part][token][row]
    __syncthreads();
    float* parts = smem;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int m = 0; m < BM / 2; ++m) {
            float lo, hi;
            unpack2(acc[r][m], lo, hi);
            parts[(warp * BM + 2 * m) * ROWS + r * 32 + lane] = lo;
            parts[(warp * BM + 2 * m + 1) * ROWS + r * 32 + lane] = hi;
        }
    __syncthreads();
    float* sums = smem + PARTS * 2 * RowsMemory<BM>::STAGE;
    auto store = [&](int e, float v) {
        const int m = e / ROWS, n = n0 + e % ROWS;
        if (m >= M || n >= N) return;
        if (bias) v += bias[n];
        C[(size_t)m * ldc + n] = v;
    };
    for (int e = threadIdx.x; e < ROWS * BM; e += PARTS * 32) {
        float v = parts[e];
#pragma unroll
        for (int w = 1; w < PARTS; ++w) v += parts[w * BM * ROWS + e];
        if (groups == 1)
            store(e, v);
        else
            sums[e] = v;
    }
    if (groups == 1) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = group * PARTS * 32 + threadIdx.x; e < ROWS * BM; e += groups * PARTS * 32) {
        float part[MAX_GROUPS];
#pragma unroll
        for (int g = 0; g < MAX_GROUPS; ++g)
            if (g < groups) part[g] = *cluster.map_shared_rank(sums + e, g);
        float v = part[0];
#pragma unroll
        for (int g = 1; g < MAX_GROUPS; ++g)
            if (g < groups) v += part[g];
        store(e, v);
    }
    cluster.sync();                   // nobody leaves while another reads its sums
}

// Thread (tx, ty) has tokens ty * 8 .. + 8 and rows tx * 4 .. + 4 and 64 + tx * 4 .. + 4 of a tile: what bounds the kernel are
// the loads from shared memory, and 64 results a thread take four of them for 32 packed products (with 32 results a thread,
// three for 16, 350 tokens of the 0.5B sizes took 118 us a product in the mean, this 100; pairs of rows against inputs
// stored twice, four loads for 16 products, 141).
template <int BM, bool VEC>
__global__ void __launch_bounds__(BM * 2)
f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias, float* __restrict__ C, int ldc,
                int M, int N, int K, int part_len, int groups, int split) {
    constexpr int THREADS = BM * 2, PASS = THREADS / 4, TM = 8, A_STRIDE = BM + 4, N_STRIDE = BN + 4;
    constexpr int A_LOADS = BM / PASS, W_LOADS = BN / PASS;
    extern __shared__ __align__(16) float smem[];
    float* As = smem;                                  // [2][BK][A_STRIDE]
    float* Ws = smem + 2 * BK * A_STRIDE;              // [2][BK][N_STRIDE]
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int ctas = split ? groups : 1;
    const int my_group = blockIdx.x % ctas, n0 = blockIdx.x / ctas * BN, m0 = blockIdx.y * BM;

    float4 a_next[A_LOADS], w_next[W_LOADS];
    auto fetch = [&](int k0) {
        auto piece = [&](const float* base, int ld, int row, int rows, int k) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row >= rows || k >= K) return v;
            const float* p = base + (size_t)row * ld + k;
            if (VEC) return *reinterpret_cast<const float4*>(p);           // K is a multiple of 4 then
            v.x = p[0];
            if (k + 1 < K) v.y = p[1];
            if (k + 2 < K) v.z = p[2];
            if (k + 3 < K) v.w = p[3];
            return v;
        };
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) a_next[i] = piece(A, lda, m0 + i * PASS + tid / 4, M, k0 + tid % 4 * 4);
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) w_next[i] = piece(W, ldw, n0 + i * PASS + tid / 4, N, k0 + tid % 4 * 4);
    };
    auto put = [&](int buffer) {
        float* as = As + buffer * BK * A_STRIDE + tid % 4 * 4 * A_STRIDE + tid / 4;
        float* ws = Ws + buffer * BK * N_STRIDE + tid % 4 * 4 * N_STRIDE + tid / 4;
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            as[i * PASS] = a_next[i].x;
            as[A_STRIDE + i * PASS] = a_next[i].y;
            as[2 * A_STRIDE + i * PASS] = a_next[i].z;
            as[3 * A_STRIDE + i * PASS] = a_next[i].w;
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            ws[i * PASS] = w_next[i].x;
            ws[N_STRIDE + i * PASS] = w_next[i].y;
            ws[2 * N_STRIDE + i * PASS] = w_next[i].z;
            ws[3 * N_STRIDE + i * PASS] = w_next[i].w;
        }
    };

    f32x2 acc[TM / 2][8], sum[TM / 2][8];
    for (int g = split ? my_group : 0; g < (split ? my_group + 1 : groups); ++g) {
        const int k_first = g * PARTS * part_len, k_last = min(K, k_first + PARTS * part_len);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = sum[i][j] = 0ull;
        __syncthreads();                               // the group in front has been read
        fetch(k_first);
        put(0);
        __syncthreads();
        int buffer = 0, left = part_len;
        for (int k0 = k_first; k0 < k_last; k0 += BK) {
            const bool more = k0 + BK < k_last;
            if (more) fetch(k0 + BK);
            const float* as = As + buffer * BK * A_STRIDE + ty * TM;
            const float* ws = Ws + buffer * BK * N_STRIDE + tx * 4;
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                f32x2 a[TM / 2];
#pragma unroll
                for (int i = 0; i < TM / 4; ++i) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(as + k * A_STRIDE + i * 4);
                    a[2 * i] = v.x;
                    a[2 * i + 1] = v.y;
                }
                const float4 w0 = *reinterpret_cast<const float4*>(ws + k * N_STRIDE), w1 = *reinterpret_cast<const float4*>(ws + k * N_STRIDE + 64);
                const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const f32x2 b = pack2(w[j], w[j]);
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i) acc[i][j] = fma2(a[i], b, acc[i][j]);
                }
            }
            left -= BK;
            if (left == 0 || !more) {                  // a part is complete
#pragma unroll
                for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        sum[i][j] = k0 + BK - k_first <= part_len ? acc[i][j] : add2(sum[i][j], acc[i][j]);
                        acc[i][j] = 0ull;
                    }
                left = part_len;
            }
            if (more) {
                buffer ^= 1;
                put(buffer);
                __syncthreads();
            }
        }
        if (split) break;
        // the groups' sums meet in C itself: every element has one thread
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + ty * TM + i;
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + (j / 4) * 64 + tx * 4 + j % 4;
                if (n >= N) continue;
                float lo, hi;
                unpack2(sum[i / 2][j], lo, hi);
                float v = i % 2 ? hi : lo;
                float* c = C + (size_t)m * ldc + n;
                if (g > 0) v = *c + v;
                if (g == groups - 1 && bias) v += bias[n];
                *c = v;
            }
        }
    }
    if (!split) return;

    __syncthreads();
    float* sums = smem;                                // [BM][BN]
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float lo, hi;
            unpack2(sum[i][j], lo, hi);
            const int n = (j / 4) * 64 + tx * 4 + j % 4;
            sums[(ty * TM + 2 * i) * BN + n] = lo;
            sums[(ty * TM + 2 * i + 1) * BN + n] = hi;
        }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int e = my_group * THREADS + tid; e < BM * BN; e += groups * THREADS) {
        const int m = m0 + e / BN, n = n0 + e % BN;
        if (m >= M || n >= N) continue;
        float part[MAX_GROUPS];
#pragma unroll
        for (int g = 0; g < MAX_GROUPS; ++g)
            if (g < groups) part[g] = *cluster.map_shared_rank(sums + e, g);
        float v = part[0];
#pragma unroll
        for (int g = 1; g < MAX_GROUPS; ++g)
            if (g < groups) v += part[g];
        if (bias) v += bias[n];
        C[(size_t)m * ldc + n] = v;
    }
    cluster.sync();
}

namespace {
template <class Kernel, class... Args>
int launch_clusters(Kernel kernel, dim3 grid, int threads, int smem, int cluster, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kernel, args...);
    return e != cudaSuccess ? (int)e : eg_launch_status();
}

template <bool VEC>
int launch_f32(cudaStream_t stream, const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N, int K) {
    const Cut cut = f32_cut(N, K);
    if (M <= ROWS_MAX_TOKENS) {
        const dim3 grid((N + ROWS - 1) / ROWS * cut.groups);
#define EG_ROWS(BM)                                                                                                                                 \
    return launch_clusters(f32_rows_kernel<BM, VEC>, grid, PARTS * 32, RowsMemory<BM>::BYTES, cut.groups, stream, A, lda, W, ldw, bias, C, ldc, M, N, K, \
                           cut.part_len, cut.groups)
        if (M <= 4) EG_ROWS(4);
        if (M <= 8) EG_ROWS(8);
        if (M <= 16) EG_ROWS(16);
        EG_ROWS(32);
#undef EG_ROWS
    }
    // tiles of 128 tokens where they fill the SMs twice over; the groups of K side by side where those of 64 do not
    const long long columns = (N + BN - 1) / BN;
    if (columns * ((M + 127) / 128) >= 296) {
        constexpr int smem = 2 * BK * (128 + 4 + BN + 4) * 4;
        return launch_clusters(f32_tile_kernel<128, VEC>, dim3((unsigned)columns, (M + 127) / 128), 2 * 128, smem, 1, stream, A, lda, W, ldw, bias, C, ldc, M, N, K,
                               cut.part_len, cut.groups, 0);
    }
    const int split = cut.groups > 1 && columns * ((M + 63) / 64) < 296;
    constexpr int tile_bytes = 2 * BK * (64 + 4 + BN + 4) * 4, sums_bytes = 64 * BN * 4;
    return launch_clusters(f32_tile_kernel<64, VEC>, dim3((unsigned)columns * (split ? cut.groups : 1), (M + 63) / 64), 2 * 64,
                           tile_bytes > sums_bytes ? tile_bytes : sums_bytes, split ? cut.groups : 1, stream, A, lda, W, ldw, bias, C, ldc, M, N, K, cut.part_len,
                           cut.groups, split);
}
}  // namespace

EG_API int eg_gemm_f32_nt(cudaStream_t stream, const float* A, int lda, const float* W, int ldw, const float* bias,
                          float* C, int ldc, int M, int N, int K) {
    if (M <= 0 || N <= 0) return 0;
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
    return vec ? launch_f32<true>(stream, A, lda, W, ldw, bias, C, ldc, M, N, K) : launch_f32<false>(stream, A, lda, W, ldw, bias, C, ldc, M, N, K);
}
