// Matrix products of a decode chain for steps of 17 to 64 tokens on tcgen05: y[m, n] = sum_k x[m, k] W[n, k].
//
// What the library's products cost here is what stands around them: 4 to 6 us each for 1.6 to 17 MB of weights, and between them
// kernels for the norms, the rotation and SwiGLU, all started one after the other (62 us a layer of the 0.5B sizes at 64 tokens).
// So, as gemm_stream.cu does for fewer tokens:
//
//   weights   boxes of 64 terms by BN rows come by TMA into a ring, asked for before the dependency wait; x's boxes behind it.
//   products  the tokens are the M side of tcgen05.mma (128 rows; those behind the last token read whatever lies there and are
//             not looked at), BN weight rows its N side; the sums are in TMEM, a token a lane.
//   sums      CTAs that share a K range are a cluster; each owns BN / CS of the columns and gets the others' parts of them by
//             st.async, counted on its mbarrier, and adds them up in their order.
//   prologue  plain rows, or rows prepared by the product in front with partial sums of squares [token][part].
//   epilogues a thread has a token: into the residual with the next norm's preparation, SwiGLU of interleaved rows, or bias,
//             rotation and cache write (a tile is a head).
//
// Bound by the chain of latencies behind the wait (x, the products, the exchange) and by the weights' stream.  A product has one wave of
// CTAs, two of which share an SM: up to 296 of them (gemm_batch_plan.h; at the 0.5B sizes 56 to 152).  Every column tile fetches all of x, as
// many bytes as its weights at 64 tokens, and of the MMA's 128 rows as many are of use as there are tokens: with more than 32 tokens the library
// is faster at most sizes, and so it is at larger widths (plans.hpp has the lines and the figures; a decode step of 32 requests at 300 keys of
// the 0.5B sizes 883 us with the library's products, 756 with these).  Every wait is bounded.
#define EG_NEEDS_TENSOR_MAPS
#include "gemm_skinny.cuh"
#include "gemm_batch_plan.h"
#include "mbarrier.cuh"

namespace {
using namespace skinny;
using batch_plan::BK;

constexpr int THREADS = 192;                  // two warps of tokens, one that copies, one that multiplies, two that help with the sums of squares
constexpr unsigned PARTS_WAIT_LIMIT = WAIT_LIMIT << 7;
constexpr int PREFETCH_PIECE = 16 * 1024;

struct Plan {
    int stages, chunks;
};

__device__ __forceinline__ void box_copy(uint32_t to, const CUtensorMap* map, int k, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(to), "l"(map), "r"(k), "r"(row), "r"(smem_addr(bar)) : "memory");
}
// K-major tile of 128-byte rows, 128-byte swizzle, groups of eight rows 1,024 bytes apart
__device__ __forceinline__ uint64_t tile_desc(uint32_t at) {
    return (uint64_t)((at & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void multiply(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_16(uint32_t at, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
    for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    if (status) atomicOr(status, EG_STATUS_WAIT_TIMEOUT);
    return false;
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}

template <int BN, int MT, int CS>
struct Sizes {
    static constexpr int X_BYTES = MT * 128, W_BYTES = BN * 128, STAGE = X_BYTES + W_BYTES;
    static constexpr int OWN = BN / CS, PART_LD = OWN + 4;
    // the products read 128 rows of x: from the last stage on as far as this
    static constexpr int BEHIND = STAGE < 16384 ? 16384 - STAGE : 0;
    static constexpr int PARTS = CS > 1 ? CS * MT * PART_LD * 4 : 0;
    static constexpr int FIXED = 1024 + (PARTS > BEHIND ? PARTS : BEHIND);
};
}  // namespace

template <int BN, int MT, int CS, int EPI, int NORM>
__global__ void __launch_bounds__(THREADS, 2)
batch_kernel(const Params p, const Plan s, const float2* __restrict__ rotations, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w) {
    using Z = Sizes<BN, MT, CS>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    float* parts = reinterpret_cast<float*>(ring + s.stages * Z::STAGE);                     // [CS][MT][PART_LD]
    __shared__ __align__(8) uint64_t full[batch_plan::MAX_STAGES], empty[batch_plan::MAX_STAGES], sums_bar, parts_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float squares[64];
    __shared__ volatile int abort_flag, asked;                    // asked: stages that have been asked for, once the copying thread is done
    TraceScope trace_scope(p.trace);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.y, n0 = blockIdx.x * BN;
    const int kb0 = s.chunks * rank / CS, k_blocks = s.chunks * (rank + 1) / CS - kb0;
    const int ahead = min(k_blocks, s.stages);

    if (threadIdx.x == 64) {
        for (int i = 0; i < s.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&sums_bar, 1);
        mbar_init(&parts_bar, 1);
        abort_flag = 0;
        asked = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if (CS > 1) mbar_expect_tx(&parts_bar, (uint32_t)(CS * MT * Z::OWN * 4));
        for (int i = 0; i < ahead; ++i) {
            mbar_expect_tx(&full[i], Z::STAGE);
            box_copy(smem_addr(ring) + i * Z::STAGE + Z::X_BYTES, &map_w, (kb0 + i) * BK, n0, &full[i]);
        }
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_slot)), "r"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (warp == 2) {
        __syncwarp();
        if (p.prefetch) {
            const int ctas = gridDim.x * gridDim.y, cta = blockIdx.y * gridDim.x + blockIdx.x;
            for (long long at = ((long long)lane * ctas + cta) * PREFETCH_PIECE; at < p.prefetch_bytes; at += 32LL * ctas * PREFETCH_PIECE) {
                const uint32_t n = (uint32_t)min((long long)PREFETCH_PIECE, p.prefetch_bytes - at) & ~15u;
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(static_cast<const char*>(p.prefetch) + at), "r"(n) : "memory");
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (CS > 1) {                                                 // the others' barriers are there before anything is sent
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot;
    // Not before this CTA has its columns of TMEM: a CTA of the kernel behind that took the last of them would wait for this one, and it for them.
    if (p.use_pdl == 1) asm volatile("griddepcontrol.launch_dependents;\n" ::);
    trace_scope.mark(0);
    if (p.use_pdl) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    trace_scope.mark(1);

    bool ok = true;
    if (warp == 2) {
        if (p.use_pdl == 2) asm volatile("griddepcontrol.launch_dependents;\n" ::);
        if (lane == 0) {                                          // ---- copies
            const uint32_t at = smem_addr(ring);
            for (int i = 0; i < ahead; ++i) box_copy(at + i * Z::STAGE, &map_x, (kb0 + i) * BK, 0, &full[i]);
            int slot = 0, phase = 0, i = ahead;
            for (; i < k_blocks; ++i) {
                ok = wait_for(&empty[slot], phase, &abort_flag, p.status);
                if (!ok) break;
                mbar_expect_tx(&full[slot], Z::STAGE);
                box_copy(at + slot * Z::STAGE + Z::X_BYTES, &map_w, (kb0 + i) * BK, n0, &full[slot]);
                box_copy(at + slot * Z::STAGE, &map_x, (kb0 + i) * BK, 0, &full[slot]);
                if (++slot == s.stages) { slot = 0; phase ^= 1; }
            }
            asked = i;
        }
    } else if (warp == 3) {
        if (lane == 0) {                                          // ---- products
            // D float32, A and B bfloat16, K-major; M 128, N BN
            constexpr uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(BN >> 3) << 17 | (uint32_t)(128 >> 4) << 24;
            int slot = 0, phase = 0;
            for (int i = 0; i < k_blocks; ++i) {
                const uint32_t at = smem_addr(ring) + slot * Z::STAGE;
                const uint64_t a = tile_desc(at), b = tile_desc(at + Z::X_BYTES);
                ok = wait_for(&full[slot], phase, &abort_flag, p.status);
                if (!ok) break;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) multiply(tmem, a + 2 * k, b + 2 * k, idesc, (i | k) != 0);
                commit(&empty[slot]);
                if (++slot == s.stages) { slot = 0; phase ^= 1; }
            }
            if (ok) commit(&sums_bar);
        }
    } else {
        // ---- the tokens' epilogue: warps 0 and 1 (TMEM lanes 0 .. 63), helped by 4 and 5
        const int m = threadIdx.x < 64 ? threadIdx.x : threadIdx.x - 128;
        const bool has_token = m < p.M, helper = threadIdx.x >= 64;
        float factor = 1.f;
        if (NORM == 2) {
            // the partial sums of squares of a token, every other four of them a thread, always in the same order
            float4 ss = make_float4(0.f, 0.f, 0.f, 0.f);
            if (has_token) {
                const float4* from = reinterpret_cast<const float4*>(p.ss_in + (size_t)m * p.ss_parts);
#pragma unroll 8
                for (int q = helper; q < p.ss_parts / 4; q += 2) {
                    const float4 v = __ldcg(from + q);
                    ss.x += v.x; ss.y += v.y; ss.z += v.z; ss.w += v.w;
                }
            }
            const float sum = (ss.x + ss.y) + (ss.z + ss.w);
            if (helper) squares[m] = sum;
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
            if (!helper) factor = 1.0f / sqrtf((sum + squares[m]) / (float)p.K + p.eps);
        }
        if (!helper && warp * 32 < MT) {
            constexpr int OWN = Z::OWN;
            // EPI_QKV_ROPE: a tile is a head; rank r of CS owns an even share of its pairs (j, j + half)
            constexpr int half = BN / 2, share = OWN / 2;
            // the residual's share is asked for here, so that its trip runs beside the product
            float v[OWN], resid[EPI == EPI_RESID_NORM ? OWN : 1];
            if (EPI == EPI_RESID_NORM && has_token) {
                const float4* from = reinterpret_cast<const float4*>(p.resid_inout + (size_t)m * p.N + n0 + rank * OWN);
#pragma unroll
                for (int i = 0; i < OWN / 4; ++i) {
                    const float4 f = from[i];
                    resid[4 * i] = f.x; resid[4 * i + 1] = f.y; resid[4 * i + 2] = f.z; resid[4 * i + 3] = f.w;
                }
            }
            const bool summed = __all_sync(0xffffffffu, wait_for(&sums_bar, 0, &abort_flag, p.status));
            trace_scope.mark(3);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t mine = tmem + ((uint32_t)(warp * 32) << 16);
            if (CS > 1) {
                const uint32_t to = smem_addr(parts + ((size_t)rank * MT + m) * Z::PART_LD), bar = smem_addr(&parts_bar);
                uint32_t far[CS], far_bar[CS];
#pragma unroll
                for (int o = 0; o < CS; ++o) {
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(far[o]) : "r"(to), "r"(o));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(far_bar[o]) : "r"(bar), "r"(o));
                }
#pragma unroll
                for (int c0 = 0; c0 < BN; c0 += 16) {
                    float t[16];
                    tmem_16(mine + c0, t);
#pragma unroll
                    for (int c = c0; c < c0 + 16; c += 4) {
                        const int jj = c % half, o = EPI == EPI_QKV_ROPE ? jj / share : c / OWN, place = EPI == EPI_QKV_ROPE ? c / half * share + jj % share : c % OWN;
                        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n"
                                     ::"r"(far[o] + (uint32_t)place * 4u), "r"(__float_as_uint(t[c - c0])), "r"(__float_as_uint(t[c - c0 + 1])),
                                       "r"(__float_as_uint(t[c - c0 + 2])), "r"(__float_as_uint(t[c - c0 + 3])), "r"(far_bar[o]) : "memory");
                    }
                }
                // (The others send their parts whatever became of their own waits, at most one limit a stage later: this CTA must
                // not be gone by then.)
                bool landed = false;
                for (unsigned i = 0; i < PARTS_WAIT_LIMIT && !landed; ++i) landed = try_wait_cluster(&parts_bar, 0);
                if (!landed && p.status) atomicOr(p.status, EG_STATUS_WAIT_TIMEOUT);
                ok = summed && __all_sync(0xffffffffu, landed);
#pragma unroll
                for (int i = 0; i < OWN; i += 4) {
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int o = 0; o < CS; ++o) {
                        const float4 f = *reinterpret_cast<const float4*>(parts + ((size_t)o * MT + m) * Z::PART_LD + i);
                        sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
                    }
                    v[i] = sum.x; v[i + 1] = sum.y; v[i + 2] = sum.z; v[i + 3] = sum.w;
                }
            } else {
                ok = summed;
#pragma unroll
                for (int c0 = 0; c0 < OWN; c0 += 16) {
                    float t[16];
                    tmem_16(mine + c0, t);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[c0 + i] = t[i];
                }
            }
            trace_scope.mark(4);
            const int first = n0 + rank * OWN;                    // of the columns owned (other than EPI_QKV_ROPE's)
            if (!ok || !has_token) {
            } else if (EPI == EPI_SWIGLU) {
                bf16* out = p.out + (size_t)m * p.ldo + first / 2;
                uint32_t packed[OWN / 4];
#pragma unroll
                for (int i = 0; i < OWN / 4; ++i) {
                    float y[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float g = v[4 * i + 2 * e], u = v[4 * i + 2 * e + 1];
                        if (NORM) { g *= factor; u *= factor; }
                        if (p.bias) { g += p.bias[first + 4 * i + 2 * e]; u += p.bias[first + 4 * i + 2 * e + 1]; }
                        // the hardware's base-2 exponent and reciprocal (2^-22 each) for a result that is rounded to bfloat16
                        float z, r;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(z) : "f"(-1.4426950408889634f * g));
                        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + z));
                        y[e] = u * (g * r);
                    }
                    const __nv_bfloat162 h = __floats2bfloat162_rn(y[0], y[1]);
                    packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
#pragma unroll
                for (int i = 0; i < OWN / 16; ++i) reinterpret_cast<uint4*>(out)[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
            } else if (EPI == EPI_RESID_NORM) {
                float sq = 0.f;
                uint32_t packed[OWN / 2];
#pragma unroll
                for (int i = 0; i < OWN; ++i) {
                    float y = v[i];
                    if (NORM) y *= factor;
                    if (p.bias) y += p.bias[first + i];
                    v[i] = resid[i] + __bfloat162float(__float2bfloat16_rn(y));      // what a stored delta would hold
                    sq = fmaf(v[i], v[i], sq);
                }
#pragma unroll
                for (int i = 0; i < OWN / 2; ++i) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(p.gain_out[first + 2 * i] * v[2 * i], p.gain_out[first + 2 * i + 1] * v[2 * i + 1]);
                    packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
#pragma unroll
                for (int i = 0; i < OWN / 4; ++i)
                    reinterpret_cast<float4*>(p.resid_inout + (size_t)m * p.N + first)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
#pragma unroll
                for (int i = 0; i < OWN / 8; ++i)
                    reinterpret_cast<uint4*>(p.xn_out + (size_t)m * p.N + first)[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
                p.ss_out[(size_t)m * (p.N / OWN) + first / OWN] = sq;
            } else {                                              // EPI_QKV_ROPE
                const int head = blockIdx.x, j0 = rank * share;
                const bool query = head < p.num_heads, key = !query && head < p.num_heads + p.num_kv_heads;
                bf16* to = nullptr;
                if (query) {
                    to = p.out + (size_t)m * p.ldo + (size_t)head * BN;
                } else {
                    const long long slot = p.slot_map[m];
                    if (slot >= p.pool_slots) atomicOr(p.status, EG_STATUS_BAD_SLOT);
                    else if (slot >= 0)
                        to = (key ? p.k_cache : p.v_cache) + (slot / p.page_size) * p.page_stride +
                             (long long)(head - p.num_heads - (key ? 0 : p.num_kv_heads)) * p.head_stride + (slot % p.page_size) * BN;
                }
#pragma unroll
                for (int i = 0; i < share; i += 2) {
                    float4 turn = make_float4(1.f, 0.f, 1.f, 0.f);                     // of values: cosine 1, sine 0
                    if (query || key) turn = __ldcg(reinterpret_cast<const float4*>(rotations + (size_t)m * half + j0 + i));
                    float x[2][2];
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int up = 0; up < 2; ++up) {
                            float y = v[up * share + i + e];
                            if (NORM) y *= factor;
                            if (p.bias) y += p.bias[head * BN + up * half + j0 + i + e];
                            x[e][up] = y;
                        }
                    if (!to) continue;
                    *reinterpret_cast<__nv_bfloat162*>(to + j0 + i) =
                        __floats2bfloat162_rn(x[0][0] * turn.x - x[0][1] * turn.y, x[1][0] * turn.z - x[1][1] * turn.w);
                    *reinterpret_cast<__nv_bfloat162*>(to + half + j0 + i) =
                        __floats2bfloat162_rn(x[0][0] * turn.y + x[0][1] * turn.x, x[1][0] * turn.w + x[1][1] * turn.z);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    // Nothing leaves while copies are on their way: the products have seen every stage full unless a wait gave up; then the last copy
    // of each stage is waited for here, with a limit.
    if (abort_flag && threadIdx.x == 64) {
        unsigned left = WAIT_LIMIT;
        for (int it = max(0, asked - s.stages); it < asked; ++it)
            while (left && !mbar_try_wait(&full[it % s.stages], (uint32_t)(it / s.stages) & 1u)) --left;
    }
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(BN) : "memory");
    }
}

namespace {
template <int BN, int MT, int CS, int EPI, int NORM>
int launch(cudaStream_t stream, const Params& p, const float2* rotations) {
    using Z = Sizes<BN, MT, CS>;
    Plan s{};
    s.chunks = p.K / BK;
    const int most = (s.chunks + CS - 1) / CS;
    s.stages = (batch_plan::SHARED - Z::FIXED) / Z::STAGE;
    if (s.stages > batch_plan::MAX_STAGES) s.stages = batch_plan::MAX_STAGES;
    if (s.stages > most) s.stages = most;
    const int smem = Z::FIXED + s.stages * Z::STAGE;
    const eg_encode_tiled_fn encode = eg_encode_tiled();
    if (!encode) return (int)cudaErrorNotSupported;
    CUtensorMap maps[2];
    for (int i = 0; i < 2; ++i) {
        const void* base = i ? (const void*)p.W : NORM == 2 ? (const void*)p.delta : (const void*)p.x;
        const cuuint64_t dims[2] = {(cuuint64_t)p.K, (cuuint64_t)(i ? p.N : p.M)}, strides[1] = {(cuuint64_t)(i ? p.ldw : NORM == 2 ? p.K : p.ldx) * 2};
        const cuuint32_t box[2] = {BK, (cuuint32_t)(i ? BN : MT)}, steps[2] = {1, 1};
        if (encode(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, i ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return (int)cudaErrorInvalidValue;
    }
    auto kernel = batch_kernel<BN, MT, CS, EPI, NORM>;
    static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, batch_plan::SHARED);
    if (configured != cudaSuccess) return (int)configured;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.N / BN), CS);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (CS > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = CS;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (p.use_pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return (int)cudaLaunchKernelEx(&cfg, kernel, p, s, rotations, maps[0], maps[1]);
}
template <int BN, int CS, int EPI, int NORM>
int launch_tokens(cudaStream_t stream, const Params& p, const float2* rotations) {
    return p.M <= 32 ? launch<BN, 32, CS, EPI, NORM>(stream, p, rotations) : launch<BN, 64, CS, EPI, NORM>(stream, p, rotations);
}
bool kind_of(int epilogue, batch_plan::Kind* kind) {
    if (epilogue == EPI_SWIGLU) *kind = batch_plan::SWIGLU;
    else if (epilogue == EPI_RESID_NORM) *kind = batch_plan::INTO_RESIDUAL;
    else if (epilogue == EPI_QKV_ROPE) *kind = batch_plan::QKV;
    else return false;
    return true;
}
}  // namespace

// Whether eg_gemm_batch takes these sizes for 17 to 64 tokens: 0, or into how many partial sums of squares a row of N goes
// (EPI_RESID_NORM; 1 for the other epilogues).
EG_API int eg_gemm_batch_takes(int epilogue, int N, int K, int head_dim) {
    batch_plan::Kind kind;
    batch_plan::Cut c{};
    if (!kind_of(epilogue, &kind) || !batch_plan::cut_for(kind, N, K, head_dim, &c)) return 0;
    return kind == batch_plan::INTO_RESIDUAL ? N / (c.columns / c.split) : 1;
}

// One product of a decode chain for M of 17 to 64 tokens.  W is read ahead, while the kernel in front still runs: nothing in the stream may
// write it.  epilogue 2 (SwiGLU of interleaved gate and up rows, out [M, N / 2]) and 3 (bias,
// rotation by `rotations` [M, head_dim / 2] cosines and sines, cache write; queries to out) read prepared rows x [M, K] with ss_in [M, ss_parts]
// partial sums of squares; epilogue 4 (resid += x W^T + bias, xn = gain * resid, ss_out [M, parts] partial sums of squares of resid) reads
// plain rows x [M, ldx].
EG_API int eg_gemm_batch(cudaStream_t stream, int epilogue, int use_pdl, const void* W, long long ldw, const float* bias, int M, int N, int K, const void* x,
                         long long ldx, float eps, const float* ss_in, int ss_parts, void* out, long long ldo, int num_heads, int num_kv_heads, int head_dim,
                         const float* rotations, const int* slot_map, void* k_cache, void* v_cache, int page_size, long long page_stride, long long head_stride,
                         long long pool_slots, float* resid, const float* gain_out, void* xn_out, float* ss_out, const void* prefetch, long long prefetch_bytes,
                         int* status) {
    batch_plan::Kind kind;
    batch_plan::Cut c{};
    auto aligned = [](const void* q) { return (uintptr_t)q % 16 == 0; };
    if (M < batch_plan::LEAST_TOKENS || M > batch_plan::MOST_TOKENS || !kind_of(epilogue, &kind) || !batch_plan::cut_for(kind, N, K, head_dim, &c) || ldw % 8 || ldx % 8 ||
        !aligned(W) || !aligned(x) || !status)
        return (int)cudaErrorInvalidValue;
    if (kind == batch_plan::INTO_RESIDUAL) {
        if (!resid || !gain_out || !xn_out || !ss_out || !aligned(resid) || !aligned(xn_out)) return (int)cudaErrorInvalidValue;
    } else if (!ss_in || ss_parts < 4 || ss_parts % 4 || !aligned(ss_in) || !out || ldx != K) {
        return (int)cudaErrorInvalidValue;
    }
    if (kind == batch_plan::SWIGLU && (!aligned(out) || ldo % 8)) return (int)cudaErrorInvalidValue;
    if (kind == batch_plan::QKV && ((num_heads + 2 * num_kv_heads) * head_dim != N || !rotations || !aligned(rotations) || !slot_map || !k_cache || !v_cache || ldo % 2 ||
                                    (uintptr_t)out % 4 || (uintptr_t)k_cache % 4 || (uintptr_t)v_cache % 4 || page_stride % 2 || head_stride % 2 || page_size < 1))
        return (int)cudaErrorInvalidValue;
    Params p{};
    p.W = (const bf16*)W;
    p.ldw = ldw;
    p.bias = bias;
    p.M = M;
    p.N = N;
    p.K = K;
    p.x = p.delta = (const bf16*)x;
    p.ldx = ldx;
    p.eps = eps;
    p.out = (bf16*)out;
    p.ldo = ldo;
    p.num_heads = num_heads;
    p.num_kv_heads = num_kv_heads;
    p.head_dim = head_dim;
    p.slot_map = slot_map;
    p.k_cache = (bf16*)k_cache;
    p.v_cache = (bf16*)v_cache;
    p.page_size = page_size;
    p.page_stride = page_stride;
    p.head_stride = head_stride;
    p.pool_slots = pool_slots;
    p.status = status;
    p.use_pdl = use_pdl;
    p.ss_in = ss_in;
    p.ss_parts = ss_parts;
    p.resid_inout = resid;
    p.gain_out = gain_out;
    p.xn_out = (bf16*)xn_out;
    p.ss_out = ss_out;
    p.prefetch = (uintptr_t)prefetch % 16 == 0 ? prefetch : nullptr;
    p.prefetch_bytes = prefetch_bytes;
    const float2* turns = (const float2*)rotations;
    if (kind == batch_plan::SWIGLU) return c.split == 1 ? launch_tokens<64, 1, EPI_SWIGLU, 2>(stream, p, turns) : launch_tokens<64, 2, EPI_SWIGLU, 2>(stream, p, turns);
    if (kind == batch_plan::INTO_RESIDUAL)
        return c.split == 4 ? launch_tokens<64, 4, EPI_RESID_NORM, 0>(stream, p, turns) : launch_tokens<64, 8, EPI_RESID_NORM, 0>(stream, p, turns);
    if (c.columns == 64) return c.split == 4 ? launch_tokens<64, 4, EPI_QKV_ROPE, 2>(stream, p, turns) : launch_tokens<64, 8, EPI_QKV_ROPE, 2>(stream, p, turns);
    return c.split == 4 ? launch_tokens<128, 4, EPI_QKV_ROPE, 2>(stream, p, turns) : launch_tokens<128, 8, EPI_QKV_ROPE, 2>(stream, p, turns);
}
