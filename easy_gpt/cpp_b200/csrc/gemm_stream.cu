// Matrix products for decode steps, weights through shared memory: y[m, n] = sum_k x[m, k] W[n, k] for up to 16 tokens.
//
// Such a product is a stream of the weights, and in a decode step a chain of such streams, each waiting for the kernel in
// front.  What bounds it is (1) how much of its stream is under way while it waits and (2) the chain of latencies behind the
// wait.  So:
//
//   weights   come by TMA (boxes of 64 terms of K by a unit's rows, 128-byte swizzle) into a ring of 16 KB stages, issued by a
//             warp of its own before the dependency wait: up to about 100 KB a CTA is on its way without a register for it,
//             and two CTAs, or this kernel's and the next one's, share an SM.  (A register-fed stream, gemm_skinny.cu, holds
//             64 KB a CTA and leaves little room for the next kernel.)
//   x         comes by asynchronous copies of the multiplying warps behind the wait, this CTA's K range of it, once.
//   products  mma.m16n8k16 with 16 weight rows as its M side and the tokens as its N side, both by ldmatrix; eight warps are
//             row blocks x slices of K, a warp has one 64-term tile of every stage.
//   sums      the slices meet in shared memory, CTAs that share a K range (a cluster) in the first one's: st.async counts
//             on its mbarrier, the others are done at once.  Always in the same order, for 1 to 16 tokens (gemm_stream_plan.h
//             decides by the epilogue, N and K alone which products are taken and how they are cut).
//
// Wide matrices: CTAs walk over consecutive row blocks, a unit at a time; the ring runs on across units.
// Prologues and epilogues are those of gemm_skinny.cu (plain rows or prepared ones with partial sums of squares).
// Every wait is bounded.
#define EG_NEEDS_TENSOR_MAPS
#include "gemm_skinny.cuh"
#include "gemm_stream_plan.h"
#include "mbarrier.cuh"
#include "mma_utils.cuh"

namespace {
using namespace skinny;
using stream_plan::MAX_STAGES;
using stream_plan::MOST_SHARED;
using stream_plan::RED_LD;
using stream_plan::STAGE_BYTES;
using stream_plan::WARPS;                     // that multiply; one more warp issues the copies

constexpr int THREADS = (WARPS + 1) * 32;
constexpr int PREFETCH_PIECE = 16 * 1024;
constexpr unsigned PARTS_WAIT_LIMIT = WAIT_LIMIT << 7;

struct Plan {
    int rb_log;                               // log2 of a unit's row blocks; the other factor of WARPS are slices of K, each one tile of a stage
    int stages;
    int k_len, k_stages;                      // terms of K a CTA has (gridDim.y CTAs share K), in stages
    int blocks;                               // row blocks of 16 in all
    int share, longer;                        // row blocks of a CTA that walks; the first `longer` CTAs have one more (share 0: every CTA has one unit)
    int x_offset, red_offset, parts_offset;   // in shared memory, bytes; the ring is at 0
};

// a box of 64 terms by the map's rows, swizzled in pieces of 16 bytes over 128-byte rows
__device__ __forceinline__ void tile_copy(uint32_t to, const CUtensorMap* map, int k, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(to), "l"(map), "r"(k), "r"(row), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix2(uint32_t& a, uint32_t& b, uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(a), "=r"(b) : "r"(at) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// mbar_wait_bounded for launches that may come without a status word
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
    for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    if (status) atomicOr(status, EG_STATUS_WAIT_TIMEOUT);
    return false;
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(WARPS * 32) : "memory"); }
}  // namespace

// GIVE_UP, for tests: every wait inside the kernel is as if it had run out at once
template <int NT, int EPI, int NORM, bool GIVE_UP>
__global__ void __launch_bounds__(THREADS, 2)
stream_kernel(const Params p, const Plan s, const __grid_constant__ CUtensorMap unit_map, const __grid_constant__ CUtensorMap block_map) {
    constexpr int MT = NT * 8;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);      // swizzled tiles start on 1,024 bytes
    __shared__ __align__(8) uint64_t full[MAX_STAGES], empty[MAX_STAGES], factor_bar, parts_bar;
    __shared__ float factor[MT];
    __shared__ volatile int abort_flag, asked;                    // asked: stages that the copying warp has asked for, once it is done
    TraceScope trace_scope(p.trace);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool clustered = gridDim.y > 1;
    // (Shifts and running counters throughout: a division by a runtime number is 100 cycles and more of a chain that has few.)
    const int RB = 1 << s.rb_log, KS = WARPS >> s.rb_log, row_log = 4 + s.rb_log, rows_per_unit = 1 << row_log;
    const int kc = KS * 64, tile_bytes = rows_per_unit * 128;
    const int k0 = blockIdx.y * s.k_len, k_len = min(s.k_len, p.K - k0), x_stride = s.k_len * 2 + 16;
    const int k_stages = min(s.k_stages, (k_len + kc - 1) >> (9 - s.rb_log));
    // this CTA's row blocks: one unit's, or an even share of consecutive ones
    const int block_lo = s.share ? blockIdx.x * s.share + min((int)blockIdx.x, s.longer) : blockIdx.x << s.rb_log;
    const int block_hi = s.share ? block_lo + s.share + ((int)blockIdx.x < s.longer) : min(s.blocks, block_lo + RB);
    const int units = (block_hi - block_lo + RB - 1) >> s.rb_log, total = units * k_stages;
    // qkv_rope: a unit is 16 rows of a head and the 16 that they are rotated with
    const int half = EPI == EPI_QKV_ROPE ? p.head_dim / 2 : 0;
    const int head = EPI == EPI_QKV_ROPE ? blockIdx.x / (half / 16) : 0, head_part = EPI == EPI_QKV_ROPE ? blockIdx.x % (half / 16) : 0;
    auto row_of = [&](int unit, int r) {                          // row r of a unit in W
        if (EPI == EPI_QKV_ROPE) return head * p.head_dim + (r >> 4) * half + head_part * 16 + (r & 15);
        return (block_lo << 4) + (unit << row_log) + r;
    };
    auto rows_of = [&](int unit) {                                // rows of a unit that exist
        if (EPI == EPI_QKV_ROPE) return 32;
        return min(min(rows_per_unit, ((block_hi - block_lo) << 4) - (unit << row_log)), p.N - row_of(unit, 0));
    };

    if (p.use_pdl == 1) asm volatile("griddepcontrol.launch_dependents;\n" ::);
    if (threadIdx.x == WARPS * 32) {
        for (int i = 0; i < s.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], WARPS);
        }
        mbar_init(&factor_bar, 1);
        mbar_init(&parts_bar, 1);
        abort_flag = GIVE_UP;
        asked = -1;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if (clustered && blockIdx.y == 0) mbar_expect_tx(&parts_bar, (gridDim.y - 1) * (uint32_t)rows_per_unit * (uint32_t)p.M * 4u);
    }
    // a stage's copies, issued by one lane: whole units by one box a tile, the rest of a share (and qkv_rope's pairs) by
    // boxes of one row block; what lies behind the matrix arrives as zeros
    int in_unit = 0, in_stage = 0, in_slot = 0, issued = 0;       // of the next stage to ask for
    auto issue = [&]() {
        const int k = in_stage * kc, rows = rows_of(in_unit), row0 = row_of(in_unit, 0), tiles = min(KS, (k_len - k + 63) >> 6);
        const bool whole = EPI != EPI_QKV_ROPE && (rows == rows_per_unit || row0 + rows >= p.N);
        const int blocks = (rows + 15) >> 4;
        uint32_t to = smem_addr(smem) + (uint32_t)in_slot * STAGE_BYTES;
        if (lane == 0) {
            mbar_expect_tx(&full[in_slot], (uint32_t)(tiles * (whole ? tile_bytes : blocks * 2048)));
            for (int t = 0; t < tiles; ++t, to += tile_bytes) {
                if (whole)
                    tile_copy(to, &unit_map, k0 + k + t * 64, row0, &full[in_slot]);
                else
                    for (int b = 0; b < blocks; ++b) tile_copy(to + b * 2048, &block_map, k0 + k + t * 64, row_of(in_unit, b * 16), &full[in_slot]);
            }
        }
        ++issued;
        if (++in_slot == s.stages) in_slot = 0;
        if (++in_stage == k_stages) { in_stage = 0; ++in_unit; }
    };
    if (warp == WARPS) {
        __syncwarp();
        const int ahead = min(s.stages, total);
        while (issued < ahead) issue();
        __syncwarp();
        if (p.prefetch) {
            const int ctas = gridDim.x * gridDim.y, cta = blockIdx.y * gridDim.x + blockIdx.x;
            for (long long at = ((long long)lane * ctas + cta) * PREFETCH_PIECE; at < p.prefetch_bytes; at += 32LL * ctas * PREFETCH_PIECE) {
                const uint32_t n = (uint32_t)min((long long)PREFETCH_PIECE, p.prefetch_bytes - at) & ~15u;
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(static_cast<const char*>(p.prefetch) + at), "r"(n) : "memory");
            }
        }
    }
    if (clustered) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    } else {
        __syncthreads();
    }

    if (warp == WARPS) {
        // ---- the warp that copies
        if (p.use_pdl) asm volatile("griddepcontrol.wait;\n" ::: "memory");
        if (p.use_pdl == 2) asm volatile("griddepcontrol.launch_dependents;\n" ::);
        if (NORM == 2) {
            // the rows' factors from the partial sums of squares, four lanes a token, always in the same order
#pragma unroll 1
            for (int tile = 0; tile < NT; ++tile) {
                const int m = tile * 8 + (lane & 7);
                float ss = 0.f;
#pragma unroll 4
                for (int q = lane >> 3; q < p.ss_parts; q += 4) ss += __ldcg(p.ss_in + (size_t)q * MT + m);
                ss += __shfl_xor_sync(0xffffffffu, ss, 8);
                ss += __shfl_xor_sync(0xffffffffu, ss, 16);
                if (lane < 8) factor[m] = m < p.M ? 1.0f / sqrtf(ss / (float)p.K + p.eps) : 0.f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&factor_bar);
        }
        bool ok = !GIVE_UP;
        for (uint32_t phase = 0; ok && issued < total;) {
            ok = wait_for(&empty[in_slot], phase, &abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) issue();
            if (in_slot == 0) phase ^= 1u;
        }
        if (lane == 0) asked = issued;
        return;
    }

    // ---- the warps that multiply
    const int rb = warp & (RB - 1), ks = warp >> s.rb_log;
    // qkv_rope: positions, cache slots, frequencies and biases were there before the step began; a thread has one token's
    // one output pair (M <= 16) and prepares its rotation and where it goes here
    float rope_cos = 1.f, rope_sin = 0.f, bias0 = 0.f, bias1 = 0.f;
    bf16* rope_out = nullptr;
    const int pair_m = threadIdx.x >> 4, pair_j = head_part * 16 + (threadIdx.x & 15);
    if (EPI == EPI_QKV_ROPE && pair_m < p.M) {
        if (head < p.num_heads + p.num_kv_heads) {
            const float a = (float)p.positions[pair_m] * p.inv_freq[pair_j];
            rope_cos = cosf(a);
            rope_sin = sinf(a);
        }
        if (p.bias) {
            bias0 = p.bias[head * p.head_dim + pair_j];
            bias1 = p.bias[head * p.head_dim + half + pair_j];
        }
        if (head < p.num_heads) {
            rope_out = p.out + (size_t)pair_m * p.ldo + (size_t)head * p.head_dim;
        } else {
            const long long slot = p.slot_map[pair_m];
            const bool key = head < p.num_heads + p.num_kv_heads;
            if (slot >= p.pool_slots) atomicOr(p.status, EG_STATUS_BAD_SLOT);
            else if (slot >= 0)
                rope_out = (key ? p.k_cache : p.v_cache) + (slot / p.page_size) * p.page_stride +
                           (long long)(head - p.num_heads - (key ? 0 : p.num_kv_heads)) * p.head_stride + (slot % p.page_size) * p.head_dim;
        }
    }
    trace_scope.mark(0);
    if (p.use_pdl) asm volatile("griddepcontrol.wait;\n" ::: "memory");       // from here on the kernel in front's results are read
    trace_scope.mark(1);
    // x: a warp has every eighth row
    {
        const bf16* x = NORM == 2 ? p.delta : p.x;
        const long long ldx = NORM == 2 ? p.K : p.ldx;
        for (int m = warp; m < p.M; m += WARPS) {
            const bf16* row = x + (size_t)m * ldx + k0;
            unsigned char* to = smem + s.x_offset + m * x_stride;
            for (int c = lane; c * 8 < k_len; c += 32) cp_async_16(to + c * 16, row + c * 8, true);
        }
        cp_async_commit();
    }
    // resid_norm: sixteen lanes have a token's rows; this lane's first element of the residual and of the gain are asked for
    // here, so that their trip from the L2 runs beside the product
    float resid_first = 0.f, gain_first = 0.f;
    if (EPI == EPI_RESID_NORM && blockIdx.y == 0) {
        const int m = warp * 2 + (lane >> 4), n = block_lo * 16 + (lane & 15);
        if (m < p.M && n < p.N) {
            resid_first = p.resid_inout[(size_t)m * p.N + n];
            gain_first = p.gain_out[n];
        }
    }
    cp_async_wait<0>();
    consumers_sync();
    bool ok = !GIVE_UP;
    trace_scope.mark(2);

    float* red = reinterpret_cast<float*>(smem + s.red_offset);              // [WARPS][MT][RED_LD]
    const uint32_t x_lane = smem_addr(smem) + s.x_offset +
                            (NT == 1 ? (uint32_t)(lane & 7) * x_stride + ((lane >> 3) & 1) * 16
                                     : (uint32_t)((lane & 7) + (lane >> 4) * 8) * x_stride + ((lane >> 3) & 1) * 16);
    uint32_t w_step[4];                                           // the four steps of 16 terms of a swizzled tile row
#pragma unroll
    for (int j = 0; j < 4; ++j)
        w_step[j] = smem_addr(smem) + ks * tile_bytes + (uint32_t)(rb * 16 + (lane & 15)) * 128 + (((j * 2 + (lane >> 4)) ^ (lane & 7)) << 4);
    int slot = 0;
    uint32_t phase = 0;
    // Nothing leaves while copies are on their way: a warp that has waited for every stage has seen all of them land, and one
    // that gave up waits here (with a limit) for the last copy of each stage.
    auto leave = [&]() {
        if (ok) return;
        if (p.status) atomicOr(p.status, EG_STATUS_WAIT_TIMEOUT);
        unsigned left = WAIT_LIMIT;
        while (asked < 0 && --left) {}
        const int in_all = max(0, asked);
        for (int it = max(0, in_all - s.stages); it < in_all; ++it)
            while (left && !mbar_try_wait(&full[it % s.stages], (uint32_t)(it / s.stages) & 1u)) --left;
    };
    for (int unit = 0; unit < units; ++unit) {
        const int rows = rows_of(unit);
        float acc[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
        for (int st = 0; st < k_stages; ++st) {
            ok = ok && wait_for(&full[slot], phase, &abort_flag, p.status);
            const int k = st * kc + ks * 64;
            if (rb * 16 < rows && k < k_len) {
                // all loads of the tile first: the products then follow one another without a trip to shared memory between them
                const uint32_t w_at = (uint32_t)slot * STAGE_BYTES, x_at = x_lane + (uint32_t)k * 2;
                uint32_t a[4][4], b[4][NT][2];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    ldmatrix4(a[j], w_step[j] + w_at);
                    if (NT == 1) {
                        ldmatrix2(b[j][0][0], b[j][0][1], x_at + j * 32);
                    } else {
#pragma unroll
                        for (int nt = 0; nt + 1 < NT; nt += 2) {
                            uint32_t t[4];
                            ldmatrix4(t, x_at + nt * 8 * x_stride + j * 32);
                            b[j][nt][0] = t[0];
                            b[j][nt][1] = t[1];
                            b[j][nt + 1][0] = t[2];
                            b[j][nt + 1][1] = t[3];
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k + j * 16 < k_len)                       // (behind it x is another row's or nobody's memory)
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) mma_bf16_16816(acc[nt], a[j], b[j][nt][0], b[j][nt][1]);
            }
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(&empty[slot]);       // (who gave up has not seen the stage full: it is not asked for again)
            if (++slot == s.stages) { slot = 0; phase ^= 1u; }
        }
        if (unit == 0) {
            trace_scope.mark(3, true);
            if (NORM == 2) ok = ok && wait_for(&factor_bar, 0, &abort_flag, p.status);
        } else {
            consumers_sync();                                     // the unit in front has been read
        }
        // ---- the slices meet: red[warp][token][row]
        const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float* base = red + ((size_t)warp * MT + nt * 8 + 2 * tig) * RED_LD + gid;
            base[0] = acc[nt][0];
            base[RED_LD] = acc[nt][1];
            base[8] = acc[nt][2];
            base[RED_LD + 8] = acc[nt][3];
        }
        consumers_sync();
        trace_scope.mark(4);
        const int slice_step = RB * MT * RED_LD;
        auto slices = [&](int r, int m) {                         // of row r of the unit, in their order
            const float* at = red + ((r >> 4) * MT + m) * RED_LD + (r & 15);
            float v = at[0];
#pragma unroll 1
            for (int i = 1; i < KS; ++i) v += at[i * slice_step];
            return v;
        };
        const int elems = rows_per_unit * p.M;                    // [token][row]
        if (clustered) {
            float* parts = reinterpret_cast<float*>(smem + s.parts_offset);     // [gridDim.y - 1][elems], of the cluster's first CTA
            if (blockIdx.y != 0) {
                uint32_t to, bar;
                asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(to) : "r"(smem_addr(parts + (size_t)(blockIdx.y - 1) * elems)));
                asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(bar) : "r"(smem_addr(&parts_bar)));
                for (int e = threadIdx.x; e < elems; e += WARPS * 32)
                    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n"
                                 ::"r"(to + (uint32_t)e * 4u), "r"(__float_as_uint(slices(e & (rows_per_unit - 1), e >> row_log))), "r"(bar) : "memory");
                leave();
                return;
            }
            // this CTA's own sum first, then the others', in their order; into the first slice's place
            for (int e = threadIdx.x; e < elems; e += WARPS * 32) {
                const int m = e >> row_log, r = e & (rows_per_unit - 1);
                red[((r >> 4) * MT + m) * RED_LD + (r & 15)] = slices(r, m);
            }
            // (The others send their parts whatever became of their own waits, at most one limit a stage later: this CTA
            // must not be gone by then.)
            bool landed = false;
            for (unsigned i = 0; i < PARTS_WAIT_LIMIT && !landed; ++i) landed = try_wait_cluster(&parts_bar, 0);
            if (!landed && p.status) atomicOr(p.status, EG_STATUS_WAIT_TIMEOUT);
            for (int e = threadIdx.x; e < elems; e += WARPS * 32) {
                const int m = e >> row_log, r = e & (rows_per_unit - 1);
                float* at = red + ((r >> 4) * MT + m) * RED_LD + (r & 15);
                float v = *at;
                for (int y = 0; y + 1 < (int)gridDim.y; ++y) v += parts[(size_t)y * elems + e];
                *at = v;
            }
            consumers_sync();
        }
        trace_scope.mark(5);
        auto sum = [&](int r, int m) { return clustered ? red[((r >> 4) * MT + m) * RED_LD + (r & 15)] : slices(r, m); };

        if (EPI == EPI_STORE || EPI == EPI_F32) {
            for (int e = threadIdx.x; e < elems; e += WARPS * 32) {
                const int m = e >> row_log, r = e & (rows_per_unit - 1);
                if (r >= rows) continue;
                const int n = row_of(unit, r);
                float v = sum(r, m);
                if (NORM) v *= factor[m];
                if (p.bias) v += p.bias[n];
                if (EPI == EPI_STORE && p.act == 1) v = v > 0.f ? fmaf(p.act_a * v, v, 0.5f * v) : fmaf(p.act_b, expm1f(v) - v, 0.5f * v);
                if (EPI == EPI_STORE && p.act == 2) v = v > 0.f ? v * v : 0.f;
                if (EPI == EPI_STORE && p.act == 4) v = gelu_erf(v);
                if (EPI == EPI_F32) p.out_f32[(size_t)m * p.ldo + n] = v;
                else p.out[(size_t)m * p.ldo + n] = __float2bfloat16_rn(v);
            }
        } else if (EPI == EPI_SWIGLU) {
            const int pairs = rows_per_unit / 2;
            for (int e = threadIdx.x; e < pairs * p.M; e += WARPS * 32) {
                const int m = e >> (row_log - 1), i = e & (pairs - 1);
                if (2 * i + 1 >= rows) continue;
                const int n = row_of(unit, 2 * i);
                float g = sum(2 * i, m), u = sum(2 * i + 1, m);
                if (NORM) { g *= factor[m]; u *= factor[m]; }
                if (p.bias) { g += p.bias[n]; u += p.bias[n + 1]; }
                bf16* out = p.out + (size_t)m * p.ldo + (n >> 1);
                if (p.act == 3) {                                         // the clamped gate: limit in act_a
                    g = fminf(g, p.act_a);
                    u = fminf(fmaxf(u, -p.act_a), p.act_a);
                    *out = __float2bfloat16_rn(g / (1.0f + expf(-1.702f * g)) * (u + 1.0f));
                    continue;
                }
                const float sig = 1.0f / (1.0f + expf(-g));
                *out = __float2bfloat16_rn(u * (g * sig));
            }
        } else if (EPI == EPI_RESID_NORM) {
            // sixteen lanes share a token: its squares are summed over them by halving, a partial sum per row block
            const int lane16 = lane & 15;
            for (int m0 = warp * 2; m0 < MT; m0 += WARPS * 2) {
                const int m = m0 + (lane >> 4);
                for (int b = 0; b * 16 < rows; ++b) {
                    const int n = row_of(unit, b * 16 + lane16);
                    float sq = 0.f;
                    if (m < p.M && n < p.N) {
                        const bool first = b == 0 && m0 == warp * 2;
                        float y = sum(b * 16 + lane16, m);
                        if (NORM) y *= factor[m];
                        if (p.bias) y += p.bias[n];
                        const float v = (first ? resid_first : p.resid_inout[(size_t)m * p.N + n]) + __bfloat162float(__float2bfloat16_rn(y));      // what a stored delta would hold
                        const float g = first ? gain_first : p.gain_out[n];
                        p.resid_inout[(size_t)m * p.N + n] = v;
                        p.xn_out[(size_t)m * p.N + n] = __float2bfloat16_rn(g * v);
                        sq = v * v;
                    }
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
                    if (lane16 == 0) p.ss_out[(size_t)((row_of(unit, 0) >> 4) + b) * MT + m] = sq;
                }
            }
        } else if (pair_m < p.M) {   // EPI_QKV_ROPE
            float x0 = sum(threadIdx.x & 15, pair_m), x1 = sum(16 + (threadIdx.x & 15), pair_m);
            if (NORM) { x0 *= factor[pair_m]; x1 *= factor[pair_m]; }
            x0 += bias0;
            x1 += bias1;
            const float y0 = x0 * rope_cos - x1 * rope_sin, y1 = x0 * rope_sin + x1 * rope_cos;      // (of values: cosine 1, sine 0)
            if (rope_out) {
                rope_out[pair_j] = __float2bfloat16_rn(y0);
                rope_out[pair_j + half] = __float2bfloat16_rn(y1);
            }
        }
    }
    leave();
}

namespace {
template <int NT, int EPI, int NORM, bool GIVE_UP = false>
int launch(cudaStream_t stream, const Params& p) {
    constexpr int MT = NT * 8;
    constexpr bool pairs = EPI == EPI_QKV_ROPE, walks = !pairs && EPI != EPI_RESID_NORM;
    stream_plan::Cut cut;
    if (!stream_plan::cut_for(p.N, p.K, pairs, walks, &cut)) return -1;
    const stream_plan::Ring ring = stream_plan::ring_of(cut, p.N, MT, walks);
    const int rows = 16 << cut.rb_log, grid = ring.grid, split = cut.split;
    Plan s{};
    s.rb_log = cut.rb_log;
    s.stages = ring.stages;
    s.k_len = cut.k_len;
    s.k_stages = cut.k_stages;
    s.blocks = (p.N + 15) / 16;
    s.share = ring.share;
    s.longer = ring.longer;
    s.x_offset = s.stages * STAGE_BYTES;
    s.red_offset = (s.x_offset + ring.x_bytes + 15) / 16 * 16;
    s.parts_offset = (s.red_offset + ring.red_bytes + 15) / 16 * 16;
    const int smem = 1024 + s.parts_offset + ring.parts_bytes;
    const eg_encode_tiled_fn encode = eg_encode_tiled();
    if (!encode) return -1;
    CUtensorMap maps[2];
    for (int i = 0; i < 2; ++i) {
        const cuuint64_t dims[2] = {(cuuint64_t)p.K, (cuuint64_t)p.N}, strides[1] = {(cuuint64_t)p.ldw * 2};
        const cuuint32_t box[2] = {64, (cuuint32_t)(i == 0 ? rows : 16)}, steps[2] = {1, 1};
        if (encode(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(p.W), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -1;
    }
    auto kernel = stream_kernel<NT, EPI, NORM, GIVE_UP>;
    static const cudaError_t configured = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SHARED);
    if (configured != cudaSuccess) return (int)configured;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, split);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (split > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = (unsigned)split;
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
    return (int)cudaLaunchKernelEx(&cfg, kernel, p, s, maps[0], maps[1]);
}

template <int EPI, int NORM>
int launch_nt(cudaStream_t stream, const Params& p) {
    if constexpr (EPI == EPI_F32 && NORM == 0)
        if (p.give_up) return p.M <= 8 ? launch<1, EPI, NORM, true>(stream, p) : p.M <= 16 ? launch<2, EPI, NORM, true>(stream, p) : -1;
    if (p.M <= 8) return launch<1, EPI, NORM>(stream, p);
    if (p.M <= 16) return launch<2, EPI, NORM>(stream, p);
    return -1;
}
}  // namespace

int eg_gemm_stream_launch(cudaStream_t stream, int epilogue, int norm, const Params& pp) {
    Params p = pp;
    if ((uintptr_t)p.prefetch % 16) p.prefetch = nullptr;
    const bf16* x = norm == 2 ? p.delta : p.x;
    const long long ldx = norm == 2 ? p.K : p.ldx;
    if (norm == 1 || p.K % 16 || p.ldw % 8 || ldx % 8 || (uintptr_t)p.W % 16 || (uintptr_t)x % 16) return -1;
    if (epilogue == EPI_QKV_ROPE && (p.head_dim % 32 || p.M > 16)) return -1;
    if (epilogue == EPI_RESID_NORM && p.RB != 1) return -1;         // its partial sums of squares are per row block here
#define EG_STREAM_CASE(E) \
    case E: return norm == 2 ? launch_nt<E, 2>(stream, p) : launch_nt<E, 0>(stream, p);
    switch (epilogue) {
        EG_STREAM_CASE(EPI_STORE)
        EG_STREAM_CASE(EPI_F32)
        EG_STREAM_CASE(EPI_SWIGLU)
        EG_STREAM_CASE(EPI_QKV_ROPE)
        EG_STREAM_CASE(EPI_RESID_NORM)
    }
#undef EG_STREAM_CASE
    return -1;
}

// The plan, for tests: out[0] whether the products of this epilogue and these sizes are taken (for 1 to 16 tokens alike), out[1..3] row
// blocks a unit (log2), CTAs a unit's K is cut across, terms of each; for `tokens` tokens out[4..7] CTAs an SM, stages of the ring, CTAs or
// clusters, row blocks of the shares (0: a unit each).
EG_API int eg_gemm_stream_plan(int epilogue, int N, int K, int tokens, int* out) {
    if (epilogue < 0 || epilogue > EPI_RESID_NORM || tokens < 1 || tokens > stream_plan::MOST_TOKENS || !out) return (int)cudaErrorInvalidValue;
    const bool pairs = epilogue == EPI_QKV_ROPE, walks = !pairs && epilogue != EPI_RESID_NORM;
    stream_plan::Cut c{};
    out[0] = stream_plan::cut_for(N, K, pairs, walks, &c);
    if (!out[0]) return 0;
    const stream_plan::Ring r = stream_plan::ring_of(c, N, (tokens + 7) / 8 * 8, walks);
    const int values[7] = {c.rb_log, c.split, c.k_len, r.per_sm, r.stages, r.grid, r.share};
    for (int i = 0; i < 7; ++i) out[i + 1] = values[i];
    return 0;
}
