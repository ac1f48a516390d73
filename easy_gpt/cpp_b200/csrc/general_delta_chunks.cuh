// The generalised delta rule (general_delta.cu) over prompts, heads of 64: tokens in chunks of 16 (counted from the entry's first
// token of the step; the last one is filled up in front with tokens that change nothing).
//
// With G_t = w_0 .. w_t channel by channel and S the state in front of a chunk, what the tokens' old states hold along their unit
// keys, H (a row h_t per token), satisfies (1 + A) H = U S + B V, where A and B are strictly lower triangular,
//   U_t = u_t G_(t-1),   A_tj = u_t . (w_(j+1) .. w_(t-1) a_j u_j),   B_tj = u_t . (w_(j+1) .. w_(t-1) k_j),
// and the outputs and the state behind the chunk are
//   O = R S + P V - Q H,   S' = diag(G_15) S + K^T V - D^T H,
//   R_t = r_t G_t,   P_tj = r_t . (w_(j+1) .. w_t k_j),   Q_tj = r_t . (w_(j+1) .. w_t a_j u_j)   (j <= t),
//   K_j = k_j w_(j+1) .. w_15,   D_j = a_j u_j w_(j+1) .. w_15
// (nothing is divided by a decay).  All that does not read S is worked out for all chunks at once: X and H0 with (1 + A) X = U,
// (1 + A) H0 = B V by forward substitution, R - Q X and P V - Q H0.  What is left in the chain of chunks is
//   H = X S + H0;   O = (R - Q X) S + (P V - Q H0);   S' = diag(G_15) S + K^T V - D^T H.
//
// Sums are float32; the running products of the decays are worked out in 64 bits and rounded once.  Where two kinds of terms meet (what
// tokens write and what they take off) each kind is added up by itself, and S gets their sum in one step: added onto S one after the
// other, sixteen roundings of S's size a chunk, the state was twice as far off the result in 64 bits as block by block.  The last term of
// K^T V is added exactly (the loss goes along): with fast decays it is most of the sum.  (2-norm errors x 1e-8 of the state and of the gated
// outputs, blocks of four / this, by the mean logit of the decays, 257 tokens: -9, 28.2 24.5 / 20.2 19.9; -2, 9.4 14.2 / 8.8 14.1; 0, 7.1 13.8 / 6.6
// 13.2; 5, 5.7 15.5 / 5.0 12.8.)
//
// What bounds the chain: its latency, two trips through shared memory a chunk (H's parts, the state) with two barriers of four warps and
// one of eight.  A chunk is 1.25 us, about 2,400 cycles; the multiply-adds of its four products, 64 x 16 a token and 16 columns each, are 512 of
// them.  A block has 16 columns of a head: 128 blocks for 32 heads and one prompt.  (Measured: the rule over 2,047 tokens, 32 heads, 357 us with
// blocks of four tokens, 253 with this; 8 entries of 256 tokens 248 and 213.)  Four warps have the state in registers and work out H and
// D^T H, four more the outputs and, a chunk ahead, K^T V.
#pragma once

constexpr int CHUNK = 16, CHUNK_DIM = 64, CHUNK_COLS = 16;
constexpr int CHUNK_SHARED = 4 * CHUNK * CHUNK_DIM + CHUNK_DIM;       // floats of X^T, (R - Q X)^T [64][16], D, K [16][64], G_15
constexpr int CHUNK_SLICE = 3 * CHUNK * CHUNK_COLS;                   // V, H0, P V - Q H0 of 16 columns, [16 tokens][16] each
constexpr int CHUNK_RECORD = CHUNK_SHARED + CHUNK_DIM / CHUNK_COLS * CHUNK_SLICE;
constexpr int CHUNK_STAGES = 3, CHUNK_STAGE = CHUNK_SHARED + CHUNK_SLICE;
constexpr int PART_LD = 18;                                            // of rows of 16 that are written in tiles of four rows

// the step's chunk `index`, of the entries' chunks one behind the other: its first token and how many it has (false: there is none)
__device__ __forceinline__ bool chunk_at(const int* seq_starts, int num_seqs, int index, int* first, int* count) {
    for (int s = 0; s < num_seqs; ++s) {
        const int lo = seq_starts[s], n = seq_starts[s + 1] - lo, chunks = (n + CHUNK - 1) / CHUNK;
        if (index < chunks) {
            *first = lo + index * CHUNK;
            *count = min(CHUNK, n - index * CHUNK);
            return true;
        }
        index -= chunks;
    }
    return false;
}

// The records of a (chunk, head), 128 threads.  Bound by its instructions: 16 x 17 / 2 pairs of tokens with four dot products of 64 each.
template <bool WIDE>
__global__ void __launch_bounds__(128) general_delta_chunks_kernel(const DeltaParams p, int num_seqs, int most_chunks) {
    pdl_enter();
    __shared__ __align__(16) float sw[CHUNK][CHUNK_DIM], su[CHUNK][CHUNK_DIM], sa[CHUNK][CHUNK_DIM], sk[CHUNK][CHUNK_DIM], sr[CHUNK][CHUNK_DIM],
        sv[CHUNK][CHUNK_DIM];
    __shared__ __align__(16) float coef[4][CHUNK][CHUNK];               // A, B, P, Q
    const int head = blockIdx.x % p.heads, index = blockIdx.x / p.heads, at = head * CHUNK_DIM, tid = threadIdx.x;
    int first = 0, count = 0;
    if (!chunk_at(p.seq_starts, num_seqs, index, &first, &count)) return;
    float* rec = p.records + ((size_t)head * most_chunks + index) * CHUNK_RECORD;
    // ---- the tokens' vectors: sixteen lanes a token, four channels each
    auto load = [&](const float* src) {
        if (WIDE) return *reinterpret_cast<const float4*>(src);
        return make_float4(src[0], src[1], src[2], src[3]);
    };
    const int d = (tid & 15) * 4;
    const float4 w0 = load(p.w0 + at + d), a0 = load(p.a0 + at + d);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int t = (tid >> 4) + half * 8;
        const bool live = t >= CHUNK - count;
        const int token = live ? first + t - (CHUNK - count) : first;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* row = p.proj + (size_t)token * p.ldp + at + d;
        const float4 k = live ? load(row + p.k_col) : zero, r = live ? load(row + p.r_col) : zero, v = live ? load(row + p.v_col) : zero;
        const float4 a = load(row + p.a_col), x = load(p.x + (size_t)token * p.ldx + at + d);
        float kk = fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w)));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) kk += __shfl_xor_sync(0xffffffffu, kk, o);
        const float inv = live ? 1.0f / sqrtf(kk + p.unit_eps) : 0.f;        // (what fills a chunk up has no key to divide by, whatever unit_eps is)
        auto decay = [&](float z) { return live ? decay_exp(-p.decay_scale * sigmoid_f(z)) : 1.0f; };
        const float4 u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
        *reinterpret_cast<float4*>(&sw[t][d]) = make_float4(decay(x.x + w0.x), decay(x.y + w0.y), decay(x.z + w0.z), decay(x.w + w0.w));
        *reinterpret_cast<float4*>(&su[t][d]) = u;
        *reinterpret_cast<float4*>(&sa[t][d]) = make_float4(sigmoid_f(a.x + a0.x) * u.x, sigmoid_f(a.y + a0.y) * u.y, sigmoid_f(a.z + a0.z) * u.z,
                                                            sigmoid_f(a.w + a0.w) * u.w);
        *reinterpret_cast<float4*>(&sk[t][d]) = k;
        *reinterpret_cast<float4*>(&sr[t][d]) = r;
        *reinterpret_cast<float4*>(&sv[t][d]) = v;
    }
    __syncthreads();
    // ---- A, B, P, Q: sixteen lanes walk from a token to the chunk's last one, then from its mirror image, so that all walk alike far
    {
        const int pair = tid >> 4;
        float dk[4], da[4];
        int j = pair, t = pair;
        auto four = [](const float* src, float (&f)[4]) {
            const float4 v = *reinterpret_cast<const float4*>(src);
            f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
        };
        four(&sk[j][d], dk);
        four(&sa[j][d], da);
#pragma unroll 1
        for (int i = 0; i <= CHUNK; ++i) {
            float u[4], r[4], w[4], sum[4] = {0.f, 0.f, 0.f, 0.f};
            four(&su[t][d], u);
            four(&sr[t][d], r);
            four(&sw[t][d], w);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sum[0] = fmaf(u[e], da[e], sum[0]);
                sum[1] = fmaf(u[e], dk[e], sum[1]);
                if (t != j) {
                    dk[e] *= w[e];
                    da[e] *= w[e];
                }
                sum[2] = fmaf(r[e], dk[e], sum[2]);
                sum[3] = fmaf(r[e], da[e], sum[3]);
            }
            // four sums over sixteen lanes: two are given away for the neighbour's half of the other two, then one
            const bool hi = tid & 8, mid = tid & 4;
            const float s0 = (hi ? sum[2] : sum[0]) + __shfl_xor_sync(0xffffffffu, hi ? sum[0] : sum[2], 8);
            const float s1 = (hi ? sum[3] : sum[1]) + __shfl_xor_sync(0xffffffffu, hi ? sum[1] : sum[3], 8);
            float s = (mid ? s1 : s0) + __shfl_xor_sync(0xffffffffu, mid ? s0 : s1, 4);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if ((tid & 3) == 0) coef[(hi ? 2 : 0) + (mid ? 1 : 0)][t][j] = s;
            if (++t == CHUNK) {
                j = t = CHUNK - 1 - pair;
                four(&sk[j][d], dk);
                four(&sa[j][d], da);
            }
        }
    }
    __syncthreads();
    if (tid < CHUNK_DIM) {
        // ---- a channel's X and R - Q X
        const int c = tid;
        // (running products in 64 bits: rounded once, they add nothing to what a step by step product of the decays would lose)
        float x[CHUNK];
        double run = 1.0;
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) {
            x[t] = (float)(su[t][c] * run);
            run *= sw[t][c];
            float off = 0.f;
#pragma unroll
            for (int j = 0; j < t; ++j) off = fmaf(-coef[0][t][j], x[j], off);
            x[t] += off;
        }
#pragma unroll
        for (int t = 0; t < CHUNK; t += 4) *reinterpret_cast<float4*>(rec + c * CHUNK + t) = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
        run = 1.0;
#pragma unroll
        for (int t = 0; t < CHUNK; t += 4) {
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                run *= sw[t + e][c];
                float off = 0.f;
#pragma unroll
                for (int j = 0; j <= t + e; ++j) off = fmaf(-coef[3][t + e][j], x[j], off);
                o[e] = (float)(sr[t + e][c] * run) + off;
            }
            *reinterpret_cast<float4*>(rec + CHUNK * CHUNK_DIM + c * CHUNK + t) = make_float4(o[0], o[1], o[2], o[3]);
        }
        rec[4 * CHUNK * CHUNK_DIM + c] = (float)run;
    } else {
        // ---- a channel's D and K, and a column's V, H0 and P V - Q H0
        const int c = tid - CHUNK_DIM;
        double run = 1.0;
#pragma unroll
        for (int t = CHUNK - 1; t >= 0; --t) {
            rec[2 * CHUNK * CHUNK_DIM + t * CHUNK_DIM + c] = (float)(sa[t][c] * run);
            rec[3 * CHUNK * CHUNK_DIM + t * CHUNK_DIM + c] = (float)(sk[t][c] * run);
            run *= sw[t][c];
        }
        float* slice = rec + CHUNK_SHARED + c / CHUNK_COLS * CHUNK_SLICE + c % CHUNK_COLS;
        float v[CHUNK], h[CHUNK];
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) {
            v[t] = sv[t][c];
            float in = 0.f, off = 0.f;
#pragma unroll
            for (int j = 0; j < t; ++j) in = fmaf(coef[1][t][j], v[j], in);
#pragma unroll
            for (int j = 0; j < t; ++j) off = fmaf(-coef[0][t][j], h[j], off);
            h[t] = in + off;
            slice[t * CHUNK_COLS] = v[t];
            slice[(CHUNK + t) * CHUNK_COLS] = h[t];
        }
#pragma unroll
        for (int t = 0; t < CHUNK; ++t) {
            float in = 0.f, off = 0.f;
#pragma unroll
            for (int j = 0; j <= t; ++j) {
                in = fmaf(coef[2][t][j], v[j], in);
                off = fmaf(-coef[3][t][j], h[j], off);
            }
            slice[(2 * CHUNK + t) * CHUNK_COLS] = in + off;
        }
    }
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t minus(uint64_t v) { return v ^ 0x8000000080000000ull; }
__device__ __forceinline__ void chunk_bar(int id) { asm volatile("bar.sync %0, 128;\n" ::"r"(id) : "memory"); }

// The chain: a block per (head, entry, 16 columns), 256 threads.
__global__ void __launch_bounds__(256, 2) general_delta_chain_kernel(const DeltaParams p, int most_chunks) {
    pdl_enter();
    extern __shared__ __align__(128) float smem[];
    __shared__ __align__(8) uint64_t full[CHUNK_STAGES];
    __shared__ int abort_flag;
    __shared__ __align__(16) float state2[2][CHUNK_DIM][CHUNK_COLS * 2];           // the state in front of a chunk, every value twice
    __shared__ __align__(16) float part[2][4][CHUNK][PART_LD];                     // of H and O: four parts of the 64 channels
    __shared__ __align__(16) float off2[CHUNK][CHUNK_COLS * 2];                    // -H, every value twice
    __shared__ __align__(16) float4 taken[2][2][128];                              // K^T V without its last term, a thread's eight values
    const int head = blockIdx.x, seq = blockIdx.y, j0 = blockIdx.z * CHUNK_COLS, tid = threadIdx.x & 127;
    const bool keeper = threadIdx.x < 128;                                          // of the state
    const int start = p.seq_starts[seq], count = p.seq_starts[seq + 1] - start, chunks = (count + CHUNK - 1) / CHUNK;
    if (chunks <= 0) return;
    int before = 0;
    for (int s = 0; s < seq; ++s) before += (p.seq_starts[s + 1] - p.seq_starts[s] + CHUNK - 1) / CHUNK;
    const float* source = p.records + ((size_t)head * most_chunks + before) * CHUNK_RECORD;
    auto fill = [&](int c) {                                                        // one thread
        float* to = smem + (c % CHUNK_STAGES) * CHUNK_STAGE;
        const float* from = source + (size_t)c * CHUNK_RECORD;
        uint64_t* bar = &full[c % CHUNK_STAGES];
        mbar_expect_tx(bar, CHUNK_STAGE * 4);
        bulk_load(to, from, CHUNK_SHARED * 4, bar);
        bulk_load(to + CHUNK_SHARED, from + CHUNK_SHARED + blockIdx.z * CHUNK_SLICE, CHUNK_SLICE * 4, bar);
    };
    auto arrived = [&](int c) { return mbar_wait_bounded(&full[c % CHUNK_STAGES], (c / CHUNK_STAGES) & 1, &abort_flag, p.status, WAIT_LIMIT); };
    auto stage_of = [&](int c) { return smem + (c % CHUNK_STAGES) * CHUNK_STAGE; };
    if (threadIdx.x == 0) {
        for (int s = 0; s < CHUNK_STAGES; ++s) mbar_init(&full[s], 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int c = 0; c < min(CHUNK_STAGES - 1, chunks); ++c) fill(c);
    }
    // tiles of four rows and two columns of the state (a warp: eight by four) and of four tokens and two columns (four by eight; the warps
    // are the parts of the channels)
    const int row = ((tid >> 2) & 7) * 4 + (tid >> 6) * 32, col = (tid & 3) * 2 + ((tid >> 5) & 1) * 8;
    const int quarter = tid >> 5, token = ((tid >> 3) & 3) * 4, token_col = (tid & 7) * 2;
    float* S = p.state + (size_t)p.seq_slots[seq] * p.slot_floats + p.state_offset + ((size_t)head * CHUNK_DIM + j0 + col) * CHUNK_DIM + row;
    uint64_t s[2][2];                                                               // [column][rows 0, 1 or 2, 3]
    auto put_state = [&](int which) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float a0, a1, b0, b1;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(s[0][i]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(s[1][i]));
            *reinterpret_cast<float4*>(&state2[which][row + 2 * i][col * 2]) = make_float4(a0, a0, b0, b0);
            *reinterpret_cast<float4*>(&state2[which][row + 2 * i + 1][col * 2]) = make_float4(a1, a1, b1, b1);
        }
    };
    if (keeper) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float4 f = *reinterpret_cast<const float4*>(S + c * CHUNK_DIM);
            s[c][0] = pair_of(f.x, f.y);
            s[c][1] = pair_of(f.z, f.w);
        }
        put_state(0);
    }
    // [16 tokens][16 columns] = m^T state, this warp's quarter of the channels, into part[which]
    auto product = [&](const float* m, const float (*st)[CHUNK_COLS * 2], int which) {
        // (two sums side by side, of the even and of the odd channels: shorter chains, fewer roundings)
        uint64_t acc[2][2] = {}, odd[2][2] = {};
        const float* mk = m + quarter * 16 * CHUNK + token;
        const float* sk = &st[quarter * 16][token_col * 2];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(mk + k * CHUNK), b = *reinterpret_cast<const ulonglong2*>(sk + k * CHUNK_COLS * 2);
            acc[0][0] = fma2(a.x, b.x, acc[0][0]);
            acc[0][1] = fma2(a.y, b.x, acc[0][1]);
            acc[1][0] = fma2(a.x, b.y, acc[1][0]);
            acc[1][1] = fma2(a.y, b.y, acc[1][1]);
            const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(mk + (k + 1) * CHUNK), d = *reinterpret_cast<const ulonglong2*>(sk + (k + 1) * CHUNK_COLS * 2);
            odd[0][0] = fma2(c.x, d.x, odd[0][0]);
            odd[0][1] = fma2(c.y, d.x, odd[0][1]);
            odd[1][0] = fma2(c.x, d.y, odd[1][0]);
            odd[1][1] = fma2(c.y, d.y, odd[1][1]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            acc[0][i] = add2(acc[0][i], odd[0][i]);
            acc[1][i] = add2(acc[1][i], odd[1][i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float a0, a1, b0, b1;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(acc[0][i]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(acc[1][i]));
            *reinterpret_cast<float2*>(&part[which][quarter][token + 2 * i][token_col]) = make_float2(a0, b0);
            *reinterpret_cast<float2*>(&part[which][quarter][token + 2 * i + 1][token_col]) = make_float2(a1, b1);
        }
    };
    const int sum_token = tid >> 3, sum_col = (tid & 7) * 2;
    auto sums = [&](int which, const float* plus) {                                 // of a token's two columns
        float2 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float2*>(&part[which][i][sum_token][sum_col]);
        const float2 z = *reinterpret_cast<const float2*>(plus + sum_token * CHUNK_COLS + sum_col);
        return make_float2((q[0].x + q[1].x) + (q[2].x + q[3].x) + z.x, (q[0].y + q[1].y) + (q[2].y + q[3].y) + z.y);
    };
    auto take_in = [&](int c) {                                                     // K^T V of chunk c, without its last term
        const float *K = stage_of(c) + 3 * CHUNK * CHUNK_DIM + row, *V = stage_of(c) + CHUNK_SHARED + col;
        uint64_t acc[2][2] = {};
#pragma unroll
        for (int j = 0; j < CHUNK - 1; ++j) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(K + j * CHUNK_DIM);
            const float2 v = *reinterpret_cast<const float2*>(V + j * CHUNK_COLS);
            const uint64_t v0 = pair_of(v.x, v.x), v1 = pair_of(v.y, v.y);
            acc[0][0] = fma2(k.x, v0, acc[0][0]);
            acc[0][1] = fma2(k.y, v0, acc[0][1]);
            acc[1][0] = fma2(k.x, v1, acc[1][0]);
            acc[1][1] = fma2(k.y, v1, acc[1][1]);
        }
        *reinterpret_cast<ulonglong2*>(&taken[c & 1][0][tid]) = make_ulonglong2(acc[0][0], acc[0][1]);
        *reinterpret_cast<ulonglong2*>(&taken[c & 1][1][tid]) = make_ulonglong2(acc[1][0], acc[1][1]);
    };
    __syncthreads();
    bool ok = true;
    if (!keeper) {
        ok = arrived(0);
        if (ok) take_in(0);
    }
    ok = __syncthreads_and(ok);
    int done = 0;
    for (int c = 0; c < chunks && ok; ++c) {
        // (the stage that is filled was read by chunk c - 1)
        if (threadIdx.x == 0 && c + CHUNK_STAGES - 1 < chunks) fill(c + CHUNK_STAGES - 1);
        const float* stage = stage_of(c);
        ok = arrived(c);
        if (keeper) {
            product(stage, state2[c & 1], 0);
            chunk_bar(1);
            const float2 h = sums(0, stage + CHUNK_SHARED + CHUNK * CHUNK_COLS);
            *reinterpret_cast<float4*>(&off2[sum_token][sum_col * 2]) = make_float4(-h.x, -h.x, -h.y, -h.y);
            const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(stage + 4 * CHUNK * CHUNK_DIM + row);
            // K^T V's last term, with what its product and its addition lose (an exact product by a fused multiply-add and Knuth's exact sum): -D^T H
            // is added up from there on
            ulonglong2 in[2], sum[2];
            {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(stage + 3 * CHUNK * CHUNK_DIM + (CHUNK - 1) * CHUNK_DIM + row);
                const float2 v = *reinterpret_cast<const float2*>(stage + CHUNK_SHARED + (CHUNK - 1) * CHUNK_COLS + col);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const ulonglong2 before = *reinterpret_cast<const ulonglong2*>(&taken[c & 1][e][tid]);
                    const uint64_t b = e ? pair_of(v.y, v.y) : pair_of(v.x, v.x);
                    auto last = [&](uint64_t a, uint64_t s, uint64_t* lost) {
                        const uint64_t p = mul2(a, b), t = add2(s, p), z = add2(t, minus(s));
                        *lost = add2(add2(add2(s, minus(add2(t, minus(z)))), add2(p, minus(z))), fma2(a, b, minus(p)));
                        return t;
                    };
                    uint64_t l0, l1;
                    in[e].x = last(k.x, before.x, &l0);
                    in[e].y = last(k.y, before.y, &l1);
                    sum[e] = make_ulonglong2(l0, l1);
                }
            }
            chunk_bar(1);
            const float* D = stage + 2 * CHUNK * CHUNK_DIM + row;
#pragma unroll
            for (int j = 0; j < CHUNK; ++j) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(D + j * CHUNK_DIM), h2 = *reinterpret_cast<const ulonglong2*>(&off2[j][col * 2]);
                sum[0].x = fma2(a.x, h2.x, sum[0].x);
                sum[0].y = fma2(a.y, h2.x, sum[0].y);
                sum[1].x = fma2(a.x, h2.y, sum[1].x);
                sum[1].y = fma2(a.y, h2.y, sum[1].y);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                s[e][0] = fma2(g.x, s[e][0], add2(in[e].x, sum[e].x));
                s[e][1] = fma2(g.y, s[e][1], add2(in[e].y, sum[e].y));
            }
            put_state((c + 1) & 1);
        } else {
            product(stage + CHUNK * CHUNK_DIM, state2[c & 1], 1);
            chunk_bar(2);
            const float2 o = sums(1, stage + CHUNK_SHARED + 2 * CHUNK * CHUNK_COLS);
            const int skip = c + 1 < chunks ? 0 : chunks * CHUNK - count, t = c * CHUNK + sum_token - skip;
            if (ok && sum_token >= skip)
                *reinterpret_cast<float2*>(p.o_raw + (size_t)(start + t) * ((size_t)p.heads * CHUNK_DIM) + head * CHUNK_DIM + j0 + sum_col) = o;
            if (c + 1 < chunks) {
                ok = arrived(c + 1) && ok;
                take_in(c + 1);
            }
        }
        ok = __syncthreads_and(ok);
        done = c + 1;
    }
    if (!ok) {                                                                      // every copy has to land before the block gives up its shared memory
        if (threadIdx.x == 0)
            for (int c = max(0, done - 1); c < min(done + CHUNK_STAGES - 1, chunks); ++c)
                for (unsigned i = 0; i < WAIT_LIMIT && !mbar_try_wait(&full[c % CHUNK_STAGES], (c / CHUNK_STAGES) & 1); ++i) {}
        return;
    }
    if (keeper) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float4 f;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(s[c][0]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(f.z), "=f"(f.w) : "l"(s[c][1]));
            *reinterpret_cast<float4*>(S + c * CHUNK_DIM) = f;
        }
    }
}
