// What the decode products' two kernels (gemm_skinny.cu, gemm_stream.cu) share: the parameters of a launch and its epilogues.
#pragma once
#include "common.cuh"

namespace skinny {

enum { EPI_STORE = 0, EPI_F32 = 1, EPI_SWIGLU = 2, EPI_QKV_ROPE = 3, EPI_RESID_NORM = 4 };

constexpr unsigned WAIT_LIMIT = 1u << 22;    // polls of a wait in gemm_stream.cu

struct Params {
    const bf16* W;
    long long ldw;
    const float* bias;
    int M, N, K;
    const bf16* x;
    long long ldx;
    const float* resid_in;
    float* resid_out;
    const bf16* delta;
    const float* gain;
    float eps;
    bf16* out;
    long long ldo;
    float* out_f32;
    int num_heads, num_kv_heads, head_dim;
    const int* positions;
    const int* slot_map;
    bf16* k_cache;
    bf16* v_cache;
    const float* inv_freq;
    int page_size;
    long long page_stride, head_stride, pool_slots;
    int* status;
    int RB, KS;
    int use_pdl;
    union {
        int stage_norm;          // gemm_skinny.cu: the norm prologue's input comes through one bulk copy into shared memory
        int give_up;             // gemm_stream.cu, for tests (EPI_F32 of plain rows): every wait inside the kernel gives up at once
    };
    int norm_mode;               // 1: add + norm here; 2: prenormed rows (delta = xn) and partial sums (ss_in)
    const float* ss_in;          // [ss_parts][padded tokens] partial sums of squares, prenormed prologue
    int ss_parts;
    float* resid_inout;          // resid_norm epilogue: the residual, updated in place
    const float* gain_out;       //   the following norm's gain
    bf16* xn_out;                //   bfloat16(gain_out * v) [M, N]
    float* ss_out;               //   [gridDim.x][padded tokens]
    // EPI_STORE with an activation on the way out: act 1: act(z) = act_a z^2 + z / 2 for z > 0, act_b (e^z - 1 - z) + z / 2
    // below; act 2: act(z) = max(z, 0)^2; act 4: the exact gelu.  EPI_SWIGLU with act 3: g = min(gate, act_a), u = clamp(up, -act_a, act_a),
    // out = g sigmoid(1.702 g) (u + 1)
    int act;
    float act_a, act_b;
    const void* prefetch;        // weights of a kernel that runs soon: pulled into L2 meanwhile
    long long prefetch_bytes;
    float* scratch;              // [gridDim.y][gridDim.x][RB*16][tokens] partial sums when K is cut across CTAs
    int* counters;               // [gridDim.x] tickets, zero before and after every launch
    unsigned long long* trace;   // optional: [2] earliest start / latest end of this launch's CTAs (%globaltimer, ns)
    int parts_offset;            // where in shared memory the cluster's parts arrive (bytes)
    int cluster_reduce;          // the gridDim.y CTAs of a row group are one cluster and sum their parts through the first one's shared memory
};

}  // namespace skinny

// gemm_stream.cu: launches the product if its kernel takes these sizes.  Returns -1 if it does not, else a cudaError_t.
int eg_gemm_stream_launch(cudaStream_t stream, int epilogue, int norm, const skinny::Params& p);
