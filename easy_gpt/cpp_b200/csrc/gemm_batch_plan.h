// Which products gemm_batch.cu takes and how it shares them out, from the sizes alone (host code, no CUDA).
#pragma once

namespace batch_plan {

constexpr int BK = 64;                          // terms of a stage: a row of 128 bytes
constexpr int MAX_STAGES = 16, SMS = 148, SHARED = 110 * 1024;
constexpr int LEAST_TOKENS = 17, MOST_TOKENS = 64;
enum Kind { SWIGLU, INTO_RESIDUAL, QKV };

struct Cut {
    int columns;                                // of a tile
    int split;                                  // CTAs (a cluster) that share a tile's K
};

// As many CTAs as have an SM each (at least about 100 where K is long enough for two stages a CTA), at most two an SM: one wave.
inline bool cut_for(Kind kind, int N, int K, int head_dim, Cut* out) {
    if (N < 64 || K < BK || K % BK) return false;
    Cut c{64, 1};
    if (kind == QKV) {
        if (head_dim != 64 && head_dim != 128) return false;          // a tile is a head
        c.columns = head_dim;
    }
    if (N % c.columns) return false;
    const int tiles = N / c.columns, chunks = K / BK;
    // SwiGLU's tiles are many; the others own 8 or 16 of a tile's columns, QKV's a share of its pairs in pieces of four at least
    const int least = kind == SWIGLU ? 1 : 4, most = kind == SWIGLU ? 2 : 8;
    c.split = least;
    while (c.split < most && tiles * c.split * 2 <= 2 * SMS && (tiles * c.split < 100 || tiles * c.split * 2 <= SMS) && chunks >= c.split * 4) c.split *= 2;
    if (chunks < c.split || tiles * c.split > 2 * SMS) return false;
    // clusters of 4 and 8 that find room with two CTAs an SM (gemm_stream_plan.h)
    if ((c.split == 4 && tiles > 71) || (c.split == 8 && tiles > 33)) return false;
    *out = c;
    return true;
}

}  // namespace batch_plan
