// How gemm_stream.cu's kernel shares a product out, from the sizes alone (host code, no CUDA): whether it takes the product and the
// order of its sums (row blocks a unit, slices and parts of K) from the epilogue, N and K, for 1 to 16 tokens alike; only the depth of
// the ring and how many CTAs share an SM hang off the token tile.
#pragma once

namespace stream_plan {

constexpr int WARPS = 8;                      // that multiply
constexpr int MAX_STAGES = 16;
constexpr int STAGE_BYTES = WARPS * 2048;     // a tile of 16 rows x 64 terms a warp
constexpr int RED_LD = 20;                    // a token's 16 row sums: stores and loads of the warps' sums meet no bank twice
constexpr int SMS = 148;                      // a constant, so that results do not hang off the GPU
constexpr int WIDE_BLOCKS = 400;              // row blocks from which on CTAs read all of K
constexpr int MOST_SHARED = 220 * 1024, HALF_SHARED = 110 * 1024;
constexpr int MOST_TOKENS = 16;

// Clusters of 1, 2, 4 and 8 CTAs that find room on a B200 together, with one CTA an SM and with two (measured with
// cudaOccupancyMaxActiveClusters; the rest would run as a second wave).  Constants, for the same reason as SMS.
constexpr int CLUSTERS[2][4] = {{148, 74, 33, 15}, {296, 148, 71, 33}};

struct Cut {
    int rb_log;                               // log2 of a unit's row blocks of 16; the other factor of WARPS are slices of K
    int split;                                // CTAs (a cluster) that share a unit's K, k_len terms each
    int k_len, k_stages;
    int units;
};

struct Ring {
    int per_sm;                               // CTAs an SM
    int stages;                               // 0: the product does not fit
    int grid, share, longer;                  // CTAs (clusters) in x; row blocks of a CTA that walks, 0: every CTA has one unit
    int x_bytes, red_bytes, parts_bytes;
};

inline Cut cut_of(int N, int K, bool pairs, int rb_log, int split) {
    Cut c{};
    const int blocks = (N + 15) / 16;
    c.rb_log = rb_log;
    c.units = pairs ? blocks / 2 : (blocks + (1 << rb_log) - 1) >> rb_log;
    c.k_len = ((K + split - 1) / split + 63) / 64 * 64;
    c.split = (K + c.k_len - 1) / c.k_len;
    const int slices = WARPS >> rb_log;
    c.k_stages = (c.k_len + slices * 64 - 1) / (slices * 64);
    return c;
}

// pairs: the epilogue that rotates pairs of row blocks; walks: units may be shared out in a row (EPI_RESID_NORM's may not).
inline Ring ring_of(const Cut& c, int N, int token_tile, bool walks) {
    Ring r{};
    const int rows = 16 << c.rb_log, blocks = (N + 15) / 16;
    r.x_bytes = token_tile * (c.k_len * 2 + 16);
    r.red_bytes = WARPS * token_tile * RED_LD * 4;
    r.parts_bytes = c.split > 1 ? (c.split - 1) * rows * token_tile * 4 : 0;
    const int rest = r.x_bytes + r.red_bytes + r.parts_bytes + 1024 + 64;
    // two CTAs an SM (or this one and the next kernel's) unless x alone is more than half of that (16 tokens at the 1.5B sizes:
    // 1,329 us a step with two, 1,463 with one)
    // ... and unless each CTA can have an SM of its own and a long walk that a ring of two or three stages would not cover (us a decode
    // step of one and 8 requests, with two / with one: 8 layers of the 3B sizes, down product in 4 parts, 494 / 487 and 520 / 516; 6
    // of 7B, QKV, 775 / 757 and 866 / 858)
    const bool lone = c.units * c.split <= SMS && c.k_stages >= 12 && (HALF_SHARED - rest) / STAGE_BYTES < 4;
    for (r.per_sm = rest <= 80 * 1024 && !lone ? 2 : 1; r.per_sm >= 1; --r.per_sm) {
        r.grid = c.units;
        r.share = r.longer = 0;
        int most = c.k_stages;
        if (walks && c.split == 1 && c.units > r.per_sm * SMS) {
            r.grid = r.per_sm * SMS;
            r.share = blocks / r.grid;
            r.longer = blocks % r.grid;
            most = c.k_stages * ((r.share + (1 << c.rb_log)) >> c.rb_log);
        }
        r.stages = ((r.per_sm == 2 ? HALF_SHARED : MOST_SHARED) - rest) / STAGE_BYTES;
        if (r.stages > MAX_STAGES) r.stages = MAX_STAGES;
        if (r.stages > most) r.stages = most;
        const int fits = CLUSTERS[r.per_sm - 1][c.split <= 1 ? 0 : c.split <= 2 ? 1 : c.split <= 4 ? 2 : 3];
        if (r.stages >= (most > 1 ? 2 : 1) && (c.split == 1 || c.units <= fits)) return r;
    }
    r.stages = 0;
    return r;
}

// Whether the kernel takes the product at every number of tokens, and its cut.  (Measured on B200, us a decode step of 8 tokens at
// the 0.5B sizes / of 4 at the 1.5B sizes.)
inline bool cut_for(int N, int K, bool pairs, bool walks, Cut* out) {
    const int blocks = (N + 15) / 16;
    if (N < 1 || K < 16) return false;
    auto fits = [&](int rb_log, int split) {
        *out = cut_of(N, K, pairs, rb_log, split);
        return ring_of(*out, N, 8, walks).stages > 0 && ring_of(*out, N, MOST_TOKENS, walks).stages > 0;
    };
    if (pairs) {
        // a unit is 32 rows; its K is cut where that leaves a CTA 768 terms (0.5B, K 896: cut in two 591, whole 586; 1.5B,
        // K 1536: 1,110 and 1,147)
        int split = 1;
        while (split < 8 && blocks * split <= SMS && K >= 768 * split * 2) split *= 2;
        return fits(1, split);
    }
    if (blocks >= WIDE_BLOCKS) return fits(2, 1);                  // (units of 128 rows: 620 / 1,155 against 623 / 1,078)
    // As many CTAs as SMs: one each leaves room for the next kernel's (down product, 56 row blocks x 4,864: 112 CTAs 597,
    // 224 CTAs 623).  Two an SM where one would have more than about 128 KB to read (1.5B: 96 CTAs 1,110, 192 CTAs 1,036),
    // if the token tile of 16 fits twice and all clusters find room, else one.
    // A CTA keeps 1,024 terms at least (K 896 cut in two: 575 against 562 for one token); of equal splits the one
    // with the most rows a unit, since every CTA reads its range of x.  Powers of two: clusters of 5 and 6 do not all
    // find room together.
    for (int per_sm = (long long)N * K * 2 > SMS * (128LL << 10) ? 2 : 1; per_sm >= 1; --per_sm) {
        const long long most = (long long)per_sm * SMS;
        long long best = -1;
        int rb_log = 0, split = 1;
        for (int rb = 0; rb <= 2; ++rb) {
            const int u = (blocks + (1 << rb) - 1) >> rb;
            int cut = 1;
            while (cut < 8 && (long long)u * cut * 2 <= most && K >= 1024 * cut * 2) cut *= 2;
            const long long ctas = u * cut > most ? 2 * most - u * cut : u * cut;
            if (ctas >= best && (rb == 0 || cut > 1)) {
                best = ctas;
                rb_log = rb;
                split = cut;
            }
        }
        if (fits(rb_log, split)) return true;
    }
    return false;
}

}  // namespace stream_plan
