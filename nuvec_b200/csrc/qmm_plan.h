// How the many-row products are cut (host side, and the device's share of it): the token tile, whether blocks work in pairs, and
// the schedule of the tiles.  No CUDA in here but the marks of functions that the kernel calls too.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define QMM_BOTH __host__ __device__
#else
#define QMM_BOTH
#endif

namespace nvc {

constexpr int QMM_BN = 128;  // weight rows per tile (UMMA M)
constexpr int QMM_BK = 64;   // k-values per block: one 128-byte swizzle row of bfloat16

// The schedule.  Every worker (block, or pair of blocks) first takes `full_waves` whole tiles (tile = worker + wave *
// workers).  The tiles left over (fewer than workers) are cut along K into `splits` parts of whole grains of k-blocks,
// dealt over the workers in `tail_rounds` rounds, so that the last wave -- or a product with fewer tiles than
// multiprocessors -- still keeps every multiprocessor busy.  Parts leave float32 partial tiles in scratch; the block that
// arrives last adds them in part order and writes the result.
struct Schedule {
    int32_t full_waves, tail_tiles, splits, tail_rounds;
};
// What the plan is weighed with, in ns: a worker's pace per 64-k block with tiles of BT tokens, and the price of cutting a tile
// (a part's way through scratch and the arrival, then the addition, which reads every part at about 100 bytes per ns).
// Measured over 16 shapes between 24 and 2048 rows: up to 128 tokens the dequantization sets the pace, from 256 on the MMAs;
// 160 and 192 have smaller stages.  More bits per code take longer to unpack.
QMM_BOTH constexpr float qmm_block_ns(int bt, bool pair, int bits) {
    return (bt <= 64 ? 220.0f : bt <= 128 ? 255.0f : bt <= 160 ? 315.0f : bt <= 192 ? 340.0f : pair ? 420.0f : 450.0f) *
           (bits == 2 || bits == 4 ? 1.0f : bt <= 192 ? 1.15f : 1.08f);
}
// tokens: of a tile, at most.  *ns: the plan's expected duration.
QMM_BOTH inline Schedule make_schedule(int tiles, int workers, int kblocks, int grain, int tokens, float block_ns, float *ns) {
    Schedule c{tiles / workers, tiles % workers, 1, 1};
    const int grains = (kblocks + grain - 1) / grain;
    float tail = 0.0f;
    if (c.tail_tiles > 0) {
        // Parts per tile: whatever makes the left-over tiles finish soonest when the parts are dealt over the workers in one or
        // two rounds; at least two grains of k-blocks per part, at most 16 parts.
        tail = (float)kblocks * block_ns;
        for (int s = 2; s <= 16 && s <= grains / 2; s++) {
            const int rounds = (c.tail_tiles * s + workers - 1) / workers;
            if (rounds > 2) break;
            const float cost = (float)(rounds * ((grains + s - 1) / s) * grain) * block_ns + 2000.0f + 5.0f * (float)(rounds * s * tokens);
            if (cost < tail) {
                tail = cost;
                c.splits = s;
            }
        }
        c.tail_rounds = (c.tail_tiles * c.splits + workers - 1) / workers;
    }
    *ns = (float)c.full_waves * (float)kblocks * block_ns + tail;
    return c;
}

// The token tile (and whether blocks work in pairs): whichever plan is expected to finish soonest.  A fixed rule on the rows
// missed by up to 1.6 (219 x 4096 x 11008: 256 tokens 45 us, 128 tokens 27): how the tiles fill the last wave matters as
// much as a tile's own pace.  Experts' rows scatter around their average: the plan is weighed with the tiles that an
// average of six counts up to 2.25 standard deviations of a random routing away needs.  Grouped products do not pair: an
// expert's last token tile is rarely full and twice as many tiles balance better (32 experts x 2880 x 2880, 128 rows each:
// 105 us with pairs, 96 without).
struct QmmPlan {
    int bt;
    bool pair;
};
inline QmmPlan qmm_plan(int64_t rows, int64_t experts /* 0: not grouped */, int64_t N, int kblocks, int bits, int sms) {
    static const QmmPlan plans[] = {{32, false}, {64, false}, {128, false}, {160, false}, {192, false}, {256, false}, {256, true}};
    QmmPlan chosen = plans[0];
    float best = INFINITY;
    for (const QmmPlan &plan : plans) {
        if (plan.pair && experts) continue;
        const int rows_per_tile = plan.pair ? 2 * QMM_BN : QMM_BN;
        const int64_t n_tiles = (N + rows_per_tile - 1) / rows_per_tile;
        float tok_tiles = (float)((rows + plan.bt - 1) / plan.bt);
        if (experts) {
            const float per = (float)rows / (float)experts, sd = sqrtf(per);
            tok_tiles = 0.0f;
            for (int z = -5; z <= 5; z += 2) tok_tiles += ceilf(fmaxf(per + 0.45f * (float)z * sd, 0.0f) / (float)plan.bt) / 6.0f;
            tok_tiles *= (float)experts;
        }
        const float tiles = fminf(tok_tiles * (float)n_tiles, 1e9f);
        float ns;
        make_schedule((int)(tiles + 0.5f), plan.pair ? sms / 2 : sms, kblocks, 4, plan.bt < rows ? plan.bt : (int)rows, qmm_block_ns(plan.bt, plan.pair, bits), &ns);
        if (ns < best) {
            best = ns;
            chosen = plan;
        }
    }
    return chosen;
}

}  // namespace nvc
