// Many-row quantized products on the 5th-generation tensor cores (tcgen05), for prefill and
// for the grouped (sorted) mixture-of-experts product:
//
//     y[tok, n] = sum_k x[tok, k] * dequantize(w)[n, k]         (weights stored [N, K], "transposed")
//
// One persistent block per multiprocessor walks output tiles of 128 weight rows x BT tokens.
// The weight tile is the UMMA "A" operand (M = 128), the activations the "B" operand (N = BT):
// the accumulator D[128 x BT] (float32) lives in tensor memory, each dequantized weight is reused
// by BT tokens, and a group of few tokens (an expert with 32 rows) still fills all 128 lanes.
//
// The ring.  A stage is SUB blocks of 64 k-values: the activations' tile in shared memory (the MMA's B operand, 128-byte
// swizzle, TMA) and the dequantized weights in tensor memory (its A operand).  Packed weights and their scales have a ring
// of their own, in slabs of KPS k-blocks, so that their latency is never behind the activation stages.
//
// Warp roles (896 threads):
//   warps 0-3   epilogue: tcgen05.ld the finished accumulator, round to the 16-bit type, store y
//   warp  4     TMA producer of activation tiles
//   warp  6     TMA producer of packed weight slabs
//   warps 24-27 producers of scales and biases (cp.async, a row per lane), in chunks of 512 k-values on a ring of their own:
//               every copy instruction touches 32 rows = 32 cache lines and holds the load unit that long, so the fewer and
//               wider the better (copying them per 128 k-values, 4 bytes a row: 71 instead of 60 us for 128 experts x 768 x 2048)
//   warps 7-22  dequantizers (four groups of four warps take stages in turn; thread = weight row = tensor-memory lane):
//               packed codes -> 16-bit values in registers, with exactly the reference's two roundings
//               (crates/nuvec-core/src/kernels.rs:835-859), so the tensor-core operands are bit-identical to the reference's
//               dequantized matrix -> tcgen05.st into the stage.  Dequantized weights never pass through shared memory.
//               They read their scales from shared memory: loads of two bytes from 32 rows are 32 cache lines each, and four
//               of them per thread and k-block kept the load unit busy for most of a k-block's time when every thread
//               fetched its own from global memory (128 experts x 768 x 2048, 32 rows each: 80 us, 62 us since)
//   warp  5     MMA issuer: 4 x tcgen05.mma.kind::f16 (K = 16, A from tensor memory) per 64-k
//               block; tcgen05.commit releases the stage / publishes the accumulator.  It waits
//               on hardware named barriers only
//   warp  23    watcher: waits on the mbarriers for the MMA warp and hands each full stage over
//               through a named barrier
// Tensor memory (512 columns): one or two accumulators of BT columns, then the weight ring of 32 columns per k-block.
// Two accumulator buffers in tensor memory let the epilogue of one tile overlap the main loop
// of the next.  All waits are bounded: a wait that gives up raises an abort flag that every
// other wait observes, the block frees its tensor memory and returns, and the host reports the
// failure at the next synchronisation.
//
// Reference behaviour covered: MLX/nuvec's qmm_t, qmm_t_splitk, nax qmm_t and gather_qmm_rhs
// kernels (crates/nuvec-kernels/src/metal/quantized.h:1358-1485, 2388-2519, 3301-3449;
// nax/quantized.metal); CPU result crates/nuvec-core/src/kernels.rs:1091-1142 and, for the
// gather, crates/nuvec-core/src/quantized.rs:679-719.
#pragma once
#include "qmm.cuh"
#include "qmm_plan.h"
#include "tcgen05.cuh"

namespace nvc {

// ── optional role timing (diagnostic builds only: -DNUVEC_TIMELINE) ─────────────────────────
// Every role of blocks 0 and 1 adds up the clock cycles it spends inside each of its waits (and
// in total); nvc_debug_qmm_timing (qmm_bf16.cu) fetches the sums of the last bfloat16 launch.
#ifdef NUVEC_TIMELINE
constexpr int QT_ROLES = 8, QT_SLOTS = 6;
static __device__ long long g_qmm_timing[2][QT_ROLES][QT_SLOTS];
#define QT_BEGIN long long qt_[QT_SLOTS] = {0, 0, 0, 0, 0, 0}; const long long qt_start_ = clock64();
#define QT(k, ...) { const long long qt_t_ = clock64(); __VA_ARGS__; qt_[k] += clock64() - qt_t_; }
#define QT_END(role, writer)                                                        \
    if (blockIdx.x < 2 && (writer)) {                                               \
        qt_[0] = clock64() - qt_start_;                                             \
        for (int q_ = 0; q_ < QT_SLOTS; q_++) g_qmm_timing[blockIdx.x][role][q_] = qt_[q_]; \
    }
#else
#define QT_BEGIN
#define QT(k, ...) { __VA_ARGS__; }
#define QT_END(role, writer)
#endif

constexpr int QMM_EPI_WARPS = 4, QMM_DQ_WARPS = 16, QMM_DQ_GROUPS = 4;  // dequantizers: groups of 4 warps
constexpr uint32_t QMM_EPI_BARRIER = 9;  // named barrier of the epilogue warps (1 .. 8 belong to the stages)
constexpr int QMM_WATCH_WARP = QMM_EPI_WARPS + 3 + QMM_DQ_WARPS;  // the warp that waits on behalf of the MMA warp
constexpr int QMM_SCALE_WARP = QMM_WATCH_WARP + 1;  // this and the three after it load scales
constexpr int QMM_CHUNK = 8;                        // k-blocks whose scales travel together
constexpr int QMM_S_STAGES_MAX = 4;                 // chunks in flight, as the groups' size allows
constexpr int QMM_THREADS = (QMM_SCALE_WARP + 4) * 32;
constexpr int QMM_TABLE_BYTES = 4112;        // the grouped products' tables: 2 x (512 + 1) ints, rounded up to 16 bytes
constexpr int QMM_ITEMS = 64;                // a worker's first items, worked out once per block (see QmmWork)
constexpr int QMM_ITEM_BYTES = QMM_ITEMS * 32;
constexpr int QMM_EPI_STAGE_BYTES = 4 * 2048;  // epilogue: 32 tokens x 32 weight rows of bfloat16 per warp

struct QmmKernelParams {
    const uint8_t *scales, *biases;   // [weight rows, K / gs]: 16-bit values, or one byte each (mxfp4 / mxfp8 / nvfp4, no biases)
    const float *global;              // nvfp4 global scale(s) or nullptr
    uint16_t *y;                      // [rows, N], 16-bit values
    const int32_t *offsets;           // grouped: first row of each expert, else nullptr
    int32_t *error;                   // host-visible word: nonzero when a wait gave up
    float *partials;                  // [tail tiles][splits][BT tokens][128 rows] float32 (K-split tiles)
    uint32_t *counters;               // [tail tiles] arrivals, zero on entry and on exit
    Schedule sched;                   // of ungrouped products; grouped ones make theirs when they know the experts' rows
    int32_t experts, rows, N, K;
    int32_t gs_shift, scale_row_bytes, expert_global;
    // A chunk's scales in shared memory: `chunk_bytes` of every row (s_pitch apart) in copies of s_vec bytes (16, 8, 4); rows
    // that are not 4-byte aligned are copied as the aligned words around them.  s_stages chunks fit the area.
    int32_t chunk_bytes, s_pitch, s_vec, s_stages;
    int32_t early;                    // 1: nothing in flight writes the weights, they may be read before the wait for the previous kernel; 0: all wait first
};

// Instruction descriptor: D = f32, A = B = bf16 (or f16), both K-major, M = m, N = n.
__host__ __device__ constexpr uint32_t umma_idesc(int n, bool f16, int m) {
    return (1u << 4) | (f16 ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ uint32_t q_lop3(uint32_t a, uint32_t mask, uint32_t orv) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(orv));
    return r;
}
__device__ __forceinline__ uint32_t q_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint32_t q_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// a + b as fma(a, 1, b): the same single rounding on the full-rate pipe (the packed bfloat16 addition issues at a quarter of it)
__device__ __forceinline__ uint32_t q_add(uint32_t a, uint32_t b) { return q_fma(a, 0x3F803F80u, b); }
__device__ __forceinline__ uint32_t q_mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h_add(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h_mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// ── dequantization of 64 k-values of one weight row ────────────────────────────────────────
// Affine, reference arithmetic: p = rn(code * scale), w = rn(p + bias), both in the 16-bit type.
// bfloat16: codes enter as the number 128 + code (code bits ORed into the mantissa of 128.0);
// fma(128 + c, s, -128 s) is the single rounding of the exact product c * s.
// float16: 1024 + code, the 1024 taken out first (-1024 s could overflow).
template <bool F16> struct Affine {
    static constexpr uint32_t MAGIC = 0x43004300u;
    uint32_t s2, ns2, b2;
    __device__ __forceinline__ void set(uint32_t s, uint32_t b) {
        s2 = s * 0x10001u;
        b2 = b * 0x10001u;
        ns2 = q_mul(s2, 0xC300C300u);  // -128 s, exact
    }
    __device__ __forceinline__ uint32_t finish(uint32_t m) const { return q_add(q_fma(m, s2, ns2), b2); }
};
template <> struct Affine<true> {
    static constexpr uint32_t MAGIC = 0x64006400u;
    uint32_t s2, b2;
    __device__ __forceinline__ void set(uint32_t s, uint32_t b) {
        s2 = s * 0x10001u;
        b2 = b * 0x10001u;
    }
    __device__ __forceinline__ uint32_t finish(uint32_t m) const { return h_add(h_mul(h_add(m, 0xE400E400u), s2), b2); }
};
// 4 bits: word = 8 codes.  a = w, b = w >> 4: byte j of a has code 2j in its low nibble, byte j of
// b has code 2j+1 there; prmt gathers the two bytes into the two halves, lop3 masks and ORs the magic number.
template <bool F16> __device__ __forceinline__ void dequant_word4(uint32_t w, const Affine<F16> &q, uint32_t *o) {
    const uint32_t b = w >> 4;
#pragma unroll
    for (int j = 0; j < 4; j++)  // selector: result byte 0 <- a.byte j, result byte 2 <- b.byte j (bytes 1 and 3 are masked away)
        o[j] = q.finish(q_lop3(q_prmt(w, b, 0x0400u + 0x0101u * (uint32_t)j), 0x000F000Fu, Affine<F16>::MAGIC));
}
// 8 bits.  bfloat16: the low seven bits as 128 + (c & 127); where bit 7 is set that is c itself, elsewhere the 128 leaves
// with -128 s in the same fma: one rounding of c * s either way.  A byte permutation that repeats sign bits makes the
// mask, one more operation applies it: 6 instructions per pair of codes where rebuilding the byte from its nibbles took 8.
// float16: a byte of 0x64 above the code is 1024 + code.
template <bool F16> __device__ __forceinline__ void dequant_word8(uint32_t w, const Affine<F16> &q, uint32_t *o) {
    if constexpr (F16) {
        o[0] = q.finish(q_prmt(w, 0x64646464u, 0x4140u));
        o[1] = q.finish(q_prmt(w, 0x64646464u, 0x4342u));
    } else {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t m = q_lop3(q_prmt(w, w, j ? 0x0302u : 0x0100u), 0x007F007Fu, 0x43004300u);
            const uint32_t off = ~q_prmt(w, w, j ? 0xBBAAu : 0x9988u) & q.ns2;
            o[j] = q_add(q_fma(m, q.s2, off), q.b2);
        }
    }
}
// 32 bits of three words' bit stream from bit `pos` on (a compile-time position once unrolled)
__device__ __forceinline__ uint32_t q_window(const uint32_t *u, int pos) {
    const int idx = pos >> 5, sh = pos & 31;
    if (sh == 0) return u[idx];
    return idx + 1 < 3 ? __funnelshift_r(u[idx], u[idx + 1], sh) : u[idx] >> sh;
}
// 3 and 6 bits: three words = 32 or 16 codes; a pair of codes is 2 * BITS consecutive bits, spread over the two halves.
template <int BITS, bool F16> __device__ __forceinline__ void dequant_words3(const uint32_t *u, const Affine<F16> &q, uint32_t *o) {
    constexpr uint32_t MASK = (1u << BITS) - 1u;
#pragma unroll
    for (int j = 0; j < 48 / BITS; j++) {
        const uint32_t v = q_window(u, 2 * BITS * j);
        o[j] = q.finish(q_lop3(v << (16 - BITS), MASK << 16, q_lop3(v, MASK, Affine<F16>::MAGIC)));
    }
}
// 2 bits: word = 16 codes; codes 2j, 2j+1 sit in bits [4j, 4j+4).
template <bool F16> __device__ __forceinline__ void dequant_word2(uint32_t w, const Affine<F16> &q, uint32_t *o) {
    const uint32_t b = w >> 2;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        // byte j/2 holds codes 4(j/2) .. 4(j/2)+3; pair j = codes (2j, 2j+1): shift the byte pair by 4 (j odd)
        uint32_t t = q_prmt(w, b, 0x0400u + 0x0101u * (uint32_t)(j >> 1));
        if (j & 1) t >>= 4;
        o[j] = q.finish(q_lop3(t, 0x00030003u, Affine<F16>::MAGIC));
    }
}

// E2M1 code pairs -> bfloat16 pairs times the group scale.  A byte permutation is an eight-entry table look-up for
// four codes at a time: the codes' magnitude bits select the high and the low byte of the bfloat16 magnitudes
// 0, .5, 1, 1.5, 2, 3, 4, 6; the signs join from the code's fourth bit.  The product with the scale (a power of two, or
// an E4M3 number with 4 significant bits) is exact: at most 6 significant bits.  It equals the reference's float32 value
// scale * code (crates/nuvec-core/src/kernels.rs:976-1009).
__device__ __forceinline__ void dequant_word_fp4(uint32_t w, uint32_t scale2, uint32_t *o) {
    const uint32_t even = w << 4;  // byte j: the sign of code 2j on top; in w itself that of code 2j + 1
    const uint32_t m = w & 0x77777777u;
#pragma unroll
    for (int q = 0; q < 2; q++) {  // codes 4q .. 4q + 3
        const uint32_t sel = q ? m >> 16 : m;
        const uint32_t hi = q_prmt(0x3F3F3F00u, 0x40404040u, sel), lo = q_prmt(0xC0800000u, 0xC0804000u, sel);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t mag = q_prmt(lo, hi, j ? 0x7362u : 0x5140u);
            const uint32_t sgn = q_prmt(even, w, j ? (q ? 0x7030u : 0x5010u) : (q ? 0x6020u : 0x4000u));  // bytes 1 and 3
            o[2 * q + j] = q_mul(q_lop3(sgn, 0x80008000u, mag), scale2);
        }
    }
}
// 8-bit floating point (mxfp8: E4M3 codes): the code's seven magnitude bits become exponent[3:0] and mantissa[6:4] of
// a bfloat16 (the value * 2^-120, subnormal codes as bfloat16 subnormals); times 2^120 and the scale (a power of two)
// it is the reference's float32 decode exactly.  The two NaN codes, which the reference's quantizer never writes, read
// as 480.  Halves: codes (0, 1) and (2, 3).
__device__ __forceinline__ void dequant_word_fp8(uint32_t w, uint32_t scale2, uint32_t *o) {
    {
        const uint32_t x = q_prmt(w, w, 0x0100u);  // bytes 0, 1 in the low byte of each half
        o[0] = q_mul(q_mul(q_lop3(x << 8, 0x80008000u, (x << 4) & 0x07F007F0u), 0x7B807B80u), scale2);
    }
    {
        const uint32_t x = q_prmt(w, w, 0x0302u);  // bytes 2, 3
        o[1] = q_mul(q_mul(q_lop3(x << 8, 0x80008000u, (x << 4) & 0x07F007F0u), 0x7B807B80u), scale2);
    }
}
// bfloat16 pair {s, s} of a scale code: E8M0 (2^(code - 127); code 0 decodes to a float32 subnormal
// that the reference flushes to zero) or E4M3.
__device__ __forceinline__ uint32_t fp_scale2(uint32_t code, bool e8m0) {
    uint32_t h;
    if (e8m0) h = code == 0u ? 0u : (code << 7);
    else h = __float_as_uint(ftz(e4m3_to_f32(code))) >> 16;
    return (h & 0xFFFFu) * 0x10001u;
}

// Tile bookkeeping shared by the roles.
struct TileInfo {
    int n0;        // first weight row of the tile inside its matrix
    int wrow0;     // first row in the stacked [experts * N] weight / scale arrays
    int tok0;      // first token row of the tile
    int tok_end;   // tokens at or past this row are not stored
    int expert;
};

// Grouped products: the experts' first rows and the number of token tiles before each expert, kept
// in shared memory (filled once per block), so that finding a tile's expert is a binary search in
// shared memory and not a walk over global memory by every role at every tile.
constexpr int QMM_MAX_TABLE_EXPERTS = 512;
struct GroupTable {
    const int *off;    // [experts + 1] first row of each expert, then the row count; nullptr: no table
    const int *tiles;  // [experts + 1] token tiles before each expert, then the total
};

// `half`: the block's rank in a pair (a pair's tiles are 2 x 128 weight rows), 0 without pairs.
template <int BT, bool PAIR>
__device__ __forceinline__ bool tile_info(const QmmKernelParams &p, const GroupTable &gt, int tile, int n_tiles, TileInfo &ti, int half) {
    const int nt = tile % n_tiles, j = tile / n_tiles;
    ti.n0 = (PAIR ? 2 * nt + half : nt) * QMM_BN;
    if (!p.offsets) {
        ti.expert = 0;
        ti.wrow0 = ti.n0;
        ti.tok0 = j * BT;
        ti.tok_end = p.rows;
        return ti.tok0 < p.rows;
    }
    if (gt.off) {
        if (j >= gt.tiles[p.experts]) return false;
        int lo = 0, hi = p.experts;  // the expert e with tiles[e] <= j < tiles[e + 1]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (gt.tiles[mid] <= j) lo = mid; else hi = mid;
        }
        ti.expert = lo;
        ti.wrow0 = lo * p.N + ti.n0;
        ti.tok0 = gt.off[lo] + (j - gt.tiles[lo]) * BT;
        ti.tok_end = gt.off[lo + 1];
        return true;
    }
    // grouped: token tile j of the concatenation of every expert's tiles
    int seen = 0;
    for (int e = 0; e < p.experts; e++) {
        const int lo = p.offsets[e], hi = e + 1 < p.experts ? p.offsets[e + 1] : p.rows;
        const int tiles_e = (hi - lo + BT - 1) / BT;
        if (j < seen + tiles_e) {
            ti.expert = e;
            ti.wrow0 = e * p.N + ti.n0;
            ti.tok0 = lo + (j - seen) * BT;
            ti.tok_end = hi;
            return true;
        }
        seen += tiles_e;
    }
    return false;
}

// One piece of a worker's share of the schedule.
struct Item {
    int tile, kb0, kb1;  // k-blocks [kb0, kb1) of this tile
    int part, parts, slot;
    int round;           // which of the worker's (at most two) parts of left-over tiles this is
};
template <int GRAIN>
__device__ __forceinline__ bool qmm_item(const Schedule &c, int kblocks, int j, Item &it, int worker, int workers) {
    if (j < c.full_waves) {
        it.tile = worker + j * workers;
        it.kb0 = 0; it.kb1 = kblocks; it.part = 0; it.parts = 1; it.slot = 0; it.round = 0;
        return true;
    }
    it.round = j - c.full_waves;
    const int pi = worker + it.round * workers;
    if (it.round >= c.tail_rounds || pi >= c.tail_tiles * c.splits) return false;
    it.slot = pi / c.splits;
    it.part = pi % c.splits;
    it.parts = c.splits;
    it.tile = c.full_waves * workers + it.slot;
    const int grains = (kblocks + GRAIN - 1) / GRAIN;  // (splits <= grains: no part is empty)
    it.kb0 = grains * it.part / c.splits * GRAIN;
    it.kb1 = min(grains * (it.part + 1) / c.splits * GRAIN, kblocks);
    return true;
}

// A worker's items, for its roles.  Finding an item (divisions, the search for the tile's expert) takes a warp 800 to 1700
// cycles beside the dequantizers, and every role needs every item: a fifth of the dequantizers' time with tiles of 12
// k-blocks.  So the first QMM_ITEMS are worked out once, a thread per item, and the roles read them from shared memory; only a
// worker with more computes the others as they come.
enum { QMM_END = 0, QMM_TAKE = 1, QMM_SKIP = 2 };
template <int BT, int GRAIN, bool PAIR> struct QmmWork {
    const QmmKernelParams &p;
    const Schedule &sched;
    const GroupTable &gt;
    int4 *list;  // [QMM_ITEMS][2]
    int kblocks, n_tiles, worker, workers, half;

    __device__ __forceinline__ int find(int j, Item &it, TileInfo &ti) const {
        if (!qmm_item<GRAIN>(sched, kblocks, j, it, worker, workers)) return QMM_END;
        return tile_info<BT, PAIR>(p, gt, it.tile, n_tiles, ti, half) ? QMM_TAKE : QMM_SKIP;
    }
    __device__ __forceinline__ void fill(int j) const {
        Item it{};
        TileInfo ti{};
        const int what = find(j, it, ti);
        list[2 * j] = make_int4(it.kb0, it.kb1, ti.tok0, ti.wrow0);
        list[2 * j + 1] = make_int4(ti.n0, ti.tok_end, ti.expert, what | it.part << 2 | it.parts << 7 | it.round << 12 | it.slot << 13);
    }
    __device__ __forceinline__ int operator()(int j, Item &it, TileInfo &ti) const {
        if (j >= QMM_ITEMS) return find(j, it, ti);
        const int4 a = list[2 * j], b = list[2 * j + 1];
        it.kb0 = a.x;
        it.kb1 = a.y;
        ti.tok0 = a.z;
        ti.wrow0 = a.w;
        ti.n0 = b.x;
        ti.tok_end = b.y;
        ti.expert = b.z;
        it.part = b.w >> 2 & 31;
        it.parts = b.w >> 7 & 31;
        it.round = b.w >> 12 & 1;
        it.slot = b.w >> 13;
        return b.w & 3;
    }
};

// Shared memory and tensor memory of an instantiation.
//
// SUB: 64-k blocks per stage.  Two halve the hand-overs wherever four such stages fit: tiles of up to 128 tokens, whose MMAs
// are short, and pairs, each of whose blocks keeps half of the activations (8-bit weights, 8192 x 12288 x 4096: 619 -> 590 us;
// 4 bits unchanged).  A slab of packed weights is then exactly a stage, read and released by the group of warps that owns the
// stage (OWNED); otherwise it serves several stages (128 or 96 bytes of a row) and all groups.
//
// Accumulators: two (the epilogue of one tile overlaps the main loop of the next) while they leave four stages for the
// weight ring; the widest tile keeps a single one.
//
// PAIR: two blocks of a cluster (cta_group::2) share a tile of 2 x 128 weight rows x BT tokens; each keeps half of the
// tokens' activations in its shared memory and its own rows' weights and accumulator in its tensor memory.  An MMA of 128
// rows reads its token operand from shared memory at half of that memory's bandwidth, and writing the stages takes the other
// half: at 256 tokens, where the MMAs set the pace, single blocks take 158 us for 2048 x 12288 x 4096, pairs 150 (8 bits: 173, 160).
template <int BITS, int BT, int MODE, bool PAIR> struct QmmShape {
    static constexpr int SUB = BT <= 128 || PAIR ? 2 : 1;
    static constexpr int KPS = SUB == 2 ? 2 : BITS == 2 ? 8 : BITS <= 4 ? 4 : 2;  // 64-k blocks per slab
    static constexpr int ROW = KPS * 8 * BITS;                                     // bytes of a slab's row
    static constexpr bool OWNED = SUB == KPS;
    // the slab's swizzle: 16-byte chunk ^= (row >> SWZ_SHIFT) & SWZ_MASK (rows of 96 and 48 bytes are not swizzled)
    static constexpr int SWZ_MASK = ROW == 128 ? 7 : ROW == 64 ? 3 : ROW == 32 ? 1 : 0, SWZ_SHIFT = ROW == 128 ? 0 : ROW == 64 ? 1 : 2;
    static constexpr int COLS = 32 * SUB;  // tensor-memory columns of a stage's weights
    static constexpr int ACC_BUFS = 2 * BT + 4 * COLS <= 512 ? 2 : 1;
    static constexpr int A_COL0 = ACC_BUFS * BT;
    static constexpr uint32_t XB_BYTES = (PAIR ? BT / 2 : BT) * QMM_BK * 2;  // activations of one k-block
    static constexpr uint32_t X_BYTES = SUB * XB_BYTES;
    static constexpr uint32_t W_BYTES = 128 * ROW;
    static constexpr int GRAIN = KPS < 4 ? 4 : KPS;  // K-split parts start at multiples of this many k-blocks
    // two chunks of scales (and biases) of the smallest groups: 32 bytes and a word of slack per row
    static constexpr uint32_t S_BYTES = (MODE == 0 ? 2 : 1) * 2 * 128 * 36;
    static constexpr int FIXED = 1024 /* alignment */ + 1024 /* barriers and flags */ + QMM_TABLE_BYTES + QMM_ITEM_BYTES + QMM_EPI_STAGE_BYTES + (int)S_BYTES;
    static constexpr int BY_TMEM = (512 - A_COL0) / COLS;
    static constexpr int BY_SMEM = (227 * 1024 - FIXED - (OWNED ? 4 : 2) * (int)W_BYTES) / (int)X_BYTES;
    static constexpr int FIT = BY_TMEM < BY_SMEM ? (BY_TMEM < 8 ? BY_TMEM : 8) : (BY_SMEM < 8 ? BY_SMEM : 8);
    // a multiple of the dequantizer groups, so that a stage is always refilled by the same group
    static constexpr int STAGES = FIT / QMM_DQ_GROUPS * QMM_DQ_GROUPS;
    static_assert(STAGES >= QMM_DQ_GROUPS, "token tile too wide for the weight ring");
    static constexpr int W_FIT = (227 * 1024 - FIXED - STAGES * (int)X_BYTES) / (int)W_BYTES;
    // OWNED: also a multiple of the groups (a slot is then always filled for the same group, which so never waits for a
    // phase two ahead of the barrier's)
    static constexpr int W_STAGES = OWNED ? (W_FIT >= 8 ? 8 : 4) : (W_FIT < 4 ? W_FIT : 4);
    static constexpr size_t SMEM = FIXED + STAGES * X_BYTES + W_STAGES * W_BYTES;
    static_assert(SMEM <= 227 * 1024 && W_FIT >= W_STAGES && W_STAGES >= 2, "not enough shared memory for the pipeline");
};

template <int BYTES> __device__ __forceinline__ void q_cp_async(uint32_t dst, const void *src) {
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ uint32_t q_lds_u16(uint32_t a) {
    uint32_t v;
    asm volatile("{\n\t.reg .b16 t;\n\tld.shared.b16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t q_lds_u8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
template <bool F16> __device__ __forceinline__ uint16_t q_bits(float f) {
    return F16 ? __half_as_ushort(__float2half_rn(f)) : __bfloat16_as_ushort(__float2bfloat16_rn(f));
}

// The scales of 64 k-values of a row: k-block kc of the chunk of scales and biases at shared addresses s_at, b_at.
template <int MODE, bool F16> struct BlockScales {  // affine: one pair per half of 32 values
    Affine<F16> q[2];
    __device__ __forceinline__ BlockScales(uint32_t s_at, uint32_t b_at, int kc, int gs_shift) {
        const uint32_t g = (uint32_t)(kc * QMM_BK) >> gs_shift;
        q[0].set(q_lds_u16(s_at + 2 * g), q_lds_u16(b_at + 2 * g));
        q[1] = q[0];
        if (gs_shift == 5) q[1].set(q_lds_u16(s_at + 2 * g + 2), q_lds_u16(b_at + 2 * g + 2));
    }
};
struct FpBlockScales {  // mxfp4, mxfp8: one scale per 32 values; nvfp4: one per 16 (two per half)
    uint32_t fa[2], fb[2];
};
template <bool F16> struct BlockScales<1, F16> : FpBlockScales {
    __device__ __forceinline__ BlockScales(uint32_t s_at, uint32_t, int kc, int) {
#pragma unroll
        for (int h = 0; h < 2; h++) fa[h] = fb[h] = fp_scale2(q_lds_u8(s_at + (uint32_t)(kc * 2 + h)), true);
    }
};
template <bool F16> struct BlockScales<2, F16> : BlockScales<1, F16> {
    using BlockScales<1, F16>::BlockScales;
};
template <bool F16> struct BlockScales<3, F16> : FpBlockScales {
    __device__ __forceinline__ BlockScales(uint32_t s_at, uint32_t, int kc, int) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            fa[h] = fp_scale2(q_lds_u8(s_at + (uint32_t)(kc * 4 + 2 * h)), false);
            fb[h] = fp_scale2(q_lds_u8(s_at + (uint32_t)(kc * 4 + 2 * h + 1)), false);
        }
    }
};
// Half h (32 values) of k-block kq of the slab row at `wrow` (its swizzle phase `sw`) -> 16 registers, register c holding
// k = 2c, 2c + 1.
template <int BITS, int MODE, bool F16>
__device__ __forceinline__ void dequant_half(const uint8_t *wrow, int sw, int kq, int h, const BlockScales<MODE, F16> &sc, uint32_t (&v)[16]) {
    if constexpr (BITS == 4) {
        const uint4 pk = *reinterpret_cast<const uint4 *>(wrow + (((kq * 2 + h) ^ sw) << 4));
        const uint32_t wv[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if constexpr (MODE == 0) dequant_word4<F16>(wv[c], sc.q[h], v + 4 * c);
            else dequant_word_fp4(wv[c], c < 2 ? sc.fa[h] : sc.fb[h], v + 4 * c);
        }
    } else if constexpr (BITS == 8) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const uint4 pk = *reinterpret_cast<const uint4 *>(wrow + (((kq * 4 + 2 * h + c) ^ sw) << 4));
            const uint32_t wv[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if constexpr (MODE == 0) dequant_word8<F16>(wv[i], sc.q[h], v + 8 * c + 2 * i);
                else dequant_word_fp8(wv[i], sc.fa[h], v + 8 * c + 2 * i);
            }
        }
    } else if constexpr (BITS == 2) {
        const uint2 pk = *reinterpret_cast<const uint2 *>(wrow + ((kq ^ sw) << 4) + 8 * h);
        dequant_word2<F16>(pk.x, sc.q[h], v);
        dequant_word2<F16>(pk.y, sc.q[h], v + 8);
    } else if constexpr (BITS == 3) {  // 12 bytes: one unit of 32 codes
        const uint32_t *src = reinterpret_cast<const uint32_t *>(wrow + kq * 24 + 12 * h);
        const uint32_t u[3] = {src[0], src[1], src[2]};
        dequant_words3<3, F16>(u, sc.q[h], v);
    } else {  // 6 bits, 24 bytes: two units of 16 codes
        const uint2 *src = reinterpret_cast<const uint2 *>(wrow + kq * 48 + 24 * h);
        const uint2 a = src[0], b = src[1], c = src[2];
        const uint32_t lo[3] = {a.x, a.y, b.x}, hi[3] = {b.y, c.x, c.y};
        dequant_words3<6, F16>(lo, sc.q[h], v);
        dequant_words3<6, F16>(hi, sc.q[h], v + 8);
    }
}

template <int BITS, int BT, int MODE /*0 affine, 1 mxfp4, 2 mxfp8, 3 nvfp4*/, bool F16, bool PAIR>
__global__ void __launch_bounds__(QMM_THREADS, 1)
qmm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, QmmKernelParams p,
           int total_tiles, int n_tiles) {
    using S = QmmShape<BITS, BT, MODE, PAIR>;
    constexpr int KPS = S::KPS, SUB = S::SUB, STAGES = S::STAGES, W_STAGES = S::W_STAGES, A_COL0 = S::A_COL0, ACC_BUFS = S::ACC_BUFS;
    constexpr int GRAIN = S::GRAIN;
    constexpr uint32_t X_BYTES = S::X_BYTES, W_BYTES = S::W_BYTES, S_BYTES = S::S_BYTES;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the swizzled tiles
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *xs = smem;                                   // [STAGES][SUB][BT x 128 B]
    uint8_t *ws = xs + STAGES * X_BYTES;                  // [W_STAGES][128 x ROW B]
    uint8_t *ss = ws + W_STAGES * W_BYTES;                // [s_stages][scales, biases][128 x s_pitch B]
    uint64_t *bars = reinterpret_cast<uint64_t *>(ss + S_BYTES);
    // empty[s]: the MMAs that read activation stage s (shared memory) and weight stage s (tensor
    // memory) are done; the activation producer and the dequantizers both wait on it.
    uint64_t *xfull = bars, *afull = xfull + STAGES, *empty = afull + STAGES;
    uint64_t *wfull = empty + STAGES, *wempty = wfull + W_STAGES;
    uint64_t *sfull = wempty + W_STAGES, *sempty = sfull + QMM_S_STAGES_MAX;
    uint64_t *accfull = sempty + QMM_S_STAGES_MAX, *accempty = accfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accempty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *last_flag = abort_flag + 1;  // epilogue: this block arrived last at a K-split tile
    int *table = reinterpret_cast<int *>(bars) + 256;  // behind the 1 KB of barriers and flags: 2 x (experts + 1) ints
    int4 *item_list = reinterpret_cast<int4 *>(reinterpret_cast<uint8_t *>(bars) + 1024 + QMM_TABLE_BYTES);
    uint8_t *epi_stage = reinterpret_cast<uint8_t *>(bars) + 1024 + QMM_TABLE_BYTES + QMM_ITEM_BYTES;  // [epilogue warp][32 tokens][32 rows] of 16 bits

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kblocks = p.K / QMM_BK;
    // A pair works as one: both blocks walk the same items.
    const int half = PAIR ? (int)pair_rank() : 0;
    const int block = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, blocks = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;
    if (!p.early) pdl_wait();
    pdl_trigger();

    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(xfull + s, 1);
            mbar_init(afull + s, (PAIR ? 2 : 1) * QMM_DQ_WARPS / QMM_DQ_GROUPS);  // (pairs: arrivals of both blocks, on the first one's)
            mbar_init(empty + s, 1);
        }
        for (int s = 0; s < W_STAGES; s++) {
            mbar_init(wfull + s, 1);
            mbar_init(wempty + s, S::OWNED ? QMM_DQ_WARPS / QMM_DQ_GROUPS : QMM_DQ_WARPS);
        }
        for (int s = 0; s < QMM_S_STAGES_MAX; s++) {
            mbar_init(sfull + s, 4 * 32);  // every loading lane's copies
            mbar_init(sempty + s, QMM_DQ_WARPS);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(accfull + s, 1);
            mbar_init(accempty + s, (PAIR ? 2 : 1) * QMM_EPI_WARPS);
        }
        *abort_flag = 0;
        *last_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {  // all of tensor memory: the accumulators and the dequantized-weight ring
        if (PAIR) {  // the same warp of both blocks
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    Schedule sched = p.sched;
    GroupTable gt{nullptr, nullptr};
    const bool tabled = p.offsets && p.experts <= QMM_MAX_TABLE_EXPERTS;
    const QmmWork<BT, GRAIN, PAIR> work{p, sched, gt, item_list, kblocks, n_tiles, block, blocks, half};
    if (p.offsets) pdl_wait();  // the experts' offsets are an earlier kernel's
    if (tabled) {
        for (int e = tid; e <= p.experts; e += QMM_THREADS) table[e] = e < p.experts ? p.offsets[e] : p.rows;
    } else if (tid >= 64 && tid < 64 + QMM_ITEMS) {
        work.fill(tid - 64);
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) pair_sync();  // the other block's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (tabled) {
        // tiles before each expert: a warp's scan over the experts, 32 at a time
        int *tiles = table + QMM_MAX_TABLE_EXPERTS + 1;
        if (warp == 0) {
            int seen = 0;
            for (int e0 = 0; e0 < p.experts; e0 += 32) {
                const int e = e0 + lane;
                const int mine = e < p.experts ? (table[e + 1] - table[e] + BT - 1) / BT : 0;
                int upto = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, upto, o);
                    if (lane >= o) upto += v;
                }
                if (e < p.experts) tiles[e] = seen + upto - mine;
                seen += __shfl_sync(0xFFFFFFFFu, upto, 31);
            }
            if (lane == 0) tiles[p.experts] = seen;
        }
        __syncthreads();
        gt.off = table;
        gt.tiles = tiles;
        // (the host knows only the most tiles there can be)
        float ns;
        sched = make_schedule(tiles[p.experts] * n_tiles, blocks, kblocks, GRAIN, BT, qmm_block_ns(BT, PAIR, BITS), &ns);
        if (tid < QMM_ITEMS) work.fill(tid);
        __syncthreads();
    }

    if (warp == 4) {
        // ── TMA producer, activations ───────────────────────────────────────────────────────
        // (the whole warp walks the loop and one elected lane issues: operands stay the warp's, see the MMA issuer)
        QT_BEGIN
        const bool elected = elect_one();
        pdl_wait();
        uint32_t s = 0, ph = 1;
        bool ok = true;
        for (int j = 0; ok; j++) {
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            const int tok0 = __shfl_sync(0xFFFFFFFFu, ti.tok0, 0);
            for (int kb = item.kb0; kb < item.kb1; kb += SUB) {
                s = __shfl_sync(0xFFFFFFFFu, s, 0);
                QT(1, ok = mbar_wait(empty + s, ph, abort_flag))
                if (!ok) break;
                if (elected) {
                    if (!PAIR || half == 0) mbar_expect_tx(xfull + s, (PAIR ? 2 : 1) * X_BYTES);
#pragma unroll
                    for (int b = 0; b < SUB; b++) {  // (a block past the end of K arrives as zeros)
                        uint8_t *dst = xs + s * X_BYTES + b * S::XB_BYTES;
                        if (PAIR)  // both blocks' halves complete on the first block's barrier
                            tma_load_2d_pair(dst, &tmap_x, (kb + b) * QMM_BK, tok0 + half * (BT / 2), pair_leader_addr(smem_u32(xfull + s)));
                        else
                            tma_load_2d(dst, &tmap_x, (kb + b) * QMM_BK, tok0, xfull + s);
                    }
                }
                __syncwarp();
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        QT_END(0, lane == 0)
    } else if (warp == 6) {
        // ── TMA producer, packed weights ────────────────────────────────────────────────────
        const bool elected = elect_one();
        uint32_t s = 0, ph = 1;
        bool ok = true;
        for (int j = 0; ok; j++) {
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            const int row0 = __shfl_sync(0xFFFFFFFFu, ti.wrow0, 0);
            for (int kb = item.kb0; kb < item.kb1; kb += KPS) {
                s = __shfl_sync(0xFFFFFFFFu, s, 0);
                ok = mbar_wait_idle(wempty + s, ph, abort_flag, 64);
                if (!ok) break;
                if (elected) {
                    mbar_expect_tx(wfull + s, W_BYTES);
                    tma_load_2d(ws + s * W_BYTES, &tmap_w, (kb / KPS) * S::ROW, row0, wfull + s);
                }
                __syncwarp();
                if (++s == W_STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp >= QMM_SCALE_WARP) {
        // ── producers of scales and biases: a row per lane ──────────────────────────────────
        const int r = (warp - QMM_SCALE_WARP) * 32 + lane;
        const uint32_t stage_bytes = (MODE == 0 ? 2 : 1) * 128 * p.s_pitch;
        int s = 0;
        uint32_t ph = 1;
        bool ok = true;
        for (int j = 0; ok; j++) {
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            // (rows past N, in the last tile, repeat the last valid row's scales; their outputs are not stored)
            const size_t row_at = (size_t)(ti.wrow0 + min(r, p.N - 1 - ti.n0)) * (size_t)p.scale_row_bytes;
            for (int kb = item.kb0; kb < item.kb1; kb += QMM_CHUNK) {
                ok = mbar_wait_idle(sempty + s, ph, abort_flag, 128);
                if (!ok) break;
                const int from = ((kb * QMM_BK) >> p.gs_shift) * (MODE == 0 ? 2 : 1), bytes = min(p.chunk_bytes, p.scale_row_bytes - from);
                uint32_t dst = smem_u32(ss) + s * stage_bytes + (uint32_t)(r * p.s_pitch);
                const uint8_t *src = p.scales + row_at + from;
#pragma unroll
                for (int array = 0; array < (MODE == 0 ? 2 : 1); array++) {
                    if (array) {
                        src = p.biases + row_at + from;
                        dst += (uint32_t)(128 * p.s_pitch);
                    }
                    if (p.s_vec == 16) {
                        for (int c = 0; c < bytes; c += 16) q_cp_async<16>(dst + c, src + c);
                    } else if (p.s_vec == 8) {
                        for (int c = 0; c < bytes; c += 8) q_cp_async<8>(dst + c, src + c);
                    } else {
                        // (every word copied holds a byte that is wanted, so none lies outside the arrays' allocations)
                        const int off = (int)((uintptr_t)src & 3);
                        for (int c = 0; c < bytes + off; c += 4) q_cp_async<4>(dst + c, src - off + c);
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(sfull + s)) : "memory");
                if (++s == p.s_stages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 5) {
        // ── MMA issuer: A (weights) from tensor memory, B (activations) from shared memory ──
        // Any shared-memory load (an mbarrier test included) issued by the thread that issues
        // tcgen05.mma was measured at ~270 cycles per round on the B200, more than four MMA issues;
        // a hardware named barrier costs ~30.  So this warp never reads shared memory: the watcher
        // warp waits on the mbarriers (stage full, accumulator drained) and passes each stage on
        // through named barrier 1 + stage.  All lanes walk the loop, one elected lane issues, and the operands are read
        // from lane 0: the compiler then knows that they are the warp's, as the instruction wants them, and not one lane's
        // (477 -> 200 cycles per 64-k block).
        constexpr uint32_t idesc = umma_idesc(BT, F16, PAIR ? 2 * QMM_BN : QMM_BN);
        QT_BEGIN
        uint32_t tcount = 0, s = 0;
        const uint32_t empty0 = smem_u32(empty);
        const uint64_t bd0 = umma_desc(smem_u32(xs));
        const bool elected = elect_one();
        const uint32_t tmem_u = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
        for (int j = 0; half == 0; j++) {  // (pairs: the first block's warp issues for both)
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            const uint32_t buf = __shfl_sync(0xFFFFFFFFu, tcount % ACC_BUFS, 0);
            const uint32_t d = tmem_u + buf * BT;
            for (int kb = item.kb0; kb < item.kb1; kb += SUB) {
                s = __shfl_sync(0xFFFFFFFFu, s, 0);
                QT(1, named_sync(1 + s))  // stage s is full (and, for the first one, the accumulator is drained)
                QT(2, if (elected) {
                    tc_fence_after();
                    const uint32_t at = tmem_u + A_COL0 + s * S::COLS;
                    const uint64_t bd = bd0 + (uint64_t)(s * (X_BYTES >> 4));
_Pragma("unroll")
                    for (int b = 0; b < SUB; b++) {
                        if (b > 0 && kb + b >= item.kb1) break;
_Pragma("unroll")
                        for (int k = 0; k < QMM_BK / 16; k++) {  // 16 k-values: 8 columns of A, 32 bytes of the swizzle row of B
                            const uint64_t bk = bd + (uint64_t)(b * (S::XB_BYTES >> 4) + 2 * k);
                            if (PAIR) tc_mma_bf16_ta_pair(d, at + 32 * b + 8 * k, bk, idesc, kb != item.kb0 || b != 0 || k != 0);
                            else tc_mma_bf16_ta(d, at + 32 * b + 8 * k, bk, idesc, kb != item.kb0 || b != 0 || k != 0);
                        }
                    }
                    // frees both halves of the stage (in both blocks of a pair) once these MMAs have read them
                    if (PAIR) tc_commit_pair(empty0 + 8 * s);
                    else tc_commit_addr(empty0 + 8 * s);
                })
                __syncwarp();
                if (++s == STAGES) s = 0;
            }
            if (elected) {
                if (PAIR) tc_commit_pair(smem_u32(accfull + buf));
                else tc_commit(accfull + buf);
            }
            __syncwarp();
            tcount++;
        }
        QT_END(1, lane == 0)
    } else if (warp == QMM_WATCH_WARP) {
        // ── watcher: the MMA warp's eyes.  It arrives on the named barrier of every stage exactly
        //    once per use whatever happens (after a wait gave up it stops waiting, not
        //    arriving), so the MMA warp can never be left behind in a barrier. ──
        uint32_t tcount = 0, s = 0, ph = 0;
        bool ok = true;
        QT_BEGIN
        for (int j = 0; half == 0; j++) {
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            const uint32_t buf = tcount % ACC_BUFS, aph = (tcount / ACC_BUFS) & 1;
            QT(4, if (lane == 0 && ok) ok = mbar_wait(accempty + buf, aph ^ 1, abort_flag))  // the epilogue has drained this buffer
            for (int kb = item.kb0; kb < item.kb1; kb += SUB) {
                QT(1, if (lane == 0 && ok) ok = mbar_wait(xfull + s, ph, abort_flag))
                QT(3, if (lane == 0 && ok) ok = mbar_wait(afull + s, ph, abort_flag))
                __syncwarp();
                QT(5, named_arrive(1 + s))
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            tcount++;
        }
        QT_END(2, lane == 0)
    } else if (warp >= 7 && warp < QMM_WATCH_WARP) {
        // ── dequantizers ─────────────────────────────────────────────────────────────────
        // Four groups of 4 warps take stages in turn.  Thread = weight row = tensor-memory lane
        // (a warp reaches the 32 lanes of its rank in the warpgroup): it rebuilds the k-values of
        // its row in registers and stores them as columns of the stage, where the MMA
        // reads its A operand.  Nothing dequantized passes through shared memory.
        const int row = 32 * (warp & 3) + lane, group = (warp - 7) >> 2;
        const int sw = (row >> S::SWZ_SHIFT) & S::SWZ_MASK;  // swizzle phase of this row in the packed slab
        const uint32_t a_cols = tmem_base + A_COL0 + ((uint32_t)(32 * (warp & 3)) << 16);
        const uint32_t s_stage_bytes = (MODE == 0 ? 2 : 1) * 128 * p.s_pitch;
        uint32_t it_base = 0, wit = 0, sph = 0;
        int sc = 0;
        bool ok = true;
        QT_BEGIN
        for (int j = 0; ok; j++) {
            Item item;
            TileInfo ti;
            const int what = work(j, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            // where the row's scales start within their aligned word (0 unless rows are not word-aligned)
            const uint32_t wr = (uint32_t)(ti.wrow0 + min(row, p.N - 1 - ti.n0));
            const uint32_t s_low = (uint32_t)(uintptr_t)p.scales + wr * (uint32_t)p.scale_row_bytes;
            const uint32_t b_low = MODE == 0 ? (uint32_t)(uintptr_t)p.biases + wr * (uint32_t)p.scale_row_bytes : 0u;
            // this group's stages are those at ring positions = group (mod groups): the same warps
            // always refill the same stages, so nobody is ever two phases ahead of a barrier
            const int first = (int)((uint32_t)(group - (int)it_base) % QMM_DQ_GROUPS);
            // announces a stage whose stores this warp has issued
            auto publish = [&](uint32_t sa) {
                tc_st_wait();
                tc_fence_before();  // the stores are ordered before the arrive the MMA thread waits on
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_leader(afull + sa);
                    else mbar_arrive(afull + sa);
                }
            };
            const int stages = (item.kb1 - item.kb0 + SUB - 1) / SUB;
            int kb = item.kb0 + first;  // (not OWNED: this group's next k-block)
            for (int ck = item.kb0; ck < item.kb1 && ok; ck += QMM_CHUNK) {
                // the chunk's scales
                QT(4, ok = mbar_wait(sfull + sc, sph, abort_flag))
                const uint32_t from = (uint32_t)(((ck * QMM_BK) >> p.gs_shift) * (MODE == 0 ? 2 : 1));
                const uint32_t area = smem_u32(ss) + sc * s_stage_bytes + (uint32_t)(row * p.s_pitch);
                const uint32_t s_at = area + ((s_low + from) & 3u), b_at = area + (uint32_t)(128 * p.s_pitch) + ((b_low + from) & 3u);
                if constexpr (S::OWNED) {
                    // a chunk is one round of the groups: at most one stage of it is this group's
                    static_assert(!S::OWNED || QMM_CHUNK == SUB * QMM_DQ_GROUPS, "a chunk is one round of the groups");
                    const int st = (ck - item.kb0) / SUB + first;
                    if (st < stages && ok) {
                        const uint32_t it = it_base + (uint32_t)st, wsi = it % W_STAGES, sa = it % STAGES;
                        QT(1, ok = mbar_wait(wfull + wsi, (it / W_STAGES) & 1, abort_flag))
                        const uint8_t *wrow = ws + wsi * W_BYTES + row * S::ROW;
                        const int blocks_here = item.kb0 + st * SUB + 1 < item.kb1 ? 2 : 1;
                        // stored by halves: the second half's registers do not wait for the first half's store to read its own
                        // (32 columns at a time: 48.8 instead of 47.3 us for 128 experts x 768 x 2048)
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            if (b == blocks_here) break;
                            const BlockScales<MODE, F16> scales(s_at, b_at, 2 * first + b, p.gs_shift);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                uint32_t v[16];
                                dequant_half<BITS, MODE, F16>(wrow, sw, b, h, scales, v);
                                if (b == 0 && h == 0) {
                                    QT(2, ok = ok && mbar_wait(empty + sa, ((it / STAGES) & 1) ^ 1, abort_flag))  // the MMAs that read this stage are done
                                    if (!ok) break;
                                    tc_fence_after();
                                }
                                tc_st16(a_cols + sa * S::COLS + 32 * b + 16 * h, v);
                            }
                            if (!ok) break;
                        }
                        if (!ok) break;
                        __syncwarp();
                        if (lane == 0) mbar_arrive(wempty + wsi);  // the slab has been read
                        QT(3, publish(sa);)
                    }
                } else {
                    const int ck_end = min(ck + QMM_CHUNK, item.kb1);
                    for (int slab = ck; slab < ck_end && ok; slab += KPS, wit++) {
                        const uint32_t wsi = wit % W_STAGES, wph = (wit / W_STAGES) & 1;
                        const int kb_end = min(slab + KPS, ck_end);
                        // (a warp none of whose blocks lie in this slab waits for it all the same before it releases it: otherwise
                        // it could run ahead and its arrival for a later slab would be counted into this one's phase)
                        QT(1, ok = mbar_wait(wfull + wsi, wph, abort_flag))
                        const uint8_t *wrow = ws + wsi * W_BYTES + row * S::ROW;
#pragma unroll 1
                        for (; kb < kb_end && ok; kb += QMM_DQ_GROUPS) {
                            const uint32_t it = it_base + (uint32_t)(kb - item.kb0), sa = it % STAGES;
                            const BlockScales<MODE, F16> scales(s_at, b_at, kb - ck, p.gs_shift);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                uint32_t v[16];
                                dequant_half<BITS, MODE, F16>(wrow, sw, kb - slab, h, scales, v);
                                if (h == 0) {
                                    QT(2, ok = mbar_wait(empty + sa, ((it / STAGES) & 1) ^ 1, abort_flag))
                                    if (!ok) break;
                                    tc_fence_after();
                                }
                                tc_st16(a_cols + sa * S::COLS + 16 * h, v);
                            }
                            if (!ok) break;
                            QT(3, publish(sa);)
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(wempty + wsi);
                    }
                }
                // (every warp releases every chunk, one that holds none of its stages included)
                __syncwarp();
                if (lane == 0) mbar_arrive(sempty + sc);
                if (++sc == p.s_stages) {
                    sc = 0;
                    sph ^= 1;
                }
            }
            it_base += (uint32_t)stages;
        }
        QT_END(3 + group, (warp & 3) == 3 && lane == 0)
    } else {
        // ── epilogue: warp q owns tensor-memory lanes 32q .. 32q+31 = weight rows n0 + 32q + lane ──
        uint32_t tcount = 0;
        bool ok = true;
        auto drained = [&](uint32_t buf) {  // the accumulator is free again
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_leader(accempty + buf);
                else mbar_arrive(accempty + buf);
            }
        };
        QT_BEGIN
        for (int jj = 0; ok; jj++) {
            Item item;
            TileInfo ti;
            const int what = work(jj, item, ti);
            if (what == QMM_END) break;
            if (what == QMM_SKIP) continue;
            const uint32_t buf = tcount % ACC_BUFS, aph = (tcount / ACC_BUFS) & 1;
            // After a wait gave up the warp keeps walking the items without touching data: the
            // named barriers of K-split tiles below must still see all four epilogue warps.
            QT(1, if (ok) ok = mbar_wait_idle(accfull + buf, aph, abort_flag, 128))
            tc_fence_after();
            const int r = warp * 32 + lane;  // row of the tile
            const uint32_t acc = tmem_base + ((uint32_t)(warp * 32) << 16) + buf * BT;
            float gmul = 1.0f;
            if (MODE != 0 && p.global) gmul = (p.expert_global ? p.global[ti.expert] : p.global[0]) / (448.0f * 6.0f);
            if (item.parts == 1) {
                // Thread = weight row, registers = 32 tokens, but y is [token][row]: the warp turns each
                // 32 x 32 piece around in shared memory ([token][row], 64 bytes per token) and stores it
                // as 16-byte pieces of 8 rows -- 4 store instructions per piece instead of 32.  Where rows are not
                // whole aligned groups of 8, a token's 32 values per store instruction.
                const bool wide = (p.N & 7) == 0 && ((uintptr_t)p.y & 15) == 0;
                uint8_t *mine = epi_stage + warp * 2048;
                const int t8 = lane >> 2, g8 = lane & 3;  // this lane's token (of 8 per pass) and group of 8 rows
#pragma unroll 1
                for (int c = 0; c < BT / 32 && ok; c++) {
                    if (ti.tok0 + c * 32 >= ti.tok_end) break;  // (the whole warp: nothing of this piece is stored)
                    uint32_t v[32];
                    QT(2, tc_ld32(acc + c * 32, v);
                    tc_ld_wait())
                    QT(3, _Pragma("unroll")
                    for (int i = 0; i < 32; i++) {
                        float f = __uint_as_float(v[i]);
                        if (MODE != 0) f *= gmul;
                        *reinterpret_cast<uint16_t *>(mine + i * 64 + lane * 2) = q_bits<F16>(f);
                    }
                    __syncwarp())
                    if (wide) {
                        const int ng = ti.n0 + warp * 32 + g8 * 8;
                        uint16_t *dst = p.y + (size_t)(ti.tok0 + c * 32 + t8) * p.N + ng;
                        QT(4, _Pragma("unroll")
                        for (int i = 0; i < 4; i++) {
                            const uint4 q = *reinterpret_cast<const uint4 *>(mine + (i * 8 + t8) * 64 + g8 * 16);
                            if (ng < p.N && ti.tok0 + c * 32 + i * 8 + t8 < ti.tok_end)
                                *reinterpret_cast<uint4 *>(dst + (size_t)(i * 8) * p.N) = q;
                        })
                    } else {
                        const int tokens = min(32, ti.tok_end - ti.tok0 - c * 32);
                        if (ti.n0 + r < p.N)
                            for (int i = 0; i < tokens; i++)
                                p.y[(size_t)(ti.tok0 + c * 32 + i) * p.N + ti.n0 + r] = *reinterpret_cast<const uint16_t *>(mine + i * 64 + lane * 2);
                    }
                    __syncwarp();  // the piece has been read before the next one overwrites it
                }
                drained(buf);
            } else {
                // One part of a tile cut along K: the float32 partial goes to scratch as
                // [token][row] (a warp writes 128 consecutive bytes per token); the block that
                // arrives last adds the parts in part order and rounds once.
                const int pslot = PAIR ? 2 * item.slot + half : item.slot;  // each block of a pair keeps its own rows' parts
                float *mine = p.partials + ((size_t)pslot * item.parts + item.part) * (size_t)(BT * QMM_BN);
#pragma unroll 1
                for (int c = 0; c < BT / 32 && ok; c++) {
                    if (ti.tok0 + c * 32 >= ti.tok_end) break;
                    uint32_t v[32];
                    tc_ld32(acc + c * 32, v);
                    tc_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (ti.tok0 + c * 32 + i < ti.tok_end) __stcg(mine + (size_t)(c * 32 + i) * QMM_BN + r, __uint_as_float(v[i]));
                }
                drained(buf);
                __threadfence();
                named_sync_n(QMM_EPI_BARRIER, QMM_EPI_WARPS * 32);
                if (tid == 0) {
                    bool last = false;
                    if (ok) {
                        const uint32_t arrived = atomicAdd(p.counters + pslot, 1u);
                        last = arrived == (uint32_t)item.parts - 1;
                        if (last) p.counters[pslot] = 0u;  // rearmed for the next launch
                    }
                    // K-split parts are a block's last items: the whole block adds the parts up
                    // after its roles have finished (below).
                    if (last) *last_flag = *last_flag | (1 << item.round);
                }
            }
            tcount++;
        }
        QT_END(7, warp == 0 && lane == 0)
    }

    // ── teardown ────────────────────────────────────────────────────────────────────────
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag && p.error) *p.error = 1;
    for (int round = 0; round < sched.tail_rounds && !*abort_flag; round++) {
        if (!(*last_flag & (1 << round))) continue;
        // This block arrived last at this K-split tile: all its threads add the float32 parts in
        // part order (the sum does not depend on who arrived when), round once and store.
        Item item;
        TileInfo ti;
        if (work(sched.full_waves + round, item, ti) == QMM_TAKE) {
            __threadfence();
            float gmul = 1.0f;
            if (MODE != 0 && p.global) gmul = (p.expert_global ? p.global[ti.expert] : p.global[0]) / (448.0f * 6.0f);
            const int pslot = PAIR ? 2 * item.slot + half : item.slot;
            const float4 *base = reinterpret_cast<const float4 *>(p.partials + (size_t)pslot * item.parts * (size_t)(BT * QMM_BN));
            constexpr int TILE4 = BT * QMM_BN / 4;  // float4 per part
            const int tokens = min(BT, ti.tok_end - ti.tok0);
            const bool wide = (p.N & 3) == 0 && ((uintptr_t)p.y & 7) == 0;
            // Two groups of four values per thread and pass, four parts of each at a time: eight loads in flight per thread (one
            // after the other they took 23 us for four parts of 128 x 256).
            const int count = tokens * (QMM_BN / 4);
            for (int idx0 = tid; idx0 < count; idx0 += 2 * QMM_THREADS) {
                float4 acc[2];
                for (int q0 = 0; q0 < item.parts; q0 += 4) {
                    float4 v[2][4];
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (idx0 + i * QMM_THREADS < count && q0 + q < item.parts) v[i][q] = __ldcg(base + (size_t)(q0 + q) * TILE4 + idx0 + i * QMM_THREADS);
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (q0 + q >= item.parts) break;
                            if (q0 + q == 0) {
                                acc[i] = v[i][q];
                            } else {
                                acc[i].x += v[i][q].x; acc[i].y += v[i][q].y; acc[i].z += v[i][q].z; acc[i].w += v[i][q].w;
                            }
                        }
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int idx = idx0 + i * QMM_THREADS;
                    if (idx >= count) break;
                    const float f[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
                    const int t = idx / (QMM_BN / 4), n = ti.n0 + 4 * (idx % (QMM_BN / 4));
                    uint16_t h[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) h[e] = q_bits<F16>(MODE != 0 ? f[e] * gmul : f[e]);
                    uint16_t *dst = p.y + (size_t)(ti.tok0 + t) * p.N + n;
                    if (wide) {
                        if (n < p.N) *reinterpret_cast<uint2 *>(dst) = make_uint2(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (n + e < p.N) dst[e] = h[e];
                    }
                }
            }
        }
    }
    if (PAIR) {
        // neither block leaves (or frees the pair's tensor memory) while the other may still arrive on its barriers
        tc_fence_before();
        pair_sync();
    }
    if (warp == 5) {
        tc_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(512) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(512) : "memory");
    }
}

// PAIR: the grid is made of clusters of two blocks (`total_tiles`, `n_tiles` then count tiles of 256 weight rows, `workers` pairs).
template <int BITS, int BT, int MODE, bool F16, bool PAIR>
static int32_t launch_cfg(nvc_device *dev, const QmmParams &q, QmmKernelParams k, int64_t token_tiles) {
    using S = QmmShape<BITS, BT, MODE, PAIR>;
    static_assert(8 * (QMM_MAX_TABLE_EXPERTS + 1) <= QMM_TABLE_BYTES, "the tables' area");
    const int64_t tile_rows = PAIR ? 2 * QMM_BN : QMM_BN, n_tiles = (q.N + tile_rows - 1) / tile_rows, total_tiles = token_tiles * n_tiles;
    if (total_tiles > INT32_MAX) return set_error(NVC_ERR_UNSUPPORTED, "qmm: too many tiles");
    CUtensorMap mx, mw;
    NVC_TRY(make_map(&mx, F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q.x, (uint64_t)q.K, (uint64_t)q.rows,
                     (uint64_t)q.ldx * 2, QMM_BK, (uint32_t)(PAIR ? BT / 2 : BT), 128));
    const uint64_t row_bytes = (uint64_t)q.K * BITS / 8;
    NVC_TRY(make_map(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, q.w, row_bytes, (uint64_t)(k.experts * q.N), row_bytes, S::ROW, QMM_BN,
                     S::SWZ_MASK ? S::ROW : 0));
    auto kernel = qmm_kernel<BITS, BT, MODE, F16, PAIR>;
    // the opt-in to this much dynamic shared memory is a per-device attribute of the instantiation
    static int workers[64] = {};  // blocks (pairs of blocks) that can be resident together; 0: not configured yet
    static std::mutex configured_mu;
    if (dev->ordinal < 0 || dev->ordinal >= 64) return set_error(NVC_ERR_UNSUPPORTED, "qmm: device ordinal %d", dev->ordinal);
    {
        std::lock_guard<std::mutex> g(configured_mu);
        if (workers[dev->ordinal] == 0) {
            NVC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
            int n = dev->prop.multiProcessorCount;
            if (PAIR) {
                cudaLaunchConfig_t probe = {};
                probe.gridDim = dim3(2 * (unsigned)n);
                probe.blockDim = dim3(QMM_THREADS);
                probe.dynamicSmemBytes = S::SMEM;
                cudaLaunchAttribute attr;
                attr.id = cudaLaunchAttributeClusterDimension;
                attr.val.clusterDim.x = 2;
                attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
                probe.attrs = &attr;
                probe.numAttrs = 1;
                NVC_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &probe));
                if (n < 1) return set_error(NVC_ERR_DRIVER, "qmm: no cluster of two blocks fits the device");
            }
            workers[dev->ordinal] = n;
        }
    }
    // How a chunk's scales are copied: the widest unit that the rows' length, the first k-blocks of parts and the addresses allow.
    const int per_value = MODE == 0 ? 2 : 1;
    k.chunk_bytes = ((QMM_CHUNK * QMM_BK) >> k.gs_shift) * per_value;
    const uintptr_t al = (uintptr_t)k.scales | (uintptr_t)k.biases | (uintptr_t)k.scale_row_bytes | (uintptr_t)(((S::GRAIN * QMM_BK) >> k.gs_shift) * per_value);
    k.s_vec = al % 16 == 0 ? 16 : al % 8 == 0 ? 8 : 4;
    k.s_pitch = al % 4 == 0 ? k.chunk_bytes : (k.chunk_bytes + 6) / 4 * 4;
    k.s_stages = (int)S::S_BYTES / (per_value * 128 * k.s_pitch);
    if (k.s_stages > QMM_S_STAGES_MAX) k.s_stages = QMM_S_STAGES_MAX;
    const int most = workers[dev->ordinal];
    int grid = most;
    size_t parts, slots;
    if (k.offsets && k.experts <= QMM_MAX_TABLE_EXPERTS) {
        parts = 2 * (size_t)most;  // whatever the experts' rows turn out to be
        slots = (size_t)most;
    } else {
        float ns;
        k.sched = make_schedule((int)total_tiles, most, k.K / QMM_BK, S::GRAIN, BT < q.rows ? BT : (int)q.rows, qmm_block_ns(BT, PAIR, BITS), &ns);
        if (k.sched.full_waves == 0 && k.sched.tail_tiles * k.sched.splits < most) grid = k.sched.tail_tiles * k.sched.splits;
        parts = k.sched.splits > 1 ? (size_t)k.sched.tail_tiles * k.sched.splits : 0;
        slots = (size_t)k.sched.tail_tiles;
    }
    if (parts) {
        const size_t blocks_per_tile = PAIR ? 2 : 1;  // each block of a pair keeps the parts of its own rows
        NVC_TRY(ensure_qmm_scratch(dev, blocks_per_tile * parts * BT * QMM_BN * sizeof(float), blocks_per_tile * slots));
        k.partials = (float *)dev->qmm_partials;
        k.counters = dev->qmm_counters;
    }
    const Writes written(k.early ? Trigger::EARLY : Trigger::LATE, {{q.y, (size_t)q.rows * (size_t)q.N * 2}});
    return launch_pdl_cluster(dev, "qmm_kernel", written, kernel, dim3((unsigned)grid * (PAIR ? 2 : 1)), dim3(QMM_THREADS), S::SMEM, PAIR ? 2 : 1, mx, mw, k,
                              (int)total_tiles, (int)n_tiles);
}

template <int BITS, int MODE, bool F16>
static int32_t launch_bt(nvc_device *dev, int bt, bool pair, const QmmParams &q, const QmmKernelParams &k, int64_t token_tiles) {
    if (pair) return launch_cfg<BITS, 256, MODE, F16, true>(dev, q, k, token_tiles);
    switch (bt) {
    case 32: return launch_cfg<BITS, 32, MODE, F16, false>(dev, q, k, token_tiles);
    case 64: return launch_cfg<BITS, 64, MODE, F16, false>(dev, q, k, token_tiles);
    case 128: return launch_cfg<BITS, 128, MODE, F16, false>(dev, q, k, token_tiles);
    case 160: return launch_cfg<BITS, 160, MODE, F16, false>(dev, q, k, token_tiles);
    case 192: return launch_cfg<BITS, 192, MODE, F16, false>(dev, q, k, token_tiles);
    default: return launch_cfg<BITS, 256, MODE, F16, false>(dev, q, k, token_tiles);
    }
}

}  // namespace nvc
