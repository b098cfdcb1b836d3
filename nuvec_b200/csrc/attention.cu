// Decode attention over an affine-quantized KV cache: fast::quantized_attention
// (crates/nuvec-core/src/fast.rs:694-722, fast/imp.rs:3940-4096; mlx-lm's quantized KV cache),
//
//     out[b, h, 0, :] = softmax(scale * q[b, h, 0, :] . K[b, h / rep, s, :] over s [, sinks[h]]) . V[b, h / rep, s, :]
//
// for every query row of every head (no mask; a row at a time), K and V as codes uint32 [B, Hkv, S, D * bits / 32] with scales and
// biases [B, Hkv, S, D / group_size], rep = Hq / Hkv query heads per key head, and an optional
// per-head sink that joins the softmax's denominator only.  The shapes the reference's kernel takes
// (fast/imp.rs:3944-3993): D 64 or 128, 3, 4 or 8 bits, groups of 32, 64 or 128, rep 1, 2, 4 or 8.
// Like that kernel it dequantizes in registers and keeps everything in float32, so it is within
// the float bound of attention over the dequantized cache (the bound the reference's test sets,
// crates/nuvec-core/tests/quantized.rs:1964-2031), not the bits of mlx-lm's composition, which
// rounds the scores to the queries' type.
//
// A cache is a view of a longer allocation (capacity beyond the keys): `capacity` is the number
// of rows between consecutive heads of every cache tensor.
//
// Every form splits the keys.  qattn_split_kernel (float32, 3-bit codes) works on the CUDA cores: one
// block of four warps per (split, key head, batch) walks its keys in tiles of 128 with a running maximum and denominator per
// query head -- scores by one thread per key, which reads the key's codes once and multiplies them with all rep query rows
// (float32 queries in shared memory, the group's scale and bias applied per group: s * sum(code * q) + b * sum(q)); values
// staged in shared memory with 16-byte loads, 64 threads x 2 key halves each own D / 64 output columns and accumulate
// p * (s * code + b) -- and qattn_combine merges the splits (and the sink) and rounds.  qattn_mma_kernel and
// qattn_tile_kernel (16-bit types, 4- and 8-bit codes) do both products on the tensor cores; see there and qattn_form.
#include "common.cuh"

#include <cstdlib>
#include <initializer_list>
#include <type_traits>

namespace nvc {

constexpr int QA_THREADS = 128, QA_TILE = 128, QA_MAX_REP = 8;

struct QAttnParams {
    const void *q;                               // [B, Hq, L, D]
    const uint32_t *kw, *vw;                     // codes
    const void *ks, *kb, *vs, *vb;               // scales, biases
    const void *sinks;                           // [Hq] or null
    float *part;                                 // [B, Hq, splits, D + 2]: acc, m, l
    void *out;                                   // [B, Hq, L, D]
    int32_t B, Hq, Hkv, S, capacity, splits, chunk;
    int32_t L, l;                                // query rows per head, and the row this launch attends for
    float scale;
    // the tensor-core form: query rows per column tile and such tiles, causal or not, whether the caches may be read before the
    // wait for the previous kernel, arrivals per (batch, row tile, key head), zero on entry and on exit
    int32_t row_pack, row_tiles, causal, early;
    uint32_t *counters;
};

// Code d of a row of BITS-bit codes packed low bits first (kernels.rs:749-756); `row` may be registers
// (d known at compile time after unrolling) or shared memory.
template <int BITS>
__device__ __forceinline__ uint32_t qa_code(const uint32_t *row, int d) {
    if (BITS == 8) return (row[d >> 2] >> (8 * (d & 3))) & 0xFFu;
    if (BITS == 4) return (row[d >> 3] >> (4 * (d & 7))) & 0xFu;
    const int bit = d * 3, w = bit >> 5, off = bit & 31;
    uint32_t v = row[w] >> off;
    if (off > 29) v |= row[w + 1] << (32 - off);
    return v & 7u;
}

// an integer below 2^23 as a float without the conversion unit (a quarter-rate instruction otherwise)
__device__ __forceinline__ float qa_float(uint32_t c) { return __uint_as_float(0x4B000000u | c) - 8388608.0f; }

template <typename T, int BITS, int D, int GS>
__global__ void __launch_bounds__(QA_THREADS, 5) qattn_split_kernel(QAttnParams p) {
    constexpr int W = D * BITS / 32, G = D / GS, DPT = D / 64;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the combine kernel's blocks may become resident meanwhile
    const int split = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    const int rep = p.Hq / p.Hkv, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int s0 = split * p.chunk, s1 = min(p.S, s0 + p.chunk);

    __shared__ __align__(16) float qs[D][QA_MAX_REP];          // scaled queries, [d][head]
    __shared__ float qsum[G][QA_MAX_REP];                      // their sums per group
    __shared__ __align__(16) float pr[QA_TILE][QA_MAX_REP];    // the tile's probabilities, [key][head]
    __shared__ float wred[2][4][QA_MAX_REP];                   // per-warp maxima / sums
    __shared__ __align__(16) uint32_t vrow[QA_TILE][W];        // the tile's value codes
    __shared__ float2 vsb[QA_TILE][G];                         // their (scale, bias)
    __shared__ float accx[64][DPT][QA_MAX_REP];                // second key half's sums, for the merge

    for (int i = t; i < D * QA_MAX_REP; i += QA_THREADS) {
        const int d = i / QA_MAX_REP, h = i % QA_MAX_REP;
        qs[d][h] = h < rep ? __fmul_rn(DT<T>::load((const T *)p.q, (((size_t)b * p.Hq + hk * rep + h) * p.L + p.l) * D + d), p.scale) : 0.0f;
    }
    __syncthreads();
    if (t < G * QA_MAX_REP) {
        const int g = t / QA_MAX_REP, h = t % QA_MAX_REP;
        float s = 0.0f;
        for (int d = 0; d < GS; d++) s += qs[g * GS + d][h];
        qsum[g][h] = s;
    }
    __syncthreads();

    const size_t head_row = ((size_t)b * p.Hkv + hk) * p.capacity;
    float m[QA_MAX_REP], l[QA_MAX_REP], acc[DPT][QA_MAX_REP];
#pragma unroll
    for (int h = 0; h < QA_MAX_REP; h++) {
        m[h] = -INFINITY;
        l[h] = 0.0f;
#pragma unroll
        for (int j = 0; j < DPT; j++) acc[j][h] = 0.0f;
    }
    const int dl = t & 63, half = t >> 6;  // value phase: columns dl * DPT .. , keys half * 64 ..

    for (int base = s0; base < s1; base += QA_TILE) {
        // ── scores of key base + t ──
        const int key = base + t;
        const bool valid = key < s1;
        float dot[QA_MAX_REP];
#pragma unroll
        for (int h = 0; h < QA_MAX_REP; h++) dot[h] = 0.0f;
        if (valid) {
            uint32_t row[W];
            const uint32_t *src = p.kw + (head_row + key) * W;
            if (W % 4 == 0) {
#pragma unroll
                for (int i = 0; i < W / 4; i++) {
                    const uint4 v = reinterpret_cast<const uint4 *>(src)[i];
                    row[4 * i] = v.x; row[4 * i + 1] = v.y; row[4 * i + 2] = v.z; row[4 * i + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < W / 2; i++) {
                    const uint2 v = reinterpret_cast<const uint2 *>(src)[i];
                    row[2 * i] = v.x; row[2 * i + 1] = v.y;
                }
            }
#pragma unroll
            for (int g = 0; g < G; g++) {
                float a[QA_MAX_REP];
#pragma unroll
                for (int h = 0; h < QA_MAX_REP; h++) a[h] = 0.0f;
#pragma unroll
                for (int d = g * GS; d < (g + 1) * GS; d++) {
                    const float c = qa_float(qa_code<BITS>(row, d));
                    const float4 q0 = *reinterpret_cast<const float4 *>(&qs[d][0]);
                    a[0] = fmaf(c, q0.x, a[0]); a[1] = fmaf(c, q0.y, a[1]); a[2] = fmaf(c, q0.z, a[2]); a[3] = fmaf(c, q0.w, a[3]);
                    if (rep > 4) {
                        const float4 q1 = *reinterpret_cast<const float4 *>(&qs[d][4]);
                        a[4] = fmaf(c, q1.x, a[4]); a[5] = fmaf(c, q1.y, a[5]); a[6] = fmaf(c, q1.z, a[6]); a[7] = fmaf(c, q1.w, a[7]);
                    }
                }
                const float sg = DT<T>::load((const T *)p.ks, (head_row + key) * G + g), bg = DT<T>::load((const T *)p.kb, (head_row + key) * G + g);
#pragma unroll
                for (int h = 0; h < QA_MAX_REP; h++) dot[h] = fmaf(sg, a[h], fmaf(bg, qsum[g][h], dot[h]));
            }
        }
        // ── the tile's values into shared memory (all threads) ──
        {
            const int keys = min(QA_TILE, s1 - base);
            constexpr int U = W % 4 == 0 ? 4 : 2;  // words per load
            const uint32_t *src = p.vw + (head_row + base) * W;
            for (int i = t; i < keys * W / U; i += QA_THREADS) {
                if (U == 4) reinterpret_cast<uint4 *>(&vrow[0][0])[i] = reinterpret_cast<const uint4 *>(src)[i];
                else reinterpret_cast<uint2 *>(&vrow[0][0])[i] = reinterpret_cast<const uint2 *>(src)[i];
            }
            for (int i = t; i < keys * G; i += QA_THREADS)
                vsb[0][i] = make_float2(DT<T>::load((const T *)p.vs, (head_row + base) * G + i), DT<T>::load((const T *)p.vb, (head_row + base) * G + i));
        }
        // ── running maximum and denominator per head ──
        float corr[QA_MAX_REP];
#pragma unroll
        for (int h = 0; h < QA_MAX_REP; h++) {
            float v = valid ? dot[h] : -INFINITY;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
            if (lane == 0) wred[0][warp][h] = v;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < QA_MAX_REP; h++) {
            const float mn = fmaxf(fmaxf(m[h], fmaxf(wred[0][0][h], wred[0][1][h])), fmaxf(wred[0][2][h], wred[0][3][h]));
            corr[h] = m[h] == -INFINITY ? 0.0f : expf(m[h] - mn);
            m[h] = mn;
            const float e = valid ? expf(dot[h] - mn) : 0.0f;
            pr[t][h] = e;
            float v = e;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            if (lane == 0) wred[1][warp][h] = v;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < QA_MAX_REP; h++) l[h] = fmaf(l[h], corr[h], (wred[1][0][h] + wred[1][1][h]) + (wred[1][2][h] + wred[1][3][h]));
        // ── values: columns dl * DPT .. of keys half * 64 .. + 63 of the tile ──
#pragma unroll
        for (int j = 0; j < DPT; j++)
#pragma unroll
            for (int h = 0; h < QA_MAX_REP; h++) acc[j][h] *= corr[h];
        const int kend = min(64, s1 - base - half * 64);
        for (int kk = 0; kk < kend; kk++) {
            const int s = half * 64 + kk;
            const float4 p0 = *reinterpret_cast<const float4 *>(&pr[s][0]);
            float4 p1 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rep > 4) p1 = *reinterpret_cast<const float4 *>(&pr[s][4]);
#pragma unroll
            for (int j = 0; j < DPT; j++) {
                const int d = dl * DPT + j;
                const float2 sb = vsb[s][d / GS];
                const float v = fmaf(sb.x, qa_float(qa_code<BITS>(vrow[s], d)), sb.y);
                acc[j][0] = fmaf(p0.x, v, acc[j][0]); acc[j][1] = fmaf(p0.y, v, acc[j][1]);
                acc[j][2] = fmaf(p0.z, v, acc[j][2]); acc[j][3] = fmaf(p0.w, v, acc[j][3]);
                if (rep > 4) {
                    acc[j][4] = fmaf(p1.x, v, acc[j][4]); acc[j][5] = fmaf(p1.y, v, acc[j][5]);
                    acc[j][6] = fmaf(p1.z, v, acc[j][6]); acc[j][7] = fmaf(p1.w, v, acc[j][7]);
                }
            }
        }
        __syncthreads();  // pr, vrow, vsb and wred are rewritten by the next tile
    }

    // ── the two key halves together, then this split's partial result ──
    if (half == 1) {
#pragma unroll
        for (int j = 0; j < DPT; j++)
#pragma unroll
            for (int h = 0; h < QA_MAX_REP; h++) accx[dl][j][h] = acc[j][h];
    }
    __syncthreads();
    if (half == 0) {
#pragma unroll
        for (int h = 0; h < QA_MAX_REP; h++) {
            if (h >= rep) break;
            float *dst = p.part + (((size_t)b * p.Hq + hk * rep + h) * p.splits + split) * (D + 2);
#pragma unroll
            for (int j = 0; j < DPT; j++) dst[dl * DPT + j] = acc[j][h] + accx[dl][j][h];
            if (dl == 0) {
                dst[D] = m[h];
                dst[D + 1] = l[h];
            }
        }
    }
}

// ── the tensor-core form (16-bit types, 4- and 8-bit codes) ─────────────────────────────────────────────
// mma.sync m16n8k16 (float16 operands, float32 accumulators) with the cache as the A operand and the queries as the eight
// columns of B: a key head's query heads, or, with several query rows, heads x rows.
//   scores   S_g[key, n] = sum over the group's dims of (1024 + code[key, d]) * q[d, n]
//            score[key, n] = sum_g  s_g[key] * (S_g - 1024 * qsum_g[n]) + b_g[key] * qsum_g[n]
//   values   O[d, n] += sum over keys of (1024 + code[key, d]) * (p[key, n] * s_g(d)[key])
//            out[d, n] = O[d, n] + sum over keys of (p * b_g(d)[key] - 1024 * p * s_g(d)[key])
// A code enters as the exact float16 integer 1024 + code (one byte permutation per pair at 8 bits, a shift and a LOP3 at 4),
// and the offset leaves with sums the kernel keeps anyway.  q * scale and p * s are rounded to float16, the latter where float16
// has all its bits (QA_TOP).
//
// Every warp works alone on steps of 16 keys: no barrier before the end.  The order of the dims in a dot
// product and of the dims among the output rows is free, so every lane's share of a row is contiguous bytes, all of which
// it uses: for the scores lane (g, c) reads GS * BITS / 32 bytes per group of keys g and g + 8, for the values GS * BITS / 64
// bytes per group of keys 2c, 2c + 1, 2c + 8, 2c + 9.  A step's rows are contiguous in memory; they travel with cp.async through
// a ring of QmRing::STAGES steps per warp (swizzled, so that both ways of reading them fall on distinct banks).  Loading them
// straight into the registers a step ahead left most of the latency exposed (16K keys, 8 bits: 17.4 us a call).
// The scores' accumulators hold [key g][n 2c, 2c + 1]; a transposing move makes them the B operand
// of the value products.  Warps keep their own maximum; the sums meet in shared memory, the splits in global memory, where
// the block that arrives last adds them in order.
// About 14 instructions per key of eight heads where the form before it (heads as the rows of A: half of them idle, one byte
// used of every word loaded, three barriers per tile of 128 keys) took some 60.
__device__ __forceinline__ void qa_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t qa_transpose(uint32_t v) {  // of the warp's 8 x 8 matrix of 16-bit values
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t qa_pack_f16(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float2 qa_unpack_f16(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2 *>(&v)); }
__device__ __forceinline__ float qa_exp2(float x) {  // 2 to the x, relative error below 2^-22; 0 for -infinity
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// p * s has to pass through float16.  The exponents' reference point is therefore placed by the value scales too: with
// 2^k the power of two at or above the largest scale met so far, the largest p * s lies between 2^11 and 2^15, 25 binary
// orders above float16's subnormals.  (With p <= 1 as the softmax has it, values of magnitude 10^-3 lose most of their codes:
// relative error 0.86 at 16K keys, 8 bits.)  It is a score plus a whole number: the key that set it has a power of two for its p,
// and so an exact p * s (whole reference points: peaked scores 8e-4 off instead of 5e-4).
constexpr float QA_SLACK = 3.0f, QA_TOP = 15.0f;  // room above the largest score when the reference moves; log2 of the largest p * s
// Scales outside are taken as these: 2^(QA_TOP - k) * p, its sums, and its products with biases of up to 2^86 stay in float32's range.
constexpr int QA_K_MIN = -26, QA_K_MAX = 55;
__device__ __forceinline__ int qa_log2_ceil(float s) {  // of s >= 0, in [QA_K_MIN, QA_K_MAX]
    const uint32_t u = __float_as_uint(s);
    return min(max((int)(u >> 23) - 127 + ((u & 0x7FFFFFu) != 0u ? 1 : 0), QA_K_MIN), QA_K_MAX);
}
__device__ __forceinline__ uint32_t qa_nibbles(uint32_t v) { return (v & 0x000F000Fu) | 0x64006400u; }
template <int WORDS> __device__ __forceinline__ void qa_load(const void *src, uint32_t *dst) {
    if constexpr (WORDS == 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(src);
        dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
    } else if constexpr (WORDS == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(src);
        dst[0] = v.x; dst[1] = v.y;
    } else {
        dst[0] = *reinterpret_cast<const uint32_t *>(src);
    }
}
// G consecutive 16-bit scales (at a shared-memory address) as floats
template <typename T, int G> struct QaScales {
    static_assert(G == 1 || G == 2 || G == 4, "groups of a head");
    uint32_t raw[G == 4 ? 2 : 1];
    __device__ __forceinline__ void load(const char *row) {
        if constexpr (G == 1) raw[0] = *reinterpret_cast<const uint16_t *>(row);
        else qa_load<G / 2>(row, raw);
    }
    __device__ __forceinline__ float get(int g) const {
        const uint16_t h = (uint16_t)(raw[g >> 1] >> (16 * (g & 1)));
        return DT<T>::load(reinterpret_cast<const T *>(&h), 0);
    }
    // the magnitudes here and in `other`, as the larger of each pair of half words: their bits are in order
    __device__ __forceinline__ uint32_t largest(const QaScales &other) const {
        uint32_t u = __vmaxu2(raw[0] & 0x7FFF7FFFu, other.raw[0] & 0x7FFF7FFFu);
        if (G == 4) u = __vmaxu2(u, __vmaxu2(raw[G / 4] & 0x7FFF7FFFu, other.raw[G / 4] & 0x7FFF7FFFu));
        return u;
    }
};
// k of the larger of two magnitudes (zero, infinities and NaN: no scale to go by), and 2^k as both half words
template <typename T> __device__ __forceinline__ int qa_scale_k(uint32_t pair) {
    constexpr uint32_t INF = std::is_same<T, __half>::value ? 0x7C00u : 0x7F80u;
    const uint32_t a = pair >> 16, b = pair & 0xFFFFu;
    const uint16_t h = (uint16_t)max(a < INF ? a : 0u, b < INF ? b : 0u);
    return qa_log2_ceil(DT<T>::load(reinterpret_cast<const T *>(&h), 0));
}
template <typename T> __device__ __forceinline__ uint32_t qa_scale_pair(int k) {
    T h[2];
    DT<T>::store(h, 0, __uint_as_float((uint32_t)(k + 127) << 23));
    h[1] = h[0];
    return *reinterpret_cast<const uint32_t *>(h);
}

constexpr int QM_WARPS = 8, QM_THREADS = QM_WARPS * 32, QM_STEP = 16;  // keys per step of a warp
constexpr int QM_BLOCKS_PER_SM = 2;

// A warp's ring: a stage holds 16 rows of keys, of values, and the four scale arrays' 16 x G values (each in a piece of its own
// with a word of slack: rows of one group start at any half word).
template <int BITS, int D, int GS> struct QmRing {
    static constexpr int G = D / GS, ROW = D * BITS / 8, CODES = QM_STEP * ROW, SPIECE = QM_STEP * 2 * G + (G == 1 ? 16 : 0);
    static constexpr int STAGE = 2 * CODES + 4 * SPIECE;
    static constexpr int FIT = 108 * 1024 / (QM_WARPS * STAGE);
    static constexpr int STAGES = FIT < 6 ? FIT : 6;
    static_assert(STAGES >= 3, "the ring");
    static constexpr int MERGE = QM_WARPS * 8 * D * 4;  // the warps' sums at the end, in the same memory
    static constexpr size_t SMEM = QM_WARPS * STAGES * STAGE > MERGE ? QM_WARPS * STAGES * STAGE : MERGE;
    // Byte offset of 16-byte chunk `chunk` of row `row` of the keys (keys 2i and 2i + 1 read together: rows of 128 bytes swap
    // halves, rows of 64 fall side by side, shorter rows are read four at a time) and of the values (rows 2c read together).
    static __device__ __forceinline__ int key_at(int row, int chunk) {
        return row * ROW + ((ROW == 128 ? chunk ^ ((row & 1) << 2) : chunk) << 4);
    }
    static __device__ __forceinline__ int value_at(int row, int chunk) {
        return row * ROW + ((ROW == 128 ? chunk ^ (((row >> 1) & 3) << 1) : ROW == 64 ? chunk ^ ((row >> 2) & 1) << 1 : chunk) << 4);
    }
};
template <int BYTES> __device__ __forceinline__ void qa_cp_async(uint32_t dst, const void *src) {
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

template <typename T, int BITS, int D, int GS>
__global__ void __launch_bounds__(QM_THREADS, QM_BLOCKS_PER_SM) qattn_mma_kernel(QAttnParams p) {
    static_assert(BITS == 4 || BITS == 8, "codes that fill bytes");
    constexpr int G = D / GS, W = D * BITS / 32, GW = GS * BITS / 32;  // groups; words of a row, of a group
    constexpr int KWD = GW / 4;                                        // words of a group per lane, scores
    constexpr int VB = GW / 2;                                         // bytes of a group per lane, values
    constexpr int VWD = VB >= 4 ? VB / 4 : 1, KS = GS / 16, MT = GS / 16;
    constexpr uint32_t MAGIC = 0x64646464u;
    const int split = blockIdx.x, hk = blockIdx.y, b = blockIdx.z / p.row_tiles, lt = blockIdx.z % p.row_tiles;
    const int rep = p.Hq / p.Hkv, t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, c = lane & 3;
    const int s0 = split * p.chunk, s1 = min(p.S, s0 + p.chunk);
    // column n of the products: query row l0 + n / rep of head hk * rep + n % rep; its keys end before `limit`
    const int l0 = lt * p.row_pack;
    auto limit_of = [&](int n) {
        const int l = l0 + n / rep;
        return p.causal && n < rep * p.row_pack && l < p.L ? p.S - (p.L - 1 - l) : p.S;  // (columns that stand for nothing: any value)
    };
    if (!p.early) pdl_wait();
    pdl_trigger();

    // This split's rows, addressed from its first by 32-bit byte offsets.
    const size_t row0 = ((size_t)b * p.Hkv + hk) * p.capacity + s0;
    const char *kbase = reinterpret_cast<const char *>(p.kw + row0 * W), *vbase = reinterpret_cast<const char *>(p.vw + row0 * W);
    const char *ksb = (const char *)p.ks + row0 * (2 * G), *kbb = (const char *)p.kb + row0 * (2 * G);
    const char *vsb = (const char *)p.vs + row0 * (2 * G), *vbb = (const char *)p.vb + row0 * (2 * G);
    const int last = s1 - s0 - 1;
    // word of a group that lane c's word j is (a 16-byte piece of either half when a lane's share is 32 bytes)
    auto kword = [&](int j) { return KWD == 8 ? (j >> 2) * 16 + c * 4 + (j & 3) : c * KWD + j; };
    // the warp's ring
    using R = QmRing<BITS, D, GS>;
    constexpr int STAGES = R::STAGES, CHUNKS = R::ROW / 16;
    extern __shared__ __align__(128) char qm_smem[];
    char *ring = qm_smem + warp * (STAGES * R::STAGE);
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    // half words by which the scale arrays' first rows miss a word (one group: rows of two bytes)
    const uint32_t off[4] = {G == 1 ? (uint32_t)(uintptr_t)ksb & 2u : 0u, G == 1 ? (uint32_t)(uintptr_t)kbb & 2u : 0u,
                             G == 1 ? (uint32_t)(uintptr_t)vsb & 2u : 0u, G == 1 ? (uint32_t)(uintptr_t)vbb & 2u : 0u};
    // Requests the 16 rows from `key0` on (rows past the end repeat the last one: their columns are
    // masked) and closes the group.
    auto request = [&](int key0, int stage) {
        if (key0 <= last) {
            const uint32_t dst = ring_s + stage * R::STAGE;
#pragma unroll
            for (int i = 0; i < QM_STEP * CHUNKS / 32; i++) {
                const int at = i * 32 + lane, row = at / CHUNKS, chunk = at % CHUNKS;
                const uint32_t src = (uint32_t)min(key0 + row, last) * (uint32_t)R::ROW + (uint32_t)(chunk * 16);
                qa_cp_async<16>(dst + R::key_at(row, chunk), kbase + src);
                qa_cp_async<16>(dst + R::CODES + R::value_at(row, chunk), vbase + src);
            }
            // the scales: words, clamped to the last row's (one group: the words around the rows)
            constexpr int SW = QM_STEP * G / 2 + (G == 1 ? 1 : 0);  // words of an array
#pragma unroll
            for (int i = 0; i < (4 * SW + 31) / 32; i++) {
                const int at = i * 32 + lane, array = at / SW, word = at % SW;
                if (at < 4 * SW) {
                    const char *base = array == 0 ? ksb : array == 1 ? kbb : array == 2 ? vsb : vbb;
                    const uint32_t o = G == 1 ? (uint32_t)(uintptr_t)base & 2u : 0u;
                    const uint32_t end = ((uint32_t)last * (2 * G) + 2 * G - 1 + o) / 4;  // the word of the last row's last value
                    const uint32_t w = min((uint32_t)key0 * (2 * G) / 4 + (uint32_t)word, end);
                    qa_cp_async<4>(dst + 2 * R::CODES + array * R::SPIECE + word * 4, base - o + w * 4);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int first = warp * QM_STEP;
    constexpr int STRIDE = QM_WARPS * QM_STEP;
#pragma unroll
    for (int i = 0; i < STAGES - 1; i++) request(first + i * STRIDE, i);
    if (p.early) pdl_wait();  // (the caches may be read ahead of it, the queries not)

    // the scaled queries (in units of log2) as B fragments, and their sums per group (of the rounded values)
    uint32_t qf[G][KS][2];
    float qs[G][2];  // of columns 2c, 2c + 1
    {
        const int l = l0 + g / rep;
        const bool have = g < rep * p.row_pack && l < p.L;
        const T *q = (const T *)p.q + (((size_t)b * p.Hq + hk * rep + (have ? g % rep : 0)) * p.L + (have ? l : 0)) * D;
        const float f = have ? p.scale * 1.4426950408889634f : 0.0f;
#pragma unroll
        for (int gr = 0; gr < G; gr++) {
            float sum = 0.0f;
            constexpr int PER = 32 / BITS;  // codes of a word
#pragma unroll
            for (int j = 0; j < KWD; j++) {
                uint32_t raw[PER / 2];
                qa_load<PER / 2>(q + gr * GS + kword(j) * PER, raw);
                const T *v = reinterpret_cast<const T *>(raw);
                auto pair = [&](int ks, int i, int lo, int hi) {
                    qf[gr][ks][i] = qa_pack_f16(DT<T>::load(v, lo) * f, DT<T>::load(v, hi) * f);
                    const float2 u = qa_unpack_f16(qf[gr][ks][i]);
                    sum += u.x + u.y;
                };
                if constexpr (BITS == 8) {
                    pair(j, 0, 0, 1);
                    pair(j, 1, 2, 3);
                } else {
                    pair(2 * j, 0, 0, 4);
                    pair(2 * j, 1, 1, 5);
                    pair(2 * j + 1, 0, 2, 6);
                    pair(2 * j + 1, 1, 3, 7);
                }
            }
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            qs[gr][0] = __shfl_sync(0xFFFFFFFFu, sum, 8 * c);
            qs[gr][1] = __shfl_sync(0xFFFFFFFFu, sum, 8 * c + 4);
        }
    }
    const int limit[2] = {limit_of(2 * c) - s0, limit_of(2 * c + 1) - s0};
    const int all_of = min(s1, p.causal ? p.S - (p.L - 1 - l0) : p.S) - s0;  // every column attends to the keys before this one

    // top: no score so far is above it; ref = top - (QA_TOP - k): the reference point of the exponents
    float top[2] = {-INFINITY, -INFINITY}, ref[2] = {0.0f, 0.0f}, l[2] = {0.0f, 0.0f};  // of columns 2c, 2c + 1 (l: this lane's keys only)
    int k = QA_K_MIN;
    uint32_t largest = 0u;  // 2^k in the scales' type, twice (0 to begin with)
    float o[G][MT][4], side[G][2];
#pragma unroll
    for (int gr = 0; gr < G; gr++) {
        side[gr][0] = side[gr][1] = 0.0f;
#pragma unroll
        for (int i = 0; i < MT; i++) o[gr][i][0] = o[gr][i][1] = o[gr][i][2] = o[gr][i][3] = 0.0f;
    }

    int stage = 0, refill = STAGES - 1;
    for (int key0 = first; key0 <= last; key0 += STRIDE) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();  // every lane's copies are visible, and every lane is through with the stage refilled next
        request(key0 + (STAGES - 1) * STRIDE, refill);
        const char *at = ring + stage * R::STAGE;
        if (++stage == STAGES) stage = 0;
        if (++refill == STAGES) refill = 0;
        uint32_t kq[2][G][KWD], vq[4][G][VWD];
        QaScales<T, G> ksc[2], kbi[2], vsc[2], vbi[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
#pragma unroll
            for (int gr = 0; gr < G; gr++) {
#pragma unroll
                for (int j = 0; j < (KWD + 3) / 4; j++) {  // byte of the row: group, then (32 bytes per lane) half, then lane
                    const int byte = gr * GW * 4 + (KWD == 8 ? j * 64 + c * 16 : c * KWD * 4);
                    qa_load<KWD < 4 ? KWD : 4>(at + R::key_at(g + 8 * r, byte >> 4) + (byte & 15), kq[r][gr] + 4 * j);
                }
            }
            ksc[r].load(at + 2 * R::CODES + off[0] + (g + 8 * r) * 2 * G);
            kbi[r].load(at + 2 * R::CODES + R::SPIECE + off[1] + (g + 8 * r) * 2 * G);
        }
        // ── scores of 16 keys ──
        float sc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // [key g: n 2c, 2c + 1][key g + 8: ...]
#pragma unroll
        for (int gr = 0; gr < G; gr++) {
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                uint32_t a[4];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if (BITS == 8) {
                        a[r] = __byte_perm(kq[r][gr][ks], MAGIC, 0x4140);
                        a[r + 2] = __byte_perm(kq[r][gr][ks], MAGIC, 0x4342);
                    } else {
                        const uint32_t w = kq[r][gr][ks >> 1];
                        a[r] = qa_nibbles(w >> (8 * (ks & 1)));
                        a[r + 2] = qa_nibbles(w >> (8 * (ks & 1) + 4));
                    }
                }
                qa_mma(acc, a[0], a[1], a[2], a[3], qf[gr][ks][0], qf[gr][ks][1]);
            }
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const float s = ksc[r].get(gr), bi = kbi[r].get(gr);
#pragma unroll
                for (int i = 0; i < 2; i++)
                    sc[2 * r + i] = fmaf(s, fmaf(-1024.0f, qs[gr][i], acc[2 * r + i]), fmaf(bi, qs[gr][i], sc[2 * r + i]));
            }
        }
        // ── probabilities ──
        if (key0 + QM_STEP > all_of) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (key0 + g + 8 * (i >> 1) >= min(limit[i & 1], last + 1)) sc[i] = -INFINITY;
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            vsc[r].load(at + 2 * R::CODES + 2 * R::SPIECE + off[2] + (g + 8 * r) * 2 * G);
            vbi[r].load(at + 2 * R::CODES + 3 * R::SPIECE + off[3] + (g + 8 * r) * 2 * G);
            // one group: the last row's word also holds a value that is not the cache's; a probability of zero times that may be NaN
            if (G == 1 && key0 + g + 8 * r > last) vsc[r].raw[0] = vbi[r].raw[0] = 0u;
        }
        // The exponents' reference point moves only when a score passes `top`, which has QA_SLACK of room when it is set, or a
        // scale the largest so far: rescaling the outputs at every new maximum, and finding it across the lanes, took a third of
        // the step.
        const float mx[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};
        const uint32_t vs = vsc[0].largest(vsc[1]);
        if (__any_sync(0xFFFFFFFFu, mx[0] > top[0] || mx[1] > top[1] || __vmaxu2(vs, largest) != largest)) {
            float corr[2];
            k = max(k, __reduce_max_sync(0xFFFFFFFFu, qa_scale_k<T>(vs)));
            largest = qa_scale_pair<T>(k);
            const float head = QA_TOP - (float)k;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float n = mx[i];
#pragma unroll
                for (int s = 4; s < 32; s <<= 1) n = fmaxf(n, __shfl_xor_sync(0xFFFFFFFFu, n, s));
                n = n > top[i] ? n + QA_SLACK : top[i];
                const float to = n == -INFINITY ? 0.0f : n - head;
                corr[i] = top[i] == -INFINITY ? 0.0f : qa_exp2(ref[i] - to);
                top[i] = n;
                ref[i] = to;
                l[i] *= corr[i];
            }
#pragma unroll
            for (int gr = 0; gr < G; gr++) {
                side[gr][0] *= corr[0];
                side[gr][1] *= corr[1];
#pragma unroll
                for (int i = 0; i < MT; i++) {
                    o[gr][i][0] *= corr[0]; o[gr][i][1] *= corr[1];
                    o[gr][i][2] *= corr[0]; o[gr][i][3] *= corr[1];
                }
            }
        }
        float pr[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            pr[i] = qa_exp2(sc[i] - ref[i & 1]);
            l[i & 1] += pr[i];
        }
        // ── values ──
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int gr = 0; gr < G; gr++) {
                const int row = 2 * c + (i & 1) + 8 * (i >> 1), byte = gr * GW * 4 + g * VB;
                const char *src = at + R::CODES + R::value_at(row, byte >> 4) + (byte & 15);
                if constexpr (VB == 2) vq[i][gr][0] = *reinterpret_cast<const uint16_t *>(src);
                else qa_load<VWD>(src, vq[i][gr]);
            }
#pragma unroll
        for (int gr = 0; gr < G; gr++) {
            uint32_t bf[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const float s = vsc[r].get(gr), bi = vbi[r].get(gr);
                const uint32_t ps = qa_pack_f16(pr[2 * r] * s, pr[2 * r + 1] * s);
                const float2 u = qa_unpack_f16(ps);
                side[gr][0] += fmaf(-1024.0f, u.x, pr[2 * r] * bi);
                side[gr][1] += fmaf(-1024.0f, u.y, pr[2 * r + 1] * bi);
                bf[r] = qa_transpose(ps);
            }
#pragma unroll
            for (int i = 0; i < MT; i++) {
                uint32_t a[4];
#pragma unroll
                for (int h = 0; h < 2; h++) {  // keys 2c, 2c + 1; then 2c + 8, 2c + 9
                    if (BITS == 8) {
                        const uint32_t tt = __byte_perm(vq[2 * h][gr][i >> 1], vq[2 * h + 1][gr][i >> 1], (i & 1) ? 0x7362 : 0x5140);
                        a[2 * h] = __byte_perm(tt, MAGIC, 0x4140);
                        a[2 * h + 1] = __byte_perm(tt, MAGIC, 0x4342);
                    } else {
                        const uint32_t tt = __byte_perm(vq[2 * h][gr][i >> 2], vq[2 * h + 1][gr][i >> 2], (i & 2) ? 0x7632 : 0x5410);
                        a[2 * h] = qa_nibbles(tt >> (8 * (i & 1)));
                        a[2 * h + 1] = qa_nibbles(tt >> (8 * (i & 1) + 4));
                    }
                }
                qa_mma(o[gr][i], a[0], a[1], a[2], a[3], bf[0], bf[1]);
            }
        }
    }

    // ── the warps' sums together ──
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the rings become the merge's memory
    float(*wsum)[8][D] = reinterpret_cast<float(*)[8][D]>(qm_smem);
    __shared__ float wm[QM_WARPS][8], wl[QM_WARPS][8];
    __shared__ float weight[QM_WARPS][8], total[2][8];
    __shared__ int is_last;
#pragma unroll
    for (int s = 4; s < 32; s <<= 1) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            l[i] += __shfl_xor_sync(0xFFFFFFFFu, l[i], s);
#pragma unroll
            for (int gr = 0; gr < G; gr++) side[gr][i] += __shfl_xor_sync(0xFFFFFFFFu, side[gr][i], s);
        }
    }
#pragma unroll
    for (int gr = 0; gr < G; gr++)
#pragma unroll
        for (int i = 0; i < MT; i++) {
            const int d = gr * GS + g * (GS / 8) + 2 * i;
#pragma unroll
            for (int n = 0; n < 2; n++)
                *reinterpret_cast<float2 *>(&wsum[warp][2 * c + n][d]) = make_float2(o[gr][i][n] + side[gr][n], o[gr][i][n + 2] + side[gr][n]);
        }
    if (g == 0) {
#pragma unroll
        for (int n = 0; n < 2; n++) {
            wm[warp][2 * c + n] = top[n] == -INFINITY ? -INFINITY : ref[n];
            wl[warp][2 * c + n] = l[n];
        }
    }
    __syncthreads();
    if (t < 8) {
        float mx = -INFINITY, sum = 0.0f;
        for (int w = 0; w < QM_WARPS; w++) mx = fmaxf(mx, wm[w][t]);
        for (int w = 0; w < QM_WARPS; w++) {
            const float f = wm[w][t] == -INFINITY ? 0.0f : qa_exp2(wm[w][t] - mx);
            weight[w][t] = f;
            sum = fmaf(wl[w][t], f, sum);
        }
        total[0][t] = mx;
        total[1][t] = sum;
    }
    __syncthreads();
    const int cols = min(rep * p.row_pack, rep * (p.L - l0));
    // output row of column n
    auto row_of = [&](int n) { return ((size_t)b * p.Hq + hk * rep + n % rep) * p.L + l0 + n / rep; };
    // the sink joins the denominator; then the quotient, rounded
    auto finish = [&](int n, int d, float4 v, float mx, float sum) {
        if (p.sinks) {
            const float sv = DT<T>::load((const T *)p.sinks, hk * rep + n % rep) * 1.4426950408889634f, nm = fmaxf(mx, sv);
            const float f = mx == -INFINITY ? 0.0f : qa_exp2(mx - nm);
            v.x *= f; v.y *= f; v.z *= f; v.w *= f;
            sum = fmaf(sum, f, qa_exp2(sv - nm));
        }
        T h[4];
        const float q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) DT<T>::store(h, i, sum > 0.0f ? __fdiv_rn(q[i], sum) : 0.0f);
        *reinterpret_cast<uint2 *>((T *)p.out + row_of(n) * D + d) = *reinterpret_cast<const uint2 *>(h);
    };
    constexpr int PITCH = D + 4;  // floats per split and row: the sums, then maximum and denominator
    for (int i = t; i < cols * (D / 4); i += QM_THREADS) {
        const int n = i / (D / 4), d = i % (D / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < QM_WARPS; w++) {
            const float4 u = *reinterpret_cast<const float4 *>(&wsum[w][n][d]);
            const float f = weight[w][n];
            v.x = fmaf(u.x, f, v.x); v.y = fmaf(u.y, f, v.y); v.z = fmaf(u.z, f, v.z); v.w = fmaf(u.w, f, v.w);
        }
        if (p.splits == 1) finish(n, d, v, total[0][n], total[1][n]);
        else {
            float *dst = p.part + (row_of(n) * p.splits + split) * PITCH;
            __stcg(reinterpret_cast<float4 *>(dst + d), v);
            if (d == 0) __stcg(reinterpret_cast<float2 *>(dst + D), make_float2(total[0][n], total[1][n]));
        }
    }
    if (p.splits == 1) return;

    // ── the splits together, by the block that arrives last ──
    __syncthreads();
    if (t == 0) {
        __threadfence();  // (after the barrier: the whole block's stores come before the arrival)
        uint32_t *counter = p.counters + ((size_t)blockIdx.z * gridDim.y + hk);
        is_last = atomicAdd(counter, 1u) == (uint32_t)p.splits - 1;
        if (is_last) *counter = 0u;
        __threadfence();
    }
    __syncthreads();
    if (!is_last) return;
    // Two threads per four outputs, each every other split, sixteen loads in flight; the first ones travel while one warp per
    // column finds the maximum and the denominator and leaves the splits' weights in shared memory.
    float *sw = &wsum[0][0][0];  // [8][splits]: splits are at most 8 * D
    constexpr int ITEMS = QM_THREADS / 2, BATCH = 16;
    const int items = cols * (D / 4);
    float4 u[BATCH];
    auto fetch = [&](int i, int j0) {
        const float *src = p.part + row_of(min(i / (D / 4), cols - 1)) * p.splits * PITCH + i % (D / 4) * 4;
#pragma unroll
        for (int j = 0; j < BATCH; j++) u[j] = __ldcg(reinterpret_cast<const float4 *>(src + (size_t)min(j0 + 2 * j, p.splits - 1) * PITCH));
    };
    fetch(t >> 1, t & 1);
    if (warp < cols) {
        const float *src = p.part + row_of(warp) * p.splits * PITCH + D;
        float mx = -INFINITY;
        for (int j = lane; j < p.splits; j += 32) mx = fmaxf(mx, __ldcg(src + (size_t)j * PITCH));
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, s));
        float sum = 0.0f;
        for (int j = lane; j < p.splits; j += 32) {
            const float2 v = __ldcg(reinterpret_cast<const float2 *>(src + (size_t)j * PITCH));
            const float f = v.x == -INFINITY ? 0.0f : qa_exp2(v.x - mx);
            sw[warp * p.splits + j] = f;
            sum = fmaf(v.y, f, sum);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, s);
        if (lane == 0) {
            total[0][warp] = mx;
            total[1][warp] = sum;
        }
    }
    __syncthreads();
    for (int i0 = 0; i0 < items; i0 += ITEMS) {
        const int i = i0 + (t >> 1), n = min(i / (D / 4), cols - 1), d = i % (D / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j0 = t & 1; j0 < p.splits; j0 += 2 * BATCH) {
            if (i0 != 0 || j0 >= 2) fetch(i, j0);
#pragma unroll
            for (int j = 0; j < BATCH; j++)
                if (j0 + 2 * j < p.splits) {
                    const float f = sw[n * p.splits + j0 + 2 * j];
                    v.x = fmaf(u[j].x, f, v.x); v.y = fmaf(u[j].y, f, v.y); v.z = fmaf(u[j].z, f, v.z); v.w = fmaf(u[j].w, f, v.w);
                }
        }
        v.x += __shfl_xor_sync(0xFFFFFFFFu, v.x, 1); v.y += __shfl_xor_sync(0xFFFFFFFFu, v.y, 1);
        v.z += __shfl_xor_sync(0xFFFFFFFFu, v.z, 1); v.w += __shfl_xor_sync(0xFFFFFFFFu, v.w, 1);
        if ((t & 1) == 0 && i < items) finish(n, d, v, total[0][n], total[1][n]);
    }
}

// ── the tensor-core form for short caches ──────────────────────────────────────────────────────────────
// The same products with the key head's query heads as the rows of A (8 of the 16 at most are used).  A warp owns 32 keys of a
// tile of 128: its score accumulators (16 heads x 8 keys) are, pairwise, exactly the A fragments (16 heads x 16 keys) of its
// value products, so the probabilities never leave registers; the four warps' outputs are added at the end.  A tile's codes
// travel into shared memory with cp.async a tile ahead (two sets of buffers), its scales and biases through registers; the
// splits are merged by qattn_combine.  See qattn_form for when it runs.
constexpr int QT_BLOCKS = 3, QT_PLAIN = 7;
__device__ __forceinline__ float qa_inverse(float x) { return __uint_as_float((254u << 23) - __float_as_uint(x)); }  // of a power of two
__device__ __forceinline__ void qa_cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ size_t head_row_of(const QAttnParams &p, int b, int hk) { return ((size_t)b * p.Hkv + hk) * p.capacity; }
template <int BITS, int D, int GS> constexpr size_t qt_smem() {
    constexpr int W = D * BITS / 32, TILE_WORDS = QA_TILE * (W + 4), RWORDS = 4 * 8 * D;
    return (size_t)(2 * TILE_WORDS + (2 * TILE_WORDS > RWORDS ? 2 * TILE_WORDS : RWORDS)) * 4 + 2 * QA_TILE * (D / GS) * 16;
}

template <typename T, int BITS, int D, int GS>
__global__ void __launch_bounds__(QA_THREADS, QT_BLOCKS) qattn_tile_kernel(QAttnParams p) {
    static_assert(BITS == 4 || BITS == 8, "codes that fill bytes");
    constexpr int W = D * BITS / 32, G = D / GS, KS = D / 16, NBD = D / 8, WP = W + 4;  // WP: padded row of the value tile
    constexpr int KS_PER_G = GS / 16, NBD_PER_G = GS / 8;
    if (!p.early) pdl_wait();
    pdl_trigger();  // the combine kernel's blocks may become resident meanwhile
    const int split = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    const int rep = p.Hq / p.Hkv, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int g8 = lane >> 2, c = lane & 3;  // the fragments' group (a head, a key or a dim) and pair index
    const int s0 = split * p.chunk, s1 = min(p.S, s0 + p.chunk);
    const bool head = g8 < rep;

    // Two sets of tile buffers: the next tile's codes arrive (cp.async) while the current tile multiplies.  Rows are
    // padded by four words: the eight rows (keys) or four rows (values) a fragment reads at once fall into distinct banks.
    __shared__ float wred[2][4][8];
    constexpr int KP = W + 4;
    constexpr int TILE_WORDS = QA_TILE * KP, RWORDS = 4 * 8 * D;
    extern __shared__ __align__(16) uint32_t qa_dyn[];
    uint32_t *kbuf = qa_dyn;                        // [2][QA_TILE * KP]
    uint32_t *vbuf = kbuf + 2 * TILE_WORDS;         // [2][QA_TILE * WP]; after the last tile the warps' sums [4][8][D]
    float4 *sbuf = reinterpret_cast<float4 *>(vbuf + (2 * TILE_WORDS > RWORDS ? 2 * TILE_WORDS : RWORDS));  // [2][QA_TILE][G]
    auto fetch_codes = [&](int base, int buf) {
        const int keys = min(QA_TILE, s1 - base);
        const uint32_t *ksrc = p.kw + (head_row_of(p, b, hk) + base) * W, *vsrc = p.vw + (head_row_of(p, b, hk) + base) * W;
        for (int i = t; i < keys * W / 4; i += QA_THREADS) {
            const int row = (4 * i) / W, col = (4 * i) % W;
            qa_cp16(kbuf + buf * TILE_WORDS + row * KP + col, ksrc + 4 * i);
            qa_cp16(vbuf + buf * TILE_WORDS + row * WP + col, vsrc + 4 * i);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch_scales = [&](int base, float4 (&r)[G]) {  // thread t: key t of the tile
        const int keys = min(QA_TILE, s1 - base);
#pragma unroll
        for (int g = 0; g < G; g++) {
            const size_t at = (head_row_of(p, b, hk) + base + min(t, keys - 1)) * G + g;
            r[g] = make_float4(DT<T>::load((const T *)p.ks, at), DT<T>::load((const T *)p.kb, at), DT<T>::load((const T *)p.vs, at),
                               DT<T>::load((const T *)p.vb, at));
        }
    };

    // The first tile's codes and scales start before the kernel in front has finished, unless it may be writing them.
    float4 nsb[G];
    if (s0 < s1) {
        fetch_codes(s0, 0);
        fetch_scales(s0, nsb);
    }
    if (p.early) pdl_wait();
    // the head's scaled queries as A fragments, and their sums per group (of the rounded values)
    uint32_t qa0[KS], qa2[KS];
    float qsum[G];
#pragma unroll
    for (int g = 0; g < G; g++) qsum[g] = 0.0f;
    {
        const T *q = (const T *)p.q + (((size_t)b * p.Hq + hk * rep + (head ? g8 : 0)) * p.L + p.l) * D;
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
            const int d = 16 * ks + 2 * c;
            qa0[ks] = head ? qa_pack_f16(DT<T>::load(q, d) * p.scale, DT<T>::load(q, d + 1) * p.scale) : 0u;
            qa2[ks] = head ? qa_pack_f16(DT<T>::load(q, d + 8) * p.scale, DT<T>::load(q, d + 9) * p.scale) : 0u;
            const float2 u = qa_unpack_f16(qa0[ks]), v = qa_unpack_f16(qa2[ks]);
            qsum[ks / KS_PER_G] += (u.x + u.y) + (v.x + v.y);
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            qsum[g] += __shfl_xor_sync(0xFFFFFFFFu, qsum[g], 1);
            qsum[g] += __shfl_xor_sync(0xFFFFFFFFu, qsum[g], 2);
        }
    }

    float m = -INFINITY, l = 0.0f;  // of head g8
    float oc[NBD][4], side[G];      // outputs times `lift` [head g8][dims 8 nbd + 2 c, + 1] (rows 8-15 idle); bias / offset terms per group, too
    float lift = 0x1p+100f, turn = 1.0f;  // what the warp's value scales and biases are multiplied by; what it changes by at the next tile
#pragma unroll
    for (int i = 0; i < NBD; i++) oc[i][0] = oc[i][1] = oc[i][2] = oc[i][3] = 0.0f;
#pragma unroll
    for (int g = 0; g < G; g++) side[g] = 0.0f;

    // Leaves a tile's scales in shared memory; a warp's threads hold the scales of the keys whose values it multiplies.  Value scales
    // of at most 2^-QT_PLAIN are lifted, by as much for all the warp's keys so far, so that p * s keeps its bits as in the ring form.
    // Above it does as it is: only p below 2^(QT_PLAIN - 14) fall among float16's subnormals, whose rounding (2^-25) is
    // 2^(QT_PLAIN - 25) of the largest term.
    auto keep_scales = [&](int to) {
        float most = 0.0f;
#pragma unroll
        for (int g = 0; g < G; g++) most = fmaxf(most, fabsf(nsb[g].z));
        const int k = qa_log2_ceil(__uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(most))));
        const float up = fminf(k > -QT_PLAIN ? 1.0f : __uint_as_float((uint32_t)((int)QA_TOP - k + 127) << 23), lift);
        turn = up * qa_inverse(lift);  // (at the first tile there is nothing to turn)
        lift = up;
#pragma unroll
        for (int g = 0; g < G; g++) sbuf[(to * QA_TILE + t) * G + g] = make_float4(nsb[g].x, nsb[g].y, nsb[g].z * up, nsb[g].w * up);
    };
    if (s0 < s1) keep_scales(0);
    int buf = 0;
    for (int base = s0; base < s1; base += QA_TILE, buf ^= 1) {
        const int keys = min(QA_TILE, s1 - base);
        const bool more = base + QA_TILE < s1;
        // the next tile's codes start travelling into the other buffers, its scales into registers
        if (more) {
            fetch_codes(base + QA_TILE, buf ^ 1);
            fetch_scales(base + QA_TILE, nsb);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t *ktile = kbuf + buf * TILE_WORDS, *vtile = vbuf + buf * TILE_WORDS;
        const float4(*sbt)[G] = reinterpret_cast<const float4(*)[G]>(sbuf + buf * QA_TILE * G);
        // ── scores of the warp's 32 keys: four blocks of 8 keys ──
        float sc[4][2];
#pragma unroll
        for (int nb = 0; nb < 4; nb++) {
            const int kfrag = warp * 32 + nb * 8;                       // first key of the block, within the tile
            const int krow = min(kfrag + g8, keys - 1);                 // the key whose codes this lane feeds (clamped: masked below)
            const uint32_t *row = ktile + krow * KP;
            float cg[G][4];
#pragma unroll
            for (int g = 0; g < G; g++) cg[g][0] = cg[g][1] = cg[g][2] = cg[g][3] = 0.0f;
#pragma unroll
            for (int q4 = 0; q4 < W / 4; q4++) {
                const uint4 v = reinterpret_cast<const uint4 *>(row)[q4];
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                if (BITS == 4) {
                    // words 4 q4 .. + 3 = dims 32 q4 .. + 31 = two steps of 16 dims; the lane's codes are byte c of every word
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        const int ks = 2 * q4 + half;
                        uint32_t bf[2];
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            const uint32_t byte = __byte_perm(w[2 * half + j], 0, 0x4440 | c);
                            bf[j] = ((byte | (byte << 12)) & 0x000F000Fu) | 0x64006400u;
                        }
                        qa_mma(cg[ks / KS_PER_G], qa0[ks], 0u, qa2[ks], 0u, bf[0], bf[1]);
                    }
                } else {
                    // words 4 q4 .. + 3 = dims 16 q4 .. + 15 = one step; dims 2 c, 2 c + 1 are a half of word c / 2, dims + 8 of word 2 + c / 2
                    const int ks = q4;
                    const uint32_t lo = (c & 2) ? w[1] : w[0], hi = (c & 2) ? w[3] : w[2];
                    const uint32_t sel = (c & 1) ? 0x4342u : 0x4140u;
                    qa_mma(cg[ks / KS_PER_G], qa0[ks], 0u, qa2[ks], 0u, __byte_perm(lo, 0, sel) | 0x64006400u, __byte_perm(hi, 0, sel) | 0x64006400u);
                }
            }
            // the C fragment holds [head g8][keys kfrag + 2 c, + 1]
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int key = min(kfrag + 2 * c + j, keys - 1);
                float sv = 0.0f;
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const float4 sb = sbt[key][g];
                    sv = fmaf(sb.x, cg[g][j] - 1024.0f * qsum[g], fmaf(sb.y, qsum[g], sv));
                }
                sc[nb][j] = sv;
            }
        }
        // ── running maximum and denominator of head g8 ──
        float tmax = -INFINITY;
#pragma unroll
        for (int nb = 0; nb < 4; nb++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const bool valid = head && warp * 32 + nb * 8 + 2 * c + j < keys;
                if (!valid) sc[nb][j] = -INFINITY;
                tmax = fmaxf(tmax, sc[nb][j]);
            }
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 1));
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 2));
        if (c == 0) wred[0][warp][g8] = tmax;
        __syncthreads();
        const float mn = fmaxf(fmaxf(m, fmaxf(wred[0][0][g8], wred[0][1][g8])), fmaxf(wred[0][2][g8], wred[0][3][g8]));
        const float corr = m == -INFINITY ? 0.0f : expf(m - mn);
        m = mn;
        float psum = 0.0f;
#pragma unroll
        for (int nb = 0; nb < 4; nb++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                sc[nb][j] = sc[nb][j] == -INFINITY ? 0.0f : expf(sc[nb][j] - mn);
                psum += sc[nb][j];
            }
        psum += __shfl_xor_sync(0xFFFFFFFFu, psum, 1);
        psum += __shfl_xor_sync(0xFFFFFFFFu, psum, 2);
        if (c == 0) wred[1][warp][g8] = psum;
        __syncthreads();
        l = fmaf(l, corr, (wred[1][0][g8] + wred[1][1][g8]) + (wred[1][2][g8] + wred[1][3][g8]));
        const float carry = corr * turn;
#pragma unroll
        for (int i = 0; i < NBD; i++) {
            oc[i][0] *= carry;
            oc[i][1] *= carry;
        }
#pragma unroll
        for (int g = 0; g < G; g++) side[g] *= carry;
        // ── values: two steps of 16 keys; the probabilities times the keys' value scales are the A fragments ──
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
            const int r0 = warp * 32 + kk * 16 + 2 * c;  // the lane's keys within the tile: r0, r0 + 1, r0 + 8, r0 + 9
            uint32_t pa0[G], pa2[G];
#pragma unroll
            for (int g = 0; g < G; g++) {
                float ps[4], pb = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int key = min(r0 + (i & 1) + 8 * (i >> 1), keys - 1);
                    const float pv = sc[2 * kk + (i >> 1)][i & 1];  // (zero for keys past the end)
                    const float4 sb = sbt[key][g];
                    ps[i] = pv * sb.z;
                    pb = fmaf(pv, sb.w, pb);
                }
                pa0[g] = qa_pack_f16(ps[0], ps[1]);
                pa2[g] = qa_pack_f16(ps[2], ps[3]);
                const float2 u = qa_unpack_f16(pa0[g]), v = qa_unpack_f16(pa2[g]);
                side[g] += pb - 1024.0f * ((u.x + u.y) + (v.x + v.y));
            }
            const uint32_t *v0 = vtile + r0 * WP, *v1 = v0 + WP, *v2 = v0 + 8 * WP, *v3 = v0 + 9 * WP;
#pragma unroll
            for (int nbd = 0; nbd < NBD; nbd++) {
                uint32_t b0, b1;
                if (BITS == 4) {
                    const int sh = 4 * g8;  // dim 8 nbd + g8 = nibble g8 of word nbd
                    b0 = (((v0[nbd] >> sh) & 0xFu) | (((v1[nbd] >> sh) & 0xFu) << 16)) | 0x64006400u;
                    b1 = (((v2[nbd] >> sh) & 0xFu) | (((v3[nbd] >> sh) & 0xFu) << 16)) | 0x64006400u;
                } else {
                    const int wd = 2 * nbd + (g8 >> 2), sh = 8 * (g8 & 3);  // byte g8 % 4 of word 2 nbd + g8 / 4
                    b0 = (((v0[wd] >> sh) & 0xFFu) | (((v1[wd] >> sh) & 0xFFu) << 16)) | 0x64006400u;
                    b1 = (((v2[wd] >> sh) & 0xFFu) | (((v3[wd] >> sh) & 0xFFu) << 16)) | 0x64006400u;
                }
                qa_mma(oc[nbd], pa0[nbd / NBD_PER_G], 0u, pa2[nbd / NBD_PER_G], 0u, b0, b1);
            }
        }
        if (more) keep_scales(buf ^ 1);
        __syncthreads();  // this tile's buffers are refilled from the next iteration on; wred is rewritten by the next tile
    }

    // ── the four warps' outputs together, then this split's partial result ──
#pragma unroll
    for (int g = 0; g < G; g++) {
        side[g] += __shfl_xor_sync(0xFFFFFFFFu, side[g], 1);
        side[g] += __shfl_xor_sync(0xFFFFFFFFu, side[g], 2);
    }
    float *wsum = reinterpret_cast<float *>(vbuf);  // [warp][head][D]
    const float unlift = qa_inverse(lift);
    if (head) {
#pragma unroll
        for (int nbd = 0; nbd < NBD; nbd++) {
            float *dst = wsum + ((warp * 8 + g8) * D) + 8 * nbd + 2 * c;
            dst[0] = (oc[nbd][0] + side[nbd / NBD_PER_G]) * unlift;
            dst[1] = (oc[nbd][1] + side[nbd / NBD_PER_G]) * unlift;
        }
    }
    __syncthreads();
    for (int i = t; i < D * rep; i += QA_THREADS) {
        const int h = i / D, d = i % D;
        float *dst = p.part + (((size_t)b * p.Hq + hk * rep + h) * p.splits + split) * (D + 2);
        dst[d] = (wsum[(0 * 8 + h) * D + d] + wsum[(1 * 8 + h) * D + d]) + (wsum[(2 * 8 + h) * D + d] + wsum[(3 * 8 + h) * D + d]);
    }
    if (warp == 0 && c == 0 && head) {
        float *dst = p.part + (((size_t)b * p.Hq + hk * rep + g8) * p.splits + split) * (D + 2);
        dst[D] = m;
        dst[D + 1] = l;
    }
}

template <typename T, int D>
__global__ void __launch_bounds__(D) qattn_combine_kernel(QAttnParams p) {
    const int h = blockIdx.x, b = blockIdx.y, d = threadIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the partial results are the split kernel's
    const float *part = p.part + ((size_t)b * p.Hq + h) * p.splits * (D + 2);
    float mx = -INFINITY;
    for (int j = 0; j < p.splits; j++) mx = fmaxf(mx, part[j * (D + 2) + D]);
    const bool sink = p.sinks != nullptr;
    const float sv = sink ? DT<T>::load((const T *)p.sinks, h) : 0.0f;
    if (sink) mx = fmaxf(mx, sv);
    float num = 0.0f, den = sink ? expf(sv - mx) : 0.0f;
    for (int j = 0; j < p.splits; j++) {
        const float mj = part[j * (D + 2) + D];
        if (mj == -INFINITY) continue;
        const float w = expf(mj - mx);
        num = fmaf(w, part[j * (D + 2) + d], num);
        den = fmaf(w, part[j * (D + 2) + D + 1], den);
    }
    DT<T>::store((T *)p.out, (((size_t)b * p.Hq + h) * p.L + p.l) * D + d, den > 0.0f ? __fdiv_rn(num, den) : 0.0f);
}

// The combine kernel, launched so that it may become resident while the split kernel runs (NUVEC_PDL=0: plain order).
template <typename T, int D>
static int32_t qattn_combine(nvc_device *dev, const QAttnParams &p) {
    const Writes written(Trigger::LATE, {{p.out, (size_t)p.B * p.Hq * p.L * D * sizeof(T)}});
    return launch_pdl(dev, "qattn_combine_kernel", written, qattn_combine_kernel<T, D>, dim3((unsigned)p.Hq, (unsigned)p.B), dim3(D), 0, p);
}

// The form of a call.  CUDA cores: float32 and 3-bit codes (NUVEC_QATTN_MMA=0: everything).  The ring form reads a row's scales
// as one word or two.  The tile form takes what is not so aligned, and one query row over few keys.
//
// Where the line lies: a block of the tile form takes a tile of 128 keys from beginning to end, with nothing to overlap it, and
// its merge is a launch that walks a head's splits one after another; the ring form's warps need a few steps each to fill their
// rings, and its merge is a round trip through global memory.  So the bytes per multiprocessor decide, and the splits per head.
// Measured over 1 to 8 batches x 1 to 8 key heads of 128 x 64 to 8000 keys, four query heads each, us by tiles over us by ring:
//     codes of the keys    up to 2 MiB     4 MiB           8 MiB           16 MiB
//     4 bits               0.77 .. 1.19    1.09 .. 1.12    1.41 .. 1.52    1.54 .. 1.62
//     8 bits               0.92 .. 1.25    0.98 .. 1.19    1.31 .. 1.34    1.68 .. 1.70
//     one to eight heads of 8000 keys (63 splits): 1.05 .. 1.45
// Up to 4 MiB and 32 splits neither form is ahead of the other by more than a quarter, 1.9 us a call; beyond, the ring form
// always is.  (Up to 128 keys are the exception: the ring form needs no merge there, 3.4 us against 6.2.)  Within the range the
// tile form stays for its results: both forms are equally exact (4 to 6e-4 before the rounding to bfloat16), but another rounding
// of the attention moves the outputs of three to six layers of a decode step by 1.1 to 1.7e-2, and gained those steps 0.2 to 1.9 %.
enum QaForm { QA_CUDA, QA_TILES, QA_RING };
static QaForm qattn_form(int dtype, int bits, int64_t groups, std::initializer_list<const void *> scales, const void *q, const void *out, int64_t L, int64_t S,
                         int64_t code_bytes) {
    static const bool mma_on = !(getenv("NUVEC_QATTN_MMA") && atoi(getenv("NUVEC_QATTN_MMA")) == 0);
    if (!mma_on || dtype == NVC_F32 || bits == 3) return QA_CUDA;
    uintptr_t al = 0;
    for (const void *p : scales) al |= (uintptr_t)p;
    if (al % (2 * (uintptr_t)groups) != 0 || (uintptr_t)q % 16 != 0 || (uintptr_t)out % 8 != 0) return QA_TILES;
    return L == 1 && S <= 4096 && code_bytes <= 4 << 20 ? QA_TILES : QA_RING;
}

template <typename T, int BITS, int D, int GS>
static int32_t qattn_launch_mma(nvc_device *dev, const QAttnParams &p, bool ring) {
    if constexpr (sizeof(T) == 2 && (BITS == 4 || BITS == 8) && D % GS == 0) {
        constexpr size_t ring_smem = QmRing<BITS, D, GS>::SMEM, tile_smem = qt_smem<BITS, D, GS>();
        static bool configured[64] = {};
        static std::mutex mu;
        if (dev->ordinal < 0 || dev->ordinal >= 64) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: device ordinal %d", dev->ordinal);
        {
            std::lock_guard<std::mutex> g(mu);
            if (!configured[dev->ordinal]) {
                NVC_CUDA(cudaFuncSetAttribute(qattn_mma_kernel<T, BITS, D, GS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring_smem));
                NVC_CUDA(cudaFuncSetAttribute(qattn_tile_kernel<T, BITS, D, GS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem));
                configured[dev->ordinal] = true;
            }
        }
        const dim3 grid((unsigned)p.splits, (unsigned)p.Hkv, (unsigned)(p.B * p.row_tiles));
        const Trigger trigger = p.early ? Trigger::EARLY : Trigger::LATE;
        if (ring)
            return launch_pdl(dev, "qattn_mma_kernel", Writes(trigger, {{p.out, (size_t)p.B * p.Hq * p.L * D * sizeof(T)}}), qattn_mma_kernel<T, BITS, D, GS>, grid,
                              dim3(QM_THREADS), ring_smem, p);
        NVC_TRY(launch_pdl(dev, "qattn_tile_kernel", Writes(trigger, {}), qattn_tile_kernel<T, BITS, D, GS>, grid, dim3(QA_THREADS), tile_smem, p));
        return qattn_combine<T, D>(dev, p);
    }
    return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: no tensor-core kernel");
}

template <typename T, int BITS, int D>
static int32_t qattn_launch(nvc_device *dev, const QAttnParams &p, int gs, QaForm form) {
    if (form != QA_CUDA) {
        if (gs == 32) return qattn_launch_mma<T, BITS, D, 32>(dev, p, form == QA_RING);
        if (gs == 64) return qattn_launch_mma<T, BITS, D, 64>(dev, p, form == QA_RING);
        return qattn_launch_mma<T, BITS, D, D == 128 ? 128 : 64>(dev, p, form == QA_RING);
    }
    dim3 grid((unsigned)p.splits, (unsigned)p.Hkv, (unsigned)p.B);
    if (gs == 32) qattn_split_kernel<T, BITS, D, 32><<<grid, QA_THREADS, 0, dev->stream>>>(p);
    else if (gs == 64) qattn_split_kernel<T, BITS, D, 64><<<grid, QA_THREADS, 0, dev->stream>>>(p);
    else if (D == 128) qattn_split_kernel<T, BITS, D, D == 128 ? 128 : 64><<<grid, QA_THREADS, 0, dev->stream>>>(p);
    NVC_TRY(check_launch(dev, "qattn_split_kernel"));
    return qattn_combine<T, D>(dev, p);
}

template <typename T>
static int32_t qattn_typed(nvc_device *dev, const QAttnParams &p, int bits, int d, int gs, QaForm form) {
    if (d == 128) {
        if (bits == 3) return qattn_launch<T, 3, 128>(dev, p, gs, form);
        if (bits == 4) return qattn_launch<T, 4, 128>(dev, p, gs, form);
        return qattn_launch<T, 8, 128>(dev, p, gs, form);
    }
    if (bits == 3) return qattn_launch<T, 3, 64>(dev, p, gs, form);
    if (bits == 4) return qattn_launch<T, 4, 64>(dev, p, gs, form);
    return qattn_launch<T, 8, 64>(dev, p, gs, form);
}

}  // namespace nvc

using namespace nvc;

extern "C" int32_t nvc_quantized_attention(nvc_device *dev, const nvc_quant *quant, int32_t dtype, const void *q, const uint32_t *k_codes,
                                           const void *k_scales, const void *k_biases, const uint32_t *v_codes, const void *v_scales,
                                           const void *v_biases, const void *sinks, int64_t B, int64_t Hq, int64_t Hkv, int64_t L, int64_t S,
                                           int64_t D, int64_t capacity, float scale, int32_t causal, void *out) {
    NVC_TRY(make_current(dev));
    NVC_TRY(check_quant("quantized_attention", quant));
    if (quant->mode != NVC_AFFINE) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_attention: keys and values need one affine quantization");
    const int bits = quant->bits, gs = quant->group_size;
    if (dtype != NVC_F16 && dtype != NVC_BF16 && dtype != NVC_F32) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: unsupported dtype %d", dtype);
    if (B < 0 || Hq < 0 || Hkv < 0 || L < 0 || S < 0 || capacity < S) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_attention: invalid shape");
    if (L > 64) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: %lld query rows per head (the cache is read once per row: up to 64)", (long long)L);
    if ((D != 64 && D != 128) || (bits != 3 && bits != 4 && bits != 8) || D % gs != 0)
        return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: head size %lld with %d bits in groups of %d (64 or 128; 3, 4 or 8; a group within a head)",
                         (long long)D, bits, gs);
    if (B * Hq * L == 0) return NVC_OK;
    if (Hkv <= 0 || Hq % Hkv != 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_attention: %lld query heads over %lld key heads", (long long)Hq, (long long)Hkv);
    const int64_t rep = Hq / Hkv;
    if (rep != 1 && rep != 2 && rep != 4 && rep != 8) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: %lld query heads per key head (1, 2, 4 or 8)", (long long)rep);
    if (B > 65535 || Hkv > 65535 || S > INT32_MAX || capacity > INT32_MAX) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: too long");
    if (!q || !out || (S > 0 && (!k_codes || !k_scales || !k_biases || !v_codes || !v_scales || !v_biases)))
        return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_attention: null operand");
    if (((uintptr_t)k_codes | (uintptr_t)v_codes) % 16 != 0) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: the codes must be 16-byte aligned");

    const QaForm form = qattn_form(dtype, bits, D / gs, {k_scales, k_biases, v_scales, v_biases}, q, out, L, S, B * Hkv * S * D * bits / 8);
    const bool ring = form == QA_RING;
    // the ring form multiplies up to eight columns (heads x query rows) in one pass over the keys
    const int64_t row_pack = ring ? (L < 8 / rep ? L : 8 / rep) : 1, row_tiles = ring ? (L + row_pack - 1) / row_pack : 1;
    if (B * row_tiles > 65535) return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: too many batches");
    // splits: one wave of as many blocks as stay resident together (what their registers allow, or the tile form's two sets
    // of buffers: two of the ring form, three and five of the others, per multiprocessor) of at least a tile of 128 keys (the
    // ring form's eight warps take 16 each)
    const int64_t tiles = S > 0 ? (S + QA_TILE - 1) / QA_TILE : 1, grain = ring ? QM_STEP : QA_TILE;
    int64_t per_sm = ring ? QM_BLOCKS_PER_SM : 5;
    if (form == QA_TILES) {
        const int64_t tile_words = QA_TILE * (D * bits / 32 + 4), sum_words = 4 * 8 * D;
        const int64_t smem = (2 * tile_words + (2 * tile_words > sum_words ? 2 * tile_words : sum_words)) * 4 + 2 * QA_TILE * (D / gs) * 16;
        per_sm = (227 * 1024) / (smem + 1024 + 256);
        if (per_sm > QT_BLOCKS) per_sm = QT_BLOCKS;
        if (per_sm < 1) per_sm = 1;
    }
    int64_t splits = per_sm * (int64_t)dev->prop.multiProcessorCount / (B * Hkv * row_tiles);
    if (splits > tiles) splits = tiles;
    if (ring && splits > 512) splits = 512;  // (their weights fit the kernel's shared memory)
    if (splits < 1) splits = 1;
    const int64_t per_split = ring ? (S + splits - 1) / splits : (tiles + splits - 1) / splits * QA_TILE;
    const int64_t chunk = (per_split + grain - 1) / grain * grain + (S == 0 ? grain : 0);
    splits = S > 0 ? (S + chunk - 1) / chunk : 1;
    // the splits' partial results: the handle's scratch block (reused between calls in stream order; it grows outside
    // recorded steps only)
    const size_t part_bytes = ring && splits == 1 ? 0 : (size_t)B * Hq * (ring ? L : 1) * splits * (D + (ring ? 4 : 2)) * sizeof(float);
    const size_t arrivals = ring && splits > 1 ? (size_t)(B * row_tiles * Hkv) : 0;
    if (dev->capturing && (dev->scratch_bytes < part_bytes || dev->counters_len < arrivals))
        return set_error(NVC_ERR_UNSUPPORTED, "quantized_attention: %zu bytes of scratch inside a recorded step (run the shape once before recording)",
                         part_bytes);
    void *part = nullptr;
    uint32_t *counters = nullptr;
    if (part_bytes) NVC_TRY(ensure_scratch(dev, part_bytes, &part));
    if (arrivals) NVC_TRY(ensure_counters(dev, arrivals, &counters));
    QAttnParams p{q, k_codes, v_codes, k_scales, k_biases, v_scales, v_biases, sinks, (float *)part, out,
                  (int32_t)B, (int32_t)Hq, (int32_t)Hkv, (int32_t)S, (int32_t)capacity, (int32_t)splits, (int32_t)chunk, (int32_t)L, 0, scale,
                  (int32_t)row_pack, (int32_t)row_tiles, causal != 0, 0, counters};
    auto run = [&]() {
        return dtype == NVC_F16 ? qattn_typed<__half>(dev, p, bits, (int)D, gs, form)
             : dtype == NVC_BF16 ? qattn_typed<__nv_bfloat16>(dev, p, bits, (int)D, gs, form) : qattn_typed<float>(dev, p, bits, (int)D, gs, form);
    };
    if (form != QA_CUDA) {
        const size_t rows = (size_t)(B * Hkv * capacity), code_bytes = rows * (size_t)(D * bits / 8), scale_bytes = rows * (size_t)(D / gs) * 2;
        p.early = early_read_ok(dev, k_codes, code_bytes) && early_read_ok(dev, v_codes, code_bytes) && early_read_ok(dev, k_scales, scale_bytes) &&
                  early_read_ok(dev, k_biases, scale_bytes) && early_read_ok(dev, v_scales, scale_bytes) && early_read_ok(dev, v_biases, scale_bytes);
    }
    if (ring) return run();
    int32_t rc = NVC_OK;
    // every query row attends to all the keys (or, causal, to those up to its position); a row at a time (the partial
    // results are reused in stream order)
    // (causal: query row l is the position S - L + l and attends to the keys up to it)
    for (int64_t l = 0; l < L && rc == NVC_OK; l++) {
        p.l = (int32_t)l;
        if (causal) p.S = (int32_t)(S - (L - 1 - l) > 0 ? S - (L - 1 - l) : 0);
        rc = run();
    }
    return rc;
}
