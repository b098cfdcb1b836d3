// quantize / dequantize kernels: the parity gates of the path.
//
// Every rounding the reference's CPU kernels perform is performed here in the same order, so
// the outputs are equal bit for bit (crates/nuvec-core/src/kernels.rs:774-859 for affine,
// :914-1009 for mxfp4 / mxfp8 / nvfp4; codecs crates/nuvec-core/src/fp8.rs:18-129).
// Intrinsics with explicit rounding (__fmul_rn, __fadd_rn, __fdiv_rn) keep the compiler from
// contracting or approximating any step.
#include "common.cuh"

namespace nvc {

// ── dequantize ─────────────────────────────────────────────────────────────────────────

// Rows picked by index (an embedding look-up: QuantizedEmbedding::forward takes the ids' rows of
// the packed table, its scales and biases, then dequantizes them, crates/nuvec-nn/src/layers.rs:246-255):
// the output's row r is source row ids[r]; an id past the end takes the last row, as `take` clamps
// (crates/nuvec-core/src/kernels.rs:120-133).  Without ids the array is one long row.
struct RowPick {
    const uint32_t *ids;     // nullptr: rows as they are
    uint32_t packs_per_row;  // cols / 8
    uint32_t rows;           // rows of the table
};
// This thread's pack of 8 values: its number in the output and in the source; false past the end.
template <bool PICK>
__device__ __forceinline__ bool pack_of(const RowPick &pick, size_t packs, size_t &i, size_t &si) {
    if (PICK) {  // a block works inside one row
        const uint32_t at = blockIdx.y * 256u + threadIdx.x;
        if (at >= pick.packs_per_row) return false;
        i = (size_t)blockIdx.x * pick.packs_per_row + at;
        si = (size_t)min(pick.ids[blockIdx.x], pick.rows - 1u) * pick.packs_per_row + at;
        return true;
    }
    i = si = (size_t)blockIdx.x * 256u + threadIdx.x;
    return i < packs;
}
// Eight results to out[first .. first + 7]: 16-byte stores where the array is aligned.
template <typename T> __device__ __forceinline__ void store8(T *out, size_t first, const float (&v)[8], bool wide) {
    T h[8];
#pragma unroll
    for (int j = 0; j < 8; j++) DT<T>::store(h, j, v[j]);
    if (wide) {
#pragma unroll
        for (int q = 0; q < (int)sizeof(T) / 2; q++) reinterpret_cast<uint4 *>(out + first)[q] = reinterpret_cast<const uint4 *>(h)[q];
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) out[first + j] = h[j];
    }
}

// One thread decodes 8 consecutive values (8 * bits bits = `bits` whole bytes, read in the widest units their alignment
// allows), which never straddle a group because every group size is a multiple of 8.  Bound by memory: 4-bit codes to
// bfloat16, 12288 x 4096: 30.8 us = 4.2 TB/s.
template <typename T, int BITS, bool FUSED, bool PICK>
__global__ void __launch_bounds__(256)
dequantize_affine_kernel(const uint8_t *__restrict__ codes, const T *__restrict__ scales,
                         const T *__restrict__ biases, T *__restrict__ out, size_t packs, int gs_shift, RowPick pick, int wide) {
    pdl_wait();
    size_t i, si;
    if (!pack_of<PICK>(pick, packs, i, si)) return;
    const uint8_t *src = codes + si * BITS;
    uint64_t stream = 0;
    if (BITS == 8) stream = reinterpret_cast<const uint32_t *>(src)[0] | (uint64_t)reinterpret_cast<const uint32_t *>(src)[1] << 32;
    else if (BITS == 4) stream = *reinterpret_cast<const uint32_t *>(src);
    else if (BITS == 2 || BITS == 6) {
#pragma unroll
        for (int b = 0; b < BITS / 2; b++) stream |= (uint64_t)reinterpret_cast<const uint16_t *>(src)[b] << (16 * b);
    } else {
#pragma unroll
        for (int b = 0; b < BITS; b++) stream |= (uint64_t)src[b] << (8 * b);
    }
    const size_t g = si * 8 >> gs_shift;
    const float s = DT<T>::load(scales, g), bias = DT<T>::load(biases, g);
    float vals[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float c = (float)(uint32_t)((stream >> (j * BITS)) & ((1u << BITS) - 1u));
        if (FUSED) {
            vals[j] = __fmaf_rn(c, s, bias);  // rounded once on store
        } else {
            float p = DT<T>::round(__fmul_rn(c, s));  // product rounded to T
            vals[j] = __fadd_rn(p, bias);             // sum rounded to T on store
        }
    }
    store8(out, i * 8, vals, wide);
}

// Floating-point modes: BITS == 4 -> two E2M1 codes per byte, low nibble first; BITS == 8 ->
// one E4M3 code per byte.  One thread decodes 8 values.  A code's magnitude bits placed at the top of a float32's
// mantissa and the bottom of its exponent are the value times 2^-126 (E2M1) or 2^-120 (E4M3), subnormal codes as float32
// subnormals; one exact multiplication restores it.
template <typename T, int BITS, bool PICK>
__global__ void __launch_bounds__(256)
dequantize_fp_kernel(const uint8_t *__restrict__ codes, const uint8_t *__restrict__ scales,
                     const float *__restrict__ global, T *__restrict__ out, size_t packs, int gs_shift, RowPick pick, int wide) {
    pdl_wait();
    size_t i, si;
    if (!pack_of<PICK>(pick, packs, i, si)) return;
    const uint32_t sc = scales[si * 8 >> gs_shift];
    float scale = ftz(gs_shift == 5 ? e8m0_to_f32(sc) : e4m3_to_f32(sc));
    if (global) {
        float inv = ftz(__fdiv_rn(*global, 448.0f * 6.0f));
        scale = ftz(__fmul_rn(scale, inv));
    }
    const uint32_t *src = reinterpret_cast<const uint32_t *>(codes + si * BITS);
    uint32_t w[2] = {src[0], BITS == 8 ? src[1] : 0u};
    // (with a finite scale the product is never NaN, and subnormal results flush in the multiplication itself)
    const bool plain = fabsf(scale) < __uint_as_float(0x7F800000u);
    float vals[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        float v;
        if (BITS == 8) {
            const uint32_t c = (w[j >> 2] >> (8 * (j & 3))) & 0xFFu;
            v = __fmul_rn(__uint_as_float((c & 0x7Fu) << 20 | (c & 0x80u) << 24), __uint_as_float((127u + 120u) << 23));
            if ((c & 0x7Fu) == 0x7Fu) v = __uint_as_float(0x7FC00000u);  // (NaN through either branch below)
        } else {
            const uint32_t c = (w[0] >> (4 * j)) & 0xFu;
            v = __fmul_rn(__uint_as_float((c & 7u) << 22 | (c & 8u) << 28), __uint_as_float((127u + 126u) << 23));
        }
        vals[j] = v;
    }
    if (plain) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(vals[j]) : "f"(scale), "f"(vals[j]));
            if (BITS == 8) vals[j] = canonical(vals[j]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) vals[j] = canonical(ftz(__fmul_rn(scale, vals[j])));
    }
    store8(out, i * 8, vals, wide);
}

// Blocks for `packs` packs: rows along x and 256 packs of a row along y with a row pick.
static dim3 pack_grid(size_t packs, const RowPick &pick) {
    if (!pick.ids) return dim3((unsigned)((packs + 255) / 256));
    return dim3((unsigned)(packs / pick.packs_per_row), (pick.packs_per_row + 255) / 256);
}

template <typename T, bool FUSED>
static int32_t launch_dequantize_affine(nvc_device *dev, int bits, const uint8_t *codes, const void *scales,
                                        const void *biases, void *out, size_t packs, int gs_shift, RowPick pick) {
    const int wide = (uintptr_t)out % 16 == 0;
    const Writes written(Trigger::LATE, {{out, packs * 8 * sizeof(T)}});
#define NVC_CASE(B)                                                                                                                     \
    case B:                                                                                                                             \
        return launch_pdl(dev, "dequantize_affine_kernel", written,                                                                              \
                          pick.ids ? dequantize_affine_kernel<T, B, FUSED, true> : dequantize_affine_kernel<T, B, FUSED, false>,        \
                          pack_grid(packs, pick), dim3(256), 0, codes, (const T *)scales, (const T *)biases, (T *)out, packs, gs_shift, pick, wide);
    switch (bits) {
        NVC_CASE(1) NVC_CASE(2) NVC_CASE(3) NVC_CASE(4) NVC_CASE(5) NVC_CASE(6) NVC_CASE(8)
    default: return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: %d bits", bits);
    }
#undef NVC_CASE
}

// ── quantize ───────────────────────────────────────────────────────────────────────────

// rint(x / scale), the quotient rounded to float32 first, where x / scale lies within 0.01 of the half-way point next to
// the integer r on rest's side (rest = x - r * scale).  The half-way point h is exact; e = x - h * scale (one rounding,
// so of the right sign).  The quotient rounds to h itself -- and rint to the even neighbour -- when |e| is at most half a
// unit in the last place of h times |scale|, a power of two times |scale| and therefore exact; it is on e's side
// otherwise.  (Below h = 0.5 the unit is half as large, but there both outcomes are 0.)  Values of few bits divided by a
// scale made of two of them meet such points for several per cent of the codes, so a division here would run in most
// warps; only |e| equal to the limit, where e's own rounding could matter, and what is not near a half-way point at all
// (NaN, infinities) divide.
__device__ __forceinline__ float near_half_code(float x, float scale, float r, float rest) {
    const float towards = (__float_as_uint(rest) ^ __float_as_uint(scale)) & 0x80000000u ? -0.5f : 0.5f;
    const float h = __fadd_rn(r, towards), e = __fmaf_rn(-h, scale, x);
    const float limit = __uint_as_float(__float_as_uint(h) & 0x7F800000u) * 5.9604645e-8f * fabsf(scale);
    if (!(fabsf(rest) <= 0.51f * fabsf(scale)) || fabsf(h) > 1024.0f || fabsf(e) == limit || limit < 1e-37f) return rintf(__fdiv_rn(x, scale));
    const float even = __fadd_rn(__fadd_rn(h, 12582912.0f), -12582912.0f);
    const float side = __fadd_rn(h, (__float_as_uint(e) ^ __float_as_uint(scale)) & 0x80000000u ? -0.5f : 0.5f);
    return fabsf(e) < limit ? even : side;
}

// One thread per 16 consecutive values; gs / 16 neighbouring lanes share a group (its extremes through shuffles).  The
// arithmetic is float32 throughout, in the reference's order.  A code is rint((v - bias) / scale): the quotient comes
// from a multiplication by 1 / scale, and the remainder v - bias - code * scale says whether the code is certain -- when
// it is below 0.4999 |scale|, the division, correctly rounded, lies on the same side of both half-way points (codes stay
// below 2^10, so its rounding moves it by less than 2^-14).  Otherwise near_half_code decides.
// Bound by issue (a dozen instructions per value, four divisions per thread for the group's constants) above memory:
// 12288 x 4096 bfloat16 to 4 bits 431 -> 46 us against one thread per group walking it in 2-byte loads.
template <typename T, int BITS>
__global__ void __launch_bounds__(256)
quantize_affine_kernel(const T *__restrict__ w, uint8_t *__restrict__ codes, T *__restrict__ scales,
                       T *__restrict__ biases, size_t packs, int lanes, int wide) {
    constexpr int V = 16, QUADS = V * (int)sizeof(T) / 16;
    pdl_trigger();
    const size_t at = (size_t)blockIdx.x * 256 + threadIdx.x;
    const bool have = at < packs;
    const size_t i = have ? at : packs - 1;  // (whole groups past the end: their lanes repeat the last pack and store nothing)
    pdl_wait();
    float v[V];
    if (wide) {
        uint4 raw[QUADS];
#pragma unroll
        for (int q = 0; q < QUADS; q++) raw[q] = reinterpret_cast<const uint4 *>(w + i * V)[q];
#pragma unroll
        for (int j = 0; j < V; j++) v[j] = DT<T>::load(reinterpret_cast<const T *>(raw), j);
    } else {
#pragma unroll
        for (int j = 0; j < V; j++) v[j] = DT<T>::load(w, i * V + j);
    }
    float lo = __int_as_float(0x7F800000), hi = __int_as_float(0xFF800000);
#pragma unroll
    for (int j = 0; j < V; j++) {
        lo = fminf(lo, v[j]);
        hi = fmaxf(hi, v[j]);
    }
    for (int o = 1; o < lanes; o <<= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    constexpr float n_bins = (float)((1u << BITS) - 1u);
    const float eps = 1e-7f;
    float scale, bias;
    if (BITS == 1) {
        scale = fmaxf(__fsub_rn(hi, lo), eps);
        bias = lo;
    } else {
        const bool far = fabsf(lo) > fabsf(hi);
        scale = fmaxf(__fdiv_rn(__fsub_rn(hi, lo), n_bins), eps);
        scale = far ? scale : -scale;
        const float edge = far ? lo : hi;
        const float q0 = rintf(__fdiv_rn(edge, scale));
        if (q0 == 0.0f) {
            bias = 0.0f;
        } else {
            scale = __fdiv_rn(edge, q0);
            bias = edge;
        }
    }
    const float inv = __frcp_rn(scale), sure = 0.4999f * fabsf(scale);
    uint32_t c[V];
#pragma unroll
    for (int j = 0; j < V; j++) {
        const float x = __fsub_rn(v[j], bias);
        const float m = __fadd_rn(__fmul_rn(x, inv), 12582912.0f);  // 1.5 * 2^23: the nearest integer in the low mantissa bits
        float r = __fsub_rn(m, 12582912.0f);
        const float rest = __fmaf_rn(-r, scale, x);
        if (!(fabsf(rest) < sure)) r = near_half_code(x, scale, r, rest);
        // to [0, n_bins] (NaN: 0) and to an integer through the mantissa
        c[j] = __float_as_uint(__fadd_rn(fminf(fmaxf(r, 0.0f), n_bins), 8388608.0f)) & 0x7FFFFFu;
    }
    if (!have) return;
    // V codes = BITS half-words
    uint32_t *dst = reinterpret_cast<uint32_t *>(codes + i * (V * BITS / 8));
    uint32_t words[(V * BITS + 31) / 32] = {};
#pragma unroll
    for (int j = 0; j < V; j++) {
        words[j * BITS / 32] |= c[j] << (j * BITS % 32);
        if (j * BITS % 32 + BITS > 32) words[j * BITS / 32 + 1] |= c[j] >> (32 - j * BITS % 32);
    }
    if (BITS == 8 && ((uintptr_t)codes & 15) == 0) *reinterpret_cast<uint4 *>(dst) = make_uint4(words[0], words[1 % ((V * BITS + 31) / 32)], words[2 % ((V * BITS + 31) / 32)], words[3 % ((V * BITS + 31) / 32)]);
    else if (BITS == 4 && ((uintptr_t)codes & 7) == 0) *reinterpret_cast<uint2 *>(dst) = make_uint2(words[0], words[1 % ((V * BITS + 31) / 32)]);
    else if (BITS % 2 == 0) {
#pragma unroll
        for (int q = 0; q < V * BITS / 32; q++) dst[q] = words[q];
    } else {
#pragma unroll
        for (int q = 0; q < BITS; q++) reinterpret_cast<uint16_t *>(dst)[q] = (uint16_t)(words[q / 2] >> (16 * (q & 1)));
    }
    if ((threadIdx.x & (lanes - 1)) == 0) {
        const size_t g = i / (unsigned)lanes;
        DT<T>::store(scales, g, scale);
        DT<T>::store(biases, g, bias);
    }
}

// fp8.rs:18-36
__device__ __forceinline__ uint32_t e4m3_from_f32(float x) {
    const uint32_t FP8_MAX = 543u << 21, DENORM_MASK = 141u << 23;
    uint32_t bits = __float_as_uint(x);
    uint32_t sign = bits & 0x80000000u;
    bits ^= sign;
    uint32_t code;
    if (bits >= FP8_MAX) {
        code = 0x7E;
    } else if (bits < (121u << 23)) {
        float sum = __fadd_rn(__uint_as_float(bits), __uint_as_float(DENORM_MASK));
        code = (__float_as_uint(sum) - DENORM_MASK) & 0xFFu;
    } else {
        uint32_t odd = (bits >> 20) & 1u;
        bits += ((uint32_t)(7 - 127) << 23) + 0x7FFFFu;
        bits += odd;
        code = (bits >> 20) & 0xFFu;
    }
    return code | (sign >> 24);
}

// fp8.rs:48-73
__device__ __forceinline__ uint32_t e2m1_from_f32(float x) {
    if (x != x) return 0x7u;
    uint32_t sign = (__float_as_uint(x) >> 31) ? 0x8u : 0x0u;
    float a = fabsf(x);
    uint32_t code = a > 5.0f ? 7u : a >= 3.5f ? 6u : a > 2.5f ? 5u : a >= 1.75f ? 4u
                  : a > 1.25f ? 3u : a >= 0.75f ? 2u : a > 0.25f ? 1u : 0u;
    return code | sign;
}

// Eight values to eight E2M1 codes in one word, value 0 in the low nibble, with the hardware's
// conversion: round to nearest even on the E2M1 grid, saturate at 6, NaN to +6 (code 7), the sign of
// a zero result kept: code for code the function above (fp8.rs:48-73; its thresholds 0.25, 0.75,
// 1.25, 1.75, 2.5, 3.5, 5 are the grid's ties, each going to the neighbour with an even mantissa).
__device__ __forceinline__ uint32_t e2m1x8_from_f32(const float *v) {
    uint32_t word;
    asm("{\n\t.reg .b8 c0, c1, c2, c3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 c0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 c1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 c2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 c3, %8, %7;\n\t"
        "mov.b32 %0, {c0, c1, c2, c3};\n\t}"
        : "=r"(word)
        : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
    return word;
}

// The E8M0 code of mx_scale_round_up(x) for x >= 0 (fp8.rs:84-93, 124-130): the smallest
// power of two that is not below x, i.e. the exponent field, plus one when any mantissa bit
// is set, capped at 254; 0 for zero and 0xFF for Inf/NaN.
__device__ __forceinline__ uint32_t mx_scale_code(float x) {
    uint32_t u = __float_as_uint(x);
    uint32_t e = (u >> 23) & 0xFFu, m = u & 0x7FFFFFu;
    if (e == 0xFFu) return 0xFFu;
    if (e == 0u) return 0u;  // x was flushed: zero
    uint32_t code = e + (m != 0u ? 1u : 0u);
    return code > 254u ? 254u : code;
}

// LAID: the scales go straight into the block-scaled tensor-core layout of the qqmm kernel instead of the plain
// [rows, groups] array: 512-byte pieces of 128 rows x 4 scales, byte (r % 32) * 16 + (r % 128 / 32) * 4 + s,
// ordered [row tile][k-block of 256][piece]; the threads then cover the padded rows and groups too and write
// the padding's zero scales.
struct ScalePieces {
    uint8_t *out;
    int64_t rows, per_row, kblocks;
    int pieces;
};
// One thread per 16 values: a group of nvfp4, or half of a group of 32, whose two lanes share its largest magnitude.
// Codes leave through the hardware's conversions (E4M3: to nearest even, saturating, as e4m3_from_f32; a NaN becomes the
// largest code there and through the minimum here).  Bound by issue above memory: 12288 x 4096 bfloat16 to mxfp8
// 64 -> 31 us, float32 to mxfp4 183 -> 34 us against one thread per group.
template <typename T, int BITS, int GS, bool LAID = false>
__global__ void __launch_bounds__(256)
quantize_fp_kernel(const T *__restrict__ w, uint8_t *__restrict__ codes, uint8_t *__restrict__ scales,
                   const float *__restrict__ global, size_t packs, ScalePieces sp = ScalePieces{}) {
    constexpr int V = 16, QUADS = V * (int)sizeof(T) / 16, LANES = GS / V;
    pdl_trigger();  // (LAID: the product kernel may set itself up meanwhile)
    size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;  // this thread's pack of V values
    bool have = i < packs;
    size_t laid_at = 0;
    pdl_wait();
    if (LAID) {
        const int64_t padded = sp.kblocks * sp.pieces * 4;  // groups per row, padding included
        const size_t g = i / LANES;
        const int64_t r = (int64_t)(g / (size_t)padded), gk = (int64_t)(g % (size_t)padded);
        const bool inside = r < (sp.rows + 127) / 128 * 128;
        laid_at = (size_t)(((r / 128 * sp.kblocks + gk / (sp.pieces * 4)) * sp.pieces + (gk / 4) % sp.pieces) * 512 + (r % 32) * 16 +
                           (r % 128 / 32) * 4 + gk % 4);
        have = r < sp.rows && gk < sp.per_row;
        if (inside && !have && i % LANES == 0) sp.out[laid_at] = 0;
        i = (size_t)(r * sp.per_row + gk) * LANES + i % LANES;
    }
    if (!have) i = 0;  // (its lanes still take part in the shuffle)
    const bool has = global != nullptr;
    const float scale_enc = has ? ftz(__fdiv_rn(448.0f * 6.0f, *global)) : 1.0f;
    float vals[V];
    if (((uintptr_t)w & 15) == 0) {
        uint4 raw[QUADS];
#pragma unroll
        for (int q = 0; q < QUADS; q++) raw[q] = reinterpret_cast<const uint4 *>(w + i * V)[q];
#pragma unroll
        for (int j = 0; j < V; j++) vals[j] = ftz(DT<T>::load(reinterpret_cast<const T *>(raw), j));
    } else {
#pragma unroll
        for (int j = 0; j < V; j++) vals[j] = ftz(DT<T>::load(w, i * V + j));
    }
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < V; j++) amax = fmaxf(amax, fabsf(vals[j]));
    if (LANES == 2) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    if (!have) return;
    float scale = ftz(__fdiv_rn(amax, BITS == 4 ? 6.0f : 448.0f));
    if (has) scale = ftz(__fmul_rn(scale, scale_enc));
    uint32_t code;
    float decoded;
    if (GS == 32 && !has) {
        code = mx_scale_code(scale);
        decoded = e8m0_to_f32(code);
    } else {
        code = e4m3_from_f32(scale);
        decoded = e4m3_to_f32(code);
    }
    if (LANES == 1 || i % LANES == 0) {
        if (LAID) sp.out[laid_at] = (uint8_t)code;
        else scales[i / LANES] = (uint8_t)code;
    }
    decoded = ftz(decoded);
    const float inverse = decoded == 0.0f ? 0.0f : ftz(__fdiv_rn(has ? scale_enc : 1.0f, decoded));
    uint32_t *dst = reinterpret_cast<uint32_t *>(codes + i * (V * BITS / 8));
    if (BITS == 4) {
        uint32_t words[2];
#pragma unroll
        for (int wd = 0; wd < 2; wd++) {
            float scaled[8];  // (a product below the normal range becomes a zero code either way)
#pragma unroll
            for (int e = 0; e < 8; e++) scaled[e] = __fmul_rn(vals[8 * wd + e], inverse);
            words[wd] = e2m1x8_from_f32(scaled);
        }
        if (((uintptr_t)codes & 7) == 0) *reinterpret_cast<uint2 *>(dst) = make_uint2(words[0], words[1]);
        else {
            dst[0] = words[0];
            dst[1] = words[1];
        }
    } else {
        uint32_t words[4];
#pragma unroll
        for (int wd = 0; wd < 4; wd++) {
            uint16_t pair[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float a = fminf(__fmul_rn(vals[4 * wd + 2 * h], inverse), 448.0f), b = fminf(__fmul_rn(vals[4 * wd + 2 * h + 1], inverse), 448.0f);
                asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pair[h]) : "f"(b), "f"(a));
            }
            words[wd] = (uint32_t)pair[0] | (uint32_t)pair[1] << 16;
        }
        if (((uintptr_t)codes & 15) == 0) *reinterpret_cast<uint4 *>(dst) = make_uint4(words[0], words[1], words[2], words[3]);
        else {
#pragma unroll
            for (int q = 0; q < 4; q++) dst[q] = words[q];
        }
    }
}

template <typename T>
static int32_t quantize_typed(nvc_device *dev, const nvc_quant *q, const void *w, size_t count,
                              const float *global, uint32_t *codes, void *scales, void *biases) {
    const size_t groups = count / (size_t)q->group_size, scale_bytes = groups * (q->mode == NVC_AFFINE ? sizeof(T) : 1);
    const Writes written(Trigger::EARLY, {{codes, count * (size_t)q->bits / 8}, {scales, scale_bytes}, {biases, scale_bytes}});
    if (q->mode == NVC_AFFINE) {
        const size_t packs = count / 16;
        const int lanes = q->group_size / 16, wide = (uintptr_t)w % 16 == 0;
#define NVC_CASE(B)                                                                                                                          \
    case B:                                                                                                                                  \
        return launch_pdl(dev, "quantize_affine_kernel", written, quantize_affine_kernel<T, B>, dim3((unsigned)((packs + 255) / 256)), dim3(256), 0, \
                          (const T *)w, (uint8_t *)codes, (T *)scales, (T *)biases, packs, lanes, wide);
        switch (q->bits) {
            NVC_CASE(1) NVC_CASE(2) NVC_CASE(3) NVC_CASE(4) NVC_CASE(5) NVC_CASE(6) NVC_CASE(8)
        default: return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize: %d bits", q->bits);
        }
#undef NVC_CASE
    }
    const size_t packs = count / 16;
    return launch_pdl(dev, "quantize_fp_kernel", written,
                      q->bits == 8 ? quantize_fp_kernel<T, 8, 32> : q->group_size == 16 ? quantize_fp_kernel<T, 4, 16> : quantize_fp_kernel<T, 4, 32>,
                      dim3((unsigned)((packs + 255) / 256)), dim3(256), 0, (const T *)w, (uint8_t *)codes, (uint8_t *)scales, global, packs,
                      ScalePieces{});
}

template <typename T>
static int32_t dequantize_typed(nvc_device *dev, const nvc_quant *q, const uint32_t *codes, const void *scales,
                                const void *biases, const float *global, size_t count, void *out, int fused,
                                RowPick pick = RowPick{nullptr, 0, 0}) {
    const size_t packs = count / 8;
    const uint8_t *bytes = (const uint8_t *)codes;
    const int gs_shift = q->group_size == 16 ? 4 : q->group_size == 32 ? 5 : q->group_size == 64 ? 6 : 7;
    if (q->mode == NVC_AFFINE) {
        return fused ? launch_dequantize_affine<T, true>(dev, q->bits, bytes, scales, biases, out, packs, gs_shift, pick)
                     : launch_dequantize_affine<T, false>(dev, q->bits, bytes, scales, biases, out, packs, gs_shift, pick);
    }
    const int wide = (uintptr_t)out % 16 == 0;
    auto kernel = q->bits == 4 ? (pick.ids ? dequantize_fp_kernel<T, 4, true> : dequantize_fp_kernel<T, 4, false>)
                               : (pick.ids ? dequantize_fp_kernel<T, 8, true> : dequantize_fp_kernel<T, 8, false>);
    return launch_pdl(dev, "dequantize_fp_kernel", Writes(Trigger::LATE, {{out, packs * 8 * sizeof(T)}}), kernel, pack_grid(packs, pick), dim3(256), 0, bytes, (const uint8_t *)scales, global, (T *)out,
                      packs, gs_shift, pick, wide);
}

}  // namespace nvc

using namespace nvc;

extern "C" int32_t nvc_quantize(nvc_device *dev, const nvc_quant *q, int32_t dtype, const void *w, int64_t rows,
                                int64_t cols, const float *global_scale, uint32_t *out_codes, void *out_scales,
                                void *out_biases) {
    NVC_TRY(make_current(dev));
    NVC_TRY(check_quant("quantize", q));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_UNSUPPORTED, "quantize: unsupported dtype %d", dtype);
    if (rows < 0 || cols < 0 || cols % q->group_size != 0)
        return set_error(NVC_ERR_INVALID_ARGUMENT,
                         "quantize: needs at least 2 dimensions with the last divisible by the group size %d, got [%lld, %lld]",
                         q->group_size, (long long)rows, (long long)cols);
    if (global_scale && q->mode != NVC_NVFP4)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize: a global scale is only supported for nvfp4");
    if (q->mode == NVC_AFFINE && !out_biases) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize: affine needs a biases output");
    size_t count = (size_t)rows * (size_t)cols;
    if (count == 0) return NVC_OK;
    if (!w || !out_codes || !out_scales) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize: null operand");
    switch (dtype) {
    case NVC_F32: return quantize_typed<float>(dev, q, w, count, global_scale, out_codes, out_scales, out_biases);
    case NVC_F16: return quantize_typed<__half>(dev, q, w, count, global_scale, out_codes, out_scales, out_biases);
    default: return quantize_typed<__nv_bfloat16>(dev, q, w, count, global_scale, out_codes, out_scales, out_biases);
    }
}

extern "C" int32_t nvc_dequantize(nvc_device *dev, const nvc_quant *q, int32_t dtype, const uint32_t *codes,
                                  const void *scales, const void *biases, const float *global_scale, int64_t rows,
                                  int64_t cols, void *out, int32_t fused) {
    NVC_TRY(make_current(dev));
    NVC_TRY(check_quant("dequantize", q));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_UNSUPPORTED, "dequantize: unsupported dtype %d", dtype);
    if (q->mode == NVC_AFFINE && !biases)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: biases must be provided for affine quantization");
    if (q->mode != NVC_AFFINE && biases)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: biases must be null for this quantization mode");
    if (global_scale && q->mode != NVC_NVFP4)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: a global scale is only supported for nvfp4");
    if (rows < 0 || cols < 0 || cols % q->group_size != 0)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: %lld columns are not divisible by the group size %d",
                         (long long)cols, q->group_size);
    size_t count = (size_t)rows * (size_t)cols;
    if (count == 0) return NVC_OK;
    if (!codes || !scales || !out) return set_error(NVC_ERR_INVALID_ARGUMENT, "dequantize: null operand");
    switch (dtype) {
    case NVC_F32: return dequantize_typed<float>(dev, q, codes, scales, biases, global_scale, count, out, fused);
    case NVC_F16: return dequantize_typed<__half>(dev, q, codes, scales, biases, global_scale, count, out, fused);
    default: return dequantize_typed<__nv_bfloat16>(dev, q, codes, scales, biases, global_scale, count, out, fused);
    }
}

extern "C" int32_t nvc_quantized_embedding(nvc_device *dev, const nvc_quant *q, int32_t dtype, const uint32_t *codes, const void *scales,
                                           const void *biases, int64_t vocab, int64_t cols, const uint32_t *ids, int64_t count, void *out) {
    NVC_TRY(make_current(dev));
    NVC_TRY(check_quant("quantized_embedding", q));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_UNSUPPORTED, "quantized_embedding: unsupported dtype %d", dtype);
    if (q->mode == NVC_AFFINE && !biases)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_embedding: biases must be provided for affine quantization");
    if (q->mode != NVC_AFFINE && biases)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_embedding: biases must be null for this quantization mode");
    if (vocab < 0 || count < 0 || cols < 0 || cols % q->group_size != 0 || vocab > 0xFFFFFFFFll)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_embedding: invalid shape (%lld rows of %lld columns, group size %d)",
                         (long long)vocab, (long long)cols, q->group_size);
    const size_t total = (size_t)count * (size_t)cols;
    if (total == 0) return NVC_OK;
    if (vocab == 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_embedding: rows taken from an empty table");
    if (!codes || !scales || !ids || !out) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantized_embedding: null operand");
    if (count > INT32_MAX || cols / 8 > 65535ll * 256) return set_error(NVC_ERR_UNSUPPORTED, "quantized_embedding: too many ids or columns");
    const RowPick pick{ids, (uint32_t)(cols / 8), (uint32_t)vocab};
    switch (dtype) {
    case NVC_F32: return dequantize_typed<float>(dev, q, codes, scales, biases, nullptr, total, out, 0, pick);
    case NVC_F16: return dequantize_typed<__half>(dev, q, codes, scales, biases, nullptr, total, out, 0, pick);
    default: return dequantize_typed<__nv_bfloat16>(dev, q, codes, scales, biases, nullptr, total, out, 0, pick);
    }
}

// The activation side of nvc_qqmm: bfloat16 x [rows, cols] to 4-bit codes (nvfp4 or mxfp4, no global scale) with the
// scales written straight into the tensor core's layout (laid: row_tiles x kblocks x pieces x 512 bytes).
int32_t nvc::quantize_fp4_laid(nvc_device *dev, const nvc_quant *q, const void *x, int64_t rows, int64_t cols, uint32_t *codes, uint8_t *laid,
                               int64_t kblocks, int pieces) {
    const int64_t padded_rows = (rows + 127) / 128 * 128, padded_groups = kblocks * pieces * 4;
    const size_t threads = (size_t)padded_rows * (size_t)padded_groups * (size_t)(q->group_size / 16);
    ScalePieces sp{laid, rows, cols / q->group_size, kblocks, pieces};
    const Writes written(Trigger::EARLY, {{codes, (size_t)(rows * cols / 2)}, {laid, (size_t)(padded_rows / 128 * kblocks) * pieces * 512}});
    return launch_pdl(dev, "quantize_fp_kernel", written,
                      q->group_size == 16 ? quantize_fp_kernel<__nv_bfloat16, 4, 16, true> : quantize_fp_kernel<__nv_bfloat16, 4, 32, true>,
                      dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, (const __nv_bfloat16 *)x, (uint8_t *)codes, nullptr, nullptr, (size_t)0,
                      sp);
}

// FastOp::QuantizeDequantize (crates/nuvec-core/src/products.rs:306-315, MLX's fp_quantize_dequantize): x through
// its quantization in a floating-point mode, the values the codes represent, in x's dtype -- the activation side of
// qqmm and gather_qqmm.  The reference's quantize followed by its dequantize; codes and scales pass through pool
// scratch (so not inside a recorded step).
extern "C" int32_t nvc_quantize_dequantize(nvc_device *dev, const nvc_quant *q, int32_t dtype, const void *x, int64_t rows, int64_t cols,
                                           const float *global_scale, void *out) {
    NVC_TRY(make_current(dev));
    NVC_TRY(check_quant("quantize_dequantize", q));
    if (q->mode == NVC_AFFINE) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize_dequantize: needs a floating-point mode (mxfp4, mxfp8 or nvfp4)");
    if (rows < 0 || cols < 0 || cols % q->group_size != 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "quantize_dequantize: invalid shape");
    if (rows * cols == 0) return NVC_OK;
    if (dev->capturing) return set_error(NVC_ERR_UNSUPPORTED, "quantize_dequantize: not inside a recorded step (it takes scratch from the pool)");
    void *codes = nullptr, *scales = nullptr;
    NVC_TRY(dev->pool.alloc((size_t)rows * cols * q->bits / 8, &codes));
    int32_t rc = dev->pool.alloc((size_t)rows * (cols / q->group_size), &scales);
    if (rc == NVC_OK) rc = nvc_quantize(dev, q, dtype, x, rows, cols, global_scale, (uint32_t *)codes, scales, nullptr);
    if (rc == NVC_OK) rc = nvc_dequantize(dev, q, dtype, (const uint32_t *)codes, scales, nullptr, global_scale, rows, cols, out, 0);
    if (codes) dev->pool.free(codes);  // (the pool hands the blocks out again in stream order)
    if (scales) dev->pool.free(scales);
    return rc;
}
