// The glue around a mixture of experts' products: the router's top-k selection with
// renormalisation and the weighted sum of the experts' outputs
// (fast::moe_route, fast::weighted_sum: crates/nuvec-core/src/fast/imp.rs:2652-2672, 2731-2747;
// their Metal kernels: crates/nuvec-kernels/src/metal/moe.metal).  Each kernel performs the
// arithmetic of the composition it stands for, in the order the reference's CPU path performs it
// (fast/imp.rs:1586-1600 over kernels.rs:231-273, 609-645, 1191-1195, 1581), so the results are
// the reference's bits:
//   moe_route   stable ascending order of a row's probabilities (NaN last), the last k indices,
//               their values, and with `normalize` those divided by their sum -- the sum taken in
//               float64 over 8 lanes combined by a fixed tree, rounded to the array's type, the
//               divide element-wise in that type (float32 arithmetic for the halves);
//   weighted_sum  the products x * w rounded to the array's type, summed over k in float64 in
//               order, rounded once;
//   moe_sort    SwitchGlu::forward's bookkeeping for many rows (crates/nuvec-lm/src/model.rs:2199-2210): the
//               stable ascending argsort of the flattened expert indices (kernels.rs:231-266), its inverse
//               (the argsort of the argsort), each sorted pair's token (pair / k) and expert, and the
//               experts' first rows (sorted_offsets); integers throughout;
//   take_rows   `take(.., 0)` of whole rows (the activations by token, the results back into pair order),
//               indices past the end clamped (kernels.rs:120-133);
//   swiglu / swiglu_oai  the activation between the up/gate and the down products
//               (crates/nuvec-nn/src/lib.rs:513-579; SwitchGlu::through, model.rs:2160-2171): on the CPU the
//               compiled function is its operations one by one (crates/nuvec-core/src/fused.rs:214-217), each
//               rounded to the array's type, the sigmoid as MLX's (kernels.rs:1538-1543) in float32.  The
//               only step that is not an IEEE operation is the exponential: where the device's expf and the
//               host's differ in their last bit a result can differ by a unit or two in the last place;
//   rms_norm / add_rms_norm  fast::rms_norm and fast::add_rms_norm (fast/imp.rs:358-412), the normalisation in
//               front of a layer's projections, with the arithmetic of their CPU expansion
//               (fast/imp.rs:1367-1379): float32 squares, their sum in float64 over 8 lanes combined by a
//               fixed tree (kernels.rs:611-624) and rounded to float32, times float32(1 / d), plus eps,
//               1 / sqrt, x * that rounded to the array's type, times the weight rounded again; the sum
//               x + residual of add_rms_norm rounded to the type first.  Every step is an IEEE operation
//               performed in the reference's order: the results are its bits;
//   expert_bias_add  SwitchProjection::forward's `y.add(bias.take(indices, 0))`
//               (crates/nuvec-lm/src/model.rs:2139-2143): every gathered row plus its expert's bias,
//               float32 arithmetic for the halves, one rounding; an index past the end selects the
//               last expert (kernels.rs:120-133).
#include "common.cuh"

#include <initializer_list>
#include <type_traits>

namespace nvc {

template <typename T> struct Glue;
template <> struct Glue<float> {
    static __device__ __forceinline__ float load(const float *p, size_t i) { return p[i]; }
    static __device__ __forceinline__ float from_f32(float x) { return x; }
    static __device__ __forceinline__ float from_f64(double x) { return (float)x; }
    static __device__ __forceinline__ float widen(float x) { return x; }
};
template <> struct Glue<__half> {
    static __device__ __forceinline__ float load(const __half *p, size_t i) { return __half2float(p[i]); }
    static __device__ __forceinline__ __half from_f32(float x) { return __float2half_rn(x); }
    static __device__ __forceinline__ __half from_f64(double x) { return __double2half(x); }  // one rounding from float64
    static __device__ __forceinline__ float widen(__half x) { return __half2float(x); }
};
template <> struct Glue<__nv_bfloat16> {
    static __device__ __forceinline__ float load(const __nv_bfloat16 *p, size_t i) { return __bfloat162float(p[i]); }
    static __device__ __forceinline__ __nv_bfloat16 from_f32(float x) { return __float2bfloat16_rn(x); }
    // bfloat16 from float64 goes through float32 (crates/nuvec-core/src/cast.rs:84-96)
    static __device__ __forceinline__ __nv_bfloat16 from_f64(double x) { return __float2bfloat16_rn((float)x); }
    static __device__ __forceinline__ float widen(__nv_bfloat16 x) { return __bfloat162float(x); }
};

// 16 bytes of a row: PER elements.
template <typename T> struct Piece {
    static constexpr int PER = 16 / sizeof(T);
    T v[PER];
};
template <typename T> __device__ __forceinline__ Piece<T> load_piece(const T *p, int64_t i) {
    const uint4 raw = reinterpret_cast<const uint4 *>(p)[i];
    return *reinterpret_cast<const Piece<T> *>(&raw);
}
template <typename T> __device__ __forceinline__ void store_piece(T *p, int64_t i, const Piece<T> &v) {
    reinterpret_cast<uint4 *>(p)[i] = *reinterpret_cast<const uint4 *>(&v);
}
static bool aligned16(std::initializer_list<const void *> ptrs) {
    uintptr_t all = 0;
    for (const void *p : ptrs) all |= (uintptr_t)p;
    return all % 16 == 0;
}

constexpr int MOE_ROUTE_MAX = 1024;  // experts
constexpr int ROUTE_WARP_MAX = 32;   // the most picks the warp form of the router makes

__device__ __forceinline__ bool route_less(float x, float y) {
    const bool xn = x != x, yn = y != y;
    if (!xn && !yn) return x < y;
    return !xn && yn;
}

// More picks than a warp has lanes: one block per row, one thread per expert: an expert's position in the sorted row is the number
// of experts that sort before it.
template <typename T>
__global__ void __launch_bounds__(MOE_ROUTE_MAX) moe_route_kernel(const T *__restrict__ probs, uint32_t *__restrict__ indices,
                                                                  T *__restrict__ scores, int experts, int k, int normalize) {
    __shared__ float p[MOE_ROUTE_MAX];
    __shared__ float top[MOE_ROUTE_MAX];
    __shared__ float total;
    const int e = threadIdx.x;
    const size_t row = blockIdx.x;
    if (e < experts) p[e] = Glue<T>::load(probs, row * experts + e);
    __syncthreads();
    if (e < experts) {
        const float v = p[e];
        int rank = 0;
        for (int j = 0; j < experts; j++) {
            const float u = p[j];
            rank += (route_less(u, v) || (!route_less(v, u) && j < e)) ? 1 : 0;
        }
        const int slot = rank - (experts - k);
        if (slot >= 0) {
            indices[row * k + slot] = (uint32_t)e;
            top[slot] = v;
        }
    }
    __syncthreads();
    if (normalize) {
        if (e == 0) {
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int j = 0; j < k; j++) acc[j & 7] += (double)top[j];
            const double sum = 0.0 + (((acc[0] + acc[4]) + (acc[1] + acc[5])) + ((acc[2] + acc[6]) + (acc[3] + acc[7])));
            total = Glue<T>::widen(Glue<T>::from_f64(sum));
        }
        __syncthreads();
        if (e < k) scores[row * k + e] = Glue<T>::from_f32(__fdiv_rn(top[e], total));
    } else if (e < k) {
        scores[row * k + e] = Glue<T>::from_f32(top[e]);
    }
}

// The usual router (k up to 32): one warp per row, k rounds of picking the largest left.  Values compare through an
// order-preserving integer (zeros alike, NaN above everything), equal values through their index, so that the picks,
// last first, are the end of the stable ascending order.  A lane keeps every 32nd expert and its own best; only the
// lane that lost its best looks again.  Bound by latency: k x (two warp-wide maxima and a look through E / 32 values)
// after one load, instead of E comparisons per expert (one thread each, the form below for larger k): 512 rows of 128
// experts, k = 8: 12.8 -> 5.2 us under ncu.
template <typename T, int PER>
__global__ void __launch_bounds__(128) moe_route_warp_kernel(const T *__restrict__ probs, uint32_t *__restrict__ indices, T *__restrict__ scores,
                                                             int64_t rows, int experts, int k, int normalize) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    pdl_trigger();
    pdl_wait();
    if (row >= rows) return;
    uint32_t key[PER];  // 0: taken, or no such expert
    const T *src = probs + row * experts;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = i * 32 + lane;
        uint32_t u = 0;
        if (e < experts) {
            const float v = Glue<T>::load(src, e);
            u = __float_as_uint(v);
            u = v != v ? 0xFFFFFFFFu : v == 0.0f ? 0x80000000u : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        }
        key[i] = u;
    }
    uint32_t best = 0;
    int at = -1;
    auto look = [&]() {
        best = 0;
        at = -1;
#pragma unroll
        for (int i = 0; i < PER; i++)
            if (key[i] != 0u && key[i] >= best) {
                best = key[i];
                at = i;
            }
    };
    look();
    float mine = 0.0f;  // lane j ends with pick j of the ascending order
    uint32_t mine_at = 0;
    for (int j = k - 1; j >= 0; j--) {
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, best);
        const uint32_t cand = best == top && at >= 0 ? (uint32_t)(at * 32 + lane) + 1u : 0u;
        const uint32_t e = __reduce_max_sync(0xFFFFFFFFu, cand) - 1u;
        if (lane == j) mine_at = e;
        if (cand == e + 1u) {
#pragma unroll
            for (int i = 0; i < PER; i++)
                if (i == at) key[i] = 0u;
            look();
        }
    }
    if (lane < k) mine = Glue<T>::load(src, mine_at);
    float total = 1.0f;
    if (normalize) {
        // float64 over 8 lanes (pick j into lane j % 8, in order), combined by the fixed tree
        double acc = 0.0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float v = __shfl_sync(0xFFFFFFFFu, mine, (lane & 7) + 8 * r);
            if ((lane & 7) + 8 * r < k) acc += (double)v;
        }
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 4);   // (0+4) (1+5) (2+6) (3+7)
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 1);   // (04+15) (26+37)
        acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 2);
        total = Glue<T>::widen(Glue<T>::from_f64(0.0 + acc));
    }
    if (lane < k) {
        indices[row * k + lane] = mine_at;
        scores[row * k + lane] = Glue<T>::from_f32(normalize ? __fdiv_rn(mine, total) : mine);
    }
}

// One thread per 16 bytes of an output row (element by element where rows are not whole 16-byte pieces).  Bound by
// memory; the k pieces of a column are independent loads.
template <typename T, bool WIDE>
__global__ void __launch_bounds__(256) weighted_sum_kernel(const T *__restrict__ x, const T *__restrict__ w, T *__restrict__ out, int k, int64_t d) {
    constexpr int PER = WIDE ? Piece<T>::PER : 1;
    pdl_trigger();
    const int64_t r = blockIdx.x, c = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x);
    if (c * PER >= d) return;
    pdl_wait();
    const T *xr = x + r * k * d;
    double s[PER];
#pragma unroll
    for (int e = 0; e < PER; e++) s[e] = 0.0;
#pragma unroll 8
    for (int j = 0; j < k; j++) {
        const float wj = Glue<T>::load(w, r * k + j);
        if (WIDE) {
            const Piece<T> p = load_piece(xr + j * d, c);
#pragma unroll
            for (int e = 0; e < PER; e++) s[e] += (double)Glue<T>::widen(Glue<T>::from_f32(__fmul_rn(Glue<T>::widen(p.v[e]), wj)));
        } else {
            s[0] += (double)Glue<T>::widen(Glue<T>::from_f32(__fmul_rn(Glue<T>::load(xr, j * d + c), wj)));
        }
    }
    if (WIDE) {
        Piece<T> o;
#pragma unroll
        for (int e = 0; e < PER; e++) o.v[e % PER] = Glue<T>::from_f64(s[e]);
        store_piece(out + r * d, c, o);
    } else {
        out[r * d + c] = Glue<T>::from_f64(s[0]);
    }
}

}  // namespace nvc

using namespace nvc;

extern "C" int32_t nvc_moe_route(nvc_device *dev, int32_t dtype, const void *probs, int64_t rows, int64_t experts, int64_t k,
                                 int32_t normalize, uint32_t *out_indices, void *out_scores) {
    NVC_TRY(make_current(dev));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_route: probabilities must be floating point (dtype %d)", dtype);
    if (rows < 0 || experts < 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_route: negative size");
    if (k < 1 || k > experts)
        return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_route: k must be in 1..=%lld for probabilities of %lld experts", (long long)experts,
                         (long long)experts);
    if (experts > MOE_ROUTE_MAX)
        return set_error(NVC_ERR_UNSUPPORTED, "moe_route: %lld experts (at most %d)", (long long)experts, MOE_ROUTE_MAX);
    if (rows == 0) return NVC_OK;
    if (!probs || !out_indices || !out_scores) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_route: null operand");
    if (rows > 0x7FFFFFFFll) return set_error(NVC_ERR_UNSUPPORTED, "moe_route: %lld rows exceed the grid limit", (long long)rows);
    if (k <= ROUTE_WARP_MAX) {
        const Writes written(Trigger::EARLY, {{out_indices, (size_t)(rows * k) * 4}, {out_scores, (size_t)(rows * k) * dtype_size(dtype)}});
        const dim3 grid((unsigned)((rows + 3) / 4));
#define NVC_ROUTE(T)                                                                                                                     \
    {                                                                                                                                    \
        auto kernel = experts <= 32    ? moe_route_warp_kernel<T, 1>                                                                     \
                      : experts <= 128 ? moe_route_warp_kernel<T, 4>                                                                     \
                      : experts <= 256 ? moe_route_warp_kernel<T, 8>                                                                     \
                                       : moe_route_warp_kernel<T, 32>;                                                                   \
        return launch_pdl(dev, "moe_route_warp_kernel", written, kernel, grid, dim3(128), 0, (const T *)probs, out_indices, (T *)out_scores, rows, \
                          (int)experts, (int)k, normalize);                                                                              \
    }
        switch (dtype) {
        case NVC_F32: NVC_ROUTE(float)
        case NVC_F16: NVC_ROUTE(__half)
        default: NVC_ROUTE(__nv_bfloat16)
        }
#undef NVC_ROUTE
    }
    const unsigned threads = (unsigned)((experts + 31) / 32 * 32);
    switch (dtype) {
    case NVC_F32:
        moe_route_kernel<float><<<(unsigned)rows, threads, 0, dev->stream>>>((const float *)probs, out_indices, (float *)out_scores,
                                                                            (int)experts, (int)k, normalize);
        break;
    case NVC_F16:
        moe_route_kernel<__half><<<(unsigned)rows, threads, 0, dev->stream>>>((const __half *)probs, out_indices, (__half *)out_scores,
                                                                             (int)experts, (int)k, normalize);
        break;
    default:
        moe_route_kernel<__nv_bfloat16><<<(unsigned)rows, threads, 0, dev->stream>>>((const __nv_bfloat16 *)probs, out_indices,
                                                                                    (__nv_bfloat16 *)out_scores, (int)experts, (int)k, normalize);
    }
    return check_launch(dev, "moe_route_kernel");
}

// Stable sort of `pairs` expert indices by one block.  Warp w owns the w-th run of pairs.  First every warp counts its
// run's experts in its row of a [warp][expert] table; then the table's columns, and the columns' totals across the
// experts, are turned into first places; then every warp walks its run again, 32 pairs at a time: the lanes that hold
// the same expert rank themselves (__match_any_sync) and the last of them moves the warp's next place for it on.
// Warps, rounds and lanes follow the pairs' order, so an expert's pairs keep theirs: the reference's stable sort.
// Bound by latency of one block (pairs are read twice, from L1 the second time); three block-wide barriers in all
// whatever the number of pairs.  4096 pairs of 128 experts 18.3 -> 11.7 us under ncu against rounds of 1024 pairs with four
// barriers and a serial scan each.  At most MOE_ROUTE_MAX experts.
__global__ void __launch_bounds__(1024) moe_sort_kernel(const uint32_t *__restrict__ indices, int64_t pairs, uint32_t k, uint32_t experts,
                                                        uint32_t *__restrict__ order, uint32_t *__restrict__ restore,
                                                        uint32_t *__restrict__ tokens, uint32_t *__restrict__ sorted,
                                                        int32_t *__restrict__ offsets) {
    extern __shared__ uint32_t table[];  // [32 warps][experts]
    __shared__ uint32_t warp_sum[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const int64_t run = ((pairs + 31) / 32 + 31) / 32 * 32;  // whole rounds of 32
    const int64_t lo = min(run * warp, pairs), hi = min(lo + run, pairs);
    uint32_t *mine = table + warp * experts;
    for (uint32_t c = lane; c < experts; c += 32u) mine[c] = 0u;
    __syncwarp();
    pdl_wait();
    for (int64_t i = lo + lane; i < hi; i += 32) atomicAdd(mine + min(indices[i], experts - 1u), 1u);
    __syncthreads();
    // expert tid: its count, and the counts before it within each warp
    uint32_t total = 0;
    if (tid < experts) {
#pragma unroll 8
        for (uint32_t w = 0; w < 32u; w++) {
            const uint32_t n = table[w * experts + tid];
            table[w * experts + tid] = total;
            total += n;
        }
    }
    uint32_t scan = total;  // inclusive over the experts of a warp, then over the warps
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, scan, o);
        if (lane >= o) scan += v;
    }
    if (lane == 31u) warp_sum[warp] = scan;
    __syncthreads();
    uint32_t before = lane < warp ? warp_sum[lane] : 0u;
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    const uint32_t base = before + scan - total;
    if (tid < experts) {
        if (offsets) offsets[tid] = (int32_t)base;
#pragma unroll 8
        for (uint32_t w = 0; w < 32u; w++) table[w * experts + tid] += base;
    }
    __syncthreads();
    for (int64_t i0 = lo; i0 < hi; i0 += 32) {
        const int64_t i = i0 + lane;
        const bool have = i < hi;
        const uint32_t e = have ? min(indices[i], experts - 1u) : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, e);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (have) {
            const uint32_t pos = mine[e] + rank;
            order[pos] = (uint32_t)i;
            restore[i] = pos;
            if (tokens) tokens[pos] = (uint32_t)i / k;
            if (sorted) sorted[pos] = e;
        }
        __syncwarp();
        if (have && (peers >> lane) == 1u) mine[e] += rank + 1u;  // the highest lane of the expert's
        __syncwarp();
    }
}

// out[i, :] = src[min(idx[i], src_rows - 1), :], rows of row_bytes bytes; 16-byte pieces when everything is aligned.
__global__ void __launch_bounds__(256) take_rows_kernel(const uint8_t *__restrict__ src, int64_t src_rows, int64_t row_bytes,
                                                        const uint32_t *__restrict__ idx, uint8_t *__restrict__ out, int wide) {
    const int64_t i = blockIdx.x;
    pdl_wait();
    const int64_t from = min((int64_t)idx[i], src_rows - 1);
    const uint8_t *a = src + from * row_bytes;
    uint8_t *b = out + i * row_bytes;
    if (wide) {
        for (int64_t c = threadIdx.x; c < row_bytes / 16; c += 512) {  // two pieces in flight (4096 rows of 5760 bytes: 10.1 -> 8.6 us)
            const bool two = c + 256 < row_bytes / 16;
            const uint4 v = reinterpret_cast<const uint4 *>(a)[c];
            uint4 w;
            if (two) w = reinterpret_cast<const uint4 *>(a)[c + 256];
            reinterpret_cast<uint4 *>(b)[c] = v;
            if (two) reinterpret_cast<uint4 *>(b)[c + 256] = w;
        }
    } else {
        for (int64_t c = threadIdx.x; c < row_bytes; c += 256) b[c] = a[c];
    }
}

// MLX's Sigmoid in float32 (kernels.rs:1538-1543): y = 1 / (1 + exp(|x|)), then x < 0 ? y : 1 - y.
__device__ __forceinline__ float sigmoid_f32(float x) {
    const float a = x < 0.0f ? -x : x;
    const float y = __frcp_rn(__fadd_rn(1.0f, expf(a)));
    return x < 0.0f ? y : __fsub_rn(1.0f, y);
}
__device__ __noinline__ float sigmoid_f32_call(float x) { return sigmoid_f32(x); }
// The sigmoid rounded to T, the same value as rounding sigmoid_f32's.  For the 16-bit types the approximate exponential and
// reciprocal decide nearly always.  Up to |x| = 16 (float16: 8, so that the result is a normal number) they and sigmoid_f32
// differ by less than 2^-18.8, relatively -- |x| log2(e) < 24 is off by 2^-20 from rounding and as much from the constant, ex2
// by 2^-22, rcp by 2^-23, sigmoid_f32 itself by 2^-21 -- at most 37 units in the last place; so a result more than 64 units from
// the middle between two values of T rounds like the exact one.  The others (one in 500; float16: one in 60) take the exact
// path.  That path for every element, about 75 instructions, bound the kernel: 4096 x 2880, swiglu_oai: 24 us, 20 since.
template <typename T> __device__ __forceinline__ float sigmoid_rounded(float x) {
    if constexpr (sizeof(T) == 4) {
        return sigmoid_f32(x);
    } else {
        constexpr bool HALF = std::is_same<T, __half>::value;
        constexpr uint32_t MIDDLE = HALF ? 0x1000u : 0x8000u;
        const float a = fabsf(x);
        float e, y;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(__fmul_rn(a, 1.4426950408889634f)));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__fadd_rn(1.0f, e)));
        float s = x < 0.0f ? y : __fsub_rn(1.0f, y);
        const uint32_t from_middle = (__float_as_uint(s) & (2u * MIDDLE - 1u)) - (MIDDLE - 64u);  // below 129: too close
        if (from_middle <= 128u || !(a <= (HALF ? 8.0f : 16.0f))) s = sigmoid_f32_call(x);
        return Glue<T>::widen(Glue<T>::from_f32(s));
    }
}
// minimum / maximum that propagate NaN (kernels.rs:1366-1367)
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// out = silu(gate) * up, op by op: s = sigmoid(g), t = g * s, out = t * up, each rounded to T.
// OAI form (alpha, limit already rounded to T): g = min(gate, limit), x = min(max(up, -limit), limit),
// out = (x + 1) * (g * sigmoid(alpha * g)), each operation rounded to T.
// One thread per 16 bytes of each operand (element by element where they are not aligned): bound by the issue of the
// ~30 float32 operations per element the roundings need; 16-byte accesses and one reciprocal (correctly rounded, the
// same number as the division 1 / x) took the OAI form at 4096 x 2880 from 40.8 to 24.7 us under ncu.
template <typename T, bool OAI, bool WIDE>
__global__ void __launch_bounds__(256) swiglu_kernel(const T *__restrict__ gate, const T *__restrict__ up, T *__restrict__ out, int64_t n,
                                                     float alpha, float limit) {
    constexpr int PER = WIDE ? Piece<T>::PER : 1;
    pdl_trigger();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i * PER >= n) return;
    pdl_wait();
    auto r = [](float v) { return Glue<T>::widen(Glue<T>::from_f32(v)); };  // one rounding to T
    auto one = [&](float g, float x) {
        if (OAI) {
            g = min_nan(g, limit);
            x = min_nan(max_nan(x, -limit), limit);
            const float s = sigmoid_rounded<T>(r(__fmul_rn(alpha, g)));
            const float gs = r(__fmul_rn(g, s));
            return Glue<T>::from_f32(__fmul_rn(r(__fadd_rn(x, 1.0f)), gs));
        } else {
            const float s = sigmoid_rounded<T>(g);
            const float t = r(__fmul_rn(g, s));
            return Glue<T>::from_f32(__fmul_rn(t, x));
        }
    };
    if (WIDE && (i + 1) * PER <= n) {
        const Piece<T> g = load_piece(gate, i), x = load_piece(up, i);
        Piece<T> o;
#pragma unroll
        for (int e = 0; e < PER; e++) o.v[e % Piece<T>::PER] = one(Glue<T>::widen(g.v[e % Piece<T>::PER]), Glue<T>::widen(x.v[e % Piece<T>::PER]));
        store_piece(out, i, o);
    } else {
        for (int64_t e = i * PER; e < n && e < (i + 1) * PER; e++) out[e] = one(Glue<T>::load(gate, e), Glue<T>::load(up, e));
    }
}

// One block per row.  The reference adds the squares in float64, eight lanes each in its order, and rounds the total to
// float32.  Any other order of the same float64 additions differs from that total by a relative d * 2^-52 at most
// (every term is non-negative), so the row is summed by all threads at once, and where both ends of that interval round
// to the same float32 -- all but about one row in 10^5 -- that is the reference's value; otherwise eight threads repeat
// the sum in its order.  The row is read once and kept in registers (NV pieces of 16 bytes per thread; NV = 0: longer
// or unaligned rows, read twice).  Bound by latency: a row of 4096 at M = 1 took 15 us under ncu while eight
// threads added 512 dependent float64 each, 4 us now.
template <typename T, int NV>
__global__ void __launch_bounds__(1024) rms_norm_kernel(const T *__restrict__ x, const T *__restrict__ residual, const T *__restrict__ weight,
                                                        T *__restrict__ sum_out, T *__restrict__ y, int64_t d, float eps, float inv_count) {
    constexpr int PER = Piece<T>::PER, HELD = NV ? NV : 1;
    __shared__ double part[32];
    __shared__ float again;
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, threads = blockDim.x;
    const T *xr = x + (size_t)blockIdx.x * d;
    const T *rr = residual ? residual + (size_t)blockIdx.x * d : nullptr;
    T *hr = sum_out ? sum_out + (size_t)blockIdx.x * d : nullptr;
    T *yr = y + (size_t)blockIdx.x * d;
    const int64_t pieces = d / PER;
    Piece<T> held[HELD];
    double acc = 0.0;
    pdl_wait();
    if (NV) {
        Piece<T> other[HELD];
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int64_t at = tid + (int64_t)i * threads;
            if (at < pieces) {
                held[i] = load_piece(xr, at);
                if (rr) other[i] = load_piece(rr, at);
            }
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int64_t at = tid + (int64_t)i * threads;
            if (at >= pieces) break;
            if (rr) {
#pragma unroll
                for (int e = 0; e < PER; e++)
                    held[i].v[e] = Glue<T>::from_f32(__fadd_rn(Glue<T>::widen(held[i].v[e]), Glue<T>::widen(other[i].v[e])));  // x + residual, rounded to T
                store_piece(hr, at, held[i]);
            }
#pragma unroll
            for (int e = 0; e < PER; e++) {
                const float v = Glue<T>::widen(held[i].v[e]);
                acc = __dadd_rn(acc, (double)__fmul_rn(v, v));
            }
        }
    } else {
        for (int64_t j = tid; j < d; j += threads) {
            float v = Glue<T>::load(xr, j);
            if (rr) {
                const T h = Glue<T>::from_f32(__fadd_rn(v, Glue<T>::load(rr, j)));
                hr[j] = h;
                v = Glue<T>::widen(h);
            }
            acc = __dadd_rn(acc, (double)__fmul_rn(v, v));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = __dadd_rn(acc, __shfl_xor_sync(0xFFFFFFFFu, acc, o));
    if (lane == 0) part[tid >> 5] = acc;
    __syncthreads();
    double total = lane < threads / 32 ? part[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total = __dadd_rn(total, __shfl_xor_sync(0xFFFFFFFFu, total, o));
    const double slack = ((double)d + 64.0) * 2.220446049250313e-16;
    float sum = __double2float_rn(total * (1.0 - slack));
    if (!(sum == __double2float_rn(total * (1.0 + slack)))) {  // (the same decision in every thread)
        double *lanes = part;
        __syncthreads();  // part has been read; hr is written
        if (tid < 8) {
            double seq = 0.0;
            for (int64_t j = tid; j < d; j += 8) {
                const float v = rr ? Glue<T>::widen(hr[j]) : Glue<T>::load(xr, j);
                seq = __dadd_rn(seq, (double)__fmul_rn(v, v));
            }
            lanes[tid] = seq;
        }
        __syncthreads();
        if (tid == 0)
            again = __double2float_rn(__dadd_rn(__dadd_rn(__dadd_rn(lanes[0], lanes[4]), __dadd_rn(lanes[1], lanes[5])),
                                                __dadd_rn(__dadd_rn(lanes[2], lanes[6]), __dadd_rn(lanes[3], lanes[7]))));
        __syncthreads();
        sum = again;
    }
    const float n = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(sum, inv_count), eps)));
    if (NV) {
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int64_t at = tid + (int64_t)i * threads;
            if (at >= pieces) break;
            Piece<T> o;
            Piece<T> wt;
            if (weight) wt = load_piece(weight, at);
#pragma unroll
            for (int e = 0; e < PER; e++) {
                o.v[e] = Glue<T>::from_f32(__fmul_rn(Glue<T>::widen(held[i].v[e]), n));
                if (weight) o.v[e] = Glue<T>::from_f32(__fmul_rn(Glue<T>::widen(o.v[e]), Glue<T>::widen(wt.v[e])));
            }
            store_piece(yr, at, o);
        }
    } else {
        for (int64_t j = tid; j < d; j += threads) {
            const float v = rr ? Glue<T>::widen(hr[j]) : Glue<T>::load(xr, j);
            T out = Glue<T>::from_f32(__fmul_rn(v, n));
            if (weight) out = Glue<T>::from_f32(__fmul_rn(Glue<T>::widen(out), Glue<T>::load(weight, j)));
            yr[j] = out;
        }
    }
}

// y[r, c] += bias[indices[r], c]: one block per row; 16-byte pieces when the rows allow it.
template <typename T>
__global__ void __launch_bounds__(256) expert_bias_add_kernel(T *__restrict__ y, const T *__restrict__ bias,
                                                              const uint32_t *__restrict__ indices, int64_t n, uint32_t experts, int wide) {
    const int64_t r = blockIdx.x;
    pdl_trigger();
    pdl_wait();
    const uint32_t e = min(indices[r], experts - 1u);
    T *row = y + r * n;
    const T *b = bias + (size_t)e * n;
    constexpr int PER = 16 / sizeof(T);
    if (wide) {
        for (int64_t c = threadIdx.x; c < n / PER; c += 256) {
            uint4 a = reinterpret_cast<uint4 *>(row)[c];
            const uint4 q = reinterpret_cast<const uint4 *>(b)[c];
            T *av = reinterpret_cast<T *>(&a);
            const T *qv = reinterpret_cast<const T *>(&q);
#pragma unroll
            for (int v = 0; v < PER; v++) av[v] = Glue<T>::from_f32(Glue<T>::widen(av[v]) + Glue<T>::widen(qv[v]));
            reinterpret_cast<uint4 *>(row)[c] = a;
        }
    } else {
        for (int64_t c = threadIdx.x; c < n; c += 256) row[c] = Glue<T>::from_f32(Glue<T>::widen(row[c]) + Glue<T>::load(b, c));
    }
}

extern "C" int32_t nvc_weighted_sum(nvc_device *dev, int32_t dtype, const void *x, const void *w, int64_t rows, int64_t k, int64_t d,
                                    void *out) {
    NVC_TRY(make_current(dev));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_INVALID_ARGUMENT, "weighted_sum: x must be floating point (dtype %d)", dtype);
    if (rows < 0 || k < 0 || d < 0 || k > 0x7FFFFFFFll) return set_error(NVC_ERR_INVALID_ARGUMENT, "weighted_sum: invalid shape");
    if (rows * d == 0) return NVC_OK;
    if (!out || (k > 0 && (!x || !w))) return set_error(NVC_ERR_INVALID_ARGUMENT, "weighted_sum: null operand");
    if (rows > 0x7FFFFFFFll) return set_error(NVC_ERR_UNSUPPORTED, "weighted_sum: %lld rows exceed the grid limit", (long long)rows);
    const int64_t per = 16 / (int64_t)dtype_size(dtype);
    // (few rows: an element per thread spreads the float64 sums over more multiprocessors)
    const bool wide = d % per == 0 && aligned16({x, out}) && rows * d >= 64 * 1024;
    const int64_t cols = wide ? d / per : d;
    const unsigned threads = (unsigned)(cols >= 256 ? 256 : (cols + 31) / 32 * 32);
    const int64_t chunks = (cols + threads - 1) / threads;
    if (chunks > 65535) return set_error(NVC_ERR_UNSUPPORTED, "weighted_sum: %lld columns exceed the grid limit", (long long)d);
    const Writes written(Trigger::EARLY, {{out, (size_t)(rows * d) * dtype_size(dtype)}});
#define NVC_WSUM(T)                                                                                                                                 \
    return launch_pdl(dev, "weighted_sum_kernel", written, wide ? weighted_sum_kernel<T, true> : weighted_sum_kernel<T, false>,                              \
                      dim3((unsigned)rows, (unsigned)chunks), dim3(threads), 0, (const T *)x, (const T *)w, (T *)out, (int)k, d);
    switch (dtype) {
    case NVC_F32: NVC_WSUM(float)
    case NVC_F16: NVC_WSUM(__half)
    default: NVC_WSUM(__nv_bfloat16)
    }
#undef NVC_WSUM
}

extern "C" int32_t nvc_expert_bias_add(nvc_device *dev, int32_t dtype, void *y, const void *bias, const uint32_t *indices, int64_t rows,
                                       int64_t n, int64_t experts) {
    NVC_TRY(make_current(dev));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_INVALID_ARGUMENT, "expert_bias_add: y must be floating point (dtype %d)", dtype);
    if (rows < 0 || n < 0 || experts < 0 || experts > 0xFFFFFFFFll) return set_error(NVC_ERR_INVALID_ARGUMENT, "expert_bias_add: invalid shape");
    if (rows * n == 0) return NVC_OK;
    if (experts == 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "expert_bias_add: no experts to take a bias from");
    if (!y || !bias || !indices) return set_error(NVC_ERR_INVALID_ARGUMENT, "expert_bias_add: null operand");
    if (rows > 0x7FFFFFFFll) return set_error(NVC_ERR_UNSUPPORTED, "expert_bias_add: %lld rows exceed the grid limit", (long long)rows);
    const size_t item = dtype == NVC_F32 ? 4 : 2;
    const int wide = (n * item) % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)bias % 16 == 0;
    const Writes written(Trigger::EARLY, {{y, (size_t)(rows * n) * item}});
#define NVC_BIAS(T)                                                                                                                               \
    return launch_pdl(dev, "expert_bias_add_kernel", written, expert_bias_add_kernel<T>, dim3((unsigned)rows), dim3(256), 0, (T *)y, (const T *)bias, indices, \
                      n, (uint32_t)experts, wide);
    switch (dtype) {
    case NVC_F32: NVC_BIAS(float)
    case NVC_F16: NVC_BIAS(__half)
    default: NVC_BIAS(__nv_bfloat16)
    }
#undef NVC_BIAS
}

extern "C" int32_t nvc_moe_sort(nvc_device *dev, const uint32_t *indices, int64_t pairs, int64_t k, int64_t experts, uint32_t *out_order,
                                uint32_t *out_restore, uint32_t *out_tokens, uint32_t *out_sorted, int32_t *out_offsets) {
    NVC_TRY(make_current(dev));
    if (pairs < 0 || k < 1 || experts < 0 || pairs > 0x7FFFFFFFll) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_sort: invalid shape");
    if (experts > MOE_ROUTE_MAX) return set_error(NVC_ERR_UNSUPPORTED, "moe_sort: %lld experts (at most %d)", (long long)experts, MOE_ROUTE_MAX);
    if (pairs > 0 && experts == 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_sort: pairs without experts");
    if (pairs == 0 && experts == 0) return NVC_OK;
    if ((pairs > 0 && (!indices || !out_order || !out_restore))) return set_error(NVC_ERR_INVALID_ARGUMENT, "moe_sort: null operand");
    const size_t smem = (size_t)32 * (size_t)experts * sizeof(uint32_t);
    if (smem > 48 * 1024) {
        static std::mutex mu;
        static bool configured[64] = {};
        if (dev->ordinal < 0 || dev->ordinal >= 64) return set_error(NVC_ERR_UNSUPPORTED, "moe_sort: device ordinal %d", dev->ordinal);
        std::lock_guard<std::mutex> g(mu);
        if (!configured[dev->ordinal]) {
            NVC_CUDA(cudaFuncSetAttribute(moe_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * MOE_ROUTE_MAX * (int)sizeof(uint32_t)));
            configured[dev->ordinal] = true;
        }
    }
    const size_t list = (size_t)pairs * 4;
    const Writes written(Trigger::LATE, {{out_order, list}, {out_restore, list}, {out_tokens, list}, {out_sorted, list}, {out_offsets, (size_t)experts * 4}});
    return launch_pdl(dev, "moe_sort_kernel", written, moe_sort_kernel, dim3(1), dim3(1024), smem, indices, pairs, (uint32_t)k, (uint32_t)experts, out_order,
                      out_restore, out_tokens, out_sorted, out_offsets);
}

extern "C" int32_t nvc_take_rows(nvc_device *dev, const void *src, int64_t src_rows, int64_t row_bytes, const uint32_t *indices, int64_t n,
                                 void *out) {
    NVC_TRY(make_current(dev));
    if (src_rows < 0 || row_bytes < 0 || n < 0 || n > 0x7FFFFFFFll) return set_error(NVC_ERR_INVALID_ARGUMENT, "take_rows: invalid shape");
    if (n * row_bytes == 0) return NVC_OK;
    if (src_rows == 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "take_rows: rows taken from an empty array");
    if (!src || !indices || !out) return set_error(NVC_ERR_INVALID_ARGUMENT, "take_rows: null operand");
    const int wide = row_bytes % 16 == 0 && (uintptr_t)src % 16 == 0 && (uintptr_t)out % 16 == 0;
    const Writes written(Trigger::LATE, {{out, (size_t)(n * row_bytes)}});
    return launch_pdl(dev, "take_rows_kernel", written, take_rows_kernel, dim3((unsigned)n), dim3(256), 0, (const uint8_t *)src, src_rows, row_bytes, indices,
                      (uint8_t *)out, wide);
}

template <bool OAI>
static int32_t launch_swiglu(nvc_device *dev, const char *op, int32_t dtype, const void *gate, const void *up, int64_t n, float alpha,
                             float limit, void *out) {
    NVC_TRY(make_current(dev));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: operands must be floating point (dtype %d)", op, dtype);
    if (n < 0) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: invalid size", op);
    if (n == 0) return NVC_OK;
    if (!gate || !up || !out) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: null operand", op);
    const bool wide = aligned16({gate, up, out});
    const int64_t per = wide ? 16 / (int64_t)dtype_size(dtype) : 1;
    const int64_t blocks = ((n + per - 1) / per + 255) / 256;
    if (blocks > 0x7FFFFFFFll) return set_error(NVC_ERR_UNSUPPORTED, "%s: %lld elements exceed the grid limit", op, (long long)n);
    const Writes written(Trigger::EARLY, {{out, (size_t)n * dtype_size(dtype)}});
#define NVC_SWIGLU(T, A, L)                                                                                                                        \
    return launch_pdl(dev, "swiglu_kernel", written, wide ? swiglu_kernel<T, OAI, true> : swiglu_kernel<T, OAI, false>, dim3((unsigned)blocks), dim3(256), 0, \
                      (const T *)gate, (const T *)up, (T *)out, n, A, L);
    // (the scalars are weak: rounded to the arrays' type, crates/nuvec-nn/src/lib.rs:504-507)
    switch (dtype) {
    case NVC_F32: NVC_SWIGLU(float, alpha, limit)
    case NVC_F16: NVC_SWIGLU(__half, __half2float(__float2half_rn(alpha)), __half2float(__float2half_rn(limit)))
    default: NVC_SWIGLU(__nv_bfloat16, __bfloat162float(__float2bfloat16_rn(alpha)), __bfloat162float(__float2bfloat16_rn(limit)))
    }
#undef NVC_SWIGLU
}

extern "C" int32_t nvc_swiglu(nvc_device *dev, int32_t dtype, const void *gate, const void *up, int64_t n, void *out) {
    return launch_swiglu<false>(dev, "swiglu", dtype, gate, up, n, 0.0f, 0.0f, out);
}

extern "C" int32_t nvc_swiglu_oai(nvc_device *dev, int32_t dtype, const void *gate, const void *up, float alpha, float limit, int64_t n,
                                  void *out) {
    return launch_swiglu<true>(dev, "swiglu_oai", dtype, gate, up, n, alpha, limit, out);
}

constexpr int RMS_MAX_D = 51180;  // longest row taken

static int32_t launch_rms_norm(nvc_device *dev, const char *op, int32_t dtype, const void *x, const void *residual, const void *weight, float eps,
                               int64_t rows, int64_t d, void *sum_out, void *y) {
    NVC_TRY(make_current(dev));
    if (!is_float_dtype(dtype)) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: the input must be floating point (dtype %d)", op, dtype);
    if (rows < 0 || d < 0 || rows > 0x7FFFFFFFll) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: invalid shape", op);
    if (rows * d == 0) return NVC_OK;
    if (!x || !y || (residual && !sum_out)) return set_error(NVC_ERR_INVALID_ARGUMENT, "%s: null operand", op);
    if (d > RMS_MAX_D) return set_error(NVC_ERR_UNSUPPORTED, "%s: rows of %lld elements (at most %d)", op, (long long)d, RMS_MAX_D);
    const float inv_count = (float)(1.0 / (double)d);
    // Rows of whole 16-byte pieces stay in registers: one piece per thread up to 1024 of them, then up to four.
    const int64_t per = 16 / (int64_t)dtype_size(dtype), pieces = d / per;
    const bool wide = d % per == 0 && pieces <= 4096 && aligned16({x, residual, weight, sum_out, y});
    const int nv = !wide ? 0 : pieces <= 1024 ? 1 : pieces <= 2048 ? 2 : 4;
    const int64_t want = nv ? (pieces + nv - 1) / nv : d;
    const unsigned threads = (unsigned)(want >= 1024 ? 1024 : (want + 31) / 32 * 32);
    const size_t bytes = (size_t)(rows * d) * dtype_size(dtype);
    const Writes written(Trigger::EARLY, {{y, bytes}, {sum_out, bytes}});
#define NVC_RMS(T)                                                                                                                              \
    return launch_pdl(dev, "rms_norm_kernel", written,                                                                                                   \
                      nv == 0 ? rms_norm_kernel<T, 0> : nv == 1 ? rms_norm_kernel<T, 1> : nv == 2 ? rms_norm_kernel<T, 2> : rms_norm_kernel<T, 4>, \
                      dim3((unsigned)rows), dim3(threads), 0, (const T *)x, (const T *)residual, (const T *)weight, (T *)sum_out, (T *)y, d, eps, inv_count);
    switch (dtype) {
    case NVC_F32: NVC_RMS(float)
    case NVC_F16: NVC_RMS(__half)
    default: NVC_RMS(__nv_bfloat16)
    }
#undef NVC_RMS
}

extern "C" int32_t nvc_rms_norm(nvc_device *dev, int32_t dtype, const void *x, const void *weight, float eps, int64_t rows, int64_t d, void *y) {
    return launch_rms_norm(dev, "rms_norm", dtype, x, nullptr, weight, eps, rows, d, nullptr, y);
}

extern "C" int32_t nvc_add_rms_norm(nvc_device *dev, int32_t dtype, const void *x, const void *residual, const void *weight, float eps,
                                    int64_t rows, int64_t d, void *out_sum, void *y) {
    if (!residual) return set_error(NVC_ERR_INVALID_ARGUMENT, "add_rms_norm: null residual");
    return launch_rms_norm(dev, "add_rms_norm", dtype, x, residual, weight, eps, rows, d, out_sum, y);
}
