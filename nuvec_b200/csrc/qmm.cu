// Host side of the many-row products (qmm_kernel.cuh): eligibility, tensor maps, choice of the token tile.  The kernel's
// instantiations live in qmm_bf16.cu, qmm_f16.cu and qmm_fp.cu.
#include "qmm_kernel.cuh"

#include <cstdlib>
#include <cstring>

namespace nvc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

int32_t make_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, uint64_t inner, uint64_t rows, uint64_t pitch_bytes, uint32_t box_inner,
                 uint32_t box_rows, int swizzle) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return set_error(NVC_ERR_DRIVER, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {inner, rows}, strides[1] = {pitch_bytes};
    cuuint32_t box[2] = {box_inner, box_rows}, estr[2] = {1, 1};
    CUresult r = fn(map, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                    : swizzle == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                    : swizzle == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                    : CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(NVC_ERR_DRIVER, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return NVC_OK;
}

bool qmm_eligible(int32_t mode, int32_t gs, int32_t bits, int32_t dtype, int32_t transpose, int64_t M, int64_t N,
                  int64_t K, const void *x, int64_t ldx, const uint32_t *w) {
    (void)gs;
    static const bool disabled = getenv("NUVEC_QMM_DISABLE") != nullptr;  // read once: products then take the other kernels
    if (disabled) return false;
    if (dtype == NVC_F32 || !transpose) return false;
    if (mode == NVC_AFFINE) {
        if (bits != 2 && bits != 3 && bits != 4 && bits != 6 && bits != 8) return false;
    } else if (dtype != NVC_BF16) {  // (a floating-point mode's scales do not fit float16)
        return false;
    } else if (mode == NVC_MXFP8) {
        if (bits != 8) return false;
    } else if (mode != NVC_MXFP4 && mode != NVC_NVFP4) {
        return false;
    }
    if (M < 1 || N < 1 || K < QMM_BK || K % QMM_BK != 0) return false;
    if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return false;
    // TMA: 16-byte aligned bases and row pitches
    if ((uintptr_t)x % 16 != 0 || (ldx * 2) % 16 != 0) return false;
    if ((uintptr_t)w % 16 != 0 || (K * bits / 8) % 16 != 0) return false;
    return true;
}

// Scratch of the K-split tiles: float32 partial tiles and their arrival counters, owned by the
// device handle (kept apart from the few-row kernel's scratch, which a gather may be using for
// its expert offsets at the same time).  Counters are zero between launches.
int32_t ensure_qmm_scratch(nvc_device *dev, size_t bytes, size_t counters) {
    if (dev->qmm_partials_bytes < bytes) {
        NVC_CUDA(cudaStreamSynchronize(dev->stream));
        if (dev->qmm_partials) dev->pool.free(dev->qmm_partials);
        dev->qmm_partials = nullptr;
        dev->qmm_partials_bytes = 0;
        NVC_TRY(dev->pool.alloc(bytes, &dev->qmm_partials));
        dev->qmm_partials_bytes = bytes;
    }
    if (dev->qmm_counters_len < counters) {
        NVC_CUDA(cudaStreamSynchronize(dev->stream));
        if (dev->qmm_counters) dev->pool.free(dev->qmm_counters);
        dev->qmm_counters = nullptr;
        dev->qmm_counters_len = 0;
        const size_t len = counters < 256 ? 256 : counters;
        void *ptr = nullptr;
        NVC_TRY(dev->pool.alloc(len * sizeof(uint32_t), &ptr));
        NVC_CUDA(cudaMemsetAsync(ptr, 0, len * sizeof(uint32_t), dev->stream));
        dev->qmm_counters = (uint32_t *)ptr;
        dev->qmm_counters_len = len;
    }
    return NVC_OK;
}

int32_t launch_qmm(nvc_device *dev, const QmmParams &p) {
    if (p.rows == 0 || p.N == 0) return NVC_OK;
    const int64_t experts = p.offsets ? p.experts : 1;
    NVC_TRY(ensure_error_word(dev));
    const QmmPlan plan = qmm_plan(p.rows, p.offsets ? experts : 0, p.N, (int)(p.K / QMM_BK), p.bits, dev->prop.multiProcessorCount);
    const int bt = plan.bt;
    const bool pair = plan.pair;
    const int64_t token_tiles = (p.rows + bt - 1) / bt + (p.offsets ? experts : 0);  // grouped: at most, one partial tile per expert
    const bool affine = p.mode == NVC_AFFINE;
    QmmKernelParams kp{};
    kp.scales = (const uint8_t *)p.scales;
    kp.biases = affine ? (const uint8_t *)p.biases : nullptr;
    kp.global = p.global;
    kp.y = (uint16_t *)p.y;
    kp.offsets = p.offsets;
    kp.error = dev->error_word_dev;
    kp.experts = (int32_t)experts;
    kp.rows = (int32_t)p.rows;
    kp.N = (int32_t)p.N;
    kp.K = (int32_t)p.K;
    kp.gs_shift = p.gs == 16 ? 4 : p.gs == 32 ? 5 : p.gs == 64 ? 6 : 7;
    kp.scale_row_bytes = (int32_t)(p.K / p.gs * (affine ? 2 : 1));
    kp.expert_global = p.expert_global;
    const size_t w_bytes = (size_t)(experts * p.N) * (size_t)(p.K * p.bits / 8), s_bytes = (size_t)(experts * p.N) * (size_t)kp.scale_row_bytes;
    kp.early = early_read_ok(dev, p.w, w_bytes) && early_read_ok(dev, p.scales, s_bytes) && (!affine || early_read_ok(dev, p.biases, s_bytes));
    if (!affine) return qmm_launch_fp(dev, bt, pair, p, kp, token_tiles);
    return p.dtype == NVC_F16 ? qmm_launch_f16(dev, bt, pair, p, kp, token_tiles) : qmm_launch_bf16(dev, bt, pair, p, kp, token_tiles);
}

}  // namespace nvc
