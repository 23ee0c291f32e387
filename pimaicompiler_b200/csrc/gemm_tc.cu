// Host side of the dense contraction  Y[j,n] = act(sum_k X[j,k] W[n,k] + b[n]):  the router over its kernels, the
// tensor-map encoders and the per-device status block of the tcgen05 kernel (gemm_rows.cu).
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "gemm_rows.cuh"
#include "tc_common.cuh"

namespace pimb200 {

int launch_gemm_wx_ragged(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx, int ldy, int act,
                          int y_is_f32, cudaStream_t st);
int launch_gemm_wx_simt(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx,
                        int ldy, int act, int y_is_f32, cudaStream_t st);

namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static std::mutex g_mu;
static EncodeTiledFn g_encode = nullptr;
static bool g_encode_tried = false;
constexpr int kMaxDevices = 64;
static int* g_status[kMaxDevices];       // per device: {sticky error code, generation of the launch that gave up}
static int g_gen = 0;                    // launch generation, never 0

EncodeTiledFn get_encode() {
    if (g_encode_tried) return g_encode;
    g_encode_tried = true;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
        g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    else
        cudaGetLastError();
    return g_encode;
}

// rows x cols of 2-byte (fp16) or 4-byte (fp32) elements, tiles of box_rows rows x 128 bytes, 128-byte swizzle
bool encode_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t row_stride_bytes, uint32_t box_rows,
               int elem_bytes) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return g_encode(map, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base),
                    dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// X as [batch][seq_rows >= steps][K] (row (b, t) at (b*seq_rows + t) * ldx), tiles of box_t timesteps x all `batch` sequences
bool encode_x_time_major(CUtensorMap* map, const void* base, uint64_t batch, uint64_t steps, uint64_t seq_rows,
                                uint64_t cols, uint64_t ldx_bytes, uint32_t box_t) {
    const cuuint64_t dims[3] = {cols, batch, steps};
    const cuuint64_t strides[2] = {seq_rows * ldx_bytes, ldx_bytes};
    const cuuint32_t box[3] = {(cuuint32_t)64, (cuuint32_t)batch, box_t};
    const cuuint32_t estr[3] = {1, 1, 1};
    return g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// [steps][batch][cols] halves, boxes of box_b rows of one step x 64 columns
bool encode_3d(CUtensorMap* map, const void* base, uint64_t cols, uint64_t batch, uint64_t steps, uint64_t row_stride_bytes,
               uint64_t step_stride_bytes, uint32_t box_b) {
    const cuuint64_t dims[3] = {cols, batch, steps};
    const cuuint64_t strides[2] = {row_stride_bytes, step_stride_bytes};
    const cuuint32_t box[3] = {64, box_b, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the device's status block and a fresh launch generation; PIMB200_ERR_UNSUPPORTED without the tensor-map encoder
int tc_prepare(int* dev, int** status, int* gen) {
    PIMB200_CUDA_TRY(cudaGetDevice(dev));
    if (*dev < 0 || *dev >= kMaxDevices) return PIMB200_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!get_encode()) return PIMB200_ERR_UNSUPPORTED;
    if (!g_status[*dev]) {
        PIMB200_CUDA_TRY(cudaMalloc(&g_status[*dev], 2 * sizeof(int)));
        PIMB200_CUDA_TRY(cudaMemset(g_status[*dev], 0, 2 * sizeof(int)));
    }
    *status = g_status[*dev];
    if (++g_gen == 0) g_gen = 1;
    *gen = g_gen;
    return PIMB200_OK;
}
int tc_sm_count(int dev) {
    static int counts[kMaxDevices];      // written with the same value by whoever comes first
    if (!counts[dev]) {
        int n = kNumSmB200;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        counts[dev] = n;
    }
    return counts[dev];
}

}  // namespace tc

static int g_force_simt = 0;

int launch_gemm_wx_skinny(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx,
                          int ldy, int act, int y_is_f32, cudaStream_t st, int fixed);

// Router of the dense contraction: up to 32 activation rows stream W on every SM (HBM-bound, like the GEMV); more rows
// go to the tcgen05 kernel; shapes neither takes (unaligned operands, K not a multiple of 8) to the ragged kernel.  `fixed`: no
// work ahead on the stream writes W, so it may be read before that work has ended.
int launch_gemm_wx(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx,
                   int ldy, int act, int y_is_f32, cudaStream_t st, int fixed) {
    if (!g_force_simt) {
        const int rs = launch_gemm_wx_skinny(W, X, bias, Y, N, K, J, ldx, ldy, act, y_is_f32, st, fixed);
        if (rs != PIMB200_ERR_UNSUPPORTED) return rs;
        const int rc = launch_gemm_rows(W, X, bias, Y, N, K, J, ldx, ldy, act, y_is_f32, 0, 0, st, fixed);
        if (rc != PIMB200_ERR_UNSUPPORTED) return rc;
        return launch_gemm_wx_ragged(W, X, bias, Y, N, K, J, ldx, ldy, act, y_is_f32, st);
    }
    return launch_gemm_wx_simt(W, X, bias, Y, N, K, J, ldx, ldy, act, y_is_f32, st);
}

// Y[t * batch + b, :] = X[b, t, :] . W^T for a batch-first X [batch][seq_rows][K] and the t < J / batch of every sequence:
// the projection of a batch-first sequence tensor written in time-major row order (up to 128 sequences).  Tensor-core path only; PIMB200_ERR_UNSUPPORTED when the shape does
// not allow it (the caller then projects in the input's own row order).
int launch_gemm_wx_time_major(const __half* W, const __half* X, void* Y, int N, int K, int J, int ldx, int ldy, int batch,
                              long seq_rows, cudaStream_t st) {
    if (g_force_simt || batch <= 0) return PIMB200_ERR_UNSUPPORTED;
    return launch_gemm_rows(W, X, nullptr, Y, N, K, J, ldx, ldy, PIMB200_ACT_NONE, 1, batch, seq_rows, st, 1);   // (a handle's weights)
}

}  // namespace pimb200

// A/B switch for profiling: 1 = always the SIMT kernel.
extern "C" int pimb200_gemm_force_simt(int on) {
    pimb200::g_force_simt = on ? 1 : 0;
    return PIMB200_OK;
}

// Status word of the tensor-core GEMM on the current device: 0, or PIMB200_ERR_TIMEOUT when one of its bounded
// waits gave up since the last call.  Synchronises the device.
extern "C" int pimb200_gemm_last_status(void) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return PIMB200_ERR_LAUNCH;
    if (dev < 0 || dev >= pimb200::tc::kMaxDevices) return PIMB200_OK;
    int* p = nullptr;
    {
        std::lock_guard<std::mutex> lk(pimb200::tc::g_mu);
        p = pimb200::tc::g_status[dev];
    }
    if (!p) return PIMB200_OK;
    int v = 0;
    if (cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return PIMB200_ERR_LAUNCH;
    if (v != 0) cudaMemset(p, 0, sizeof(int));
    return v;
}
