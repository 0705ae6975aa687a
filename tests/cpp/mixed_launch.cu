// One launch of the one-tile linear kernel with a projection that has per-head RMSNorm and one that has none, for
// tests/test_mixed_launch_gpu.py: no C entry point builds such a launch.
#include "../../brodiffusion_b200/csrc/gemm_tc05.cu"

using namespace bdattn;

namespace {
// (cols, rows) BF16 matrix, box = 64 columns x box_rows rows, 128-byte swizzle
bool map_2d(CUtensorMap* m, const void* base, int cols, int rows, int box_rows) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || fn == nullptr) return false;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)}, strides[1] = {dims[0] * 2};
    cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)}, step[2] = {1, 1};
    return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn)(
               m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// y0 = RMSNorm per head of 64 columns (x . w0^T) * gain, y1 = x . w1^T + bias; M rows, K columns of x, n0 and n1 outputs
extern "C" int mixed_launch(const void* x, int M, int K, const void* w0, int n0, const float* gain, float eps, void* y0,
                            const void* w1, int n1, const void* bias, void* y1) {
    GemmLaunch L = {};
    L.bf16 = true;
    L.n_problems = 2;
    L.args.split = 1;
    const void* w[2] = {w0, w1};
    void* y[2] = {y0, y1};
    const int n[2] = {n0, n1};
    for (int i = 0; i < 2; ++i) {
        GemmProblem& p = L.args.p[i];
        p.M = M; p.N = n[i]; p.K = K; p.C = y[i]; p.ldc = n[i];
        p.n_tile = 64;
        p.tiles_m = gemm_row_tiles(M);
        p.tiles_n = (n[i] + 63) / 64;
        if (!map_2d(&L.tmA[i], x, K, M, 128) || !map_2d(&L.tmB[i], w[i], K, n[i], 64)) return -1;
    }
    L.args.p[0].norm_rope = 1; L.args.p[0].gain = gain; L.args.p[0].gain_is_f32 = 1; L.args.p[0].eps = eps;
    L.args.p[1].bias = bias;
    L.tmA[2] = L.tmA[0]; L.tmB[2] = L.tmB[0];
    if (launch_gemm_tc05(L, nullptr) != cudaSuccess) return -1;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : -1;
}
