// fp32 SIMT complex GEMM on generic strides: the products that are too small or too narrow for the tensor-core tiles,
// and all of them where the arena has no room for packed operands; every operand orientation of the Linear backward
// without staging copies.
#include "cgemm_fma.cuh"

namespace {

struct Strided {
    const float* re; const float* im;
    long row, k;
    bool k_fast;
    __device__ __forceinline__ float2 operator()(int r, int kk) const {
        const size_t o = (size_t) r * row + (size_t) kk * k;
        return make_float2(re[o], im[o]);            // not __ldg: that may move ahead of the wait for the kernel before
    }
};

__global__ void __launch_bounds__(256) cgemm_simt_k(const Strided a, const Strided b, const cnb_fma::Result p) {
    cnb_pdl_enter();
    __shared__ __align__(16) cnb_fma::Slabs s;
    cnb_fma::tile(a, b, p, s, blockIdx.y * cnb_fma::TM, blockIdx.x * cnb_fma::TN, threadIdx.x, [] { __syncthreads(); });
}

}  // namespace

namespace cnb {

int cgemm_simt(cnb_ctx* ctx, const float* a_re, const float* a_im, long sam, long sak, const float* b_re,
               const float* b_im, long sbn, long sbk, int conjB, const float* r_re, const float* r_im,
               float* d_re, float* d_im, int M, int N, int K, int accumulate, cudaStream_t st) {
    (void) ctx;
    const dim3 grid((N + cnb_fma::TN - 1) / cnb_fma::TN, (M + cnb_fma::TM - 1) / cnb_fma::TM);
    const Strided a = {a_re, a_im, sam, sak, sak == 1}, b = {b_re, b_im, sbn, sbk, sbk == 1};
    const cnb_fma::Result p = {d_re, d_im, r_re, r_im, M, N, K, conjB, accumulate};
    cnb::launch(cgemm_simt_k, grid, dim3(256), 0, st, 1, a, b, p);
    CNB_LAUNCH_CHECK("cgemm_simt");
    return CNB_OK;
}

}  // namespace cnb
