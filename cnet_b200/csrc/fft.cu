// Dispatch of FourierTrans between its kernels: the persistent, bulk-copy pipelined one at N = 1024 (fft_pipe.cu) and
// the mixed-radix one at every other length that fits shared memory (fft_mixed.cu).  At 1024 x 4000 rows the first
// takes 14.5 us and the second 24.8; at 256 and 4096 the mixed-radix kernel took over from a fixed four-step one
// (16000 x 256: 23.1 -> 19.6 us, 1000 x 4096: 37.9 -> 26.6 us).
#include "common.cuh"
#include "fft_regs.cuh"

namespace {

using cnb_fft::FftEpilogue;

// tw[k1 * R + t] = e^{-2 pi i t k1 / N}: laid out so that the R threads of a row read one contiguous line
// per frequency k1 (a table indexed by the product t*k1 costs one cache line per thread).
__global__ void fft_twiddle_k(float2* __restrict__ tw, int R) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= R * R) return;
    int k1 = i / R, t = i % R;
    double s, c;
    sincospi(-2.0 * (double) (t * k1) / (double) (R * R), &s, &c);
    tw[i] = make_float2((float) c, (float) s);
}

int make_pipe_table(cnb_ctx* ctx, int, cudaStream_t st, cnb_twiddle* t) {
    constexpr int R = 32;
    void* p = nullptr;
    const int rc = cnb_alloc(ctx, R * R * sizeof(float2), &p);
    if (rc != CNB_OK) return rc;
    t->re = static_cast<float*>(p);
    fft_twiddle_k<<<(R * R + 255) / 256, 256, 0, st>>>(static_cast<float2*>(p), R);
    CNB_LAUNCH_CHECK("fft_twiddle");
    return CNB_OK;
}

bool aligned16(const void* a, const void* b, const void* c, const void* d) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
             reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

}  // namespace

namespace cnb {

bool fft_supported(int N) { return N == 1024 || fft_mixed_supported(N); }

static int fft_dispatch(cnb_ctx* ctx, const float* xr, const float* xi, float* yr, float* yi, int B, int N, int inverse,
                        int accumulate, const FftEpilogue& ep, cudaStream_t st) {
    // the bulk copies of the pipelined kernel need 16-byte aligned planes
    if (N != 1024 || !aligned16(xr, xi, yr, yi)) return fft_mixed(ctx, xr, xi, yr, yi, B, N, inverse, accumulate, ep, st);
    // its inter-pass twiddle table lives in the arena; DFT matrices have positive map keys, fft_mixed's tables -N
    constexpr int key = -(1 << 20);
    cnb_twiddle t;
    const int rc = table(ctx, key, st, make_pipe_table, &t);
    if (rc != CNB_OK) return rc;
    return fft1024_pipe(ctx, xr, xi, yr, yi, reinterpret_cast<const float2*>(t.re), B, inverse, accumulate, ep, st);
}

int fft_run(cnb_ctx* ctx, const float* xr, const float* xi, float* yr, float* yi, int B, int N, int inverse,
            int accumulate, cudaStream_t st) {
    return fft_dispatch(ctx, xr, xi, yr, yi, B, N, inverse, accumulate, FftEpilogue(), st);
}

int fft_hadamard_gelu(cnb_ctx* ctx, const float* xr, const float* xi, const float* hr, const float* hi, float* ur,
                      float* ui, float* ar, float* ai, float* yr, float* yi, float* sp, int B, int N, cudaStream_t st) {
    FftEpilogue ep;
    ep.ar = ar; ep.ai = ai;
    ep.hr = hr; ep.hi = hi; ep.gr = yr; ep.gi = yi; ep.sp = sp;
    ep.np = ((size_t) B * N + 63) & ~size_t(63);
    return fft_dispatch(ctx, xr, xi, ur, ui, B, N, 0, 0, ep, st);
}

}  // namespace cnb
