// Shared declarations of the device library: context, error plumbing, launch helpers.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <algorithm>
#include <map>
#include <string>

#include "../../include/cnet_b200.h"

struct cnb_twiddle {
    float* re = nullptr;   // [N, N] planes, F[p,q] = N^-1/2 e^{-2 pi i pq/N}
    float* im = nullptr;
    void* pack = nullptr;  // the matrix packed (made once; head, then planes), or null when the tiles cannot take it
    cudaEvent_t built = nullptr;           // recorded behind the kernels that make the table; null once they are known to be done
    unsigned long long stream_id = 0;      // the stream they run on
};

// Head of a packed operand: the scale's exponent; on their way to becoming that, the largest component and the
// complement of the least group maximum (as bits of magnitudes); how many blocks of the packing launch have read them.
struct cnb_pack_head { int exponent; unsigned max_bits, ticket, low_bits; };

struct cnb_ctx {
    int device = 0;
    int sm_count = 148;
    char* base = nullptr;
    size_t size = 0;
    size_t used = 0;
    bool owns = false;
    int* d_status = nullptr;          // device error word (bounded waits report here)
    int* d_counters = nullptr;        // 8 sets of 64 "CTAs done" counters, zero between launches
    unsigned counter_set = 0;
    // Column-reduction partials and packed operands of raw products: the last bytes of the arena, so that growing it
    // takes in what it had.
    size_t scratch_bytes = 0;
    size_t scratch_kept = 0;          // of them, what no allocation may take back
    std::map<int, cnb_twiddle> twiddles;
    int gemm_cta_limit = 0;           // > 0: the tensor-core GEMM uses at most this many CTAs (SMs)
    bool force_dft_gemm = false;      // FourierTrans as a GEMM even where the FFT kernel applies
};

namespace cnb {

int set_error(int code, const char* fmt, ...);
void count_launch();
// keep: the caller has no way of doing without.  What packed operands alone asked for is given back to an allocation that
// finds no other room; their products have the SIMT tiles.
int ensure_scratch(cnb_ctx* ctx, size_t bytes, bool keep, cudaStream_t st, float** out);
extern thread_local int g_last_engine;

// A table of constants from the context's cache, made by `make(stream, &table)` (arena memory and launches) at its first
// use.  On return work on `st` may read it: its kernels ran on `st` before, or have completed.  While `st` is being
// captured the table is made on a stream of its own, since what is captured does not run until the graph does.
typedef int (*TableMake)(cnb_ctx* ctx, int key, cudaStream_t st, cnb_twiddle* t);
int table(cnb_ctx* ctx, int key, cudaStream_t st, TableMake make, cnb_twiddle* out);
void drop_tables(cnb_ctx* ctx);

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// SMs a kernel sized as "one wave" should count on: all of them, or fewer while some are set aside for a
// collective's kernels (cnb_set_gemm_sm_limit); sized for the whole device such a kernel would run a second,
// nearly empty wave.
inline int usable_sms(const cnb_ctx* ctx) {
    return ctx->gemm_cta_limit > 0 && ctx->gemm_cta_limit < ctx->sm_count ? ctx->gemm_cta_limit : ctx->sm_count;
}

// fp32 SIMT complex GEMM on generic strides:
//   D[m,n] (+)= sum_k A(m,k) * (conjB ? conj(B(n,k)) : B(n,k)) (+ R[m,n])
//   A(m,k) = a[m*sam + k*sak], B(n,k) = b[n*sbn + k*sbk], D/R row-major with ld = N.
int cgemm_simt(cnb_ctx* ctx, const float* a_re, const float* a_im, long sam, long sak,
               const float* b_re, const float* b_im, long sbn, long sbk, int conjB,
               const float* r_re, const float* r_im, float* d_re, float* d_im,
               int M, int N, int K, int accumulate, cudaStream_t st);

// tcgen05 complex GEMM on split operands:
//   D[m,n] (+)= sum_k A[m,k] * (conjB ? conj(B[n,k]) : B[n,k]) (+ R[m,n]); A [M,K], B [N,K].
// The sizes that its tiles are made for, and those of them for which it beats the SIMT tiles with the operands still to be packed:
bool cgemm_tc_fits(int M, int N, int K);
bool cgemm_tc_shape_ok(int M, int N, int K);
// Products left to the SIMT tiles by that line whose chains in tensor memory would be shorter than K: summed one by one they
// would be less exact.
bool cgemm_fma_in_chains(int M, int N, int K);
// A packed operand: fp16 high and low parts of a matrix scaled by one power of two (cgemm_tc.cu), the form that
// everything but the C ABI's split buffers goes through.
struct PackRequest {
    const float* re; const float* im;  // [rows, cols]
    int rows, cols, pitch;             // pitch of the packed rows: a multiple of 8, of 64 where they are read MN-major
    void* planes;                      // 8 * rows * pitch bytes, 128-byte aligned
    cnb_pack_head* head;               // zeroed before the first use
};
int pack(cnb_ctx* ctx, const PackRequest* r, int n, cudaStream_t st);
// fp32 operands, packed into scratch first: a_trans / b_trans = the source planes are stored [K, rows]; b_packed: a
// constant B that its owner has packed.
int cgemm_tc_run(cnb_ctx* ctx, const float* a_re, const float* a_im, int a_trans, const float* b_re,
                 const float* b_im, int b_trans, int conjB, const float* r_re, const float* r_im, float* d_re,
                 float* d_im, int M, int N, int K, int accumulate, cudaStream_t st,
                 const PackRequest* b_packed = nullptr);
size_t cgemm_tc_workspace_bytes(int M, int N, int K);
// An operand that is already split (see cnb_split_component below): slots plane_pitch floats apart, stored rows
// [rows, K] (mn = 0) or [K, rows] (mn = 1) at `pitch` elements.
struct SplitOperand {
    const float* base;
    size_t plane_pitch;
    int pitch, mn;
    const int* exponent;               // not NULL: a packed operand (fp16 high and low parts, cgemm_tc.cu), base its first plane
};
int cgemm_tc_presplit(cnb_ctx* ctx, const SplitOperand& a, const SplitOperand& b, int conjB,
                      const float* r_re, const float* r_im, float* d_re, float* d_im, int M, int N, int K,
                      int accumulate, cudaStream_t st);
SplitOperand packed_operand(const PackRequest& r, int mn);
// split = 4 consecutive slots of pad64(n) floats (see cnb_split_component below)
int split_planes(cnb_ctx* ctx, const float* re, const float* im, size_t n, float* split, cudaStream_t st);

// Skinny Linear (out <= 16): HBM-bound fp32 kernels.
bool skinny_ok(int B, int in, int out);
size_t skinny_workspace_bytes(int B, int in, int out, int sm_count);
int skinny_fwd(cnb_ctx* ctx, const float* xr, const float* xi, const float* wr, const float* wi, float* yr, float* yi,
               int B, int in, int out, cudaStream_t st);
int skinny_bwd_x(cnb_ctx* ctx, const float* gr, const float* gi, const float* wr, const float* wi, float* dr,
                 float* di, int B, int in, int out, int accumulate, cudaStream_t st);
int skinny_bwd_w(cnb_ctx* ctx, const float* gr, const float* gi, const float* xr, const float* xi, float* dr,
                 float* di, int B, int in, int out, int accumulate, cudaStream_t st);

// Shared-memory FFT (fft_pipe.cu at N = 1024, fft_mixed.cu elsewhere); inverse = conjugate direction.
bool fft_supported(int N);
int fft_run(cnb_ctx* ctx, const float* xr, const float* xi, float* yr, float* yi, int B, int N, int inverse,
            int accumulate, cudaStream_t st);
// Forward FFT whose epilogue also applies Hadamard(h) -> CGelu: u = FFT(x) -> (ur, ui); y = gelu(u o h) ->
// (yr, yi) and, when sp != NULL, the operand split of y; u o h -> (ar, ai) where these are given (not at N = 1024).
int fft_hadamard_gelu(cnb_ctx* ctx, const float* xr, const float* xi, const float* hr, const float* hi, float* ur,
                      float* ui, float* ar, float* ai, float* yr, float* yi, float* sp, int B, int N, cudaStream_t st);

}  // namespace cnb

// CGelu of the reference (impl/relu.h:119-131): tanh form; the derivative uses sech^2 = 1 - tanh^2.
// tanh(y) = 1 - 2 / (e^{2y} + 1) on the special-function unit: absolute error below 1e-7 (the
// approximate exp2 is good to 2^-22; both tails saturate to +-1 exactly), a third of tanhf's instructions.
__device__ __forceinline__ float cnb_tanh(float y) {
    return 1.0f - __fdividef(2.0f, __expf(2.0f * y) + 1.0f);
}

__device__ __forceinline__ float cnb_gelu(float x) {
    float t = cnb_tanh(0.7978845608028654f * (x + 0.044715f * x * x * x));
    return 0.5f * x * (1.0f + t);
}

__device__ __forceinline__ float cnb_dgelu(float x) {
    float x2 = x * x;
    float t = cnb_tanh(0.7978845608028654f * (x + 0.044715f * x * x2));
    float sech2 = 1.0f - t * t;
    return 0.5f * (1.0f + t) + 0.5f * x * sech2 * 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x2);
}

// The operand split of the tensor-core product.  x = hi + lo with hi = x cut to TF32 (low 13 mantissa bits
// cleared) and lo = x - hi, exact in fp32.  A product x.y is taken as hi.hi on the TF32 pipe plus the two cross
// terms hi.lo + lo.hi on the BF16 pipe, for which hi and lo are also kept rounded to bf16 (h16, l16).  A split
// buffer of n elements is four slots of np = pad64(n) floats:
//   slot 0: hi of the real plane (fp32)      slot 2: h16 of the real plane, then of the imaginary plane (bf16)
//   slot 1: hi of the imaginary plane        slot 3: l16 of the real plane, then of the imaginary plane
__device__ __forceinline__ float cnb_tf32_hi(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); }
__device__ __forceinline__ unsigned short cnb_bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

struct cnb_split_dst {
    float* hi;               // fp32 hi plane of this component (real or imaginary)
    unsigned short* h16;     // its bf16 planes
    unsigned short* l16;
};

// component c (0 = real, 1 = imaginary) of a split buffer with plane pitch np
__host__ __device__ __forceinline__ cnb_split_dst cnb_split_component(float* sp, size_t np, int c) {
    cnb_split_dst d;
    d.hi = sp + (size_t) c * np;
    d.h16 = reinterpret_cast<unsigned short*>(sp + 2 * np) + (size_t) c * np;
    d.l16 = reinterpret_cast<unsigned short*>(sp + 3 * np) + (size_t) c * np;
    return d;
}

__device__ __forceinline__ void cnb_split_store1(const cnb_split_dst& d, size_t i, float x) {
    const float h = cnb_tf32_hi(x);
    d.hi[i] = h;
    d.h16[i] = cnb_bf16_bits(h);
    d.l16[i] = cnb_bf16_bits(x - h);
}

// four consecutive elements, i % 4 == 0 (16-byte store of hi, 8-byte stores of the bf16 planes)
__device__ __forceinline__ void cnb_split_store4(const cnb_split_dst& d, size_t i, float x0, float x1, float x2, float x3) {
    const float h0 = cnb_tf32_hi(x0), h1 = cnb_tf32_hi(x1), h2 = cnb_tf32_hi(x2), h3 = cnb_tf32_hi(x3);
    *reinterpret_cast<float4*>(d.hi + i) = make_float4(h0, h1, h2, h3);
    uint2 a, b;
    a.x = (uint32_t) cnb_bf16_bits(h0) | ((uint32_t) cnb_bf16_bits(h1) << 16);
    a.y = (uint32_t) cnb_bf16_bits(h2) | ((uint32_t) cnb_bf16_bits(h3) << 16);
    b.x = (uint32_t) cnb_bf16_bits(x0 - h0) | ((uint32_t) cnb_bf16_bits(x1 - h1) << 16);
    b.y = (uint32_t) cnb_bf16_bits(x2 - h2) | ((uint32_t) cnb_bf16_bits(x3 - h3) << 16);
    *reinterpret_cast<uint2*>(d.h16 + i) = a;
    *reinterpret_cast<uint2*>(d.l16 + i) = b;
}

// The magnitude of a component as an ordered integer for the scale of a packed operand.  Infinities and NaN count as
// zero: they stay what they are under any scale, and must not take the finite rows beside them out of range.
__device__ __forceinline__ unsigned cnb_scale_bits(float x) {
    const unsigned b = __float_as_uint(x) & 0x7fffffffu;
    return b < 0x7f800000u ? b : 0u;
}

// Programmatic dependent launch.  Every kernel of the step is launched with the "programmatic stream
// serialization" attribute (cnb::launch below): it may be scheduled as soon as every CTA of the kernel before
// it in the stream has called cnb_pdl_trigger() (or exited), so its launch latency and its set-up (barriers,
// tensor memory, tables that no kernel writes) run under the predecessor's tail.  cnb_pdl_wait() returns when
// the predecessor grid has completed and its memory is visible: nothing a predecessor writes or reads may be
// touched before it.  Both are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void cnb_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cnb_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void cnb_pdl_enter() { cnb_pdl_trigger(); cnb_pdl_wait(); }

// A value that kernels before this one may have written, read among this kernel's own stores: not through __ldg, which is not
// held behind cnb_pdl_wait, and without the order that a plain load has against the stores before it.
__device__ __forceinline__ float cnb_ld_behind_wait(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Whether `mine` holds for any of the `threads` threads (whole warps) that meet at the CTA's barrier `barrier`: the same
// answer for all of them.
__device__ __forceinline__ bool cnb_group_any(int barrier, int threads, bool mine) {
    unsigned any;
    asm volatile(
        "{\n\t.reg .pred m, a;\n\t"
        "setp.ne.u32 m, %1, 0;\n\t"
        "barrier.cta.red.or.pred a, %2, %3, m;\n\t"
        "selp.u32 %0, 1, 0, a;\n\t}"
        : "=r"(any) : "r"((unsigned) mine), "r"(barrier), "r"(threads) : "memory");
    return any != 0;
}

namespace cnb {

bool pdl_enabled();                // CNB_PDL=0 in the environment launches every kernel fully serialised

// Launch of a kernel that starts with cnb_pdl_enter() (or does its own trigger / wait); cluster > 1 adds a
// thread-block cluster of that many CTAs along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_ex(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster,
                             bool dependent, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (dependent && pdl_enabled()) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned) cluster;
        at[n].val.clusterDim.y = 1;
        at[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster,
                          Args... args) {
    return launch_ex(kernel, grid, block, smem, st, cluster, true, args...);
}

}  // namespace cnb

#define CNB_CHECK_ARG(cond, ...) \
    do { if (!(cond)) return cnb::set_error(CNB_ERR_ARG, __VA_ARGS__); } while (0)

#define CNB_CUDA(call) \
    do { cudaError_t e_ = (call); \
         if (e_ != cudaSuccess) return cnb::set_error(CNB_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); } while (0)

#define CNB_LAUNCH_CHECK(name) \
    do { cnb::count_launch(); cudaError_t e_ = cudaGetLastError(); \
         if (e_ != cudaSuccess) return cnb::set_error(CNB_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e_)); } while (0)
