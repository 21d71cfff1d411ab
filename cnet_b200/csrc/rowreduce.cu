// Row reductions of the complex training step: L2 normalisation (the reference's "SoftMax") forward / backward, the
// fused CrossEntropy forward + backward seed, and L2Out.
//
// All are HBM-bound: a row is read once and kept in registers between its reduction and the element-wise pass.  G
// threads share a row and hold E elements of every plane each, so that a row of any usual length finds a form in which
// most of them work and enough loads are in flight: 8 lanes (rows up to 32, four rows to a warp), a warp (up to 512), a
// CTA of 128 (2048) or 512 threads (8192), a cluster of up to eight such CTAs (65536, partial sums through distributed
// shared memory).  Elements that a row does not have still take registers, and so CTAs from an SM: with 16 a thread for all
// rows beyond 128, forward, loss and backward one behind the other took 34.8 us at 4096 x 1000 (now, with 8, 28.9), 82.4 at
// 2000 x 3000 (53.4), 119 at 65000 x 130 (78.9), 131 at 9000 x 777 (69.8), 109 at 1000 x 6001 (with 12, 82.1); the same
// sums.  16-byte accesses where the row length and the planes allow them, else consecutive threads take
// consecutive elements.  65536 x 20 through a CTA of one warp per row took 69 us a kernel, 300 x 27000 through two
// passes over each row 60 to 82.
#include <algorithm>
#include <initializer_list>

#include "common.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the CTA; result valid in every thread.  blockDim.x is a multiple of 32, <= 1024.
__device__ __forceinline__ float block_sum(float v, float* smem) {
    v = warp_sum(v);
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    float r = (lane < nw) ? smem[lane] : 0.f;
    r = warp_sum(r);
    return r;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Sum over the G threads of a row, or over the whole cluster when it has `parts` CTAs; valid in every thread.
template <int G> __device__ __forceinline__ float row_sum(float v, int parts) {
    if constexpr (G <= 32) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    } else {
        __shared__ float sm[32], part;
        v = block_sum(v, sm);
        if (parts > 1) {
            if (threadIdx.x == 0) part = v;
            cluster_sync();
            const uint32_t local = (uint32_t) __cvta_generic_to_shared(&part);
            v = 0.f;
            for (int c = 0; c < parts; ++c) {                // the same order in every CTA
                uint32_t remote;
                float x;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(c));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(remote) : "memory");
                v += x;
            }
            cluster_sync();                                  // no CTA leaves while a peer still reads its part
        }
        return v;
    }
}

// What a thread holds of a row: element k is at at(k).
template <int G, int E, int VEC> struct Tile {
    size_t base;                    // first element of the row
    int t0, n;                      // this thread's place among the row's, row length
    bool live;
    int row;

    __device__ __forceinline__ Tile(int rows, int n_, int parts) : n(n_) {
        if constexpr (G <= 32) {
            row = (int) (blockIdx.x * (blockDim.x / G) + threadIdx.x / G);       // not of a product that passes 2^32
            t0 = threadIdx.x % G;
        } else {
            row = (int) (blockIdx.x / (unsigned) parts);
            t0 = threadIdx.x + (int) (blockIdx.x % (unsigned) parts) * G;
        }
        live = row < rows;
        base = (size_t) row * n;
        stride = (G <= 32 ? 1 : parts) * G;
    }
    int stride;                     // threads on the row, over all CTAs of its cluster
    __device__ __forceinline__ int at(int k) const { return VEC == 4 ? 4 * (t0 + (k / 4) * stride) + k % 4 : t0 + k * stride; }
    __device__ __forceinline__ void load(const float* p, float (&v)[E]) const {
#pragma unroll
        for (int k = 0; k < E; k += VEC) {
            const bool on = live && at(k) < n;
            if constexpr (VEC == 4) {
                const float4 x = on ? *reinterpret_cast<const float4*>(p + base + at(k)) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[k] = x.x; v[k + 1] = x.y; v[k + 2] = x.z; v[k + 3] = x.w;
            } else {
                v[k] = on ? p[base + at(k)] : 0.f;
            }
        }
    }
    __device__ __forceinline__ void store(float* p, const float (&v)[E]) const {
#pragma unroll
        for (int k = 0; k < E; k += VEC) {
            if (!live || at(k) >= n) continue;
            if constexpr (VEC == 4) *reinterpret_cast<float4*>(p + base + at(k)) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
            else p[base + at(k)] = v[k];
        }
    }
};

// Whether rows that twelve elements a thread would hold take that form and not the one of sixteen: with fewer registers more CTAs
// are resident, which is no gain where few are launched, and twelve scattered loads are slower than sixteen then (us, with 16 and with
// 12: loss of 95 x 4903 3.5 and 4.6, forward of 185 x 5452 3.8 and 4.5, of 417 x 1296 2.8 and 2.9; 164 x 4394 5.7 and 4.4, 567 x 1025 4.0
// and 2.9, 4607 x 1116 9.7 and 9.2; backward, of four planes, 95 x 4903 6.1 and 4.6, 185 x 5452 5.5 and 4.6, but 523 x 1436 3.3 and 3.8; eight
// rows to a CTA 2276 x 378 forward 3.1 and 4.0, backward 2.9 and 3.5).
bool twelve(int g, int vec, int planes, size_t ctas, int sms) {
    if (g == 32) return ctas >= 5 * (size_t) sms;
    if (planes == 4) return g != 128 || vec == 1 || ctas >= 5 * (size_t) sms;
    return ctas >= (vec == 1 ? 1 : 5) * (size_t) sms;
}

constexpr int cta_threads(int g) { return g < 128 ? 256 : g; }

template <int G, int E, int VEC>
__global__ void __launch_bounds__(cta_threads(G))
softmax_fwd_k(const float* __restrict__ zr, const float* __restrict__ zi, float* __restrict__ yr, float* __restrict__ yi,
              float* __restrict__ inv_norm, int rows, int n, int parts) {
    cnb_pdl_enter();
    const Tile<G, E, VEC> t(rows, n, parts);
    float a[E], b[E], s = 0.f;
    t.load(zr, a); t.load(zi, b);
#pragma unroll
    for (int k = 0; k < E; ++k) s += a[k] * a[k] + b[k] * b[k];
    s = row_sum<G>(s, parts);
    const float inv = 1.0f / fmaxf(sqrtf(s), 1e-15f);
    if (t.live && t.t0 == 0) inv_norm[t.row] = inv;
#pragma unroll
    for (int k = 0; k < E; ++k) { a[k] *= inv; b[k] *= inv; }
    t.store(yr, a); t.store(yi, b);
}

template <int G, int E, int VEC>
__global__ void __launch_bounds__(cta_threads(G))
softmax_bwd_k(const float* __restrict__ gr, const float* __restrict__ gi, const float* __restrict__ zr,
              const float* __restrict__ zi, const float* __restrict__ inv_norm, float* __restrict__ dr,
              float* __restrict__ di, int rows, int n, int parts, int accumulate) {
    cnb_pdl_enter();
    const Tile<G, E, VEC> t(rows, n, parts);
    float a[E], b[E], x[E], y[E], s = 0.f;
    t.load(gr, a); t.load(gi, b); t.load(zr, x); t.load(zi, y);
    const float inv = t.live ? inv_norm[t.row] : 0.f;
#pragma unroll
    for (int k = 0; k < E; ++k) s += a[k] * x[k] + b[k] * y[k];          // Re(g* conj(z))
    s = row_sum<G>(s, parts);
    const float c = s * inv * inv * inv;
#pragma unroll
    for (int k = 0; k < E; ++k) { a[k] = a[k] * inv - x[k] * c; b[k] = b[k] * inv - y[k] * c; }
    if (accumulate) {
        t.load(dr, x); t.load(di, y);
#pragma unroll
        for (int k = 0; k < E; ++k) { a[k] += x[k]; b[k] += y[k]; }
    }
    t.store(dr, a); t.store(di, b);
}

template <int G, int E, int VEC>
__global__ void __launch_bounds__(cta_threads(G))
crossent_k(const float* __restrict__ zr, const float* __restrict__ zi, const int32_t* __restrict__ labels,
           float* __restrict__ loss, float* __restrict__ dr, float* __restrict__ di, int rows, int n, int parts) {
    cnb_pdl_enter();
    const Tile<G, E, VEC> t(rows, n, parts);
    const int l = t.live ? min(max(labels[t.row], 0), n - 1) : 0;
    float a[E], b[E], s = 0.f;
    t.load(zr, a); t.load(zi, b);
    // the label's element, asked for again (it is on its way to this SM) rather than passed between threads
    const float lr = t.live ? zr[t.base + l] : 0.f, li = t.live ? zi[t.base + l] : 0.f;
#pragma unroll
    for (int k = 0; k < E; ++k) s += a[k] * a[k] + b[k] * b[k];
    s = row_sum<G>(s, parts);
    const float S = fmaxf(s, 1e-15f), m2 = lr * lr + li * li;
    if (t.live && t.t0 == 0) loss[t.row] = -logf(fmaxf(m2 / S, 1e-15f));
    if (dr == nullptr) return;
    const float m = fmaxf(m2, 1e-15f);
    const float cl = -(S - m) / (m * S), co = 1.0f / S;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const float c = t.at(k) == l ? cl : co;
        a[k] *= c; b[k] *= c;
    }
    t.store(dr, a); t.store(di, b);
}

// L2Out: loss[b] = sum |z|^2; seed dz* = z
template <int G, int E, int VEC>
__global__ void __launch_bounds__(cta_threads(G))
l2out_k(const float* __restrict__ zr, const float* __restrict__ zi, float* __restrict__ loss, float* __restrict__ dr,
        float* __restrict__ di, int rows, int n, int parts) {
    cnb_pdl_enter();
    const Tile<G, E, VEC> t(rows, n, parts);
    float a[E], b[E], s = 0.f;
    t.load(zr, a); t.load(zi, b);
#pragma unroll
    for (int k = 0; k < E; ++k) s += a[k] * a[k] + b[k] * b[k];
    if (dr) { t.store(dr, a); t.store(di, b); }
    s = row_sum<G>(s, parts);
    if (t.live && t.t0 == 0) loss[t.row] = s;
}

// Rows beyond the longest cluster: one CTA reads the row once to reduce and again for the element-wise pass.
__global__ void softmax_fwd_long_k(const float* __restrict__ zr, const float* __restrict__ zi,
                                   float* __restrict__ yr, float* __restrict__ yi, float* __restrict__ inv_norm, int N) {
    cnb_pdl_enter();
    __shared__ float sm[32];
    size_t base = (size_t) blockIdx.x * N;
    float s = 0.f;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        float a = zr[base + i], b = zi[base + i];
        s += a * a + b * b;
    }
    s = block_sum(s, sm);
    float n = fmaxf(sqrtf(s), 1e-15f);
    float inv = 1.0f / n;
    if (threadIdx.x == 0) inv_norm[blockIdx.x] = inv;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        yr[base + i] = zr[base + i] * inv;
        yi[base + i] = zi[base + i] * inv;
    }
}

__global__ void softmax_bwd_long_k(const float* __restrict__ gr, const float* __restrict__ gi,
                                   const float* __restrict__ zr, const float* __restrict__ zi,
                                   const float* __restrict__ inv_norm, float* __restrict__ dr, float* __restrict__ di,
                                   int N, int accumulate) {
    cnb_pdl_enter();
    __shared__ float sm[32];
    size_t base = (size_t) blockIdx.x * N;
    float s = 0.f;
    for (int i = threadIdx.x; i < N; i += blockDim.x)   // Re(g* conj(z))
        s += gr[base + i] * zr[base + i] + gi[base + i] * zi[base + i];
    s = block_sum(s, sm);
    float inv = inv_norm[blockIdx.x];
    float c = s * inv * inv * inv;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        float a = gr[base + i] * inv - zr[base + i] * c;
        float b = gi[base + i] * inv - zi[base + i] * c;
        if (accumulate) { a += dr[base + i]; b += di[base + i]; }
        dr[base + i] = a; di[base + i] = b;
    }
}

__global__ void crossent_long_k(const float* __restrict__ zr, const float* __restrict__ zi,
                                const int32_t* __restrict__ labels, float* __restrict__ loss,
                                float* __restrict__ dr, float* __restrict__ di, int M) {
    cnb_pdl_enter();
    __shared__ float sm[32];
    size_t base = (size_t) blockIdx.x * M;
    float s = 0.f;
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
        float a = zr[base + i], b = zi[base + i];
        s += a * a + b * b;
    }
    s = block_sum(s, sm);
    float S = fmaxf(s, 1e-15f);
    int l = labels[blockIdx.x];
    l = min(max(l, 0), M - 1);
    float lr = zr[base + l], li = zi[base + l];
    float m2 = lr * lr + li * li;
    if (threadIdx.x == 0) loss[blockIdx.x] = -logf(fmaxf(m2 / S, 1e-15f));
    if (dr == nullptr) return;
    float m = fmaxf(m2, 1e-15f);
    float cl = -(S - m) / (m * S), co = 1.0f / S;
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
        float c = (i == l) ? cl : co;
        dr[base + i] = zr[base + i] * c;
        di[base + i] = zi[base + i] * c;
    }
}

__global__ void l2out_long_k(const float* __restrict__ zr, const float* __restrict__ zi, float* __restrict__ loss,
                             float* __restrict__ dr, float* __restrict__ di, int N) {
    cnb_pdl_enter();
    __shared__ float sm[32];
    size_t base = (size_t) blockIdx.x * N;
    float s = 0.f;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        float a = zr[base + i], b = zi[base + i];
        s += a * a + b * b;
        if (dr) { dr[base + i] = a; di[base + i] = b; }
    }
    s = block_sum(s, sm);
    if (threadIdx.x == 0) loss[blockIdx.x] = s;
}

bool vec_ok(int n, std::initializer_list<const void*> planes) {
    if (n % 4) return false;
    for (const void* p : planes) if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

}  // namespace

// The form for rows of n elements (the lines are where a thread's 4, 8, 12 or 16 elements are used up) and its launch; NAME is
// the kernel, the argument list ends with rows, n, parts and what may follow them.
#define CNB_ROWS_GO(NAME, G, E, V, CTAS, PARTS, ...)                                                                     \
    cnb::launch(NAME<G, E, V>, dim3((unsigned) (CTAS)), dim3(cta_threads(G)), 0, st, PARTS, __VA_ARGS__)
#define CNB_ROWS_V(NAME, PLANES, V, rows, n, ...)                                                                                \
    do {                                                                                                                 \
        if ((n) <= 32) CNB_ROWS_GO(NAME, 8, 4, V, ((size_t) (rows) + 31) / 32, 1, __VA_ARGS__);                          \
        else if ((n) <= 128) CNB_ROWS_GO(NAME, 32, 4, V, ((size_t) (rows) + 7) / 8, 1, __VA_ARGS__);                     \
        else if ((n) <= 256) CNB_ROWS_GO(NAME, 32, 8, V, ((size_t) (rows) + 7) / 8, 1, __VA_ARGS__);                     \
        else if ((n) <= 384 && twelve(32, V, PLANES, ((size_t) (rows) + 7) / 8, ctx->sm_count))                          \
            CNB_ROWS_GO(NAME, 32, 12, V, ((size_t) (rows) + 7) / 8, 1, __VA_ARGS__);                                     \
        else if ((n) <= 512) CNB_ROWS_GO(NAME, 32, 16, V, ((size_t) (rows) + 7) / 8, 1, __VA_ARGS__);                    \
        else if ((n) <= 1024) CNB_ROWS_GO(NAME, 128, 8, V, rows, 1, __VA_ARGS__);                                        \
        else if ((n) <= 1536 && twelve(128, V, PLANES, rows, ctx->sm_count)) CNB_ROWS_GO(NAME, 128, 12, V, rows, 1, __VA_ARGS__); \
        else if ((n) <= 2048) CNB_ROWS_GO(NAME, 128, 16, V, rows, 1, __VA_ARGS__);                                       \
        else if ((n) <= 4096) CNB_ROWS_GO(NAME, 512, 8, V, rows, 1, __VA_ARGS__);                                        \
        else if ((n) <= 6144 && twelve(512, V, PLANES, rows, ctx->sm_count)) CNB_ROWS_GO(NAME, 512, 12, V, rows, 1, __VA_ARGS__); \
        else CNB_ROWS_GO(NAME, 512, 16, V, (size_t) (rows) * parts, parts, __VA_ARGS__);                                 \
    } while (0)
#define CNB_ROWS(NAME, PLANES, vec, rows, n, ...)                                                                                \
    do {                                                                                                                 \
        if (vec) CNB_ROWS_V(NAME, PLANES, 4, rows, n, __VA_ARGS__);                                                              \
        else CNB_ROWS_V(NAME, PLANES, 1, rows, n, __VA_ARGS__);                                                                  \
        CNB_LAUNCH_CHECK(#NAME);                                                                                         \
    } while (0)

namespace {
constexpr int kLongest = 65536;
int parts_for(int n) { return n <= 8192 ? 1 : n <= 16384 ? 2 : n <= 32768 ? 4 : 8; }
}  // namespace

extern "C" {

int cnb_softmax_fwd(cnb_ctx* ctx, const float* z_re, const float* z_im, float* y_re, float* y_im,
                    float* inv_norm, int B, int N, void* stream) {
    CNB_CHECK_ARG(ctx && z_re && z_im && y_re && y_im && inv_norm, "cnb_softmax_fwd: null pointer");
    CNB_CHECK_ARG(B > 0 && N > 0, "cnb_softmax_fwd: B=%d N=%d", B, N);
    cudaStream_t st = cnb::S(stream);
    const int parts = parts_for(N);
    if (N > kLongest) {
        cnb::launch(softmax_fwd_long_k, dim3(B), dim3(512), 0, st, 1, z_re, z_im, y_re, y_im, inv_norm, N);
        CNB_LAUNCH_CHECK("softmax_fwd");
    } else {
        CNB_ROWS(softmax_fwd_k, 2, vec_ok(N, {z_re, z_im, y_re, y_im}), B, N, z_re, z_im, y_re, y_im, inv_norm, B, N, parts);
    }
    return CNB_OK;
}

int cnb_softmax_bwd(cnb_ctx* ctx, const float* g_re, const float* g_im, const float* z_re, const float* z_im,
                    const float* inv_norm, float* dz_re, float* dz_im, int B, int N, int accumulate,
                    void* stream) {
    CNB_CHECK_ARG(ctx && g_re && g_im && z_re && z_im && inv_norm && dz_re && dz_im,
                  "cnb_softmax_bwd: null pointer");
    CNB_CHECK_ARG(B > 0 && N > 0, "cnb_softmax_bwd: B=%d N=%d", B, N);
    cudaStream_t st = cnb::S(stream);
    const int parts = parts_for(N);
    if (N > kLongest) {
        cnb::launch(softmax_bwd_long_k, dim3(B), dim3(512), 0, st, 1, g_re, g_im, z_re, z_im, inv_norm, dz_re, dz_im, N, accumulate);
        CNB_LAUNCH_CHECK("softmax_bwd");
    } else {
        CNB_ROWS(softmax_bwd_k, 4, vec_ok(N, {g_re, g_im, z_re, z_im, dz_re, dz_im}), B, N, g_re, g_im, z_re, z_im, inv_norm, dz_re,
                 dz_im, B, N, parts, accumulate);
    }
    return CNB_OK;
}

int cnb_crossent_fwd_bwd(cnb_ctx* ctx, const float* z_re, const float* z_im, const int32_t* labels, float* loss,
                         float* dz_re, float* dz_im, int B, int M, void* stream) {
    CNB_CHECK_ARG(ctx && z_re && z_im && labels && loss, "cnb_crossent_fwd_bwd: null pointer");
    CNB_CHECK_ARG((dz_re == nullptr) == (dz_im == nullptr), "cnb_crossent_fwd_bwd: dz planes must be a pair");
    CNB_CHECK_ARG(B > 0 && M > 0, "cnb_crossent_fwd_bwd: B=%d M=%d", B, M);
    cudaStream_t st = cnb::S(stream);
    const int parts = parts_for(M);
    if (M > kLongest) {
        cnb::launch(crossent_long_k, dim3(B), dim3(512), 0, st, 1, z_re, z_im, labels, loss, dz_re, dz_im, M);
        CNB_LAUNCH_CHECK("crossent");
    } else {
        CNB_ROWS(crossent_k, 2, vec_ok(M, {z_re, z_im, dz_re, dz_im}), B, M, z_re, z_im, labels, loss, dz_re, dz_im, B, M, parts);
    }
    return CNB_OK;
}

int cnb_l2out_fwd_bwd(cnb_ctx* ctx, const float* z_re, const float* z_im, float* loss, float* dz_re, float* dz_im,
                      int B, int N, void* stream) {
    CNB_CHECK_ARG(ctx && z_re && z_im && loss, "cnb_l2out_fwd_bwd: null pointer");
    CNB_CHECK_ARG((dz_re == nullptr) == (dz_im == nullptr), "cnb_l2out_fwd_bwd: dz planes must be a pair");
    CNB_CHECK_ARG(B > 0 && N > 0, "cnb_l2out_fwd_bwd: B=%d N=%d", B, N);
    cudaStream_t st = cnb::S(stream);
    const int parts = parts_for(N);
    if (N > kLongest) {
        cnb::launch(l2out_long_k, dim3(B), dim3(512), 0, st, 1, z_re, z_im, loss, dz_re, dz_im, N);
        CNB_LAUNCH_CHECK("l2out");
    } else {
        CNB_ROWS(l2out_k, 2, vec_ok(N, {z_re, z_im, dz_re, dz_im}), B, N, z_re, z_im, loss, dz_re, dz_im, B, N, parts);
    }
    return CNB_OK;
}

}  // extern "C"
