// fp32 SIMT complex GEMM on generic strides: the products that are too small, too narrow or too short for the tensor-core
// tiles, and all of them where the arena has no room for packed operands; every operand orientation of the Linear backward
// without staging copies.
//
// Tiles of T x T outputs (16, 32 or 64), one, four or sixteen of them a thread, k-slabs in two shared-memory buffers, the next
// one on its way while one is worked on.  What bounds them is the chain of a CTA's slabs, each a round trip to L2, and few CTAs:
// with tiles of 64 x 64 and slabs of 16, fetched and then worked on, 64 x 64 -> 32 took 12 us and 128 x 128, K = 128 23 us
// (now 2.8 and 5.2), 2000 x 50 -> 50 13 (6.0), 500 x 900, K = 26 9.1 (6.8), 2000 x 2000, K = 18 54 (32).  The terms of an
// output are added one by one in the order of k whatever the tile, but for the products that cgemm_fma_in_chains names.
#include "common.cuh"

namespace {

// What the kernels before this one may still be writing is read by ordinary loads behind cnb_pdl_enter.
// CHAINS: the terms of an output are added up in sixteens, and the sums of these in turn.
template <int T, int SLAB, bool CHAINS>
__global__ void __launch_bounds__(256)
cgemm_simt_k(const float* a_re, const float* a_im, long sam, long sak, const float* b_re, const float* b_im, long sbn, long sbk,
             int conjB, const float* r_re, const float* r_im, float* d_re, float* d_im, int M, int N, int K, int accumulate) {
    cnb_pdl_enter();
    constexpr int U = T / 16, LOADS = T * SLAB / 256, CHAIN = 16;
    static_assert(SLAB % CHAIN == 0, "a slab is whole chains");
    __shared__ float2 As[2][SLAB][T + 1], Bs[2][SLAB][T + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int tiles_n = (N + T - 1) / T, m0 = (int) (blockIdx.x / (unsigned) tiles_n) * T, n0 = (int) (blockIdx.x % (unsigned) tiles_n) * T;
    // loader mapping: the index that is contiguous in memory is the fast one
    const bool a_kfast = sak == 1, b_kfast = sbk == 1;
    float2 na[LOADS], nb[LOADS];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int e = tid + j * 256;
            const int gm = m0 + (a_kfast ? e / SLAB : e % T), ka = k0 + (a_kfast ? e % SLAB : e / T);
            const int gn = n0 + (b_kfast ? e / SLAB : e % T), kb = k0 + (b_kfast ? e % SLAB : e / T);
            na[j] = nb[j] = make_float2(0.f, 0.f);
            if (gm < M && ka < K) { const size_t o = (size_t) gm * sam + (size_t) ka * sak; na[j] = make_float2(a_re[o], a_im[o]); }
            if (gn < N && kb < K) { const size_t o = (size_t) gn * sbn + (size_t) kb * sbk; nb[j] = make_float2(b_re[o], b_im[o]); }
        }
    };
    float cr[U][U] = {}, ci[U][U] = {}, sr[U][U] = {}, si[U][U] = {};
    auto end_chain = [&] {
#pragma unroll
        for (int i = 0; i < U; ++i)
#pragma unroll
            for (int j = 0; j < U; ++j) { sr[i][j] += cr[i][j]; si[i][j] += ci[i][j]; cr[i][j] = ci[i][j] = 0.f; }
    };
    fetch(0);
    for (int k0 = 0, s = 0; k0 < K; k0 += SLAB, s ^= 1) {
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int e = tid + j * 256;
            As[s][a_kfast ? e % SLAB : e / T][a_kfast ? e / SLAB : e % T] = na[j];
            Bs[s][b_kfast ? e % SLAB : e / T][b_kfast ? e / SLAB : e % T] = make_float2(nb[j].x, conjB ? -nb[j].y : nb[j].y);
        }
        __syncthreads();                                 // the other buffer was last read before the barrier of the slab before
        if (k0 + SLAB < K) fetch(k0 + SLAB);
        const float2* as = &As[s][0][ty];
        const float2* bs = &Bs[s][0][tx];
        auto step = [&](int kk) {
            float2 a[U], b[U];
#pragma unroll
            for (int i = 0; i < U; ++i) { a[i] = as[kk * (T + 1) + 16 * i]; b[i] = bs[kk * (T + 1) + 16 * i]; }
#pragma unroll
            for (int i = 0; i < U; ++i)
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    cr[i][j] += a[i].x * b[j].x - a[i].y * b[j].y;
                    ci[i][j] += a[i].x * b[j].y + a[i].y * b[j].x;
                }
        };
        if (K - k0 >= SLAB) {
#pragma unroll
            for (int kk = 0; kk < SLAB; ++kk) {
                step(kk);
                if (CHAINS && kk % CHAIN == CHAIN - 1) end_chain();
            }
        } else {
#pragma unroll 4
            for (int kk = 0; kk < K - k0; ++kk) {
                step(kk);
                if (CHAINS && (kk % CHAIN == CHAIN - 1 || kk + 1 == K - k0)) end_chain();
            }
        }
    }
#pragma unroll
    for (int i = 0; i < U; ++i)
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int gm = m0 + ty + 16 * i, gn = n0 + tx + 16 * j;
            if (gm >= M || gn >= N) continue;
            const size_t o = (size_t) gm * N + gn;
            float vr = CHAINS ? sr[i][j] : cr[i][j], vi = CHAINS ? si[i][j] : ci[i][j];
            if (r_re) { vr += r_re[o]; vi += r_im[o]; }
            if (accumulate) { vr += d_re[o]; vi += d_im[o]; }
            d_re[o] = vr; d_im[o] = vi;
        }
}

// The same for few outputs: tiles of 8 x 8, an output a thread, two warps, and five slabs on their way (asynchronous copies of 4 bytes,
// which take any alignment) while one is worked on, which makes up for the round trip to L2.  The terms are rounded and added as
// above.  What bounds it is issue, two fifths of it the copies': 10 ns a k where both operands lie along k, 15 where neither does,
// beside 29 in tiles of 16 (64 x 26, K = 784 23.4 -> 9.6 us; 53 x 27, K = 993 30.0 -> 13.7; 64 x 32, K = 64 2.9 -> 1.9).  With the copies left to
// two warps of their own, or through registers and ordinary loads, two slabs ahead: 10.4 and 11.2 us, 17.6 and 17.7.
constexpr int SLIM = 8, SLIM_SLAB = 32, STAGES = 6, SLIM_THREADS = SLIM * SLIM;

__device__ __forceinline__ void copy4(float* dst, const float* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                 ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 4 : 0) : "memory");
}

// One plane of an operand's slab, rows of k (KFAST: k is contiguous in memory; four of them are read at a time) or lines of rows.
template <bool KFAST> struct SlimPlane {
    static constexpr int PITCH = KFAST ? SLIM_SLAB + 4 : SLIM;
    float v[KFAST ? SLIM * PITCH : SLIM_SLAB * PITCH];
    __device__ __forceinline__ float* at(int row, int k) { return v + (KFAST ? row * PITCH + k : k * PITCH + row); }
    __device__ __forceinline__ void four(int row, int k, float (&x)[4]) {
        if constexpr (KFAST) {
            const float4 f = *reinterpret_cast<const float4*>(at(row, k));
            x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = *at(row, k + i);
        }
    }
};

template <bool AK, bool BK, bool CHAINS>
__global__ void __launch_bounds__(SLIM_THREADS)
cgemm_slim_k(const float* a_re, const float* a_im, long sam, long sak, const float* b_re, const float* b_im, long sbn, long sbk,
             int conjB, const float* r_re, const float* r_im, float* d_re, float* d_im, int M, int N, int K, int accumulate) {
    cnb_pdl_enter();
    struct Slab { SlimPlane<AK> ar, ai; SlimPlane<BK> br, bi; };
    __shared__ __align__(16) Slab slabs[STAGES];
    constexpr int CHAIN = 16;
    const int tid = threadIdx.x, tx = tid % SLIM, ty = tid / SLIM;
    const int tiles_n = (N + SLIM - 1) / SLIM, m0 = (int) (blockIdx.x / (unsigned) tiles_n) * SLIM, n0 = (int) (blockIdx.x % (unsigned) tiles_n) * SLIM;
    // This thread's copies of a slab: always the same elements of it, one slab further each time.
    constexpr int COPIES = SLIM * SLIM_SLAB / SLIM_THREADS;
    const float *pa[COPIES], *pb[COPIES];
    int ka[COPIES], kb[COPIES];                          // k of the next copy; K or more: nothing is left, or the row does not exist
    const ptrdiff_t a_im_at = a_im - a_re, b_im_at = b_im - b_re;
#pragma unroll
    for (int j = 0; j < COPIES; ++j) {
        const int e = tid + j * SLIM_THREADS;
        const int ma = AK ? e / SLIM_SLAB : e % SLIM, nb = BK ? e / SLIM_SLAB : e % SLIM;
        ka[j] = AK ? e % SLIM_SLAB : e / SLIM;
        kb[j] = BK ? e % SLIM_SLAB : e / SLIM;
        pa[j] = a_re + (size_t) (m0 + ma) * sam + (size_t) ka[j] * sak;
        pb[j] = b_re + (size_t) (n0 + nb) * sbn + (size_t) kb[j] * sbk;
        if (m0 + ma >= M) ka[j] = K;
        if (n0 + nb >= N) kb[j] = K;
    }
    const ptrdiff_t a_step = (ptrdiff_t) SLIM_SLAB * sak, b_step = (ptrdiff_t) SLIM_SLAB * sbk;
    auto fetch = [&](int slab) {
        if (slab * SLIM_SLAB < K) {
            Slab& s = slabs[slab % STAGES];
#pragma unroll
            for (int j = 0; j < COPIES; ++j) {
                const int e = tid + j * SLIM_THREADS;
                const int ra = AK ? e / SLIM_SLAB : e % SLIM, rb = BK ? e / SLIM_SLAB : e % SLIM;
                const int la = AK ? e % SLIM_SLAB : e / SLIM, lb = BK ? e % SLIM_SLAB : e / SLIM;
                const bool ina = ka[j] < K, inb = kb[j] < K;
                const float *qa = ina ? pa[j] : a_re, *qb = inb ? pb[j] : b_re;
                copy4(s.ar.at(ra, la), qa, ina); copy4(s.ai.at(ra, la), qa + a_im_at, ina);
                copy4(s.br.at(rb, lb), qb, inb); copy4(s.bi.at(rb, lb), qb + b_im_at, inb);
                pa[j] += a_step; pb[j] += b_step;
                ka[j] += SLIM_SLAB; kb[j] += SLIM_SLAB;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    const unsigned sign = conjB ? 0x80000000u : 0u;
    float cr = 0.f, ci = 0.f, sr = 0.f, si = 0.f;
    const int slab_count = (K + SLIM_SLAB - 1) / SLIM_SLAB;
    for (int n = 0; n < slab_count; ++n) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                 // this slab is here, and nobody reads the one before any more
        fetch(n + STAGES - 1);
        Slab& s = slabs[n % STAGES];
        const int left = min(SLIM_SLAB, K - n * SLIM_SLAB);
        auto step = [&](float ax, float ay, float bx, float by) {
            by = __uint_as_float(__float_as_uint(by) ^ sign);
            cr += fmaf(ax, bx, -(ay * by));              // rounded as in the other kernel
            ci += fmaf(ax, by, ay * bx);
        };
        auto end_chain = [&] { sr += cr; si += ci; cr = ci = 0.f; };
        if (left == SLIM_SLAB) {
#pragma unroll
            for (int k = 0; k < SLIM_SLAB; k += 4) {
                float ax[4], ay[4], bx[4], by[4];
                s.ar.four(ty, k, ax); s.ai.four(ty, k, ay); s.br.four(tx, k, bx); s.bi.four(tx, k, by);
#pragma unroll
                for (int i = 0; i < 4; ++i) step(ax[i], ay[i], bx[i], by[i]);
                if (CHAINS && (k + 4) % CHAIN == 0) end_chain();
            }
        } else {
            for (int k = 0; k < left; ++k) {
                step(*s.ar.at(ty, k), *s.ai.at(ty, k), *s.br.at(tx, k), *s.bi.at(tx, k));
                if (CHAINS && (k % CHAIN == CHAIN - 1 || k + 1 == left)) end_chain();
            }
        }
    }
    const int gm = m0 + ty, gn = n0 + tx;
    if (gm >= M || gn >= N) return;
    const size_t o = (size_t) gm * N + gn;
    float vr = CHAINS ? sr : cr, vi = CHAINS ? si : ci;
    if (r_re) { vr += r_re[o]; vi += r_im[o]; }
    if (accumulate) { vr += d_re[o]; vi += d_im[o]; }
    d_re[o] = vr; d_im[o] = vi;
}

// Where tiles of 8 x 8 are the faster ones, in 210 products of up to 8 million multiplications (us, tiles of 16 or 32 and of 8): up to
// one and a half to an SM, two where both operands lie along k, one and a quarter where neither does (128 x 128, K = 128, 1.7: 5.0 and 4.6, and
// 5.0 and 5.7; 260 x 35, K = 223, 1.1, 7.8 and 7.0).  Beyond, where A lies along k: from 1.25 tiles of 16 to an SM on, which are the second
// round of those (177 x 285, K = 35 4.3 and 3.4; 87 x 794, K = 89 8.9 and 6.4; but 108 x 403, K = 107, 1.23, 5.8 and 6.6), up to eight of
// these (91 x 899, K = 36, 9.2, 4.3 and 4.8), and where a tile of 16 would be a quarter empty at a K that counts (1241 x 20, K = 204 14.4 and 10.5).
// Below a K of 16 five slabs on their way are none, and their set-up is what counts (16 x 31, K = 3 1.15 and 1.43, 123 x 381, K = 2 2.0 and
// 2.2; 60 sizes of K from 16 to 23 0.95 of the time in the mean).
bool slim_tiles(int M, int N, int K, bool ak, bool bk, int sms) {
    if (K < 16) return false;
    const long slim = (long) ((M + SLIM - 1) / SLIM) * ((N + SLIM - 1) / SLIM), small = (long) ((M + 15) / 16) * ((N + 15) / 16);
    if (4 * slim <= (ak && bk ? 8 : ak || bk ? 6 : 5) * sms) return true;
    if (!ak) return false;
    return (4 * small > 5L * sms && slim <= 8L * sms) || (slim <= 3 * small && slim <= 4L * sms && K >= 96);
}

}  // namespace

namespace cnb {

int cgemm_simt(cnb_ctx* ctx, const float* a_re, const float* a_im, long sam, long sak, const float* b_re,
               const float* b_im, long sbn, long sbk, int conjB, const float* r_re, const float* r_im,
               float* d_re, float* d_im, int M, int N, int K, int accumulate, cudaStream_t st) {
    auto go = [&](auto kernel, long tiles, bool dependent = true) {
        return cnb::launch_ex(kernel, dim3((unsigned) tiles), dim3(256), 0, st, 1, dependent, a_re, a_im, sam, sak, b_re, b_im, sbn, sbk, conjB, r_re,
                              r_im, d_re, d_im, M, N, K, accumulate);
    };
    // Small tiles while they hardly fill the device, where twice the loads for an output cost nothing: one to an SM whatever
    // K (30 x 20, K = 3000: 156 us with the others, 85), up to six of a short K (4096 x 16, K = 100: 14.6 and 9.8; 1000 x
    // 60, K = 1000, two to an SM: 77 and 81).
    const long small = (long) ((M + 15) / 16) * ((N + 15) / 16), large = (long) ((M + 31) / 32) * ((N + 31) / 32);
    const bool tile16 = small <= ctx->sm_count || (K <= 256 && small <= 6L * ctx->sm_count);
    const bool chains = cgemm_fma_in_chains(M, N, K), ak = sak == 1, bk = sbk == 1;
    if (slim_tiles(M, N, K, ak, bk, ctx->sm_count)) {
        const long slim = (long) ((M + SLIM - 1) / SLIM) * ((N + SLIM - 1) / SLIM);
#define CNB_SLIM_K(A, B) (chains ? cgemm_slim_k<A, B, true> : cgemm_slim_k<A, B, false>)
        CNB_CUDA(cnb::launch(ak ? (bk ? CNB_SLIM_K(true, true) : CNB_SLIM_K(true, false)) : bk ? CNB_SLIM_K(false, true) : CNB_SLIM_K(false, false),
                             dim3((unsigned) slim), dim3(SLIM_THREADS), 0, st, 1, a_re, a_im, sam, sak, b_re, b_im, sbn, sbk, conjB, r_re, r_im, d_re, d_im,
                             M, N, K, accumulate));
#undef CNB_SLIM_K
        CNB_LAUNCH_CHECK("cgemm_slim");
        return CNB_OK;
    }
    if (chains) {
        CNB_CUDA(tile16 ? go(cgemm_simt_k<16, 32, true>, small) : go(cgemm_simt_k<32, 32, true>, large));
    } else {
        // Tiles of 64 read half as much for an output, in slabs of 16, two to an SM, which share its issue slots: as many rounds
        // as the fullest SM has tiles, three quarters of them full at least (tiles of 32 and of 64, us: 2000 x 2000, K = 2000,
        // 6.9 tiles to an SM, 2290 and 1930; 777 x 1333, K = 1001, 1.8, 347 and 283; 300 x 3000, K = 700, 1.6, 214 and 199; 512 x
        // 1024, K = 512, 0.9, 92 and 82; but 777 x 1001, K = 1333, 1.4, 347 and 374, 1500 x 200, K = 1500, 0.7, 200 and 325).
        // Not launched ahead of the kernel before: its tiles would take what is free on that one's SMs by twos, with others
        // empty (0.9 to an SM: 92 and 135).
        const long huge = (long) ((M + 63) / 64) * ((N + 63) / 64), rounds = (huge + ctx->sm_count - 1) / ctx->sm_count;
        if (K >= 64 && 4 * huge >= 3 * rounds * ctx->sm_count) CNB_CUDA(go(cgemm_simt_k<64, 16, false>, huge, false));
        else CNB_CUDA(tile16 ? go(cgemm_simt_k<16, 32, false>, small) : go(cgemm_simt_k<32, 32, false>, large));
    }
    CNB_LAUNCH_CHECK("cgemm_simt");
    return CNB_OK;
}

}  // namespace cnb
