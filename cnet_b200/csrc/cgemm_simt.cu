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
    if (cgemm_fma_in_chains(M, N, K)) {
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
