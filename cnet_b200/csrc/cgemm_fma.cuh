// One 64 x 64 tile of a complex product of packed operands in fp32 FMAs (cgemm_tc.cu): 256 threads with a 4 x 4 block of complex accumulators each, k-slabs
// of 16 in shared memory, the next slab on its way while one is worked on.  The terms of an element are added in the
// order of k.
#pragma once
#include "common.cuh"

namespace cnb_fma {

constexpr int TM = 64, TN = 64, TK = 16;
struct Slabs { float a_re[TK][TM + 4], a_im[TK][TM + 4], b_re[TK][TN + 4], b_im[TK][TN + 4]; };

struct Result {
    float* d_re; float* d_im;
    const float* r_re; const float* r_im;    // added, or NULL
    int M, N, K, conjB, accumulate;
};

// Operands: float2 operator()(row, k), and k_fast, whether k or the row is the index that is contiguous in memory.
// tid 0..255; sync is a barrier of these threads.
template <class A, class B, class Sync>
__device__ __forceinline__ void tile(const A& a, const B& b, const Result& p, Slabs& s, int m0, int n0, int tid, Sync sync) {
    const int tx = tid & 15, ty = tid >> 4;
    float cr[4][4] = {}, ci[4][4] = {};
    float2 na[4], nb[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = tid + j * 256;                 // 0..1023 = TM * TK
            const int mm = a.k_fast ? e / TK : e % TM, ka = k0 + (a.k_fast ? e % TK : e / TM);
            const int nn = b.k_fast ? e / TK : e % TN, kb = k0 + (b.k_fast ? e % TK : e / TN);
            na[j] = nb[j] = make_float2(0.f, 0.f);
            if (m0 + mm < p.M && ka < p.K) na[j] = a(m0 + mm, ka);
            if (n0 + nn < p.N && kb < p.K) nb[j] = b(n0 + nn, kb);
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < p.K; k0 += TK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = tid + j * 256;
            const int mm = a.k_fast ? e / TK : e % TM, ka = a.k_fast ? e % TK : e / TM;
            const int nn = b.k_fast ? e / TK : e % TN, kb = b.k_fast ? e % TK : e / TN;
            s.a_re[ka][mm] = na[j].x; s.a_im[ka][mm] = na[j].y;
            s.b_re[kb][nn] = nb[j].x; s.b_im[kb][nn] = p.conjB ? -nb[j].y : nb[j].y;
        }
        sync();
        if (k0 + TK < p.K) fetch(k0 + TK);
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            float ar[4], ai[4], br[4], bi[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                ar[i] = s.a_re[kk][ty * 4 + i]; ai[i] = s.a_im[kk][ty * 4 + i];
                br[i] = s.b_re[kk][tx * 4 + i]; bi[i] = s.b_im[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    cr[i][j] += ar[i] * br[j] - ai[i] * bi[j];
                    ci[i][j] += ar[i] * bi[j] + ai[i] * br[j];
                }
        }
        sync();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= p.N) continue;
            const size_t o = (size_t) gm * p.N + gn;
            float vr = cr[i][j], vi = ci[i][j];
            if (p.r_re) { vr += p.r_re[o]; vi += p.r_im[o]; }
            if (p.accumulate) { vr += p.d_re[o]; vi += p.d_im[o]; }
            p.d_re[o] = vr; p.d_im[o] = vi;
        }
    }
}

}  // namespace cnb_fma
