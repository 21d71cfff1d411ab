// FourierTrans at any length that fits shared memory: a mixed-radix Stockham transform, rows in shared memory.
//
// N is factored into radices of at most 16 (2..16; primes up to 13), as few passes as that takes: 784 = 8 x 14 x 7,
// 1500 = 10 x 15 x 10, 4096 = 16 x 16 x 16.  A thread takes one butterfly of R points at a time in registers; pass p
// with L = the product of the radices before it reads x[j + q N/R], multiplies by e^{-2 pi i (j % L) q / (L R)},
// transforms over q and writes (j / L) L R + j % L + q L, so the last pass comes out in natural order.  The first
// pass reads the planes and the last one writes them (consecutive threads, consecutive elements); the passes between
// go through shared memory, whose elements are spread by one in every 16 against bank conflicts where that helps (choose_spread).
//
// Lengths with a prime factor above 13 use the chirp form (Bluestein): X[k] = c[k] sum_n (x[n] c[n]) conj(c[k-n]),
// c[n] = e^{-pi i n^2 / N}, the convolution as two transforms of a length M >= 2N-1 that factors well, in the same
// launch and the same shared memory.
//
// The conjugate transform is the forward one with the planes swapped on both sides.  HBM traffic: one read and one
// write of the tensor; a product with the N x N twiddle matrix (the only other form for these lengths) costs 8 N
// flops an element and the matrix.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "fft_mixed.cuh"
#include "fft_regs.cuh"

namespace {

using namespace cnb_mixed;
using cnb_fft::FftEpilogue;

constexpr int MAX_PASSES = 6, MAX_THREADS = 256;
constexpr size_t MAX_SMEM = 224 * 1024;

struct Pass {
    int radix, L, nb;                 // nb = length / radix butterflies per row
    unsigned mag_nb, mag_L;           // reciprocals for the two divisions of an index (0: the divisor is 1)
    int tw;                           // first entry of the pass's twiddles: [q - 1][k], q = 1..radix-1, k < L
};

struct MixedPlan {
    int n, m;                         // row length; transform length (m > n: chirp form)
    int passes, rows, threads, stride; // rows per CTA; float2 per row of a buffer
    int buffers, shift;               // shift: spread of the buffers' rows, 4 or NO_SPREAD
    Pass p[MAX_PASSES];
    float scale;
    unsigned mag_n;                   // reciprocal of n
};

// Where element i of a row lies in a buffer: every 16th set one further (shift 4), or as it is.  Constants of the kernel: a
// shift read from the plan cost every length 1 to 3 %.
constexpr int SPREAD = 4, NO_SPREAD = 31;
template <int SHIFT> __host__ __device__ __forceinline__ int pad_of(int i) { return i + (SHIFT == NO_SPREAD ? 0 : i >> SHIFT); }

__device__ __forceinline__ int div_by(int i, unsigned mag) { return mag ? (int) __umulhi((unsigned) i, mag) : i; }

struct Io {
    const float *xr, *xi;             // planes of this CTA's first row
    float *yr, *yi;
    const float2 *tw, *chirp, *spectrum;
    const float2* src;                // shared-memory buffers, NULL: the planes
    float2* dst;
    int rows;
    bool spectral;                    // chirp form: this pass opens the inverse transform
    size_t row0;
};

// What becomes of a finished row: stored, stored and taken through the tail (by the threads that hold its last butterflies, or from
// shared memory by all in turn), or added to what is there.
enum Finish { STORE = 0, TAIL = 1, ADD = 2, TAIL_LOOP = 3 };

// The tail of an element whose transform is u: u, u o h where it is kept, CGelu of that.
__device__ __forceinline__ void tail_store(const Io& io, const FftEpilogue& ep, size_t g, size_t at, float2 u, float hr, float hi) {
    io.yr[g] = u.x;
    io.yi[g] = u.y;
    const float ar = u.x * hr - u.y * hi, ai = u.x * hi + u.y * hr;
    const float gr = cnb_gelu(ar), gi = cnb_gelu(ai);
    if (ep.ar) { ep.ar[at] = ar; ep.ai[at] = ai; }
    if (ep.gr) { ep.gr[at] = gr; ep.gi[at] = gi; }
    if (ep.sp) {
        cnb_split_store1(cnb_split_component(ep.sp, ep.np, 0), at, gr);
        cnb_split_store1(cnb_split_component(ep.sp, ep.np, 1), at, gi);
    }
}

template <int R, int FINISH, bool CHIRP, int SHIFT>
__device__ __forceinline__ void run_pass(const MixedPlan& pl, const Pass& d, Io& io, const FftEpilogue& ep) {
    const int items = io.rows * d.nb;
    for (int i = threadIdx.x; i < items; i += blockDim.x) {
        const int row = div_by(i, d.mag_nb), j = i - row * d.nb;
        float2 v[R];
        if (io.src) {
            const float2* s = io.src + row * pl.stride;
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = s[pad_of<SHIFT>(j + q * d.nb)];
            if (CHIRP && io.spectral) {
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const float2 t = cmul(v[q], __ldg(io.spectrum + j + q * d.nb));
                    v[q] = make_float2(t.y, t.x);          // swapped: the inverse transform
                }
            }
        } else {
            const float* pr = io.xr + (size_t) row * pl.n + j;
            const float* pi = io.xi + (size_t) row * pl.n + j;
            if (CHIRP) {
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const int e = j + q * d.nb;
                    v[q] = make_float2(0.f, 0.f);
                    if (e < pl.n) v[q] = cmul(make_float2(pr[q * d.nb], pi[q * d.nb]), __ldg(io.chirp + e));
                }
            } else {
#pragma unroll
                for (int q = 0; q < R; ++q) v[q] = make_float2(pr[q * d.nb], pi[q * d.nb]);
            }
        }
        const int k = j - div_by(j, d.mag_L) * d.L;
        if (d.L > 1) {
            const float2* w = io.tw + d.tw + k;
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = cmul(v[q], __ldg(w + (q - 1) * d.L));
        }
        dft<R>(v);
        const int o = (j - k) * R + k;
        if (io.dst) {
            float2* t = io.dst + row * pl.stride;
#pragma unroll
            for (int q = 0; q < R; ++q) t[pad_of<SHIFT>(o + q * d.L)] = v[q];
        } else {
            const size_t base = (size_t) row * pl.n + o;
            // Old values are requested together, before the first store: between the stores each load waited for the
            // store before it, R round trips one after another.  A form of its own, because the registers they sit
            // in cost the plain transform a CTA per SM (1000 x 1500 both ways 26.5 -> 30.2 us).
            float2 old[FINISH == ADD ? R : 1];
            if (FINISH == ADD) {
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const size_t g = (size_t) row * pl.n + (CHIRP ? min(o + q * d.L, pl.n - 1) : o + q * d.L);
                    old[FINISH == ADD ? q : 0] = make_float2(io.yr[g], io.yi[g]);
                }
            }
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int e = o + q * d.L;
                if (CHIRP && e >= pl.n) break;
                const size_t g = base + (size_t) q * d.L;
                float2 u = v[q];
                if (CHIRP) u = cmul(make_float2(u.y, u.x), __ldg(io.chirp + e));
                u.x *= pl.scale; u.y *= pl.scale;
                if (FINISH == ADD) { u.x += old[FINISH == ADD ? q : 0].x; u.y += old[FINISH == ADD ? q : 0].y; }
                if (FINISH == TAIL) {
                    // the kernels before may have written h: the read-only path only behind a barrier of this one
                    const bool lone = pl.passes == 1;
                    const float hr = lone ? cnb_ld_behind_wait(ep.hr + e) : __ldg(ep.hr + e), hi = lone ? cnb_ld_behind_wait(ep.hi + e) : __ldg(ep.hi + e);
                    tail_store(io, ep, g, (io.row0 + row) * (size_t) pl.n + e, u, hr, hi);
                } else {
                    io.yr[g] = u.x;
                    io.yi[g] = u.y;
                }
            }
        }
    }
}

// TAIL_LOOP: the rows lie finished, but for their scale (and chirp), at `s`.
template <bool CHIRP, int SHIFT>
__device__ __forceinline__ void tail_loop(const MixedPlan& pl, const Io& io, const FftEpilogue& ep, const float2* s) {
    const int total = io.rows * pl.n, step = blockDim.x;
    for (int i0 = threadIdx.x; i0 < total; i0 += 2 * step) {
        float2 u[2], h[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = i0 + k * step, row = div_by(i, pl.mag_n), e = i - row * pl.n;
            if (i >= total) break;
            h[k] = make_float2(__ldg(ep.hr + e), __ldg(ep.hi + e));
            u[k] = s[row * pl.stride + pad_of<SHIFT>(e)];
            if (CHIRP) u[k] = cmul(make_float2(u[k].y, u[k].x), __ldg(io.chirp + e));
            u[k].x *= pl.scale; u[k].y *= pl.scale;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = i0 + k * step;
            if (i < total) tail_store(io, ep, i, io.row0 * (size_t) pl.n + i, u[k], h[k].x, h[k].y);
        }
    }
}

// CTAS: how many of 256 threads an SM's registers are to hold, two or three (fewer_waves).
template <int FINISH, bool CHIRP, int SHIFT, int CTAS>
__global__ void __launch_bounds__(MAX_THREADS, CTAS)
fft_mixed_k(const float* __restrict__ xr, const float* __restrict__ xi, float* yr, float* yi,
            const float2* __restrict__ tw, const float2* __restrict__ chirp, const float2* __restrict__ spectrum, int B,
            const FftEpilogue ep, const __grid_constant__ MixedPlan pl) {
    cnb_pdl_enter();
    extern __shared__ __align__(16) float2 bufs[];
    Io io;
    io.row0 = (size_t) blockIdx.x * pl.rows;
    io.rows = min(pl.rows, B - (int) io.row0);
    io.xr = xr + io.row0 * pl.n; io.xi = xi + io.row0 * pl.n;
    io.yr = yr + io.row0 * pl.n; io.yi = yi + io.row0 * pl.n;
    io.tw = tw; io.chirp = chirp; io.spectrum = spectrum;
    const int total = CHIRP ? 2 * pl.passes : pl.passes;
    for (int s = 0; s < total; ++s) {
        const Pass& d = pl.p[CHIRP && s >= pl.passes ? s - pl.passes : s];
        io.src = s == 0 ? nullptr : bufs + (s & 1 ? 0 : pl.rows * pl.stride);
        io.dst = s == total - 1 && FINISH != TAIL_LOOP ? nullptr : bufs + (s & 1 ? pl.rows * pl.stride : 0);
        io.spectral = CHIRP && s == pl.passes;
        switch (d.radix) {
#define CNB_RADIX(R) case R: run_pass<R, FINISH, CHIRP, SHIFT>(pl, d, io, ep); break
            CNB_RADIX(2); CNB_RADIX(3); CNB_RADIX(4); CNB_RADIX(5); CNB_RADIX(6); CNB_RADIX(7); CNB_RADIX(8); CNB_RADIX(9);
            CNB_RADIX(10); CNB_RADIX(11); CNB_RADIX(12); CNB_RADIX(13); CNB_RADIX(14); CNB_RADIX(15); CNB_RADIX(16);
#undef CNB_RADIX
        }
        if (s < total - 1 || FINISH == TAIL_LOOP) __syncthreads();
    }
    if (FINISH == TAIL_LOOP) tail_loop<CHIRP, SHIFT>(pl, io, ep, bufs + ((total - 1) & 1 ? pl.rows * pl.stride : 0));
}

// twiddles of every pass, packed as Pass::tw says, in double
__global__ void mixed_twiddle_k(float2* __restrict__ tw, const __grid_constant__ MixedPlan pl) {
    for (int p = 0; p < pl.passes; ++p) {
        const Pass d = pl.p[p];
        if (d.L == 1) continue;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (d.radix - 1) * d.L; i += gridDim.x * blockDim.x) {
            const int q = i / d.L + 1, k = i % d.L;
            double s, c;
            sincospi(-2.0 * (double) (k * q) / ((double) d.L * d.radix), &s, &c);
            tw[d.tw + i] = make_float2((float) c, (float) s);
        }
    }
}

// chirp[n] = e^{-pi i n^2 / N}; spectrum = DFT_M of b, b[n] = b[M - n] = conj(chirp[n]) for n < N, 0 between, over M
__global__ void mixed_chirp_k(float2* __restrict__ chirp, float2* __restrict__ spectrum, int N, int M) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        double s, c;
        sincospi((double) ((long) i * i % (2L * N)) / N, &s, &c);
        chirp[i] = make_float2((float) c, (float) -s);
    }
    for (int k = warp; k < M; k += warps) {
        double re = 0.0, im = 0.0;
        for (int n = 1 + lane; n < N; n += 32) {           // b is even: 2 sum b[n] cos(2 pi n k / M)
            double s, c;
            sincospi((double) ((long) n * n % (2L * N)) / N, &s, &c);
            const double t = 2.0 * cospi(2.0 * (double) ((long) n * k % M) / M);
            re += c * t; im += s * t;
        }
        for (int o = 16; o > 0; o >>= 1) { re += __shfl_xor_sync(0xffffffffu, re, o); im += __shfl_xor_sync(0xffffffffu, im, o); }
        if (lane == 0) spectrum[k] = make_float2((float) ((re + 1.0) / M), (float) (im / M));
    }
}

// ------------------------------------------------------------------------------------------------------- plans
unsigned reciprocal(int d) { return d == 1 ? 0u : (unsigned) ((1ull << 32) / (unsigned) d + 1); }

// Work of a butterfly of R points in the units of an element's trip through shared memory: primes cost their
// square, and every butterfly some index arithmetic.
double butterfly_cost(int r) {
    const int p = r % 13 == 0 ? 13 : r % 11 == 0 ? 11 : r % 7 == 0 ? 7 : r % 5 == 0 ? 5 : 2;
    return 4.0 + r * (1.0 + 0.04 * p);
}

// every factorisation of m into exactly `left` radices, non-increasing
void factorisations(int m, int left, int most, std::vector<int>& cur, std::vector<std::vector<int> >& out) {
    if (left == 0) { if (m == 1) out.push_back(cur); return; }
    for (int r = std::min(most, 16); r >= 2; --r) {
        if (m % r) continue;
        cur.push_back(r);
        factorisations(m / r, left - 1, r, cur, out);
        cur.pop_back();
    }
}

// The radices of a transform of length m, or false when a prime factor exceeds 13.  Of the factorisations with the
// fewest passes the one of least work; the largest radix goes into the middle, where consecutive threads need not
// touch consecutive elements of the planes (narrow first and last passes keep those runs long).
bool choose_radices(int m, std::vector<int>* radices, double* cost) {
    for (int n = 1; n <= MAX_PASSES; ++n) {
        std::vector<int> cur;
        std::vector<std::vector<int> > all;
        factorisations(m, n, 16, cur, all);
        if (all.empty()) continue;
        double best = 1e30;
        for (auto& f : all) {
            double c = 0;
            for (int r : f) c += butterfly_cost(r) / r;
            if (c < best) { best = c; *radices = f; }
        }
        if (radices->size() > 2) std::swap((*radices)[0], (*radices)[1]);
        *cost = best * m;
        return true;
    }
    return false;
}

int row_stride(int m) { return pad_of<SPREAD>(m) + 1; }
size_t smem_bytes(int m, int rows, int buffers) { return (size_t) buffers * rows * row_stride(m) * sizeof(float2); }

// Wavefronts of the 8-byte accesses of up to 32 lanes: 16 at a time, a word pair per bank pair.
int wavefronts(const int (&at)[32], int lanes) {
    int sum = 0;
    for (int h = 0; h < lanes; h += 16) {
        int most = 0, count[16] = {};
        for (int l = h; l < std::min(lanes, h + 16); ++l) most = std::max(most, ++count[at[l] & 15]);
        sum += most;
    }
    return sum;
}

// The spread of fewest wavefronts over the first warps' butterflies of every pass, weighed by the butterflies they stand for.
// Radix 16 wants every 16th element set apart; runs 10 apart get into each other's way by it: 1500 = 10 x 15 x 10 had 4.8
// wavefronts too many a store (1000 rows 12.9 -> 11.0 us; 10000 x 100 8.8 -> 7.9, 1000 x 1000 11.4 -> 9.7).
int choose_spread(const MixedPlan& pl) {
    double cost[2] = {0, 0};
    for (int v = 0; v < 2; ++v)
        for (int p = 0; p < pl.passes; ++p) {
            const Pass& d = pl.p[p];
            const int warps = std::min(4, (d.nb + 31) / 32);
            int sum = 0;
            for (int w = 0; w < warps; ++w)
                for (int q = 0; q < d.radix; ++q) {
                    int to[32], from[32], n = 0;
                    for (int i = 32 * w; i < std::min(32 * w + 32, d.nb); ++i, ++n) {
                        const int o = (i - i % d.L) * d.radix + i % d.L + q * d.L, s = i + q * d.nb;
                        to[n] = v ? pad_of<SPREAD>(o) : o;
                        from[n] = v ? pad_of<SPREAD>(s) : s;
                    }
                    sum += (p + 1 < pl.passes ? wavefronts(to, n) : 0) + (p > 0 ? wavefronts(from, n) : 0);
                }
            cost[v] += (double) sum * d.nb / std::min(32 * warps, d.nb);
        }
    return cost[0] < 0.95 * cost[1] ? NO_SPREAD : SPREAD;
}


int buffers_for(int passes, bool chirp) {
    const int hops = (chirp ? 2 * passes : passes) - 1;     // passes that write shared memory
    return hops > 1 ? 2 : hops;
}

// The length-dependent part of a plan; false: this length has no kernel here.
bool plan_length(int N, MixedPlan* out) {
    if (N < 2) return false;
    std::vector<int> radices, r;
    double cost = 0, c;
    int m = N;
    if (!choose_radices(N, &radices, &cost)) {
        // chirp: of the lengths up to a fifth above the least one, the cheapest
        cost = 1e30;
        const int least = 2 * N - 1;
        for (int t = least; t <= least + std::max(8, least / 5); ++t)
            if (choose_radices(t, &r, &c) && c < cost) { cost = c; m = t; radices = r; }
        if (radices.empty()) return false;
    }
    MixedPlan pl = {};
    pl.n = N; pl.m = m;
    pl.passes = (int) radices.size();
    pl.stride = row_stride(m);
    pl.buffers = buffers_for(pl.passes, m > N);
    if (smem_bytes(m, 1, pl.buffers) > MAX_SMEM) return false;
    int L = 1, tw = 0;
    for (int p = 0; p < pl.passes; ++p) {
        Pass& d = pl.p[p];
        d.radix = radices[p]; d.L = L; d.nb = m / radices[p];
        d.mag_nb = reciprocal(d.nb); d.mag_L = reciprocal(d.L);
        d.tw = tw;
        if (L > 1) tw += (d.radix - 1) * L;
        L *= d.radix;
    }
    pl.shift = m > N ? SPREAD : choose_spread(pl);
    pl.scale = (float) (1.0 / std::sqrt((double) N));
    pl.mag_n = reciprocal(N);
    *out = pl;
    return true;
}

bool cached_plan(int N, MixedPlan* out) {
    static std::mutex mu;
    static std::map<int, MixedPlan> plans;                  // at most one entry per length; n = 0: no kernel
    std::lock_guard<std::mutex> lock(mu);
    auto it = plans.find(N);
    if (it == plans.end()) {
        MixedPlan pl = {};
        if (!plan_length(N, &pl)) pl.n = 0;
        it = plans.emplace(N, pl).first;
    }
    *out = it->second;
    return out->n != 0;
}

// Rows per CTA and threads: about four CTAs to an SM (up to 52 KB of shared memory each), so that some load or store
// while others transform; rows are spread over the SMs first when the batch is small; of the thread counts the one
// that wastes the fewest lanes over the passes, or, with no more than 1.75 CTAs to an SM, the one with the fewest butterflies
// one after another (64 x 784, 128 threads instead of 64: 5.7 -> 5.1 us, with the tail 8.3 -> 6.4; at 1.5 to 1.7, 900 x 303 19.8 -> 13.6, 1000 x 300
// 4.5 -> 3.7, 250 x 784 4.5 -> 3.9; at 2.0, 3000 x 137 16.0 and 16.6, 2662 x 77 3.2 and 3.7).
void plan_batch(MixedPlan* pl, int B, int sms) {
    const size_t budget = 52 * 1024;
    int rows = 1;
    while (rows < 64 && smem_bytes(pl->m, rows + 1, std::max(1, pl->buffers)) <= budget && (long) (rows + 1) * pl->m <= 4096) ++rows;
    rows = std::max(1, std::min(rows, (B + 2 * sms - 1) / (2 * sms)));
    const long ctas = (B + rows - 1) / rows;
    const bool alone = 4 * ctas <= 7L * sms;
    double best = 1e30;
    for (int t = 64; t <= MAX_THREADS; t += 32) {
        double c = 0;
        for (int p = 0; p < pl->passes; ++p) {
            const int items = rows * pl->p[p].nb;
            c += (double) ((items + t - 1) / t) * butterfly_cost(pl->p[p].radix);
        }
        if (!alone) c *= t + 32;                            // lanes held, and a little for every CTA
        if (c < best * 0.999) { best = c; pl->threads = t; }
    }
    pl->rows = rows;
}

// Whether the form of fewer registers (80 a thread in the place of 96, with the tail 112) is the faster one: it has to save a wave of
// CTAs, since what it costs in loads and arithmetic ahead is more than it gives where it does not, and to hold a third more of them
// (us, with more registers and with 80: 4096 x 784 plain 22.3 and 19.7, 2282 x 396 8.9 and 7.1, 2000 x 2000 36.2 and 29.6; but four
// CTAs or five to an SM 2500 x 1600 23.4 and 23.9, 12361 x 208 backward 17.4 and 17.9, 39267 x 50 11.4 and 11.5).
//
// With the tail, short rows store runs of a few floats into four planes, and more CTAs at once are in each other's way there: a saved
// wave may stand for three and a half CTAs an SM, five and a half where two were resident (1000 x 1500 22.6 and 16.9, 28360 x 32 10.2
// and 7.7; but 47095 x 50 23.0 and 25.8, 82001 x 50 34.3 and 38.6, 48007 x 72 33.4 and 36.1, 64750 x 49
// 36.6 and 38.0; of 247 sizes that save a wave, 33 that lost by it are left out so, and 27 % of what the others gain).
bool fewer_waves(long ctas, int threads, size_t smem, int regs, int fewer, int sms, int n, bool tail) {
    auto fit = [&](int r) {
        const long by_registers = 65536 / ((long) threads * ((r + 7) / 8 * 8)), by_memory = (long) (227 * 1024 / (smem + 1024));
        return std::max(1L, std::min({by_registers, by_memory, 2048L / threads}));
    };
    auto waves = [&](long f) { return (ctas + f * sms - 1) / (f * sms); };
    const long before = fit(regs), after = fit(fewer), saved = waves(before) - waves(after);
    if (saved <= 0 || 3 * after < 4 * before) return false;
    return !tail || n > 256 || 2 * ctas <= (before == 2 ? 11 : 7) * saved * sms;
}

// The tail in a loop through shared memory, by all threads: written out behind a butterfly of 16 points it is 30 KB of
// instructions, which a small batch runs through once, at the pace of their first fetch, on the few threads that have a last
// butterfly (16 x 256 5.7 -> 3.0 us, 296 x 100 4.3 -> 2.9, 296 x 500 5.6 -> 4.2; in a training step, where other
// kernels' instructions lie between, more: calls back to back of rows whose last pass is light are slower by the loop, 9462 x 48 5.0 and 5.3,
// 8310 x 56 5.0 and 5.6, 512 x 784 5.8 and 6.2, and steps are not, 512 x 784 in 4 blocks 349 and 339, 359 x 273 30.9 and 29.0).  Not where the trip through shared memory counts, whose row one CTA then has on its way twice: from
// half a million elements (1024 x 512 6.2 and 6.3, 1024 x 900 11.2 and 16.3; half of that in the chirp form, 1024 x 137 7.6 and 7.4, 4096 x 137 16.8
// and 19.5) and beyond 1024 points (86 x 2000 7.3 and 7.5).  Two elements a thread, in one round: as many threads as that takes (16 x 256
// 3.0 us, with four 3.5).
bool loop_tail(MixedPlan* pl, int B) {
    const bool chirp = pl->m > pl->n;
    if (pl->n > 1024 || (long) B * pl->n >= (chirp ? 1 << 18 : 1 << 19)) return false;
    const int buffers = (chirp ? 2 : 1) * pl->passes > 1 ? 2 : 1;
    if (smem_bytes(pl->m, pl->rows, buffers) > MAX_SMEM) return false;
    pl->buffers = buffers;
    pl->threads = std::max(pl->threads, std::min(MAX_THREADS, (pl->rows * pl->n / 2 + 31) / 32 * 32));
    return true;
}

size_t twiddle_entries(const MixedPlan& pl) {
    size_t n = 0;
    for (int p = 0; p < pl.passes; ++p) if (pl.p[p].L > 1) n += (size_t) (pl.p[p].radix - 1) * pl.p[p].L;
    return n;
}

// twiddles of the passes, then for the chirp form c[0..n) and the spectrum
int make_mixed_tables(cnb_ctx* ctx, int key, cudaStream_t st, cnb_twiddle* t) {
    MixedPlan pl;
    cached_plan(-key, &pl);
    const size_t tw_entries = twiddle_entries(pl);
    const bool chirp = pl.m > pl.n;
    void* p = nullptr;
    const int rc = cnb_alloc(ctx, std::max<size_t>(1, tw_entries + (chirp ? (size_t) pl.n + pl.m : 0)) * sizeof(float2), &p);
    if (rc != CNB_OK) return rc;
    t->re = static_cast<float*>(p);
    float2* tab = static_cast<float2*>(p);
    mixed_twiddle_k<<<16, 256, 0, st>>>(tab, pl);
    CNB_LAUNCH_CHECK("mixed_twiddle");
    if (chirp) {
        mixed_chirp_k<<<ctx->sm_count * 4, 256, 0, st>>>(tab + tw_entries, tab + tw_entries + pl.n, pl.n, pl.m);
        CNB_LAUNCH_CHECK("mixed_chirp");
    }
    return CNB_OK;
}

}  // namespace

namespace cnb {

bool fft_mixed_supported(int N) {
    MixedPlan pl;
    return cached_plan(N, &pl);
}

int fft_mixed(cnb_ctx* ctx, const float* xr, const float* xi, float* yr, float* yi, int B, int N, int inverse,
              int accumulate, const FftEpilogue& ep, cudaStream_t st) {
    MixedPlan pl;
    if (!cached_plan(N, &pl)) return set_error(CNB_ERR_UNSUPPORTED, "fft: N=%d", N);
    plan_batch(&pl, B, usable_sms(ctx));
    const bool chirp = pl.m > pl.n;
    // the tables live in the arena; the map key -N keeps them apart from DFT matrices
    cnb_twiddle t;
    const int rc = table(ctx, -N, st, make_mixed_tables, &t);
    if (rc != CNB_OK) return rc;
    const size_t tw_entries = twiddle_entries(pl);
    const float2* tw = reinterpret_cast<const float2*>(t.re);
    const float2* ch = tw + tw_entries;
    const float2* spec = ch + pl.n;
    if (inverse) { std::swap(xr, xi); std::swap(yr, yi); }
    Finish finish = ep.hr ? TAIL : accumulate ? ADD : STORE;
    if (finish == TAIL && loop_tail(&pl, B)) finish = TAIL_LOOP;
    const size_t smem = smem_bytes(pl.m, pl.rows, pl.buffers);
    static bool attr_done[64] = {};                         // the attribute is per device
    static int registers[3][2];                             // of a thread in each form, as the kernels were built (all devices alike)
    if (!attr_done[ctx->device & 63]) {
#define CNB_MIXED_ATTR(F, C, S, N) \
    CNB_CUDA(cudaFuncSetAttribute(fft_mixed_k<F, C, S, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) MAX_SMEM))
#define CNB_MIXED_ATTRS(F, N) CNB_MIXED_ATTR(F, false, SPREAD, N); CNB_MIXED_ATTR(F, false, NO_SPREAD, N)
        CNB_MIXED_ATTRS(STORE, 2); CNB_MIXED_ATTRS(TAIL, 2); CNB_MIXED_ATTRS(ADD, 2); CNB_MIXED_ATTRS(TAIL_LOOP, 2);
        CNB_MIXED_ATTRS(STORE, 3); CNB_MIXED_ATTRS(TAIL, 3); CNB_MIXED_ATTRS(ADD, 3);
        CNB_MIXED_ATTR(STORE, true, SPREAD, 2); CNB_MIXED_ATTR(TAIL, true, SPREAD, 2); CNB_MIXED_ATTR(ADD, true, SPREAD, 2);
        CNB_MIXED_ATTR(TAIL_LOOP, true, SPREAD, 2);
#undef CNB_MIXED_ATTRS
#undef CNB_MIXED_ATTR
#define CNB_MIXED_REGS(F, N)                                                                                  \
    do {                                                                                                      \
        cudaFuncAttributes a, b;                                                                              \
        CNB_CUDA(cudaFuncGetAttributes(&a, fft_mixed_k<F, false, SPREAD, N>));                                \
        CNB_CUDA(cudaFuncGetAttributes(&b, fft_mixed_k<F, false, NO_SPREAD, N>));                             \
        registers[F][N - 2] = std::max(a.numRegs, b.numRegs);                                                 \
    } while (0)
        CNB_MIXED_REGS(STORE, 2); CNB_MIXED_REGS(TAIL, 2); CNB_MIXED_REGS(ADD, 2);
        CNB_MIXED_REGS(STORE, 3); CNB_MIXED_REGS(TAIL, 3); CNB_MIXED_REGS(ADD, 3);
#undef CNB_MIXED_REGS
        attr_done[ctx->device & 63] = true;
    }
    const dim3 grid((unsigned) ((B + pl.rows - 1) / pl.rows)), block((unsigned) pl.threads);
    auto go = [&](auto kernel) { return cnb::launch(kernel, grid, block, smem, st, 1, xr, xi, yr, yi, tw, ch, spec, B, ep, pl); };
    const bool spread = pl.shift == SPREAD;
#define CNB_MIXED(F, N) CNB_CUDA(spread ? go(fft_mixed_k<F, false, SPREAD, N>) : go(fft_mixed_k<F, false, NO_SPREAD, N>))
    if (chirp) {
        CNB_CUDA(finish == TAIL ? go(fft_mixed_k<TAIL, true, SPREAD, 2>) : finish == TAIL_LOOP ? go(fft_mixed_k<TAIL_LOOP, true, SPREAD, 2>) :
                 finish == ADD ? go(fft_mixed_k<ADD, true, SPREAD, 2>) : go(fft_mixed_k<STORE, true, SPREAD, 2>));
    } else if (finish == TAIL_LOOP) {
        CNB_MIXED(TAIL_LOOP, 2);
    } else if (fewer_waves((long) grid.x, pl.threads, smem, registers[finish][0], registers[finish][1], usable_sms(ctx), pl.n, finish == TAIL)) {
        if (finish == TAIL) CNB_MIXED(TAIL, 3);
        else if (finish == ADD) CNB_MIXED(ADD, 3);
        else CNB_MIXED(STORE, 3);
    } else if (finish == TAIL) {
        CNB_MIXED(TAIL, 2);
    } else if (finish == ADD) {
        CNB_MIXED(ADD, 2);
    } else {
        CNB_MIXED(STORE, 2);
    }
#undef CNB_MIXED
    CNB_LAUNCH_CHECK("fft_mixed");
    return CNB_OK;
}

}  // namespace cnb

extern "C" int cnb_fft_form(int N, int B, int tail, int sm_count, int regs, int fewer_regs, int* out4) {
    MixedPlan pl;
    if (!out4 || B <= 0 || sm_count <= 0 || regs <= 0 || fewer_regs <= 0) return cnb::set_error(CNB_ERR_ARG, "cnb_fft_form: B=%d sm_count=%d", B, sm_count);
    if (!cached_plan(N, &pl)) return cnb::set_error(CNB_ERR_UNSUPPORTED, "cnb_fft_form: N=%d", N);
    plan_batch(&pl, B, sm_count);
    const bool loop = tail && loop_tail(&pl, B);
    const long ctas = (B + pl.rows - 1) / pl.rows;
    out4[0] = (int) ctas;
    out4[1] = pl.threads;
    out4[2] = loop ? 1 : 0;
    out4[3] = !loop && pl.m == pl.n && fewer_waves(ctas, pl.threads, smem_bytes(pl.m, pl.rows, pl.buffers), regs, fewer_regs, sm_count, N, tail != 0);
    return CNB_OK;
}

extern "C" int cnb_fft_plan(int N, int B, int sm_count, int* out, int capacity) {
    MixedPlan pl;
    if (!out || capacity < 6 + MAX_PASSES || N < 1 || B < 1 || sm_count < 1)
        return cnb::set_error(CNB_ERR_ARG, "cnb_fft_plan: N=%d B=%d", N, B);
    if (!cached_plan(N, &pl)) return 0;
    plan_batch(&pl, B, sm_count);
    out[0] = pl.m; out[1] = pl.rows; out[2] = pl.threads; out[3] = pl.buffers; out[4] = pl.stride;
    out[5] = (int) smem_bytes(pl.m, pl.rows, pl.buffers);
    for (int p = 0; p < pl.passes; ++p) out[6 + p] = pl.p[p].radix;
    return pl.passes;
}
