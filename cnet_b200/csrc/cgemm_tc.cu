// tcgen05 complex GEMM on error-compensated operands, for sm_100a.
//
//   D[m,n] (+)= sum_k A[m,k] * (conjB ? conj(B[n,k]) : B[n,k]) (+ R[m,n])
//   A [M,K], B [N,K] complex, K-major (row-major) or MN-major ([K, rows]).
//
// Numerics.  Two operand forms, each three tensor-core MMAs per real product with fp32 accumulation in tensor memory.
// PACKED, what everything but the C ABI's split buffers runs on: two fp16 parts, high and low, of the matrix scaled by one
// power of two (22 bits; see pack_k below, also for matrices whose range is too wide for that and which run as fp32
// FMAs); high.low + low.high + high.high on the FP16 pipe, 1.5 TF32-equivalents, 4 operand bytes per real element.  Sizes
// whose alternative are fp32 FMAs are summed in chains short enough not to be less exact than those (max_chain).
// SPLIT, the split buffers: hi = x with the 13 low mantissa bits cleared (exactly a TF32 value) and lo = x - hi (exact in
// fp32);
//     hi*hi                on the TF32 pipe (exact products), and
//     hi*lo + lo*hi        on the BF16 pipe, from hi and lo rounded to bf16 (h16, l16).
// Its cross terms are 2^-10 of the product, so their bf16 rounding (2^-9 each factor) costs 2^-18 of the
// product per cross term at worst (2^-19.5 rms for both), next to the 2^-20 of the dropped lo*lo term; fp32's
// exponent range is kept (no scaling).  Two TF32-equivalents a real product, 8 operand bytes per real element.
//
// Tiling.  One CTA computes a 128 x 128 complex tile.  The B tile is staged as ONE 256-row
// operand [B_re rows ; B_im rows], so every MMA is 128 x 256 and the complex structure
// costs two accumulators instead of four MMA shapes:
//     acc1 = A_re * [B_re ; B_im]^T      (TMEM columns   0..255)
//     acc2 = A_im * [B_re ; B_im]^T      (TMEM columns 256..511)
//     D_re = acc1[:, :128] -/+ acc2[:, 128:],   D_im = acc1[:, 128:] +/- acc2[:, :128]   (epilogue)
// A stage holds 8 operand slots of 8 KB = 64 KB; 3 stages.  PACKED, a k-block of 32:
//     A high re, high im, low re, low im, then the same of B (fp16, 64-byte swizzle);
// per k-block and accumulator: 6 FP16 MMAs (k-steps of 16).  SPLIT, a k-block of 16:
//     A hi_re, A hi_im (fp32, 64-byte swizzle),  A h16 [re ; im], A l16 [re ; im] (bf16, 32-byte swizzle),
//     B hi_re, B hi_im,                          B h16 [re ; im], B l16 [re ; im];
// per k-block and accumulator: 2 TF32 MMAs (k-steps of 8) + 2 BF16 MMAs (one k-step of 16).
// Each CTA issues its own plain TMA tile loads; their zero fill handles every M/N/K edge.
//
// CTA pairs.  The large launches (cgemm_tc_k<true>) give a 256 x 128 tile to a cluster of two CTAs that work as
// one tensor core (cta_group::2): each CTA stages its own 128 rows of A and one half of the stacked B operand
// (B_re rows in the first CTA, B_im rows in the second), i.e. 48 KB per k-block instead of 64 KB, four stages
// instead of three.  The first CTA issues every MMA (M = 256); both CTAs load, drain their own accumulator rows
// and write them out.  Completion bytes of both CTAs' loads go to the first CTA's full barrier; its
// tcgen05.commit arrives on the stage's empty barrier (and on the "accumulators ready" barrier) of both.
//
// Scheduling.  Stream-K: the (tile, k-block) work units are cut into equal consecutive runs, one
// per CTA and one CTA per SM, so every SM finishes together whatever the tile count; a tile whose
// k-range is shared by several CTAs is summed with fp32 atomics into a pre-zeroed output.
//
// Roles.  warp 0: TMA producer; warp 1: TMEM allocation + MMA issue (one elected thread);
// the last eight warps: epilogue (tcgen05.ld, combine, stage through shared memory, coalesced 16-byte
// stores / atomics with residual or accumulate), two groups of four warps with half of a tile's columns each;
// tensor memory is handed back to the MMA warp as soon as it has been read, so the write-out overlaps the next
// run of MMAs.  With one group a whole tile left in 4.6 us after its last MMA, 8.9 with a residual and 18.8 where
// rows are not 16-byte aligned; 777 x 1333 x 1001 forward and both gradients 179 -> 157 us, 512 x 1024 x 1024 in a
// cluster of four 17.4 -> 16.6 (what is left there: 3.9 us of reading the peers' partial tiles).
// Every mbarrier wait is bounded (2 s); on expiry the kernel records an error word, skips to
// the common exit, frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <bitset>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "cgemm_fma.cuh"
#include "common.cuh"

namespace {

constexpr int BM = 128, BN = 128, NARROW = 64;
constexpr int PLANE_BYTES = 8192;                    // one operand slot of one stage: 128 rows of 64 bytes

// Operand forms.  SPLIT: fp32 hi, bf16 of hi and lo, k-blocks of 16 (the split buffers of the C ABI).  PACKED: two fp16
// parts of the scaled value, k-blocks of 32 in the same bytes.
enum Form { SPLIT = 0, PACKED = 1 };
template <int FORM> struct FormCfg {
    static constexpr int BK = FORM == PACKED ? 32 : 16;
    static constexpr int MAPS = FORM == PACKED ? 4 : 8;
};
// tensor maps of A, then of B.  SPLIT: hi_re, hi_im, h16, l16 each; PACKED: high parts, low parts (both planes a map).
template <int FORM> struct OperandMaps { CUtensorMap m[FormCfg<FORM>::MAPS]; };
// One CTA per tile: 8 slots (A: 4, B: 4) = 64 KB per stage, 3 stages.  A pair of CTAs per 256-row tile
// (cta_group::2): each CTA stages its own 128 rows of A (4 slots) and one of the two halves of the stacked B
// operand (B_re rows in the first CTA, B_im rows in the second: 2 slots) = 48 KB per stage, 4 stages.
// A narrow tile of 128 x 64 (PACKED, one CTA): half the slots for B, as in a pair.
template <bool PAIR, int TN> struct Cfg {
    static constexpr int STAGES = PAIR || TN == NARROW ? 4 : 3;
    static constexpr int STAGE_BYTES = (PAIR || TN == NARROW ? 6 : 8) * PLANE_BYTES;
    static constexpr int TILE_M = PAIR ? 2 * BM : BM;
};
constexpr int OPERAND_BYTES = 3 * 8 * PLANE_BYTES;   // 192 KB of operand stages in both forms
constexpr int EPI_GROUPS = 2, EPI_THREADS = 128 * EPI_GROUPS;
// What becomes of the accumulators: written out (NONE), or taken into running sums in registers, each while the other is still
// multiplied (OVERLAP) or both together (EXACT).
enum Drain { NONE = 0, OVERLAP = 1, EXACT = 2 };
// Threads: running sums, three warpgroups (two warps of the first have nothing to do), with this many registers a thread of the
// first and of the epilogue's two out of what all are launched with; else the two warps and the epilogue.
template <int DRAIN> struct Threads { static constexpr int FIRST_EPI = DRAIN ? 128 : 64, ALL = FIRST_EPI + EPI_THREADS; };
constexpr int LAUNCH_REGS = 168, ISSUE_REGS = 56, EPI_REGS = 224;
static_assert(128 * ISSUE_REGS + EPI_THREADS * EPI_REGS <= Threads<true>::ALL * LAUNCH_REGS, "registers");
constexpr int EPI_BYTES = EPI_GROUPS * 2 * 128 * 16 * 4;  // 32 KB: one epilogue round of both groups, re and im staging
constexpr int SMEM_BYTES = OPERAND_BYTES + EPI_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
template <bool PAIR, int TN> constexpr bool fills = Cfg<PAIR, TN>::STAGES * Cfg<PAIR, TN>::STAGE_BYTES == OPERAND_BYTES;
static_assert(fills<false, BN> && fills<true, BN> && fills<false, NARROW>, "stages");
constexpr uint32_t TMEM_COLS = 512;
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

struct TcParams {
    float* d_re; float* d_im;
    const float* r_re; const float* r_im;
    int M, N, K, conjB, accumulate;
    int units_per_cta;        // consecutive (tile, k-block) work units per CTA (stream-K)
    int a_mn, b_mn;           // operand stored [K, rows] (MN-major) instead of [rows, K] (K-major)
    int cluster;              // > 1: that many CTAs of one cluster share a tile, each a slice of K
    int whole_per_cta;        // > 0: every CTA first takes that many whole tiles, then its run of the remaining units
    int segments;             // > 0: CTA r takes k-segment r / tiles of tile r % tiles (units_per_cta k-blocks each)
    int chain, first;         // PACKED: k-blocks that are summed in tensor memory at most; the same of a tile's first ones
    const int* a_exp;         // PACKED: the powers of two that A and B were scaled by, or kPlain
    const int* b_exp;
    const void* a_planes; const void* b_planes;       // PACKED: what the tensor maps describe, for the FMA form
    size_t a_np, b_np;
    int a_pitch, b_pitch;
    int* status;
    // The pair form (cgemm_tc_k<true>): cluster = K slices per tile, each slice a CTA pair (cluster of 2 * cluster CTAs).
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait: false (and the error word set) if the phase did not complete in WAIT_LIMIT_NS
// or another role already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                          int code) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > WAIT_LIMIT_NS) {
            *abort_flag = 1;
            atomicCAS(status, 0, code);
            atomicExch(status + 1, (int) blockIdx.x);
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// The pair form's loads: the data goes to this CTA's shared memory, the completion bytes to the barrier `bar`,
// a shared::cluster address that may lie in the peer CTA (the pair's first CTA collects both halves).
__device__ __forceinline__ void tma2_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma2_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma2_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// shared::cluster address of `local_addr` (a shared::cta address of this CTA's layout) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local_addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    return remote;
}

// Hands a CTA's accumulators back to the pair's first CTA.  What the arrival orders are tensor-memory loads, which the
// tcgen05 fence in front of it has ordered; release at cluster scope would also wait for every store of the thread before
// it (1.4 us of idle MMAs after each chain and each tile).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// MN-major operand tile (source stored [K, rows]): slabs of 32 rows-of-the-operand, each slab
// 16 k-lines of 128 B.  The only layout the tensor core accepts for MN-major TF32 is the 128-byte
// swizzle with 32-byte atomicity: atoms of 4 k-lines (512 B).  Leading byte offset = distance
// between slabs (2 KB), stride byte offset = distance between 4-line k atoms (512 B).
__device__ __forceinline__ uint64_t smem_desc_mn128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t) ((addr >> 4) & 0x3FFF);
    d |= (uint64_t) (2048 >> 4) << 16;
    d |= (uint64_t) (512 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 1 << 61;                          // layout type: 128-byte swizzle, 32-byte base
    return d;
}

// K-major operand tile, 64-byte swizzle: rows of 64 B, 8-row groups 512 B apart.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t) ((addr >> 4) & 0x3FFF);           // start address, 16-byte units
    d |= (uint64_t) 1 << 16;                          // leading byte offset (unused with swizzle): 1
    d |= (uint64_t) (512 >> 4) << 32;                 // stride byte offset between 8-row groups
    d |= (uint64_t) 1 << 46;                          // descriptor version of sm_100
    d |= (uint64_t) 4 << 61;                          // layout type: 64-byte swizzle
    return d;
}

// bf16 K-major operand tile, 32-byte swizzle: rows of 32 B (16 bf16 = one MMA's depth), 8-row groups 256 B apart.
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t) ((addr >> 4) & 0x3FFF);
    d |= (uint64_t) 1 << 16;
    d |= (uint64_t) (256 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 6 << 61;                          // layout type: 32-byte swizzle
    return d;
}

// bf16 MN-major operand tile (source stored [K, rows]): slabs of 64 rows-of-the-operand (128 B), each slab 16
// k-lines; plain 128-byte swizzle, atoms of 8 k-lines (1 KB).  Leading byte offset = slab to slab (2 KB),
// stride byte offset = k atom to k atom (1 KB).
__device__ __forceinline__ uint64_t smem_desc_mn128_b16(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t) ((addr >> 4) & 0x3FFF);
    d |= (uint64_t) (2048 >> 4) << 16;
    d |= (uint64_t) (1024 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 2 << 61;                          // layout type: 128-byte swizzle
    return d;
}

// fp16 MN-major operand tile with 32 k-lines a slab: as above, slabs 4 KB apart.
__device__ __forceinline__ uint64_t smem_desc_mn128_h(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t) ((addr >> 4) & 0x3FFF);
    d |= (uint64_t) (4096 >> 4) << 16;
    d |= (uint64_t) (1024 >> 4) << 32;
    d |= (uint64_t) 1 << 46;
    d |= (uint64_t) 2 << 61;                          // layout type: 128-byte swizzle
    return d;
}

// kind::f16 with fp16 operands, fp32 accumulate, M = 128, N = both planes of a tile's TN columns
template <int TN> constexpr uint32_t kInstrDescH = (1u << 4) | (((2u * TN) >> 3) << 17) | ((128u >> 4) << 24);

// kind::f16 with bf16 operands, fp32 accumulate, M = 128, N = 256
constexpr uint32_t kInstrDesc16 = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// kind::tf32, fp32 accumulate, A and B K-major, M = 128, N = 256
constexpr uint32_t kInstrDesc = (1u << 4) | (2u << 7) | (2u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// The pair form: one MMA of the pair's first CTA multiplies the 256 rows of A held by both CTAs (128 each, at the
// same shared-memory offsets) with the B operand whose two 128-row halves the two CTAs hold; each CTA's tensor
// memory receives the accumulator rows of its own A.
__device__ __forceinline__ void umma2_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void umma2_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// arrives on the barrier at this shared-memory offset in both CTAs of the pair once the MMAs issued so far are done
// (the pair = cluster ranks first_rank and first_rank + 1)
__device__ __forceinline__ void umma2_commit_both(uint32_t bar, uint32_t first_rank) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short) (3u << first_rank)) : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Packed operands: a matrix that is stored as fp32 planes instead of fp16 parts has this for its exponent.
constexpr int kPlain = 1 << 20;

struct PackedElement {
    const void* planes;
    size_t np;
    int pitch, exponent;
    bool k_fast;                             // stored [rows, K]
    __device__ __forceinline__ float2 operator()(int row, int k) const {
        const size_t o = k_fast ? (size_t) row * pitch + k : (size_t) k * pitch + row;
        if (exponent == kPlain) {
            const float* f = static_cast<const float*>(planes) + o;
            return make_float2(f[0], f[np]);
        }
        const __half* h = static_cast<const __half*>(planes) + o;
        const float unscale = __uint_as_float((unsigned) (127 - exponent) << 23);
        return make_float2((__half2float(h[0]) + __half2float(h[2 * np])) * unscale, (__half2float(h[np]) + __half2float(h[3 * np])) * unscale);
    }
};

// The product where an operand is plain: fp32 FMAs by the epilogue's threads, the CTAs of the launch taking 64 x 64 tiles
// in turn whatever the schedule, after the tile product of the same bytes (which meant nothing) has run without a store.
// Nothing waits for the exponents that way where no operand is plain.  1.7 ms at 4096 x 1024 x 1024
// (80 us as a tile product), 0.24 ms at 512 rows (17 us).
__device__ __noinline__ void fma_product(const TcParams& p, void* smem) {
    const PackedElement a = {p.a_planes, p.a_np, p.a_pitch, *p.a_exp, !p.a_mn}, b = {p.b_planes, p.b_np, p.b_pitch, *p.b_exp, !p.b_mn};
    const cnb_fma::Result r = {p.d_re, p.d_im, p.r_re, p.r_im, p.M, p.N, p.K, p.conjB, p.accumulate};
    const int tiles_n = (p.N + cnb_fma::TN - 1) / cnb_fma::TN, tiles = (p.M + cnb_fma::TM - 1) / cnb_fma::TM * tiles_n;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        cnb_fma::tile(a, b, r, *static_cast<cnb_fma::Slabs*>(smem), t / tiles_n * cnb_fma::TM, t % tiles_n * cnb_fma::TN,
                      (int) threadIdx.x - ((int) blockDim.x - EPI_THREADS),
                      [] { asm volatile("bar.sync %0, %1;" ::"n"(1 + EPI_GROUPS), "n"(EPI_THREADS) : "memory"); });
}

// One accumulator of a chain (this thread's row, the half of the tile's columns of its group from `tl` on) into the running sums, rounded
// to nearest: acc1 holds A_re.[B_re ; B_im], acc2 A_im.[B_re ; B_im].  The last load has completed on return.
template <int ACC, int TN> __device__ __forceinline__ void drain_chain(uint32_t tl, float sgn, float (&sr)[TN / 2], float (&si)[TN / 2]) {
#pragma unroll
    for (int c = 0; c < TN / 2; c += 16) {
        float x[16], y[16];
        tmem_ld16(tl + ACC * 256 + c, x);                // . B_re
        tmem_ld16(tl + ACC * 256 + TN + c, y);           // . B_im
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (ACC == 0) { sr[c + i] += x[i]; si[c + i] -= sgn * y[i]; }
            else { si[c + i] += x[i]; sr[c + i] += sgn * y[i]; }
        }
    }
}

// Both accumulators together: their difference is rounded at the chain's magnitude, and only the sum at the running sums'.
template <int TN> __device__ __forceinline__ void drain_exact(uint32_t tl, float sgn, float (&sr)[TN / 2], float (&si)[TN / 2]) {
#pragma unroll
    for (int c = 0; c < TN / 2; c += 8) {
        float a[8], f[8], b[8], e[8];
        tmem_ld8(tl + c, a);                             // A_re.B_re
        tmem_ld8(tl + 256 + TN + c, f);                  // A_im.B_im
        tmem_ld8(tl + TN + c, b);                        // A_re.B_im
        tmem_ld8(tl + 256 + c, e);                       // A_im.B_re
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            sr[c + i] += a[i] + sgn * f[i];
            si[c + i] += e[i] - sgn * b[i];
        }
    }
}

// the four warps of one epilogue group
__device__ __forceinline__ void epi_bar_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }
// One decision for the group.  The flag may be set at any time by the producer, the MMA thread or the other group, so threads
// that each looked at it after the barrier could part ways, some to the role's end and some to the group's next barrier.
__device__ __forceinline__ bool epi_gave_up(int group, volatile int* abort_flag) { return cnb_group_any(1 + group, 128, *abort_flag != 0); }

// Shared memory by its 32-bit address: through a generic pointer the compiler keeps every load behind the global store
// before it, which made a round trip of each 16 bytes written out.
__device__ __forceinline__ void st_shared4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ float4 ld_shared4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float ld_shared1(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// Staging tile of one epilogue round: 128 rows x 16 floats per plane, 16-byte chunks XOR-swizzled by the row so that
// both the row-per-thread writes and the row-segment reads are conflict-free.  In bytes.
__device__ __forceinline__ uint32_t stage_off(int row, int chunk) {
    return (uint32_t) (row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4));
}
constexpr uint32_t STAGE_PLANE = 128 * 16 * 4;

// Partial tile of one CTA in cluster mode: 128 rows x TN floats per plane over the (then idle) operand
// stages, 16-byte chunks XOR-swizzled by the row like the staging tile.
template <int TN> __device__ __forceinline__ int part_off(int row, int chunk) { return row * TN + ((chunk ^ (row & 7)) << 2); }
template <int TN> constexpr int PART_PLANE_BYTES = 128 * TN * 4;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Brings `bytes` (a multiple of 16, 16-byte aligned) of global memory into L2 through the bulk-copy engine.
// The epilogue reads residual / old-D tiles 128 bytes per row and round; fetched like that from DRAM each
// row segment costs four scattered accesses, fetched here as one 512-byte piece per row, while the tile's
// MMAs run, the later reads hit L2.
__device__ __forceinline__ void l2_prefetch(const float* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

template <int TN>
__device__ __forceinline__ void prefetch_tile_rows(const TcParams& p, const float* re, const float* im, int row,
                                                  int n0) {
    if (row >= p.M || (p.N & 3)) return;
    const uint32_t bytes = (uint32_t) min(TN, p.N - n0) * 4u;
    const size_t o = (size_t) row * p.N + n0;
    if (((reinterpret_cast<uintptr_t>(re + o) | reinterpret_cast<uintptr_t>(im + o)) & 15) != 0) return;
    l2_prefetch(re + o, bytes);
    l2_prefetch(im + o, bytes);
}

// A 16-byte global load that stays where it is written (volatile asm keeps its place among the other
// volatile asms: the tensor-memory loads and barriers), so a batch of them is in flight together.
__device__ __forceinline__ float4 ld_global_now(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float ld_global_now1(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Four consecutive floats of a row of which `left` (>= 1) remain: one 16-byte access, or (VEC = false: rows at any
// 4-byte alignment, ragged ends) up to four single ones.
template <bool VEC> __device__ __forceinline__ float4 ld_global_part(const float* p, int left) {
    if constexpr (VEC) return ld_global_now(p);
    float4 v = make_float4(ld_global_now1(p), 0.f, 0.f, 0.f);
    if (left > 1) v.y = ld_global_now1(p + 1);
    if (left > 2) v.z = ld_global_now1(p + 2);
    if (left > 3) v.w = ld_global_now1(p + 3);
    return v;
}

template <bool VEC> __device__ __forceinline__ void st_global_part(float* p, int left, float4 v) {
    if constexpr (VEC) { *reinterpret_cast<float4*>(p) = v; return; }
    p[0] = v.x;
    if (left > 1) p[1] = v.y;
    if (left > 2) p[2] = v.z;
    if (left > 3) p[3] = v.w;
}

// all threads of all CTAs of the cluster; orders shared-memory writes before the peers' reads
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ float4 ld_peer(uint32_t local_addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    float4 v;   // volatile keeps it between the two cluster barriers; no memory clobber, so loads can be in flight together
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote));
    return v;
}

// Cluster mode, after the first cluster barrier: this CTA sums its band of rows of the tile over the CL
// partial tiles (its own and its peers', through distributed shared memory), adds residual / old D and
// stores.  Two 16-byte chunks per thread and round: every load of both (2 * CL peer loads per plane pair,
// residual, old D) is issued before the first sum, so a round costs one round trip.  Fixed summation order.
// The CL partial tiles sit in the CTAs of cluster rank peer0 + c * peer_step (one CTA per tile: 0 and 1; CTA pairs:
// this CTA's rank in its pair and 2: the peers are the CTAs that hold the same 128 rows).
template <int CL, bool VEC, int TN>
__device__ __forceinline__ void cluster_reduce(const TcParams& p, uint32_t smem_base, uint32_t crank, int m0, int n0,
                                               int et, uint32_t peer0, uint32_t peer_step) {
    constexpr int ROWS = BM / CL, LINE = TN / 4;         // chunks in a row
    constexpr int U = CL <= 4 ? 2 : 1;                   // chunks per thread and round
    for (int base = et; base < ROWS * LINE; base += EPI_THREADS * U) {
        float4 xr[U][CL], xi[U][CL], vr[U], vi[U];
        size_t o[U];
        bool live[U];
        int gn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = base + EPI_THREADS * u;
            const int r = (int) crank * ROWS + idx / LINE, ch = idx % LINE;
            const int gm = m0 + r;
            gn[u] = n0 + ch * 4;
            live[u] = idx < ROWS * LINE && gm < p.M && gn[u] < p.N;
            o[u] = (size_t) gm * p.N + gn[u];
            vr[u] = make_float4(0.f, 0.f, 0.f, 0.f); vi[u] = vr[u];
            if (!live[u]) continue;
            const uint32_t local = smem_base + 4u * (uint32_t) part_off<TN>(r, ch);
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                const uint32_t peer = peer0 + (uint32_t) c * peer_step;
                xr[u][c] = ld_peer(local, peer); xi[u][c] = ld_peer(local + PART_PLANE_BYTES<TN>, peer);
            }
            if (p.r_re) { vr[u] = ld_global_part<VEC>(p.r_re + o[u], p.N - gn[u]); vi[u] = ld_global_part<VEC>(p.r_im + o[u], p.N - gn[u]); }
            if (p.accumulate) {
                const float4 dr = ld_global_part<VEC>(p.d_re + o[u], p.N - gn[u]), di = ld_global_part<VEC>(p.d_im + o[u], p.N - gn[u]);
                vr[u].x += dr.x; vr[u].y += dr.y; vr[u].z += dr.z; vr[u].w += dr.w;
                vi[u].x += di.x; vi[u].y += di.y; vi[u].z += di.z; vi[u].w += di.w;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!live[u]) continue;
            float4 sr = make_float4(0.f, 0.f, 0.f, 0.f), si = sr;
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                sr.x += xr[u][c].x; sr.y += xr[u][c].y; sr.z += xr[u][c].z; sr.w += xr[u][c].w;
                si.x += xi[u][c].x; si.y += xi[u][c].y; si.z += xi[u][c].z; si.w += xi[u][c].w;
            }
            vr[u].x += sr.x; vr[u].y += sr.y; vr[u].z += sr.z; vr[u].w += sr.w;
            vi[u].x += si.x; vi[u].y += si.y; vi[u].z += si.z; vi[u].w += si.w;
            st_global_part<VEC>(p.d_re + o[u], p.N - gn[u], vr[u]);
            st_global_part<VEC>(p.d_im + o[u], p.N - gn[u], vi[u]);
        }
    }
}

// Phase stamps of CTA 0 (a build with -DCNB_GEMM_TIMING only; read back from the status block): %globaltimer ns.
#ifdef CNB_GEMM_TIMING
#define CNB_GSTAMP(k, cond)                                                                        \
    do { if (blockIdx.x == 0 && (cond)) p.status[900 + (k)] = (int) global_ns(); } while (0)
#else
#define CNB_GSTAMP(k, cond) do { } while (0)
#endif

// VEC: rows of D and R are 16-byte aligned (N % 4 == 0); the form without it writes 32 consecutive floats of a row per
// warp instruction instead of four 16-byte pieces of four rows.
// DRAIN: a run of more than p.chain k-blocks is cut into chains of that many; after each the epilogue takes the
// accumulators into running sums in registers (max_chain says why).
// OVERLAP: one while the other is still multiplied, so that the MMAs hardly wait.  Where a CTA goes through several tiles (one
// leaves tensor memory in 0.3 us and is written out under the next one's MMAs: 4096 x 1024 x 1024 74.4 -> 69.8 us), and where
// chains are long or many (chain_blocks).
// EXACT: both together, so that a chain costs one rounding at the magnitude of the running sums and not two.  For the few or short
// chains of sizes that are to be no further off than fp32 FMAs: 466 x 2805, K = 97, four chains of one block, 1.14e-7 off
// float64 and 1.19e-7 as OVERLAP.
// Launches of one chain and one tile a CTA (NONE) leave registers of the SM to the kernels around them, and their set-up
// runs under the tail of the kernel before (512-row training step 772 -> 743 us).
// TN: columns of a tile, BN or NARROW (choose_schedule).
template <bool PAIR, bool VEC, int FORM, int DRAIN, int TN>
__global__ void __launch_bounds__(Threads<DRAIN>::ALL, 1)
cgemm_tc_k(const __grid_constant__ OperandMaps<FORM> om, const __grid_constant__ TcParams p) {
    static_assert(TN == BN || (TN == NARROW && !PAIR && FORM == PACKED && DRAIN != OVERLAP), "narrow tiles");
    extern __shared__ uint8_t smem_raw[];
    constexpr int BK = FormCfg<FORM>::BK;
    CNB_GSTAMP(0, threadIdx.x == 0);
    // operand stages need the alignment of their swizzle pattern; 1024 B covers every mode
    constexpr int STAGES = Cfg<PAIR, TN>::STAGES, STAGE_BYTES = Cfg<PAIR, TN>::STAGE_BYTES, TILE_M = Cfg<PAIR, TN>::TILE_M;
    constexpr int B_LOW = STAGE_BYTES / PLANE_BYTES == 8 ? 6 : 5;          // PACKED: slot of B's low parts
    constexpr int HALF = TN / 2;                         // columns of an epilogue group
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OPERAND_BYTES + EPI_BYTES);
    // bars[0..S) full, bars[S..2S) empty, bars[2S] accumulators ready, bars[2S+1] accumulators drained; OVERLAP: these two
    // of acc1, bars[2S+2] and bars[2S+3] of acc2
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (p.N + TN - 1) / TN;
    const int tiles_m = (p.M + TILE_M - 1) / TILE_M;
    const int k_blocks = (p.K + BK - 1) / BK;
    const long total_units = (long) tiles_m * tiles_n * k_blocks;
    // In the pair form the two CTAs of a cluster work through the same units (each on its own 128 rows of the
    // 256-row tile): "CTA" below is the pair.
    // Cluster ranks: one CTA per tile: rank = K slice (cluster split-K) or none; pairs: rank = 2 * K slice + place in
    // the pair.
    const uint32_t rank_all = (PAIR || p.cluster > 1) ? cluster_rank() : 0u;
    const uint32_t prank = PAIR ? (rank_all & 1u) : 0u;
    const uint32_t lead_rank = rank_all & ~1u;           // pairs: the pair's first CTA
    const long cta_idx = PAIR ? (long) (blockIdx.x >> 1) : (long) blockIdx.x;
    const long cta_cnt = PAIR ? (long) (gridDim.x >> 1) : (long) gridDim.x;
    const int row_off = PAIR ? (int) prank * BM : 0;
    // Whole tiles first, every cta_cnt-th (so that the CTAs work on neighbours at any time), then one run of (tile, k-block)
    // units of those that are left.
    const long left = (long) p.whole_per_cta * cta_cnt * k_blocks;
    long u_begin = min(total_units, left + cta_idx * p.units_per_cta);
    long u_end = min(total_units, u_begin + p.units_per_cta);
    if (p.segments > 0) {
        // Capped chains (K > 4096): consecutive CTAs take the SAME k-segment of consecutive tiles, so the CTAs that
        // run together read the same columns of A and B and share them through L2 (tile-major runs had every CTA
        // of a wave on its own k-range: 5.0 GB of DRAM reads for 0.8 GB of operands at 1024 x 2048 x 16384).
        const long tiles = (long) tiles_m * tiles_n;
        const long seg = cta_idx / tiles, tile = cta_idx % tiles;
        u_begin = tile * k_blocks + seg * p.units_per_cta;
        u_end = min(u_begin + p.units_per_cta, (tile + 1) * k_blocks);
        if (u_begin > u_end) u_begin = u_end;
    }
    const bool split_cluster = p.cluster > 1;
    const uint32_t crank = split_cluster ? (PAIR ? rank_all >> 1 : rank_all) : 0;     // the K slice
    const int cluster_ctas = p.cluster * (PAIR ? 2 : 1);
    if (split_cluster) {                                 // one tile per cluster, an even slice of its k-blocks per CTA (pair)
        const long tile = blockIdx.x / cluster_ctas;
        u_begin = tile * k_blocks + (long) k_blocks * crank / p.cluster;
        u_end = tile * k_blocks + (long) k_blocks * (crank + 1) / p.cluster;
    }
    auto run_begin = [&](int r) { return r < p.whole_per_cta ? min(total_units, (cta_idx + r * cta_cnt) * k_blocks) : u_begin; };
    auto run_end = [&](int r) { return r < p.whole_per_cta ? min(total_units, (cta_idx + r * cta_cnt + 1) * k_blocks) : u_end; };
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    const uint32_t acc_full = bar_base + 8u * (2 * STAGES);
    const uint32_t acc_empty = bar_base + 8u * (2 * STAGES + 1);
    const uint32_t acc2_full = bar_base + 8u * (2 * STAGES + 2), acc2_empty = bar_base + 8u * (2 * STAGES + 3);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        mbar_init(acc_full, 1);
        mbar_init(acc2_full, 1);
        // every epilogue group, or (DRAIN) every one of their warps, hands the accumulators back; pair: of both CTAs
        const uint32_t hands = (PAIR ? 2 : 1) * (DRAIN ? EPI_THREADS / 32 : EPI_GROUPS);
        mbar_init(acc_empty, hands);
        mbar_init(acc2_empty, hands);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {   // whole warp: allocate all 512 tensor-memory columns (1 CTA per SM by shared-memory size)
        if constexpr (PAIR) {                            // the same warp of both CTAs of the pair
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    if (warp == 0 && lane < FormCfg<FORM>::MAPS)   // descriptor fetch of the operand maps, off the first TMA's critical path
        asm volatile("prefetch.tensormap [%0];" ::"l"(&om.m[lane]) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) cluster_sync();                  // the peer's barriers exist before anything signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // Everything above touched no memory another kernel writes: under programmatic dependent launch it ran
    // while the kernel before this one in the stream was finishing.  Operands, residual and old D are read
    // (and D written) only after that kernel has completed.
    cnb_pdl_trigger();
    cnb_pdl_wait();
    CNB_GSTAMP(1, threadIdx.x == 0);
    // Where the roles end, each in its own branch: behind a common end the registers of the smaller share would hold for
    // both.  Every thread of every CTA reaches these barriers, also after a bounded wait gave up.  A pair's CTA neither
    // leaves nor frees tensor memory while the other may still signal its barriers, read its shared memory (the first CTA's
    // MMAs read the peer's operand stages) or write its tensor memory; with a K split all partial tiles are in shared memory.
    auto finish = [&] {
        __syncwarp();
        asm volatile("barrier.cta.sync.aligned 0;" ::: "memory");
        if (PAIR || split_cluster) cluster_sync();
    };

    // DRAIN: the epilogue's running sums want more registers than an equal share.  The shares change once: a group that took
    // its own back could do so before the others have theirs.
    constexpr int EPI_WARP = Threads<DRAIN>::FIRST_EPI / 32;
    if (warp < EPI_WARP) {
    if (DRAIN) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ISSUE_REGS));
    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            long it = 0;
            bool live = true;
            for (int r = 0; r <= p.whole_per_cta && live; ++r)
            for (long u = run_begin(r), ue = run_end(r); u < ue; ++u, ++it) {
                int tile = (int) (u / k_blocks), kb = (int) (u % k_blocks);
                int m0 = (tile / tiles_n) * TILE_M + row_off, n0 = (tile % tiles_n) * TN;
                int s = (int) (it % STAGES);
                uint32_t phase = (uint32_t) (it / STAGES) & 1;
                if (!mbar_wait(empty_bar(s), phase ^ 1, abort_flag, p.status, 1)) { live = false; break; }
                uint32_t dst = smem_base + s * STAGE_BYTES;
                if constexpr (FORM == PACKED) {
                    // slots 0..3: A high re, im, low re, im; then B: all four, or (pair) this CTA's plane of high and low
                    const uint32_t bar = PAIR ? map_to_rank(full_bar(s), lead_rank) : full_bar(s);
                    if (prank == 0) mbar_expect_tx(full_bar(s), (PAIR ? 2 : 1) * STAGE_BYTES);
                    auto load = [&](uint32_t to, const CUtensorMap* m, bool mn, int r0, int plane) {
                        if (mn) {
                            if constexpr (PAIR) tma2_load_4d(to, m, bar, 0, kb * BK, r0 / 64, plane);
                            else tma_load_4d(to, m, bar, 0, kb * BK, r0 / 64, plane);
                        } else {
                            if constexpr (PAIR) tma2_load_3d(to, m, bar, kb * BK, r0, plane);
                            else tma_load_3d(to, m, bar, kb * BK, r0, plane);
                        }
                    };
                    load(dst, &om.m[0], p.a_mn, m0, 0);
                    load(dst + 2 * PLANE_BYTES, &om.m[1], p.a_mn, m0, 0);
                    load(dst + 4 * PLANE_BYTES, &om.m[2], p.b_mn, n0, PAIR ? (int) prank : 0);
                    load(dst + B_LOW * PLANE_BYTES, &om.m[3], p.b_mn, n0, PAIR ? (int) prank : 0);
                    continue;
                } else {
                const CUtensorMap* maps = om.m;
                if constexpr (PAIR) {
                    // Both CTAs fill their own stage; all completion bytes go to the full barrier of the pair's
                    // first CTA, which expects the bytes of both.
                    const uint32_t bar = map_to_rank(full_bar(s), lead_rank);
                    if (prank == 0) mbar_expect_tx(full_bar(s), 2 * STAGE_BYTES);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {        // this CTA's 128 rows of A: hi_re, hi_im, h16 pair, l16 pair
                        if (q < 2) {
                            if (p.a_mn) tma2_load_3d(dst + q * PLANE_BYTES, maps + q, bar, 0, kb * BK, m0 / 32);
                            else tma2_load_2d(dst + q * PLANE_BYTES, maps + q, bar, kb * BK, m0);
                        } else {
                            if (p.a_mn) tma2_load_4d(dst + q * PLANE_BYTES, maps + q, bar, 0, kb * BK, m0 / 64, 0);
                            else tma2_load_3d(dst + q * PLANE_BYTES, maps + q, bar, kb * BK, m0, 0);
                        }
                    }
                    // this CTA's half of the stacked B operand: the real planes (first CTA) or the imaginary ones
                    const int c = (int) prank;
                    uint32_t db = dst + 4 * PLANE_BYTES;
                    if (p.b_mn) tma2_load_3d(db, maps + 4 + c, bar, 0, kb * BK, n0 / 32);
                    else tma2_load_2d(db, maps + 4 + c, bar, kb * BK, n0);
                    db += PLANE_BYTES;
                    for (int q = 6; q < 8; ++q, db += PLANE_BYTES / 2) {      // h16, l16: boxes of one plane
                        if (p.b_mn) tma2_load_4d(db, maps + q, bar, 0, kb * BK, n0 / 64, c);
                        else tma2_load_3d(db, maps + q, bar, kb * BK, n0, c);
                    }
                    continue;
                }
                mbar_expect_tx(full_bar(s), STAGE_BYTES);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int r0 = q < 4 ? m0 : n0;
                    const bool mn = q < 4 ? p.a_mn : p.b_mn;
                    if ((q & 3) < 2) {                   // an fp32 hi plane
                        if (mn) tma_load_3d(dst + q * PLANE_BYTES, maps + q, full_bar(s), 0, kb * BK, r0 / 32);
                        else tma_load_2d(dst + q * PLANE_BYTES, maps + q, full_bar(s), kb * BK, r0);
                    } else {                             // a pair of bf16 planes [re ; im]
                        if (mn) tma_load_4d(dst + q * PLANE_BYTES, maps + q, full_bar(s), 0, kb * BK, r0 / 64, 0);
                        else tma_load_3d(dst + q * PLANE_BYTES, maps + q, full_bar(s), kb * BK, r0, 0);
                    }
                }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (pair: its first CTA only)
        if (lane == 0 && prank == 0) {
            bool ok = true;
            long it = 0;
            int seg = 0;
            // bits 15 / 16 of the instruction descriptor: operand A / B is MN-major
            const uint32_t mn_bits = (p.a_mn ? (1u << 15) : 0u) | (p.b_mn ? (1u << 16) : 0u);
            // pair: M = 256 over the two CTAs
            const uint32_t m_bits = PAIR ? ((256u >> 4) << 24) - ((128u >> 4) << 24) : 0u;
            const uint32_t idesc = (kInstrDesc | mn_bits) + m_bits, idesc16 = (kInstrDesc16 | mn_bits) + m_bits;
            // PACKED: one thread issues an MMA every 140 cycles; a descriptor is one addition to what is known here
            const uint32_t idesch = (kInstrDescH<TN> | mn_bits) + m_bits;
            const uint64_t a_desc = p.a_mn ? smem_desc_mn128_h(0) : smem_desc_sw64(0), b_desc = p.b_mn ? smem_desc_mn128_h(0) : smem_desc_sw64(0);
            const uint32_t a_step = (p.a_mn ? 2048 : 32) >> 4, b_step = (p.b_mn ? 2048 : 32) >> 4;
            for (int r = 0; r <= p.whole_per_cta; ++r)
            for (long u = run_begin(r), ue = run_end(r); u < ue && ok; ++seg) {
                int kb0 = (int) (u % k_blocks);
                int kb1 = (int) min((long) k_blocks, kb0 + (ue - u));
                if constexpr (DRAIN) kb1 = min(kb1, kb0 + (kb0 == 0 ? p.first : p.chain));    // every chain is a segment of its own here
                // the epilogue must have drained the previous segment's accumulators
                auto drained = [&](uint32_t bar) {
                    const bool done = mbar_wait(bar, (uint32_t) (seg & 1) ^ 1, abort_flag, p.status, 4);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    return done;
                };
                if constexpr (DRAIN != OVERLAP) { ok = drained(acc_empty); if (!ok) break; }
                for (int kb = kb0; kb < kb1 && ok; ++kb, ++it) {
                    int s = (int) (it % STAGES);
                    uint32_t phase = (uint32_t) (it / STAGES) & 1;
                    ok = mbar_wait(full_bar(s), phase, abort_flag, p.status, 2);
                    if (!ok) break;
                    CNB_GSTAMP(2, it == 0);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t st = smem_base + s * STAGE_BYTES;
                    const uint32_t first = kb == kb0 ? 0u : 1u;
                    if constexpr (FORM == PACKED) {
                        const uint32_t at = (st >> 4) & 0x3FFF;      // (in a cluster the CTA's rank stands above the offset)
                        // term 0: low.high, 1: high.low, 2: high.high
                        auto mma = [&](int j, int acc, int term) {
                            const uint64_t ad = a_desc + (at + (term == 0 ? 2 + acc : acc) * (PLANE_BYTES >> 4) + j * a_step);
                            const uint64_t bd = b_desc + (at + (term == 1 ? B_LOW : 4) * (PLANE_BYTES >> 4) + j * b_step);
                            const uint32_t add = j == 0 && term == 0 ? first : 1u;
                            if constexpr (PAIR) umma2_bf16(tmem_base + 256 * acc, ad, bd, idesch, add);
                            else umma_bf16(tmem_base + 256 * acc, ad, bd, idesch, add);
                        };
                        // OVERLAP: at a chain's ends the accumulators take turns by the block: acc1 is summed up while acc2 of
                        // the chain's last block is multiplied, acc2 while acc1 of the next chain's first block is.
                        // EXACT: the small terms of a block come first, so that in a chain of one block they meet a small
                        // accumulator (K = 50: 1.5e-7 -> 1.1e-7 off float64, FMAs 1.3e-7).
                        const bool last = kb + 1 == kb1;
                        if (DRAIN == OVERLAP && (kb == kb0 || last)) {
#pragma unroll
                            for (int acc = 0; acc < 2; ++acc) {
                                if (kb == kb0 && !drained(acc ? acc2_empty : acc_empty)) { ok = false; break; }
#pragma unroll
                                for (int j = 0; j < BK / 16; ++j) { mma(j, acc, 0); mma(j, acc, 1); mma(j, acc, 2); }
                                if (acc == 1) { if constexpr (PAIR) umma2_commit_both(empty_bar(s), lead_rank); else umma_commit(empty_bar(s)); }
                                if (last) {
                                    const uint32_t bar = acc ? acc2_full : acc_full;
                                    if constexpr (PAIR) umma2_commit_both(bar, lead_rank); else umma_commit(bar);
                                }
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < BK / 16; ++j)
#pragma unroll
                                for (int acc = 0; acc < 2; ++acc) {
                                    mma(j, acc, 0); mma(j, acc, 1);
                                    if (DRAIN != EXACT) mma(j, acc, 2);
                                }
                            if (DRAIN == EXACT) {
#pragma unroll
                                for (int j = 0; j < BK / 16; ++j) { mma(j, 0, 2); mma(j, 1, 2); }
                            }
                            if constexpr (PAIR) umma2_commit_both(empty_bar(s), lead_rank); else umma_commit(empty_bar(s));
                        }
                        continue;
                    } else {
                    if constexpr (PAIR) {
                        // slots: 0 / 1 A hi_re / hi_im, 2 / 3 A h16 / l16 [re ; im], 4 B hi, 5 B h16 then l16
                        auto a16 = [&](int slot, int im) {
                            const uint32_t a = st + slot * PLANE_BYTES + im * (PLANE_BYTES / 2);
                            return p.a_mn ? smem_desc_mn128_b16(a) : smem_desc_sw32(a);
                        };
                        auto b16 = [&](int half) {
                            const uint32_t a = st + 5 * PLANE_BYTES + half * (PLANE_BYTES / 2);
                            return p.b_mn ? smem_desc_mn128_b16(a) : smem_desc_sw32(a);
                        };
                        const uint64_t b_h16 = b16(0), b_l16 = b16(1);
                        umma2_bf16(tmem_base, a16(3, 0), b_h16, idesc16, first);
                        umma2_bf16(tmem_base, a16(2, 0), b_l16, idesc16, 1u);
                        umma2_bf16(tmem_base + 256, a16(3, 1), b_h16, idesc16, first);
                        umma2_bf16(tmem_base + 256, a16(2, 1), b_l16, idesc16, 1u);
#pragma unroll
                        for (int j = 0; j < BK / 8; ++j) {
                            const uint32_t ka = p.a_mn ? j * 1024 : j * 32, kbo = p.b_mn ? j * 1024 : j * 32;
                            auto adesc = [&](int plane) {
                                uint32_t a = st + plane * PLANE_BYTES + ka;
                                return p.a_mn ? smem_desc_mn128(a) : smem_desc_sw64(a);
                            };
                            const uint32_t bb = st + 4 * PLANE_BYTES + kbo;
                            const uint64_t b_h = p.b_mn ? smem_desc_mn128(bb) : smem_desc_sw64(bb);
                            umma2_tf32(tmem_base, adesc(0), b_h, idesc, 1u);
                            umma2_tf32(tmem_base + 256, adesc(1), b_h, idesc, 1u);
                        }
                        umma2_commit_both(empty_bar(s), lead_rank);  // the stage is free in both CTAs once these MMAs have read it
                        continue;
                    }
                    {
                        // the cross terms first (small terms first): one BF16 k-step covers the whole 16-deep block.
                        // A slots 2 / 3 hold [re ; im] of h16 / l16 (4 KB each), B slots 6 / 7 the 256-row operands.
                        auto a16 = [&](int slot, int im) {
                            const uint32_t a = st + slot * PLANE_BYTES + im * (PLANE_BYTES / 2);
                            return p.a_mn ? smem_desc_mn128_b16(a) : smem_desc_sw32(a);
                        };
                        auto b16 = [&](int slot) {
                            const uint32_t a = st + slot * PLANE_BYTES;
                            return p.b_mn ? smem_desc_mn128_b16(a) : smem_desc_sw32(a);
                        };
                        const uint64_t b_h16 = b16(6), b_l16 = b16(7);
                        umma_bf16(tmem_base, a16(3, 0), b_h16, idesc16, first);          // lo(A_re) . hi(B)
                        umma_bf16(tmem_base, a16(2, 0), b_l16, idesc16, 1u);             // hi(A_re) . lo(B)
                        umma_bf16(tmem_base + 256, a16(3, 1), b_h16, idesc16, first);    // lo(A_im) . hi(B)
                        umma_bf16(tmem_base + 256, a16(2, 1), b_l16, idesc16, 1u);       // hi(A_im) . lo(B)
                    }
#pragma unroll
                    for (int j = 0; j < BK / 8; ++j) {
                        // one k-step = 8 TF32: 32 bytes along a K-major swizzled row, or one 1 KB atom of k-lines
                        const uint32_t ka = p.a_mn ? j * 1024 : j * 32, kbo = p.b_mn ? j * 1024 : j * 32;
                        auto adesc = [&](int plane) {
                            uint32_t a = st + plane * PLANE_BYTES + ka;
                            return p.a_mn ? smem_desc_mn128(a) : smem_desc_sw64(a);
                        };
                        const uint32_t bb = st + 4 * PLANE_BYTES + kbo;             // [B_re ; B_im] hi, 256 rows
                        const uint64_t b_h = p.b_mn ? smem_desc_mn128(bb) : smem_desc_sw64(bb);
                        umma_tf32(tmem_base, adesc(0), b_h, idesc, 1u);              // hi(A_re) . hi(B)
                        umma_tf32(tmem_base + 256, adesc(1), b_h, idesc, 1u);        // hi(A_im) . hi(B)
                    }
                    umma_commit(empty_bar(s));       // the stage is free once these MMAs have read it
                    }
                }
                if (ok && DRAIN != OVERLAP) { if constexpr (PAIR) umma2_commit_both(acc_full, lead_rank); else umma_commit(acc_full); }
                CNB_GSTAMP(3, true);
                u += kb1 - kb0;
            }
        }
    }
    finish();
    if (split_cluster) cluster_sync();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    } else {
        // -------------------------------------------------------------------- epilogue
        bool plain = false;
        if (DRAIN) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
        const int q = warp & 3;                      // TMEM lane quarter this warp may read
        const int row = q * 32 + lane;
        const int group = (warp - EPI_WARP) >> 2;           // the half of the columns this warp takes
        const int et = ((warp - EPI_WARP) & 3) * 32 + lane; // 0..127 within the epilogue group
        const uint32_t tl = tmem_base + ((uint32_t) (q * 32) << 16);
        const float sgn = p.conjB ? 1.f : -1.f;
        // PACKED: the scales of both operands are taken out again, in two factors so that neither leaves fp32's range
        float u0 = 1.f, u1 = 1.f;
        if constexpr (FORM == PACKED) {
            const int ea = *p.a_exp, eb = *p.b_exp;
            plain = ea == kPlain || eb == kPlain;
            const int e = -(ea + eb), h = e >> 1;
            u0 = __uint_as_float((uint32_t) (h + 127) << 23);
            u1 = __uint_as_float((uint32_t) (e - h + 127) << 23);
        }
        auto out = [&](float v) { return FORM == PACKED ? v * u0 * u1 : v; };
        const int rows = plain ? 0 : p.M;                // plain: nothing is read of D or R, or stored
        const uint32_t stage = smem_base + OPERAND_BYTES + (uint32_t) group * 2 * STAGE_PLANE;
        int seg = 0;
        // DRAIN: the chains of the k-blocks from `kb` to `end` of a tile into the running sums; false after a wait gave up
        float sr[DRAIN ? HALF : 1], si[DRAIN ? HALF : 1];
        auto sum_chains = [&](int kb, int end) {
            if constexpr (DRAIN) {
#pragma unroll
                for (int i = 0; i < HALF; ++i) sr[i] = si[i] = 0.f;
                for (; kb < end; kb += kb == 0 ? p.first : p.chain, ++seg) {
                    // every warp by itself; after a wait gave up the others end at once
                    auto sum = [&](auto acc, uint32_t full, uint32_t empty) {
                        mbar_wait(full, (uint32_t) seg & 1, abort_flag, p.status, 3);
                        __syncwarp();
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if constexpr (DRAIN == EXACT) drain_exact<TN>(tl + group * HALF, sgn, sr, si);
                        else drain_chain<decltype(acc)::value, TN>(tl + group * HALF, sgn, sr, si);
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            if constexpr (PAIR) mbar_arrive_cluster(map_to_rank(empty, lead_rank));
                            else mbar_arrive(empty);
                        }
                    };
                    sum(std::integral_constant<int, 0>(), acc_full, acc_empty);
                    if constexpr (DRAIN == OVERLAP) sum(std::integral_constant<int, 1>(), acc2_full, acc2_empty);
                }
                if (epi_gave_up(group, abort_flag)) return false;
            }
            return true;
        };
        if (split_cluster) {
            // the whole k-slice is one segment; its partial sums go to shared memory for the cluster reduction
            {
                const int tile = blockIdx.x / cluster_ctas, rows_per = BM / p.cluster;
                const int row = (tile / tiles_n) * TILE_M + row_off + (int) crank * rows_per + et, n0 = (tile % tiles_n) * TN;
                if (group == 0 && et < rows_per) {       // the band of rows this CTA will write out
                    if (p.r_re) prefetch_tile_rows<TN>(p, p.r_re, p.r_im, row, n0);
                    if (p.accumulate) prefetch_tile_rows<TN>(p, p.d_re, p.d_im, row, n0);
                }
            }
            if constexpr (DRAIN) {
                if (sum_chains((int) (u_begin % k_blocks), (int) (u_begin % k_blocks) + (int) (u_end - u_begin))) {           // after the last chain the stages are idle
#pragma unroll
                    for (int i = 0; i < HALF; i += 4) {
                        const uint32_t o = smem_base + 4u * (uint32_t) part_off<TN>(row, (group * HALF + i) >> 2);
                        st_shared4(o, out(sr[i]), out(sr[i + 1]), out(sr[i + 2]), out(sr[i + 3]));
                        st_shared4(o + PART_PLANE_BYTES<TN>, out(si[i]), out(si[i + 1]), out(si[i + 2]), out(si[i + 3]));
                    }
                }
            } else {
            mbar_wait(acc_full, 0u, abort_flag, p.status, 3);
            CNB_GSTAMP(4, et == 0);
            if (!epi_gave_up(group, abort_flag)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = group * HALF; c0 < group * HALF + HALF; c0 += 16) {
                    float a[16], f[16], b[16], e[16];
                    tmem_ld16(tl + c0, a);                   // A_re.B_re
                    tmem_ld16(tl + 256 + TN + c0, f);             // A_im.B_im
                    tmem_ld16(tl + TN + c0, b);             // A_re.B_im
                    tmem_ld16(tl + 256 + c0, e);             // A_im.B_re
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const uint32_t o = smem_base + 4u * (uint32_t) part_off<TN>(row, (c0 + i) >> 2);
                        st_shared4(o, out(a[i] + sgn * f[i]), out(a[i + 1] + sgn * f[i + 1]), out(a[i + 2] + sgn * f[i + 2]),
                                   out(a[i + 3] + sgn * f[i + 3]));
                        st_shared4(o + PART_PLANE_BYTES<TN>, out(e[i] - sgn * b[i]), out(e[i + 1] - sgn * b[i + 1]),
                                   out(e[i + 2] - sgn * b[i + 2]), out(e[i + 3] - sgn * b[i + 3]));
                    }
                }
            }
            }
            CNB_GSTAMP(5, et == 0);
            u_end = u_begin;                             // nothing left for the loop below
        }
        bool live = true;
        for (int r = 0; r <= p.whole_per_cta && live; ++r)
        for (long u = run_begin(r), ue = run_end(r); u < ue; seg += DRAIN ? 0 : 1) {
            int tile = (int) (u / k_blocks), kb0 = (int) (u % k_blocks);
            int kb1 = (int) min((long) k_blocks, kb0 + (ue - u));
            int m0 = (tile / tiles_n) * TILE_M + row_off, n0 = (tile % tiles_n) * TN;
            const bool partial = !(kb0 == 0 && kb1 == k_blocks);   // split tiles are summed with atomics
            const bool add_res = p.r_re != nullptr && kb0 == 0;
            const bool need_old = !partial && p.accumulate;
            const bool pre = VEC && (add_res || need_old);
            // one row of the tile per epilogue thread, requested before the wait for the MMAs
            if (group == 0) {
                if (add_res) prefetch_tile_rows<TN>(p, p.r_re, p.r_im, m0 + et, n0);
                if (need_old) prefetch_tile_rows<TN>(p, p.d_re, p.d_im, m0 + et, n0);
            }
            // What a round adds from global memory (the residual if there is one, else old D) is requested a round
            // ahead, the first one's under the MMAs: asked for in the round itself it doubled the round's time, and
            // asked for between the stores each load would wait for the store before it.
            constexpr int U = 4;
            float4 gr[U], gi[U];
            auto request = [&](int c0, int h) {
                const float* xr = add_res ? p.r_re : p.d_re;
                const float* xi = add_res ? p.r_im : p.d_im;
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const int idx = et + 128 * (h + j);
                    const int gm = m0 + (idx >> 2), gn = n0 + c0 + (idx & 3) * 4;
                    gr[j] = make_float4(0.f, 0.f, 0.f, 0.f); gi[j] = gr[j];
                    if (gm >= rows || gn >= p.N) continue;
                    const size_t o = (size_t) gm * p.N + gn;
                    gr[j] = ld_global_now(xr + o);
                    gi[j] = ld_global_now(xi + o);
                }
            };
            const int c_first = group * HALF, c_last = c_first + HALF - 16;
            if (pre) request(c_first, 0);
            if constexpr (DRAIN) {
                if (!sum_chains(kb0, kb1)) { live = false; break; }
            } else {
                mbar_wait(acc_full, (uint32_t) seg & 1, abort_flag, p.status, 3);
                if (epi_gave_up(group, abort_flag)) { live = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
#pragma unroll(DRAIN ? 4 : 1)
            for (int round = 0; round < HALF / 16; ++round) {
                const int c0 = c_first + 16 * round;
                if constexpr (DRAIN) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const uint32_t o = stage + stage_off(row, i / 4);
                        const int k = DRAIN ? 16 * round + i : 0;        // (the other form has one element)
                        st_shared4(o, out(sr[k]), out(sr[k + 1]), out(sr[k + 2]), out(sr[k + 3]));
                        st_shared4(o + STAGE_PLANE, out(si[k]), out(si[k + 1]), out(si[k + 2]), out(si[k + 3]));
                    }
                } else {
                    float a[16], f[16], b[16], e[16];
                    tmem_ld16(tl + c0, a);                   // A_re.B_re
                    tmem_ld16(tl + 256 + TN + c0, f);             // A_im.B_im
                    tmem_ld16(tl + TN + c0, b);             // A_re.B_im
                    tmem_ld16(tl + 256 + c0, e);             // A_im.B_re
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const uint32_t o = stage + stage_off(row, i / 4);
                        st_shared4(o, out(a[i] + sgn * f[i]), out(a[i + 1] + sgn * f[i + 1]), out(a[i + 2] + sgn * f[i + 2]),
                                   out(a[i + 3] + sgn * f[i + 3]));
                        st_shared4(o + STAGE_PLANE, out(e[i] - sgn * b[i]), out(e[i + 1] - sgn * b[i + 1]),
                                   out(e[i + 2] - sgn * b[i + 2]), out(e[i + 3] - sgn * b[i + 3]));
                    }
                }
                if (!DRAIN && c0 == c_last) {
                    // last TMEM read of this segment done: hand the accumulators back to the MMA warp
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                }
                epi_bar_sync(group);
                if (!DRAIN && c0 == c_last && et == 0) {
                    if constexpr (PAIR) mbar_arrive_cluster(map_to_rank(acc_empty, lead_rank));   // the first CTA's MMA thread waits for both
                    else mbar_arrive(acc_empty);
                }
                if constexpr (VEC) {
                    // coalesced write-out: each warp instruction covers 8 rows x 64 contiguous bytes
#pragma unroll
                    for (int h = 0; h < 4; h += U) {
                        float4 vr[U], vi[U];
#pragma unroll
                        for (int j = 0; j < U; ++j) {
                            const int idx = et + 128 * (h + j);
                            const uint32_t at = stage + stage_off(idx >> 2, idx & 3);
                            vr[j] = ld_shared4(at);
                            vi[j] = ld_shared4(at + STAGE_PLANE);
                        }
                        if (pre) {
#pragma unroll
                            for (int j = 0; j < U; ++j) {
                                vr[j].x += gr[j].x; vr[j].y += gr[j].y; vr[j].z += gr[j].z; vr[j].w += gr[j].w;
                                vi[j].x += gi[j].x; vi[j].y += gi[j].y; vi[j].z += gi[j].z; vi[j].w += gi[j].w;
                            }
                            if (c0 != c_last) request(c0 + 16, 0);
                        }
#pragma unroll
                        for (int j = 0; j < U; ++j) {
                            const int idx = et + 128 * (h + j);
                            const int gm = m0 + (idx >> 2), gn = n0 + c0 + (idx & 3) * 4;
                            if (gm >= rows || gn >= p.N) continue;
                            const size_t o = (size_t) gm * p.N + gn;
                            if (add_res && need_old) {   // both at once: old D is read here
                                const float4 xr = *reinterpret_cast<const float4*>(p.d_re + o), xi = *reinterpret_cast<const float4*>(p.d_im + o);
                                vr[j].x += xr.x; vr[j].y += xr.y; vr[j].z += xr.z; vr[j].w += xr.w;
                                vi[j].x += xi.x; vi[j].y += xi.y; vi[j].z += xi.z; vi[j].w += xi.w;
                            }
                            if (partial) {
                                atomicAdd(reinterpret_cast<float4*>(p.d_re + o), vr[j]);
                                atomicAdd(reinterpret_cast<float4*>(p.d_im + o), vi[j]);
                            } else {
                                *reinterpret_cast<float4*>(p.d_re + o) = vr[j];
                                *reinterpret_cast<float4*>(p.d_im + o) = vi[j];
                            }
                        }
                    }
                } else {
                    // a warp takes 32 rows, 16 floats of two rows per instruction; what is added to sixteen rows is
                    // requested before the first of them is stored
                    const int gn = n0 + c0 + (lane & 15), half = lane >> 4;
#pragma unroll 1
                    for (int r0 = q * 32 + half; r0 < q * 32 + 32; r0 += 16) {
                        float ar[8], ai[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int gm = m0 + r0 + 2 * j;
                            const size_t o = (size_t) gm * p.N + gn;
                            const bool on = gm < rows && gn < p.N;
                            ar[j] = ai[j] = 0.f;
                            if (on && add_res) { ar[j] = ld_global_now1(p.r_re + o); ai[j] = ld_global_now1(p.r_im + o); }
                            if (on && need_old) { ar[j] += ld_global_now1(p.d_re + o); ai[j] += ld_global_now1(p.d_im + o); }
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t at = stage + stage_off(r0 + 2 * j, (lane & 15) >> 2) + 4u * (uint32_t) (lane & 3);
                            ar[j] += ld_shared1(at);
                            ai[j] += ld_shared1(at + STAGE_PLANE);
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int gm = m0 + r0 + 2 * j;
                            if (gm >= rows || gn >= p.N) continue;
                            const size_t o = (size_t) gm * p.N + gn;
                            if (partial) { atomicAdd(p.d_re + o, ar[j]); atomicAdd(p.d_im + o, ai[j]); }
                            else { p.d_re[o] = ar[j]; p.d_im[o] = ai[j]; }
                        }
                    }
                }
                epi_bar_sync(group);                 // staging is reused by the next round
            }
            u += kb1 - kb0;
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        finish();
        if (split_cluster) {
            CNB_GSTAMP(6, threadIdx.x == Threads<DRAIN>::FIRST_EPI);
            if (!plain && !*abort_flag) {
                const int tile = blockIdx.x / cluster_ctas;
                const int m0 = (tile / tiles_n) * TILE_M + row_off, n0 = (tile % tiles_n) * TN;
                const int et = (warp - EPI_WARP) * 32 + lane;
                const uint32_t peer0 = PAIR ? prank : 0u, peer_step = PAIR ? 2u : 1u;
                switch (p.cluster) {
                    case 2: cluster_reduce<2, VEC, TN>(p, smem_base, crank, m0, n0, et, peer0, peer_step); break;
                    case 4: cluster_reduce<4, VEC, TN>(p, smem_base, crank, m0, n0, et, peer0, peer_step); break;
                    default: cluster_reduce<8, VEC, TN>(p, smem_base, crank, m0, n0, et, peer0, peer_step); break;
                }
            }
            CNB_GSTAMP(7, threadIdx.x == Threads<DRAIN>::FIRST_EPI);
            __syncwarp();                                // (lanes beyond the tile have left the loops one by one)
            cluster_sync();                              // no CTA leaves while a peer still reads its shared memory
            CNB_GSTAMP(8, threadIdx.x == Threads<DRAIN>::FIRST_EPI);
        }
        if (FORM == PACKED && plain) fma_product(p, smem);   // shared memory is idle: every chain has been read out
    }
}

// The operand split (cnb_split_store*, common.cuh) of a pair of planes into a split buffer with plane pitch np.
__global__ void split_k(const float* __restrict__ s0, const float* __restrict__ s1, float* __restrict__ sp, size_t np,
                        size_t n) {
    cnb_pdl_enter();
    const cnb_split_dst d0 = cnb_split_component(sp, np, 0), d1 = cnb_split_component(sp, np, 1);
    size_t stride = (size_t) gridDim.x * blockDim.x * 4;
    for (size_t i = ((size_t) blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += stride) {
        if (i + 3 < n) {
            const float4 x = *reinterpret_cast<const float4*>(s0 + i), y = *reinterpret_cast<const float4*>(s1 + i);
            cnb_split_store4(d0, i, x.x, x.y, x.z, x.w);
            cnb_split_store4(d1, i, y.x, y.y, y.z, y.w);
        } else {
            for (size_t j = i; j < n; ++j) { cnb_split_store1(d0, j, s0[j]); cnb_split_store1(d1, j, s1[j]); }
        }
    }
}

// Packed operands.  x = 2^-e (high + low), high = fp16(x 2^e), low = fp16(x 2^e - high), with one e for the whole
// matrix that brings its largest component into [2^14, 2^15): 22 bits of every component down to 2^-17 of the largest,
// fewer below, an absolute error of 2^-39 of the largest at most (half of fp16's least subnormal, 2^-25, beside 2^14).
//
// That must not cost what fp32's exponent range gave: rows of another scale than their neighbours keep their own
// relative precision in the forward product and dX*, columns in dW*.  So the first pass also finds the largest component
// of every group of 1 x 128 and of 32 x 1 elements (down to about half of that where the sizes are no multiples: a remainder of
// a few elements would be small by chance, which the values of a CGelu often are), and a matrix in which one of these (not
// all zero) lies below 2^-17 of the largest is stored as it is, as fp32 planes in the same bytes, and multiplied in fp32
// FMAs.
struct PackJob {
    const float* re; const float* im;
    __half* dst;                       // four planes of rows * pitch: high re, high im, low re, low im (or two of float)
    cnb_pack_head* head;               // max_bits, low_bits and ticket are zero between uses
    int rows, cols, pitch, blocks, max_blocks;
    int tiles_x, tiles_y;              // groups of the first pass; the first rows % tiles_y of them have a row more, likewise columns
};
template <int N> struct PackJobs { PackJob j[N]; };

constexpr int GROUP_ROWS = 32, GROUP_COLS = 128;

__host__ __device__ __forceinline__ bool pack_vec(const float* re, const float* im, int cols) {
    return cols % 4 == 0 && ((reinterpret_cast<uintptr_t>(re) | reinterpret_cast<uintptr_t>(im)) & 15) == 0;
}
__device__ __forceinline__ bool pack_vec(const PackJob& job) { return pack_vec(job.re, job.im, job.cols); }

// kPlain: some group is too small beside the largest component, or that itself is so small that no scale of fp32 brings it to 2^14.
__device__ __forceinline__ int pack_exponent(unsigned max_bits, unsigned low_bits) {
    if (max_bits == 0) return 0;
    const int e = 14 + 127 - (int) (max_bits >> 23);
    const bool wide = low_bits != 0 && __uint_as_float(~low_bits) < __uint_as_float(max_bits) * 0x1p-17f;
    return wide || e > 126 ? kPlain : e;
}

// Two components as high and low parts under the matrix's scale.
__device__ __forceinline__ void pack_pair(float a, float b, float scale, __half2* hi, __half2* lo) {
    a *= scale; b *= scale;
    *hi = __floats2half2_rn(a, b);
    const float2 f = __half22float2(*hi);
    *lo = __floats2half2_rn(a - f.x, b - f.y);
}

// Blocks take tiles of up to GROUP_ROWS x GROUP_COLS in turn, a warp four rows of a tile and a lane four elements of each.
template <int N>
__global__ void __launch_bounds__(256) pack_max_k(const __grid_constant__ PackJobs<N> jobs) {
    cnb_pdl_enter();
    const PackJob& job = jobs.j[blockIdx.y];
    if ((int) blockIdx.x >= job.max_blocks) return;
    __shared__ unsigned col[8][GROUP_COLS], block_most[8], block_low[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = pack_vec(job);
    const int unit = vec ? 4 : 1, units = job.cols / unit, tiles = job.tiles_x * job.tiles_y;
    const int width = units / job.tiles_x, wider = units % job.tiles_x, height = job.rows / job.tiles_y, higher = job.rows % job.tiles_y;
    unsigned most = 0, low = 0;        // low: ~ of the least group maximum, 0 while there is none
    for (int t = blockIdx.x; t < tiles; t += job.max_blocks) {
        const int y = t / job.tiles_x, x = t % job.tiles_x;
        const int top = y * height + min(y, higher), r0 = top + warp, r1 = top + height + (y < higher);
        const int c0 = (x * width + min(x, wider)) * unit, c1 = c0 + (width + (x < wider)) * unit;
        float re[4][4], im[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + 8 * i;
            const size_t at = (size_t) row * job.cols + c0;
            if (vec) {
                const bool on = row < r1 && c0 + 4 * lane < c1;
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 x = on ? *reinterpret_cast<const float4*>(job.re + at + 4 * lane) : z;
                const float4 y = on ? *reinterpret_cast<const float4*>(job.im + at + 4 * lane) : z;
                re[i][0] = x.x; re[i][1] = x.y; re[i][2] = x.z; re[i][3] = x.w;
                im[i][0] = y.x; im[i][1] = y.y; im[i][2] = y.z; im[i][3] = y.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const bool on = row < r1 && c0 + lane + 32 * k < c1;
                    re[i][k] = on ? job.re[at + lane + 32 * k] : 0.f;
                    im[i][k] = on ? job.im[at + lane + 32 * k] : 0.f;
                }
            }
        }
        unsigned c[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            unsigned g = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned m = max(cnb_scale_bits(re[i][k]), cnb_scale_bits(im[i][k]));
                c[k] = max(c[k], m);
                g = max(g, m);
            }
            g = __reduce_max_sync(0xffffffffu, g);
            most = max(most, g);
            if (g) low = max(low, ~g);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) col[warp][k * 32 + lane] = c[k];      // every column has a place of its own
        __syncthreads();
        if (threadIdx.x < GROUP_COLS) {
            unsigned g = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) g = max(g, col[w][threadIdx.x]);
            if (g) low = max(low, ~g);
        }
        __syncthreads();
    }
    low = __reduce_max_sync(0xffffffffu, low);
    if (lane == 0) { block_most[warp] = most; block_low[warp] = low; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) { most = max(most, block_most[w]); low = max(low, block_low[w]); }
        atomicMax(&job.head->max_bits, most);
        atomicMax(&job.head->low_bits, low);
    }
}

// Small matrices (those of a 512-row batch, 4 MB) are a chain of round trips: the head, then the data.  AHEAD: what a thread
// converts first is requested before the head is read, each further piece before the stores of the one before, and the head is
// given back at the end (4096 x 4096 65.9 -> 63.7 us, 300 x 500 5.0 -> 4.5, 1000 x 1001 9.8 -> 8.4).  Two columns at a time that
// is no gain where there are more blocks than are resident: it takes registers, six CTAs to an SM instead of eight, from loads of
// 4 bytes that want many in flight (5306 x 3317 82.8 us, as plain loops of loads and stores 77.9; 1001 x 1333, nine blocks to an
// SM, 10.2 and 9.5; 777 x 1333, seven, 8.6 and 9.1).
template <int N, bool AHEAD>
__global__ void __launch_bounds__(256) pack_k(const __grid_constant__ PackJobs<N> jobs) {
    cnb_pdl_enter();
    const PackJob& job = jobs.j[blockIdx.y];
    if ((int) blockIdx.x >= job.blocks) return;
    // Consecutive threads take consecutive columns: four each where the rows allow 16-byte loads (8-byte stores), else
    // two (4-byte accesses), so that every access of a warp is one run.
    const bool vec = pack_vec(job);
    const size_t np = (size_t) job.rows * job.pitch;
    const int groups = vec ? job.cols / 4 : (job.cols + 1) / 2;
    const size_t total = (size_t) job.rows * groups;
    // rows without padding are one run; else a 32-bit division where it does (a 64-bit one was half the kernel's time)
    const bool flat = vec && job.pitch == job.cols;
    struct Item { float4 x, y; size_t dst; };
    auto fetch = [&](size_t i) {
        Item v;
        const int row = flat ? 0 : total >> 32 ? (int) (i / groups) : (int) ((unsigned) i / (unsigned) groups);
        const int g = (int) (i - (size_t) row * groups);
        if (!AHEAD || vec) {
            const size_t src = flat ? 4 * i : (size_t) row * job.cols + 4 * g;
            v.dst = flat ? 4 * i : (size_t) row * job.pitch + 4 * g;
            v.x = *reinterpret_cast<const float4*>(job.re + src);
            v.y = *reinterpret_cast<const float4*>(job.im + src);
        } else {
            const int c = 2 * g;
            const bool two = c + 1 < job.cols;
            const size_t src = (size_t) row * job.cols + c;
            v.dst = (size_t) row * job.pitch + c;
            v.x = make_float4(job.re[src], two ? job.re[src + 1] : 0.f, 0.f, 0.f);
            v.y = make_float4(job.im[src], two ? job.im[src + 1] : 0.f, 0.f, 0.f);
        }
        return v;
    };
    const size_t stride = (size_t) job.blocks * 256;
    size_t i = (size_t) blockIdx.x * 256 + threadIdx.x;
    Item item = {};
    if ((AHEAD || vec) && i < total) item = fetch(i);
    __shared__ int s_exp;
    if (threadIdx.x == 0) {
        const int e = pack_exponent(__ldcg(&job.head->max_bits), __ldcg(&job.head->low_bits));
        s_exp = e;
        if (blockIdx.x == 0) job.head->exponent = e;
    }
    __syncthreads();
    const bool plain = s_exp == kPlain;
    const float scale = plain ? 1.f : __uint_as_float((unsigned) (s_exp + 127) << 23);
    float* const plain_dst = reinterpret_cast<float*>(job.dst);
    auto part = [&](float a, float b, __half2* hi, __half2* lo) { pack_pair(a, b, scale, hi, lo); };
    auto put2 = [&](float x0, float x1, float y0, float y1, size_t dst) {
        if (plain) {
            *reinterpret_cast<float2*>(plain_dst + dst) = make_float2(x0, x1);
            *reinterpret_cast<float2*>(plain_dst + np + dst) = make_float2(y0, y1);
            return;
        }
        __half2 hi, lo;
        part(x0, x1, &hi, &lo);
        *reinterpret_cast<__half2*>(job.dst + dst) = hi;
        *reinterpret_cast<__half2*>(job.dst + 2 * np + dst) = lo;
        part(y0, y1, &hi, &lo);
        *reinterpret_cast<__half2*>(job.dst + np + dst) = hi;
        *reinterpret_cast<__half2*>(job.dst + 3 * np + dst) = lo;
    };
    if (!AHEAD && !vec) {
        // (the planes of a pack are nobody else's, so that the loads of several rounds may go before the stores)
        const float* __restrict__ re = job.re;
        const float* __restrict__ im = job.im;
        for (; i < total; i += stride) {
            const int row = total >> 32 ? (int) (i / groups) : (int) ((unsigned) i / (unsigned) groups), c = 2 * (int) (i - (size_t) row * groups);
            const bool two = c + 1 < job.cols;
            const size_t src = (size_t) row * job.cols + c;
            const float x0 = re[src], y0 = im[src];
            put2(x0, two ? re[src + 1] : 0.f, y0, two ? im[src + 1] : 0.f, (size_t) row * job.pitch + c);
        }
    }
    while (i < total) {
        const float4 x = item.x, y = item.y;
        const size_t dst = item.dst;
        i += stride;
        if (i < total) item = fetch(i);                  // the next one, before this one's stores
        if (AHEAD && !vec) {
            put2(x.x, x.y, y.x, y.y, dst);
            continue;
        }
        if (plain) {
            *reinterpret_cast<float4*>(plain_dst + dst) = x;
            *reinterpret_cast<float4*>(plain_dst + np + dst) = y;
            continue;
        }
        __align__(8) __half2 hi[2], lo[2];
        part(x.x, x.y, &hi[0], &lo[0]); part(x.z, x.w, &hi[1], &lo[1]);
        *reinterpret_cast<uint2*>(job.dst + dst) = *reinterpret_cast<uint2*>(hi);
        *reinterpret_cast<uint2*>(job.dst + 2 * np + dst) = *reinterpret_cast<uint2*>(lo);
        part(y.x, y.y, &hi[0], &lo[0]); part(y.z, y.w, &hi[1], &lo[1]);
        *reinterpret_cast<uint2*>(job.dst + np + dst) = *reinterpret_cast<uint2*>(hi);
        *reinterpret_cast<uint2*>(job.dst + 3 * np + dst) = *reinterpret_cast<uint2*>(lo);
    }
    // every block has read the head (this one's thread 0 before the barrier above): the last one makes it ready for the next use
    if (threadIdx.x == 0 && atomicAdd(&job.head->ticket, 1u) == (unsigned) job.blocks - 1) {
        job.head->max_bits = 0;
        job.head->low_bits = 0;
        job.head->ticket = 0;
    }
}

// Matrices of up to 16 tiles (65536 elements): both passes in one launch, a cluster to a matrix and a CTA to a tile, which holds it
// in registers while the CTAs tell each other their largest and least through distributed shared memory: a cluster barrier in the
// place of a launch and of the second read.  86 x 256 3.9 -> 3.4 us, 128 x 512 4.3 -> 3.8, in clusters of 8 and 16 CTAs; 17 to 32 tiles, two
// to a CTA, 4.8 and 5.5.
constexpr int ONE_CTAS = 8, ONE_TILES = 16;              // (more than eight tiles: a cluster of sixteen, which a device may not have)

template <int N>
__global__ void __launch_bounds__(256) pack_one_k(const __grid_constant__ PackJobs<N> jobs) {
    cnb_pdl_enter();
    const PackJob& job = jobs.j[blockIdx.y];
    __shared__ unsigned col[8][GROUP_COLS], warp_most[8], warp_low[8];
    __shared__ __align__(8) unsigned cta[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = pack_vec(job);
    const int unit = vec ? 4 : 1, units = job.cols / unit, tiles = job.tiles_x * job.tiles_y;
    const int width = units / job.tiles_x, wider = units % job.tiles_x, height = job.rows / job.tiles_y, higher = job.rows % job.tiles_y;
    const int ctas = (int) gridDim.x, t = (int) blockIdx.x, y = t / job.tiles_x, x = t % job.tiles_x;
    const int top = y * height + min(y, higher), r0 = top + warp, r1 = t < tiles ? top + height + (y < higher) : 0;
    const int c0 = (x * width + min(x, wider)) * unit, c1 = c0 + (width + (x < wider)) * unit;
    float re[4][4], im[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = r0 + 8 * i;
        const size_t at = (size_t) row * job.cols + c0;
        if (vec) {
            const bool on = row < r1 && c0 + 4 * lane < c1;
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 u = on ? *reinterpret_cast<const float4*>(job.re + at + 4 * lane) : z;
            const float4 v = on ? *reinterpret_cast<const float4*>(job.im + at + 4 * lane) : z;
            re[i][0] = u.x; re[i][1] = u.y; re[i][2] = u.z; re[i][3] = u.w;
            im[i][0] = v.x; im[i][1] = v.y; im[i][2] = v.z; im[i][3] = v.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool on = row < r1 && c0 + lane + 32 * k < c1;
                re[i][k] = on ? job.re[at + lane + 32 * k] : 0.f;
                im[i][k] = on ? job.im[at + lane + 32 * k] : 0.f;
            }
        }
    }
    unsigned c[4] = {0, 0, 0, 0}, most = 0, low = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        unsigned g = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned m = max(cnb_scale_bits(re[i][k]), cnb_scale_bits(im[i][k]));
            c[k] = max(c[k], m);
            g = max(g, m);
        }
        g = __reduce_max_sync(0xffffffffu, g);
        most = max(most, g);
        if (g) low = max(low, ~g);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) col[warp][k * 32 + lane] = c[k];
    __syncthreads();
    if (threadIdx.x < GROUP_COLS) {
        unsigned g = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) g = max(g, col[w][threadIdx.x]);
        if (g) low = max(low, ~g);
    }
    low = __reduce_max_sync(0xffffffffu, low);
    if (lane == 0) { warp_most[warp] = most; warp_low[warp] = low; }
    __syncthreads();
    if (warp == 0) {
        most = __reduce_max_sync(0xffffffffu, warp_most[lane & 7]);
        low = __reduce_max_sync(0xffffffffu, warp_low[lane & 7]);
        if (lane == 0) { cta[0] = most; cta[1] = low; }
    }
    __syncwarp();                                        // (a barrier of the aligned form takes a warp's threads together)
    cluster_sync();
    most = low = 0;
    if (lane < ctas) {
        const uint32_t at = map_to_rank(smem_u32(cta), (uint32_t) lane);
        asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(most), "=r"(low) : "r"(at) : "memory");
    }
    const int e = pack_exponent(__reduce_max_sync(0xffffffffu, most), __reduce_max_sync(0xffffffffu, low));
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x == 0) job.head->exponent = e;
    const bool plain = e == kPlain;
    const float scale = plain ? 1.f : __uint_as_float((unsigned) (e + 127) << 23);
    const size_t np = (size_t) job.rows * job.pitch;
    float* const plain_dst = reinterpret_cast<float*>(job.dst);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = r0 + 8 * i;
        if (row >= r1) continue;
        const size_t line = (size_t) row * job.pitch + c0;
        if (vec) {
            if (c0 + 4 * lane >= c1) continue;
            const size_t dst = line + 4 * lane;
            if (plain) {
                *reinterpret_cast<float4*>(plain_dst + dst) = make_float4(re[i][0], re[i][1], re[i][2], re[i][3]);
                *reinterpret_cast<float4*>(plain_dst + np + dst) = make_float4(im[i][0], im[i][1], im[i][2], im[i][3]);
                continue;
            }
            __align__(8) __half2 hi[2], lo[2];
            pack_pair(re[i][0], re[i][1], scale, &hi[0], &lo[0]); pack_pair(re[i][2], re[i][3], scale, &hi[1], &lo[1]);
            *reinterpret_cast<uint2*>(job.dst + dst) = *reinterpret_cast<uint2*>(hi);
            *reinterpret_cast<uint2*>(job.dst + 2 * np + dst) = *reinterpret_cast<uint2*>(lo);
            pack_pair(im[i][0], im[i][1], scale, &hi[0], &lo[0]); pack_pair(im[i][2], im[i][3], scale, &hi[1], &lo[1]);
            *reinterpret_cast<uint2*>(job.dst + np + dst) = *reinterpret_cast<uint2*>(hi);
            *reinterpret_cast<uint2*>(job.dst + 3 * np + dst) = *reinterpret_cast<uint2*>(lo);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (c0 + lane + 32 * k >= c1) continue;
                const size_t dst = line + lane + 32 * k;
                if (plain) { plain_dst[dst] = re[i][k]; plain_dst[np + dst] = im[i][k]; continue; }
                __half2 hi, lo;
                pack_pair(re[i][k], im[i][k], scale, &hi, &lo);
                job.dst[dst] = __low2half(hi); job.dst[np + dst] = __high2half(hi);
                job.dst[2 * np + dst] = __low2half(lo); job.dst[3 * np + dst] = __high2half(lo);
            }
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // no CTA leaves while a peer still reads its shared memory
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// In every map `pitch` is the distance in elements between two stored rows (a multiple of 8: TMA wants a 16-byte row
// pitch, of 64 for the MN-major forms) and may exceed their length; what lies between them is never used: a K-major
// box beyond K is zero-filled, and operand rows beyond the last one only reach output columns or rows that do not exist.

// [rows, K] fp32 row-major plane; box = BK x 128 rows; 64-byte swizzle; zero fill outside.
int make_map(CUtensorMap* m, const float* base, int rows, int K, int pitch) {
    constexpr int BK = FormCfg<SPLIT>::BK;
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {(cuuint64_t) K, (cuuint64_t) rows};
    cuuint64_t strides[1] = {(cuuint64_t) pitch * sizeof(float)};
    cuuint32_t box[2] = {(cuuint32_t) BK, 128u};
    cuuint32_t estr[2] = {1u, 1u};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a [%d,%d] plane", (int) r, rows, K);
    return CNB_OK;
}

// MN-major plane stored [K, rows] (rows contiguous, pitch % 32 == 0), seen as [pitch/32][K][32]:
// one box {32, BK, 4} brings four 32-row slabs of 16 k-lines, slab after slab (128-byte swizzle,
// 32-byte atomicity).
int make_map_mn(CUtensorMap* m, const float* base, int K, int pitch) {
    constexpr int BK = FormCfg<SPLIT>::BK;
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[3] = {32u, (cuuint64_t) K, (cuuint64_t) (pitch / 32)};
    cuuint64_t strides[2] = {(cuuint64_t) pitch * sizeof(float), 32u * sizeof(float)};
    cuuint32_t box[3] = {32u, (cuuint32_t) BK, 4u};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for an MN-major [%d,%d] plane", (int) r, K, pitch);
    return CNB_OK;
}

// A pair of 16-bit planes (real, imaginary; np elements apart), each [rows, K] row-major, seen as [2][rows][K]: one
// box {BK, 128, 2} brings the 128 rows of both planes, real then imaginary (planes_per_box = 1: of one plane; box_rows: of
// 64 rows for narrow tiles);
// the swizzle is the box's row of 2 BK bytes.
int make_map16(CUtensorMap* m, const void* base, int rows, int K, int pitch, size_t np, unsigned planes_per_box, unsigned box_rows,
               int BK, CUtensorMapDataType type) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[3] = {(cuuint64_t) K, (cuuint64_t) rows, 2u};
    cuuint64_t strides[2] = {(cuuint64_t) pitch * 2u, (cuuint64_t) np * 2u};
    cuuint32_t box[3] = {(cuuint32_t) BK, box_rows, planes_per_box};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    CUresult r = fn(m, type, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, BK == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a 16-bit [%d,%d] plane pair", (int) r, rows, K);
    return CNB_OK;
}

// The same pair stored [K, rows] (rows contiguous, pitch % 64 == 0), seen as [2][pitch/64][K][64]: one box
// {64, BK, 2, 2} brings two 64-row slabs of 16 k-lines of both planes, slab after slab (128-byte swizzle).
int make_map16_mn(CUtensorMap* m, const void* base, int K, int pitch, size_t np, unsigned planes_per_box, unsigned box_rows,
                  int BK, CUtensorMapDataType type) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[4] = {64u, (cuuint64_t) K, (cuuint64_t) (pitch / 64), 2u};
    cuuint64_t strides[3] = {(cuuint64_t) pitch * 2u, 128u, (cuuint64_t) np * 2u};
    cuuint32_t box[4] = {64u, (cuuint32_t) BK, box_rows / 64, planes_per_box};
    cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    CUresult r = fn(m, type, 4, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cnb::set_error(CNB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for an MN-major 16-bit [%d,%d] plane pair", (int) r, K, pitch);
    return CNB_OK;
}

// Clears the two output planes of a product whose tiles are summed with atomics.
__global__ void zero_pair_k(float* __restrict__ a, float* __restrict__ b, size_t n) {
    cnb_pdl_enter();
    const size_t n4 = n / 4;
    const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
    const size_t tid = (size_t) blockIdx.x * blockDim.x + threadIdx.x, step = (size_t) gridDim.x * blockDim.x;
    if (vec) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        for (size_t i = tid; i < n4; i += step) {
            reinterpret_cast<float4*>(a)[i] = z;
            reinterpret_cast<float4*>(b)[i] = z;
        }
        for (size_t i = 4 * n4 + tid; i < n; i += step) { a[i] = 0.f; b[i] = 0.f; }
    } else {
        for (size_t i = tid; i < n; i += step) { a[i] = 0.f; b[i] = 0.f; }
    }
}

// The schedule of one product: which form (one CTA per tile or CTA pairs), how many CTAs, how the (tile, k-block)
// units are dealt.  Host arithmetic only (also reachable as cnb_gemm_schedule, for tests that need no GPU).
struct Schedule { bool pair; long ctas, upc; int whole_per_cta, clear_from_row, cluster, segments; bool splits_tiles, joined; int tile_n, first, rest; bool exact; };

// Sizes whose products have always been split ones here, at 19 bits an operand: packed ones are nearer to float64 there
// whatever the length of the chain (512 x 1024 x 1024: 1.9e-6 -> 0.9e-6, 4096 x 1024 x 1024: 4.5e-6 -> 3.1e-6).
bool split_sizes(int M, int N, int K) { return K % 8 == 0 && K >= 32 && M >= 64 && N >= 64; }

// The longest chain of a product with K > 4096, in k-blocks of 16 (see choose_schedule).
constexpr int kMaxChain16 = 64;

// Every other size could run as fp32 FMAs (cgemm_simt.cu), and the tiles must not be less exact than those.  The tensor
// core truncates as it accumulates: measured on balanced data one chain of C products is off by 4.2e-9 C of the result,
// rounded FMAs over K products by 1.8e-8 sqrt(K), and a sum of chains rounded to nearest by what one chain is.  So a chain
// may be 4.28 sqrt(K) long, in blocks of 32.
int max_chain(int K) { return std::max(1, (int) (4.28 * std::sqrt((double) K) / FormCfg<PACKED>::BK)); }

// The longest run of k-blocks that one CTA sums for a tile.
int longest_run(const Schedule& q, int k_blocks) {
    return q.cluster > 1 ? (k_blocks + q.cluster - 1) / q.cluster : q.whole_per_cta > 0 ? k_blocks : (int) std::min<long>(q.upc, k_blocks);
}

// The chains of a packed product in k-blocks of 32: a tile's first ones, and those of all others.
//
// At sizes that were split products, whole tiles of K <= 4096 are one chain, and a longer K is cut at choose_schedule's cap.  Whole
// tiles that used to be shared runs (`joined`) take two chains at least, of 24 at most: what was shared had shorter chains than a
// whole tile (4096 x 1024, K = 512: 1.57e-6 off float64, 1.83e-6 as one chain, 0.93e-6 as two; K = 1024 3.11e-6, and 1.83e-6 as
// two).  A second chain takes up to 2.5 us (K = 256: 34.8 us as shared runs, 23.7 as one chain, 26.2 as two; K = 512 47.1,
// 37.8, 38.0).
//
// At others max_chain is the line.  A run of K > 4096 that is longer than the cap is cut as evenly as runs of that length were:
// 1500 x 1500, K = 4100 in chains of 8, 8, 8 and 2 a run 8.7e-7 off, in chains of 8 throughout 9.3e-7, of 7 7.8e-7.
// `joined` there: what whole chains leave of K, or one of them, goes to both ends (4089 x 1019, K = 500, 16 blocks: 2.29e-7 off
// as shared runs, 2.30e-7 as 8 x 2, 2.21e-7 as 1 + 7 x 2 + 1; 3321 x 1275, K = 250, 8 blocks: 2.22e-7, 2.27e-7, 2.06e-7).
//
// Runs by CTA pairs that make five chains or more of at least three blocks take the accumulators out one after the other, and a
// block less a chain for it: the MMAs wait less, and the second rounding weighs less than the block (4089 x 1019, K = 1001 4.47e-7
// off as shared runs, 91 us as EXACT, 81 and 3.72e-7 so; 777 x 1001, K = 1333 47.6 -> 45.0 us, 4.44e-7 -> 3.75e-7; a mean of
// 0.95 over 28 sizes).  In fewer chains, or by single CTAs, that is no gain (1.00 to 1.04 over 85).
struct Chains { int first, rest; bool exact; };
Chains chain_blocks(int M, int N, int K, const Schedule& q) {
    const int n = (K + FormCfg<PACKED>::BK - 1) / FormCfg<PACKED>::BK, cap = kMaxChain16 * FormCfg<SPLIT>::BK / FormCfg<PACKED>::BK;
    auto evenly = [](int blocks, int most) { const int chains = (blocks + most - 1) / most; return (blocks + chains - 1) / chains; };
    if (q.rest > 0) return {q.first, q.rest, true};      // (narrow_tiles)
    if (split_sizes(M, N, K)) {
        const int c = evenly(n, K > 4096 ? cap : q.joined ? std::max(2, std::min(24, (n + 1) / 2)) : n);
        return {c, c, false};
    }
    const int run = longest_run(q, n), c = K > 4096 && run > cap ? evenly(evenly(n, cap), max_chain(K)) : max_chain(K);
    if (q.pair && max_chain(K) >= 3 && run > 4 * c) return {c - 1, c - 1, false};
    return {q.joined && n > c ? (n % c + c + 1) / 2 : c, c, true};
}

// The form of a packed launch: chains are taken out of tensor memory one after the other wherever a run is cut, also where only the
// run of a tile's first blocks is (785 x 1218, K = 616 added to a gradient, slices of 9 and 10 blocks and a first chain of 9: launched
// as one chain each, which the plan is not, 1.13e-6 off float64 in the place of 1.08e-6).
Drain drain_form(int M, int N, int K, const Schedule& q, const Chains& chains) {
    const int k_blocks = (K + FormCfg<PACKED>::BK - 1) / FormCfg<PACKED>::BK, run = longest_run(q, k_blocks);
    const int first_run = q.cluster > 1 ? k_blocks / q.cluster : run;
    // several tiles a CTA (a single tile's runs are not: 83 x 102, K = 13688 took 1.4 us more in that form)
    const int tiles = (M + (q.pair ? 2 * BM : BM) - 1) / (q.pair ? 2 * BM : BM) * ((N + BN - 1) / BN);
    const bool several = q.cluster == 1 && q.segments == 0 && tiles > 1 && (q.whole_per_cta > 0 || q.upc != k_blocks);
    const bool cut = run > chains.rest || first_run > chains.first;
    return q.exact || (cut && chains.exact) ? EXACT : cut || several ? OVERLAP : NONE;
}

// Clusters of `ctas` CTAs, each with an SM to itself, that are resident at once: 15 of eight and 33 of four on 148 SMs.
int resident_clusters(int ctas, int sms) { return ctas == 8 ? sms * 15 / 148 : ctas == 4 ? sms * 33 / 148 : sms / ctas; }

// The chains of a run from k-block `from` to `to`: how many, and the sum of the cubes of their lengths, which is what the square of
// the error goes with: what is truncated in a chain of C, C at the magnitude of sqrt(C).
struct Sum { long chains, cubes; };
Sum chains_of(int from, int to, int first, int rest) {
    const int head = from == 0 ? std::min(first, to) : 0, whole = (to - from - head) / rest, left = (to - from - head) % rest;
    auto cube = [](long n) { return n * n * n; };
    return {(head > 0) + whole + (left > 0), cube(head) + whole * cube(rest) + cube(left)};
}

// The cubes of a packed launch, of a tile in the mean.
double tile_cubes(int M, int N, int K, const Schedule& q) {
    const int k_blocks = (K + FormCfg<PACKED>::BK - 1) / FormCfg<PACKED>::BK, tile_m = q.pair ? 2 * BM : BM;
    const long tiles = (long) ((M + tile_m - 1) / tile_m) * ((N + q.tile_n - 1) / q.tile_n), units = tiles * k_blocks;
    Chains chains = chain_blocks(M, N, K, q);
    if (drain_form(M, N, K, q, chains) == NONE) chains.first = chains.rest = k_blocks;
    double cubes = 0;
    auto run = [&](long from, long to) { if (to > from) cubes += (double) chains_of((int) from, (int) to, chains.first, chains.rest).cubes; };
    const long pieces = q.cluster > 1 ? q.cluster : q.segments;              // of every tile alike
    if (pieces > 0) {
        for (long k = 0; k < pieces; ++k)
            if (q.cluster > 1) run(k_blocks * k / pieces, k_blocks * (k + 1) / pieces);
            else run(k * q.upc, std::min<long>(k_blocks, (k + 1) * q.upc));
        return cubes;
    }
    const long whole = std::min(tiles, q.whole_per_cta * q.ctas);
    cubes = (double) whole * chains_of(0, k_blocks, chains.first, chains.rest).cubes;
    long run_end = whole * k_blocks + q.upc, tile = whole * k_blocks;       // where a run ends; a tile's first unit
    for (long u = tile; u < units && q.upc > 0;) {
        const long end = std::min(run_end, tile + k_blocks);
        run(u - tile, end - tile);
        u = end;
        if (u == run_end) run_end += q.upc;
        if (u == tile + k_blocks) tile = u;
    }
    return cubes / tiles;
}

// Narrow tiles (128 x 64) for products of few tiles, one CTA to a tile's slice of K.  Past the MMAs such a launch takes as long as
// half a tile of 128 x 128 needs three times: out of tensor memory (1.1 us), between the CTAs of a cluster (2.5 to 3.5 us, 38 bytes
// a ns into an SM, and a barrier), into memory (1.2); and it leaves most SMs without a tile.
//
// Where twice the tiles still are one wave in the clusters of the wide ones, every element's sum is what it was, in order too
// (product and packs, us: 300 x 300, K = 300 18.1 -> 14.6, 64 x 784, K = 784 18.4 -> 16.1, 128 x 128, K = 4096 29.6 -> 23.3).
//
// Where they are not, smaller clusters may be faster; clusters that are not all resident at once (15 of eight CTAs and 33 of four
// are, on 148 SMs) never are, and neither are short runs summed with atomics.  The estimate below, fitted to 20 sizes at every
// width and cluster that has room and to 40 that ran as such sums, has to promise a microsecond (300 x 500, K = 500 19.2 -> 17.3,
// 256 x 512, K = 512 17.1 -> 15.2, 128 x 2048, K = 512 30.4 -> 18.7, 350 x 401, K = 1081 35.6 -> 22.7; 512 x 1024, K = 1024 stays
// as it is).  Of 2100 products of 16 to 3000 rows and columns that run otherwise with narrow tiles than without, the time is 0.83 of
// what it was in the mean; seven take 2 to 6 % more (390 x 108, K = 1639 20.9 -> 22.1, 1048 x 928, K = 3432 104 -> 108), the others no
// more than runs of one program differ.  Chains are as short as it takes that sums in another order are no further off float64: a
// twentieth fewer cubes (below), since as many, cut elsewhere, are up to 1.02 times as far off.  None of the 2100 is more than 1.002
// times as far, and in the mean they are 0.92 times.
//
// Products with an N of up to 128, and gradients with an M of up to 128, are those of a head.  The gradient of a loss divides by
// what they give, which magnifies a sum in another order, so they keep theirs where it is fixed.
void narrow_tiles(Schedule& r, int M, int N, int K, int k_blocks, int accumulate, int sms) {
    auto fit = [&](int c) { return resident_clusters(c, sms); };
    const long rows = (M + BM - 1) / BM, wide = rows * ((N + BN - 1) / BN), narrow = rows * ((N + NARROW - 1) / NARROW);
    auto take = [&](int tile_n, int c) {
        r.pair = false;
        r.tile_n = tile_n;
        r.cluster = c;
        r.ctas = (tile_n == NARROW ? narrow : wide) * c;
        r.upc = c > 1 ? 0 : k_blocks;
        r.splits_tiles = false;
    };
    const int c0 = r.cluster;
    if (r.whole_per_cta > 0 || r.segments > 0) return;
    if (c0 == 1 && !r.splits_tiles) {                    // a CTA or a pair to a tile
        const Chains now = chain_blocks(M, N, K, r);
        const bool whole = r.pair ? now.rest >= k_blocks || now.exact : r.ctas == wide;
        if (whole && narrow <= sms) take(NARROW, 1);
        return;
    }
    if (c0 > 1 && (k_blocks + c0 - 1) / c0 > kMaxChain16 / 2) return;        // (chains that are taken out one after the other)
    if (c0 > 1 && !r.pair && narrow <= fit(c0)) return take(NARROW, c0);
    if ((c0 > 1 && (N <= BN || (accumulate && M <= BM))) || K > 4096) return;

    auto cluster_of = [&](int c, int first, int rest) {                      // most chains of a CTA, and all cubes of a tile
        Sum v = {0, 0};
        for (int k = 0; k < c; ++k) {
            const Sum w = chains_of(k_blocks * k / c, k_blocks * (k + 1) / c, first, rest);
            v = {std::max(v.chains, w.chains), v.cubes + w.cubes};
        }
        return v;
    };
    const Chains now = chain_blocks(M, N, K, r);
    const long tiles = c0 > 1 ? 1 : r.pair ? (long) ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN) : wide;
    long all_cubes = 0;                                  // of `tiles` tiles, as they are; 0: not asked for yet
    auto cubes = [&] {
        if (all_cubes > 0) return all_cubes;
        if (c0 > 1) return all_cubes = cluster_of(c0, now.first, now.rest).cubes;
        long run_end = r.upc, tile = 0;                  // where the run ends; the tile's first unit
        for (long u = 0; u < tiles * k_blocks;) {
            const long end = std::min(run_end, tile + k_blocks);
            all_cubes += chains_of((int) (u - tile), (int) (end - tile), now.first, now.rest).cubes;
            u = end;
            if (u == run_end) run_end += r.upc;
            if (u == tile + k_blocks) tile = u;
        }
        return all_cubes;
    };
    // Where chains begin (K <= 4096), and how many of them the sums hold, over all additions of a tile: each is rounded at its magnitude.
    struct Sums { std::bitset<128> at; int adds; };
    auto sums = [&](int c, int first, int rest) {
        Sums v = {{}, 0};
        for (int k = 0, all = 0; k < c; ++k) {
            int n = 0;
            for (int kb = k_blocks * k / c, end = k_blocks * (k + 1) / c; kb < end; kb += kb == 0 ? first : rest) {
                v.at.set(kb);
                v.adds += n > 0 ? n + 1 : 0;
                ++n;
            }
            v.adds += all > 0 ? all + n : 0;
            all += n;
        }
        return v;
    };
    const bool several = now.rest < (c0 > 1 ? (k_blocks + c0 - 1) / c0 : r.upc), vec = N % 4 == 0;
    // Costs in hundredths of a microsecond: blocks, what a cluster adds, taking a chain out of tensor memory before the next.
    struct { int tile_n, c, first, rest; long cost; } best = {0, 0, 0, 0, 0};
    long before = 1 << 30;
    auto consider = [&](int tile_n, int c, bool as_it_is) {
        if ((tile_n == NARROW ? narrow : wide) > fit(c)) return;
        static const int wide_add[4] = {140, 430, 590, 690}, narrow_add[4] = {0, 235, 345, 470};
        const bool thin = tile_n == NARROW, crowd = (thin ? narrow : wide) * c > 100 * sms / 148;
        const int log_c = c == 8 ? 3 : c == 4 ? 2 : c - 1, run = (k_blocks + c - 1) / c;
        long fixed = (thin ? (crowd ? 85 : 70) * run + narrow_add[log_c] : 90 * run + wide_add[log_c]) + (crowd && c == 8 ? 200 : 0);
        // What is added to is read by the CTAs themselves: by one CTA for its whole tile, four bytes a lane where 16 do not fit, and
        // by fewer CTAs of a smaller cluster (1013 x 1747, K = 366 as one run a tile 43.4 -> 55.6 us, 824 x 240, K = 680 in clusters of
        // four 20.0 -> 21.6, 438 x 880, K = 104 as one run 16.2 -> 17.1).
        if (accumulate && c == 1) fixed += vec ? (thin ? 300 : 100) : (thin ? 900 : 1900);
        else if (accumulate && c0 > 1 && !r.pair && !as_it_is) fixed += 250;
        const int chain = thin ? 50 : 100;
        // the longest chains that are no less exact than those of the form before; a shorter first one where that does.  No further
        // than a cost that would be taken (the search through all of it took up to 14 us of the host's time a launch, 437 x 89, K = 3952).
        const long most = best.c ? best.cost - 1 : before - 100;
        for (int rest = std::min(run, now.rest); rest >= 1 && fixed + chain * ((run + rest - 1) / rest - 1) <= most; --rest)
            for (int first = rest; first >= std::max(1, rest - 1); --first) {
                const Sum v = cluster_of(c, first, rest);
                // As many cubes in other runs may be 1.03 as far off (1010 x 1595, K = 323), and so may the same chains added up one after
                // the other (346 x 1698, K = 199: four in a row 1.027 as far as two by two).
                if (!as_it_is && v.cubes * tiles * 20 > cubes() * 19) {
                    if (c0 == 1 || c == 1 || v.cubes != cubes()) continue;
                    const Sums before_it = sums(c0, now.first, now.rest), it = sums(c, first, rest);
                    if (it.at != before_it.at || it.adds > before_it.adds) continue;
                }
                const long cost = fixed + chain * (v.chains - 1);
                if (best.c == 0 || cost < best.cost) best = {tile_n, c, first, rest, cost};
                return;
            }
    };
    if (c0 == 1) {
        before = (vec ? 800 : 1500) + (split_sizes(M, N, K) ? 0 : 300) - (accumulate ? 300 : 0) + 80 * r.upc;
    } else if (r.pair) {                                 // two pairs to a tile of 256 x 128: as two CTAs to one of 128 x 128
        before = 90 * ((k_blocks + 1) / 2) + 430 + 100 * (cluster_of(c0, now.first, now.rest).chains - 1);
    } else {
        consider(BN, c0, true);
        if (best.c) before = best.cost;
        best.c = 0;
    }
    for (int c = c0 == 1 || r.pair ? 8 : c0 / 2; c >= 1; c /= 2) { consider(BN, c, false); consider(NARROW, c, false); }
    // Runs with atomics may take less than the estimate where large clusters would replace them, of eight for a single column of tiles (257 x
    // 112, K = 2375 21.3 -> 24.1, 1022 x 107, K = 2390 33.6 -> 35.0) or of four for rows of 4-byte alignment (409 x 594, K = 1538 33.9 -> 37.7):
    // those have to promise more than a microsecond.  One row of tiles gains a little less by a smaller cluster.
    const bool column = best.c == 8 && N <= BN;
    const long promise = c0 > 1 ? (M <= BM && !r.pair ? 120 : 100) : accumulate || best.c < 4 ? 100 :
                         column ? (!vec ? 550 : split_sizes(M, N, K) ? 250 : 400) : best.c == 4 && !vec ? 350 : 100;
    if (best.c == 0 || best.cost > before - promise) return;
    r.first = best.first;
    r.rest = best.rest;
    r.exact = several && now.exact;                      // runs of a single chain too
    take(best.tile_n, best.c);
}

Schedule choose_schedule(int M, int N, int K, int accumulate, int sm_count, int sm_limit, int bk) {
    // Schedule, by tile count ("CTA" = one CTA, or the CTA pair of a 256-row tile; sms = how many of them this launch
    // may fill: leaving a few SMs free (gemm_cta_limit) lets a concurrent collective's kernels run beside the GEMM):
    //  * tiles >= 4 x SMs, or one nearly full wave of one-tile CTAs when D is not read: whole tiles, plain stores, fixed
    //    summation order; grid = tiles, or (packed operands) one CTA per SM that stays and takes every n-th tile;
    //  * more tiles than SMs: persistent CTAs, one per SM; each takes tiles / SMs whole tiles and then an
    //    equal run of the remaining tiles' k-blocks (summed with atomics), so every SM finishes together
    //    and only the remainder needs atomics and a cleared output.  Packed operands: a remainder that is nearly a wave is
    //    taken as whole tiles too (below);
    //  * few tiles and short runs: a cluster per tile (below); otherwise plain stream-K.
    // K > 4096: one fp32 accumulation chain in tensor memory that long costs accuracy.  Split operands keep to runs of kMaxChain16
    // at most; packed ones cut their runs into chains (chain_blocks), and a tile into as few segments as cost least, or none.
    struct Plan { long ctas, upc; int whole_per_cta, clear_from_row, cluster, segments; bool splits_tiles, joined; };
    const int k_blocks = (K + bk - 1) / bk;
    const bool packed = bk == FormCfg<PACKED>::BK;
    auto blocks = [&](int of16) { return (long) std::max(1, of16 * 16 / bk); };
    auto plan = [&](bool pair) {
        Plan q = {};
        const int tile_m = pair ? 2 * BM : BM;
        const int tiles = ((M + tile_m - 1) / tile_m) * ((N + BN - 1) / BN);
        const long total = (long) tiles * k_blocks;
        const long min_units = blocks(8);                    // do not split below 8 k-blocks per CTA
        const int all = pair ? sm_count / 2 : sm_count;
        // Pairs under an SM limit (a few SMs set aside for a collective's kernel): a pair needs both SMs of a TPC and
        // each SM set aside may cost a pair its partner, so they are counted twice (6 set aside: 68 pairs).
        // A limit of exactly half the device (two products side by side, no collective) leaves half the pairs, less
        // a margin of 4.
        const int set_aside = sm_count - sm_limit;
        const bool halved = sm_limit * 2 == sm_count;
        const int pairs_left = halved ? sm_limit / 2 - 4 : (sm_limit - set_aside) / 2;
        const int sms = sm_limit > 0
            ? std::min(pair ? std::max(1, pairs_left) : sm_limit, all) : all;
        const bool full_wave = !accumulate && tiles <= sms && (long) tiles * 100 >= (long) sms * 85 && k_blocks <= blocks(256);
        const bool whole_tiles = (tiles >= all * 4 && sm_limit <= 0 && k_blocks <= blocks(256)) || full_wave;
        const bool lead_whole = !whole_tiles && tiles > sms && k_blocks <= blocks(256);
        // min_units is about splitting tiles: whole ones are dealt to as many CTAs as there are.  (With a short K
        // total / min_units alone put 16 tiles of 2 blocks on 8 CTAs: 2000 x 50 x 50 36 -> 23 us, 777 x 1001 x 60 36 -> 23.)
        long ctas = std::min<long>(sms, std::max<long>(tiles, total / min_units));
        if (whole_tiles) ctas = tiles;                        // many tiles: whole tiles, no atomics
        long upc = (total + ctas - 1) / ctas;
        if (whole_tiles) upc = k_blocks;
        // The tensor core adds into its fp32 accumulator with truncation, so the error of one accumulation chain
        // in tensor memory grows with its length: measured ~2e-6 of the accumulator's magnitude per k-block, which
        // reached 1e-3 on a 443-k-block chain whose accumulator one large term dominated (the gradient of a loss
        // through a K = 8192 product).  Runs are therefore capped at kMaxChain k-blocks (the partial tiles are summed
        // outside, in fp32 round-to-nearest): several equal waves of CTAs instead of one persistent wave.
        // Only K > 4096 gets here with longer runs; a whole tile of K <= 4096 is at most 256 k-blocks.  Each tile is
        // cut into equal segments and the CTAs are numbered segment-major (see the kernel).
        // (packed operands: the running sums in registers cut the chains, whatever the run)
        const long kMaxChain = blocks(kMaxChain16);
        if (packed && !whole_tiles && upc > kMaxChain && k_blocks > blocks(256)) {
            // As few segments as cost least: waves of runs, and what a run costs beside its k-blocks (start, write-out) as
            // about 9 of them, the cleared output and the atomics as another 5.  At 15 sizes, K from 4100 to 65536, the choice took
            // at most 6.4 % more than the best of one to five (300 x 1024, K = 8192 71.6 us, 67.3 in four; 1024 x 2048, K = 16384
            // 544, 525 in one), at twelve of them at most 2.1 %.
            long best = 0;
            for (int c = 1; (c - 1) * kMaxChain < k_blocks; ++c) {
                const long cost = ((long) tiles * c + sms - 1) / sms * ((k_blocks + c - 1) / c + 9) + (c > 1 ? 5 : 0);
                if (best == 0 || cost < best) { best = cost; q.segments = c; }
            }
            upc = (k_blocks + q.segments - 1) / q.segments;
            ctas = (long) tiles * q.segments;
            if (q.segments == 1) {
                q.segments = 0;
                upc = 0;
                ctas = std::min<long>(tiles, sms);
                q.whole_per_cta = (int) ((tiles + ctas - 1) / ctas);
            }
        } else if (!whole_tiles && upc > kMaxChain && k_blocks > blocks(256)) {
            q.segments = (int) ((k_blocks + kMaxChain - 1) / kMaxChain);     // per tile, each at most kMaxChain k-blocks
            upc = (k_blocks + q.segments - 1) / q.segments;
            ctas = (long) tiles * q.segments;
        } else {
            ctas = (total + upc - 1) / upc;
        }
        if (packed && tiles > sms && (whole_tiles || (lead_whole && tiles % sms * 10 >= sms * 7))) {
            // Whole tiles by CTAs that stay: the write-out of one runs under the MMAs of the next.  Also where a remainder of
            // tiles, seven tenths of a wave or more, would be shared: no cleared output and no atomics.  Shared and whole on 74 pairs,
            // us: 0.95 of a wave left (4096 x 1152) K = 512 42.0 and 39.5, K = 1024 80.5 and 74.4, K = 2048 150 and 144; 0.73 (4096 x 1024)
            // 41.4 and 38.0, 69.7 and 69.8, 134 and 136; 0.62 (2560 x 1536) 40.5 and 36.8, 65.9 and 66.9, 123 and 132.  On top of
            // what is there, K = 1024: 0.95 79.1 and 76.7, 0.73 67.9 and 71.5, 0.84 of a third wave 111 and 119.  (The line is one for
            // all K: a long one, and an accumulating product, would have it nearer to a whole wave, a short one at a third.)
            ctas = sms;
            upc = 0;
            q.whole_per_cta = (tiles + sms - 1) / sms;
            q.joined = lead_whole;
        } else if (lead_whole) {
            ctas = sms;
            q.whole_per_cta = tiles / sms;
            const long rest = (long) (tiles - q.whole_per_cta * sms) * k_blocks;
            upc = (rest + ctas - 1) / ctas;
            q.clear_from_row = (q.whole_per_cta * sms / ((N + BN - 1) / BN)) * tile_m;   // rows below are only ever stored whole
        }
        // Few tiles (small batches): a cluster of 2, 4 or 8 CTAs takes one tile, every CTA a slice of K, and
        // the partial tiles are summed through distributed shared memory: no atomics, no cleared output,
        // a fixed summation order.
        // Worth it while a stream-K run would be short (<= 48 k-blocks): with long runs the atomics are
        // amortised and using every SM wins over the clusters' rounded-down CTA count.
        q.cluster = 1;
        if (!whole_tiles && q.whole_per_cta == 0 && upc <= blocks(48)) {
            // pairs: two slices at most (clusters of 8 CTAs do not all fit a GPC side by side: measured 0.043 ms
            // against 0.025 at 512 x 1024 x 1024)
            for (int c = pair ? 2 : 8; c >= 2; c >>= 1)
                if ((long) tiles * c <= sms && k_blocks / c >= blocks(4)) { q.cluster = c; break; }
            // Long K over few tiles leaves the cluster form most of the device idle: 83 x 102 x 13688, one tile, ran
            // 107 k-blocks on each of 8 CTAs (126 us) where stream-K runs are 8 k-blocks long.  The atomics and the
            // cleared output of that form cost about as much as 16 k-blocks.
            if (q.cluster > 1 && k_blocks / q.cluster > 2 * upc + blocks(16)) q.cluster = 1;
        }
        if (q.cluster > 1) { ctas = (long) tiles * q.cluster; upc = 0; }
        q.splits_tiles = q.cluster == 1 && (q.whole_per_cta > 0 ? upc > 0 : (q.segments > 0 || (upc % k_blocks) != 0));
        q.ctas = ctas; q.upc = upc;
        return q;
    };
    // The pair form (two CTAs, cta_group::2, per 256-row tile: each CTA stages half of the B operand, so a k-block
    // costs 48 KB of shared-memory fill per CTA instead of 64 KB): at least one whole pair tile of rows; with few
    // tiles, a cluster of two pairs per tile, each pair a slice of K.
    static const bool pair_allowed = [] { const char* e = getenv("CNB_GEMM_PAIR"); return !(e && e[0] == '0'); }();
    // beside a collective (SMs set aside): measured 2.145 -> 2.115 ms per step at 2 GPUs; CNB_GEMM_PAIR_DP=0 turns it off
    static const bool pair_beside_collective = [] { const char* e = getenv("CNB_GEMM_PAIR_DP"); return !(e && e[0] == '0'); }();
    // not under a limit that halves the device (two products side by side at small batches: measured 1.25 -> 1.31 ms
    // per step at 4 GPUs with pairs there)
    const bool small_reserve = sm_limit > 0 &&
        (sm_count - sm_limit <= 16 || sm_limit * 2 == sm_count);   // or exactly half, no collective
    bool pair = pair_allowed && (sm_limit <= 0 || (pair_beside_collective && small_reserve)) && M >= 2 * BM;
    Plan q = plan(pair);
    if (pair && q.cluster > 1) {                         // K-split clusters: pairs only if they fill as many SMs
        const Plan single = plan(false);
        if (single.ctas > 2 * q.ctas) { pair = false; q = single; }
    }
    Schedule r;
    r.pair = pair; r.ctas = q.ctas; r.upc = q.upc; r.whole_per_cta = q.whole_per_cta; r.clear_from_row = q.clear_from_row;
    r.cluster = q.cluster; r.segments = q.segments; r.splits_tiles = q.splits_tiles; r.joined = q.joined;
    r.tile_n = BN;
    r.first = r.rest = 0;
    r.exact = false;
    if (packed) narrow_tiles(r, M, N, K, k_blocks, accumulate, sm_limit > 0 ? std::min(sm_limit, sm_count) : sm_count);
    return r;
}

}  // namespace

namespace cnb {

bool cgemm_tc_fits(int M, int N, int K) {
    if (split_sizes(M, N, K)) return true;
    // Other sizes leave more of the 128 x 128 tiles empty: from about two million complex multiplications on packing
    // and tiles together take less than the fp32 SIMT tiles (64 x 64, K = 512: 15.5 against 12.3 us), below it they do not.
    // A short K leaves little to gain on either: 2000 x 50 takes 6 us in FMAs and 23 in tiles at K = 50; with more 64 x 64
    // blocks than SMs the FMAs take several waves (1000 x 1000 x 60: 21 and 20).
    if (K < 96 && (long) ((M + 63) / 64) * ((N + 63) / 64) <= 148) return false;
    return K >= 48 && (double) M * N * K >= (double) (1 << 21);
}

bool cgemm_tc_shape_ok(int M, int N, int K) {
    // Small products are done by the SIMT tiles before the operands would be packed.  FMAs, packing and tiles, us: 128 x 128,
    // K = 128 4.9 and 13.6, K = 256 8.6 and 14.3, 200 x 100, K = 200 9.9 and 16.7, 200 x 200, K = 200 17.0 and 17.8; 300 x 256,
    // K = 200, 15 million, 17.9 and 16.7; 300 x 256, K = 256 21.9 and 14.5.  The line is on the safe side: FMAs are ahead to
    // K = 400 or so where outputs are few (128 x 128, K = 300 9.9 and 17.0, K = 400 12.7 and 16.1, K = 512 15.7 and 14.7), and
    // beyond 8 million where K is short (1000 x 256, K = 64 9.9 and 12.6; 4000 x 64, K = 100 15.6 and 15.9).
    if (K <= 256 && (double) M * N * K <= 8e6) return false;
    return cgemm_tc_fits(M, N, K);
}

// K of 48 to 256 in chains of one or two blocks is 1.13e-7 to 2.5e-7 off float64 here, and in FMAs added one by one 1.8e-8 sqrt(K):
// 268 x 117, K = 213 1.17e-7 and 2.67e-7; in sums of sixteen 1.10e-7 (11.0 and 11.5 us).
bool cgemm_fma_in_chains(int M, int N, int K) { return cgemm_tc_fits(M, N, K) && !cgemm_tc_shape_ok(M, N, K) && !split_sizes(M, N, K); }

static size_t padded(int n, int to) { return ((size_t) n + to - 1) / to * to; }

// An operand of `rows` x K as cgemm_tc_run stores it: K-major rows at a pitch of K rounded up to 8 (TMA's 16 bytes), or,
// from a source stored [K, rows], MN-major lines at a pitch of rows rounded up to 64.
static int operand_pitch(int rows, int K, int trans) { return (int) (trans ? padded(rows, 64) : padded(K, 8)); }
static size_t operand_bytes(int rows, int K, int trans) {
    return (8 * (size_t) (trans ? K : rows) * operand_pitch(rows, K, trans) + 255) & ~size_t(255);
}

size_t cgemm_tc_workspace_bytes(int M, int N, int K) {
    return std::max(operand_bytes(M, K, 0), operand_bytes(M, K, 1)) + std::max(operand_bytes(N, K, 0), operand_bytes(N, K, 1)) + 4096;
}

// The GEMM proper on operands that are already split: the four slots of a split buffer (hi_re, hi_im,
// [h16_re ; h16_im], [l16_re ; l16_im]) lie plane_pitch floats apart, elements are stored [rows, K] (mn = 0) or
// [K, rows] (mn = 1) with stored rows at `pitch`.
int cgemm_tc_presplit(cnb_ctx* ctx, const SplitOperand& a, const SplitOperand& b, int conjB,
                      const float* r_re, const float* r_im, float* d_re, float* d_im, int M, int N, int K,
                      int accumulate, cudaStream_t st) {
    static bool attr_set[64] = {};                       // the attribute is per device
    if (!attr_set[ctx->device & 63]) {
#define CNB_TC_ATTR(F, D)                                                                                                   \
    do {                                                                                                                    \
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, false, F, D, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES)); \
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, true, F, D, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));  \
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<true, false, F, D, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));  \
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<true, true, F, D, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));   \
    } while (0)
        CNB_TC_ATTR(SPLIT, NONE); CNB_TC_ATTR(PACKED, NONE); CNB_TC_ATTR(PACKED, OVERLAP); CNB_TC_ATTR(PACKED, EXACT);
#undef CNB_TC_ATTR
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, false, PACKED, NONE, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, true, PACKED, NONE, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, false, PACKED, EXACT, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        CNB_CUDA(cudaFuncSetAttribute(cgemm_tc_k<false, true, PACKED, EXACT, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        // the shares of a launch with running sums must add up to what it starts with
#define CNB_TC_REGS(P, V, D, T)                                                                                              \
    do {                                                                                                                    \
        cudaFuncAttributes f;                                                                                               \
        CNB_CUDA(cudaFuncGetAttributes(&f, cgemm_tc_k<P, V, PACKED, D, T>));                                                   \
        if (f.numRegs < LAUNCH_REGS) return set_error(CNB_ERR_CUDA, "cgemm_tc: built with %d registers a thread, not %d", f.numRegs, LAUNCH_REGS); \
    } while (0)
        CNB_TC_REGS(false, false, OVERLAP, BN); CNB_TC_REGS(false, true, OVERLAP, BN); CNB_TC_REGS(true, false, OVERLAP, BN); CNB_TC_REGS(true, true, OVERLAP, BN);
        CNB_TC_REGS(false, false, EXACT, BN); CNB_TC_REGS(false, true, EXACT, BN); CNB_TC_REGS(true, false, EXACT, BN); CNB_TC_REGS(true, true, EXACT, BN);
        CNB_TC_REGS(false, false, EXACT, NARROW); CNB_TC_REGS(false, true, EXACT, NARROW);
#undef CNB_TC_REGS
        attr_set[ctx->device & 63] = true;
    }
    if ((reinterpret_cast<uintptr_t>(d_re) | reinterpret_cast<uintptr_t>(d_im)) & 3)
        return set_error(CNB_ERR_ARG, "cgemm_tc: misaligned output");
    if (a.pitch % (a.mn ? 64 : 8) || b.pitch % (b.mn ? 64 : 8))
        return set_error(CNB_ERR_ARG, "cgemm_tc: operand pitches %d and %d", a.pitch, b.pitch);
    const bool packed = a.exponent != nullptr;
    const int bk = packed ? FormCfg<PACKED>::BK : FormCfg<SPLIT>::BK;
    const Schedule q = choose_schedule(M, N, K, accumulate, ctx->sm_count, ctx->gemm_cta_limit, bk);
    const bool pair = q.pair;
    const long ctas = q.ctas;
    const int cluster = q.cluster;

    int rc;
    OperandMaps<SPLIT> maps_s;
    OperandMaps<PACKED> maps_p;
    const unsigned b_planes = pair ? 1u : 2u;            // pair: a CTA loads the real or the imaginary plane of B
    for (int side = 0; side < 2; ++side) {
        const SplitOperand& o = side ? b : a;
        const int rows = side ? N : M;
        const unsigned planes = side ? b_planes : 2u, box_rows = side ? (unsigned) q.tile_n : 128u;
        if (packed) {
            for (int k = 0; k < 2; ++k) {                // high parts, low parts
                CUtensorMap* m = &maps_p.m[2 * side + k];
                const __half* base = reinterpret_cast<const __half*>(o.base) + 2 * k * o.plane_pitch;
                rc = o.mn ? make_map16_mn(m, base, K, o.pitch, o.plane_pitch, planes, box_rows, bk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16)
                          : make_map16(m, base, rows, K, o.pitch, o.plane_pitch, planes, box_rows, bk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
                if (rc != CNB_OK) return rc;
            }
            continue;
        }
        for (int k = 0; k < 4; ++k) {
            CUtensorMap* m = &maps_s.m[4 * side + k];
            const float* base = o.base + k * o.plane_pitch;
            if (k < 2) rc = o.mn ? make_map_mn(m, base, K, o.pitch) : make_map(m, base, rows, K, o.pitch);
            else rc = o.mn ? make_map16_mn(m, base, K, o.pitch, o.plane_pitch, planes, 128u, bk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16)
                           : make_map16(m, base, rows, K, o.pitch, o.plane_pitch, planes, 128u, bk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
            if (rc != CNB_OK) return rc;
        }
    }
    if (q.splits_tiles && !accumulate) {
        // one launch clears both planes (they need not be adjacent or in one allocation)
        const size_t first = (size_t) q.clear_from_row * N;
        const size_t plane = (size_t) M * N - first;
        const size_t vec = plane / 4 + 1;
        const int blocks = (int) std::min<size_t>((vec + 255) / 256, (size_t) ctx->sm_count * 8);
        cnb::launch(zero_pair_k, dim3(blocks), dim3(256), 0, st, 1, d_re + first, d_im + first, plane);
        CNB_LAUNCH_CHECK("zero_pair");
    }
    TcParams p;
    p.d_re = d_re; p.d_im = d_im; p.r_re = r_re; p.r_im = r_im;
    p.M = M; p.N = N; p.K = K; p.conjB = conjB; p.accumulate = accumulate;
    p.units_per_cta = (int) q.upc;
    p.a_mn = a.mn; p.b_mn = b.mn;
    p.a_exp = a.exponent; p.b_exp = b.exponent;
    p.a_planes = a.base; p.b_planes = b.base;
    p.a_np = a.plane_pitch; p.b_np = b.plane_pitch;
    p.a_pitch = a.pitch; p.b_pitch = b.pitch;
    p.cluster = cluster;
    p.whole_per_cta = q.whole_per_cta;
    p.segments = q.segments;
    p.status = ctx->d_status;
    const bool vec = N % 4 == 0 && ((reinterpret_cast<uintptr_t>(d_re) | reinterpret_cast<uintptr_t>(d_im) |
                                     reinterpret_cast<uintptr_t>(r_re) | reinterpret_cast<uintptr_t>(r_im)) & 15) == 0;
    const Chains chains = chain_blocks(M, N, K, q);
    p.chain = chains.rest;
    p.first = chains.first;
    const Drain drain = packed ? drain_form(M, N, K, q, chains) : NONE;
    auto go = [&](auto kernel, const auto& maps) {
        return cnb::launch(kernel, dim3((unsigned) (pair ? 2 * ctas : ctas)), dim3(drain == NONE ? Threads<NONE>::ALL : Threads<OVERLAP>::ALL), SMEM_BYTES, st,
                           pair ? 2 * cluster : cluster, maps, p);
    };
    cudaError_t e;
#define CNB_TC_GO(F, D, maps)                                                                                              \
    (pair ? (vec ? go(cgemm_tc_k<true, true, F, D, BN>, maps) : go(cgemm_tc_k<true, false, F, D, BN>, maps))               \
          : (vec ? go(cgemm_tc_k<false, true, F, D, BN>, maps) : go(cgemm_tc_k<false, false, F, D, BN>, maps)))
#define CNB_TC_GO_NARROW(D) (vec ? go(cgemm_tc_k<false, true, PACKED, D, NARROW>, maps_p) : go(cgemm_tc_k<false, false, PACKED, D, NARROW>, maps_p))
    if (q.tile_n == NARROW) e = drain == EXACT ? CNB_TC_GO_NARROW(EXACT) : CNB_TC_GO_NARROW(NONE);
    else if (!packed) e = CNB_TC_GO(SPLIT, NONE, maps_s);
    else if (drain == EXACT) e = CNB_TC_GO(PACKED, EXACT, maps_p);
    else if (drain == OVERLAP) e = CNB_TC_GO(PACKED, OVERLAP, maps_p);
    else e = CNB_TC_GO(PACKED, NONE, maps_p);
#undef CNB_TC_GO
#undef CNB_TC_GO_NARROW
    CNB_CUDA(e);
    CNB_LAUNCH_CHECK("cgemm_tc");
    return CNB_OK;
}

// ------------------------------------------------------------------------------------------------ packed operands
SplitOperand packed_operand(const PackRequest& r, int mn) {
    return {static_cast<const float*>(r.planes), (size_t) r.rows * r.pitch, r.pitch, mn, &r.head->exponent};
}

// Whether the device holds clusters of ONE_TILES CTAs of pack_one_k, which are beyond the portable size.
template <int N> static bool wide_clusters(int device) {
    static std::atomic<signed char> known[64];           // 0: not asked yet
    std::atomic<signed char>& k = known[device & 63];
    if (k == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim = {ONE_TILES, 1, 1};
        cfg.gridDim = dim3(ONE_TILES);
        cfg.blockDim = dim3(256);
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool ok = cudaFuncSetAttribute(pack_one_k<N>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, pack_one_k<N>, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        k = ok ? 1 : -1;
    }
    return k > 0;
}

// Jobs in pairs of launches of at most 32, or in one where all are small.
template <int N> static int pack_some(cnb_ctx* ctx, const PackRequest* r, int n, cudaStream_t st) {
    PackJobs<N> jobs;
    int blocks = 0, max_blocks = 0;
    bool vec = true;
    for (int k = 0; k < n; ++k) vec = vec && pack_vec(r[k].re, r[k].im, r[k].cols);
    // Enough blocks in all to fill the device a few times over, whatever the number of jobs.  Of two operands the large one's
    // blocks are to be one wave, of six CTAs to an SM or (in plain loops) eight: 829 x 4812 -> 13 dW*, all in fours, 37.5 us with
    // eight blocks to an SM for each of its operands, 35.9 with six.
    const size_t cap = std::max<size_t>(16, (size_t) ctx->sm_count * (vec && n > 1 ? 12 : 16) / n);
    size_t all = 0;
    for (int k = 0; k < n; ++k) {
        if (reinterpret_cast<uintptr_t>(r[k].planes) & 127 || r[k].pitch % 8)
            return set_error(CNB_ERR_ARG, "pack: planes must be 128-byte aligned, pitch %d a multiple of 8", r[k].pitch);
        const size_t items = (size_t) r[k].rows * ((r[k].cols + 3) / 4);
        const int tiles_x = (r[k].cols - 1) / GROUP_COLS + 1, tiles_y = (r[k].rows - 1) / GROUP_ROWS + 1;
        const size_t tiles = (size_t) tiles_x * tiles_y;
        jobs.j[k] = {r[k].re, r[k].im, static_cast<__half*>(r[k].planes), r[k].head, r[k].rows, r[k].cols, r[k].pitch,
                     (int) std::min((items + 255) / 256, cap), (int) std::min(tiles, cap), tiles_x, tiles_y};
        blocks = std::max(blocks, jobs.j[k].blocks);
        all += jobs.j[k].blocks;
        max_blocks = std::max(max_blocks, jobs.j[k].max_blocks);
    }
    long tiles = 0;
    for (int k = 0; k < n; ++k) tiles = std::max(tiles, (long) jobs.j[k].tiles_x * jobs.j[k].tiles_y);
    if (tiles <= ONE_CTAS || (tiles <= ONE_TILES && wide_clusters<N>(ctx->device))) {
        const int ctas = tiles <= ONE_CTAS ? ONE_CTAS : ONE_TILES;
        CNB_CUDA(cnb::launch(pack_one_k<N>, dim3(ctas, n), dim3(256), 0, st, ctas, jobs));
        CNB_LAUNCH_CHECK("pack_one");
        return CNB_OK;
    }
    cnb::launch(pack_max_k<N>, dim3(max_blocks, n), dim3(256), 0, st, 1, jobs);
    CNB_LAUNCH_CHECK("pack_max");
    if (vec || all <= 7 * (size_t) ctx->sm_count) cnb::launch(pack_k<N, true>, dim3(blocks, n), dim3(256), 0, st, 1, jobs);
    else cnb::launch(pack_k<N, false>, dim3(blocks, n), dim3(256), 0, st, 1, jobs);
    CNB_LAUNCH_CHECK("pack");
    return CNB_OK;
}

int pack(cnb_ctx* ctx, const PackRequest* r, int n, cudaStream_t st) {
    if (n <= 2) return pack_some<2>(ctx, r, n, st);
    for (int k = 0; k < n; k += 32) {
        const int rc = pack_some<32>(ctx, r + k, std::min(32, n - k), st);
        if (rc != CNB_OK) return rc;
    }
    return CNB_OK;
}

// fp32 operands, packed into scratch first.  a_trans / b_trans say the source is stored [K, rows]; it is then consumed
// MN-major.  The heads sit in the context's status block, which starts at zero.
int cgemm_tc_run(cnb_ctx* ctx, const float* a_re, const float* a_im, int a_trans, const float* b_re,
                 const float* b_im, int b_trans, int conjB, const float* r_re, const float* r_im, float* d_re,
                 float* d_im, int M, int N, int K, int accumulate, cudaStream_t st, const PackRequest* b_packed) {
    float* ws = nullptr;
    const size_t na = operand_bytes(M, K, a_trans), nb = b_packed ? 0 : operand_bytes(N, K, b_trans);
    int rc = ensure_scratch(ctx, na + nb, false, st, &ws);
    if (rc != CNB_OK) return rc;
    cnb_pack_head* heads = reinterpret_cast<cnb_pack_head*>(ctx->d_status + 768);
    PackRequest r[2];
    r[0] = {a_re, a_im, a_trans ? K : M, a_trans ? M : K, operand_pitch(M, K, a_trans), ws, heads};
    if (b_packed) r[1] = *b_packed;
    else r[1] = {b_re, b_im, b_trans ? K : N, b_trans ? N : K, operand_pitch(N, K, b_trans), reinterpret_cast<char*>(ws) + na, heads + 1};
    rc = pack(ctx, r, b_packed ? 1 : 2, st);
    if (rc != CNB_OK) return rc;
    return cgemm_tc_presplit(ctx, packed_operand(r[0], a_trans), packed_operand(r[1], b_trans), conjB, r_re, r_im, d_re, d_im, M, N,
                             K, accumulate, st);
}

static void split_launch(cnb_ctx* ctx, const float* s0, const float* s1, float* sp, size_t np, size_t n, cudaStream_t st) {
    const size_t blocks = (n / 4 + 255) / 256 + 1, cap = (size_t) ctx->sm_count * 16;
    cnb::launch(split_k, dim3((unsigned) std::min(blocks, cap)), dim3(256), 0, st, 1, s0, s1, sp, np, n);
}

int split_planes(cnb_ctx* ctx, const float* re, const float* im, size_t n, float* split, cudaStream_t st) {
    if (((reinterpret_cast<uintptr_t>(re) | reinterpret_cast<uintptr_t>(im) | reinterpret_cast<uintptr_t>(split)) & 15) != 0)
        return set_error(CNB_ERR_ARG, "split: planes must be 16-byte aligned");
    split_launch(ctx, re, im, split, (n + 63) & ~size_t(63), n, st);
    CNB_LAUNCH_CHECK("split");
    return CNB_OK;
}

}  // namespace cnb

static int schedule_of(int M, int N, int K, int accumulate, int sm_count, int sm_limit, int bk, int* out8) {
    if (!out8 || M <= 0 || N <= 0 || K <= 0 || sm_count <= 0)
        return cnb::set_error(CNB_ERR_ARG, "cnb_gemm_schedule: M=%d N=%d K=%d sm_count=%d", M, N, K, sm_count);
    const Schedule q = choose_schedule(M, N, K, accumulate, sm_count, sm_limit, bk);
    out8[0] = q.pair ? 1 : 0;
    out8[1] = (int) (q.pair ? 2 * q.ctas : q.ctas);      // CTAs of the launch
    out8[2] = q.cluster * (q.pair ? 2 : 1);              // CTAs per cluster (1: no cluster)
    out8[3] = (int) q.upc;
    out8[4] = q.whole_per_cta;
    out8[5] = q.segments;
    out8[6] = q.splits_tiles ? 1 : 0;
    out8[7] = q.clear_from_row;
    return CNB_OK;
}

extern "C" int cnb_gemm_schedule(int M, int N, int K, int accumulate, int sm_count, int sm_limit, int* out8) {
    return schedule_of(M, N, K, accumulate, sm_count, sm_limit, FormCfg<SPLIT>::BK, out8);
}

extern "C" int cnb_gemm_schedule_packed(int M, int N, int K, int accumulate, int sm_count, int sm_limit, int* out8) {
    return schedule_of(M, N, K, accumulate, sm_count, sm_limit, FormCfg<PACKED>::BK, out8);
}

extern "C" int cnb_gemm_chain_packed(int M, int N, int K, int accumulate, int sm_count, int sm_limit) {
    if (M <= 0 || N <= 0 || K <= 0 || sm_count <= 0)
        return cnb::set_error(CNB_ERR_ARG, "cnb_gemm_chain_packed: M=%d N=%d K=%d sm_count=%d", M, N, K, sm_count);
    const Schedule q = choose_schedule(M, N, K, accumulate, sm_count, sm_limit, FormCfg<PACKED>::BK);
    return chain_blocks(M, N, K, q).rest;
}

extern "C" double cnb_gemm_share_packed(int M, int N, int K, int accumulate, int sm_count) {
    if (M <= 0 || N <= 0 || K <= 0 || sm_count <= 0) return -1.0;
    const Schedule q = choose_schedule(M, N, K, accumulate, sm_count, 0, FormCfg<PACKED>::BK);
    const int ctas = q.cluster * (q.pair ? 2 : 1);
    return (double) q.ctas / q.cluster / std::max(1, resident_clusters(ctas, sm_count));
}

extern "C" double cnb_gemm_truncation_packed(int M, int N, int K, int accumulate, int sm_count, int sm_limit) {
    if (M <= 0 || N <= 0 || K <= 0 || sm_count <= 0) return -1.0;
    return tile_cubes(M, N, K, choose_schedule(M, N, K, accumulate, sm_count, sm_limit, FormCfg<PACKED>::BK));
}

extern "C" int cnb_gemm_form_packed(int M, int N, int K, int accumulate, int sm_count, int sm_limit, int* out4) {
    if (!out4 || M <= 0 || N <= 0 || K <= 0 || sm_count <= 0)
        return cnb::set_error(CNB_ERR_ARG, "cnb_gemm_form_packed: M=%d N=%d K=%d sm_count=%d", M, N, K, sm_count);
    const Schedule q = choose_schedule(M, N, K, accumulate, sm_count, sm_limit, FormCfg<PACKED>::BK);
    const Chains chains = chain_blocks(M, N, K, q);
    out4[0] = q.tile_n;
    out4[1] = chains.first;
    out4[2] = chains.rest;
    out4[3] = drain_form(M, N, K, q, chains);
    return CNB_OK;
}
