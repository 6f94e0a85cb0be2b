// Tensor-core path of the binned parse (sm_100a): the kernel template and its launcher,
// instantiated per path and tile variant in ldk_tc_hap0.cu, ldk_tc_hap1.cu, ldk_tc_geno.cu.
//
// Counting as a Gram product.  For SNPs i, j and one population, with per-haplotype spins
// sigma = 1 - 2 [allele == 1] (0 where missing) and v = [allele != missing], the four products
//   R = sum_k sigma_ik sigma_jk,  S = sum_k sigma_ik v_jk,  T = sum_k v_ik sigma_jk,  n = sum_k v_ik v_jk
// determine the two-locus counts exactly (n11 = (n - S - T + R) / 4, ...; pg_gpu
// ld_pipeline.py:155-172) and are the moments the estimators are polynomials of
// (ldk_spin.cuh), so no count is rebuilt per pair.  Genotypes: sigma = 1 - g, sigma^2 and v.
//
// Layout in HBM (built by k_prep_planes): per SNP two s8 planes (sigma, v) over the
// concatenated haplotypes of all populations, each population padded to a multiple of
// 32 bytes, the whole K axis to a multiple of 128 bytes:  planes[snp][plane][k].
// A 3-D TMA box {128 k, 2 planes, R snps} then lands in shared memory as 2R interleaved
// rows (sigma_i0, v_i0, sigma_i1, ...) in the 128-byte-swizzled K-major layout that
// tcgen05.mma reads directly.  One MMA per 32-byte K step and population:
//   D[128 x 2NJ] (+)= A[128 rows = 64 SNPs x {sigma, v}] . B[2NJ rows = NJ SNPs x {sigma, v}]^T
// with s8 inputs and s32 accumulation in tensor memory: TMEM lane 2r holds (R, S) and
// lane 2r+1 holds (T, n) of SNP i0+r against every j of the tile.
//
// What bounds it: with two or more populations the FP64 estimators of the epilogue, not the
// counts.  The spin forms take 30 / 112 / 267 FP64 operations a pair for 1 / 2 / 3 haplotype
// populations (the factored raw-call forms they replaced: 404 measured for three) and
// 35 / 144 / 316 for genotypes (the nine-cell polynomials: 404 for one population's numerators
// alone).  B200, 1965 MHz, a pass with the old forms -> with the spin forms -> with what the
// comments below describe: 500 diploids x 100,000 SNPs 9.63 -> 3.79 -> 2.57 ms, two genotype
// populations x 20,001 SNPs 5.28 -> 2.77 -> 0.99, three haplotype populations x 200 windows
// 48.0 -> 39.5 -> 31.4 (FP64 pipe about 56%: estimators 12 of a warp's 17 thousand cycles a
// tile), two x 50,000 SNPs 6.93 -> 5.74 -> 4.86.  With one population the loads weigh as much as
// the estimators: 2,000 haplotypes x 10^6 SNPs 28.3 -> 21.2 ms, where a tile's 21.7 thousand
// cycles hold 10 of waiting for TMA traffic (about 10 TB/s from L2) and the epilogue takes 20.
//
// Warp roles (one CTA per SM, persistent over work items: runs of one row block's partner
// tiles, claimed dynamically):
//   warp 0     TMA producer (A: row block, B: 8..128 partner SNPs, per 128-byte K chunk)
//   warp 1     TMEM allocator and MMA issuer, double-buffered accumulators
//   epilogue   8, 12 or 16 warps (see Cfg), two to four per TMEM lane quarter, each
//              taking its share of every partner tile: tcgen05.ld the moments (QROWS: all
//              four of a pair in one thread), evaluate the estimators in FP64, sum per
//              distance bin in registers (bins are monotone in j for a fixed i), flush each
//              finished bin run into an FP64 staging copy in shared memory, and add the
//              staged sums to the per-bootstrap-block fixed-point accumulators once per work
//              item (integer atomics, so the result does not depend on the order of the
//              items).
// Every wait is bounded (LDK_DEVERR_TIMEOUT) so a fault cannot hang the GPU.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <utility>

#include "ldk_estimators.cuh"
#include "ldk_internal.h"

namespace ldk {
namespace {

constexpr int kKChunk = 128;            // K bytes per TMA box / swizzle row
constexpr int kRing = 2;                // claimed work items in flight between the roles
constexpr int kTmemCols = 512;
constexpr uint64_t kTimeoutNs = 5000000000ull;  // 5 s per wait
// Register split of the SPLIT layouts: the launch gives every thread Cfg::REG_LAUNCH
// registers; warpgroup 0 drops to Cfg::REG_CTRL and the epilogue warpgroups rise to Cfg::REG_EPI,
// which the freed registers cover (Cfg asserts the sum).  The host launches only a kernel
// compiled to Cfg::REG_LAUNCH registers.
constexpr size_t kMinSmem = 116 * 1024;
constexpr size_t kMaxSmem = 227 * 1024;  // of a CTA, its __shared__ variables (Cfg::SHARED) included
constexpr size_t kSpareSmem = 1536;      // kept free of flush rows and further ring stages
constexpr int kMaxStages = 8;

// Tile geometry.  Haplotype path: a row block of 64 SNPs x {sigma, v} = 128 MMA rows against
// NJ partners x {sigma, v} (N = 2 NJ), one MMA per K step and population.  Genotype path: a row
// block of 128 SNPs; four stored planes per SNP {sigma, sigma^2, valid, 0}; per K step and
// population three MMAs, plane x (< 3) of the row block against all four planes of NJ
// partners (N = 4 NJ) into region x, so TMEM lane r holds all nine Gram products of SNP r
// (and a zero column per partner, which keeps every partner's columns 4-aligned).
// Partners per tile: tile variant 0 is the default, variant 1 the alternative the
// autotuner also times (half the width on the haplotype path; on the genotype path 8 for
// one population, 16 for two -- one TMEM buffer -- and the default for more).
// One genotype population: 12 (or 24), so that each of the three epilogue warps of a lane
// quarter takes an equal share of the tile.
constexpr int tile_nj(int P, bool GENO, int V) {
    return GENO ? (V == 0 ? (P == 1 ? 12 : 8) : (P == 1 ? 24 : P == 2 ? 16 : 8))
                : ((P == 1 ? 128 : P == 2 ? 48 : 32) >> V);
}

template <int P, bool GENO = false, int V = 0, bool IL = false>
struct Cfg {
    static constexpr int ROWS = GENO ? 128 : 64;                      // SNPs per row block
    static constexpr int PLANES = GENO ? 4 : 2;                        // stored planes per SNP
    static constexpr int NJ = tile_nj(P, GENO, V);                     // partners per tile
    static constexpr int N = PLANES * NJ;                              // MMA N
    static constexpr int REGIONS = GENO ? 3 : 1;                       // MMAs per K step and population
    static constexpr int COLS = P * REGIONS * N;                       // TMEM columns per buffer
    static constexpr int NBUF = 2 * COLS <= kTmemCols ? 2 : 1;         // accumulator buffers
    // four genotype populations: two stages, so that the per-bin staging of more bins fits
    // beside them (their epilogue, not the loads, sets the pace)
    static constexpr int STAGES = GENO ? (P == 4 ? 2 : 3) : (P == 1) ? 2 : (P == 2) ? 3 : 4;
    static constexpr int A_BOX = 128 * kKChunk;                        // one 128-row A box
    static constexpr int A_BYTES = REGIONS * A_BOX;
    static constexpr int B_BYTES = N * kKChunk;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int NS = HapNStats<P>::value;
    static constexpr int SLOTS = GENO ? 4 : 2;                         // bootstrap blocks staged per row block
    // QROWS (one to three haplotype populations): A rows come in groups of sixteen, eight
    // SNPs' sigma rows and the same SNPs' v rows, so that one tcgen05.ld.16x256b hands a
    // thread all four moments (R, S, T, n) of one pair -- SNP lane / 4 of the eight, partner
    // lane % 4 of four -- with no exchange between lanes (eighteen selects and six shuffles a
    // pair for three populations).  Otherwise rows are interleaved
    // (sigma, v per SNP; genotypes: one plane per region) and read with 32x32b.
    // IL (two and three populations of many haplotypes, interleave_k): interleaved all the same,
    // because QROWS loads a row block in eight boxes of 2 KB instead of one of 16.
    static constexpr bool QROWS = !GENO && P <= 3 && !IL;
    // Warp layout.  Warp w may read only TMEM lane quarter w % 4, and each of the four
    // schedulers of an SM holds warps w, w + 4, ... with a quarter of the register file.
    //  * SPLIT (genotypes; haplotypes with two or more populations -- estimators that want
    //    150 to 240 registers): 12 warps.  Warpgroup 0 (TMA, MMA, two idle warps) gives its
    //    registers up with setmaxnreg (24 or 40 each) and the eight epilogue warps 4..11
    //    take them (240 or 232 each), so that every scheduler holds two full-register epilogue
    //    warps beside one control warp (launch: 168 per thread).  Two haplotype populations
    //    with twelve epilogue warps at 160 registers: 5.65 ms, with eight 5.14.
    //  * one genotype population, also SPLIT: 16 warps, twelve epilogue warps 4..15 at 160
    //    registers, three per scheduler and lane quarter (launch: 128).
    //  * one haplotype population: 18 warps, TMA and MMA in warps 0 and 1, sixteen epilogue
    //    warps 2..17, four per lane quarter and scheduler (96 registers: five warps share a
    //    scheduler's quarter of the register file).
    static constexpr int EPI = (!GENO && P == 1) ? 16 : (GENO && P == 1) ? 12 : 8;
    static constexpr bool SPLIT = GENO || P >= 2;
    static constexpr int W0 = SPLIT ? 4 : 2;  // first epilogue warp
    static constexpr int THREADS = 32 * (W0 + EPI);
    static constexpr int REG_LAUNCH = (EPI == 16) ? 96 : (EPI == 12) ? 128 : 168;  // SPLIT layouts only
    // control and epilogue registers; three and four haplotype populations need every register
    // in the epilogue, the others give the control warps enough not to spill
    static constexpr int REG_CTRL = (EPI == 12) ? 32 : (!GENO && P >= 3) ? 24 : 40;
    static constexpr int REG_EPI = (EPI == 16) ? 112 : (EPI == 12) ? 160 : (!GENO && P >= 3) ? 240 : 232;
    // SSPL (four haplotype populations): the two warps of a lane quarter split the
    // statistics, not the partners -- both take every pair, part 0 accumulates statistics
    // [0, K) (DD, Dz) and counts pairs, part 1 the pi2 statistics [K, NS) and r^2 -- so that
    // each holds about half of the 105 accumulators.
    static constexpr bool SSPL = !GENO && P == 4;
    static constexpr int PARTS = SSPL ? 2 : 1;
    // Steps (TMEM reads) per tile and their shares: with QROWS two warps of a quarter split
    // its SNPs, further ones the partners; otherwise the warps split the partners.
    static constexpr int STEPS = GENO ? NJ : QROWS ? NJ / 4 : NJ / 2;
    static constexpr int SHARES = EPI / (4 * PARTS * (QROWS ? 2 : 1));
    static constexpr int MY_STEPS = STEPS / SHARES;
    // Pairs a lane evaluates together: one population's chain of ~45 FP64 operations waits for
    // itself, two interleaved chains less (1,000,000 SNPs x 2,000 haplotypes 21.7 -> 20.7 ms,
    // 5,000 x 100 0.099 -> 0.090); with two populations a pair at a time is faster (5.18 against
    // 5.44 ms), and two pairs of three do not fit the registers.
    static constexpr int U = P == 1 ? 2 : 1;
    static_assert(MY_STEPS % U == 0, "pairs per step");
    using Recip = typename std::conditional<P == 1, double, double4>::type;
    // The ring: as many stages as shared memory has left (STAGES at least), or STAGES where the
    // control warps have 24 registers, which do not hold a run-time length.
    static constexpr bool MORE_STAGES = !SPLIT || REG_CTRL >= 32;
    static constexpr int MAX_STAGES = !MORE_STAGES ? STAGES
                                      : kMaxSmem / STAGE_BYTES < kMaxStages ? (int)(kMaxSmem / STAGE_BYTES) : kMaxStages;
    // bytes of the kernel's __shared__ variables: barriers of the ring, of the accumulators and of the
    // claimed items, the item ring, two words, bin edges (the launch checks it against the build)
    static constexpr size_t SHARED = 16 * MAX_STAGES + 16 * NBUF + 16 * kRing + 8 * kRing + 8 + 8 * (LDK_MAX_BINS + 1);
    // Staging row of the bin flush: a lane's sums, then {pairs, finite r^2, key, -}
    static constexpr int K = GENO ? 0 : SpinSplit<P>::value;
    static constexpr int NA = SSPL ? (K > NS + 1 - K ? K : NS + 1 - K) : NS + 1;  // sums per lane
    static constexpr int FROW = P == 1 ? 0 : (NA + 2) | 1;  // odd: rows in other banks; one population reduces in registers
    static constexpr int FROWS_MAX = 8;
    // The rows of a warp's 32 SNPs (8 with QROWS) cross a bin edge a few partners apart.
    // LATE: a lane's finished sums wait in registers until some lane of the warp leaves the
    // next bin, so one flush serves a whole edge: 500 diploids x 100,000 SNPs 3.10 -> 2.79 ms,
    // 1,000,000 SNPs x 2,000 haplotypes 20.7 -> 20.1 (two haplotype populations 4.80 -> 5.22:
    // their registers cost more than the few flushes).
    // PEND: rows wait in the scratch until it is full, where the staged sums are shared by
    // atomics: two genotype populations 1.03 -> 0.94 ms, four haplotype 2.25 -> 2.23 (two
    // haplotype populations 4.80 -> 5.0, three 31.8 -> 31.9).
    static constexpr bool LATE = P == 1;
    static constexpr bool PEND = P > 1 && (GENO || P == 4);
    static_assert(!SPLIT || 4 * REG_CTRL + EPI * REG_EPI <= (W0 + EPI) * REG_LAUNCH,
                  "register split must fit the launch allocation");
    static_assert(!SPLIT || THREADS * REG_LAUNCH <= 65536, "register file");
    static_assert(EPI % 4 == 0 && STEPS % SHARES == 0 && (!QROWS || NJ % 4 == 0), "epilogue warps share tiles equally");
    static_assert(NBUF * COLS <= kTmemCols, "TMEM budget");
    static_assert(N % 16 == 0 && N <= 256, "MMA N");
};

// ---------------------------------------------------------------------------
// PTX wrappers (tcgen05, TMA, mbarrier)
// ---------------------------------------------------------------------------

LDK_DEV uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

LDK_DEV void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count));
}
LDK_DEV void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
LDK_DEV void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
LDK_DEV bool mbar_test(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on a barrier phase.  False on timeout or when another role aborted.
LDK_DEV bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag, unsigned* status) {
    if (mbar_test(b, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_test(b, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > kTimeoutNs) {
            atomicOr(status, LDK_DEVERR_TIMEOUT);
            *abort_flag = 1;
            return false;
        }
    }
}

LDK_DEV void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(su32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

LDK_DEV void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(dst)), "r"(ncols));
}
LDK_DEV void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;"); }
LDK_DEV void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
LDK_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
LDK_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand in the 128-byte swizzle layout: 8-row groups 1024 bytes apart.
LDK_DEV uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;              // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
    d |= (uint64_t)1 << 46;              // descriptor version for sm_100
    d |= (uint64_t)2 << 61;              // SWIZZLE_128B
    return d;
}

// kind::i8 instruction descriptor: s8 x s8 -> s32, K-major A and B, M = 128.
template <int N>
__host__ __device__ constexpr uint32_t idesc_s8() {
    return (2u << 4)                      // D format s32
           | (1u << 7) | (1u << 10)       // A, B signed 8-bit
           | ((uint32_t)(N >> 3) << 17)   // N / 8
           | ((uint32_t)(128 >> 4) << 24);  // M / 16
}

LDK_DEV void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}
LDK_DEV void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
                 : "memory");
}

// The same from a whole warp, issued by the lane whose `one` is set: predicated, not branched,
// so that the descriptors stay in uniform registers.
LDK_DEV void mma_i8_one(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc, uint32_t one) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(one));
}
LDK_DEV void mma_commit_one(uint64_t* bar, uint32_t one) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(su32(bar)),
        "r"(one)
        : "memory");
}
LDK_DEV uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}

LDK_DEV void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
// Sixteen lanes x eight columns: thread t gets columns 2 (t % 4), + 1 of lane t / 4 in r[0],
// r[1] and of lane t / 4 + 8 in r[2], r[3].
LDK_DEV void tmem_ld_q(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
template <int P>
LDK_DEV void tmem_wait4(uint32_t (&r)[P][4]) {
#pragma unroll
    for (int p = 0; p < P; ++p)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[p][0]), "+r"(r[p][1]), "+r"(r[p][2]), "+r"(r[p][3])
                     :
                     : "memory");
}

template <int EPI>
LDK_DEV void epi_bar() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI) : "memory"); }
template <int EPI>
LDK_DEV bool epi_bar_or(bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "n"(32 * EPI)
        : "memory");
    return r != 0;
}

// Warpgroup-wide register budget changes (all four warps of the warpgroup execute them).
template <int N>
LDK_DEV void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
LDK_DEV void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

LDK_DEV void spin_ns(uint64_t ns) {
    const uint64_t t0 = global_ns();
    while (global_ns() - t0 < ns) {
    }
}

// ---------------------------------------------------------------------------
// the fused count + estimator + bin kernel
// ---------------------------------------------------------------------------

// Flush of one population's four sums: for every (block, bin) among the flushing lanes the
// warp adds the lanes' values with a butterfly that halves the values each lane carries (two
// exchanges leave lane / 8 % 4 with one value, three more add it up), and the four lanes that
// hold a total add it to the staged sums.  About ten lanes of a warp hold the same key when a row
// block crosses a bin edge (all of them since they wait for one another); one lane per round,
// ~60 cycles each, took 25.0 ms for 1,000,000 SNPs x 2,000 haplotypes in 32 bins, this 21.6 (5,000 SNPs x 100:
// 0.119 -> 0.098; 500 diploids x 100,000: 3.82 -> 3.43), all kernel times before the later steps.
template <bool PRIV>
LDK_DEV void flush_one_pop(unsigned mask, int key, const double* acc, unsigned np, unsigned nr2, double* my_sacc,
                           unsigned* my_scnt, int lane) {
    while (mask) {
        const int kk = __shfl_sync(0xffffffffu, key, __ffs(mask) - 1);
        const bool in = ((mask >> lane) & 1u) && key == kk;
        mask &= ~__ballot_sync(0xffffffffu, in);
        const bool h1 = lane & 16, h2 = lane & 8;
        double v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) v[s] = in ? acc[s] : 0.0;
        const unsigned cp = __reduce_add_sync(0xffffffffu, in ? np : 0u);
        const unsigned cr = __reduce_add_sync(0xffffffffu, in ? nr2 : 0u);
        double x0 = h1 ? v[2] : v[0], x1 = h1 ? v[3] : v[1];
        x0 += __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[2], 16);
        x1 += __shfl_xor_sync(0xffffffffu, h1 ? v[1] : v[3], 16);
        double y = h2 ? x1 : x0;
        y += __shfl_xor_sync(0xffffffffu, h2 ? x0 : x1, 8);
        y += __shfl_xor_sync(0xffffffffu, y, 4);
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        if ((lane & 7) == 0) {  // lanes 0, 8, 16, 24 hold sums 0, 1, 2, 3
            double* dst = my_sacc + kk * 4 + (lane >> 3);
            if constexpr (PRIV) *dst += y;
            else atomicAdd(dst, y);
        } else if (lane == 1) {
            if constexpr (PRIV) {
                my_scnt[2 * kk] += cp;
                my_scnt[2 * kk + 1] += cr;
            } else {
                atomicAdd(my_scnt + 2 * kk, cp);
                atomicAdd(my_scnt + 2 * kk + 1, cr);
            }
        }
        __syncwarp();
    }
}

struct TcArgs {
    const double* coord;
    const int32_t* jmax;
    const int32_t* snp_block;
    int n_blocks;
    const int32_t* items;  // (n_items, 4): rows [row0, row1), partner tiles [t0, t1) of that row block
    const int* n_items;    // items in use (written with the list)
    int* item_counter;     // next unclaimed item (zero at launch)
    int nkc;               // K chunks of 128 bytes
    int kofs[LDK_MAX_POPS + 1];
    int max_n;             // largest population (reciprocal table size - 1)
    BinEdges edges;
    unsigned long long* fx;  // fixed-point bin sums [block][bin][NS + 1][kFxLimbs] (r^2 last)
    unsigned long long* pairs;
    unsigned long long* r2_counts;
    unsigned* status;
    int slots;              // bootstrap blocks staged per row block (1 without snp_block)
    int stages;             // ring stages
    int frows;              // staging rows per epilogue warp of the bin flush
    int dense;              // DN: an item of fewer partners per bin flushes lane by lane
    const double4* rtab_g;  // haplotype path: reciprocal table in global memory, or null when
                            // each CTA builds it in shared memory
    const double4* gtab;    // genotype path: reciprocal table in global memory
};

// Shared-memory state of the persistent pipeline (one CTA).
struct Pipe {
    uint32_t stages;  // shared address of the ring
    uint64_t* full_bar;
    uint64_t* empty_bar;
    uint64_t* tfull;
    uint64_t* tempty;
    uint64_t* ifull;
    uint64_t* iempty;
    volatile int* ring;  // [kRing] claimed items, then [kRing] their tile counts
    volatile int* abort_s;
};

// Item `item`: rows [row0, row1) and the partner tiles [t0, t1) of that row block, t1
// clipped to the row block's tiles (partners up to jmax[row1 - 1]).  Returns the number of
// tiles; the first starts at partner jt0.  The items of one row block partition its tile
// indices (its last item runs to INT32_MAX), so every tile is counted once whatever the
// partner range is when the kernel runs.
template <class C>
LDK_DEV int item_tiles(const TcArgs& a, int item, int& row0, int& row1, int& jt0) {
    const int4 it = reinterpret_cast<const int4*>(a.items)[item];
    row0 = it.x;
    row1 = it.y;
    const int jend = a.jmax[row1 - 1];
    const int n_jt = jend > row0 + 1 ? (jend - row0 + C::NJ - 1) / C::NJ : 0;
    const int te = it.w < n_jt ? it.w : n_jt;
    jt0 = row0 + it.z * C::NJ;
    return te > it.z ? te - it.z : 0;
}

// TMA loads of K chunk c of a row block into `dst`, signalled on `bar`.
template <class C, bool QR>
LDK_DEV void load_rows(uint32_t dst, const CUtensorMap* tmA, uint64_t* bar, int c, int row0) {
    if constexpr (QR) {  // box {128 k, 8 SNPs, 2 planes}: one group of sixteen rows
#pragma unroll
        for (int g = 0; g < C::ROWS / 8; ++g) tma_load_3d(dst + g * 16 * kKChunk, tmA, bar, c * kKChunk, row0 + 8 * g, 0);
    } else {
#pragma unroll
        for (int x = 0; x < C::REGIONS; ++x) tma_load_3d(dst + x * C::A_BOX, tmA, bar, c * kKChunk, x, row0);
    }
}

// MMAs of K chunk c (staged at a_addr) into accumulator buffer buf.
template <class C, int P>
LDK_DEV void issue_mmas(uint32_t tmem, const TcArgs& a, uint32_t a_addr, int c, uint32_t buf, uint32_t one) {
    constexpr uint32_t idesc = idesc_s8<C::N>();
    const uint32_t b_addr = a_addr + C::A_BYTES;
#pragma unroll
    for (int ks = 0; ks < kKChunk / 32; ++ks) {
        const int kbyte = c * kKChunk + ks * 32;
        int p = 0;
#pragma unroll
        for (int q = 1; q < P; ++q) p += (kbyte >= a.kofs[q]) ? 1 : 0;
        const uint32_t first = (kbyte == a.kofs[p]) ? 1u : 0u;
#pragma unroll
        for (int x = 0; x < C::REGIONS; ++x) {
            const uint32_t d = tmem + buf * C::COLS + (p * C::REGIONS + x) * C::N;
            mma_i8_one(d, sw128_desc(a_addr + x * C::A_BOX + ks * 32), sw128_desc(b_addr + ks * 32), idesc, first ^ 1u, one);
        }
    }
}

// Warp 0: claims work items from the global counter, publishes each with its tile count
// through the ring and issues the TMA loads of every partner tile's K chunks.
template <class C, bool QR>
LDK_DEV void run_producer(const Pipe& S, const CUtensorMap* tmA, const CUtensorMap* tmB, const TcArgs& a,
                          int lane) {
    if (lane == 0) {
        const int nst = C::MORE_STAGES ? a.stages : C::STAGES;
        int s = 0;        // ring stage and its phase
        uint32_t ph = 0;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            // claim the next item and publish it to the MMA issuer and the epilogue
            const int sl = k % kRing;
            if (!mbar_wait(&S.iempty[sl], ((k / kRing) & 1u) ^ 1u, S.abort_s, a.status)) { ok = false; break; }
            int item = atomicAdd(a.item_counter, 1);
            if (item >= *a.n_items) item = -1;
            int row0 = 0, row1 = 0, jt0 = 0, n_jt = 0;
            if (item >= 0) n_jt = item_tiles<C>(a, item, row0, row1, jt0);
            S.ring[sl] = item;
            S.ring[kRing + sl] = n_jt;
            mbar_arrive(&S.ifull[sl]);
            if (item < 0) break;
            for (int t = 0; t < n_jt && ok; ++t) {
                for (int c = 0; c < a.nkc; ++c) {
                    if (!mbar_wait(&S.empty_bar[s], ph ^ 1u, S.abort_s, a.status)) { ok = false; break; }
                    const uint32_t dst = S.stages + s * C::STAGE_BYTES;
                    mbar_expect_tx(&S.full_bar[s], C::STAGE_BYTES);
                    load_rows<C, QR>(dst, tmA, &S.full_bar[s], c, row0);
                    tma_load_3d(dst + C::A_BYTES, tmB, &S.full_bar[s], c * kKChunk, 0, jt0 + t * C::NJ);
                    if (++s == nst) { s = 0; ph ^= 1u; }
                }
            }
        }
        if (!ok) spin_ns(2000000);  // let copies already issued land before teardown
    }
    __syncwarp();
}

// Warp 1: the MMAs of every tile into the double-buffered accumulators.  The whole warp runs the
// loop, one elected lane issues: in code that only one lane runs, every MMA's descriptors went
// through vector registers, and issuing took longer than the small MMAs themselves (a tile of
// 48 MMAs with N = 48 3,680 -> 2,170 cycles, near the 48 each that the tensor core takes for
// N <= 64; 500 diploids x 100,000 SNPs 3.33 -> 3.11 ms, two haplotype populations 4.95 -> 4.82).
template <class C, int P>
LDK_DEV void run_mma(const Pipe& S, uint32_t tmem, const TcArgs& a) {
    const int nst = C::MORE_STAGES ? a.stages : C::STAGES;
    const uint32_t one = elect_one();
    int s = 0;
    uint32_t ph = 0, buf = 0, tph = 0;
    bool ok = true;
    for (uint32_t k = 0; ok; ++k) {
        const int sl = k % kRing;
        if (!__all_sync(0xffffffffu, mbar_wait(&S.ifull[sl], (k / kRing) & 1u, S.abort_s, a.status))) { ok = false; break; }
        const int item = __shfl_sync(0xffffffffu, S.ring[sl], 0), n_jt = __shfl_sync(0xffffffffu, S.ring[kRing + sl], 0);
        if (one) mbar_arrive(&S.iempty[sl]);
        __syncwarp();
        if (item < 0) break;
        for (int t = 0; t < n_jt && ok; ++t) {
            if (!__all_sync(0xffffffffu, mbar_wait(&S.tempty[buf], tph ^ 1u, S.abort_s, a.status))) { ok = false; break; }
            tc_fence_after();
            for (int c = 0; c < a.nkc; ++c) {
                if (!__all_sync(0xffffffffu, mbar_wait(&S.full_bar[s], ph, S.abort_s, a.status))) { ok = false; break; }
                tc_fence_after();
                issue_mmas<C, P>(tmem, a, S.stages + s * C::STAGE_BYTES, c, buf, one);
                mma_commit_one(&S.empty_bar[s], one);
                if (++s == nst) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            mma_commit_one(&S.tfull[buf], one);
            if (++buf == C::NBUF) { buf = 0; tph ^= 1u; }
        }
    }
    if (!ok) spin_ns(2000000);
    __syncwarp();
}

// GT: the haplotype path's reciprocal table is read from the workspace (a.rtab_g) instead of
// being built in shared memory -- a compile-time choice, so that the shared-memory form keeps
// its hot loop unchanged.
// CNT: populations of more than kSpinMaxN, where the spin forms are no longer exact; the
// statistics come from the counts behind the moments.  Loads and MMAs of so many haplotypes hide
// most of the raw calls' extra FP64 operations: 6,000 haplotypes x 20,000 SNPs 3.33 ms with the spin
// forms, 3.36 with this; 100,000 x 1,000 0.523, 0.527; 6,000 + 6,000 x 4,000 0.84, 0.86; genotypes,
// whose raw calls are long polynomials, 20,000 x 2,000 0.43, 0.47, 6,000 + 60 + 60 x 2,000 0.45, 0.80.
// DN: items whose bins hold few partners (dense_partners) have a tile loop of their own, whose flush
// adds lane by lane.
template <int P, bool PRIV, bool GENO, int V, bool GT, bool CNT, bool DN, bool IL>
__global__ void __launch_bounds__(Cfg<P, GENO, V>::THREADS, 1)
    k_parse_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcArgs a) {
    using C = Cfg<P, GENO, V, IL>;
    constexpr int NS = C::NS;
    constexpr int EPI = C::EPI;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int nb = a.edges.n_bins;
    const int slots = a.slots;
    unsigned char* stages = base;
    constexpr int NCOPY = PRIV ? EPI : 1;  // staging copies: one per epilogue warp, or shared
    double* sacc = reinterpret_cast<double*>(stages + a.stages * C::STAGE_BYTES);  // [NCOPY][slots][nb][NS+1]
    unsigned* scnt = reinterpret_cast<unsigned*>(sacc + NCOPY * slots * nb * (NS + 1));  // [NCOPY][slots][nb][2]
    // reciprocals of the valid counts [max_n + 1] (one population reads the last one only)
    using Recip = typename C::Recip;
    Recip* rtab = reinterpret_cast<Recip*>(scnt + ((NCOPY * slots * nb * 2 + 7) & ~7));
    double* fstage = reinterpret_cast<double*>(rtab + (GENO || GT ? 0 : (a.max_n + 2) & ~1));  // [EPI][frows][FROW]

    __shared__ __align__(8) uint64_t full_bar[C::MAX_STAGES], empty_bar[C::MAX_STAGES], tfull[C::NBUF], tempty[C::NBUF];
    __shared__ __align__(8) uint64_t ifull[kRing], iempty[kRing];
    __shared__ volatile int ring[2 * kRing];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    __shared__ double sedges[LDK_MAX_BINS + 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < C::NBUF; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], EPI);
        }
        for (int b = 0; b < kRing; ++b) {
            mbar_init(&ifull[b], 1);
            mbar_init(&iempty[b], 1 + EPI);  // the MMA issuer and every epilogue warp
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) sedges[b] = a.edges.e[b];
    for (int idx = threadIdx.x; idx < NCOPY * slots * nb * (NS + 1); idx += blockDim.x) sacc[idx] = 0.0;
    for (int idx = threadIdx.x; idx < NCOPY * slots * nb * 2; idx += blockDim.x) scnt[idx] = 0u;
    if constexpr (!GENO && !GT)
        for (int idx = threadIdx.x; idx <= a.max_n; idx += blockDim.x) {
            if constexpr (P == 1) rtab[idx] = recip_entry(idx).w;
            else rtab[idx] = recip_entry(idx);
        }
    if (warp == 1) {
        tmem_alloc(&tmem_base_s, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const Pipe pipe{su32(stages), full_bar, empty_bar, tfull, tempty, ifull, iempty, ring, &abort_s};
    // Each side changes its register budget once, at its start, and never back: warpgroup
    // 0 releases registers (setmaxnreg.dec never waits) and the epilogue warps take them
    // (setmaxnreg.inc waits only for that release, which comes unconditionally first).
    // No later increase exists that could wait on registers another warp holds -- a
    // restore to the launch count by warpgroup 0, whose idle warps would reach it at once,
    // could take the registers back before the epilogue's increase and starve it.  The
    // code both sides share, the teardown below, fits the smaller budget.  Neither the
    // roles nor the teardown may call a function (printf, a non-inlined helper): a
    // callee's registers are not bounded by the budget, and a call from a warp holding
    // 24 registers raised an illegal-instruction fault.
    if (warp < C::W0) {
        if constexpr (C::SPLIT) setmaxnreg_dec<C::REG_CTRL>();
        if (warp == 0) run_producer<C, C::QROWS>(pipe, &tmA, &tmB, a, lane);
        else if (warp == 1) run_mma<C, P>(pipe, tmem, a);
    } else {
        if constexpr (C::SPLIT) setmaxnreg_inc<C::REG_EPI>();
        // ------------------------------------------------------------- epilogue
        const int e = warp - C::W0, quarter = warp & 3;
        const int unit = e >> 2;  // this warp among its lane quarter's
        constexpr bool SSPL = C::SSPL;
        constexpr int K = C::K, NA = C::NA;
        const int half = C::QROWS ? unit & 1 : 0;  // which eight SNPs of the quarter's sixteen
        const int rest = C::QROWS ? unit >> 1 : unit;
        const int part = SSPL ? rest : 0, share = SSPL ? 0 : rest;
        // SNP r of the row block and partner jb + stride * step of a tile
        const int r = C::QROWS ? quarter * 16 + half * 8 + (lane >> 2)
                      : GENO   ? quarter * 32 + lane
                               : (quarter * 32 + lane) >> 1;
        const int role = (GENO || C::QROWS) ? 0 : lane & 1;
        constexpr int JSTRIDE = GENO ? 1 : C::QROWS ? 4 : 2;
        const int q0 = share * C::MY_STEPS;
        const int jb = JSTRIDE * q0 + (GENO ? 0 : lane & (JSTRIDE - 1));
        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32 + half * 16) << 16) +
                               (uint32_t)q0 * (C::QROWS ? 8 : 4);
        const int stage_n = slots * nb * (NS + 1);
        const int copy = PRIV ? e : 0;
        double* my_sacc = sacc + copy * stage_n;
        unsigned* my_scnt = scnt + copy * slots * nb * 2;
        double* my_fst = fstage + e * a.frows * C::FROW;
        uint32_t tcount = 0;
        for (uint32_t k = 0;; ++k) {
            const int sl = k % kRing;
            int item = -1;
            if (lane == 0) {
                if (mbar_wait(&ifull[sl], (k / kRing) & 1u, &abort_s, a.status)) {
                    item = ring[sl];
                    mbar_arrive(&iempty[sl]);
                }
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (epi_bar_or<EPI>(abort_s != 0 || item < 0)) break;
            // the item's tiles [tb, te) of row block [row0, row1) (as item_tiles; scalar loads
            // and a loop over tile indices keep this 240-register epilogue free of spills)
            const int row0 = a.items[4 * item], row1 = a.items[4 * item + 1];
            const int jend = a.jmax[row1 - 1];
            const int n_full = jend > row0 + 1 ? (jend - row0 + C::NJ - 1) / C::NJ : 0;
            const int tw = a.items[4 * item + 3];
            const int tb = a.items[4 * item + 2];
            const int te = tw < n_full ? tw : n_full;
            if (te <= tb) continue;
            const int i = row0 + r;
            bool row_ok = i < row1;
            const double ci = row_ok ? a.coord[i] : 0.0;
            const int blk0 = a.snp_block ? a.snp_block[row0] : 0;
            int slot = 0;
            if (row_ok && a.snp_block) {
                slot = a.snp_block[i] - blk0;
                if (slot < 0 || slot >= slots) {
                    atomicOr(a.status, LDK_DEVERR_BLOCK_SPAN);
                    row_ok = false;
                }
            }
            // partners i < j < jmax[i]: j - i - 1 < span as unsigned numbers
            const unsigned span = row_ok ? (unsigned)(a.jmax[i] - i - 1) : 0u;
            // Sums of the current bin live in registers.  Partners come in increasing j,
            // so the distance to them never decreases and each (row, bin) run is flushed
            // to shared memory once, when the lane's next partner falls past the bin's
            // upper edge (held in `nxt`).
            auto run_tiles = [&](auto dense_c) {
            constexpr bool DENSE = decltype(dense_c)::value;
            double acc[NA];
            // statistic s of this warp's accumulators and where it goes in the staging row
            const int na = SSPL ? (part == 0 ? K : NS + 1 - K) : NS + 1;
            const int gofs = SSPL && part == 1 ? K : 0;
#pragma unroll
            for (int s = 0; s < NA; ++s) acc[s] = 0.0;
            unsigned np = 0, nr2 = 0;
            [[maybe_unused]] double pacc[C::LATE ? NA : 1];  // LATE: sums of the bin this lane left last
            [[maybe_unused]] unsigned pnp = 0, pnr2 = 0;
            [[maybe_unused]] int pkey = 0;
            int cur = -1;
            bool in_bin = false;  // 0 <= cur < nb
            double nxt = sedges[0];
            // Adds lanes' sums into the staged sums; called by all 32 lanes.  With more than one
            // population they go into rows of the warp's scratch (all lanes of a batch at
            // once), and for every (block, bin) among the rows the warp adds the rows that hold
            // it, lane s taking value s.  One lane per round adding its own 46 values took one
            // pass per lane of a key -- on average 6.5 for 200 windows x 3 populations, 39.5 ->
            // 32.4 ms with eight rows of odd stride (four rows: 33.5; rows added one after the
            // other: 33.4); with shared staging (atomics) two genotype populations 2.77 -> 1.07
            // ms, four haplotype 4.72 -> 2.32.  With PRIV every epilogue warp owns its staged
            // sums and plain adds suffice; otherwise the warps share them (atomics).  The pairs
            // are counted by the first of two warps that share them.
            int used = 0;  // rows of the scratch that wait
            auto drain = [&]() {
                constexpr int VPL = (NA + 31) / 32;  // values per lane; lane 31 also adds the counts
                constexpr int RB = C::FROWS_MAX;
                __syncwarp();
                // lane r knows row r's key; one pass per key adds the rows that hold it
                const int my_key = lane < used ? *reinterpret_cast<const int*>(my_fst + lane * C::FROW + NA + 1) : -1;
                unsigned left = (1u << used) - 1u;
                while (left) {
                    const int kk = __shfl_sync(0xffffffffu, my_key, __ffs(left) - 1);
                    const unsigned grp = __ballot_sync(0xffffffffu, my_key == kk);
                    left &= ~grp;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        const int s = lane + 32 * v;
                        if (s < na) {
                            double* dst = my_sacc + kk * (NS + 1) + gofs + s;
                            double d = PRIV ? *dst : 0.0;
#pragma unroll
                            for (int rr = 0; rr < RB; ++rr)
                                if ((grp >> rr) & 1u) d += my_fst[rr * C::FROW + s];
                            if constexpr (PRIV) *dst = d;
                            else atomicAdd(dst, d);
                        }
                    }
                    if (part == 0 && lane == 31) {
                        unsigned* dst = my_scnt + 2 * kk;
                        uint2 dc = PRIV ? make_uint2(dst[0], dst[1]) : make_uint2(0u, 0u);
#pragma unroll
                        for (int rr = 0; rr < RB; ++rr)
                            if ((grp >> rr) & 1u) {
                                const uint2 c = *reinterpret_cast<const uint2*>(my_fst + rr * C::FROW + NA);
                                dc.x += c.x;
                                dc.y += c.y;
                            }
                        if constexpr (PRIV) {
                            dst[0] = dc.x;
                            dst[1] = dc.y;
                        } else {
                            atomicAdd(dst, dc.x);
                            atomicAdd(dst + 1, dc.y);
                        }
                    }
                }
                __syncwarp();
                used = 0;
            };
            auto add = [&](bool want, bool last, const double* acc, unsigned np, unsigned nr2, int key) {
                const unsigned mask = __ballot_sync(0xffffffffu, want);
                if constexpr (P == 1 && !DENSE) flush_one_pop<PRIV>(mask, key, acc, np, nr2, my_sacc, my_scnt, lane);
                const int rank = __popc(mask & ((1u << lane) - 1u)), total = __popc(mask);
                if constexpr (P > 1 || DENSE) {
                if (DENSE || (!DN && a.frows == 0)) {  // one lane per (block, bin) at a time
                    const unsigned grp = __match_any_sync(0xffffffffu, want ? key : -1);
                    const int turn = __popc(grp & ((1u << lane) - 1u));
                    const int turns = PRIV ? (int)__reduce_max_sync(0xffffffffu, want ? (unsigned)__popc(grp) : 0u) : 1;
                    double* dst = my_sacc + key * (NS + 1) + gofs;
                    unsigned* cnt = my_scnt + 2 * key;
                    for (int rr = 0; rr < turns; ++rr) {
                        if (want && (!PRIV || turn == rr)) {
#pragma unroll
                            for (int s = 0; s < NA; ++s)
                                if (!SSPL || s < na) {
                                    if constexpr (PRIV) dst[s] += acc[s];
                                    else atomicAdd(dst + s, acc[s]);
                                }
                            if (part == 0) {
                                if constexpr (PRIV) {
                                    cnt[0] += np;
                                    cnt[1] += nr2;
                                } else {
                                    atomicAdd(cnt, np);
                                    atomicAdd(cnt + 1, nr2);
                                }
                            }
                        }
                        __syncwarp();
                    }
                    return;
                }
                if constexpr (!DENSE) {
                int b0 = 0;
                do {
                    const int rows = total - b0 < a.frows - used ? total - b0 : a.frows - used;
                    if (want && rank >= b0 && rank < b0 + rows) {
                        double* row = my_fst + (used + rank - b0) * C::FROW;
#pragma unroll
                        for (int s = 0; s < NA; ++s)
                            if (!SSPL || s < na) row[s] = acc[s];
                        *reinterpret_cast<uint2*>(row + NA) = make_uint2(np, nr2);
                        *reinterpret_cast<int*>(row + NA + 1) = key;
                    }
                    used += rows;
                    b0 += rows;
                    if (!C::PEND || used == a.frows || (last && b0 == total)) drain();
                } while (b0 < total);
                }
                }
            };
            auto flush = [&](bool want, bool last) {
                if constexpr (C::LATE) {
                    if (__ballot_sync(0xffffffffu, want && pnp > 0)) {
                        add(pnp > 0, false, pacc, pnp, pnr2, pkey);
                        pnp = 0;
                    }
                    if (want) {
#pragma unroll
                        for (int s = 0; s < NA; ++s) pacc[s] = acc[s];
                        pnp = np;
                        pnr2 = nr2;
                        pkey = slot * nb + cur;
                    }
                    if (last) add(pnp > 0, true, pacc, pnp, pnr2, pkey);
                } else {
                    add(want, last, acc, np, nr2, slot * nb + cur);
                }
            };
            // One TMEM read per step, indexed with constants only so the counts stay in
            // registers.  (Issuing the next step's read before this step's estimators, so that
            // it lands under them, measured slower: the raw counts held across the estimators
            // cost the scheduler registers -- 200 windows x 3 populations 35.0 -> 37.4 ms, two
            // populations spilled.)
            constexpr int CREGS = (C::NJ + 31) / 32;  // partner coordinates per lane
            constexpr int U = C::U;
            bool ok = true;
            for (int t = tb; t < te; ++t, ++tcount) {
                const uint32_t buf = tcount % C::NBUF, tph = (tcount / C::NBUF) & 1u;
                const int j0 = row0 + t * C::NJ;
                double creg[CREGS];  // partner coordinates of this tile, one per lane and register
#pragma unroll
                for (int kk = 0; kk < CREGS; ++kk) {
                    const int j = j0 + 32 * kk + lane;
                    creg[kk] = (32 * kk + lane < C::NJ && j < jend) ? a.coord[j] : 0.0;
                }
                if (!mbar_wait(&tfull[buf], tph, &abort_s, a.status)) { ok = false; break; }
                tc_fence_after();
#pragma unroll 1
                for (int qq = 0; qq < C::MY_STEPS; qq += U) {
                    uint32_t v[U][P][C::REGIONS][4];
                    double dist[U];
                    bool valid[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int p = 0; p < P; ++p)
#pragma unroll
                            for (int x = 0; x < C::REGIONS; ++x) {
                                const uint32_t ta = tbase + buf * C::COLS + (p * C::REGIONS + x) * C::N +
                                                    (qq + u) * (C::QROWS ? 8 : 4);
                                if constexpr (C::QROWS) tmem_ld_q(ta, v[u][p][x]);
                                else tmem_ld4(ta, v[u][p][x]);
                            }
                    bool any = false;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int jj = jb + JSTRIDE * (qq + u);
                        double csrc = creg[0];
#pragma unroll
                        for (int kk = 1; kk < CREGS; ++kk)
                            if ((jj >> 5) == kk) csrc = creg[kk];
                        dist[u] = fabs(__shfl_sync(0xffffffffu, csrc, jj & 31) - ci);
                        valid[u] = (unsigned)(j0 + jj - i - 1) < span;
                        any |= valid[u] && dist[u] >= nxt;
                    }
                    const bool change = __ballot_sync(0xffffffffu, any) != 0u;
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int p = 0; p < P; ++p) tmem_wait4<C::REGIONS>(v[u][p]);
                    SpinPop f[U][P];
                    int nval[U][P];
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int p = 0; p < P; ++p) {
                            SpinPop& m = f[u][p];
                            if constexpr (GENO) {
                                // G[x][y]: plane x of SNP i . plane y of SNP j (0: sigma,
                                // 1: sigma^2, 2: valid)
                                const uint32_t (&G)[3][4] = v[u][p];
                                m.R = i2d_exact((int)G[0][0]);
                                m.STT = i2d_exact((int)G[0][1]);
                                m.S = i2d_exact((int)G[0][2]);
                                m.SST = i2d_exact((int)G[1][0]);
                                m.SSTT = i2d_exact((int)G[1][1]);
                                m.SS = i2d_exact((int)G[1][2]);
                                m.T = i2d_exact((int)G[2][0]);
                                m.TT = i2d_exact((int)G[2][1]);
                                nval[u][p] = (int)G[2][2];
                            } else if constexpr (C::QROWS) {
                                m.R = i2d_exact((int)v[u][p][0][0]);
                                m.S = i2d_exact((int)v[u][p][0][1]);
                                m.T = i2d_exact((int)v[u][p][0][2]);
                                nval[u][p] = (int)v[u][p][0][3];
                            } else {
                                // lane 2r: (R, S) of partners 2q, 2q+1; lane 2r+1: (T, n)
                                const uint32_t* w = v[u][p][0];
                                const uint32_t rx = __shfl_xor_sync(0xffffffffu, role ? w[0] : w[2], 1);
                                const uint32_t ry = __shfl_xor_sync(0xffffffffu, role ? w[1] : w[3], 1);
                                m.R = i2d_exact((int)(role ? rx : w[0]));
                                m.S = i2d_exact((int)(role ? ry : w[1]));
                                m.T = i2d_exact((int)(role ? w[2] : rx));
                                nval[u][p] = (int)(role ? w[3] : ry);
                            }
                        }
                    if (qq == C::MY_STEPS - U) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&tempty[buf]);
                    }
                    auto evaluate = [&](int u, bool counts) {  // pair u into the current bin's sums
#pragma unroll
                        for (int p = 0; p < P; ++p) {
                            SpinPop& m = f[u][p];
                            m.n = i2d_exact(nval[u][p]);
                            if constexpr (GENO) spin_reciprocals(m, a.gtab[nval[u][p]]);
                            else if constexpr (GT) spin_reciprocals(m, a.rtab_g[nval[u][p]]);
                            else if constexpr (P == 1) m.r4 = rtab[nval[u][p]];
                            else spin_reciprocals(m, rtab[nval[u][p]]);
                            if (U > 1 && !counts) m.r1 = m.r2 = m.r3 = m.r4 = 0.0;
                        }
                        if constexpr (CNT) {  // called for counted pairs only
                            if constexpr (!SSPL) count_stats<P, GENO, 0>(f[u], acc, nr2);
                            else if (part == 0) count_stats<P, GENO, 1>(f[u], acc, nr2);
                            else count_stats<P, GENO, 2>(f[u], acc, nr2);
                        } else if constexpr (SSPL) {
                            if (part == 0) spin_stats<P, GENO, 1>(f[u], counts, acc, nr2);
                            else spin_stats<P, GENO, 2>(f[u], counts, acc, nr2);
                        } else {
                            spin_stats<P, GENO, 0>(f[u], counts, acc, nr2);
                        }
                        np += counts;
                    };
                    if (U > 1 && !CNT && !DENSE && !change) {
                        // every pair stays in its lane's bin: evaluated together, without branches
#pragma unroll
                        for (int u = 0; u < U; ++u) evaluate(u, valid[u] && in_bin);
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const bool step = valid[u] && dist[u] >= nxt;
                            if (U == 1 ? change : __ballot_sync(0xffffffffu, step) != 0u) {
                                const bool want = step && in_bin && np > 0;
                                if (__ballot_sync(0xffffffffu, want)) flush(want, false);
                                if (step) {
                                    cur = bin_advance(sedges, nb, cur, dist[u]);
                                    nxt = cur < nb ? sedges[cur + 1] : CUDART_INF;
                                    in_bin = (unsigned)cur < (unsigned)nb;
#pragma unroll
                                    for (int s = 0; s < NA; ++s) acc[s] = 0.0;
                                    np = nr2 = 0;
                                }
                            }
                            if (valid[u] && in_bin) evaluate(u, true);
                        }
                    }
                }
            }
            flush(in_bin && np > 0, true);
            (void)ok;
            };
            bool dense = false;
            if constexpr (DN) {  // the first row's partners and the bins up to its last one
                const int last = a.jmax[row0] - 1;
                const double far = fabs(a.coord[last] - a.coord[row0]);
                int bins = __popc(__ballot_sync(0xffffffffu, lane < nb && far >= sedges[lane]));
                if (nb > 32) bins += __popc(__ballot_sync(0xffffffffu, lane + 32 < nb && far >= sedges[lane + 32]));
                dense = last - row0 < (int64_t)a.dense * bins || a.frows == 0;
                if (dense) run_tiles(std::true_type{});
            }
            if (!dense) run_tiles(std::false_type{});
            // staging -> global, once per work item
            epi_bar<EPI>();
            const int et = threadIdx.x - 32 * C::W0;
            for (int idx = et; idx < stage_n; idx += 32 * EPI) {
                double val = 0.0;
#pragma unroll
                for (int w = 0; w < NCOPY; ++w) {
                    val += sacc[w * stage_n + idx];
                    sacc[w * stage_n + idx] = 0.0;
                }
                const int sl = idx / (nb * (NS + 1));
                const int rem = idx % (nb * (NS + 1));
                const int bb = rem / (NS + 1), s = rem % (NS + 1);
                const int blk = blk0 + sl;
                if (val != 0.0 && (unsigned)blk < (unsigned)a.n_blocks)  // others: reported by pair_range
                    fx_add(a.fx + (((int64_t)blk * nb + bb) * (NS + 1) + spin_stat<P, GENO>(s)) * kFxLimbs,
                           CNT ? val : val * spin_weight<P, GENO>(s), a.status);
            }
            for (int idx = et; idx < slots * nb; idx += 32 * EPI) {
                unsigned long long c0 = 0, c1 = 0;
#pragma unroll
                for (int w = 0; w < NCOPY; ++w) {
                    unsigned* sc = scnt + w * slots * nb * 2;
                    c0 += sc[2 * idx];
                    c1 += sc[2 * idx + 1];
                    sc[2 * idx] = 0u;
                    sc[2 * idx + 1] = 0u;
                }
                const int blk = blk0 + idx / nb, bb = idx % nb;
                if ((unsigned)blk < (unsigned)a.n_blocks) {
                    if (c0) atomicAdd(&a.pairs[(int64_t)blk * nb + bb], c0);
                    if (c1) atomicAdd(&a.r2_counts[(int64_t)blk * nb + bb], c1);
                }
            }
            epi_bar<EPI>();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// planes[snp][plane][k]: boxes of 128 k x plane_box planes x rows_box SNPs
// (snp_first: 128 k x rows_box SNPs x plane_box planes, coordinates in that order)
bool make_map(CUtensorMap* m, const uint8_t* planes, int64_t n_var, int ktot, int n_planes, int plane_box,
              int rows_box, bool snp_first = false) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)ktot, (cuuint64_t)n_planes, (cuuint64_t)n_var};
    cuuint64_t strides[2] = {(cuuint64_t)ktot, (cuuint64_t)ktot * n_planes};
    cuuint32_t box[3] = {(cuuint32_t)kKChunk, (cuuint32_t)plane_box, (cuuint32_t)rows_box};
    cuuint32_t estr[3] = {1, 1, 1};
    if (snp_first) {
        std::swap(dims[1], dims[2]);
        std::swap(strides[0], strides[1]);
        std::swap(box[1], box[2]);
    }
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(planes), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Shared memory of a CTA but for flush rows and further ring stages: `ncopy` staging copies of
// `slots` bootstrap blocks, `table` reciprocal table entries of `entry` bytes.
template <class C>
size_t smem_bytes(int nb, int ncopy, int slots, int table, size_t entry) {
    return 1024 + (size_t)C::STAGES * C::STAGE_BYTES + (size_t)ncopy * slots * nb * (C::NS + 1) * sizeof(double) +
           (size_t)((ncopy * slots * nb * 2 + 7) & ~7) * sizeof(unsigned) + (size_t)table * entry + 32;
}

// Whether a shape fits with `ncopy` staging copies and `table` table entries in shared memory.
// Decided for every bootstrap slot and entries of 32 bytes, whatever the call stages, and it has to
// fit as it is launched: the slots in use, the kernel's entries, its __shared__ variables.
template <class C>
bool smem_fits(const ParseShape& sh, int ncopy, int table) {
    return smem_bytes<C>(sh.n_bins, ncopy, C::SLOTS, table, sizeof(double4)) <= kMaxSmem &&
           smem_bytes<C>(sh.n_bins, ncopy, sh.slots, table, sizeof(typename C::Recip)) + C::SHARED <= kMaxSmem;
}

// Two and three haplotype populations: bytes of K from which the row block's rows are interleaved
// (Cfg::IL), and with them the table kept in the workspace.  The loads bound such parses, and the
// small boxes take about twice as long: ms with QROWS / interleaved, 16 bins, two populations x
// 6,000 SNPs: 1,000 + 1,000 haplotypes 0.375 / 0.375 (60 bins 0.47 / 0.52), 1,500 + 1,500 0.495 /
// 0.421, 3,000 + 3,000 0.866 / 0.551, 5,000 + 5,000 1.376 / 0.765; three: 400 each 0.531 / 0.546, 600
// each 0.616 / 0.593, 2,000 each x 5,000 SNPs 1.164 / 0.683.  Fewer haplotypes: QROWS, whose reads
// need no exchange between lanes (100 + 100 x 8,000 SNPs 0.444 / 0.483).
inline int interleave_k(int P) { return P == 2 ? 3072 : P == 3 ? 1920 : INT32_MAX; }

// Ring stages in `room` bytes: C::STAGES, or as many as fit (two stages of 48 KB left the MMAs of
// 2,000 haplotypes waiting 1,000 cycles a chunk for their loads; three: 20.7 -> 20.3 ms).
template <class C>
int ring_stages(size_t room) {
    const size_t n = room / C::STAGE_BYTES;
    return C::MORE_STAGES && n > (size_t)C::STAGES ? (int)std::min<size_t>(n, C::MAX_STAGES) : C::STAGES;
}

// Reciprocal table entries held in shared memory (none on the genotype path, none when the
// table lives in the workspace).
inline int smem_table(const ParseShape& sh) { return (sh.genotypes || sh.rtab_global) ? 0 : sh.max_n + 1; }

// Per-warp staging copies when they fit next to the pipeline stages.
template <int P, bool GENO, int V>
bool private_staging(const ParseShape& sh) {
    return smem_fits<Cfg<P, GENO, V>>(sh, Cfg<P, GENO, V>::EPI, smem_table(sh));
}

// Haplotype path: the reciprocal table goes to the workspace when it does not fit in shared
// memory beside the widest tile's pipeline -- with per-warp staging if that fits without
// the table (per-warp staging matters more than a shared-memory table), else beside one
// shared staging copy -- and with interleaved rows.
template <int P>
bool rtab_global_t(const ParseShape& sh) {
    using C = Cfg<P, false, 0>;
    const int t = sh.max_n + 1;
    if (sh.ktot >= interleave_k(P)) return true;
    if (smem_fits<C>(sh, C::EPI, t)) return false;
    if (smem_fits<C>(sh, C::EPI, 0)) return true;
    return !smem_fits<C>(sh, 1, t);
}

// DN: partners per bin below which an item's flush adds lane by lane.  Adding key by key or through
// scratch rows pays where many lanes leave a bin together; in bins of a few partners every lane of
// every step leaves one, with another key.  Kernel ms of 12,000 SNPs, lane by lane / the other way:
//   three populations (40 + 30 + 20 haplotypes, bootstrap blocks), 8 scratch rows, 16 bins: 1
//   partner per bin 0.095 / 0.183, 2.5 0.249 / 0.247, 5 0.54 / 0.31; 4 rows, 18 bins: 1 0.105 /
//   0.290, 2.5 0.27 / 0.43, 5 0.60 / 0.51; 2 rows, 20 bins: 1 0.11 / 0.39, 5 0.65 / 0.92, 10 0.93 /
//   0.84; 1 row, 21 bins: 75 1.24 / 1.74;
//   60 haplotypes, 64 bins: 1.6 0.073 / 0.124; 16 bins: 2.5 0.056 / 0.062, 6 0.097 / 0.064;
//   600 genotypes (10,000 SNPs), 16 bins: 2.5 0.074 / 0.143, 25 0.134 / 0.109.
template <int P, bool GENO, bool PRIV>
int dense_partners(int frows) {
    if (P == 1) return GENO ? 8 : 3;
    if (!PRIV) return 0;  // shared sums: lanes of one key would wait for one another's atomics
    return frows >= 8 ? 2 : frows == 4 ? 4 : frows == 2 ? 7 : 1 << 20;
}

template <int P, bool PRIV, bool GENO, int V, bool GT, bool CNT, bool DN, bool IL>
cudaError_t launch_parse_tc_p(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w,
                                     const ParseShape& sh, int max_items, cudaStream_t s) {
    using C = Cfg<P, GENO, V, IL>;
    // A: the row block (haplotypes: both planes of 64 SNPs, with QROWS of eight per box;
    // genotypes: one plane of 128 SNPs per box); B: every plane of NJ partners
    CUtensorMap mA, mB;
    if (!make_map(&mA, w.hv, d->n_var, sh.ktot, C::PLANES, GENO ? 1 : C::PLANES, C::QROWS ? 8 : C::ROWS, C::QROWS) ||
        !make_map(&mB, w.hv, d->n_var, sh.ktot, C::PLANES, C::PLANES, C::NJ))
        return cudaErrorInvalidValue;
    TcArgs a;
    a.coord = d->coord ? d->coord : d->pos;
    a.jmax = w.jmax;
    a.snp_block = d->snp_block;
    a.n_blocks = d->n_blocks;
    a.items = w.items;
    a.n_items = w.n_items;
    a.item_counter = w.item_counter;
    a.nkc = sh.ktot / kKChunk;
    for (int p = 0; p <= LDK_MAX_POPS; ++p) a.kofs[p] = sh.kofs[p];
    a.max_n = sh.max_n;
    a.edges.n_bins = d->n_bins;
    for (int b = 0; b <= LDK_MAX_BINS; ++b) a.edges.e[b] = b <= d->n_bins ? d->edges[b] : 0.0;
    a.fx = w.fx;
    a.pairs = reinterpret_cast<unsigned long long*>(o->pairs);
    a.r2_counts = reinterpret_cast<unsigned long long*>(o->r2_counts);
    a.status = w.status;
    a.rtab_g = static_cast<const double4*>(w.rtab);
    a.gtab = static_cast<const double4*>(w.gtab);
    const int ncopy = PRIV ? C::EPI : 1;
    // What the staging (smem_fits) leaves of shared memory goes to flush rows, then to the ring.
    a.slots = sh.slots;
    size_t other = smem_bytes<C>(d->n_bins, ncopy, a.slots, smem_table(sh), sizeof(typename C::Recip)) -
                   (size_t)C::STAGES * C::STAGE_BYTES;
    const size_t row = (size_t)C::EPI * C::FROW * sizeof(double), full = kMaxSmem - kSpareSmem;
    a.frows = C::FROWS_MAX;
    while (a.frows > 0 && other + (size_t)C::STAGES * C::STAGE_BYTES + a.frows * row > full) a.frows >>= 1;
    // two populations with one or two rows flush lane by lane (82 + 15 haplotypes x 12,000 SNPs, 64 bins of
    // 3 partners 1.75 -> 0.38 ms, of 23 2.61 -> 1.25; with four rows of 62 bins 0.28 / 0.37 in bins of
    // one partner, 1.00 / 0.85 of ten)
    if (P == 2 && PRIV && a.frows <= 2) a.frows = 0;
    a.dense = dense_partners<P, GENO, PRIV>(a.frows);
    if (a.frows > 0) other += a.frows * row + sizeof(typename C::Recip);  // they start at an even table entry
    a.stages = ring_stages<C>(full > other ? full - other : 0);
    size_t smem = other + (size_t)a.stages * C::STAGE_BYTES;
    // at least half of an SM's shared memory, so that one CTA (holding all 512 TMEM
    // columns) runs per SM
    if (smem < kMinSmem) smem = kMinSmem;
    if (smem + C::SHARED > kMaxSmem) return cudaErrorInvalidConfiguration;
    cudaError_t e =
        cudaFuncSetAttribute(k_parse_tc<P, PRIV, GENO, V, GT, CNT, DN, IL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    {
        // the register split adds up only at C::REG_LAUNCH registers per thread (any other
        // allocation would leave setmaxnreg.inc waiting) and what fits is decided with C::SHARED,
        // so a build with others is not launched
        static std::atomic<int> built{-1};  // of this build's kernel: asked for once
        if (built.load() < 0) {
            cudaFuncAttributes fa;
            e = cudaFuncGetAttributes(&fa, k_parse_tc<P, PRIV, GENO, V, GT, CNT, DN, IL>);
            if (e != cudaSuccess) return e;
            built.store((!C::SPLIT || fa.numRegs == C::REG_LAUNCH) && fa.sharedSizeBytes <= C::SHARED);
        }
        if (!built.load()) return cudaErrorInvalidKernelImage;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (max_items == 0) return cudaSuccess;
    const int grid = max_items < sms ? max_items : sms;
    k_parse_tc<P, PRIV, GENO, V, GT, CNT, DN, IL><<<grid, C::THREADS, smem, s>>>(mA, mB, a);
    return cudaGetLastError();
}


// One population count of one tile variant: per-warp or shared staging, and the reciprocal
// table in shared memory or (FP64 estimators, widest tile only) in the workspace.  Other
// variants answer cudaErrorInvalidConfiguration for a workspace table, which the tile
// autotuner reads as "does not fit this shape".
// The kernel with or without DN.  The choice inside one tile loop makes that loop 1.4 to 2.7% slower;
// two loops leave three haplotype populations (200 windows 31.8 -> 31.0 ms) and the wide genotype
// tile (500 x 100,000 2.56 -> 2.51) faster, other kernels' main loop 2 to 3% slower: those of one
// population have it from so many bins on that narrow ones are likely (38 haplotypes x 24,864 SNPs
// in 64 bins of 26 partners 0.45 -> 0.48 ms), two populations do not (16 bins of 2.5 partners take
// 0.115 ms, lane by lane 0.093).
template <int PP, bool PRIV, bool GENO, int V, bool GT, bool CNT>
cudaError_t launch_parse_tc_d(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w, const ParseShape& sh,
                              int max_items, cudaStream_t s) {
    constexpr bool always = !CNT && ((!GENO && PP == 3) || (GENO && PP == 1 && V == 1));
    if constexpr (!CNT && PP == 1 && !always)
        if (sh.n_bins > (GENO ? 24 : 32))
            return launch_parse_tc_p<PP, PRIV, GENO, V, GT, CNT, true, false>(d, o, w, sh, max_items, s);
    constexpr bool il = !GENO && GT && (PP == 2 || PP == 3);
    if constexpr (il && CNT) return launch_parse_tc_p<PP, PRIV, GENO, V, GT, CNT, always, true>(d, o, w, sh, max_items, s);
    if constexpr (il && !CNT)
        if (sh.ktot >= interleave_k(PP))
            return launch_parse_tc_p<PP, PRIV, GENO, V, GT, CNT, always, true>(d, o, w, sh, max_items, s);
    if constexpr (!(il && CNT)) return launch_parse_tc_p<PP, PRIV, GENO, V, GT, CNT, always, false>(d, o, w, sh, max_items, s);
}

template <int PP, bool GENO, int V, bool CNT>
cudaError_t launch_staged(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w, const ParseShape& sh,
                          int max_items, cudaStream_t s) {
    const bool priv = private_staging<PP, GENO, V>(sh);
    if (!GENO && sh.rtab_global) {
        if constexpr (!GENO && V == 0)
            return priv ? launch_parse_tc_d<PP, true, GENO, V, true, CNT>(d, o, w, sh, max_items, s)
                        : launch_parse_tc_d<PP, false, GENO, V, true, CNT>(d, o, w, sh, max_items, s);
        else
            return cudaErrorInvalidConfiguration;
    }
    if constexpr (!GENO && CNT) {  // a table of kSpinMaxN entries never fits in shared memory
        static_assert((size_t)kSpinMaxN * sizeof(double4) + Cfg<PP, GENO, V>::STAGES * Cfg<PP, GENO, V>::STAGE_BYTES > kMaxSmem,
                      "counted haplotypes keep their table in the workspace");
        return cudaErrorInvalidConfiguration;
    } else {
        return priv ? launch_parse_tc_d<PP, true, GENO, V, false, CNT>(d, o, w, sh, max_items, s)
                    : launch_parse_tc_d<PP, false, GENO, V, false, CNT>(d, o, w, sh, max_items, s);
    }
}

// One tile variant of one path, over the population count and staging.
template <bool GENO, int V, bool CNT = false>
cudaError_t dispatch_tc(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w, const ParseShape& sh,
                        int max_items, cudaStream_t s) {
#define LDK_TC_CASE(PP)                                                                                   \
    case PP:                                                                                              \
        return launch_staged<PP, GENO, V, CNT>(d, o, w, sh, max_items, s);
    switch (sh.P) {
        LDK_TC_CASE(1)
        LDK_TC_CASE(2)
        LDK_TC_CASE(3)
        LDK_TC_CASE(4)
        default: return cudaErrorInvalidValue;
    }
#undef LDK_TC_CASE
}

}  // namespace
}  // namespace ldk
