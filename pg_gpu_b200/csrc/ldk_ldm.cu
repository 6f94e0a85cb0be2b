// All-pairs LD of one SNP set on the tensor-core count pipeline: pairwise r^2, the
// unbiased sigma_D^2, r^2 from jointly valid counts, dosage r^2 and Rogers-Huff r for every
// pair i < j, written as a full symmetric matrix and/or reduced to the sum and count behind
// ZnS.
//
// The Gram moments come from the same TMA + tcgen05 pipeline as the binned parse (64-SNP
// row blocks against 128-SNP partner tiles, no distance cutoff, so every partner j > i of
// the set; work items of a few tiles, claimed dynamically, because the row blocks shrink
// along the triangle: whole row blocks left 148 SMs waiting for the longest).  Sixteen
// epilogue warps each take eight SNPs x 64 partners of a tile; a thread holds one SNP and
// every fourth partner and stores its value to the upper and the lower triangle straight
// from registers (32-byte and 64-byte runs).  Everything that depends on one SNP alone
// (frequency, reciprocal variance) is tabulated first, so a pair costs no division.
#include <algorithm>
#include <cmath>

#include "ldk_tc_kernel.cuh"

namespace ldk {

namespace {

using LdmCfg = Cfg<1, false, 0>;
constexpr int kLdmEpi = 16;                    // epilogue warps: four per TMEM lane quarter
constexpr int kLdmPart = LdmCfg::NJ / 2;       // partners per epilogue warp and tile
constexpr int kLdmGroup = 4;                   // steps (four partners each) in flight together
constexpr int kLdmTable = 8192;                // most entries of the 1/n table in shared memory

struct LdmArgs {
    const double2* site;  // per SNP, by estimator (k_site)
    double* out;          // (n_var rows, stride ld_out) or null
    int64_t ld_out;
    double* sums;         // [sum over pairs i < j, pairs counted] or null
};

// Per SNP over the selected rows, into site[v]:
//   LDK_LDM_R2              {p, 1 / (p (1 - p))}, p = derived / valid calls (haplotype_matrix.py:1119-1120)
//   LDK_LDM_DIPLOID_R2      {m, 1 / V}, m the mean spin (1 - dosage) of the valid calls, V their sum
//                           of squared deviations (ld_statistics.py:1000-1011)
//   LDK_LDM_ROGERS_HUFF_R   {d, 1 / sqrt(V)}, d the mean dosage
// with 0 for the reciprocal of 0; and the partner range (the rest of the set) and the matrix
// diagonal.  For the Rogers-Huff and sigma_D^2 genotype estimators, which take complete data
// (ld_statistics.py:389-399), a missing call sets LDK_DEVERR_BAD_INPUT, unless the set has no pair.
// A block takes 128 SNPs (four a lane, one word per row), its sixteen warps every sixteenth
// group of eight rows: 12,000 SNPs x 200 rows 24 us with a thread per SNP walking the rows, 13.
constexpr int kSiteWarps = 16;
__global__ void __launch_bounds__(32 * kSiteWarps)
    k_site(const int8_t* __restrict__ X, int64_t ld, int64_t n_var, const int32_t* __restrict__ rows, int n_rows,
           int estimator, double2* __restrict__ site, int32_t* __restrict__ jmax, double* __restrict__ out,
           int64_t ld_out, double diag, unsigned* status) {
    __shared__ int cnt[3][128];  // valid calls, codes 1, codes 2
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < 3 * 128; k += blockDim.x) (&cnt[0][0])[k] = 0;
    __syncthreads();
    const int64_t vq = (int64_t)blockIdx.x * 128 + 4 * lane;
    const int left = n_var - vq < 4 ? (int)(n_var - vq) : 4;
    const bool read = estimator == LDK_LDM_R2 || estimator >= LDK_LDM_DIPLOID_R2;
    if (read && left > 0) {
        int N[3][4] = {};
        for (int k0 = 8 * warp; k0 < n_rows; k0 += 8 * kSiteWarps) {
            uint32_t x[8];
#pragma unroll
            for (int b = 0; b < 8; ++b)
                x[b] = k0 + b < n_rows ? load_quad(X + (int64_t)rows[k0 + b] * ld + vq, left) : 0xFFFFFFFFu;
            uint32_t c[3] = {};
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                c[0] += ~(x[b] >> 7) & 0x01010101u;
                c[1] += __vcmpeq4(x[b], 0x01010101u) & 0x01010101u;
                c[2] += __vcmpeq4(x[b], 0x02020202u) & 0x01010101u;
            }
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int j = 0; j < 4; ++j) N[q][j] += (c[q] >> (8 * j)) & 0xFF;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (N[q][j]) atomicAdd(&cnt[q][4 * lane + j], N[q][j]);
    }
    __syncthreads();
    const int64_t v = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (threadIdx.x >= 128 || v >= n_var) return;
    const int c[3] = {cnt[0][threadIdx.x], cnt[1][threadIdx.x], cnt[2][threadIdx.x]};
    jmax[v] = (int32_t)n_var;
    if (out) out[v * ld_out + v] = diag;
    double2 r = make_double2(0.0, 0.0);
    if (estimator == LDK_LDM_R2) {
        r.x = c[0] > 0 ? (double)c[1] / (double)c[0] : 0.0;
        const double pq = r.x * (1.0 - r.x);
        r.y = pq > 0.0 ? 1.0 / pq : 0.0;
    } else if (estimator >= LDK_LDM_DIPLOID_R2) {
        if (estimator != LDK_LDM_DIPLOID_R2 && n_var > 1 && c[0] < n_rows) atomicOr(status, LDK_DEVERR_BAD_INPUT);
        // spins: 1 for dosage 0, 0 for 1, -1 for 2; V = (n sum s^2 - (sum s)^2) / n, exact numerator
        const double n = c[0], S = (double)(c[0] - c[1] - 2 * c[2]), SS = (double)(c[0] - c[1]);
        const double V = c[0] > 0 ? fma(n, SS, -(S * S)) / n : 0.0;
        if (c[0] > 0) r.x = (estimator == LDK_LDM_DIPLOID_R2 ? S : (double)(c[1] + 2 * c[2])) / n;
        if (V > 0.0) r.y = estimator == LDK_LDM_DIPLOID_R2 ? 1.0 / V : 1.0 / sqrt(V);
    }
    site[v] = r;
}

// CNT (sigma_D^2 of more than kSpinMaxN rows): the numerators from the counts, because the moment
// form's n^4 terms no longer cancel exactly there (two singletons on one haplotype of 20,000: 0 / 0
// became -16 / -16).  6,000 haplotypes x 4,000 SNPs 0.371 ms with the moment form, 0.375 with this;
// genotypes 1.157, 1.208.
template <int EST, bool CNT = false>
__global__ void __launch_bounds__(128 + 32 * kLdmEpi, 1)
    k_ld_matrix(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcArgs a,
                const LdmArgs m) {
    using C = LdmCfg;
    constexpr int NJ = C::NJ;
    constexpr bool SITE = EST == LDK_LDM_R2 || EST >= LDK_LDM_DIPLOID_R2;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* stages = base;
    double* rn = reinterpret_cast<double*>(stages + a.stages * C::STAGE_BYTES);  // EST R2: 1 / n

    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], tfull[C::NBUF], tempty[C::NBUF];
    __shared__ __align__(8) uint64_t ifull[kRing], iempty[kRing];
    __shared__ volatile int ring[2 * kRing];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < C::NBUF; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kLdmEpi);
        }
        for (int b = 0; b < kRing; ++b) {
            mbar_init(&ifull[b], 1);
            mbar_init(&iempty[b], 1 + kLdmEpi);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const bool table = EST == LDK_LDM_R2 && a.max_n < kLdmTable;
    if (table)
        for (int n = threadIdx.x; n <= a.max_n; n += blockDim.x) rn[n] = n > 0 ? 1.0 / (double)n : 0.0;
    if (warp == 1) {
        tmem_alloc(&tmem_base_s, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const Pipe pipe{su32(stages), full_bar, empty_bar, tfull, tempty, ifull, iempty, ring, &abort_s};
    if (warp == 0) run_producer<C, true>(pipe, &tmA, &tmB, a, lane);
    else if (warp == 1) run_mma<C, 1>(pipe, tmem, a);
    if (warp >= 4) {
        // thread: SNP `r` of the row block, partners jb + 4 step of the tile
        const int e = warp - 4, quarter = warp & 3, half = (e >> 2) & 1, share = e >> 3;
        const int r = quarter * 16 + half * 8 + (lane >> 2), jb = share * kLdmPart + (lane & 3);
        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32 + half * 16) << 16) + (uint32_t)share * (2 * kLdmPart);
        double zsum = 0.0;
        unsigned long long zcnt = 0;
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
            if (epi_bar_or<kLdmEpi>(abort_s != 0 || item < 0)) break;
            int row0, row1, jt0;
            const int n_jt = item_tiles<C>(a, item, row0, row1, jt0);
            if (n_jt == 0) continue;
            const int jend = a.jmax[row1 - 1];
            const int i = row0 + r;
            const bool row_ok = i < row1;
            double2 si = make_double2(0.0, 0.0);
            if (SITE && row_ok) si = m.site[i];
            bool ok = true;
            for (int t = 0; t < n_jt; ++t, ++tcount) {
                const uint32_t buf = tcount % C::NBUF, tph = (tcount / C::NBUF) & 1u;
                const int j0 = jt0 + t * NJ;
                // a tile off the diagonal, inside the matrix and of a whole row block needs no bounds
                const bool whole = row1 - row0 == C::ROWS && j0 >= row1 && j0 + NJ <= jend;
                if (!mbar_wait(&tfull[buf], tph, &abort_s, a.status)) { ok = false; break; }
                tc_fence_after();
                int j = j0 + jb;
                double* up = m.out ? m.out + (int64_t)i * m.ld_out + j : nullptr;
                double* lo = m.out ? m.out + (int64_t)j * m.ld_out + i : nullptr;
                unsigned cnt = 0;
#pragma unroll 1
                for (int q = 0; q < kLdmPart / 4; q += kLdmGroup) {
                    uint32_t v[kLdmGroup][4];
                    double2 sj[kLdmGroup];
#pragma unroll
                    for (int g = 0; g < kLdmGroup; ++g) tmem_ld_q(tbase + buf * C::COLS + (q + g) * 8, v[g]);
                    if constexpr (SITE) {
#pragma unroll
                        for (int g = 0; g < kLdmGroup; ++g)
                            sj[g] = whole || j + 4 * g < jend ? __ldg(m.site + j + 4 * g) : make_double2(0.0, 0.0);
                    }
                    tmem_wait4<kLdmGroup>(v);
                    if (q == kLdmPart / 4 - kLdmGroup) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&tempty[buf]);
                    }
#pragma unroll
                    for (int g = 0; g < kLdmGroup; ++g, j += 4) {
                        const int iR = (int)v[g][0], iS = (int)v[g][1], iT = (int)v[g][2], in = (int)v[g][3];
                        double val;
                        bool counted = true;  // enters the sum and count
                        if constexpr (EST == LDK_LDM_R2) {
                            // haplotype_matrix.py:1122-1128, 1171-1175; n11 = (n - S - T + R) / 4
                            const double c1 = i2d_exact((in - iS - iT + iR) >> 2);
                            const double r1 = table ? rn[in] : (in > 0 ? recip_cubic(i2d_exact(in)) : 0.0);
                            const double D = fma(c1, r1, -(si.x * sj[g].x));
                            val = (D * D) * (si.y * sj[g].y);
                        } else if constexpr (EST == LDK_LDM_DIPLOID_R2) {
                            // covariance of the centred spins of the jointly called individuals
                            // (centred dosages with the other sign, ld_statistics.py:1000-1018)
                            const double S = i2d_exact(iS), T = i2d_exact(iT), R = i2d_exact(iR), n = i2d_exact(in);
                            const double cov = fma(-sj[g].x, fma(-si.x, n, S), fma(-si.x, T, R));
                            val = (cov * cov) * (si.y * sj[g].y);
                        } else if constexpr (EST == LDK_LDM_ROGERS_HUFF_R) {
                            // ld_statistics.py:392-437 (complete data); NaN where a site is constant.
                            // Of dosages 1 - sigma, not spins: of rare alleles their sums are small,
                            // where R - mean mean n cancels n - n
                            const double cov = fma(-(si.x * sj[g].x), i2d_exact(in), i2d_exact(in - iS - iT + iR));
                            const double s = si.y * sj[g].y;
                            counted = s > 0.0;
                            val = counted ? cov * s : CUDART_NAN;
                        } else {
                            const double n = i2d_exact(in), S = i2d_exact(iS), T = i2d_exact(iT), R = i2d_exact(iR);
                            if constexpr (EST == LDK_LDM_SIGMA_D2) {
                                // ld_statistics.py:326-343: the DD and pi2 numerators, exact
                                // integers in FP64 (up to kSpinMaxN; 16 times each) or, from the
                                // counts, where these are small
                                double dd, pi2;
                                if constexpr (CNT)
                                    hap_numerators(i2d_exact((in - iS - iT + iR) >> 2), i2d_exact((in - iS + iT - iR) >> 2),
                                                   i2d_exact((in + iS - iT - iR) >> 2), i2d_exact((in + iS + iT + iR) >> 2),
                                                   dd, pi2);
                                else
                                    spin_hap_numerators(n, S, T, R, dd, pi2);
                                counted = in >= 4;
                                val = (counted && pi2 != 0.0) ? dd * recip_cubic(pi2) : 0.0;
                            } else {
                                // haplotype_kernels.py:32-42: NaN where pA qA pB qB = 0
                                const double E = fma(n, R, -(S * T));
                                const double den = fma(n, n, -(S * S)) * fma(n, n, -(T * T));
                                counted = den > 0.0;
                                val = counted ? (E * E) * recip_cubic(den) : CUDART_NAN;
                            }
                        }
                        const bool valid = whole || (row_ok && j > i && j < jend);
                        if (m.sums && valid && counted) {
                            zsum += EST == LDK_LDM_ROGERS_HUFF_R ? val * val : val;
                            ++cnt;
                        }
                        if (m.out) {
                            if (valid) {
                                *up = val;
                                *lo = val;
                            }
                            up += 4;
                            lo += 4 * m.ld_out;
                        }
                    }
                }
                zcnt += cnt;
            }
            (void)ok;
        }
        if (m.sums) {
            double zc = (double)zcnt;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                zsum += __shfl_xor_sync(0xffffffffu, zsum, o);
                zc += __shfl_xor_sync(0xffffffffu, zc, o);
            }
            if (lane == 0) {
                atomicAdd(&m.sums[0], zsum);
                atomicAdd(&m.sums[1], zc);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}


// ---- sigma_D^2 of genotype pairs: nine moments per pair ----------------------------------

using LdmGCfg = Cfg<1, true, 0>;               // 128-SNP row blocks, 12-partner tiles
constexpr int kLdmGEpi = 8;                    // two epilogue warps per TMEM lane quarter
constexpr int kLdmGPart = LdmGCfg::NJ / 2;     // partners per epilogue warp and tile
constexpr int kLdmGStride = kLdmGPart + 1;

struct LdmGArgs {
    double* out;
    int64_t ld_out;
    double* sums;
};

template <bool CNT>  // as for k_ld_matrix
__global__ void __launch_bounds__(128 + 32 * kLdmGEpi, 1)
    k_ld_matrix_geno(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcArgs a,
                     const LdmGArgs m) {
    using C = LdmGCfg;
    constexpr int NJ = C::NJ, SP = kLdmGStride;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* stages = base;
    double* stile = reinterpret_cast<double*>(stages + a.stages * C::STAGE_BYTES);  // [kLdmGEpi][32][SP]

    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], tfull[C::NBUF], tempty[C::NBUF];
    __shared__ __align__(8) uint64_t ifull[kRing], iempty[kRing];
    __shared__ volatile int ring[2 * kRing];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < C::NBUF; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kLdmGEpi);
        }
        for (int b = 0; b < kRing; ++b) {
            mbar_init(&ifull[b], 1);
            mbar_init(&iempty[b], 1 + kLdmGEpi);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
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
    if (warp == 0) run_producer<C, false>(pipe, &tmA, &tmB, a, lane);
    else if (warp == 1) run_mma<C, 1>(pipe, tmem, a);
    if (warp >= 4) {
        // lane = SNP of the row block (32 per warp); the warp takes half `part` of every tile
        const int e = warp - 4, quarter = warp & 3, part = e >> 2;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        double* st = stile + e * 32 * SP;
        double zsum = 0.0, zcnt = 0.0;
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
            if (epi_bar_or<kLdmGEpi>(abort_s != 0 || item < 0)) break;
            int row0, row1, jt0;
            const int n_jt = item_tiles<C>(a, item, row0, row1, jt0);
            if (n_jt == 0) continue;
            const int jend = a.jmax[row1 - 1];
            const int i = row0 + quarter * 32 + lane;
            const bool row_ok = i < row1;
            bool ok = true;
            for (int t = 0; t < n_jt; ++t, ++tcount) {
                const uint32_t buf = tcount % C::NBUF, tph = (tcount / C::NBUF) & 1u;
                const int j0 = jt0 + t * NJ;
                if (!mbar_wait(&tfull[buf], tph, &abort_s, a.status)) { ok = false; break; }
                tc_fence_after();
#pragma unroll 1
                for (int cl = 0; cl < kLdmGPart; ++cl) {
                    const int c = part * kLdmGPart + cl;
                    uint32_t G[3][4];
#pragma unroll
                    for (int x = 0; x < 3; ++x) tmem_ld4(tmem + lane_base + buf * C::COLS + x * C::N + 4 * c, G[x]);
                    const int j = j0 + c;
                    tmem_wait4<3>(G);
                    if (cl == kLdmGPart - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&tempty[buf]);
                    }
                    const bool valid = row_ok && j > i && j < jend;
                    double val = 0.0;
                    if (valid) {
                        // G[x][y]: plane x of SNP i . plane y of SNP j (0: sigma = 1 - g,
                        // 1: sigma^2, 2: valid); DD over pi2 of one population
                        // (genotype_kernels.py:91-170)
                        double dd, pi2;
                        if constexpr (CNT) {
                            const SpinPop s{i2d_exact((int)G[2][2]), i2d_exact((int)G[0][2]), i2d_exact((int)G[2][0]),
                                            i2d_exact((int)G[0][0]), i2d_exact((int)G[1][2]), i2d_exact((int)G[2][1]),
                                            i2d_exact((int)G[1][0]), i2d_exact((int)G[0][1]), i2d_exact((int)G[1][1])};
                            double c[9];
                            spin_geno_cells(s, c);
                            GenoFeat<double> f{};
                            f.w4 = 1.0;  // n(n-1)(n-2)(n-3) cancels
                            geno_set_counts(f, c);
                            geno_features<double, 1, false>(f);
                            dd = 0.25 * f.DD1;  // the genotype DD is four times the moment form's
                            pi2 = f.PI1;
                        } else {
                            spin_geno_numerators(G, dd, pi2);
                        }
                        if ((int)G[2][2] >= 4 && pi2 > 0.0) {
                            val = 4.0 * dd * recip_cubic(pi2);
                            zsum += val;
                            zcnt += 1.0;
                        } else {
                            val = CUDART_NAN;
                        }
                    }
                    st[lane * SP + cl] = val;
                }
                __syncwarp();
                if (m.out) {
                    const int gi0 = row0 + quarter * 32, gj0 = j0 + part * kLdmGPart;
                    for (int idx = lane; idx < 32 * kLdmGPart; idx += 32) {  // rows: upper triangle
                        const int r = idx / kLdmGPart, cc = idx % kLdmGPart, gi = gi0 + r, gj = gj0 + cc;
                        if (gi < row1 && gj > gi && gj < jend) m.out[(int64_t)gi * m.ld_out + gj] = st[r * SP + cc];
                    }
                    for (int idx = lane; idx < 32 * kLdmGPart; idx += 32) {  // columns: lower triangle
                        const int r = idx % 32, cc = idx / 32, gi = gi0 + r, gj = gj0 + cc;
                        if (gi < row1 && gj > gi && gj < jend) m.out[(int64_t)gj * m.ld_out + gi] = st[r * SP + cc];
                    }
                }
                __syncwarp();
            }
            (void)ok;
        }
        if (m.sums) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                zsum += __shfl_xor_sync(0xffffffffu, zsum, o);
                zcnt += __shfl_xor_sync(0xffffffffu, zcnt, o);
            }
            if (lane == 0) {
                atomicAdd(&m.sums[0], zsum);
                atomicAdd(&m.sums[1], zcnt);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

struct LdmLayout {
    size_t jmax = 0, items = 0, planes = 0, site = 0, total = 0;
    int n_row_blocks = 0, rows = 0, ktot = 0;
};

LdmLayout ldm_layout(int64_t n_var, int32_t n_sel, bool geno) {
    LdmLayout L;
    L.ktot = (int)(((n_sel + 31) / 32 * 32 + 127) / 128 * 128);
    L.rows = geno ? LdmGCfg::ROWS : LdmCfg::ROWS;
    L.n_row_blocks = (int)((n_var + L.rows - 1) / L.rows);
    auto up = [](size_t x, size_t a) { return (x + a - 1) / a * a; };
    size_t off = 256;
    L.jmax = off;
    off = up(off + (size_t)n_var * 4, 256);
    L.items = off;
    off = up(off + (size_t)tc_item_capacity(L.n_row_blocks) * 16, 1024);
    L.planes = off;
    off = up(off + (size_t)n_var * (geno ? 4 : 2) * L.ktot, 256);
    L.site = off;
    off = up(off + (size_t)n_var * sizeof(double2), 256);
    L.total = off;
    return L;
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Shared memory of a launch: `other` bytes beside the pipeline of C::STAGES stages.  (A longer
// ring takes the L1 that serves the per-SNP factors: r^2 matrix 369 -> 392 us.)
template <class C>
size_t ldm_smem(TcArgs& a, size_t other) {
    a.stages = C::STAGES;
    return other + (size_t)a.stages * C::STAGE_BYTES;
}

template <bool CNT>
cudaError_t launch_ldm_geno(const CUtensorMap& mA, const CUtensorMap& mB, TcArgs& a, const LdmGArgs& m,
                            cudaStream_t s) {
    size_t smem = ldm_smem<LdmGCfg>(a, 1024 + (size_t)kLdmGEpi * 32 * kLdmGStride * sizeof(double));
    if (smem < kMinSmem) smem = kMinSmem;
    if (smem > kMaxSmem) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaFuncSetAttribute(k_ld_matrix_geno<CNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ld_matrix_geno<CNT><<<sm_count(), 128 + 32 * kLdmGEpi, smem, s>>>(mA, mB, a, m);
    return cudaGetLastError();
}

template <int EST, bool CNT = false>
cudaError_t launch_ldm(const CUtensorMap& mA, const CUtensorMap& mB, TcArgs& a, const LdmArgs& m, cudaStream_t s) {
    size_t smem = ldm_smem<LdmCfg>(a, 1024 + (a.max_n < kLdmTable ? a.max_n + 1 : 0) * sizeof(double));
    if (smem < kMinSmem) smem = kMinSmem;
    cudaError_t e = cudaFuncSetAttribute(k_ld_matrix<EST, CNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_ld_matrix<EST, CNT><<<sm_count(), 128 + 32 * kLdmEpi, smem, s>>>(mA, mB, a, m);
    return cudaGetLastError();
}

}  // namespace

size_t ld_matrix_workspace(int64_t n_var, int32_t n_sel) {
    return std::max(ldm_layout(n_var, n_sel, true).total, ldm_layout(n_var, n_sel, false).total);
}

// Enqueues the all-pairs LD of the n_sel selected rows of X (see ldk_ld_matrix).
cudaError_t launch_ld_matrix(const int8_t* X, int64_t ld_x, int64_t n_var, const int32_t* rows, int32_t n_sel,
                             int estimator, double* out, int64_t ld_out, double* sums, unsigned char* ws,
                             unsigned* status, cudaStream_t s) {
    const bool dosage = estimator >= LDK_LDM_DIPLOID_R2;       // codes {-1, 0, 1, 2}
    const bool nine = estimator == LDK_LDM_SIGMA_D2_GENO;      // the nine-moment kernel
    const LdmLayout L = ldm_layout(n_var, n_sel, nine);
    cudaError_t e;
    if (sums && (e = cudaMemsetAsync(sums, 0, 2 * sizeof(double), s)) != cudaSuccess) return e;
    if (n_var < 1) return cudaSuccess;
    Scratch w{};
    w.status = status;
    w.jmax = reinterpret_cast<int32_t*>(ws + L.jmax);
    w.items = reinterpret_cast<int32_t*>(ws + L.items);
    w.n_items = reinterpret_cast<int*>(ws + 192);
    w.item_counter = reinterpret_cast<int*>(ws + 128);
    w.hv = ws + L.planes;
    double2* site = reinterpret_cast<double2*>(ws + L.site);
    const bool nan_diag = estimator == LDK_LDM_R2_COUNTS || estimator >= LDK_LDM_ROGERS_HUFF_R;
    k_site<<<(unsigned)((n_var + 127) / 128), 32 * kSiteWarps, 0, s>>>(X, ld_x, n_var, rows, n_sel, estimator, site, w.jmax,
                                                                    out, ld_out, nan_diag ? std::nan("") : 0.0, status);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (n_var < 2) return cudaSuccess;
    // the spin planes of the selected rows, as for a one-population parse
    ldk_parse_t d{};
    d.genotypes = dosage ? 1 : 0;
    d.X = X;
    d.ld_x = ld_x;
    d.n_var = n_var;
    d.pop_rows = rows;
    d.n_pops = 1;
    d.pop_offsets[0] = 0;
    for (int p = 1; p <= LDK_MAX_POPS; ++p) d.pop_offsets[p] = n_sel;
    ParseShape sh{};
    sh.P = 1;
    sh.genotypes = dosage ? 1 : 0;
    sh.planes = nine ? 4 : 2;
    sh.ktot = L.ktot;
    for (int p = 0; p <= LDK_MAX_POPS; ++p) sh.kofs[p] = p == 0 ? 0 : (n_sel + 31) / 32 * 32;
    sh.max_n = n_sel;
    if ((e = launch_prep_planes(&d, w, sh, nullptr, s)) != cudaSuccess) return e;
    // items of one tile at least: unlike the parse's, they end without a flush
    if ((e = launch_split_items(w, L.n_row_blocks, nine ? LdmGCfg::NJ : LdmCfg::NJ, 1, L.rows, (int)n_var, s)) !=
        cudaSuccess)
        return e;
    CUtensorMap mA, mB;
    if (nine ? (!make_map(&mA, w.hv, n_var, L.ktot, 4, 1, LdmGCfg::ROWS) ||
                !make_map(&mB, w.hv, n_var, L.ktot, 4, 4, LdmGCfg::NJ))
             : (!make_map(&mA, w.hv, n_var, L.ktot, 2, 2, 8, true) ||
                !make_map(&mB, w.hv, n_var, L.ktot, 2, 2, LdmCfg::NJ)))
        return cudaErrorInvalidValue;
    TcArgs a{};
    a.jmax = w.jmax;
    a.items = w.items;
    a.n_items = w.n_items;
    a.item_counter = w.item_counter;
    a.nkc = L.ktot / kKChunk;
    for (int p = 0; p <= LDK_MAX_POPS; ++p) a.kofs[p] = sh.kofs[p];
    a.max_n = n_sel;
    a.status = status;
    const bool counts = n_sel > kSpinMaxN;
    if (nine) {
        const LdmGArgs g{out, ld_out, sums};
        return counts ? launch_ldm_geno<true>(mA, mB, a, g, s) : launch_ldm_geno<false>(mA, mB, a, g, s);
    }
    const LdmArgs m{site, out, ld_out, sums};
    switch (estimator) {
        case LDK_LDM_R2: return launch_ldm<LDK_LDM_R2>(mA, mB, a, m, s);
        case LDK_LDM_SIGMA_D2:
            return counts ? launch_ldm<LDK_LDM_SIGMA_D2, true>(mA, mB, a, m, s) : launch_ldm<LDK_LDM_SIGMA_D2>(mA, mB, a, m, s);
        case LDK_LDM_R2_COUNTS: return launch_ldm<LDK_LDM_R2_COUNTS>(mA, mB, a, m, s);
        case LDK_LDM_DIPLOID_R2: return launch_ldm<LDK_LDM_DIPLOID_R2>(mA, mB, a, m, s);
        default: return launch_ldm<LDK_LDM_ROGERS_HUFF_R>(mA, mB, a, m, s);
    }
}

}  // namespace ldk
