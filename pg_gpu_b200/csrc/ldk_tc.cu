// Tensor-core path of the binned parse: spin-plane preparation, tile-variant
// dispatch and the peak probes (the kernel itself is in ldk_tc_kernel.cuh).
#include "ldk_tc_kernel.cuh"
#include "ldk_jmax.cuh"

namespace ldk {

namespace {
// ---------------------------------------------------------------------------
// spin planes (s8).  Haplotypes: planes[v][0][k] = sigma = 1 - 2x, planes[v][1][k] = [x in {0, 1}].
// Genotypes: planes[v][0..3][k] = sigma = 1 - x, sigma^2, [x in {0, 1, 2}], 0.  Missing: 0.
// ---------------------------------------------------------------------------

struct PrepArgs {
    const int8_t* X;
    int64_t ld;
    int64_t n_var;
    const int32_t* pop_rows;
    int pop_off[LDK_MAX_POPS + 1];
    int kofs[LDK_MAX_POPS + 1];
    int P;
    int ktot;
    uint8_t* planes_out;
    unsigned* status;
    int64_t nx;  // SNP tiles
    int ny;      // K tiles, and one more slice for a parse's other preparations (slice < 0: none)
    int slice;
    JmaxArgs ranges;
    unsigned long long* zero[3];  // accumulators to clear and their 64-bit words
    int64_t zero_n[3];
    double4* table;  // reciprocal table in the workspace, or null
    int table_n;
};  // X: int8 codes, or (PACKED) 2-bit codes + 1, four SNPs per byte (LDK_X_PACKED2)

constexpr int kPrepV = 128, kPrepK = 128;
// Blocks run in groups of eight SNP tiles x all K tiles: what is in flight together then reads
// rows of X in runs of a kilobyte and completes whole rows of planes.  2,000 haplotypes x 10^6
// SNPs (2 GB read, 4 GB written, DRAM the bound): K tile by K tile 2.2 ms, in groups 1.85, and
// with the sixteen-row gather below 1.2 (5 TB/s).
constexpr int kPrepGroup = 8;

// Pair ranges of the block's 128 SNPs (first half of the threads); zeroed accumulators and the
// reciprocal table (second half).
template <bool GENO>
LDK_DEV void prepare_rest(const PrepArgs& a, int64_t bx) {
    if (threadIdx.x < 128) {
        const int64_t i = bx * 128 + threadIdx.x;
        if (i < a.n_var) pair_range(a.ranges, i);
        return;
    }
    const int64_t t = bx * 128 + threadIdx.x - 128, step = a.nx * 128;
#pragma unroll
    for (int z = 0; z < 3; ++z)
        for (int64_t k = t; k < a.zero_n[z]; k += step) a.zero[z][k] = 0ull;
    for (int64_t k = t; k < a.table_n; k += step) a.table[k] = GENO ? recip_entry_geno((int)k) : recip_entry((int)k);
}

// One block: 128 K positions (haplotypes / individuals) x 128 SNPs.  The rows of the 128 K
// positions are resolved once; the gather reads 128-byte row segments of X (a lane four
// consecutive SNPs) into a SNP-major shared tile, the scatter turns sixteen K positions of a SNP
// into their plane bytes and writes every plane as 128-byte runs along K.  Plane bytes (GENO: 4
// planes, haplotypes: 2):
//   haplotypes  sigma = 1 - 2x, v = [x in {0, 1}]
//   genotypes   sigma = 1 - x, sigma^2, v = [x in {0, 1, 2}], 0 (PL = 2: sigma, v)
// Padding (127) and invalid codes give 0 in every plane; invalid codes also raise
// LDK_DEVERR_BAD_INPUT.
//
// Gather: a warp takes sixteen K rows, all of them in flight before the first is used (what
// bounds this kernel is how many bytes are under way); each row's four codes come as one 32-bit
// word (int8 input) or one byte (packed input: four 2-bit fields holding code + 1, SNP v in bits
// 2 (v % 4) of byte v / 4), 4 x 4 byte blocks are transposed in registers with byte permutes,
// and each SNP's sixteen K bytes go to the tile in one 128-bit store, at a place rotated by the
// lane so that eight lanes fall in the 32 banks.  An int8 row segment that does not start on a
// 4-byte boundary (odd row stride, or an unaligned base) is read as the two aligned words around
// it and joined with a funnel shift; the offset is the same for the 32 lanes of a row, so the
// branch is warp-uniform.  The second word is read only where it holds SNPs of the quad, and an
// aligned word holding one byte of the matrix lies in that byte's memory page, so no read can
// fault; its other bytes are shifted or masked out.  The range check and the plane bytes are
// computed on four bytes at a time in plain 32-bit arithmetic.
template <bool GENO, bool PACKED, int PL = GENO ? 4 : 2>
__global__ void __launch_bounds__(256) k_prep_planes(PrepArgs a) {
    static_assert(kPrepV == 128 && kPrepK == 128, "a warp gathers 16 K rows, a lane four SNPs");
    constexpr uint32_t kOne = 0x01010101u, kPad = 0x7F7F7F7Fu;
    __shared__ uint4 tile[kPrepV][kPrepK / 16];  // 16 K positions at [v][their index ^ (v / 4) % 8]
    __shared__ int srow[kPrepK];
    const int64_t g = blockIdx.x / ((int64_t)kPrepGroup * a.ny), q = blockIdx.x % ((int64_t)kPrepGroup * a.ny);
    const int64_t bx = g * kPrepGroup + q % kPrepGroup;
    const int by = (int)(q / kPrepGroup);
    if (bx >= a.nx) return;
    if (by == a.slice) {
        prepare_rest<GENO>(a, bx);
        return;
    }
    const int64_t v0 = bx * kPrepV;
    const int k0 = by * kPrepK;
    if (threadIdx.x < kPrepK) {
        const int k = k0 + threadIdx.x;
        int p = 0;
        while (p + 1 < a.P && k >= a.kofs[p + 1]) ++p;
        const int local = k - a.kofs[p];
        const int np = a.pop_off[p + 1] - a.pop_off[p];
        srow[threadIdx.x] = (local >= 0 && local < np && k < a.kofs[a.P]) ? a.pop_rows[a.pop_off[p] + local] : -1;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // gather: tile[v][k] = X[row(k), v0 + v]; 127 marks padding
    {
        const int64_t v = v0 + 4 * lane;
        const int64_t left = a.n_var - v;
        const int nv = left >= 4 ? 4 : (left > 0 ? (int)left : 0);  // SNPs of this quad in the matrix
        const uint32_t keep = nv >= 4 ? 0xFFFFFFFFu : ((1u << (8 * nv)) - 1u);
        const int8_t* base = a.X + (PACKED ? (v >> 2) : v);
        uint32_t w[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int row = srow[16 * warp + m];
            w[m] = kPad;
            if (row >= 0 && nv > 0) {
                if constexpr (PACKED) {
                    w[m] = (uint8_t)__ldg(base + (int64_t)row * a.ld);
                } else {
                    const uintptr_t ad = reinterpret_cast<uintptr_t>(base + (int64_t)row * a.ld);
                    const uint32_t* q = reinterpret_cast<const uint32_t*>(ad & ~uintptr_t(3));
                    const int s = (int)(ad & 3u);
                    w[m] = __ldg(q);
                    if (s != 0) {
                        const uint32_t hi = s + nv > 4 ? __ldg(q + 1) : 0u;
                        w[m] = __funnelshift_r(w[m], hi, 8 * s);
                    }
                }
            }
        }
        uint32_t bad = 0u;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            if constexpr (PACKED) {
                // field j = code + 1 -> byte j = code (two's complement), or 0xFF for missing
                if (srow[16 * warp + m] >= 0 && nv > 0) {
                    const uint32_t b = w[m];
                    w[m] = 0u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[m] |= (((b >> (2 * j)) & 3u) - 1u & 0xFFu) << (8 * j);
                }
            }
            // code + 1 of each byte (no carry between bytes); valid: 0 .. 2 (haplotypes), 0 .. 3
            if (srow[16 * warp + m] >= 0) {
                const uint32_t y = (((w[m] & 0x7F7F7F7Fu) + kOne) ^ (w[m] & 0x80808080u)) & keep;
                uint32_t odd = y & 0xFCFCFCFCu;
                if constexpr (!GENO) odd |= y & (y >> 1) & kOne;
                if (odd) {  // invalid codes become padding
                    bad |= odd;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if ((odd >> (8 * j)) & 0xFFu) w[m] |= 0x7Fu << (8 * j);
                }
                w[m] = (w[m] & keep) | (kPad & ~keep);
            }
        }
        if (bad) atomicOr(a.status, LDK_DEVERR_BAD_INPUT);
        // 4 x 4 byte transposes: t[q][j] holds SNP j's codes of rows 4 q .. 4 q + 3
        uint32_t t[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t x0 = __byte_perm(w[4 * q], w[4 * q + 1], 0x5140), x1 = __byte_perm(w[4 * q], w[4 * q + 1], 0x7362);
            const uint32_t x2 = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x5140);
            const uint32_t x3 = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x7362);
            t[q][0] = __byte_perm(x0, x2, 0x5410);
            t[q][1] = __byte_perm(x0, x2, 0x7632);
            t[q][2] = __byte_perm(x1, x3, 0x5410);
            t[q][3] = __byte_perm(x1, x3, 0x7632);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            tile[4 * lane + j][warp ^ (lane & 7)] = make_uint4(t[0][j], t[1][j], t[2][j], t[3][j]);
    }
    __syncthreads();
    // scatter: a warp takes four SNPs at a time, a lane 16 K positions of one
    const int kg = lane & 7;
    uint8_t* out = a.planes_out + k0 + 16 * kg;
#pragma unroll
    for (int it = 0; it < kPrepV / 32; ++it) {
        const int vv = 32 * it + 4 * warp + (lane >> 3);
        const int64_t v = v0 + vv;
        if (v >= a.n_var) break;
        const uint4 q = tile[vv][kg ^ ((vv >> 2) & 7)];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        uint32_t sg[4], sq[4], va[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // the codes are 0, 1 (, 2), 0x7F or 0xFF: bit 1 (2) is clear in the valid ones only,
            // and adding 254 to a byte of 1 makes it -1
            va[k] = (~w[k] >> (GENO ? 2 : 1)) & kOne;
            if constexpr (GENO) {
                sq[k] = va[k] & ~w[k];
                sg[k] = sq[k] + ((w[k] >> 1) & va[k]) * 254u;
            } else {
                sg[k] = va[k] + (w[k] & va[k]) * 254u;
            }
        }
        uint8_t* dst = out + v * PL * (int64_t)a.ktot;
        auto put = [&](int plane, const uint32_t (&x)[4]) {
            *reinterpret_cast<uint4*>(dst + plane * (int64_t)a.ktot) = make_uint4(x[0], x[1], x[2], x[3]);
        };
        put(0, sg);
        if constexpr (PL == 4) {
            put(1, sq);
            put(2, va);
            *reinterpret_cast<uint4*>(dst + 3 * (int64_t)a.ktot) = make_uint4(0u, 0u, 0u, 0u);
        } else {
            put(1, va);
        }
    }
}

// ---------------------------------------------------------------------------
// peak probes: the two rates the fused parse's roofline is stated against
// ---------------------------------------------------------------------------

// Back-to-back kind::i8 MMAs (M = 128, N = 256, K = 32) from zero-filled shared-memory
// tiles into one TMEM accumulator, issued by one thread per CTA.
constexpr int kProbeN = 256;
__device__ unsigned g_probe_status;  // LDK_DEVERR_* of the probes
__device__ double g_probe_sink;      // keeps the FP64 chains live

__global__ void __launch_bounds__(128, 1) k_probe_i8(int iters) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int A_BYTES = 128 * kKChunk, B_BYTES = kProbeN * kKChunk;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    for (int idx = threadIdx.x; idx < (A_BYTES + B_BYTES) / 16; idx += blockDim.x)
        reinterpret_cast<uint4*>(base)[idx] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        tmem_alloc(&tmem_base_s, kProbeN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    if (threadIdx.x == 0) {
        constexpr uint32_t idesc = idesc_s8<kProbeN>();
        const uint32_t a_addr = su32(base), b_addr = a_addr + A_BYTES;
        for (int it = 0; it < iters; ++it)
#pragma unroll
            for (int ks = 0; ks < kKChunk / 32; ++ks)
                mma_i8(tmem, sw128_desc(a_addr + ks * 32), sw128_desc(b_addr + ks * 32), idesc, (it | ks) ? 1u : 0u);
        mma_commit(&bar);
        mbar_wait(&bar, 0u, &abort_s, &g_probe_status);
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        tmem_dealloc(tmem, kProbeN);
    }
}

// Eight independent FP64 FMA chains per thread.
__global__ void __launch_bounds__(512) k_probe_fp64(int iters, double b, double c) {
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-3 + k;
    for (int it = 0; it < iters; ++it)
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = fma(x[k], b, c);
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += x[k];
    if (t == 1234.5678) g_probe_sink = t;  // never true for these inputs
}


}  // namespace

int tc_rows_per_block(const ParseShape& sh) { return sh.genotypes ? Cfg<1, true>::ROWS : Cfg<1, false>::ROWS; }
int tc_block_slots(const ParseShape& sh) { return sh.genotypes ? Cfg<1, true>::SLOTS : Cfg<1, false>::SLOTS; }
int tc_tile_width(const ParseShape& sh, int variant) { return tile_nj(sh.P, sh.genotypes != 0, variant); }
int tc_planes(const ParseShape& sh) { return sh.genotypes ? Cfg<1, true>::PLANES : Cfg<1, false>::PLANES; }

namespace {
template <bool GENO>
bool tc_fits_g(const ParseShape& sh) {
    const int t = smem_table(sh);
    switch (sh.P) {
        case 1: return smem_fits<Cfg<1, GENO>>(sh, 1, t);
        case 2: return smem_fits<Cfg<2, GENO>>(sh, 1, t);
        case 3: return smem_fits<Cfg<3, GENO>>(sh, 1, t);
        default: return smem_fits<Cfg<4, GENO>>(sh, 1, t);
    }
}

template <bool GENO, int V>
bool private_staging_of(const ParseShape& sh) {
    switch (sh.P) {
        case 1: return private_staging<1, GENO, V>(sh);
        case 2: return private_staging<2, GENO, V>(sh);
        case 3: return private_staging<3, GENO, V>(sh);
        default: return private_staging<4, GENO, V>(sh);
    }
}
}  // namespace

bool tc_fits(const ParseShape& sh) { return sh.genotypes ? tc_fits_g<true>(sh) : tc_fits_g<false>(sh); }

// The narrow haplotype tile reads no table in the workspace; the wide genotype tiles fit with any
// number of bins (one staging copy of 64: 196 and 208 KB).
bool tc_variant_runs(const ParseShape& sh, int variant) { return variant == 0 || sh.genotypes || !sh.rtab_global; }

bool tc_private_staging(const ParseShape& sh, int variant) {
    if (sh.genotypes) return (variant == 1 && sh.P <= 2) ? private_staging_of<true, 1>(sh) : private_staging_of<true, 0>(sh);
    return variant == 1 ? private_staging_of<false, 1>(sh) : private_staging_of<false, 0>(sh);
}

bool tc_rtab_global(const ParseShape& sh) {
    switch (sh.P) {
        case 1: return rtab_global_t<1>(sh);
        case 2: return rtab_global_t<2>(sh);
        case 3: return rtab_global_t<3>(sh);
        default: return rtab_global_t<4>(sh);
    }
}

bool tc_from_counts(const ParseShape& sh) { return sh.max_n > kSpinMaxN; }

// The spin planes, and with `o` the rest of a parse's preparation in the same launch: pair
// ranges, the cleared accumulators and pair tallies, the reciprocal table.  (Separate kernels and
// memsets each waited for the one before: with the outputs' own memsets, which the bin sums
// overwrite anyway, thirteen operations for a window of 400 SNPs, 92 us a call; five, 56, of
// which the narrower tile and one-tile pieces on more SMs give 18.)
cudaError_t launch_prep_planes(const ldk_parse_t* d, const Scratch& w, const ParseShape& sh, const ldk_parse_out_t* o,
                               cudaStream_t s) {
    if (d->n_var == 0) return cudaSuccess;
    PrepArgs a{};
    a.slice = -1;
    a.X = d->X;
    a.ld = d->ld_x;
    a.n_var = d->n_var;
    a.pop_rows = d->pop_rows;
    for (int p = 0; p <= LDK_MAX_POPS; ++p) {
        a.pop_off[p] = d->pop_offsets[p];
        a.kofs[p] = sh.kofs[p];
    }
    a.P = sh.P;
    a.ktot = sh.ktot;
    a.planes_out = w.hv;
    a.status = w.status;
    a.nx = (d->n_var + kPrepV - 1) / kPrepV;
    a.ny = sh.ktot / kPrepK;
    if (o) {
        a.slice = a.ny++;
        a.ranges = jmax_args(d, w);
        const int64_t cells = (int64_t)d->n_blocks * d->n_bins;
        a.zero[0] = w.fx;
        a.zero_n[0] = cells * (sh.n_stats + 1) * kFxLimbs;
        a.zero[1] = reinterpret_cast<unsigned long long*>(o->pairs);
        a.zero[2] = reinterpret_cast<unsigned long long*>(o->r2_counts);
        a.zero_n[1] = a.zero_n[2] = cells;
        // more than a few words a thread (many blocks of few SNPs): by memset.  400 SNPs, 20 bins,
        // 1,000,000 blocks: 2,437 us with the tallies always cleared here, 1,103 with memsets
        for (int z = 0; z < 3; ++z)
            if (a.zero_n[z] > 64ll * 128 * a.nx) {
                cudaError_t e = cudaMemsetAsync(a.zero[z], 0, a.zero_n[z] * sizeof(unsigned long long), s);
                if (e != cudaSuccess) return e;
                a.zero_n[z] = 0;
            }
        a.table = static_cast<double4*>(w.rtab ? w.rtab : w.gtab);
        a.table_n = a.table ? sh.max_n + 1 : 0;
    }
    const int64_t blocks = (a.nx + kPrepGroup - 1) / kPrepGroup * kPrepGroup * a.ny;
    if (blocks > INT32_MAX) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)blocks;
    const bool packed = d->x_format == LDK_X_PACKED2;
    if (sh.genotypes && sh.planes == 2) {
        k_prep_planes<true, false, 2><<<grid, 256, 0, s>>>(a);
    } else if (sh.genotypes) {
        if (packed) k_prep_planes<true, true><<<grid, 256, 0, s>>>(a);
        else k_prep_planes<true, false><<<grid, 256, 0, s>>>(a);
    } else {
        if (packed) k_prep_planes<false, true><<<grid, 256, 0, s>>>(a);
        else k_prep_planes<false, false><<<grid, 256, 0, s>>>(a);
    }
    return cudaGetLastError();
}

namespace {
// Work items of the persistent parse kernel.  A row block alone is too coarse a unit where
// there are few row blocks per SM (a 5,000-SNP window has 79) or where their count leaves a
// partial last wave; pieces of at most c partner tiles bound the spread of the CTAs' finishing
// times by one piece.  c = max(min_tiles, ceil(total tiles / kItemTarget)) -- min_tiles at
// most the tiles there are per SM -- so shapes with many small row blocks keep one item per row
// block, and no piece is so short that the flush of its staged sums (which ends every item)
// outweighs its tiles.  Where there are fewer tiles than SMs a tile is a piece: 400 SNPs
// (28 tiles of 64 partners) x 60 haplotypes 0.028 ms with pieces of four, 0.020 with one; x 2,000
// haplotypes 0.050 and 0.028; from 2,000 SNPs on the same.  Not, though, where these pieces are
// more than the SMs and pieces of four tiles are not: 5,500 SNPs of 75 partners (86 row blocks of
// three tiles), two populations, 172 pieces 0.110 ms, 86 0.081 (8 bins 0.064, 0.048).
// Pieces of one row block are consecutive (the claim order of the row blocks stays), its last
// piece runs to INT32_MAX, and a row block without partners gets no item.  One block of 1024
// threads: the total, then a block-wide scan of the pieces per row block, 1024 row blocks per round.
constexpr int kSplitThreads = 1024;

// Row block k: from the list, or (no list: one window) [k * rows, (k + 1) * rows) up to `end`.
struct RowBlocks {
    const int32_t* list;
    int rows, end;
    __device__ __forceinline__ int2 at(int k) const {
        if (list) return make_int2(list[2 * k], list[2 * k + 1]);
        const int r0 = k * rows;
        return make_int2(r0, end - r0 < rows ? end : r0 + rows);
    }
};

__device__ __forceinline__ int rb_tiles(const RowBlocks& rb, const int32_t* __restrict__ jmax, int k, int nj) {
    const int2 b = rb.at(k);
    const int r0 = b.x, r1 = b.y;
    const int jend = jmax[r1 - 1];
    return jend > r0 + 1 ? (jend - r0 + nj - 1) / nj : 0;
}

// Sum over the block's threads, in every thread; `s_sum` must not be in use.
__device__ __forceinline__ long long block_sum(long long t, long long (&s_sum)[kSplitThreads / 32]) {
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = t;
    __syncthreads();
    long long total = 0;
#pragma unroll 4
    for (int x = 0; x < kSplitThreads / 32; ++x) total += s_sum[x];
    return total;
}

__global__ void __launch_bounds__(kSplitThreads) k_split_items(const RowBlocks rb, int n_rb,
                                                               const int32_t* __restrict__ jmax, int nj,
                                                               int min_tiles, int4* __restrict__ items,
                                                               int* __restrict__ n_items) {
    __shared__ long long s_sum[3][kSplitThreads / 32];
    __shared__ int s_scan[kSplitThreads / 32];
    __shared__ int s_base;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int NW = kSplitThreads / 32;
    long long t = 0;
    for (int k = tid; k < n_rb; k += kSplitThreads) t += rb_tiles(rb, jmax, k, nj);
    if (tid == 0) s_base = 0;
    const long long total = block_sum(t, s_sum[0]);
    const long long cl = (total + kItemTarget - 1) / kItemTarget, spread = (total + kSpreadCtas - 1) / kSpreadCtas;
    int least = spread < min_tiles ? (spread > 0 ? (int)spread : 1) : min_tiles;
    if (least < kMinItemTiles && min_tiles >= kMinItemTiles && n_rb >= kSpreadCtas / 2) {
        // a second round of shorter pieces (more than a few) costs more than one round of kMinItemTiles
        long long now = 0, whole = 0;
        for (int k = tid; k < n_rb; k += kSplitThreads) {
            const int nt = rb_tiles(rb, jmax, k, nj);
            now += (nt + least - 1) / least;
            whole += (nt + kMinItemTiles - 1) / kMinItemTiles;
        }
        if (block_sum(now, s_sum[1]) > kSpreadCtas + kSpreadCtas / 16 && block_sum(whole, s_sum[2]) <= kSpreadCtas) least = kMinItemTiles;
    }
    const int c = cl > least ? (int)cl : least;
    for (int b0 = 0; b0 < n_rb; b0 += kSplitThreads) {
        const int k = b0 + tid;
        const int nt = k < n_rb ? rb_tiles(rb, jmax, k, nj) : 0;
        const int parts = (nt + c - 1) / c;
        int x = parts;  // inclusive scan within the warp, then over the warps
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_scan[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int v = s_scan[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += y;
            }
            s_scan[lane] = v;
        }
        __syncthreads();
        const int first = s_base + (wid ? s_scan[wid - 1] : 0) + x - parts;
        if (parts) {
            const int r0 = rb.at(k).x, r1 = rb.at(k).y;
            for (int q = 0; q < parts; ++q)
                items[first + q] = make_int4(r0, r1, q * c, q == parts - 1 ? INT32_MAX : (q + 1) * c);
        }
        const int round_total = s_scan[NW - 1];
        __syncthreads();
        if (tid == 0) s_base += round_total;
        __syncthreads();
    }
    if (tid == 0) *n_items = s_base;
}
}  // namespace

int tc_min_item_tiles(const ParseShape& sh) {
    const int staged = sh.slots * sh.n_bins * (sh.n_stats + 1);
    const int t = (staged + kFlushValuesPerTile - 1) / kFlushValuesPerTile;
    return t > kMinItemTiles ? t : kMinItemTiles;
}

cudaError_t launch_split_items(const Scratch& w, int n_row_blocks, int nj, int min_tiles, int rows, int end,
                               cudaStream_t s) {
    k_split_items<<<1, kSplitThreads, 0, s>>>(RowBlocks{w.row_blocks, rows, end}, n_row_blocks, w.jmax, nj, min_tiles,
                                              reinterpret_cast<int4*>(w.items), w.n_items);
    return cudaGetLastError();
}

cudaError_t launch_parse_tc(const ldk_parse_t* d, const ldk_parse_out_t* o, const Scratch& w,
                            const ParseShape& sh, int max_items, int variant, cudaStream_t s) {
    if (sh.from_counts)
        return sh.genotypes ? launch_tc_counts_geno(d, o, w, sh, max_items, variant, s)
                            : launch_tc_counts_hap(d, o, w, sh, max_items, variant, s);
    if (sh.genotypes) return launch_tc_geno(d, o, w, sh, max_items, variant, s);
    return variant == 1 ? launch_tc_hap_v1(d, o, w, sh, max_items, s) : launch_tc_hap_v0(d, o, w, sh, max_items, s);
}


// Peak probes, each timed with CUDA events on `s` after one untimed warm-up launch.
// *status receives the probes' device status word.
cudaError_t probe_peaks(double* int8_ops_per_s, double* fp64_fma_per_s, unsigned* status, cudaStream_t s) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = 1024 + 128 * kKChunk + kProbeN * kKChunk;
    cudaError_t e = cudaFuncSetAttribute(k_probe_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const unsigned zero = 0u;
    if ((e = cudaMemcpyToSymbolAsync(g_probe_status, &zero, sizeof(unsigned), 0, cudaMemcpyHostToDevice, s)) !=
        cudaSuccess)
        return e;
    cudaEvent_t e0, e1;
    if ((e = cudaEventCreate(&e0)) != cudaSuccess) return e;
    if ((e = cudaEventCreate(&e1)) != cudaSuccess) { cudaEventDestroy(e0); return e; }
    float ms = 0.f;
    const int i8_iters = 20000, f64_iters = 2000;
    k_probe_i8<<<sms, 128, smem, s>>>(64);
    cudaEventRecord(e0, s);
    k_probe_i8<<<sms, 128, smem, s>>>(i8_iters);
    cudaEventRecord(e1, s);
    if ((e = cudaEventSynchronize(e1)) == cudaSuccess && (e = cudaEventElapsedTime(&ms, e0, e1)) == cudaSuccess)
        *int8_ops_per_s = 2.0 * 128 * kProbeN * kKChunk * (double)i8_iters * sms / (ms * 1e-3);
    if (e == cudaSuccess) {
        k_probe_fp64<<<sms, 512, 0, s>>>(16, 0.999999, 1e-9);
        cudaEventRecord(e0, s);
        k_probe_fp64<<<sms, 512, 0, s>>>(f64_iters, 0.999999, 1e-9);
        cudaEventRecord(e1, s);
        if ((e = cudaEventSynchronize(e1)) == cudaSuccess && (e = cudaEventElapsedTime(&ms, e0, e1)) == cudaSuccess)
            *fp64_fma_per_s = 64.0 * 512 * (double)f64_iters * sms / (ms * 1e-3);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyFromSymbolAsync(status, g_probe_status, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

}  // namespace ldk
