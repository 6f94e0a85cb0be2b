// Pair-list haplotype counts from bit planes, and per-SNP call counts.
//
// The byte-wise count reads two codes and updates five sums per row and pair; with the
// population's rows packed 32 to a word (three planes: code 1, code 0, code >= 0) a pair takes
// five AND + POPC per word.  Packing reads the selected rows of the matrix once, which also
// answers whether any entry is missing -- a question every call asks and that took a gather,
// a compare and a reduction over the same rows.  1,000,000 pairs of 50,000 SNPs, 100 rows:
// byte-wise 137 us and 32 us for the missing test; packed 21 us (both answers' reading of the
// matrix) and 17 us.  Packing costs about one byte-wise count of n_var / 4 pairs, and the missing
// test alone read as much, so every call takes this path.
#include "ldk_internal.h"

namespace ldk {

namespace {

constexpr uint32_t kOnes = 0x01010101u;

// planes[plane][word][n_var]: bit b of word w is row 32 w + b of the selection; plane 0 code == 1,
// 1 code == 0, 2 code >= 0.  A thread takes four SNPs of one word: each row's four codes come as
// one word, its comparison bytes are shifted into four byte accumulators, and after eight rows
// each byte is a byte of one SNP's word.  flag: 1 = a code -1 was seen, 2 = a row outside the matrix.
constexpr int kPackThreads = 128;
__global__ void __launch_bounds__(kPackThreads)
    k_pack_bits(const int8_t* __restrict__ X, int64_t ld, int64_t n_var, int64_t n_total,
                const int32_t* __restrict__ rows, int n_rows, uint32_t* __restrict__ planes, int words,
                int* __restrict__ flag) {
    const int64_t v = 4 * ((int64_t)blockIdx.x * kPackThreads + threadIdx.x);
    if (v >= n_var) return;
    const int left = n_var - v < 4 ? (int)(n_var - v) : 4;
    for (int w = blockIdx.y; w < words; w += gridDim.y) {
        uint32_t out[3][4] = {};
        uint32_t missing = 0u;
        bool outside = false;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t x[8];
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const unsigned k = 32u * w + 8 * g + b;
                x[b] = 0xFEFEFEFEu;  // past the selection: in no plane, and not missing
                if (k < (unsigned)n_rows) {
                    const int row = rows[k];
                    if (row >= 0 && row < n_total) x[b] = load_quad(X + row * ld + v, left);
                    else outside = true;
                }
            }
            uint32_t one = 0u, zero = 0u, valid = 0u;  // byte j: eight rows of SNP v + j
#pragma unroll
            for (int b = 7; b >= 0; --b) {
                one = (one << 1) | (__vcmpeq4(x[b], kOnes) & kOnes);
                zero = (zero << 1) | (__vcmpeq4(x[b], 0u) & kOnes);
                valid = (valid << 1) | (~(x[b] >> 7) & kOnes);
                missing |= __vcmpeq4(x[b], 0xFFFFFFFFu);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                out[0][j] |= ((one >> (8 * j)) & 0xFFu) << (8 * g);
                out[1][j] |= ((zero >> (8 * j)) & 0xFFu) << (8 * g);
                out[2][j] |= ((valid >> (8 * j)) & 0xFFu) << (8 * g);
            }
        }
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < left) planes[((int64_t)pl * words + w) * n_var + v + j] = out[pl][j];
        if (left < 4) missing &= (1u << (8 * left)) - 1u;  // the bytes beyond the matrix
        const int f = (missing ? 1 : 0) | (outside ? 2 : 0);
        if (f) atomicOr(flag, f);
    }
}

__global__ void __launch_bounds__(256)
    k_counts_bits(const uint32_t* __restrict__ planes, int words, int64_t n_var, const int32_t* __restrict__ ii,
                  const int32_t* __restrict__ jj, int64_t n, int32_t* __restrict__ counts, int32_t* __restrict__ n_valid) {
    const int64_t pl = (int64_t)words * n_var;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t* pi = planes + ii[t];
        const uint32_t* pj = planes + jj[t];
        int c11 = 0, c10 = 0, c01 = 0, c00 = 0, v = 0;
#pragma unroll 4
        for (int w = 0; w < words; ++w, pi += n_var, pj += n_var) {
            const uint32_t oi = __ldg(pi), zi = __ldg(pi + pl), oj = __ldg(pj), zj = __ldg(pj + pl);
            c11 += __popc(oi & oj);
            c10 += __popc(oi & zj);
            c01 += __popc(zi & oj);
            c00 += __popc(zi & zj);
            v += __popc(__ldg(pi + 2 * pl) & __ldg(pj + 2 * pl));
        }
        reinterpret_cast<int4*>(counts)[t] = make_int4(c11, c10, c01, c00);
        if (n_valid) n_valid[t] = v;
    }
}

int pack_words(int n_rows) { return (int)(((int64_t)n_rows + 31) / 32); }

}  // namespace

size_t counts_workspace(int64_t n_var, int32_t n_rows) {
    return 256 + (size_t)3 * pack_words(n_rows) * n_var * sizeof(uint32_t);
}

cudaError_t launch_counts_bits(const int8_t* X, int64_t ld, int64_t n_var, int64_t n_total, const int32_t* rows,
                               int n_rows, const int32_t* ii, const int32_t* jj, int64_t n, int32_t* counts,
                               int32_t* n_valid, unsigned char* ws, cudaStream_t s) {
    int* flag = reinterpret_cast<int*>(ws);
    uint32_t* planes = reinterpret_cast<uint32_t*>(ws + 256);
    const int words = pack_words(n_rows);
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    if (n_var > 0 && words > 0) {
        const dim3 grid((unsigned)((n_var + 4 * kPackThreads - 1) / (4 * kPackThreads)), (unsigned)(words < 65535 ? words : 65535));
        k_pack_bits<<<grid, kPackThreads, 0, s>>>(X, ld, n_var, n_total, rows, n_rows, planes, words, flag);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (n > 0) {
        const int64_t blocks = (n + 255) / 256;
        k_counts_bits<<<(unsigned)(blocks < (1 << 20) ? blocks : (1 << 20)), 256, 0, s>>>(planes, words, n_var, ii, jj, n,
                                                                                        counts, n_valid);
    }
    return cudaGetLastError();
}

namespace {
// Per SNP over the selected rows (null: every row): the sum of its positive codes and how many
// codes are not negative.  As k_pack_bits, four SNPs a thread; a block's warps share 128 SNPs and
// take every sixteenth group of eight rows, so that a few thousand SNPs fill the GPU.
constexpr int kSumWarps = 16;
__global__ void __launch_bounds__(32 * kSumWarps)
    k_site_counts(const int8_t* __restrict__ X, int64_t ld, int64_t n_var, const int32_t* __restrict__ rows, int n_rows,
                  int32_t* __restrict__ pos, int32_t* __restrict__ valid) {
    __shared__ int sum[128], cnt[128];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < 128; k += blockDim.x) sum[k] = cnt[k] = 0;
    __syncthreads();
    const int64_t v = (int64_t)blockIdx.x * 128 + 4 * lane;
    const int64_t rest = n_var - v;
    const int left = rest < 4 ? (int)rest : 4;
    if (left > 0) {
        int S[4] = {}, N[4] = {};
        for (int k0 = 8 * warp; k0 < n_rows; k0 += 8 * kSumWarps) {
            uint32_t x[8];
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const int k = k0 + b;
                x[b] = k < n_rows ? load_quad(X + (int64_t)(rows ? rows[k] : k) * ld + v, left) : 0xFFFFFFFFu;
            }
            uint32_t nv = 0u, lo = 0u, hi = 0u;  // eight rows: at most 8 per byte, 1016 per half word
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint32_t c = __vmaxs4(x[b], 0u);
                nv += ~(x[b] >> 7) & kOnes;
                lo += c & 0x00FF00FFu;
                hi += (c >> 8) & 0x00FF00FFu;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                N[j] += (nv >> (8 * j)) & 0xFF;
                S[j] += ((j & 1 ? hi : lo) >> (16 * (j >> 1))) & 0xFFFF;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (S[j]) atomicAdd(&sum[4 * lane + j], S[j]);
            if (N[j]) atomicAdd(&cnt[4 * lane + j], N[j]);
        }
    }
    __syncthreads();
    const int64_t u = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (threadIdx.x < 128 && u < n_var) {
        pos[u] = sum[threadIdx.x];
        valid[u] = cnt[threadIdx.x];
    }
}
}  // namespace

cudaError_t launch_site_counts(const int8_t* X, int64_t ld, int64_t n_var, const int32_t* rows, int n_rows, int32_t* pos,
                               int32_t* valid, cudaStream_t s) {
    if (n_var == 0) return cudaSuccess;
    k_site_counts<<<(unsigned)((n_var + 127) / 128), 32 * kSumWarps, 0, s>>>(X, ld, n_var, rows, n_rows, pos, valid);
    return cudaGetLastError();
}

}  // namespace ldk
