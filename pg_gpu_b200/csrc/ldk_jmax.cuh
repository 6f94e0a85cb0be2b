// Pair ranges: jmax[i] = end of SNP i's partners (cutoff on pos, window end); i + 1 for SNPs
// after their window's anchor end (a split parse's right halo).  Also the input checks a parse
// makes once per SNP.
#pragma once
#include "ldk_internal.h"

namespace ldk {
namespace {

struct JmaxArgs {
    const double* pos;
    const double* coord;     // or null
    int64_t n_var;
    const int64_t* win_off;  // (n_win + 1) window offsets and (n_win) anchor ends; one window: null,
    const int64_t* anc_end;  // [0, n_var) with the anchors ending at anchor0
    int n_win;
    int64_t anchor0;
    double max_dist;
    const int32_t* snp_block;
    int n_blocks;
    int32_t* jmax;
    unsigned* status;
};

JmaxArgs jmax_args(const ldk_parse_t* d, const Scratch& w) {
    const bool one = !d->window_offsets || d->n_windows == 1;
    return JmaxArgs{d->pos, d->coord, d->n_var, one ? nullptr : w.win_off, one ? nullptr : w.anc_end, one ? 1 : d->n_windows,
                    d->anchor_end ? d->anchor_end[0] : d->n_var, d->max_dist, d->snp_block, d->n_blocks, w.jmax, w.status};
}

LDK_DEV void pair_range(const JmaxArgs& a, int64_t i) {
    int64_t we = a.n_var, ae = a.anchor0;
    if (a.win_off) {
        int lo = 0, hi = a.n_win;  // window w with win_off[w] <= i < win_off[w+1]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (a.win_off[mid] <= i) lo = mid; else hi = mid;
        }
        we = a.win_off[lo + 1];
        ae = a.anc_end[lo];
    }
    const double lim = a.pos[i] + a.max_dist;
    int64_t b = i + 1, e = we;  // first j in [i+1, we) with pos[j] > lim
    while (b < e) {
        const int64_t m = (b + e) >> 1;
        if (a.pos[m] <= lim) b = m + 1; else e = m;
    }
    a.jmax[i] = (int32_t)(i < ae ? b : i + 1);  // SNPs past the anchors have no pairs of their own
    if (i + 1 < we && a.pos[i + 1] < a.pos[i]) atomicOr(a.status, LDK_DEVERR_BAD_INPUT);
    if (a.coord && i + 1 < we && a.coord[i + 1] < a.coord[i]) atomicOr(a.status, LDK_DEVERR_BAD_INPUT);
    if (a.snp_block) {
        const int blk = a.snp_block[i];
        if (blk < 0 || blk >= a.n_blocks) atomicOr(a.status, LDK_DEVERR_BLOCK_RANGE);
    }
}

}  // namespace
}  // namespace ldk
