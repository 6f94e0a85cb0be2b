// Spin moments of one SNP pair and population: the tensor-core counts and what the
// statistic-level forms (spin_hap_P*, spin_geno_P*) read.
#pragma once
#include "ldk_common.cuh"

// n jointly called individuals, S = sum sigma, T = sum tau, R = sum sigma tau (sigma, tau the
// spins of the left and right SNP: 1 - 2a, a the individual's frequency of allele 1); the
// genotype path adds SS = sum sigma^2, TT, SST = sum sigma^2 tau, STT, SSTT.  r1..r4:
// reciprocals of n, n(n-1), n(n-1)(n-2), n(n-1)(n-2)(n-3).
struct SpinPop {
    double n, S, T, R, SS, TT, SST, STT, SSTT;
    double r1, r2, r3, r4;
};

// Haplotype table entry for n: each reciprocal 0 where its product is 0, the reference's
// ``den > 0 ? num / den : 0`` (haplotype_kernels.py:78).
LDK_DEV double4 recip_entry(int n) {
    const double d = (double)n;
    double4 r;
    r.x = n >= 1 ? 1.0 / d : 0.0;
    r.y = n >= 2 ? 1.0 / (d * (d - 1.0)) : 0.0;
    r.z = n >= 3 ? 1.0 / (d * (d - 1.0) * (d - 2.0)) : 0.0;
    r.w = n >= 4 ? 1.0 / (d * (d - 1.0) * (d - 2.0) * (d - 3.0)) : 0.0;
    return r;
}

// Genotype table entry: the reference divides by n, n(n-1) and n(n-1)(n-2) unguarded
// (genotype_kernels.py:183-197), so the statistics of several populations are not finite where
// one has fewer than three jointly called individuals; only the four-fold one is guarded.
LDK_DEV double4 recip_entry_geno(int n) {
    const double d = (double)n;
    double4 r = recip_entry(n);
    r.x = 1.0 / d;
    r.y = 1.0 / (d * (d - 1.0));
    r.z = 1.0 / (d * (d - 1.0) * (d - 2.0));
    return r;
}

LDK_DEV void spin_reciprocals(SpinPop& x, const double4& r) {
    x.r1 = r.x;
    x.r2 = r.y;
    x.r3 = r.z;
    x.r4 = r.w;
}

// 1/x in double: the hardware estimate r (relative error e = 1 - x r, |e| < 2^-19) and one
// third-order iteration r (1 + e + e^2), which leaves e^3 -- one FMA fewer than two
// second-order ones.
LDK_DEV double recip_cubic(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
