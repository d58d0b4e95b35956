/*
 * ntlp_recip.h -- the reciprocals of the FP64 deposition's denominators, which
 * div_by (ntlp_deposit.cuh) divides with.  Host code without CUDA.
 */
#ifndef NTLP_RECIP_H
#define NTLP_RECIP_H

#include "ntlp_math.h"

namespace ntlp {

/* whether division by reciprocal is exact for a denominator: a significand
 * that is not all ones, within 2^-100 .. 2^100 */
inline bool recip_exact(double d) {
    const uint64_t m = ntlp_bits(d) & 0x000fffffffffffffULL;
    return d > 0x1p-100 && d < 0x1p100 && m != 0x000fffffffffffffULL;
}

/* rec[k] = 1/dzu(k), rec[nnz+3+k] = 1/(dx dy dzu(k)) for the cells' levels
 * k = 1..nnz+1, each correctly rounded, and 1 for dzu(0) and dzu(nnz+2), which
 * the deposition does not divide by and a caller may leave unset.  False when
 * a denominator does not qualify; the deposition then divides. */
inline bool deposit_reciprocals(double dx, double dy, const double *dzu, int nnz, double *rec) {
    const int n = nnz + 3;
    bool all = recip_exact(dx) && recip_exact(dy);
    for (int k = 0; k < 2 * n; ++k) rec[k] = 1.0;
    for (int k = 1; k <= nnz + 1; ++k) {
        const double dV = dx * dy * dzu[k];
        all = all && recip_exact(dzu[k]) && recip_exact(dV);
        rec[k] = 1.0 / dzu[k];
        rec[n + k] = 1.0 / dV;
    }
    return all;
}

}  // namespace ntlp

#endif
