// DoubleDouble pieces shared by the double-double integrand's kernels
// (cdet_dd.cu, cdet_wide.cu): the operators beyond those in cdet_device.cuh,
// the LU fallback's minor and the order-1 branch, in the reference's
// arrangement (utility/types.h:30-182).
#pragma once

#include "cdet_device.cuh"
#include "cdet_kernels.cuh"

namespace cdet {

// ------------------------------------------------ DoubleDouble (the rest) ---
// operator/ (utility/types.h:114-120): q1 = x.hi / y.hi, the remainder
// x - q1 y, q2 = (r.hi + r.lo) / y.hi, q1 + q2 renormalised.
__device__ __forceinline__ DD dd_div(DD x, DD y) {
    const double q1 = ddiv(x.hi, y.hi);
    const DD r = dd_sub(x, dd_mul(DD{q1, 0.0}, y));
    const double q2 = ddiv(dadd(r.hi, r.lo), y.hi);
    DD q = dd_add(DD{q1, 0.0}, DD{q2, 0.0});
    const double s = dadd(q.hi, q.lo);
    q.lo = dsub(q.lo, dsub(s, q.hi));
    q.hi = s;
    return q;
}
// dd_abs (utility/types.h:221-223)
__device__ __forceinline__ DD dd_abs(DD x) { return x.hi < 0.0 ? DD{-x.hi, -x.lo} : x; }
// the comparison operators (utility/types.h:146-168): lexicographic on (hi, lo)
__device__ __forceinline__ bool dd_lt(DD a, DD b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
__device__ __forceinline__ bool dd_gt(DD a, DD b) { return dd_lt(b, a); }
__device__ __forceinline__ bool dd_eq(DD a, DD b) { return a.hi == b.hi && a.lo == b.lo; }
__device__ __forceinline__ bool dd_zero(DD a) { return a.hi == 0.0 && a.lo == 0.0; }
// subtract_product for DoubleDouble (fast_principle_minors.h:30-37): base - left * right
__device__ __forceinline__ DD dd_sub_prod(DD left, DD right, DD base) { return dd_sub(base, dd_mul(left, right)); }

// determinant_principal_minor_from_buffer<DoubleDouble> (fast_principle_minors.h:39-105)
// for one mask on one lane; m is this lane's n x n DoubleDouble scratch.
static __device__ DD minor_by_lu_dd(const DD* a, int n, uint32_t mask, DD* m) {
    int idx[kMaxOrder];
    int k = 0;
    for (int i = 0; i < n; ++i)
        if (mask & (1u << i)) idx[k++] = i;
    if (k == 0) return DD{1.0, 0.0};
    for (int r = 0; r < k; ++r)
        for (int c = 0; c < k; ++c) m[r * k + c] = a[idx[r] * n + idx[c]];
    DD det{1.0, 0.0};
    int sign = 1;
    for (int col = 0; col < k; ++col) {
        int pivot_row = col;
        DD pivot_abs = dd_abs(m[col * k + col]);
        for (int row = col + 1; row < k; ++row) {
            const DD cand = dd_abs(m[row * k + col]);
            if (dd_gt(cand, pivot_abs)) {
                pivot_abs = cand;
                pivot_row = row;
            }
        }
        if (dd_zero(pivot_abs)) return DD{0.0, 0.0};
        if (pivot_row != col) {
            for (int c = col; c < k; ++c) {
                const DD t = m[col * k + c];
                m[col * k + c] = m[pivot_row * k + c];
                m[pivot_row * k + c] = t;
            }
            sign = -sign;
        }
        const DD pivot = m[col * k + col];
        det = dd_mul(det, pivot);
        for (int row = col + 1; row < k; ++row) {
            const DD factor = dd_div(m[row * k + col], pivot);
            if (dd_zero(factor)) continue;
            m[row * k + col] = DD{0.0, 0.0};
            for (int c = col + 1; c < k; ++c) m[row * k + c] = dd_sub_prod(factor, m[col * k + c], m[row * k + c]);
        }
    }
    return sign < 0 ? DD{-det.hi, -det.lo} : det;
}

// order1_density_integrand_from_sampled_vertex (:173-213) with IntegrandRealT =
// DoubleDouble: the unshifted diagonal widened, the DoubleDouble shifts added;
// no finiteness check on this branch.
__device__ __forceinline__ DD dd_order1_value(const Problem& p, const Scratch& w, int64_t c, int set) {
    const int r = set == 0 ? 2 : 1;
    const double* diag = w.diag + c * 2 * 2 * p.max_order;
    const DD shu{p.dd_shift[0].hi, p.dd_shift[0].lo}, shd{p.dd_shift[1].hi, p.dd_shift[1].lo};
    const DD su = dd_add(DD{diag[(set * 2) * p.max_order], 0.0}, shu);
    const DD sd = dd_add(DD{diag[(set * 2 + 1) * p.max_order], 0.0}, shd);
    const DD ru = dd_mul(dd_mul(DD{static_cast<double>(-r), 0.0}, DD{p.dd_u.hi, p.dd_u.lo}),
                         DD{p.dd_beta.hi, p.dd_beta.lo});
    return dd_mul(ru, dd_sub(dd_mul(su, sd), dd_mul(shu, shd)));
}

}  // namespace cdet
