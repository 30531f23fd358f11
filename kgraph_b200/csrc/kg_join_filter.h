// The tensor-core join's filter (kg_join_tc.cu): which pairs are too far apart
// to enter either endpoint's pool, and the audit of that decision.  Host and
// device: the same lines are compiled for the host and checked there against
// FP64 distances.
#pragma once
#include <cfloat>
#include <cmath>

#ifdef __CUDACC__
#define KG_HD_FILTER __host__ __device__ __forceinline__
#else
#define KG_HD_FILTER inline
#endif

namespace kgb {

enum FilterMetric { FILTER_EUCLIDEAN = 0, FILTER_ANGULAR = 1, FILTER_L2SQR = 2 };   // the values of METRIC_*

// The test, approx d - E > max radius, without a square root or a division per
// pair: both sides times the denominator (angular), the margin's terms split into
// one part per row, |x_u - x_n| |x_j - x_n| = s_u s_j with s = sqrt(2 h) per row.
// euclidean and l2sqr (halved): A_u + A_j - g - 2 et s_u s_j > max radius;
// angular, full = g + A_u + A_j, w = n_u n_j:
//   -full - 2 et s_u s_j - C_u - C_j - 2 gam w - 4 gam |full| - 4.8e-7 |g|
//   > max radius (w + FLT_EPSILON).
// Its rounding is a few parts in 2^24 of the same terms, inside the factor 2 of E;
// the constants cover what underflows.
// h = |x_u - x_n|^2 / 2, c = (x_u - x_n) . x_n, qn = |x_n|^2, nrm the canonical
// norm term.
struct FilterRow { float A, s, rad, C, nrm; };

KG_HD_FILTER FilterRow filter_row(FilterMetric m, float h, float c, float nrm, float qn, float gam, float rad) {
    const float sr = sqrtf(2.0f * h);
    if (m == FILTER_ANGULAR)
        return FilterRow{c + 0.5f * qn, sr, rad,
                         2.0f * (gam * sr * sqrtf(qn) + 0.5f * gam * qn + 2.4e-7f * (fabsf(c) + 0.5f * qn)) + 6e-38f, nrm};
    if (m == FILTER_L2SQR) return FilterRow{h - 6.0f * gam * h - 5e-31f, sr, 0.5f * rad, 0.f, nrm};   // halved, the radius exactly
    return FilterRow{h - 2.0f * gam * h - 4.0f * gam * nrm - 5e-31f, sr, rad, 0.f, nrm};
}

// The relative product error et of E4M3 rows, f = 1 + their relative errors (g8:
// the products' accumulation).
KG_HD_FILTER float filter_et8(float fu, float fj, float g8) { return fu * fj * (1.f + g8) - 1.f; }

// The pair is skipped where lhs > rhs.  g: Gram entry, t2 = 2 et s_u s_j.
struct FilterTest { float lhs, rhs; };

KG_HD_FILTER FilterTest filter_pair(FilterMetric m, float g, float t2, float gam, float Au, float Aj, float radu,
                                    float radj, float Cu, float Cj, float nu, float nj) {
    const float rad = fmaxf(radu, radj);
    if (m == FILTER_ANGULAR) {
        const float full = g + (Au + Aj), w = nu * nj;
        return FilterTest{-full - t2 - (Cu + Cj) - 2.f * gam * w - 4.f * gam * fabsf(full) - 4.8e-7f * fabsf(g),
                          rad * (w + FLT_EPSILON)};
    }
    return FilterTest{(Au + Aj) - g - t2, rad};
}

// Whether the test went wrong on a pair of which the exact distance d64 and the
// canonical FP32 distance dc are known: its lower bound lies above either, or it
// skipped a pair that a pool would take.  rad: the larger radius as the test held
// it (FilterRow::rad).
KG_HD_FILTER bool filter_wrong(FilterMetric m, float lhs, bool skip, float rad, float nu, float nj, double d64, float dc) {
    const double unit = m == FILTER_ANGULAR ? (double)nu * (double)nj + (double)FLT_EPSILON : m == FILTER_L2SQR ? 0.5 : 1.0;
    const double radius = m == FILTER_L2SQR ? 2.0 * (double)rad : (double)rad;
    return (double)lhs > unit * fmin(d64, (double)dc) || (skip && !((double)dc > radius));
}

}  // namespace kgb
