// Shared by the beam ODE (rk4.cu) and the trajectory surrogate (surrogate.cu):
// the sound speed interpolant with its derivatives, the beam state, and the
// writer of trajectory records (FP64 records, FP32 summation records, and the
// per-time-tile culling boxes) in the layout msgb_trajectories documents.
#pragma once

#include <climits>
#include <type_traits>

#include "common.cuh"

namespace msgb {
namespace {

struct MediumArgs {
    int kind, boundary;
    int n[3];
    double spacing[3], origin[3];
    double inv_spacing[3];  // 1 / spacing (multiplications instead of FP64 divisions)
    const double *coeffs;
    double c, lam;
    const float *coeffs32;  // (coeffs - c_ref) in FP32, or nullptr
    double c_ref;
    // factors of the interpolant's sums (see speed_eval_k): the value's, the
    // gradient's per axis and the Hessian's per pair of axes
    double sv, sg[3], sh[3][3];
};

__device__ __forceinline__ int map_index(int i, int n, int boundary) {
    if (n == 1) return 0;
    switch (boundary) {
        case 0: return i < 0 ? 0 : (i > n - 1 ? n - 1 : i);
        case 1: { int r = i % n; return r < 0 ? r + n : r; }
        case 2: { const int per = 2 * n; int r = i % per; if (r < 0) r += per; return r < n ? r : per - 1 - r; }
        default: { const int per = 2 * n - 2; int r = i % per; if (r < 0) r += per; return r < n ? r : per - r; }
    }
}

// Indices of the 4 (cubic) or 2 taps starting at lo by the boundary rule: only
// for cells at the edge of the grid, kept out of the integrators' loop.
static __device__ __noinline__ int4 edge_taps(int lo, int n, int boundary) {
    return make_int4(map_index(lo, n, boundary), map_index(lo + 1, n, boundary), map_index(lo + 2, n, boundary),
                     map_index(lo + 3, n, boundary));
}

// The taps x taps values of a 2D stencil whose first tap is (lo0, lo1): inside
// the grid (the usual case) from one base address with constant row offsets.
template <int TAPS, typename T>
__device__ __forceinline__ void gather_plane(const T *__restrict__ g, const int *n, int lo0, int lo1, int boundary,
                                             T (*v)[4]) {
    if (lo0 >= 0 && lo0 <= n[0] - TAPS && lo1 >= 0 && lo1 <= n[1] - TAPS) {
        const T *p = g + ((int64_t)lo0 * n[1] + lo1);
#pragma unroll
        for (int i = 0; i < TAPS; ++i) {
#pragma unroll
            for (int k = 0; k < TAPS; ++k) v[i][k] = __ldg(p + k);
            p += n[1];
        }
        return;
    }
    const int4 a = edge_taps(lo0, n[0], boundary), b = edge_taps(lo1, n[1], boundary);
    const int ia[4] = {a.x, a.y, a.z, a.w}, ib[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < TAPS; ++i)
#pragma unroll
        for (int k = 0; k < TAPS; ++k) v[i][k] = __ldg(g + ((int64_t)ia[i] * n[1] + ib[k]));
}

// A lane's stencil of a 2D cubic medium, kept in shared memory across evaluations:
// a beam stays in its grid cell for about three steps (18 evaluations), and 16
// scattered loads per lane and evaluation are 16 x 32 L1 lookups per warp -- they
// took half of the beam ODE's time.  at: this lane's first vector; the rows are
// strided by the block (16-byte accesses without bank conflicts).
struct NoCache {
    static constexpr bool on = false;
};

template <typename T>
struct StencilCache {
    static constexpr bool on = true;
    using V = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
    static constexpr int NV = 16 * sizeof(T) / sizeof(V);
    static constexpr int kLanes = 64;  // the integrators' block size
    static constexpr size_t kBytes = sizeof(V) * NV * kLanes;
    V *at;
    int lo0 = INT_MIN, lo1 = 0;
    T centre;  // FP32: the value at tap (1, 1), subtracted from the stored ones

    // v: the stencil at (lo0, lo1); FP32: minus its centre value c
    __device__ __forceinline__ void get(const T *__restrict__ g, const int *n, int l0, int l1, int boundary, T (*v)[4],
                                        T &c) {
        if (l0 != lo0 || l1 != lo1) {
            gather_plane<4>(g, n, l0, l1, boundary, v);
            centre = sizeof(T) == 4 ? v[1][1] : T(0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[i][k] = sizeof(T) == 4 ? v[i][k] - centre : v[i][k];
                if constexpr (sizeof(T) == 4) {
                    at[i * kLanes] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
                } else {
                    at[2 * i * kLanes] = make_double2(v[i][0], v[i][1]);
                    at[(2 * i + 1) * kLanes] = make_double2(v[i][2], v[i][3]);
                }
            }
            lo0 = l0;
            lo1 = l1;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (sizeof(T) == 4) {
                const float4 q = at[i * kLanes];
                v[i][0] = q.x, v[i][1] = q.y, v[i][2] = q.z, v[i][3] = q.w;
            } else {
                const double2 q = at[2 * i * kLanes], r = at[(2 * i + 1) * kLanes];
                v[i][0] = q.x, v[i][1] = q.y, v[i][2] = r.x, v[i][3] = r.y;
            }
        }
        c = centre;
    }
};

// The integrators' cache for a medium: 2D cubic only (a 3D stencil, 64 values,
// would cost a resident block).
template <int D, int KIND, typename T>
using MediumCache = typename std::conditional<D == 2 && KIND == MSGB_MEDIUM_BSPLINE3, StencilCache<T>, NoCache>::type;
template <int D, int KIND, typename T>
constexpr size_t medium_cache_bytes() {
    return D == 2 && KIND == MSGB_MEDIUM_BSPLINE3 ? StencilCache<T>::kBytes : 0;
}

// The taps along one axis starting at lo (offsets into that axis).
template <int TAPS>
__device__ __forceinline__ void axis_taps(int lo, int n, int boundary, int *idx) {
    if (lo >= 0 && lo <= n - TAPS) {
#pragma unroll
        for (int k = 0; k < TAPS; ++k) idx[k] = lo + k;
        return;
    }
    const int4 a = edge_taps(lo, n, boundary);
    const int ia[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int k = 0; k < TAPS; ++k) idx[k] = ia[k];
}

// floor(u) and u's cell, from adding 1.5 * 2^52 (|u| < 2^31, as any position within
// two thousand million cells; others give some cell, which the boundary rule maps
// into the grid): floor and the conversion to int run at a fraction of the rate.
__device__ __forceinline__ double floor_cell(double u, int &i) {
    const double m = u + 6755399441055744.0;
    i = __double2loint(m);
    double fl = m - 6755399441055744.0;
    if (fl > u) fl -= 1.0, i -= 1;
    return fl;
}

// c, grad c (D), hess c (D x D, row-major) at x, for a medium of kind KIND
// (the tap count and the weights are then compile-time constants).
template <int D, int KIND, typename Cache = NoCache>
__device__ __forceinline__ void speed_eval_k(const MediumArgs &m, const double *x, double &c, double *g, double *H,
                                             Cache *cache = nullptr) {
    if (KIND == MSGB_MEDIUM_CONSTANT) {
        c = m.c;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            g[i] = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) H[i * D + k] = 0.0;
        }
        return;
    }
    constexpr bool cubic = KIND == MSGB_MEDIUM_BSPLINE3;
    constexpr int taps = cubic ? 4 : 2;
    constexpr int off0 = cubic ? -1 : 0;
    double w[D][4], d1[D][4], d2[D][4];
    int lo[D], idx[D][4];
#pragma unroll
    for (int a = 0; a < D; ++a) {
        const double u = (x[a] - m.origin[a]) * m.inv_spacing[a];
        int i0;
        const double t = u - floor_cell(u, i0);
        if (cubic) {
            // 6 x the B-spline weights (the factors 1/6 are applied to the
            // sums at the end: no FP64 division per weight)
            const double omt = 1.0 - t, t2 = t * t, t3 = t2 * t;
            w[a][0] = omt * omt * omt;
            w[a][1] = 3.0 * t3 - 6.0 * t2 + 4.0;
            w[a][2] = -3.0 * t3 + 3.0 * t2 + 3.0 * t + 1.0;
            w[a][3] = t3;
            d1[a][0] = -(omt * omt) / 2.0;
            d1[a][1] = 1.5 * t2 - 2.0 * t;
            d1[a][2] = -1.5 * t2 + t + 0.5;
            d1[a][3] = t2 / 2.0;
            d2[a][0] = omt;
            d2[a][1] = 3.0 * t - 2.0;
            d2[a][2] = -3.0 * t + 1.0;
            d2[a][3] = t;
        } else {
            w[a][0] = 1.0 - t;
            w[a][1] = t;
            d1[a][0] = -1.0;
            d1[a][1] = 1.0;
            d2[a][0] = d2[a][1] = 0.0;
            w[a][2] = w[a][3] = d1[a][2] = d1[a][3] = d2[a][2] = d2[a][3] = 0.0;
        }
        lo[a] = i0 + off0;
        if (D != 2) axis_taps<taps>(lo[a], m.n[a], m.boundary, idx[a]);
    }
    // Separable reduction, last axis first: the tensor-product weights factor,
    // so the value, gradient and Hessian need 3 sums per line of the last
    // axis instead of D^2 products per grid corner.
    double cc = 0.0, gg[D], hh[D][D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        gg[i] = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) hh[i][k] = 0.0;
    }
    if (D == 1) {
#pragma unroll
        for (int k = 0; k < taps; ++k) {
            const double v = __ldg(m.coeffs + idx[0][k]);
            cc = fma(w[0][k], v, cc);
            gg[0] = fma(d1[0][k], v, gg[0]);
            hh[0][0] = fma(d2[0][k], v, hh[0][0]);
        }
    } else if (D == 2) {
        const int L = D - 1;  // last axis
        double v2[4][4];
        if constexpr (Cache::on) {
            double centre;
            cache->get(m.coeffs, m.n, lo[0], lo[L], m.boundary, v2, centre);
        } else {
            gather_plane<taps>(m.coeffs, m.n, lo[0], lo[L], m.boundary, v2);
        }
#pragma unroll
        for (int i = 0; i < taps; ++i) {
            double rw = 0.0, rd = 0.0, rdd = 0.0;
#pragma unroll
            for (int k = 0; k < taps; ++k) {
                const double v = v2[i][k];
                rw = fma(w[L][k], v, rw);
                rd = fma(d1[L][k], v, rd);
                rdd = fma(d2[L][k], v, rdd);
            }
            cc = fma(w[0][i], rw, cc);
            gg[0] = fma(d1[0][i], rw, gg[0]);
            gg[L] = fma(w[0][i], rd, gg[L]);
            hh[0][0] = fma(d2[0][i], rw, hh[0][0]);
            hh[0][L] = fma(d1[0][i], rd, hh[0][L]);
            hh[L][L] = fma(w[0][i], rdd, hh[L][L]);
        }
    } else {
        const int Y = 1 % D, Z = 2 % D;
#pragma unroll
        for (int i = 0; i < taps; ++i) {
            double tw = 0.0, ty = 0.0, tyy = 0.0, tz = 0.0, tyz = 0.0, tzz = 0.0;
#pragma unroll
            for (int j = 0; j < taps; ++j) {
                const double *line = m.coeffs + ((int64_t)idx[0][i] * m.n[Y] + idx[Y][j]) * m.n[Z];
                double sw = 0.0, sd = 0.0, sdd = 0.0;
#pragma unroll
                for (int k = 0; k < taps; ++k) {
                    const double v = __ldg(line + idx[Z][k]);
                    sw = fma(w[Z][k], v, sw);
                    sd = fma(d1[Z][k], v, sd);
                    sdd = fma(d2[Z][k], v, sdd);
                }
                tw = fma(w[Y][j], sw, tw);
                ty = fma(d1[Y][j], sw, ty);
                tyy = fma(d2[Y][j], sw, tyy);
                tz = fma(w[Y][j], sd, tz);
                tyz = fma(d1[Y][j], sd, tyz);
                tzz = fma(w[Y][j], sdd, tzz);
            }
            cc = fma(w[0][i], tw, cc);
            gg[0] = fma(d1[0][i], tw, gg[0]);
            gg[Y] = fma(w[0][i], ty, gg[Y]);
            gg[Z] = fma(w[0][i], tz, gg[Z]);
            hh[0][0] = fma(d2[0][i], tw, hh[0][0]);
            hh[0][Y] = fma(d1[0][i], ty, hh[0][Y]);
            hh[0][Z] = fma(d1[0][i], tz, hh[0][Z]);
            hh[Y][Y] = fma(w[0][i], tyy, hh[Y][Y]);
            hh[Y][Z] = fma(w[0][i], tyz, hh[Y][Z]);
            hh[Z][Z] = fma(w[0][i], tzz, hh[Z][Z]);
        }
    }
    // (the cubic weights are 6 x the true ones: see medium_args for the factors)
    c = cc * m.sv;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        g[a] = gg[a] * m.sg[a];
#pragma unroll
        for (int b = 0; b < D; ++b) H[a * D + b] = (a <= b ? hh[a][b] : hh[b][a]) * m.sh[a][b];
    }
}

// The same in FP32 for the FP32 path: the fractional position is formed in
// FP64 and rounded, the B-spline weights and tap sums run in FP32 on
// (coefficient - c_ref) values centred on tap (1, 1[, 1]) of the stencil (the
// weights of every derivative sum to zero, so the centring leaves the
// gradient and Hessian unchanged and keeps their sums free of cancellation;
// the value gets the centre back), and the results return to FP64 with c_ref.
template <int D, int KIND, typename Cache>
__device__ __forceinline__ void speed_eval_f32(const MediumArgs &m, const double *x, double &c, double *g, double *H,
                                               Cache *cache) {
    constexpr bool cubic = KIND == MSGB_MEDIUM_BSPLINE3;
    constexpr int taps = cubic ? 4 : 2;
    constexpr int off0 = cubic ? -1 : 0;
    constexpr int ctr = cubic ? 1 : 0;  // the tap at the cell's lower corner
    float w[D][4], d1[D][4], d2[D][4];
    int lo[D], idx[D][4];
#pragma unroll
    for (int a = 0; a < D; ++a) {
        const double u = (x[a] - m.origin[a]) * m.inv_spacing[a];
        int i0;
        const float t = (float)(u - floor_cell(u, i0));
        if (cubic) {
            const float omt = 1.0f - t, t2 = t * t, t3 = t2 * t;
            w[a][0] = omt * omt * omt;
            w[a][1] = fmaf(3.0f, t3, fmaf(-6.0f, t2, 4.0f));
            w[a][2] = fmaf(-3.0f, t3, fmaf(3.0f, t2, fmaf(3.0f, t, 1.0f)));
            w[a][3] = t3;
            d1[a][0] = -0.5f * omt * omt;
            d1[a][1] = fmaf(1.5f, t2, -2.0f * t);
            d1[a][2] = fmaf(-1.5f, t2, t + 0.5f);
            d1[a][3] = 0.5f * t2;
            d2[a][0] = omt;
            d2[a][1] = fmaf(3.0f, t, -2.0f);
            d2[a][2] = fmaf(-3.0f, t, 1.0f);
            d2[a][3] = t;
        } else {
            w[a][0] = 1.0f - t;
            w[a][1] = t;
            d1[a][0] = -1.0f;
            d1[a][1] = 1.0f;
            d2[a][0] = d2[a][1] = 0.0f;
            w[a][2] = w[a][3] = d1[a][2] = d1[a][3] = d2[a][2] = d2[a][3] = 0.0f;
        }
        lo[a] = i0 + off0;
        if (D != 2) axis_taps<taps>(lo[a], m.n[a], m.boundary, idx[a]);
    }
    float cc = 0.0f, gg[D], hh[D][D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        gg[i] = 0.0f;
#pragma unroll
        for (int k = 0; k < D; ++k) hh[i][k] = 0.0f;
    }
    float vc;
    if (D == 1) {
        vc = __ldg(m.coeffs32 + idx[0][ctr]);
#pragma unroll
        for (int k = 0; k < taps; ++k) {
            const float v = __ldg(m.coeffs32 + idx[0][k]) - vc;
            cc = fmaf(w[0][k], v, cc);
            gg[0] = fmaf(d1[0][k], v, gg[0]);
            hh[0][0] = fmaf(d2[0][k], v, hh[0][0]);
        }
    } else if (D == 2) {
        const int L = D - 1;
        float v2[4][4];
        if constexpr (Cache::on) {
            cache->get(m.coeffs32, m.n, lo[0], lo[L], m.boundary, v2, vc);
        } else {
            gather_plane<taps>(m.coeffs32, m.n, lo[0], lo[L], m.boundary, v2);
            vc = v2[ctr][ctr];
#pragma unroll
            for (int i = 0; i < taps; ++i)
#pragma unroll
                for (int k = 0; k < taps; ++k) v2[i][k] -= vc;
        }
#pragma unroll
        for (int i = 0; i < taps; ++i) {
            float rw = 0.0f, rd = 0.0f, rdd = 0.0f;
#pragma unroll
            for (int k = 0; k < taps; ++k) {
                const float v = v2[i][k];
                rw = fmaf(w[L][k], v, rw);
                rd = fmaf(d1[L][k], v, rd);
                rdd = fmaf(d2[L][k], v, rdd);
            }
            cc = fmaf(w[0][i], rw, cc);
            gg[0] = fmaf(d1[0][i], rw, gg[0]);
            gg[L] = fmaf(w[0][i], rd, gg[L]);
            hh[0][0] = fmaf(d2[0][i], rw, hh[0][0]);
            hh[0][L] = fmaf(d1[0][i], rd, hh[0][L]);
            hh[L][L] = fmaf(w[0][i], rdd, hh[L][L]);
        }
    } else {
        const int Y = 1 % D, Z = 2 % D;
        vc = __ldg(m.coeffs32 + ((int64_t)idx[0][ctr] * m.n[Y] + idx[Y][ctr]) * m.n[Z] + idx[Z][ctr]);
#pragma unroll
        for (int i = 0; i < taps; ++i) {
            float tw = 0.0f, ty = 0.0f, tyy = 0.0f, tz = 0.0f, tyz = 0.0f, tzz = 0.0f;
#pragma unroll
            for (int j = 0; j < taps; ++j) {
                const float *line = m.coeffs32 + ((int64_t)idx[0][i] * m.n[Y] + idx[Y][j]) * m.n[Z];
                float sw = 0.0f, sd = 0.0f, sdd = 0.0f;
#pragma unroll
                for (int k = 0; k < taps; ++k) {
                    const float v = __ldg(line + idx[Z][k]) - vc;
                    sw = fmaf(w[Z][k], v, sw);
                    sd = fmaf(d1[Z][k], v, sd);
                    sdd = fmaf(d2[Z][k], v, sdd);
                }
                tw = fmaf(w[Y][j], sw, tw);
                ty = fmaf(d1[Y][j], sw, ty);
                tyy = fmaf(d2[Y][j], sw, tyy);
                tz = fmaf(w[Y][j], sd, tz);
                tyz = fmaf(d1[Y][j], sd, tyz);
                tzz = fmaf(w[Y][j], sdd, tzz);
            }
            cc = fmaf(w[0][i], tw, cc);
            gg[0] = fmaf(d1[0][i], tw, gg[0]);
            gg[Y] = fmaf(w[0][i], ty, gg[Y]);
            gg[Z] = fmaf(w[0][i], tz, gg[Z]);
            hh[0][0] = fmaf(d2[0][i], tw, hh[0][0]);
            hh[0][Y] = fmaf(d1[0][i], ty, hh[0][Y]);
            hh[0][Z] = fmaf(d1[0][i], tz, hh[0][Z]);
            hh[Y][Y] = fmaf(w[0][i], tyy, hh[Y][Y]);
            hh[Y][Z] = fmaf(w[0][i], tyz, hh[Y][Z]);
            hh[Z][Z] = fmaf(w[0][i], tzz, hh[Z][Z]);
        }
    }
    // (the cubic weights are 6 x the true ones: see medium_args for the factors)
    // the value's weights sum to 1: the centre comes back in FP64
    c = m.c_ref + (double)vc + (double)cc * m.sv;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        g[a] = (double)gg[a] * m.sg[a];
#pragma unroll
        for (int b = 0; b < D; ++b) H[a * D + b] = (a <= b ? (double)hh[a][b] : (double)hh[b][a]) * m.sh[a][b];
    }
}

// The same for a medium kind known only at run time.
template <int D>
__device__ void speed_eval(const MediumArgs &m, const double *x, double &c, double *g, double *H) {
    switch (m.kind) {
        case MSGB_MEDIUM_CONSTANT: speed_eval_k<D, MSGB_MEDIUM_CONSTANT>(m, x, c, g, H); break;
        case MSGB_MEDIUM_LINEAR: speed_eval_k<D, MSGB_MEDIUM_LINEAR>(m, x, c, g, H); break;
        default: speed_eval_k<D, MSGB_MEDIUM_BSPLINE3>(m, x, c, g, H); break;
    }
}

template <int D>
struct State {
    double x[D], p[D];
    cd M[D][D];
    cd A;
};

// Smallest eigenvalue of a symmetric D x D matrix (exact for D <= 2,
// Gershgorin lower bound for D = 3).
template <int D>
__device__ __forceinline__ double lam_min(const double (*S)[D]) {
    if (D == 1) return S[0][0];
    if (D == 2) {
        const double a = S[0][0], b = 0.5 * (S[0][1 % D] + S[1 % D][0]), c = S[1 % D][1 % D];
        const double m = 0.5 * (a + c), r = sqrt(0.25 * (a - c) * (a - c) + b * b);
        return m - r;
    }
    double lo = 1e300;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        double s = S[i][i];
#pragma unroll
        for (int k = 0; k < D; ++k)
            if (k != i) s -= fabs(0.5 * (S[i][k] + S[k][i]));
        lo = fmin(lo, s);
    }
    return lo;
}

struct TrajArgs {
    int64_t nb, b_first, n;
    double *rec64;
    void *rec32;
    float *cull;
    int32_t *status;
    // compact FP32 store (pool != nullptr): see msgb_trajectories
    int32_t *slot = nullptr;
    void *pool = nullptr;
    float *pool_cull = nullptr;
    int64_t pool_blocks = 0;
    unsigned long long *pool_next = nullptr;
    bool align16 = false;  // the FP32 record base is 16-byte aligned (16-byte stores in 1D and 2D)
    const float *boxes = nullptr;
    int64_t n_boxes = 0;
    float live_cutoff = 0.0f;
};

// Host: the compact-store fields of a msgb_trajectories descriptor.
inline void set_compact(TrajArgs &T, const msgb_trajectories *t) {
    T.slot = t->slot;
    T.pool = t->pool;
    T.pool_cull = t->pool_cull;
    T.align16 = ((uintptr_t)(t->pool ? t->pool : t->rec32) & 15) == 0;
    T.pool_blocks = t->pool_blocks;
    T.pool_next = t->pool_next;
    T.boxes = t->live_boxes;
    T.n_boxes = t->n_boxes;
    T.live_cutoff = (float)t->live_cutoff;
}

inline int check_compact(const msgb_trajectories *t, int ndim) {
    if (!t->pool) return MSGB_OK;
    if (t->rec32) return fail(MSGB_ERR_ARG, "trajectories: rec32 and a compact pool are exclusive");
    if (!t->slot || !t->pool_cull || !t->pool_next || t->pool_blocks < 1)
        return fail(MSGB_ERR_ARG, "trajectories: compact store needs slot, pool_cull, pool_next and pool_blocks > 0");
    if (t->n_boxes < 0 || (t->n_boxes > 0 && !t->live_boxes))
        return fail(MSGB_ERR_ARG, "trajectories: live_boxes is NULL");
    if (!(t->live_cutoff >= 0.0)) return fail(MSGB_ERR_ARG, "trajectories: live_cutoff must be >= 0");
    (void)ndim;
    return MSGB_OK;
}


// Writes the records of one beam (index bl within the chunk) at every time k,
// and the culling box of each time tile as its last time is written.
template <int D>
struct RecordWriter {
    static constexpr int S = D * (D + 1) / 2;
    static constexpr int NR64 = 2 * D + 2 * D * D + 2;
    const ProbArgs &P;
    const TrajArgs &T;
    int64_t bl;
    double w;
    static constexpr int tt_len = MSGB_TIME_TILE;  // a power of two: no 64-bit division per record
    float lo[D], hi[D];
    double lmin = 1e300;
    bool bad = false;
    // compact store: this lane's block for the current time tile (-1: none
    // taken yet; kept across beams when a dead tile did not use it)
    int64_t blk = -1;

    __device__ RecordWriter(const ProbArgs &P_, const TrajArgs &T_, int64_t bl_, double w_)
        : P(P_), T(T_), bl(bl_), w(w_) {
#pragma unroll
        for (int i = 0; i < D; ++i) lo[i] = 3.4e38f, hi[i] = -3.4e38f;
    }

    // Start the records of another beam of the same chunk.
    __device__ void reset(int64_t bl_, double w_) {
        bl = bl_;
        w = w_;
        lmin = 1e300;
        bad = false;
#pragma unroll
        for (int i = 0; i < D; ++i) lo[i] = 3.4e38f, hi[i] = -3.4e38f;
    }

    // `failed`: the state is not trustworthy from here on (never culled).
    __device__ void put(int64_t k, const State<D> &y, bool failed) {
        bad |= failed;
        double xw[D];
#pragma unroll
        for (int i = 0; i < D; ++i) xw[i] = P.periodic[i] ? pymod(y.x[i], P.L[i]) : y.x[i];
        if (T.rec64) {
            double *r = T.rec64 + (k * T.nb + bl) * NR64;
            int q = 0;
#pragma unroll
            for (int i = 0; i < D; ++i) r[q++] = y.x[i];
#pragma unroll
            for (int i = 0; i < D; ++i) r[q++] = y.p[i];
#pragma unroll
            for (int i = 0; i < D; ++i)
#pragma unroll
                for (int l = 0; l < D; ++l) {
                    r[q++] = y.M[i][l].re;
                    r[q++] = y.M[i][l].im;
                }
            r[q++] = y.A.re;
            r[q++] = y.A.im;
        }
        char *base = record32(k);
        if (base) {
            float q[S], p[S];
#pragma unroll
            for (int i = 0; i < D; ++i)
#pragma unroll
                for (int l = i; l < D; ++l) {
                    const int e = sym_index<D>(i, l);
                    const double fac = 0.5 * w;  // off-diagonal: (M_il + M_li)/2 doubled
                    const double mre = i == l ? y.M[i][i].re : (y.M[i][l].re + y.M[l][i].re);
                    const double mim = i == l ? y.M[i][i].im : (y.M[i][l].im + y.M[l][i].im);
                    q[e] = (float)(fac * mre);
                    p[e] = (float)(fac * mim);
                }
            // arg A and 2|A| are stored as floats: FP32 arithmetic on the
            // rounded components gives them to FP32 precision
            store32(base, xw, y.p, q, p, (float)y.A.re, (float)y.A.im);
        }
        if (T.cull || T.pool) {
            double Sm[D][D];
#pragma unroll
            for (int i = 0; i < D; ++i)
#pragma unroll
                for (int l = 0; l < D; ++l) Sm[i][l] = y.M[i][l].im;
            bound(k, xw, lam_min<D>(Sm));
        }
    }

    // put() for the mixed-precision state: centre and momentum r (2 D doubles), the
    // Hessian and the amplitude f (re, im pairs in sym_index order, then A).
    __device__ __forceinline__ void put_mix(int64_t k, const double *r, const float *f, bool failed) {
        bad |= failed;
        double xw[D];
#pragma unroll
        for (int i = 0; i < D; ++i) xw[i] = P.periodic[i] ? pymod(r[i], P.L[i]) : r[i];
        char *base = record32(k);
        if (base) {
            float q[S], p[S];
#pragma unroll
            for (int i = 0; i < D; ++i)
#pragma unroll
                for (int l = i; l < D; ++l) {
                    const int e = sym_index<D>(i, l);
                    const double fac = (i == l ? 0.5 : 1.0) * w;
                    q[e] = (float)(fac * (double)f[2 * e]);
                    p[e] = (float)(fac * (double)f[2 * e + 1]);
                }
            store32(base, xw, r + D, q, p, f[2 * S], f[2 * S + 1]);
        }
        if (T.cull || T.pool) {
            double lam;
            if (D == 2) {
                // smaller eigenvalue as det / larger: the determinant in FP64, the
                // rest in FP32 (relative error below 1e-6, taken off here; zero, which
                // leaves no beam out, where a square would leave FP32's range)
                const double a = f[1], b = f[3 % (2 * S)], c = f[5 % (2 * S)];
                const float m = 0.5f * (f[1] + f[5 % (2 * S)]), h = 0.5f * (f[1] - f[5 % (2 * S)]);
                const float den = m + sqrtf(fmaf(h, h, f[3 % (2 * S)] * f[3 % (2 * S)]));
                const float det = (float)fma(a, c, -b * b);
                const float l = m > 1e-15f && m < 1e18f ? __fdividef(det, den) : 0.0f;
                lam = (double)(l - 1e-6f * fabsf(l));
            } else {
                double Sm[D][D];
#pragma unroll
                for (int i = 0; i < D; ++i)
#pragma unroll
                    for (int l = 0; l < D; ++l) Sm[i][l] = (double)f[2 * sym_index<D>(i, l) + 1];
                lam = lam_min<D>(Sm);
            }
            bound(k, xw, lam);
        }
    }

    // Where the FP32 record of time k goes, or nullptr.  A compact lane takes a
    // block at the start of a time tile unless it still has one.
    __device__ __forceinline__ char *record32(int64_t k) {
        if (T.pool) {
            const int kk = (int)((uint64_t)k % tt_len);
            if (kk == 0 && blk < 0) blk = (int64_t)atomicAdd(T.pool_next, 1ULL);
            if (blk >= 0 && blk < T.pool_blocks) return (char *)T.pool + (blk * tt_len + kk) * (int64_t)(16 * D + 8 * S + 8);
            return nullptr;
        }
        return T.rec32 ? (char *)T.rec32 + (k * T.nb + bl) * (int64_t)(16 * D + 8 * S + 8) : nullptr;
    }

    // The FP32 summation's BeamTime<D> record: x, w p, q, p, arg A, 2 |A|.
    __device__ __forceinline__ void store32(char *base, const double *xw, const double *mom, const float *q, const float *p,
                                            float are, float aim) {
        constexpr int NF = 2 * S + 2;
        float f[NF];
#pragma unroll
        for (int e = 0; e < S; ++e) f[e] = q[e], f[S + e] = p[e];
        f[2 * S] = atan2f(aim, (are == 0.0f && aim == 0.0f) ? 1e-12f : are);
        f[2 * S + 1] = 2.0f * hypotf(are, aim);
        if (D != 3 && T.align16) {  // 32 B (1D) or 64 B (2D) in 16-byte stores
            double d[2 * D];
#pragma unroll
            for (int i = 0; i < D; ++i) d[i] = xw[i], d[D + i] = w * mom[i];
            double2 *b2 = (double2 *)base;
#pragma unroll
            for (int i = 0; i < D; ++i) b2[i] = make_double2(d[2 * i], d[2 * i + 1]);
            float4 *b4 = (float4 *)(b2 + D);
#pragma unroll
            for (int i = 0; i < NF / 4; ++i) b4[i] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
            return;
        }
        double *xd = (double *)base;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            xd[i] = xw[i];
            xd[D + i] = w * mom[i];
        }
        float2 *b2 = (float2 *)(xd + 2 * D);
#pragma unroll
        for (int i = 0; i < NF / 2; ++i) b2[i] = make_float2(f[2 * i], f[2 * i + 1]);
    }

    // The culling box of the time tile: the centre xw and the smallest eigenvalue
    // lam of Im M at time k; written (with the tile's slot) at the tile's end.
    __device__ __forceinline__ void bound(int64_t k, const double *xw, double lam) {
        const int kk = (int)((uint64_t)k % tt_len);
        if (kk == 0) {
            lmin = 1e300;
#pragma unroll
            for (int i = 0; i < D; ++i) lo[i] = 3.4e38f, hi[i] = -3.4e38f;
        }
        lmin = fmin(lmin, lam);
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const float xf = (float)xw[i];
            lo[i] = fminf(lo[i], xf);
            hi[i] = fmaxf(hi[i], xf);
        }
        {
            if (kk == tt_len - 1 || k == P.nt - 1) {
                float box[2 * D + 1];
#pragma unroll
                for (int i = 0; i < D; ++i) {
                    // periodic axes and non-finite states are never culled
                    const bool open = P.periodic[i] || bad;
                    box[i] = open ? -3.4e38f : lo[i];
                    box[D + i] = open ? 3.4e38f : hi[i];
                }
                box[2 * D] = bad ? 0.0f : (float)fmax(0.0, 0.5 * w * lmin * (1.0 - 1e-6));
                if (T.pool) {
                    // live: within the cutoff of some sensor tile (the summation's
                    // own test, with the cutoff widened by 1e-4 so that every
                    // tile the summation keeps is stored)
                    bool live = bad || T.n_boxes == 0;
                    for (int64_t q = 0; q < T.n_boxes && !live; ++q) {
                        const float *tb = T.boxes + q * 2 * D;
                        float d2 = 0.0f;
#pragma unroll
                        for (int i = 0; i < D; ++i) {
                            const float gap = fmaxf(0.0f, fmaxf(tb[i] - box[D + i], box[i] - tb[D + i]));
                            d2 = fmaf(gap, gap, d2);
                        }
                        live = box[2 * D] * d2 * 0.999f <= T.live_cutoff * 1.0001f;
                    }
                    int32_t *sl = T.slot + (int64_t)((uint64_t)k / tt_len) * T.nb + bl;
                    if (live && blk >= 0 && blk < T.pool_blocks) {
                        *sl = (int32_t)blk;
                        float *c = T.pool_cull + blk * (2 * D + 1);
#pragma unroll
                        for (int i = 0; i < 2 * D + 1; ++i) c[i] = box[i];
                        blk = -1;  // the block belongs to this tile now
                    } else {
                        *sl = -1;  // dead tile (or pool exhausted): the block is reused
                    }
                } else {
                    float *c = T.cull + ((int64_t)((uint64_t)k / tt_len) * T.nb + bl) * (2 * D + 1);
#pragma unroll
                    for (int i = 0; i < 2 * D + 1; ++i) c[i] = box[i];
                }
            }
        }
    }
};

// Host: medium description -> kernel arguments (MSGB_OK or an error code).
inline int medium_args(const msgb_problem *prob, const msgb_medium *med, MediumArgs &M) {
    if (!med) return fail(MSGB_ERR_ARG, "medium is NULL");
    if (med->kind != MSGB_MEDIUM_CONSTANT) {
        if (med->kind != MSGB_MEDIUM_LINEAR && med->kind != MSGB_MEDIUM_BSPLINE3)
            return fail(MSGB_ERR_ARG, "unknown medium kind %d", med->kind);
        if (!med->coeffs) return fail(MSGB_ERR_ARG, "medium grid is NULL");
        if (med->boundary < 0 || med->boundary > 3) return fail(MSGB_ERR_ARG, "unknown boundary %d", med->boundary);
        for (int a = 0; a < prob->ndim; ++a)
            if (med->n[a] < 1 || !(med->spacing[a] > 0.0)) return fail(MSGB_ERR_ARG, "bad medium grid");
    } else if (!(med->c > 0.0)) {
        return fail(MSGB_ERR_ARG, "constant medium speed must be > 0");
    }
    M = MediumArgs{};
    M.kind = med->kind;
    M.boundary = med->boundary;
    for (int a = 0; a < 3; ++a) {
        M.n[a] = med->n[a];
        M.spacing[a] = med->spacing[a];
        M.origin[a] = med->origin[a];
    }
    for (int a = 0; a < 3; ++a) M.inv_spacing[a] = 1.0 / M.spacing[a];
    M.coeffs = med->coeffs;
    M.c = med->c;
    M.lam = med->lam;
    M.coeffs32 = med->coeffs32;
    M.c_ref = med->c_ref;
    // The cubic sums carry 6 x the B-spline weights (no FP64 division per
    // weight): a sum whose terms carry the plain weight of q axes is 6^q too
    // large (value: all axes; gradient and diagonal Hessian: ndim - 1; mixed
    // Hessian: ndim - 2).
    const double s6 = med->kind == MSGB_MEDIUM_BSPLINE3 ? 1.0 / 6.0 : 1.0;
    const int D = prob->ndim;
    M.sv = D == 1 ? s6 : (D == 2 ? s6 * s6 : s6 * s6 * s6);
    const double sg = D == 1 ? 1.0 : (D == 2 ? s6 : s6 * s6), sm = D == 3 ? s6 : 1.0;
    for (int a = 0; a < D; ++a) {
        M.sg[a] = sg * M.inv_spacing[a];
        for (int b = 0; b < D; ++b) M.sh[a][b] = (a == b ? sg : sm) * M.inv_spacing[a] * M.inv_spacing[b];
    }
    return MSGB_OK;
}

}  // namespace
}  // namespace msgb
