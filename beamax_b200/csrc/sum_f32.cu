// FP32 Gaussian-beam summation with Gaussian-cutoff culling, and its transpose.
//
// Same operator as compute_gaussian_beam_real (beamax gb/core.py:194-329)
// with solve_hom_diag (gb/gb_solvers.py:356-422):
//   out(t, s) = sum_b Re[z_b(t, s)],  z = 2|A| exp(i theta - chi),
//   theta = w (p.D + D^T Re M D / 2) + arg A,  chi = w D^T Im M D / 2,
//   D = s - x_b(t).
//
// Precision plan
//  * Sensors are grouped into tiles of TS sensors, ordered so that tiles hold
//    straight, evenly spaced runs (coarse-cell Morton order, row-major inside a
//    cell).  Each tile has an FP64 anchor s0.  Per (beam, time) the large phase
//    w p.(s0 - x(t)) + arg A is formed in FP64 and reduced to [-pi, pi) before
//    it meets FP32; per sensor only w p.(s - s0) (bounded by the tile) is FP32.
//  * Along a run s_k = s_a + k h the exponent i theta - chi is a quadratic in k,
//    so z_{k+1} = z_k r_k, r_{k+1} = r_k q with r_0 = exp(a1 + a2), q =
//    exp(2 a2): two complex multiplies per sensor.  Every run starts with a
//    direct evaluation (MUFU sincos/exp after explicit range reduction) and
//    runs are at most GS sensors long, which bounds the recurrence's relative
//    error growth (~k^2 eps / 2 < 1e-5).
//  * Accumulation across beams is Kahan-compensated FP32.
// Culling: for a (beam, time tile, sensor tile) triple
//   chi >= (w/2) lambda_min(Im M(t)) |D|^2 >= (w/2) lam_lo(t_b) dist^2,
// lam_lo(t) = 1 / (1/beta_min + (c t/|p|)^2 beta_max): with M0 = i diag(beta),
// Im M(t) = (S + R S^-1 R)^-1, S = diag(1/beta), R = (c t/|p|) P_perp, which is
// Loewner-decreasing in |t|; dist is the gap between the bounding boxes of the
// centre's path over the time tile and of the sensor tile.  A triple is
// skipped when that bound exceeds `cutoff` e-folds.
#include <cub/cub.cuh>

#include <mutex>

#include "common.cuh"

namespace msgb {
namespace {

constexpr int TT = 32;               // times per tile (= lanes)
constexpr int GS = 16;               // sensors per warp group and maximal run length
constexpr int NW = 8;                // warps per CTA (forward)
constexpr int TS = GS * NW;          // sensors per tile
constexpr int THREADS = NW * 32;
// Beams per record pass.  Every warp then evaluates only the beams that reach
// its own sensor group (about a quarter to a half of them), so the pass has to
// be long enough for the warps' shares to even out between the barriers: 8
// beams per pass left the warps idle there, 32 is the most that two CTAs' records
// (80 KB each in 3D) leave room for on an SM.
constexpr int G = 32;
static_assert(G == 32, "a warp's share of a pass is one 32-bit mask");
constexpr float kTwoPi = 6.283185307179586f;
constexpr float kInvTwoPi = 0.15915494309189535f;

// Reduce an FP32 angle to [-pi, pi] (bounded inputs, |th| < 2^22 turns).  The
// nearest integer comes from adding 1.5 * 2^23 on the FMA pipe: rintf runs on
// the MUFU pipe, which the seeds' sin/cos/exp already fill (a complex
// exponential measured 25.4 cycles per warp and scheduler instead of 32.8).
__device__ __forceinline__ float reduce_angle(float th) {
    const float k = __fadd_rn(fmaf(th, kInvTwoPi, 12582912.0f), -12582912.0f);
    return fmaf(-k, kTwoPi, th);
}

struct cf {
    float re, im;
};
__device__ __forceinline__ cf cmul(cf a, cf b) {
    return cf{fmaf(a.re, b.re, -a.im * b.im), fmaf(a.re, b.im, a.im * b.re)};
}
__device__ __forceinline__ cf cdiv(cf a, cf b) {
    const float inv = __frcp_rn(fmaf(b.re, b.re, b.im * b.im));
    return cf{(a.re * b.re + a.im * b.im) * inv, (a.im * b.re - a.re * b.im) * inv};
}
__device__ __forceinline__ cf csqrtf_(cf z) {
    const float m = sqrtf(fmaf(z.re, z.re, z.im * z.im));
    if (m == 0.0f) return cf{0.0f, 0.0f};
    const float r = sqrtf(0.5f * (m + fabsf(z.re)));
    if (z.re >= 0.0f) return cf{r, z.im / (2.0f * r)};
    return cf{fabsf(z.im) / (2.0f * r), copysignf(r, z.im)};
}
// Two complex numbers, component-packed, for the paired FP32 instructions of
// sm_100 (FFMA2 / FMUL2 / FADD2).  Each lane of a paired operation rounds
// exactly as the scalar instruction, so these produce the same bits as cmul
// and kahan_add applied to each half.
struct cf2 {
    float2 re, im;
};
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ cf2 cmul2(cf2 a, cf2 b) {
    return cf2{__ffma2_rn(a.re, b.re, neg2(__fmul2_rn(a.im, b.im))), __ffma2_rn(a.re, b.im, __fmul2_rn(a.im, b.re))};
}
__device__ __forceinline__ void kahan_add2(float2 &acc, float2 &cmp, float2 v) {
    const float2 y = __fadd2_rn(v, neg2(cmp));
    const float2 t = __fadd2_rn(acc, y);
    cmp = __fadd2_rn(__fadd2_rn(t, neg2(acc)), neg2(y));
    acc = t;
}
__device__ __forceinline__ cf2 pack2(cf a, cf b) { return cf2{make_float2(a.re, b.re), make_float2(a.im, b.im)}; }

// exp(x + i y) with y range-reduced first.
__device__ __forceinline__ cf cexpf_(float x, float y) {
    float s, c;
    __sincosf(reduce_angle(y), &s, &c);
    const float e = __expf(x);
    return cf{e * c, e * s};
}

template <int D>
struct Sym {
    static constexpr int S = D * (D + 1) / 2;
};

// Quadratic form with packed coefficients (off-diagonals already doubled).
template <int D>
__device__ __forceinline__ float quad(const float *c, const float *v) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) r = fmaf(c[sym_index<D>(i, k)], v[i] * v[k], r);
    return r;
}
// 2 u^T C v for the same packed coefficients.
template <int D>
__device__ __forceinline__ float bilin2(const float *c, const float *u, const float *v) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) {
            const float ck = c[sym_index<D>(i, k)];
            r = (i == k) ? fmaf(2.0f * ck, u[i] * v[i], r) : fmaf(ck, fmaf(u[i], v[k], u[k] * v[i]), r);
        }
    return r;
}

// Per (beam, time) evaluation record.
template <int D>
struct Rec {
    float d0[D];             // s0 - x(t)
    float wp[D];             // w p
    float q[Sym<D>::S];      // w/2 Re M (off-diagonals doubled)
    float p[Sym<D>::S];      // w/2 Im M (off-diagonals doubled)
    float th0;               // reduce(w p.(s0 - x(t)) + arg A)
    float amp;               // 2 |A(t)|
    static constexpr int NF = 2 * D + 2 * Sym<D>::S + 2;
};

// Tile-independent part of a record (the FP64 centre and the FP32 shape).
template <int D>
struct BeamTime {
    double x[D];
    double wp[D];
    float q[Sym<D>::S], p[Sym<D>::S];
    float ang, amp;
};

// Per selected coefficient culling data (mode independent).
template <int D>
struct Cull {
    float x0[D];
    float dir[D];   // p0 / |p0|
    float bmin, bmax, w, inv_np;
    int ok;         // 0: M0 not of the form i diag(beta) -> never culled
};

template <int D>
struct TileInfo {
    double s0[D];
    float lo[D], hi[D];
};

// Closed-form Hessian and amplitude in FP32 (gb_solvers.py:306-353, :194-264).
template <int D>
__device__ __forceinline__ void hom_mA_f32(const float *p0, const cf *al, cf a0, float c0t, cf *M, cf &A) {
    float n2 = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) n2 = fmaf(p0[i], p0[i], n2);
    const float np = sqrtf(n2);
    const float inv_np = 1.0f / np;
    const float np3 = n2 * np;
    cf Ainv[D], Ainv_u[D], vT[D];
    float u[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        const float f = c0t * inv_np;
        cf Ad = cf{fmaf(f, al[i].re, 1.0f), f * al[i].im};
        Ainv[i] = cdiv(cf{1.0f, 0.0f}, Ad);
        u[i] = -c0t * p0[i] / np3;
        Ainv_u[i] = cf{u[i] * Ainv[i].re, u[i] * Ainv[i].im};
        cf t = cmul(al[i], Ainv[i]);
        vT[i] = cf{p0[i] * t.re, p0[i] * t.im};
    }
    cf sc = cf{1.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < D; ++j) sc = cf{fmaf(u[j], vT[j].re, sc.re), fmaf(u[j], vT[j].im, sc.im)};
    const cf isc = cdiv(cf{1.0f, 0.0f}, sc);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = i; j < D; ++j) {
            cf Y = cmul(cmul(Ainv_u[i], vT[j]), isc);
            Y = cf{-Y.re, -Y.im};
            if (i == j) Y = cf{Y.re + Ainv[i].re, Y.im + Ainv[i].im};
            M[sym_index<D>(i, j)] = cmul(al[i], Y);
        }
    if (D == 3) {
        const float p1 = p0[0] * p0[0], p2 = p0[1 % D] * p0[1 % D], p3 = p0[2 % D] * p0[2 % D];
        const cf a1 = al[0], a2 = al[1 % D], a3 = al[2 % D];
        const float tsc = c0t / (n2 * n2);
        auto term = [&](cf x, cf y) {
            cf xy = cmul(x, y);
            return cf{fmaf(c0t, xy.re, np * (x.re + y.re)), fmaf(c0t, xy.im, np * (x.im + y.im))};
        };
        cf t1 = term(a2, a3), t2 = term(a1, a3), t3 = term(a1, a2);
        cf s = cf{p1 * t1.re + p2 * t2.re + p3 * t3.re, p1 * t1.im + p2 * t2.im + p3 * t3.im};
        cf den = cf{fmaf(tsc, s.re, 1.0f), tsc * s.im};
        A = cdiv(a0, csqrtf_(den));
    } else if (D == 2) {
        cf ap = cf{(p0[0] * p0[0] * al[1 % D].re + p0[1 % D] * p0[1 % D] * al[0].re) / np3,
                   (p0[0] * p0[0] * al[1 % D].im + p0[1 % D] * p0[1 % D] * al[0].im) / np3};
        A = cdiv(a0, csqrtf_(cf{fmaf(c0t, ap.re, 1.0f), c0t * ap.im}));
    } else {
        A = a0;
    }
}

// Beam b in [0, 2n) (b >= n: mode -1) at time t, anchor-independent part.
template <int D>
__device__ __forceinline__ void beam_time(const ProbArgs &P, const BeamArgs &B, int64_t b, double t,
                                          BeamTime<D> &r) {
    const int64_t j = b < B.n ? b : b - B.n;
    const double c0 = b < B.n ? P.c : -P.c;
    double p0d[D], n2 = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        p0d[i] = B.p0[j * D + i];
        n2 += p0d[i] * p0d[i];
    }
    const double np = sqrt(n2);
    const double w = B.omega[j];
    float p0f[D];
    cf al[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        double x = B.x0[j * D + i] + c0 * (p0d[i] / np) * t;
        if (P.periodic[i]) x = pymod(x, P.L[i]);
        r.x[i] = x;
        r.wp[i] = w * p0d[i];
        p0f[i] = (float)p0d[i];
        al[i] = cf{(float)B.alpha[2 * (j * D + i)], (float)B.alpha[2 * (j * D + i) + 1]};
    }
    cf M[Sym<D>::S], A;
    hom_mA_f32<D>(p0f, al, cf{(float)B.a0[2 * j], (float)B.a0[2 * j + 1]}, (float)(c0 * t), M, A);
    const float wf = (float)w;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) {
            const int q = sym_index<D>(i, k);
            const float f = (i == k ? 0.5f : 1.0f) * wf;
            r.q[q] = f * M[q].re;
            r.p[q] = f * M[q].im;
        }
    float re = A.re;
    if (A.re == 0.0f && A.im == 0.0f) re = 1e-12f;
    r.ang = atan2f(A.im, re);
    r.amp = 2.0f * sqrtf(fmaf(A.re, A.re, A.im * A.im));
}

// What the closed form needs per selected coefficient (mode independent),
// prepared in FP64 once per call.  With M0 = i diag(beta), u = p0/|p0| and n_j the
// eigenvectors of diag(beta) restricted to the plane normal to u (eigenvalues d_j),
// diag(beta) = e u u^T + sum_j d_j nu_j nu_j^T, nu_j = n_j + (n_j.beta u / d_j) u, and
//   M(t) = i e u u^T + sum_j d_j k_j (x_j + i) nu_j nu_j^T,  x_j = c t d_j / |p0|,
//   k_j = 1 / (1 + x_j^2),  A(t) = a0 prod_j (1 + i x_j)^(-1/2),
// the Sherman-Morrison closed form (gb_solvers.py:194-264, :306-353) written as a sum
// of positive terms: no cancellation in FP32 and one division per transverse axis
// instead of complex divisions and a complex square root per record.
template <int D>
struct alignas(16) HomBeam {
    static constexpr int NT = D - 1;  // transverse axes
    double x0[D], v[D], wp[D];        // centre, velocity c u (mode +1), w p0
    float N[NT > 0 ? NT : 1][Sym<D>::S];  // w/2 d_j nu_j nu_j^T (off-diagonals doubled)
    float U[Sym<D>::S];                   // w/2 e u u^T (off-diagonals doubled)
    float td[NT > 0 ? NT : 1];            // c d_j / |p0|
    float aabs, aarg;                     // a0
    int ok;                               // 0: M0 not i diag(beta > 0): beam_time is used
};

template <int D>
__device__ __forceinline__ HomBeam<D> make_hom_beam(const ProbArgs &P, const BeamArgs &B, int64_t j) {
    HomBeam<D> h;
    double p0[D], beta[D], n2 = 0.0;
    h.ok = 1;
    const double w = B.omega[j];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        p0[i] = B.p0[j * D + i];
        n2 += p0[i] * p0[i];
        beta[i] = B.alpha[2 * (j * D + i) + 1];
        if (B.alpha[2 * (j * D + i)] != 0.0 || !(beta[i] > 0.0)) h.ok = 0;
    }
    const double np = sqrt(n2);
    if (!(np > 0.0)) h.ok = 0;
    double u[D], n[D][D];  // n[j]: transverse directions, j < D - 1
#pragma unroll
    for (int i = 0; i < D; ++i) {
        u[i] = p0[i] / np;
        h.x0[i] = B.x0[j * D + i];
        h.v[i] = P.c * u[i];
        h.wp[i] = w * p0[i];
    }
    if (D == 2) {
        n[0][0] = -u[1 % D];
        n[0][1 % D] = u[0];
    } else if (D == 3) {
        // any orthonormal pair normal to u, then turned onto the eigenvectors
        const int ax = fabs(u[0]) < 0.6 ? 0 : 1;
        double e0[3] = {ax == 0 ? 1.0 : 0.0, ax == 1 ? 1.0 : 0.0, 0.0};
        double a[3], b[3], aa = 0.0;
        const double eu = e0[0] * u[0] + e0[1] * u[1 % D];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = e0[i] - eu * u[i % D];
            aa += a[i] * a[i];
        }
        const double ia = 1.0 / sqrt(aa);
#pragma unroll
        for (int i = 0; i < 3; ++i) a[i] *= ia;
        b[0] = u[1 % D] * a[2] - u[2 % D] * a[1];
        b[1] = u[2 % D] * a[0] - u[0] * a[2];
        b[2] = u[0] * a[1] - u[1 % D] * a[0];
        double daa = 0.0, dab = 0.0, dbb = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            daa += beta[i % D] * a[i] * a[i];
            dab += beta[i % D] * a[i] * b[i];
            dbb += beta[i % D] * b[i] * b[i];
        }
        double sn, cs;
        sincos(0.5 * atan2(2.0 * dab, daa - dbb), &sn, &cs);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            n[0][i % D] = cs * a[i] + sn * b[i];
            n[1 % D][i % D] = cs * b[i] - sn * a[i];
        }
    }
    double e = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) e += beta[i] * u[i] * u[i];
#pragma unroll
    for (int q = 0; q < D - 1; ++q) {
        double d = 0.0, b = 0.0, nu[D];
#pragma unroll
        for (int i = 0; i < D; ++i) {
            d += beta[i] * n[q][i] * n[q][i];
            b += beta[i] * n[q][i] * u[i];
        }
        e -= b * b / d;
#pragma unroll
        for (int i = 0; i < D; ++i) nu[i] = n[q][i] + (b / d) * u[i];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int k = i; k < D; ++k)
                h.N[q][sym_index<D>(i, k)] = (float)((i == k ? 0.5 : 1.0) * w * d * nu[i] * nu[k]);
        h.td[q] = (float)(P.c * d / np);
    }
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) h.U[sym_index<D>(i, k)] = (float)((i == k ? 0.5 : 1.0) * w * e * u[i] * u[k]);
    const float ar = (float)B.a0[2 * j], ai = (float)B.a0[2 * j + 1];
    h.aabs = hypotf(ar, ai);
    h.aarg = atan2f(ai, (ar == 0.0f && ai == 0.0f) ? 1e-12f : ar);
    return h;
}

template <int D>
__global__ void hom_prep_kernel(ProbArgs P, BeamArgs B, HomBeam<D> *out) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j < B.n) out[j] = make_hom_beam<D>(P, B, j);
}

// Largest e-fold count the run recurrence may meet: at the seed (chi), in the
// first step's ratio and in the ratio's own step.  Beyond it the factors leave
// FP32's range (e^88) and the recurrence would produce 0 * inf; such runs are
// evaluated directly.  Only very narrow beams (e-fold width under about one
// sensor spacing over a 16-sensor run, e.g. after focusing in a
// heterogeneous medium) reach it.
constexpr float kRecurrenceEfolds = 60.0f;
// A run whose smallest exponent over its 16 sensors exceeds this many e-folds
// contributes below 4e-18 of the beam's amplitude and is skipped (only when
// culling is enabled, cutoff > 0).
constexpr float kNegligibleEfolds = 40.0f;

// Margin, in e-folds beyond the cutoff, of the per-group test: a (beam, time
// tile) whose smallest exponent over a group of GS sensors and the 32 times is
// larger than cutoff + margin is left out for that group.  The tile test
// (survives, traj_survives) bounds the exponent with the smallest eigenvalue of
// Im M and a box around 128 sensors, so most of what it keeps lies far outside the
// beam: at 1024^2 heterogeneous 67 % of the (beam, group) pairs it kept were
// beyond 24 e-folds, 33 % at 512^2 homogeneous, 56 % at 128^3.
constexpr float kGroupMarginEfolds = 4.0f;

// One warp's sensor group: its straight run's start and step.
template <int D>
struct Run {
    float ds[D], h[D];
};

// Smallest exponent chi(k) = chi + B k + A k^2 over k in [0, GS - 1].
__device__ __forceinline__ float run_chi_min(float chi, float Bq, float Aq) {
    constexpr float kl = (float)(GS - 1);
    const float kv = Aq > 0.0f ? fminf(fmaxf(__fdividef(-0.5f * Bq, Aq), 0.0f), kl) : 0.0f;
    return fminf(fminf(chi, fmaf(kl, fmaf(Aq, kl, Bq), chi)), fmaf(kv, fmaf(Aq, kv, Bq), chi));
}

// Direct evaluation at sensor offset ds: z.
template <int D, bool PERIODIC>
__device__ __forceinline__ cf direct_eval(const Rec<D> &r, const float *ds, const ProbArgs &P) {
    float Dl[D];
    float th = r.th0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        Dl[i] = ds[i] + r.d0[i];
        if (PERIODIC && P.periodic[i]) Dl[i] -= (float)P.L[i] * rintf(Dl[i] / (float)P.L[i]);
        th = fmaf(r.wp[i], ds[i], th);
    }
    th += quad<D>(r.q, Dl);
    cf z = cexpf_(-quad<D>(r.p, Dl), th);
    return cf{z.re * r.amp, z.im * r.amp};
}

// Run start: z, the ratio f to the next sensor and the ratio's own step q.
// Returns true when the run has to be evaluated directly (z = f = q = 0 then):
// its factors would leave FP32's range and some sensor of it is not negligible.
template <int D>
__device__ __forceinline__ bool seed_eval(const Rec<D> &r, const Run<D> &g, bool skip_negligible, cf &z, cf &f, cf &q) {
    float Dl[D];
    float th = r.th0, wh = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        Dl[i] = g.ds[i] + r.d0[i];
        th = fmaf(r.wp[i], g.ds[i], th);
        wh = fmaf(r.wp[i], g.h[i], wh);
    }
    th += quad<D>(r.q, Dl);
    const float chi = quad<D>(r.p, Dl);
    z = cexpf_(-chi, th);
    z.re *= r.amp;
    z.im *= r.amp;
    const float a1r = -bilin2<D>(r.p, g.h, Dl), a1i = wh + bilin2<D>(r.q, g.h, Dl);
    const float a2r = -quad<D>(r.p, g.h), a2i = quad<D>(r.q, g.h);
    f = cexpf_(a1r + a2r, a1i + a2i);
    q = cexpf_(2.0f * a2r, 2.0f * a2i);
    bool direct = false;
    if (chi > kRecurrenceEfolds || a1r + a2r > kRecurrenceEfolds || -2.0f * a2r > kRecurrenceEfolds) {
        direct = !(skip_negligible && run_chi_min(chi, -a1r, -a2r) > kNegligibleEfolds);
        z = f = q = cf{0.0f, 0.0f};
    }
    return direct;
}

template <int D>
__device__ __forceinline__ bool survives(const Cull<D> &cb, float c0, float ta, float tb, const TileInfo<D> &ti,
                                         const ProbArgs &P, float cutoff) {
    if (!cb.ok || cutoff <= 0.0f) return true;
    float d2 = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        if (P.periodic[i]) continue;
        const float v = c0 * cb.dir[i];
        const float xa = fmaf(v, ta, cb.x0[i]), xb = fmaf(v, tb, cb.x0[i]);
        const float mn = fminf(xa, xb), mx = fmaxf(xa, xb);
        const float gap = fmaxf(0.0f, fmaxf(ti.lo[i] - mx, mn - ti.hi[i]));
        d2 = fmaf(gap, gap, d2);
    }
    const float k = fabsf(c0) * fmaxf(fabsf(ta), fabsf(tb)) * cb.inv_np;
    const float lam = 1.0f / (1.0f / cb.bmin + k * k * cb.bmax);
    return 0.5f * cb.w * lam * d2 * 0.999f <= cutoff;
}

// ------------------------------------------------------------------ prep
// Sort key: Morton order of coarse cells (32 per axis), row-major inside a
// cell, so axis-aligned lines and planes form evenly spaced runs.
template <int D>
__global__ void sensor_key_kernel(const double *sens, int64_t ns, ProbArgs P, uint32_t *key, int32_t *val) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= ns) return;
    const int bits = D == 1 ? 31 : (D == 2 ? 16 : 10);
    const int cellbits = 5;
    const int lowbits = bits - cellbits;
    uint32_t q[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        double u = sens[s * D + i] / P.L[i];
        u = fmin(fmax(u, 0.0), 1.0 - 1e-12);
        q[i] = (uint32_t)(u * (double)(1u << bits));
    }
    uint32_t k = 0;
    if (D == 1) {
        k = q[0];
    } else {
        for (int b = cellbits - 1; b >= 0; --b)
#pragma unroll
            for (int i = 0; i < D; ++i) k = (k << 1) | ((q[i] >> (lowbits + b)) & 1u);
#pragma unroll
        for (int i = 0; i < D; ++i) k = (k << lowbits) | (q[i] & ((1u << lowbits) - 1u));
    }
    key[s] = k;
    val[s] = (int32_t)s;
}

// Per tile: anchor, bounding box, FP32 offsets, steps and the per-group fast flag (one
// straight run of GS sensors, no periodic wrap).
template <int D>
__global__ void tile_kernel(const double *sens, const int32_t *perm, const int32_t *offs, ProbArgs P,
                            TileInfo<D> *tiles, float *ds, float *hn, uint8_t *gfast) {
    const int64_t tile = blockIdx.x;
    const int64_t first = offs[tile];
    const int cnt = offs[tile + 1] - offs[tile];
    __shared__ double lo[D], hi[D];
    __shared__ double pos[TS][D];
    for (int k = threadIdx.x; k < cnt; k += blockDim.x)
        for (int i = 0; i < D; ++i) pos[k][i] = sens[(int64_t)perm[first + k] * D + i];
    __syncthreads();
    bool any_periodic = false;
    for (int i = 0; i < D; ++i) any_periodic |= (P.periodic[i] != 0);
    if (threadIdx.x == 0) {
        for (int i = 0; i < D; ++i) {
            double a = 1e300, b = -1e300;
            for (int k = 0; k < cnt; ++k) {
                a = fmin(a, pos[k][i]);
                b = fmax(b, pos[k][i]);
            }
            lo[i] = a;
            hi[i] = b;
            tiles[tile].s0[i] = 0.5 * (a + b);
            tiles[tile].lo[i] = (float)a;
            tiles[tile].hi[i] = (float)b;
        }
        // run starts: a run continues while the step stays the same
        bool have_h = false;
        double hh[D];
        unsigned fastmask = 0;
        for (int k = 0; k < TS; ++k) {
            bool s = true;
            if (k < cnt) {
                s = (k % GS == 0) || any_periodic;
                if (!s) {
                    double st[D], n2 = 0.0, e2 = 0.0;
                    for (int i = 0; i < D; ++i) {
                        st[i] = pos[k][i] - pos[k - 1][i];
                        n2 += st[i] * st[i];
                    }
                    if (!have_h) {
                        for (int i = 0; i < D; ++i) hh[i] = st[i];
                        have_h = n2 > 0.0;
                        s = !have_h;
                    } else {
                        for (int i = 0; i < D; ++i) e2 += (st[i] - hh[i]) * (st[i] - hh[i]);
                        s = e2 > 1e-12 * n2;
                    }
                }
            }
            if (s) have_h = false;
            if (k % GS == 0) fastmask = 1;
            if (k % GS != 0 && s) fastmask = 0;
            if (k % GS == GS - 1) gfast[tile * NW + k / GS] = (fastmask && (k < cnt) && !any_periodic) ? 1 : 0;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
        for (int i = 0; i < D; ++i) {
            const double c = 0.5 * (lo[i] + hi[i]);
            ds[(first + k) * D + i] = (float)(pos[k][i] - c);
            hn[(first + k) * D + i] = (k + 1 < cnt) ? (float)(pos[k + 1][i] - pos[k][i]) : 0.0f;
        }
    }
}

__global__ void fixed_offsets_kernel(int32_t *offs, int64_t n_tiles, int64_t ns) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i <= n_tiles) offs[i] = (int32_t)min((int64_t)i * TS, ns);
}

template <int D>
__global__ void cull_prep_kernel(BeamArgs B, Cull<D> *out) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= B.n) return;
    Cull<D> c;
    double n2 = 0.0;
    for (int i = 0; i < D; ++i) n2 += B.p0[j * D + i] * B.p0[j * D + i];
    const double np = sqrt(n2);
    float bmin = 1e30f, bmax = 0.0f;
    int ok = 1;
    for (int i = 0; i < D; ++i) {
        c.x0[i] = (float)B.x0[j * D + i];
        c.dir[i] = (float)(B.p0[j * D + i] / np);
        const double re = B.alpha[2 * (j * D + i)], im = B.alpha[2 * (j * D + i) + 1];
        if (re != 0.0 || !(im > 0.0)) ok = 0;
        bmin = fminf(bmin, (float)im);
        bmax = fmaxf(bmax, (float)im);
    }
    c.bmin = bmin;
    c.bmax = bmax;
    c.w = (float)B.omega[j];
    c.inv_np = (float)(1.0 / np);
    c.ok = ok && np > 0.0;
    out[j] = c;
}

// data (nt, ns) in caller order -> (ns, nt) in sorted sensor order.
__global__ void transpose_permute_kernel(const float *data, const int32_t *perm, int64_t nt, int64_t ns, float *out) {
    __shared__ float tile[32][33];
    const int64_t s0 = (int64_t)blockIdx.x * 32, t0 = (int64_t)blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t t = t0 + k, s = s0 + threadIdx.x;
        tile[k][threadIdx.x] = (t < nt && s < ns) ? data[t * ns + perm[s]] : 0.0f;
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t s = s0 + k, t = t0 + threadIdx.x;
        if (s < ns && t < nt) out[s * nt + t] = tile[threadIdx.x][k];
    }
}

// ------------------------------------------------------------------ trajectories
// Records written by msgb_rk4_trajectories (rec32) for a chunk of beams, the
// per-time-tile culling boxes, and the Kahan state carried across chunks.
template <int D>
struct TrajSrc {
    int64_t nb, b_first;
    const BeamTime<D> *rec;   // dense: (nt, nb)
    const float *cull;        // dense: (n_tt, nb, 2D + 1)
    const int32_t *slot;      // compact: (n_tt, nb) block or -1
    const BeamTime<D> *pool;  // compact: (blocks, TT)
    const float *pool_cull;   // compact: (blocks, 2D + 1)
    float *state;             // (2, nt, ns) Kahan sum / compensation, sorted sensor order
    const uint32_t *limits;   // (n_tt, nb): see traj_limits_kernel; nullptr: refine is not run
    int first, last;
};

template <int D>
__device__ __forceinline__ bool traj_survives(const TrajSrc<D> &T, int64_t bl, int64_t tt, const TileInfo<D> &ti,
                                              float cutoff) {
    const float *c;
    if (T.pool) {
        const int32_t blk = T.slot[tt * T.nb + bl];
        if (blk < 0) return false;  // no sensor tile within the cutoff: not stored
        if (cutoff <= 0.0f) return true;
        c = T.pool_cull + (int64_t)blk * (2 * D + 1);
    } else {
        if (cutoff <= 0.0f) return true;
        c = T.cull + (tt * T.nb + bl) * (2 * D + 1);
    }
    float d2 = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        const float gap = fmaxf(0.0f, fmaxf(ti.lo[i] - c[D + i], c[i] - ti.hi[i]));
        d2 = fmaf(gap, gap, d2);
    }
    return c[2 * D] * d2 * 0.999f <= cutoff;
}

constexpr int SCAN = 4;  // beams tested per thread and scan

// ------------------------------------------------------------------ record passes
// A record pass holds up to G beams' records at the tile's 32 times in shared
// memory, rec[field][beam][time], and per beam an 8-bit mask of the warps (sensor
// groups) it reaches.  Warp w of the pass writes beams w, w + 8, ...: lane = time.
template <int D>
constexpr size_t rec_bytes() {
    return sizeof(float) * Rec<D>::NF * G * TT;
}

// One group of GS sensors, for the test of the record pass: the run's start and
// step (one straight run), or a ball around the sensors.
template <int D>
struct GroupInfo {
    float ds[D], h[D];  // straight run: start and step; else: centre (ds)
    float rad;          // else: largest distance of a sensor from the centre
    int kind;           // 0 no sensors, 1 straight run, 2 other, 3 never left out (periodic)
};

template <int D>
struct TileGroups {
    GroupInfo<D> g[NW];
    // lattice: the n groups are straight runs with one step, starting at
    // g[0].ds + k e (a 128-sensor line, or rows of a detector plane)
    float e[D];
    int lattice, n;
    unsigned present;  // groups that hold sensors
};

// Is Im M positive definite?  (Not where it is not finite.)
template <int D>
__device__ __forceinline__ bool positive_form(const float *p) {
    if (D == 1) return p[0] > 0.0f;
    // leading minors, the off-diagonals of p being doubled
    const float a = p[sym_index<D>(0, 0)], b = 0.5f * p[sym_index<D>(0, 1 % D)], d = p[sym_index<D>(1 % D, 1 % D)];
    const float m = fmaf(a, d, -b * b);
    if (D == 2) return a > 0.0f && m > 0.0f;
    const float c = 0.5f * p[sym_index<D>(0, 2 % D)], e = 0.5f * p[sym_index<D>(1 % D, 2 % D)];
    const float f = p[sym_index<D>(2 % D, 2 % D)];
    return a > 0.0f && m > 0.0f && fmaf(m, f, -fmaf(a * e, e, c * fmaf(d, c, -2.0f * b * e))) > 0.0f;
}

// Does a record reach group g within thr e-folds?  No only if a lower bound on its
// exponent is above thr: a NaN is not, and such a record is evaluated.  positive: Im M
// is positive definite.
template <int D>
__device__ __forceinline__ bool group_reached(const Rec<D> &r, bool positive, const GroupInfo<D> &g, float thr) {
    float Dl[D];
#pragma unroll
    for (int i = 0; i < D; ++i) Dl[i] = g.ds[i] + r.d0[i];
    const float chi = quad<D>(r.p, Dl);
    if (g.kind == 1) return !(run_chi_min(chi, bilin2<D>(r.p, g.h, Dl), quad<D>(r.p, g.h)) > thr);
    // sqrt(chi) is a norm where Im M is positive definite: over the ball it is then at
    // least sqrt(chi(centre)) - sqrt(tr P) rad
    if (!positive) return true;
    float tr = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) tr += r.p[sym_index<D>(i, i)];
    return !(sqrtf(fmaxf(chi, 0.0f)) - sqrtf(tr) * g.rad > sqrtf(thr));
}

// Describe the tile's groups (warp w describes group w; sds / shn loaded).
template <int D>
__device__ __forceinline__ void describe_group(const float (*sds)[D], const float (*shn)[D], int s_cnt, bool fast,
                                               bool periodic, TileGroups<D> &tg) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gbase = warp * GS;
    const int cnt = min(GS, s_cnt - gbase);
    if (lane == 0) {
        GroupInfo<D> g;
        float r2 = 0.0f;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            float lo = sds[gbase][i], hi = lo;
            if (!fast)
                for (int k = 1; k < cnt; ++k) lo = fminf(lo, sds[gbase + k][i]), hi = fmaxf(hi, sds[gbase + k][i]);
            g.ds[i] = fast ? lo : 0.5f * (lo + hi);
            g.h[i] = shn[gbase][i];
            const float e = 0.5f * (hi - lo);
            r2 = fmaf(e, e, r2);
        }
        g.rad = sqrtf(r2) * 1.00001f;
        g.kind = cnt <= 0 ? 0 : (fast ? 1 : (periodic ? 3 : 2));
        tg.g[warp] = g;
    }
}

template <int D>
__device__ __forceinline__ void find_lattice(TileGroups<D> &tg) {
    int n = 0;
    while (n < NW && tg.g[n].kind == 1) ++n;
    bool ok = n > 0 && (n == NW || tg.g[n].kind == 0);  // groups without sensors come last
    float hh = 0.0f;
    for (int i = 0; i < D; ++i) hh += fabsf(tg.g[0].h[i]);
    for (int i = 0; i < D; ++i) {
        const float e = n > 1 ? tg.g[1].ds[i] - tg.g[0].ds[i] : 0.0f;
        tg.e[i] = e;
        // a thousandth of a sensor step is far below the test's margin
        for (int g = 0; g < n; ++g)
            ok = ok && fabsf(tg.g[g].h[i] - tg.g[0].h[i]) <= 1e-4f * hh &&
                 fabsf(tg.g[g].ds[i] - fmaf((float)g, e, tg.g[0].ds[i])) <= 1e-3f * hh;
    }
    tg.n = n;
    tg.lattice = ok ? 1 : 0;
    tg.present = 0;
    for (int g = 0; g < NW; ++g) tg.present |= tg.g[g].kind ? 1u << g : 0u;
}

// Mask of the groups of the tile that this lane's record reaches within thr, for any
// Im M: growing beams and records that are not finite among them.  UNROLL: of the loop
// over groups that are no lattice.  Eight copies of the ball test are faster where it
// runs (ring sensor at 256^2, forward: 3.43 ms, two copies 3.50) but slow the
// transpose's instruction fetches where it does not (512^2: 56.1 against 53.4 ms).
template <int D, int UNROLL>
__device__ __forceinline__ unsigned reached_mask(const Rec<D> &r, const TileGroups<D> &tg, float thr) {
    unsigned m = 0;
    if (tg.lattice) {
        // chi on the lattice: chi(g, k) = c0 + Bg g + Ag g^2 + (Bk + C g) k + Ak k^2
        const float *h = tg.g[0].h, *e = tg.e;
        float Dl[D];
#pragma unroll
        for (int i = 0; i < D; ++i) Dl[i] = tg.g[0].ds[i] + r.d0[i];
        const float c0 = quad<D>(r.p, Dl), Bk = bilin2<D>(r.p, h, Dl), Ak = quad<D>(r.p, h);
        const float Bg = bilin2<D>(r.p, e, Dl), Ag = quad<D>(r.p, e), C = bilin2<D>(r.p, h, e);
        // a run's smallest exponent: at the vertex, or (Ak not positive) at the end that
        // the chord of slope B + 15 Ak falls to
        // (finite also for a subnormal Ak: the factor 0 below would make infinity a NaN)
        const float im = Ak > 0.0f ? fmaxf(__fdividef(-0.5f, Ak), -1e18f) : -1e18f;
        const float kn = (float)(GS - 1) * fminf(Ak, 0.0f) * im;
        const float lim = fmaf(2e-6f, fabsf(c0), thr);  // round-off of the expansion
        const int n = tg.n;
#pragma unroll
        for (int g = 0; g < NW; ++g) {
            const float gf = (float)g;
            const float B = fmaf(C, gf, Bk), cg = fmaf(fmaf(Ag, gf, Bg), gf, c0);
            const float kv = fminf(fmaxf(fmaf(B, im, kn), 0.0f), (float)(GS - 1));
            if (!(fmaf(fmaf(Ak, kv, B), kv, cg) > lim) && g < n) m |= 1u << g;
        }
        return m;
    }
    const bool positive = positive_form<D>(r.p);
#pragma unroll UNROLL
    for (int g = 0; g < NW; ++g) {
        const GroupInfo<D> &q = tg.g[g];
        if (q.kind && (q.kind == 3 || group_reached<D>(r, positive, q, thr))) m |= 1u << g;
    }
    return m;
}

// The closed-form beams of a pass, staged per warp (4 beams each).
template <int D, bool TRAJ>
struct HomStage {
    HomBeam<D> b[G];
};
template <int D>
struct HomStage<D, true> {};

template <int D>
__device__ __noinline__ void general_beam_time(const ProbArgs &P, const BeamArgs &B, int64_t b, double t,
                                               BeamTime<D> &bt) {
    beam_time<D>(P, B, b, t, bt);
}

// Write the records of the pass's beams beam_of(0 .. nb) and their masks alive[].
// Bound: latency (dependent FP64 and MUFU chains of one record per warp); a third of
// the homogeneous forward (15.7 of 48.6 ms at 512^2), half of the trajectory sums
// before refine.  What a record needs beyond the test (the anchor phase, the amplitude) is formed
// only when the beam reaches some group at some time.
template <int D, bool PERIODIC, bool TRAJ, int UNROLL, typename BeamOf>
__device__ __forceinline__ void record_pass(const ProbArgs &P, const BeamArgs &B, const TrajSrc<D> &T,
                                            const HomBeam<D> *hom, HomStage<D, TRAJ> &stage, int64_t t_first, int t_cnt,
                                            const TileInfo<D> &ti, const TileGroups<D> &tg, float thr, float *rec,
                                            uint8_t *alive, int nb, const BeamOf &beam_of) {
    constexpr int PW = G / NW;  // beams per warp and pass
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool tv = lane < t_cnt;
    const int mine = warp < nb ? (nb - warp + NW - 1) / NW : 0;  // this warp's beams: warp + k NW, k < mine
    // lane k < PW looks up beam k of the warp
    int64_t b_lane = 0;
    int32_t blk_lane = 0;
    float aabs_lane = 0.0f, aarg_lane = 0.0f;
    if (lane < mine) {
        b_lane = beam_of(warp + lane * NW);
        if constexpr (TRAJ) {
            if (T.pool) blk_lane = T.slot[(t_first / TT) * T.nb + b_lane];
            // the coefficient's amplitude and phase join the record's FP32 |A| and
            // arg A in FP32 (the record already holds them to FP32 precision)
            const int64_t b = T.b_first + b_lane, j = b < B.n ? b : b - B.n;
            const float ar = (float)B.a0[2 * j], ai = (float)B.a0[2 * j + 1];
            aabs_lane = hypotf(ar, ai);
            aarg_lane = atan2f(ai, (ar == 0.0f && ai == 0.0f) ? 1e-12f : ar);
        }
    }
    if constexpr (!TRAJ) {
        if (hom) {
            constexpr int W = sizeof(HomBeam<D>) / 16;
            __syncwarp();
#pragma unroll 1
            for (int q = lane; q < PW * W; q += 32) {
                const int k = q / W;
                const int64_t b = k < mine ? beam_of(warp + k * NW) : -1;
                if (b >= 0)
                    reinterpret_cast<int4 *>(&stage.b[warp * PW + k])[q % W] =
                        __ldg(reinterpret_cast<const int4 *>(&hom[b < B.n ? b : b - B.n]) + q % W);
            }
        } else if (lane < mine) {  // no table in the caller's scratch
            stage.b[warp * PW + lane] = make_hom_beam<D>(P, B, b_lane < B.n ? b_lane : b_lane - B.n);
        }
        __syncwarp();
    }
    const double t = !TRAJ && tv ? P.ts[t_first + lane] : 0.0;
#pragma unroll (TRAJ ? 2 : 1)
    for (int k = 0; k < PW; ++k) {
        if (k >= mine) break;
        const int i = warp + k * NW;
        const int64_t b = __shfl_sync(0xffffffffu, b_lane, k);
        Rec<D> r;
        double dd[D], wpd[D];
        float ang = 0.0f, xk[D];  // xk: the closed form's x_j
#pragma unroll
        for (int a = 0; a < D; ++a) r.d0[a] = 0.0f, wpd[a] = 0.0, dd[a] = 0.0, xk[a] = 0.0f;
#pragma unroll
        for (int q = 0; q < Sym<D>::S; ++q) r.q[q] = r.p[q] = 0.0f;
        r.amp = 0.0f;
        bool closed = false;
        if constexpr (TRAJ) {
            const int32_t blk = __shfl_sync(0xffffffffu, blk_lane, k);
            const float aabs = __shfl_sync(0xffffffffu, aabs_lane, k), aarg = __shfl_sync(0xffffffffu, aarg_lane, k);
            if (tv) {
                const BeamTime<D> bt = T.pool ? T.pool[(int64_t)blk * TT + lane] : T.rec[(t_first + lane) * T.nb + b];
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    dd[a] = ti.s0[a] - bt.x[a];
                    wpd[a] = bt.wp[a];
                }
#pragma unroll
                for (int q = 0; q < Sym<D>::S; ++q) r.q[q] = bt.q[q], r.p[q] = bt.p[q];
                r.amp = bt.amp * aabs;
                ang = bt.ang + aarg;
            }
        } else {
            const HomBeam<D> &h = stage.b[warp * PW + k];
            const double tm = b < B.n ? t : -t;
            if (h.ok) {
                closed = true;
                const float tf = (float)tm;
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    dd[a] = fma(-h.v[a], tm, ti.s0[a] - h.x0[a]);
                    wpd[a] = h.wp[a];
                }
#pragma unroll
                for (int q = 0; q < Sym<D>::S; ++q) r.p[q] = h.U[q];
                float kk = 1.0f;
#pragma unroll
                for (int n = 0; n < D - 1; ++n) {
                    xk[n] = h.td[n] * tf;
                    const float kn = __frcp_rn(fmaf(xk[n], xk[n], 1.0f)), xn = xk[n] * kn;
                    kk *= kn;
#pragma unroll
                    for (int q = 0; q < Sym<D>::S; ++q) {
                        r.p[q] = fmaf(kn, h.N[n][q], r.p[q]);
                        r.q[q] = fmaf(xn, h.N[n][q], r.q[q]);
                    }
                }
                r.amp = kk;  // to the power 1/4 below
                ang = h.aarg;
            } else if (tv) {
                BeamTime<D> bt;
                general_beam_time<D>(P, B, b, t, bt);
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    dd[a] = ti.s0[a] - bt.x[a];
                    wpd[a] = bt.wp[a];
                }
#pragma unroll
                for (int q = 0; q < Sym<D>::S; ++q) r.q[q] = bt.q[q], r.p[q] = bt.p[q];
                r.amp = bt.amp;
                ang = bt.ang;
            }
        }
#pragma unroll
        for (int a = 0; a < D; ++a) {
            if (P.periodic[a]) dd[a] -= P.L[a] * nearbyint(dd[a] / P.L[a]);
            r.d0[a] = (float)dd[a];
            r.wp[a] = (float)wpd[a];
        }
        // (periodic domains: no group is left out)
        const unsigned reach = !tv ? 0u : (!PERIODIC && thr > 0.0f ? reached_mask<D, UNROLL>(r, tg, thr) : tg.present);
        const unsigned m = __reduce_or_sync(0xffffffffu, reach);
        if (m) {
            double lin = 0.0;
#pragma unroll
            for (int a = 0; a < D; ++a) lin = fma(wpd[a], dd[a], lin);
            if (!TRAJ && closed) {
                if constexpr (!TRAJ) r.amp = 2.0f * stage.b[warp * PW + k].aabs * sqrtf(sqrtf(r.amp));
#pragma unroll
                for (int n = 0; n < D - 1; ++n) ang = fmaf(-0.5f, atanf(xk[n]), ang);
            }
            const double th = lin + (double)ang;
            r.th0 = (float)(th - 6.283185307179586 * nearbyint(th * 0.15915494309189535));
            if (!tv) r.amp = 0.0f;
            const float *rf = reinterpret_cast<const float *>(&r);
#pragma unroll
            for (int f = 0; f < Rec<D>::NF; ++f) rec[(f * G + i) * TT + lane] = rf[f];
        }
        if (lane == 0) alive[i] = (uint8_t)m;
    }
}

template <int D>
__device__ __forceinline__ void load_rec(const float *rec, int i, int lane, Rec<D> &r) {
    float *rf = reinterpret_cast<float *>(&r);
#pragma unroll
    for (int f = 0; f < Rec<D>::NF; ++f) rf[f] = rec[(f * G + i) * TT + lane];
}

// Seeds of beams i0 and i1 (i1 < 0: none) as one pair; bit 0 / 1 of the
// result: this lane has to evaluate beam i0 / i1 directly.
template <int D>
__device__ __forceinline__ int seed_pair(const float *rec, int i0, int i1, int lane, const Run<D> &g, bool skip, cf2 &z,
                                         cf2 &f, cf2 &q) {
    cf za, fa, qa, zb{0.0f, 0.0f}, fb{0.0f, 0.0f}, qb{0.0f, 0.0f};
    Rec<D> r;
    load_rec<D>(rec, i0, lane, r);
    int direct = seed_eval<D>(r, g, skip, za, fa, qa) ? 1 : 0;
    if (i1 >= 0) {
        load_rec<D>(rec, i1, lane, r);
        direct |= seed_eval<D>(r, g, skip, zb, fb, qb) ? 2 : 0;
    }
    z = pack2(za, zb);
    f = pack2(fa, fb);
    q = pack2(qa, qb);
    return direct;
}

__device__ __forceinline__ int take_bit(unsigned &bits) {
    const int i = __ffs((int)bits) - 1;  // -1 when none is left
    bits &= bits - 1u;
    return i;
}

// Exclusive offset of this warp's entry (row k of NROW) in the CTA-wide order
// (row, warp), from the per-warp counts cnt[row * NW + warp]; total in tot.
template <int NROW>
__device__ __forceinline__ int scan_counts(const int *cnt, int row, int warp, int &tot) {
    static_assert(NROW * NW <= 32, "one count per lane");
    const int lane = threadIdx.x & 31;
    const int v = lane < NROW * NW ? cnt[lane] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    tot = __shfl_sync(0xffffffffu, x, 31);
    return __shfl_sync(0xffffffffu, x - v, row * NW + warp);
}

// What four of a tile's records say about all of them.  Segment s of a (time tile,
// beam) is its times 8 s .. 8 s + 7, its sample the time segment_sample(s).  With P the
// sample's w/2 Im M, rho the smallest eigenvalue of P^-1 P_t over the segment's times t
// and way the largest distance, in the norm of P, of a centre from the sample's,
//   sqrt(chi_t(y)) >= sqrt(rho) (sqrt(chi(y)) - way)  for every t and sensor y,
// chi being the sample's exponent: a sensor where sqrt(chi) exceeds
// root = sqrt(thr / rho) + way is beyond thr at all of the segment's times.  Byte s of
// limits[tt][b] is that root, rounded up, in steps of sqrt(thr) / kLimitSteps above
// sqrt(thr); 255: none is known (P or some P_t not positive definite or not finite, or
// the beam changes too much), and the beam stays.
constexpr int kLimitSteps = 32;
constexpr int kNoLimit = 255;
__device__ __forceinline__ int segment_sample(int s, int t_cnt) { return min(8 * s + 4, t_cnt - 1); }

// A lower bound on the smallest eigenvalue of P^-1 Q (at most 0 or NaN when none is
// known), for symmetric P (positive definite where the result is positive) and Q.
template <int D>
__device__ __forceinline__ float pencil_min(const double *P, const double *Q) {
    if (D == 1) return P[0] > 0.0 ? 0.99999f * (float)(Q[0] / P[0]) : 0.0f;
    if (D == 2) {
        // the smaller root of x^2 - T x + det Q / det P, T = tr(adj(P) Q) / det P: FP64
        // where thin beams' determinants cancel, then FP32 with the discriminant
        // raised by more than its rounding (all in FP64 took 11 ms for 200,000 beams
        // over 5,667 save times, a third of it in sqrt and divisions)
        const double a = P[0], b = P[1 % Sym<D>::S], d = P[2 % Sym<D>::S];
        const double q = Q[0], r = Q[1 % Sym<D>::S], u = Q[2 % Sym<D>::S];
        const double det = fma(a, d, -b * b);
        if (!(a > 0.0 && det > 0.0)) return 0.0f;
        const double inv = 1.0 / det;
        const float T = (float)((fma(d, q, a * u) - 2.0 * b * r) * inv), N = (float)(fma(q, u, -r * r) * inv);
        const float disc = fmaxf(0.0f, fmaf(T, T, -4.0f * N)) + 1e-6f * T * T;
        return T > 0.0f ? 0.99999f * __fdividef(2.0f * N, T + sqrtf(disc)) : 0.0f;
    }
    // 1 - |L^-1 (Q - P) L^-T|_F with P = L L^T; the norm's square is tr (P^-1 (Q - P))^2
    auto at = [](const double *M, int i, int k) { return M[i <= k ? sym_index<D>(i, k) : sym_index<D>(k, i)]; };
    double adj[D][D], det = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int i1 = (i + 1) % D, i2 = (i + 2) % D, k1 = (k + 1) % D, k2 = (k + 2) % D;
            adj[i][k] = at(P, k1, i1) * at(P, k2, i2) - at(P, k1, i2) * at(P, k2, i1);
        }
#pragma unroll
    for (int k = 0; k < D; ++k) det = fma(at(P, 0, k), adj[k][0], det);
    // leading minors: P00, adj[2][2] = P00 P11 - P01^2, det
    if (!(P[0] > 0.0 && adj[D - 1][D - 1] > 0.0 && det > 0.0)) return 0.0;
    double G[D][D], f = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = 0; k < D; ++k) {
            G[i][k] = 0.0;
#pragma unroll
            for (int l = 0; l < D; ++l) G[i][k] = fma(adj[i][l], at(Q, l, k) - at(P, l, k), G[i][k]);
        }
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = 0; k < D; ++k) f = fma(G[i][k], G[k][i], f);
    return 0.99999f * (1.0f - 1.00001f * (float)(sqrt(fmax(0.0, f)) / det));
}

// A warp takes `per` (at most 32) consecutive (time tile, beam) pairs, then those of
// them that are stored one at a time, lane = time: every record is read once.  32 pairs
// share the index division and the look at the slots; few pairs are spread over the
// GPU instead (2,000 beams over 700 times: 42 us with 32 a warp).
// Bound: HBM, and the instructions of the pencils: 200,000 beams over 5,667 times (a
// third of the tiles stored, 26 GB) 6.4 ms; a pair per warp with FP64 roots 11.0.
// (This and the four samples replace a test of four records alone, which assumed how
// a beam changes between them.  Testing all 32 of each candidate's records in refine
// instead made the summation 247 and 226 ms where it is 185 and 166, no better than
// without refine, 259 and 233.)
template <int D>
__global__ void __launch_bounds__(THREADS) traj_limits_kernel(TrajSrc<D> T, int64_t nt, float thr, int per,
                                                              uint32_t *limits) {
    constexpr int S = Sym<D>::S;
    const int lane = threadIdx.x & 31;
    const int64_t n = (nt + TT - 1) / TT * T.nb, stride = (int64_t)gridDim.x * NW * per;
    for (int64_t i0 = (blockIdx.x * (int64_t)NW + (threadIdx.x >> 5)) * per; i0 < n; i0 += stride) {
        const int64_t mine = min(i0 + lane, n - 1), tt_lane = mine / T.nb;
        const int32_t blk_lane = T.pool ? T.slot[mine] : 0;
        const unsigned live = __ballot_sync(0xffffffffu, lane < per && i0 + lane < n && blk_lane >= 0);
        unsigned word_lane = 0;
        for (unsigned left = live; left;) {
            const int l = take_bit(left);
            const int64_t tt = __shfl_sync(0xffffffffu, tt_lane, l), b = i0 + l - tt * T.nb;
            const int32_t blk = __shfl_sync(0xffffffffu, blk_lane, l);
            const int t_cnt = (int)min((int64_t)TT, nt - tt * TT), t = min(lane, t_cnt - 1);
            const BeamTime<D> *bt = T.pool ? T.pool + ((int64_t)blk * TT + t) : T.rec + ((tt * TT + t) * T.nb + b);
            const int at = segment_sample(lane >> 3, t_cnt);
            float q[S], p[S], dx[D], mag = 0.0f;  // this record's form, the sample's (off-diagonals doubled)
            double Q[S], P[S];
#pragma unroll
            for (int e = 0; e < S; ++e) q[e] = bt->p[e];
#pragma unroll
            for (int e = 0; e < S; ++e) p[e] = __shfl_sync(0xffffffffu, q[e], at);
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int k = a; k < D; ++k) {
                    const int e = sym_index<D>(a, k);
                    Q[e] = (a == k ? 1.0 : 0.5) * (double)q[e];
                    P[e] = (a == k ? 1.0 : 0.5) * (double)p[e];
                }
#pragma unroll
            for (int a = 0; a < D; ++a) {
                const double x = bt->x[a];
                dx[a] = (float)(x - __shfl_sync(0xffffffffu, x, at));
            }
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int k = a; k < D; ++k) mag = fmaf(fabsf(p[sym_index<D>(a, k)]), fabsf(dx[a] * dx[k]), mag);
            // (the quadratic form's rounding is below 1e-6 of its terms' magnitudes)
            float rho = pencil_min<D>(P, Q);
            const float way = quad<D>(p, dx) + 1e-6f * mag;
            float w = sqrtf(fmaxf(way, 0.0f)) * 1.00001f;
            // a value that is not a number is not a limit
            bool known = rho > 0.0f && way < 1e30f;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                rho = fminf(rho, __shfl_xor_sync(0xffffffffu, rho, o));
                w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
                known = __shfl_xor_sync(0xffffffffu, (int)known, o) != 0 && known;
            }
            const float c = ceilf((rsqrtf(rho) * 1.00001f + w * rsqrtf(thr) * 1.00001f - 1.0f) * (float)kLimitSteps);
            const unsigned code = known && c < (float)kNoLimit ? (unsigned)fmaxf(c, 0.0f) : (unsigned)kNoLimit;
            unsigned word = code << (8 * (lane >> 3));
            word |= __shfl_xor_sync(0xffffffffu, word, 8);
            word |= __shfl_xor_sync(0xffffffffu, word, 16);
            if (lane == l) word_lane = word;
        }
        if (live >> lane & 1u) limits[mine] = word_lane;
    }
}

// Trajectory candidates surv[old .. nq) (kept by the tile test) against the groups
// of the tile, from 4 of their tile's 32 times and their limits: the tile test's
// isotropic bound keeps 2 to 3 candidates for each that reaches the tile (live: 34 % at
// 1024^2 heterogeneous, 40 % at 128^3), and fetching a dead one's whole record (2 KB in
// 2D) cost more than half of the summation.  A candidate goes if no group is within
// its limit of any of the four samples: the record pass would leave it out at every
// group.  Four lanes per candidate; the survivors move to surv[old ..) in order.
// Returns the new end.  All threads; ends with a barrier.
template <int D, typename BeamOf>
__device__ __forceinline__ int refine(const TrajSrc<D> &T, int64_t t_first, int t_cnt, const TileInfo<D> &ti,
                                      const TileGroups<D> &tg, float thr, int32_t *surv, int old, int nq, uint8_t *keep,
                                      int *warp_cnt, const BeamOf &beam_of) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, smp = lane & 3;
    const int64_t tt = t_first / TT;
    const int ts = segment_sample(smp, t_cnt);
    int out = old;
    for (int base = old; base < nq; base += SCAN * THREADS) {
        const int end = min(nq, base + SCAN * THREADS);
#pragma unroll 2
        for (int c0 = base + warp * 8; c0 < end; c0 += NW * 8) {
            const int c = min(c0 + lane / 4, end - 1);
            const int64_t b = beam_of(c);
            const BeamTime<D> *bt =
                T.pool ? T.pool + ((int64_t)T.slot[tt * T.nb + b] * TT + ts) : T.rec + ((t_first + ts) * T.nb + b);
            const int code = T.limits[tt * T.nb + b] >> (8 * smp) & 255u;
            Rec<D> r;
#pragma unroll
            for (int a = 0; a < D; ++a) r.d0[a] = (float)(ti.s0[a] - bt->x[a]);
#pragma unroll
            for (int q = 0; q < Sym<D>::S; ++q) r.p[q] = bt->p[q];
            const float up = fmaf((float)code, 1.0f / kLimitSteps, 1.0f);
            const unsigned hit =
                __ballot_sync(0xffffffffu, code == kNoLimit || reached_mask<D, 2>(r, tg, thr * up * up) != 0);
            if (smp == 0 && c0 + lane / 4 < end) keep[c0 + lane / 4 - base] = (hit >> lane & 15u) ? 1 : 0;
        }
        __syncthreads();
        int32_t v[SCAN];
        unsigned bk[SCAN];
#pragma unroll
        for (int k = 0; k < SCAN; ++k) {
            const int i = base + k * THREADS + tid;
            v[k] = i < end ? surv[i] : 0;
            bk[k] = __ballot_sync(0xffffffffu, i < end && keep[i - base]);
            if (lane == 0) warp_cnt[k * NW + warp] = __popc(bk[k]);
        }
        __syncthreads();
        int tot = 0;
#pragma unroll
        for (int k = 0; k < SCAN; ++k) {
            const int off = out + scan_counts<SCAN>(warp_cnt, k, warp, tot);
            if (bk[k] >> lane & 1u) surv[off + __popc(bk[k] & ((1u << lane) - 1u))] = v[k];
        }
        out += tot;
        __syncthreads();
    }
    return out;
}

// ------------------------------------------------------------------ forward
__device__ __forceinline__ void kahan_add(float &acc, float &cmp, float v) {
    const float y = v - cmp;
    const float t = acc + y;
    cmp = (t - acc) - y;
    acc = t;
}

// A tile's beams in n ranges of len, each its own work item with a partial
// (compensated sum, compensation) per output, added in order by
// combine_parts_kernel.  n = 1: the item writes the output itself.  part = nullptr (a
// workspace without room for the partials) and n > 1: an item takes all of its tile's
// ranges, one after the other, and adds them in the same order in shared memory, so
// that the result is the same bits whatever the workspace.
struct Split {
    int n;
    int64_t len;
    float2 *part;  // (n, ns, nt)
    __host__ __device__ bool serial() const { return n > 1 && !part; }
    __host__ __device__ int items_per_tile() const { return part ? n : 1; }
};
// Shared memory of the ranges' totals in that case: (sensor, time) of the tile.
constexpr size_t kTotalBytes = sizeof(float2) * TS * TT;

// Work items a launch should have: 8 per resident CTA (2 per SM of the 148), so that
// the last, unevenly filled wave is a small part of it (a constant, not the device's
// own count: the order of the sums follows from it).  Fewer tiles than that are
// split over the beams, in ranges of at least kSplitMin (8 passes of both modes):
// 4,096 coefficients at 128^2 ran 19 blocks for 3.9 ms, now 0.24 ms; a 512-point
// sensor at 512^2 304 blocks in two waves for 31.0 ms, 18.9 ms without the split
// after the other steps, 10.5 with it.
constexpr int64_t kItemsWanted = 8 * 2 * 148;
constexpr int64_t kSplitMin = 128;

// out (or the chunk state) = sum over the ranges, in order, and over earlier
// chunks; one 32 x 32 block of (sorted sensor, time) per CTA.
__device__ __forceinline__ void add_part(float &a, float &c, float2 v) {
    kahan_add(a, c, v.x);
    kahan_add(a, c, -v.y);
}

__global__ void combine_parts_kernel(const float2 *part, int n, const int32_t *perm, int64_t nt, int64_t ns, float *state,
                                     int first, int last, float *out) {
    __shared__ float2 tile[32][33];
    const int64_t s0 = (int64_t)blockIdx.x * 32, t0 = (int64_t)blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t s = s0 + k, t = t0 + threadIdx.x;
        float a = 0.0f, c = 0.0f;
        if (s < ns && t < nt) {
            for (int q = 0; q < n; ++q) add_part(a, c, part[((int64_t)q * ns + s) * nt + t]);
        }
        tile[k][threadIdx.x] = make_float2(a, c);
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t s = s0 + threadIdx.x, t = t0 + k;
        if (s >= ns || t >= nt) continue;
        float2 v = tile[threadIdx.x][k];
        if (!first) add_part(v.x, v.y, make_float2(state[t * ns + s], state[(nt + t) * ns + s]));
        if (last) {
            out[t * ns + perm[s]] = v.x - v.y;
        } else {
            state[t * ns + s] = v.x;
            state[(nt + t) * ns + s] = v.y;
        }
    }
}

// Persistent CTAs take (time tile, sensor tile, beam range) work items from a
// counter.  Warp w owns sensor group w (GS sensors) of the tile; lane l owns time l.
// Per item: beams are scanned 1024 at a time against the tile (survives /
// traj_survives), survivors queue up, and every G of them make a record pass;
// then each warp evaluates the pass's beams that reach its group, four at a
// time (two independent paired recurrences; two values of a sensor are added
// before each compensated addition).
//
// Bound: FP32 pipe (recurrence 8 FMA-pipe operations per triple, seed ~75 per 16
// triples) with the seeds' MUFU work beside it; measured 55 % (512^2), 51 % (1024^2
// heterogeneous) and 59 % (128^3) of that pipe's cycles, the rest in pass barriers and latency.  512^2
// homogeneous (65,536 coefficients, 2,414 times, 2,044 sensors): 78.3 ms when every
// group evaluated every survivor of the tile, 46.7 now (45.5 with four beams' values
// added before each compensated addition instead of two); 1024^2 heterogeneous,
// 200,000 beams: 538 -> 168 ms; 128^3: 300 -> 116 ms.
template <int D, bool PERIODIC, bool TRAJ>
__global__ void __launch_bounds__(THREADS, 2)
fwd32_kernel(ProbArgs P, BeamArgs B, const Cull<D> *cull, const HomBeam<D> *hom, const TileInfo<D> *tiles, const int32_t *offs,
             const float *ds_g, const float *hn_g, const uint8_t *gfast_g, const int32_t *perm, float cutoff,
             float *out, unsigned long long *eval_count, int *work, int n_st, int n_items, Split sp, TrajSrc<D> T) {
    extern __shared__ __align__(16) float rec[];  // rec_bytes<D>(), then (sp.serial()) the ranges' totals
    __shared__ float sds[TS][D], shn[TS][D];
    __shared__ TileGroups<D> ginfo;
    __shared__ HomStage<D, TRAJ> hstage;
    __shared__ int32_t surv[2 * SCAN * THREADS + G];
    __shared__ int warp_cnt[SCAN * NW];
    __shared__ uint8_t alive[G], keep[TRAJ ? SCAN * THREADS : 1];
    __shared__ int tile_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float thr = cutoff > 0.0f ? cutoff + kGroupMarginEfolds : 0.0f;
    const bool skip = cutoff > 0.0f;
    unsigned long long evals = 0;
    while (true) {
        if (tid == 0) tile_s = atomicAdd(work, 1);
        __syncthreads();
        const int item = tile_s;
        if (item >= n_items) break;
        const int per_tile = sp.items_per_tile(), tile = item / per_tile;
        const int64_t st = tile % n_st, tt = tile / n_st;
        const int64_t s_first = offs[st], t_first = tt * TT;
        const int s_cnt = offs[st + 1] - offs[st];
        const int t_cnt = (int)min((int64_t)TT, P.nt - t_first);
        const TileInfo<D> ti = tiles[st];
        const float ta = (float)P.ts[t_first], tb = (float)P.ts[t_first + t_cnt - 1];
        for (int k = tid; k < TS; k += THREADS) {
#pragma unroll
            for (int i = 0; i < D; ++i) {
                sds[k][i] = k < s_cnt ? ds_g[(s_first + k) * D + i] : 0.0f;
                shn[k][i] = k < s_cnt ? hn_g[(s_first + k) * D + i] : 0.0f;
            }
        }
        __syncthreads();
        const bool fast = gfast_g[st * NW + warp] != 0;
        const int gbase = warp * GS;
        const bool active = gbase < s_cnt;
        describe_group<D>(sds, shn, s_cnt, fast, PERIODIC, ginfo);
        __syncthreads();
        if (tid == 0) find_lattice<D>(ginfo);
        Run<D> run;
#pragma unroll
        for (int i = 0; i < D; ++i) run.ds[i] = sds[gbase][i], run.h[i] = shn[gbase][i];
        const int g_cnt = max(0, min(GS, s_cnt - gbase));
        // one range, or with sp.serial() all of the tile's in order
        for (int part = item % per_tile, end = sp.serial() ? sp.n : part + 1; part < end; ++part) {
            // Kahan sums of sensors 2h and 2h + 1 in .x and .y
            float2 acc2[GS / 2], cmp2[GS / 2];
#pragma unroll
            for (int h = 0; h < GS / 2; ++h) acc2[h] = make_float2(0.0f, 0.0f), cmp2[h] = make_float2(0.0f, 0.0f);
            if (TRAJ && sp.n == 1 && !T.first && lane < t_cnt && active) {
                const int64_t t = t_first + lane;
#pragma unroll
                for (int k = 0; k < GS; ++k) {
                    const int s = gbase + k;
                    if (s < s_cnt) {
                        const float a = T.state[t * P.ns + s_first + s];
                        const float c = T.state[(P.nt + t) * P.ns + s_first + s];
                        if (k & 1)
                            acc2[k / 2].y = a, cmp2[k / 2].y = c;
                        else
                            acc2[k / 2].x = a, cmp2[k / 2].x = c;
                    }
                }
            }
            const int64_t jb = part * sp.len;
            const int64_t nbeam = min(jb + sp.len, TRAJ ? T.nb : B.n);
            int nq = 0;  // queued survivors (the same in every thread)

            for (int64_t j0 = jb; j0 < nbeam; j0 += SCAN * THREADS) {
                unsigned bp[SCAN], bm[SCAN];
#pragma unroll
                for (int k = 0; k < SCAN; ++k) {
                    const int64_t j = j0 + k * THREADS + tid;
                    bool keep_p = false, keep_m = false;
                    if (j < nbeam) {
                        if (TRAJ) {
                            keep_p = traj_survives<D>(T, j, tt, ti, cutoff);
                        } else {
                            const Cull<D> cb = cull[j];
                            keep_p = mode_on(B.modes, 0) && survives<D>(cb, (float)P.c, ta, tb, ti, P, cutoff);
                            keep_m = mode_on(B.modes, 1) && survives<D>(cb, -(float)P.c, ta, tb, ti, P, cutoff);
                        }
                    }
                    bp[k] = __ballot_sync(0xffffffffu, keep_p);
                    bm[k] = TRAJ ? 0u : __ballot_sync(0xffffffffu, keep_m);
                    if (lane == 0) warp_cnt[k * NW + warp] = __popc(bp[k]) + __popc(bm[k]);
                }
                __syncthreads();
                int tot = 0;
                const unsigned lt = (1u << lane) - 1u;
#pragma unroll
                for (int k = 0; k < SCAN; ++k) {
                    const int off = nq + scan_counts<SCAN>(warp_cnt, k, warp, tot);
                    const int32_t j = (int32_t)(j0 + k * THREADS + tid);
                    if (bp[k] >> lane & 1u) surv[off + __popc(bp[k] & lt)] = j;
                    if (!TRAJ && (bm[k] >> lane & 1u)) surv[off + __popc(bp[k]) + __popc(bm[k] & lt)] = (int32_t)(j + B.n);
                }
                const int old = nq;
                nq += tot;
                __syncthreads();
                if constexpr (TRAJ && !PERIODIC) {
                    if (T.limits)
                        nq = refine<D>(T, t_first, t_cnt, ti, ginfo, thr, surv, old, nq, keep, warp_cnt,
                                       [&](int c) { return (int64_t)surv[c]; });
                }
                const bool last_scan = j0 + SCAN * THREADS >= nbeam;
                int g0 = 0;
                while (nq - g0 >= G || (last_scan && g0 < nq)) {
                    const int nb = min(G, nq - g0);
                    record_pass<D, PERIODIC, TRAJ, 8>(P, B, T, hom, hstage, t_first, t_cnt, ti, ginfo, thr, rec, alive, nb,
                                         [&](int i) { return (int64_t)surv[g0 + i]; });
                    __syncthreads();
                    unsigned bits = __ballot_sync(0xffffffffu, active && lane < nb && (alive[lane] >> warp & 1));
                    evals += (unsigned long long)__popc(bits) * (unsigned)(t_cnt * g_cnt);
                    while (bits) {
                        if (fast) {
                            const int i0 = take_bit(bits), i1 = take_bit(bits), i2 = take_bit(bits), i3 = take_bit(bits);
                            cf2 za, fa, qa, zb, fb, qb;
                            int direct = seed_pair<D>(rec, i0, i1, lane, run, skip, za, fa, qa);
                            zb = fb = qb = cf2{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                            if (i2 >= 0) direct |= seed_pair<D>(rec, i2, i3, lane, run, skip, zb, fb, qb) << 2;
                            {
                                // z_{k+1} = z_k f_k, f_{k+1} = f_k q; sensors 2h, 2h + 1
                                // share a paired compensated addition per two beams (one or
                                // two beams left: the other pair is zero -- a second loop for
                                // them costs more in instruction fetches than it saves)
#pragma unroll
                                for (int h = 0; h < GS / 2; ++h) {
                                    if (h > 0) {
                                        za = cmul2(za, fa);
                                        zb = cmul2(zb, fb);
                                        fa = cmul2(fa, qa);
                                        fb = cmul2(fb, qb);
                                    }
                                    const float2 a0 = za.re, b0 = zb.re;
                                    za = cmul2(za, fa);
                                    zb = cmul2(zb, fb);
                                    fa = cmul2(fa, qa);
                                    fb = cmul2(fb, qb);
                                    kahan_add2(acc2[h], cmp2[h], make_float2(a0.x + a0.y, za.re.x + za.re.y));
                                    if (i2 >= 0) kahan_add2(acc2[h], cmp2[h], make_float2(b0.x + b0.y, zb.re.x + zb.re.y));
                                }
                            }
                            if (!__any_sync(0xffffffffu, direct != 0)) continue;
                            // rare: recurrences out of FP32's range
#pragma unroll 1
                            for (int e = 0; e < 4; ++e) {
                                if (!__any_sync(0xffffffffu, direct >> e & 1)) continue;
                                Rec<D> r;
                                load_rec<D>(rec, e == 0 ? i0 : (e == 1 ? i1 : (e == 2 ? i2 : i3)), lane, r);
                                float v[GS];
#pragma unroll 1
                                for (int k = 0; k < GS; ++k)
                                    v[k] = (direct >> e & 1) ? direct_eval<D, false>(r, sds[gbase + k], P).re : 0.0f;
#pragma unroll
                                for (int h = 0; h < GS / 2; ++h)
                                    kahan_add2(acc2[h], cmp2[h], make_float2(v[2 * h], v[2 * h + 1]));
                            }
                        } else {
                            // broken runs (sensors off the grid, periodic domains): every
                            // sensor directly, values staged in a small array (one copy
                            // of the evaluation in the instruction cache)
                            const int i0 = take_bit(bits), i1 = take_bit(bits);
                            Rec<D> ra, rb;
                            load_rec<D>(rec, i0, lane, ra);
                            load_rec<D>(rec, i1 >= 0 ? i1 : i0, lane, rb);
                            if (i1 < 0) rb.amp = 0.0f;
                            float v[GS];
#pragma unroll 1
                            for (int k = 0; k < GS; ++k)
                                v[k] = direct_eval<D, PERIODIC>(ra, sds[gbase + k], P).re +
                                       direct_eval<D, PERIODIC>(rb, sds[gbase + k], P).re;
#pragma unroll
                            for (int h = 0; h < GS / 2; ++h)
                                kahan_add2(acc2[h], cmp2[h], make_float2(v[2 * h], v[2 * h + 1]));
                        }
                    }
                    g0 += nb;
                    __syncthreads();
                }
                if (g0 > 0 && g0 < nq) {  // fewer than G survivors wait for the next scan
                    const int32_t left = tid < nq - g0 ? surv[g0 + tid] : 0;
                    __syncthreads();
                    if (tid < nq - g0) surv[tid] = left;
                }
                nq -= g0;
            }
            if (lane < t_cnt && active) {
                const int64_t t = t_first + lane;
#pragma unroll
                for (int k = 0; k < GS; ++k) {
                    const int s = gbase + k;
                    if (s < s_cnt) {
                        const float a = (k & 1) ? acc2[k / 2].y : acc2[k / 2].x;
                        const float c = (k & 1) ? cmp2[k / 2].y : cmp2[k / 2].x;
                        if (sp.part) {
                            sp.part[((int64_t)part * P.ns + s_first + s) * P.nt + t] = make_float2(a, c);
                        } else if (sp.n > 1) {
                            // this thread's own entries
                            float2 &tot = reinterpret_cast<float2 *>(rec + rec_bytes<D>() / sizeof(float))[s * TT + lane];
                            float sa = part ? tot.x : 0.0f, sc = part ? tot.y : 0.0f;
                            add_part(sa, sc, make_float2(a, c));
                            tot = make_float2(sa, sc);
                            if (part < sp.n - 1) continue;
                            const int64_t at = t * P.ns + s_first + s;
                            if (TRAJ && !T.first) add_part(sa, sc, make_float2(T.state[at], T.state[P.nt * P.ns + at]));
                            if (TRAJ && !T.last) {
                                T.state[at] = sa;
                                T.state[P.nt * P.ns + at] = sc;
                            } else {
                                out[t * P.ns + perm[s_first + s]] = sa - sc;
                            }
                        } else if (TRAJ && !T.last) {
                            T.state[t * P.ns + s_first + s] = a;
                            T.state[(P.nt + t) * P.ns + s_first + s] = c;
                        } else {
                            out[t * P.ns + perm[s_first + s]] = a - c;
                        }
                    }
                }
            }
            __syncthreads();
        }
    }
    if (eval_count && lane == 0 && evals) atomicAdd(eval_count, evals);
}

// ------------------------------------------------------------------ adjoint
// Deterministic tile-parallel transpose (no floating-point atomics).
//
// Work item = (time tile tt, range of RJ consecutive beam indices j; fewer per
// range when the launch would have too few items, kItemsWanted): for the
// homogeneous entry point j is a selected coefficient and both of its modes
// are summed; for trajectories j is a beam of the chunk.  Items run tt-major,
// so consecutive items read the same time tile of the data.  For each sensor
// tile in order, the CTA tests the range's beams for survival, loads the tile's
// data (registers: warp w holds sensor group w, lane l time l) and makes
// record passes as the forward does; each warp runs the forward's recurrence
// for the beams that reach its group while the lane accumulates
// sum_s d(t, s) conj(z(t, s)).  The partials are reduced over the 32 times
// (FP32 shuffles) and over the 8 warps (FP64), in fixed orders, into the range's
// per-beam FP64 accumulators in shared memory (one owner thread per value and
// pass).  The item then writes every accumulator (zeros included) to
// part[tt][slot], and reduce_parts_kernel sums part over the time tiles in
// order.  Bound: as the forward, with more time at the pass barriers (FMA pipe
// 44-49 %).  512^2: 86.4 -> 54.2 ms; 1024^2 heterogeneous 576 -> 185 ms; 128^3 504 ->
// 147 ms.  Each partial has one writer and every sum has a fixed order, so the
// result is bit-identical between runs; the work counter only hands out items.
template <int D, bool TRAJ>
struct AdjRange {
    // accumulator slots (re, im FP64) per item; 3D's larger records leave room
    // for half as many when two CTAs share an SM
    static constexpr int NACC = D == 3 ? 1024 : 2048;
    static constexpr int RJ = TRAJ ? NACC : NACC / 2;  // most beam indices per item
};

template <int D, bool PERIODIC, bool TRAJ>
__global__ void __launch_bounds__(THREADS, 2)
adj32_kernel(ProbArgs P, BeamArgs B, const Cull<D> *cull, const HomBeam<D> *hom, const TileInfo<D> *tiles, const int32_t *offs,
             const float *ds_g, const float *hn_g, const uint8_t *gfast_g, const float *dataT, float cutoff,
             double *part, unsigned long long *eval_count, int *work, int n_st, int RJ, int n_ranges, int n_items,
             TrajSrc<D> T) {
    constexpr int NACC = AdjRange<D, TRAJ>::NACC;
    extern __shared__ double acc_smem[];  // (NACC, 2), then the records
    float *rec = reinterpret_cast<float *>(acc_smem + 2 * NACC);
    __shared__ float sds[TS][D], shn[TS][D];
    __shared__ TileGroups<D> ginfo;
    __shared__ HomStage<D, TRAJ> hstage;
    __shared__ int32_t surv[NACC];  // a range's survivors in one tile (local slots)
    __shared__ int warp_cnt[SCAN * NW];
    __shared__ uint8_t keep[TRAJ ? SCAN * THREADS : 1];
    __shared__ float wpart[NW][G][2];
    __shared__ uint8_t alive2[2][G];
    __shared__ int item_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t nbeam = TRAJ ? T.nb : B.n;
    const int64_t nslots = TRAJ ? T.nb : 2 * B.n;
    const float thr = cutoff > 0.0f ? cutoff + kGroupMarginEfolds : 0.0f;
    const bool skip = cutoff > 0.0f;
    unsigned long long evals = 0;
    int flip = 0;
    for (int q = tid; q < 2 * NACC; q += THREADS) acc_smem[q] = 0.0;
    while (true) {
        if (tid == 0) item_s = atomicAdd(work, 1);
        __syncthreads();
        const int item = item_s;
        if (item >= n_items) break;
        const int64_t tt = item / n_ranges, r0 = (int64_t)(item % n_ranges) * RJ;
        const int64_t r1 = min(r0 + RJ, nbeam);
        const int64_t t_first = tt * TT;
        const int t_cnt = (int)min((int64_t)TT, P.nt - t_first);
        const float ta = (float)P.ts[t_first], tb = (float)P.ts[t_first + t_cnt - 1];
        const bool tv = lane < t_cnt;
        for (int st = 0; st < n_st; ++st) {
            const int64_t s_first = offs[st];
            const int s_cnt = offs[st + 1] - offs[st];
            if (s_cnt <= 0) continue;
            const TileInfo<D> ti = tiles[st];
            // survivors of the range: local slot j - r0 (mode +1 / trajectories), RJ + j - r0 (mode -1)
            int nq = 0;
            for (int64_t j0 = r0; j0 < r1; j0 += THREADS) {
                const int64_t j = j0 + tid;
                bool keep_p = false, keep_m = false;
                if (j < r1) {
                    if (TRAJ) {
                        keep_p = traj_survives<D>(T, j, tt, ti, cutoff);
                    } else {
                        const Cull<D> cb = cull[j];
                        keep_p = mode_on(B.modes, 0) && survives<D>(cb, (float)P.c, ta, tb, ti, P, cutoff);
                        keep_m = mode_on(B.modes, 1) && survives<D>(cb, -(float)P.c, ta, tb, ti, P, cutoff);
                    }
                }
                const unsigned bp = __ballot_sync(0xffffffffu, keep_p);
                const unsigned bm = TRAJ ? 0u : __ballot_sync(0xffffffffu, keep_m);
                __syncthreads();  // warp_cnt and (first trip) the previous tile's surv are done with
                if (lane == 0) warp_cnt[warp] = __popc(bp) + __popc(bm);
                __syncthreads();
                int tot;
                const int off = nq + scan_counts<1>(warp_cnt, 0, warp, tot);
                const unsigned lt = (1u << lane) - 1u;
                if (keep_p) surv[off + __popc(bp & lt)] = (int32_t)(j - r0);
                if (keep_m) surv[off + __popc(bp) + __popc(bm & lt)] = (int32_t)(RJ + j - r0);
                nq += tot;
            }
            if (nq == 0) continue;
            for (int k = tid; k < TS; k += THREADS) {
#pragma unroll
                for (int i = 0; i < D; ++i) {
                    sds[k][i] = k < s_cnt ? ds_g[(s_first + k) * D + i] : 0.0f;
                    shn[k][i] = k < s_cnt ? hn_g[(s_first + k) * D + i] : 0.0f;
                }
            }
            __syncthreads();
            const bool fast = gfast_g[st * NW + warp] != 0;
            const int gbase = warp * GS;
            const bool active = gbase < s_cnt;
            const int g_cnt = max(0, min(GS, s_cnt - gbase));
            describe_group<D>(sds, shn, s_cnt, fast, PERIODIC, ginfo);
            Run<D> run;
#pragma unroll
            for (int i = 0; i < D; ++i) run.ds[i] = sds[gbase][i], run.h[i] = shn[gbase][i];
            const float *dcol = dataT + (int64_t)s_first * P.nt + t_first + lane;
            __syncthreads();
            if (tid == 0) find_lattice<D>(ginfo);
            __syncthreads();  // ginfo, surv
            if constexpr (TRAJ && !PERIODIC) {
                if (T.limits) {
                    nq = refine<D>(T, t_first, t_cnt, ti, ginfo, thr, surv, 0, nq, keep, warp_cnt,
                                   [&](int c) { return r0 + surv[c]; });
                    if (nq == 0) continue;
                }
            }
            float dv[GS];
#pragma unroll
            for (int k = 0; k < GS; ++k)
                dv[k] = (tv && gbase + k < s_cnt) ? __ldg(dcol + (int64_t)(gbase + k) * P.nt) : 0.0f;

            for (int g0 = 0; g0 < nq; g0 += G) {
                const int nb = min(G, nq - g0);
                uint8_t *alive = alive2[flip];
                flip ^= 1;
                record_pass<D, PERIODIC, TRAJ, 2>(P, B, T, hom, hstage, t_first, t_cnt, ti, ginfo, thr, rec, alive, nb, [&](int i) {
                    const int q = surv[g0 + i];
                    return TRAJ || q < RJ ? r0 + q : B.n + r0 + q - RJ;
                });
                __syncthreads();
                unsigned bits = __ballot_sync(0xffffffffu, active && lane < nb && (alive[lane] >> warp & 1));
                evals += (unsigned long long)__popc(bits) * (unsigned)(t_cnt * g_cnt);
                while (bits) {
                    const int i0 = take_bit(bits), i1 = take_bit(bits);
                    float2 ar = make_float2(0.0f, 0.0f), ai = ar, br = ar, bi = ar;
                    int i2 = -1, i3 = -1;
                    if (fast) {
                        i2 = take_bit(bits);
                        i3 = take_bit(bits);
                        cf2 za, fa, qa, zb, fb, qb;
                        int direct = seed_pair<D>(rec, i0, i1, lane, run, skip, za, fa, qa);
                        zb = fb = qb = cf2{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                        if (i2 >= 0) direct |= seed_pair<D>(rec, i2, i3, lane, run, skip, zb, fb, qb) << 2;
                        {
#pragma unroll
                            for (int k = 0; k < GS; ++k) {
                                if (k > 0) {
                                    za = cmul2(za, fa);
                                    zb = cmul2(zb, fb);
                                    fa = cmul2(fa, qa);
                                    fb = cmul2(fb, qb);
                                }
                                const float2 dk = make_float2(dv[k], dv[k]);
                                ar = __ffma2_rn(dk, za.re, ar);
                                ai = __ffma2_rn(neg2(dk), za.im, ai);
                                br = __ffma2_rn(dk, zb.re, br);
                                bi = __ffma2_rn(neg2(dk), zb.im, bi);
                            }
                        }
                        if (__any_sync(0xffffffffu, direct != 0)) {
                            // rare: recurrences out of FP32's range
#pragma unroll 1
                            for (int e = 0; e < 4; ++e) {
                                if (!(direct >> e & 1)) continue;
                                Rec<D> r;
                                load_rec<D>(rec, e == 0 ? i0 : (e == 1 ? i1 : (e == 2 ? i2 : i3)), lane, r);
                                float sr = 0.0f, si = 0.0f;
#pragma unroll 1
                                for (int k = 0; k < GS; ++k) {
                                    const float d = tv ? __ldg(dcol + (int64_t)(gbase + k) * P.nt) : 0.0f;
                                    const cf z = direct_eval<D, false>(r, sds[gbase + k], P);
                                    sr = fmaf(d, z.re, sr);
                                    si = fmaf(-d, z.im, si);
                                }
                                if (e == 0) ar.x = sr, ai.x = si;
                                if (e == 1) ar.y = sr, ai.y = si;
                                if (e == 2) br.x = sr, bi.x = si;
                                if (e == 3) br.y = sr, bi.y = si;
                            }
                        }
                    } else {
                        Rec<D> ra, rb;
                        load_rec<D>(rec, i0, lane, ra);
                        load_rec<D>(rec, i1 >= 0 ? i1 : i0, lane, rb);
#pragma unroll 1
                        for (int k = 0; k < g_cnt; ++k) {
                            const float d = tv ? __ldg(dcol + (int64_t)(gbase + k) * P.nt) : 0.0f;
                            const cf z0 = direct_eval<D, PERIODIC>(ra, sds[gbase + k], P);
                            const cf z1 = direct_eval<D, PERIODIC>(rb, sds[gbase + k], P);
                            ar.x = fmaf(d, z0.re, ar.x);
                            ai.x = fmaf(-d, z0.im, ai.x);
                            ar.y = fmaf(d, z1.re, ar.y);
                            ai.y = fmaf(-d, z1.im, ai.y);
                        }
                    }
                    // over the 32 times (the partials are sums of 16 terms): a
                    // reduce-scatter of the eight partials (re, im of four beams), 9
                    // shuffles.  Lane 4 v ends with value v; FP64 from here on.
                    {
                        const bool u4 = (lane & 16) != 0, u3 = (lane & 8) != 0, u2 = (lane & 4) != 0;
                        float k0 = u4 ? br.x : ar.x, k1 = u4 ? bi.x : ai.x, k2 = u4 ? br.y : ar.y, k3 = u4 ? bi.y : ai.y;
                        k0 += __shfl_xor_sync(0xffffffffu, u4 ? ar.x : br.x, 16);
                        k1 += __shfl_xor_sync(0xffffffffu, u4 ? ai.x : bi.x, 16);
                        k2 += __shfl_xor_sync(0xffffffffu, u4 ? ar.y : br.y, 16);
                        k3 += __shfl_xor_sync(0xffffffffu, u4 ? ai.y : bi.y, 16);
                        float m0 = u3 ? k2 : k0, m1 = u3 ? k3 : k1;
                        m0 += __shfl_xor_sync(0xffffffffu, u3 ? k0 : k2, 8);
                        m1 += __shfl_xor_sync(0xffffffffu, u3 ? k1 : k3, 8);
                        float v = u2 ? m1 : m0;
                        v += __shfl_xor_sync(0xffffffffu, u2 ? m0 : m1, 4);
                        v += __shfl_xor_sync(0xffffffffu, v, 2);
                        v += __shfl_xor_sync(0xffffffffu, v, 1);
                        const int i = u4 ? (u3 ? i3 : i2) : (u3 ? i1 : i0);
                        if ((lane & 3) == 0 && i >= 0) wpart[warp][i][u2 ? 1 : 0] = v;
                    }
                }
                __syncthreads();
                if (tid < 2 * nb) {
                    const int i = tid >> 1, c = tid & 1;
                    const unsigned m = alive[i];
                    double sum = 0.0;
#pragma unroll
                    for (int w = 0; w < NW; ++w)
                        if (m >> w & 1u) sum += (double)wpart[w][i][c];
                    acc_smem[2 * surv[g0 + i] + c] += sum;  // slots are distinct within a pass
                }
            }
        }
        __syncthreads();
        // every slot of the item, zeros included, then clear for the next item
        for (int q = tid; q < (TRAJ ? RJ : 2 * RJ); q += THREADS) {
            const int64_t jl = TRAJ ? q : (q < RJ ? q : q - RJ);
            const int64_t j = r0 + jl;
            if (j < r1) {
                const int64_t slot = TRAJ ? j : (q < RJ ? j : B.n + j);
                double *dst = part + 2 * (tt * nslots + slot);
                dst[0] = acc_smem[2 * q];
                dst[1] = acc_smem[2 * q + 1];
            }
            acc_smem[2 * q] = 0.0;
            acc_smem[2 * q + 1] = 0.0;
        }
    }
    if (eval_count && lane == 0 && evals) atomicAdd(eval_count, evals);
}

// g[j] = sum over time tiles, in order, of part[tt][j] (trajectories) or of
// part[tt][j] + part[tt][n + j] (both modes of coefficient j).
__global__ void reduce_parts_kernel(const double *part, int64_t n_tt, int64_t nslots, int64_t n_out, int both_modes,
                                    double *g) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n_out) return;
    double re = 0.0, im = 0.0;
    for (int64_t tt = 0; tt < n_tt; ++tt) {
        const double *p = part + 2 * (tt * nslots + j);
        re += p[0];
        im += p[1];
        if (both_modes) {
            re += p[2 * n_out];
            im += p[2 * n_out + 1];
        }
    }
    g[2 * j] = re;
    g[2 * j + 1] = im;
}

// ------------------------------------------------------------------ workspace
struct Layout {
    size_t keys_in, keys_out, vals_in, vals_out, cub, tiles, offs, gfast, ds, hn, cull, data, work, part, total;
    size_t cub_bytes;
    int64_t n_st;
    int64_t cull_cap;  // beams the culling table has room for
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

int64_t tile_count(const msgb_problem *p, const msgb_sum_opts *o) {
    if (o && o->tiling) return o->tiling->n_tiles;
    return (p->ns + TS - 1) / TS;
}

Layout layout(const msgb_problem *p, int64_t n_beams, bool with_data, int64_t n_st) {
    Layout l{};
    const int D = p->ndim;
    const int64_t ns = p->ns;
    l.n_st = n_st;
    size_t cub_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                    (const int32_t *)nullptr, (int32_t *)nullptr, (int)ns);
    l.cub_bytes = cub_bytes;
    size_t o = 0;
    l.keys_in = o; o = align256(o + ns * 4);
    l.keys_out = o; o = align256(o + ns * 4);
    l.vals_in = o; o = align256(o + ns * 4);
    l.vals_out = o; o = align256(o + ns * 4);
    l.cub = o; o = align256(o + cub_bytes);
    l.tiles = o; o = align256(o + n_st * sizeof(TileInfo<3>));
    l.offs = o; o = align256(o + (n_st + 1) * 4);
    l.gfast = o; o = align256(o + n_st * NW);
    l.ds = o; o = align256(o + ns * D * 4);
    l.hn = o; o = align256(o + ns * D * 4);
    l.cull_cap = n_beams > 0 ? n_beams : 1;
    l.cull = o; o = align256(o + l.cull_cap * sizeof(Cull<3>));
    l.data = o; o = align256(o + (with_data ? p->nt * ns * 4 : 0));
    l.work = o; o = align256(o + 64);
    // (the closed-form beam table follows when the caller's workspace has room: see hom_bytes)
    // adjoint partials: one complex FP64 per (time tile, beam mode) of the coefficients
    l.part = o; o = align256(o + (with_data ? (size_t)((p->nt + TT - 1) / TT) * 2 * (n_beams > 0 ? n_beams : 0) * 16 : 0));
    l.total = o;
    return l;
}

// The closed-form beam table (HomBeam), after everything else in a workspace
// sized by msgb_sum_f32_workspace_size; a smaller scratch (the static one, for
// many coefficients) goes without and every record pass prepares its beams.
size_t hom_bytes(int ndim, int64_t n) {
    const size_t per = ndim == 1 ? sizeof(HomBeam<1>) : (ndim == 2 ? sizeof(HomBeam<2>) : sizeof(HomBeam<3>));
    return align256(per * (size_t)(n > 0 ? n : 0));
}

template <int D>
const HomBeam<D> *prepare_hom(const msgb_problem *p, const msgb_beam_set *b, char *at, size_t spare, cudaStream_t st) {
    if (b->n == 0 || spare < hom_bytes(D, b->n)) return nullptr;
    HomBeam<D> *h = (HomBeam<D> *)at;
    hom_prep_kernel<D><<<(unsigned)((b->n + 127) / 128), 128, 0, st>>>(to_args(p), to_args(b), h);
    return h;
}

// Ranges of the beams per tile for a forward over n_tiles tiles and nbeam beams
// (2^62: as many as the tiles ask for).
int split_count(int64_t n_tiles, int64_t nbeam) {
    if (n_tiles <= 0) return 1;
    const int64_t want = (kItemsWanted + n_tiles - 1) / n_tiles, most = (nbeam + kSplitMin - 1) / kSplitMin;
    const int64_t n = want < most ? want : most;
    return (int)(n < 1 ? 1 : n);
}

// Partials of the split forward for any tiling of the problem's sensors.
size_t split_bytes(const msgb_problem *p, int64_t nbeam) {
    const int64_t n = split_count((p->ns + TS - 1) / TS * ((p->nt + TT - 1) / TT), nbeam);
    return n > 1 ? align256((size_t)n * (size_t)p->ns * (size_t)p->nt * sizeof(float2)) : 0;
}

// The ranges of a problem, with their partials at `at` where `spare` bytes hold them.
Split make_split(const msgb_problem *p, int64_t n_tiles, int64_t nbeam, char *at, size_t spare) {
    const size_t per = (size_t)p->ns * (size_t)p->nt * sizeof(float2);
    int64_t n = split_count(n_tiles, nbeam);
    if (n < 2) return Split{1, nbeam > 0 ? nbeam : 1, nullptr};
    const int64_t len = ((nbeam + n - 1) / n + G - 1) / G * G;
    n = (nbeam + len - 1) / len;
    return Split{(int)n, len, n > 1 && per * (size_t)n <= spare ? (float2 *)at : nullptr};
}

// Limits of a trajectory chunk of nb beams (refine).  They follow everything else in a
// workspace sized by msgb_sum_f32_traj_workspace_size; a smaller one goes without.
size_t traj_limit_bytes(const msgb_problem *p, int64_t nb) {
    return align256((size_t)((p->nt + TT - 1) / TT) * (size_t)(nb > 0 ? nb : 0) * sizeof(uint32_t));
}

// Adjoint partials of a trajectory chunk of nb beams: (n_tt, nb) complex FP64.
size_t traj_part_bytes(const msgb_problem *p, int64_t nb) {
    return align256((size_t)((p->nt + TT - 1) / TT) * (size_t)(nb > 0 ? nb : 0) * 16);
}

__global__ void copy_i32_kernel(const int32_t *in, int64_t n, int32_t *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

// Caller-provided tile offsets are clamped so that every tile lies in
// [0, ns) and holds at most TS sensors; order entries outside [0, ns) are
// replaced by 0.  (A malformed tiling gives wrong numbers, never an
// out-of-bounds access.)
__global__ void sanitize_tiling_kernel(const int32_t *offs_in, int64_t n_st, int64_t ns, int32_t *offs,
                                       int32_t *order) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i <= n_st) {
        int64_t v = offs_in[i];
        v = v < 0 ? 0 : (v > ns ? ns : v);
        offs[i] = (int32_t)v;
    }
    for (int64_t k = i; k < ns; k += (int64_t)gridDim.x * blockDim.x)
        if (order[k] < 0 || order[k] >= ns) order[k] = 0;
}

__global__ void clamp_tiles_kernel(int32_t *offs, int64_t n_st) {
    // serial pass (n_st is small): non-decreasing, at most TS per tile
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int64_t i = 1; i <= n_st; ++i) {
        int32_t lo = offs[i - 1];
        int32_t v = offs[i] < lo ? lo : offs[i];
        if (v - lo > TS) v = lo + TS;
        offs[i] = v;
    }
}

template <int D>
int prep(const msgb_problem *p, const msgb_beam_set *b, const msgb_sum_opts *o, const Layout &l, char *ws,
         cudaStream_t st) {
    const int64_t ns = p->ns;
    if (b->n > l.cull_cap) return fail(MSGB_ERR_WORKSPACE, "culling table sized for %lld beams, got %lld",
                                       (long long)l.cull_cap, (long long)b->n);
    uint32_t *kin = (uint32_t *)(ws + l.keys_in), *kout = (uint32_t *)(ws + l.keys_out);
    int32_t *vin = (int32_t *)(ws + l.vals_in), *vout = (int32_t *)(ws + l.vals_out);
    int32_t *offs = (int32_t *)(ws + l.offs);
    const int blk = 256;
    if (o && o->tiling) {
        if (!o->tiling->order || !o->tiling->tile_offsets || o->tiling->n_tiles <= 0)
            return fail(MSGB_ERR_ARG, "sensor tiling: NULL arrays or no tiles");
        copy_i32_kernel<<<(unsigned)((ns + blk - 1) / blk), blk, 0, st>>>(o->tiling->order, ns, vout);
        sanitize_tiling_kernel<<<(unsigned)((l.n_st + 1 + blk - 1) / blk), blk, 0, st>>>(o->tiling->tile_offsets,
                                                                                        l.n_st, ns, offs, vout);
        clamp_tiles_kernel<<<1, 1, 0, st>>>(offs, l.n_st);
    } else {
        sensor_key_kernel<D><<<(unsigned)((ns + blk - 1) / blk), blk, 0, st>>>(p->sensors, ns, to_args(p), kin, vin);
        size_t cb = l.cub_bytes;
        cudaError_t e = cub::DeviceRadixSort::SortPairs(ws + l.cub, cb, kin, kout, vin, vout, (int)ns, 0, 32, st);
        if (e != cudaSuccess) return fail(MSGB_ERR_CUDA, "sensor sort: %s", cudaGetErrorString(e));
        fixed_offsets_kernel<<<(unsigned)((l.n_st + 1 + blk - 1) / blk), blk, 0, st>>>(offs, l.n_st, ns);
    }
    tile_kernel<D><<<(unsigned)l.n_st, 128, 0, st>>>(p->sensors, vout, offs, to_args(p), (TileInfo<D> *)(ws + l.tiles),
                                                    (float *)(ws + l.ds), (float *)(ws + l.hn), (uint8_t *)(ws + l.gfast));
    if (b->n > 0)
        cull_prep_kernel<D><<<(unsigned)((b->n + blk - 1) / blk), blk, 0, st>>>(to_args(b), (Cull<D> *)(ws + l.cull));
    return check_launch("msgb sum f32 prep");
}

int sm_count() {
    int dev = 0, n = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

// The limits of T's records at `at`, where cutoff, domain and the `spare` bytes there
// allow; returns the bytes taken.
template <int D>
size_t prepare_limits(const msgb_problem *p, const msgb_sum_opts *o, TrajSrc<D> &T, char *at, size_t spare,
                      cudaStream_t st) {
    const size_t bytes = traj_limit_bytes(p, T.nb);
    const float cutoff = o ? (float)o->cutoff : 0.0f;
    for (int i = 0; i < D; ++i)
        if (p->periodic[i]) return 0;
    if (!(cutoff > 0.0f) || T.nb == 0 || spare < bytes) return 0;
    const int64_t items = (p->nt + TT - 1) / TT * T.nb, want = 8LL * sm_count(), share = items / (want * NW);
    const int per = (int)(share < 1 ? 1 : (share > 32 ? 32 : share));
    const int64_t need = (items + (int64_t)per * NW - 1) / ((int64_t)per * NW);
    traj_limits_kernel<D><<<(unsigned)(want < need ? want : need), THREADS, 0, st>>>(
        T, p->nt, cutoff + kGroupMarginEfolds, per, (uint32_t *)at);
    T.limits = (const uint32_t *)at;
    return bytes;
}

template <int D, bool TRAJ>
int run_fwd(const msgb_problem *p, const msgb_beam_set *b, const msgb_sum_opts *o, char *ws, const Layout &l,
            size_t ws_used, size_t ws_bytes, float *out, cudaStream_t st, TrajSrc<D> T) {
    // trajectory sums cull with the records' own boxes: the closed-form
    // culling table (sized for no beams in their layout) is not built
    msgb_beam_set none{};
    if (int e = prep<D>(p, TRAJ ? &none : b, o, l, ws, st)) return e;
    const int64_t n_st = l.n_st, n_tt = (p->nt + TT - 1) / TT;
    if (n_st * n_tt > 0x7fffffffLL) return fail(MSGB_ERR_UNSUPPORTED, "msgb_sum_fwd_f32: too many tiles");
    const ProbArgs P = to_args(p);
    int *work = (int *)(ws + l.work);
    cudaMemsetAsync(work, 0, sizeof(int), st);
    bool periodic = false;
    for (int i = 0; i < D; ++i) periodic |= (p->periodic[i] != 0);
    size_t at = ws_used, spare = ws_bytes - ws_used;
    const HomBeam<D> *hom = nullptr;
    if (!TRAJ) {
        hom = prepare_hom<D>(p, b, ws + at, spare, st);
        if (hom) at += hom_bytes(D, b->n), spare -= hom_bytes(D, b->n);
    } else {
        const size_t taken = prepare_limits<D>(p, o, T, ws + at, spare, st);
        at += taken, spare -= taken;
    }
    const Split sp = make_split(p, n_st * n_tt, TRAJ ? T.nb : b->n, ws + at, spare);
    if (n_st * n_tt * sp.items_per_tile() > 0x7fffffffLL)
        return fail(MSGB_ERR_UNSUPPORTED, "msgb_sum_fwd_f32: too many tiles");
    const int n_items = (int)(n_st * n_tt * sp.items_per_tile());
    const int64_t want = 2LL * sm_count();
    const unsigned grid = (unsigned)(want < n_items ? want : n_items);
    const size_t smem = rec_bytes<D>() + (sp.serial() ? kTotalBytes : 0);
    auto args = [&](auto kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<grid, THREADS, smem, st>>>(P, to_args(b), (const Cull<D> *)(ws + l.cull), hom,
                                          (const TileInfo<D> *)(ws + l.tiles), (const int32_t *)(ws + l.offs),
                                          (const float *)(ws + l.ds), (const float *)(ws + l.hn),
                                          (const uint8_t *)(ws + l.gfast), (const int32_t *)(ws + l.vals_out),
                                          o ? (float)o->cutoff : 0.0f, out, o ? o->eval_count : nullptr, work,
                                          (int)n_st, n_items, sp, T);
    };
    if (periodic)
        args(fwd32_kernel<D, true, TRAJ>);
    else
        args(fwd32_kernel<D, false, TRAJ>);
    if (int e = check_launch("msgb_sum_fwd_f32")) return e;
    if (sp.part) {
        const dim3 cg((unsigned)((p->ns + 31) / 32), (unsigned)n_tt);
        if (cg.y > 65535u) return fail(MSGB_ERR_UNSUPPORTED, "msgb_sum_fwd_f32: nt too large");
        combine_parts_kernel<<<cg, dim3(32, 8), 0, st>>>(sp.part, sp.n, (const int32_t *)(ws + l.vals_out), p->nt, p->ns,
                                                         T.state, T.first, T.last, out);
        return check_launch("msgb_sum_fwd_f32 combine");
    }
    return MSGB_OK;
}

template <int D, bool TRAJ>
int run_adj(const msgb_problem *p, const msgb_beam_set *b, const msgb_sum_opts *o, char *ws, const Layout &l,
            size_t ws_used, size_t ws_bytes, const float *data, double *part, double *g, cudaStream_t st, TrajSrc<D> T) {
    msgb_beam_set none{};
    if (int e = prep<D>(p, TRAJ ? &none : b, o, l, ws, st)) return e;
    dim3 tg((unsigned)((p->ns + 31) / 32), (unsigned)((p->nt + 31) / 32));
    if (tg.y > 65535u) return fail(MSGB_ERR_UNSUPPORTED, "msgb_adj_gather_f32: nt too large");
    transpose_permute_kernel<<<tg, dim3(32, 8), 0, st>>>(data, (const int32_t *)(ws + l.vals_out), p->nt, p->ns,
                                                         (float *)(ws + l.data));
    const ProbArgs P = to_args(p);
    bool periodic = false;
    for (int i = 0; i < D; ++i) periodic |= (p->periodic[i] != 0);
    const int64_t nw = TRAJ ? T.nb : b->n;  // beam indices j of the items
    const int64_t n_st = l.n_st, n_tt = (p->nt + TT - 1) / TT;
    constexpr int64_t RJ = AdjRange<D, TRAJ>::RJ;
    int64_t rj = nw * n_tt / kItemsWanted / G * G;
    rj = rj > RJ ? RJ : (rj < G ? G : rj);
    const int64_t n_ranges = (nw + rj - 1) / rj;
    if (n_ranges * n_tt > 0x7fffffffLL || n_st > 0x7fffffffLL)
        return fail(MSGB_ERR_UNSUPPORTED, "msgb_adj_gather_f32: too many work items");
    int *work = (int *)(ws + l.work);
    cudaMemsetAsync(work, 0, sizeof(int), st);
    const int n_items = (int)(n_ranges * n_tt);
    const int64_t want = 2LL * sm_count();
    const unsigned grid = (unsigned)(want < n_items ? want : n_items);
    constexpr size_t smem = (size_t)AdjRange<D, TRAJ>::NACC * 2 * sizeof(double) + rec_bytes<D>();
    const HomBeam<D> *hom = TRAJ ? nullptr : prepare_hom<D>(p, b, ws + ws_used, ws_bytes - ws_used, st);
    if (TRAJ) prepare_limits<D>(p, o, T, ws + ws_used, ws_bytes - ws_used, st);
    auto args = [&](auto kern) {
        // static + dynamic shared memory exceed the default 48 KB: opt in
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<grid, THREADS, smem, st>>>(P, to_args(b), (const Cull<D> *)(ws + l.cull), hom,
                                          (const TileInfo<D> *)(ws + l.tiles), (const int32_t *)(ws + l.offs),
                                          (const float *)(ws + l.ds), (const float *)(ws + l.hn),
                                          (const uint8_t *)(ws + l.gfast), (const float *)(ws + l.data),
                                          o ? (float)o->cutoff : 0.0f, part, o ? o->eval_count : nullptr, work,
                                          (int)n_st, (int)rj, (int)n_ranges, n_items, T);
    };
    if (periodic)
        args(adj32_kernel<D, true, TRAJ>);
    else
        args(adj32_kernel<D, false, TRAJ>);
    if (int e = check_launch("msgb_adj_gather_f32")) return e;
    const int blk = 256;
    reduce_parts_kernel<<<(unsigned)((nw + blk - 1) / blk), blk, 0, st>>>(part, n_tt, TRAJ ? nw : 2 * nw, nw,
                                                                          TRAJ ? 0 : 1, g);
    return check_launch("msgb_adj_gather_f32 reduce");
}

template <int D>
TrajSrc<D> traj_src(const msgb_trajectories *t, float *state, int first, int last) {
    TrajSrc<D> T{};
    if (t) {
        T.nb = t->nb;
        T.b_first = t->b_first;
        T.rec = (const BeamTime<D> *)t->rec32;
        T.cull = t->cull;
        if (t->pool) {
            T.slot = t->slot;
            T.pool = (const BeamTime<D> *)t->pool;
            T.pool_cull = t->pool_cull;
        }
    }
    T.state = state;
    T.first = first;
    T.last = last;
    return T;
}

}  // namespace
}  // namespace msgb

using namespace msgb;

extern "C" size_t msgb_sum_f32_workspace_size(const msgb_problem *prob, int64_t n) {
    if (validate_problem(prob) || n < 0) return 0;
    // The default tiling has the most tiles a valid tiling of ns sensors needs
    // when every tile is full; reserve for one tile per 16 sensors so that
    // caller tilings with partial tiles fit as well.
    return layout(prob, n, true, (prob->ns + GS - 1) / GS).total + hom_bytes(prob->ndim, n) +
           split_bytes(prob, n);
}

static int check_ws(const msgb_problem *p, const msgb_beam_set *b, const msgb_sum_opts *o, bool with_data, void *ws,
                    size_t bytes, Layout &l) {
    l = layout(p, b->n, with_data, tile_count(p, o));
    if (l.n_st <= 0) return fail(MSGB_ERR_ARG, "sensor tiling has no tiles");
    if (b->n > (int64_t(1) << 26)) return fail(MSGB_ERR_UNSUPPORTED, "at most 2^26 selected coefficients");
    if (!ws || bytes < l.total)
        return fail(MSGB_ERR_WORKSPACE, "workspace too small: need %zu bytes, got %zu", l.total, bytes);
    if (((uintptr_t)ws & 255) != 0) return fail(MSGB_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    if (p->ns > 0x7fffffffLL) return fail(MSGB_ERR_UNSUPPORTED, "too many sensors");
    return MSGB_OK;
}

extern "C" int msgb_sum_fwd_f32(const msgb_problem *prob, const msgb_beam_set *beams, const msgb_sum_opts *opts,
                                void *workspace, size_t workspace_bytes, float *out, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!out) return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f32: out is NULL");
    if (prob->nt == 0 || prob->ns == 0) return MSGB_OK;
    Layout l;
    if (int e = check_ws(prob, beams, opts, false, workspace, workspace_bytes, l)) return e;
    cudaStream_t st = as_stream(stream);
    char *ws = (char *)workspace;
    switch (prob->ndim) {
        case 1: return run_fwd<1, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, out, st, traj_src<1>(nullptr, nullptr, 1, 1));
        case 2: return run_fwd<2, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, out, st, traj_src<2>(nullptr, nullptr, 1, 1));
        default: return run_fwd<3, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, out, st, traj_src<3>(nullptr, nullptr, 1, 1));
    }
}

extern "C" int msgb_adj_gather_f32(const msgb_problem *prob, const msgb_beam_set *beams, const msgb_sum_opts *opts,
                                   void *workspace, size_t workspace_bytes, const float *data, double *g,
                                   msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!data || !g) return fail(MSGB_ERR_ARG, "msgb_adj_gather_f32: NULL data or g");
    if (beams->n == 0) return MSGB_OK;
    if (prob->nt == 0 || prob->ns == 0) {
        cudaMemsetAsync(g, 0, sizeof(double) * 2 * beams->n, as_stream(stream));
        return check_launch("msgb_adj_gather_f32");
    }
    Layout l;
    if (int e = check_ws(prob, beams, opts, true, workspace, workspace_bytes, l)) return e;
    cudaStream_t st = as_stream(stream);
    char *ws = (char *)workspace;
    switch (prob->ndim) {
        case 1: return run_adj<1, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, data, (double *)(ws + l.part), g, st,
                                         traj_src<1>(nullptr, nullptr, 1, 1));
        case 2: return run_adj<2, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, data, (double *)(ws + l.part), g, st,
                                         traj_src<2>(nullptr, nullptr, 1, 1));
        default: return run_adj<3, false>(prob, beams, opts, ws, l, l.total, workspace_bytes, data, (double *)(ws + l.part), g, st,
                                          traj_src<3>(nullptr, nullptr, 1, 1));
    }
}

// ---- trajectory entry points ------------------------------------------------
static size_t traj_state_offset(const Layout &l) { return l.total; }

static size_t traj_state_bytes(const msgb_problem *p) { return align256((size_t)2 * p->nt * p->ns * sizeof(float)); }

extern "C" size_t msgb_sum_f32_traj_workspace_size(const msgb_problem *prob, int64_t nb_max) {
    if (validate_problem(prob) || nb_max < 0) return 0;
    const Layout l = layout(prob, 0, true, (prob->ns + GS - 1) / GS);
    // after the Kahan state: the adjoint's partials, or those of the split forward, and
    // the limits
    const size_t part = traj_part_bytes(prob, nb_max), split = split_bytes(prob, int64_t(1) << 62);
    return l.total + traj_state_bytes(prob) + (part > split ? part : split) + traj_limit_bytes(prob, nb_max);
}

// with_part: the adjoint's partials (n_tt, nb) follow the Kahan state.
static int check_traj32(const msgb_problem *p, const msgb_beam_set *b, const msgb_trajectories *t,
                        const msgb_sum_opts *o, void *ws, size_t bytes, bool with_part, Layout &l) {
    if (!t || (!t->rec32 && !t->pool)) return fail(MSGB_ERR_ARG, "FP32 trajectory records are NULL");
    if (t->pool) {
        if (!t->slot || !t->pool_cull) return fail(MSGB_ERR_ARG, "compact trajectories: slot or pool_cull is NULL");
    } else if (!t->cull && o && o->cutoff > 0.0) {
        return fail(MSGB_ERR_ARG, "culling boxes are NULL");
    }
    if (t->nb < 0 || t->b_first < 0 || t->b_first + t->nb > 2 * b->n)
        return fail(MSGB_ERR_ARG, "trajectory beam range outside [0, 2n)");
    l = layout(p, 0, true, tile_count(p, o));
    if (l.n_st <= 0) return fail(MSGB_ERR_ARG, "sensor tiling has no tiles");
    const size_t need = l.total + traj_state_bytes(p) + (with_part ? traj_part_bytes(p, t->nb) : 0);
    if (!ws || bytes < need) return fail(MSGB_ERR_WORKSPACE, "workspace too small: need %zu bytes, got %zu", need, bytes);
    if (((uintptr_t)ws & 255) != 0) return fail(MSGB_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    return MSGB_OK;
}

extern "C" int msgb_sum_fwd_f32_traj(const msgb_problem *prob, const msgb_beam_set *beams,
                                     const msgb_trajectories *traj, const msgb_sum_opts *opts, int first_chunk,
                                     int last_chunk, void *workspace, size_t workspace_bytes, float *out,
                                     msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!out) return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f32_traj: out is NULL");
    if (prob->nt == 0 || prob->ns == 0) return MSGB_OK;
    Layout l;
    if (int e = check_traj32(prob, beams, traj, opts, workspace, workspace_bytes, false, l)) return e;
    cudaStream_t st = as_stream(stream);
    char *ws = (char *)workspace;
    float *state = (float *)(ws + traj_state_offset(l));
    const int f = first_chunk != 0, la = last_chunk != 0;
    switch (prob->ndim) {
        case 1: return run_fwd<1, true>(prob, beams, opts, ws, l, traj_state_offset(l) + traj_state_bytes(prob), workspace_bytes, out, st, traj_src<1>(traj, state, f, la));
        case 2: return run_fwd<2, true>(prob, beams, opts, ws, l, traj_state_offset(l) + traj_state_bytes(prob), workspace_bytes, out, st, traj_src<2>(traj, state, f, la));
        default: return run_fwd<3, true>(prob, beams, opts, ws, l, traj_state_offset(l) + traj_state_bytes(prob), workspace_bytes, out, st, traj_src<3>(traj, state, f, la));
    }
}

extern "C" int msgb_adj_gather_f32_traj(const msgb_problem *prob, const msgb_beam_set *beams,
                                        const msgb_trajectories *traj, const msgb_sum_opts *opts, void *workspace,
                                        size_t workspace_bytes, const float *data, double *g, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!data || !g) return fail(MSGB_ERR_ARG, "msgb_adj_gather_f32_traj: NULL data or g");
    if (!traj || traj->nb == 0) return MSGB_OK;
    if (prob->nt == 0 || prob->ns == 0) {
        cudaMemsetAsync(g, 0, sizeof(double) * 2 * traj->nb, as_stream(stream));
        return check_launch("msgb_adj_gather_f32_traj");
    }
    Layout l;
    if (int e = check_traj32(prob, beams, traj, opts, workspace, workspace_bytes, true, l)) return e;
    cudaStream_t st = as_stream(stream);
    char *ws = (char *)workspace;
    double *part = (double *)(ws + traj_state_offset(l) + traj_state_bytes(prob));
    const size_t used = traj_state_offset(l) + traj_state_bytes(prob) + traj_part_bytes(prob, traj->nb);
    switch (prob->ndim) {
        case 1: return run_adj<1, true>(prob, beams, opts, ws, l, used, workspace_bytes, data, part, g, st, traj_src<1>(traj, nullptr, 1, 1));
        case 2: return run_adj<2, true>(prob, beams, opts, ws, l, used, workspace_bytes, data, part, g, st, traj_src<2>(traj, nullptr, 1, 1));
        default: return run_adj<3, true>(prob, beams, opts, ws, l, used, workspace_bytes, data, part, g, st, traj_src<3>(traj, nullptr, 1, 1));
    }
}

// ---- sensor-tile boxes (for the compact trajectory store) -------------------
namespace msgb {
namespace {
template <int D>
__global__ void tile_boxes_kernel(const TileInfo<D> *tiles, int64_t n_st, float *boxes) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n_st) return;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        boxes[i * 2 * D + a] = tiles[i].lo[a];
        boxes[i * 2 * D + D + a] = tiles[i].hi[a];
    }
}

template <int D>
int tile_boxes(const msgb_problem *p, const msgb_sum_opts *o, char *ws, const Layout &l, float *boxes,
               cudaStream_t st) {
    msgb_beam_set none{};
    if (int e = prep<D>(p, &none, o, l, ws, st)) return e;
    tile_boxes_kernel<D><<<(unsigned)((l.n_st + 127) / 128), 128, 0, st>>>((const TileInfo<D> *)(ws + l.tiles),
                                                                           l.n_st, boxes);
    return check_launch("msgb_sum_f32_tile_boxes");
}
}  // namespace
}  // namespace msgb

extern "C" int64_t msgb_sum_f32_tile_count(const msgb_problem *prob, const msgb_sum_opts *opts) {
    if (validate_problem(prob)) return -1;
    return tile_count(prob, opts);
}

extern "C" int msgb_sum_f32_tile_boxes(const msgb_problem *prob, const msgb_sum_opts *opts, void *workspace,
                                       size_t workspace_bytes, float *boxes, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (!boxes) return fail(MSGB_ERR_ARG, "msgb_sum_f32_tile_boxes: boxes is NULL");
    if (prob->ns == 0) return MSGB_OK;
    const Layout l = layout(prob, 0, true, tile_count(prob, opts));
    if (l.n_st <= 0) return fail(MSGB_ERR_ARG, "sensor tiling has no tiles");
    if (!workspace || workspace_bytes < l.total)
        return fail(MSGB_ERR_WORKSPACE, "workspace too small: need %zu bytes, got %zu", l.total, workspace_bytes);
    if (((uintptr_t)workspace & 255) != 0) return fail(MSGB_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    cudaStream_t st = as_stream(stream);
    char *ws = (char *)workspace;
    switch (prob->ndim) {
        case 1: return tile_boxes<1>(prob, opts, ws, l, boxes, st);
        case 2: return tile_boxes<2>(prob, opts, ws, l, boxes, st);
        default: return tile_boxes<3>(prob, opts, ws, l, boxes, st);
    }
}

// ---- forward summation for callers that cannot allocate ----------------------
//
// Some hosts cannot hand this library device memory: an XLA custom-call or
// plugin handler registered without a scratch allocator, a runtime whose
// device memory belongs entirely to another framework's pool, or a process
// with allocation forbidden once serving starts.  For them the FP32 forward
// takes its scratch from the fixed array below instead of a caller workspace.
// The array is part of the module: every GPU that loads the library holds it
// until the process exits.  In host code `sum32_static_scratch` only stands in
// for the symbol; the device address comes from cudaGetSymbolAddress, taken
// once per device on the first call made with that device current.
static __device__ __align__(256) unsigned char sum32_static_scratch[MSGB_SUM_F32_STATIC_SCRATCH_BYTES];

namespace {
constexpr int kMaxStaticDevices = 64;
std::mutex static_scratch_mu;
void *static_scratch_ptr[kMaxStaticDevices] = {};

int static_scratch_address(void **ptr) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(MSGB_ERR_CUDA, "msgb_sum_fwd_f32_static: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxStaticDevices)
        return fail(MSGB_ERR_UNSUPPORTED, "msgb_sum_fwd_f32_static: device ordinal %d beyond %d", dev,
                    kMaxStaticDevices - 1);
    std::lock_guard<std::mutex> lock(static_scratch_mu);
    if (!static_scratch_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, sum32_static_scratch);
        if (e != cudaSuccess || !p)
            return fail(MSGB_ERR_CUDA, "msgb_sum_fwd_f32_static: cudaGetSymbolAddress on device %d: %s", dev,
                        cudaGetErrorString(e));
        static_scratch_ptr[dev] = p;
    }
    *ptr = static_scratch_ptr[dev];
    return MSGB_OK;
}
}  // namespace

extern "C" int msgb_sum_fwd_f32_static(const msgb_problem *prob, const msgb_beam_set *beams,
                                       const msgb_sum_opts *opts, float *out, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!out) return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f32_static: out is NULL");
    if (prob->nt == 0 || prob->ns == 0) return MSGB_OK;
    const Layout need = layout(prob, beams->n, false, tile_count(prob, opts));
    if (need.total > (size_t)MSGB_SUM_F32_STATIC_SCRATCH_BYTES)
        return fail(MSGB_ERR_UNSUPPORTED,
                    "msgb_sum_fwd_f32_static: %lld coefficients and %lld sensors need %zu bytes of scratch, more "
                    "than the %zu-byte static scratch; call msgb_sum_fwd_f32 with a workspace instead",
                    (long long)beams->n, (long long)prob->ns, need.total, (size_t)MSGB_SUM_F32_STATIC_SCRATCH_BYTES);
    cudaStream_t st = as_stream(stream);
    if (st) {
        // the array's address is per device: the stream must run on the current one
        int cur = 0, sdev = 0;
        cudaError_t e = cudaGetDevice(&cur);
        if (e == cudaSuccess) e = cudaStreamGetDevice(st, &sdev);
        if (e != cudaSuccess)
            return fail(MSGB_ERR_CUDA, "msgb_sum_fwd_f32_static: device of the stream: %s", cudaGetErrorString(e));
        if (sdev != cur)
            return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f32_static: the stream belongs to device %d but device %d is current",
                        sdev, cur);
    }
    void *scratch = nullptr;
    if (int e = static_scratch_address(&scratch)) return e;
    Layout l;
    if (int e = check_ws(prob, beams, opts, false, scratch, MSGB_SUM_F32_STATIC_SCRATCH_BYTES, l)) return e;
    // Only the persistent kernel's work counter must start at zero; run_fwd
    // clears it on the stream before the launch.  Everything else in the
    // scratch is written by this call's preparation kernels before it is read.
    char *ws = (char *)scratch;
    switch (prob->ndim) {
        case 1: return run_fwd<1, false>(prob, beams, opts, ws, l, l.total, (size_t)MSGB_SUM_F32_STATIC_SCRATCH_BYTES, out, st, traj_src<1>(nullptr, nullptr, 1, 1));
        case 2: return run_fwd<2, false>(prob, beams, opts, ws, l, l.total, (size_t)MSGB_SUM_F32_STATIC_SCRATCH_BYTES, out, st, traj_src<2>(nullptr, nullptr, 1, 1));
        default: return run_fwd<3, false>(prob, beams, opts, ws, l, l.total, (size_t)MSGB_SUM_F32_STATIC_SCRATCH_BYTES, out, st, traj_src<3>(nullptr, nullptr, 1, 1));
    }
}
