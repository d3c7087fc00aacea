// Dense FP64 Gaussian-beam summation and its exact transpose.
//
// Forward: restates compute_gaussian_beam_real (beamax gb/core.py:194-329)
// with solve_hom_diag (gb/gb_solvers.py:356-422) fused in: every beam is
// evaluated at every (time, sensor) pair, as the reference does; there is no
// cutoff.  Each CTA owns a tile of times x sensors, keeps its outputs in
// registers and streams the beams through shared memory, so every output is
// written exactly once and the summation order is fixed (deterministic).  Where
// there are few tiles, a cluster of 2 to 8 CTAs shares a tile's beams and adds its
// partials, in rank order, through distributed shared memory.
//
// Transpose: one CTA (or cluster, over the times) per selected coefficient gathers
//   g_j = sum_{mode, t, s} 2 d(t, s) conj(A_j(t)) exp(-i w phi) exp(-w chi)
// over all times and sensors in a fixed order (no atomics).
//
// Bound: FP64 pipe (16 lanes per scheduler), 45 operations per evaluation in 2D
// forward and 55 in the transpose; 83 % and 67 % of its cycles busy.  With the
// library's cos, sincos and exp an evaluation issued 148 instructions, 62 of them
// FP64.  256^2, 3,000 coefficients, 1,207 times, 1,020 sensors: forward 52.5 -> 24.0
// ms, transpose 51.6 -> 34.0 ms.
#include <cooperative_groups.h>

#include "common.cuh"

namespace msgb {
namespace {

namespace cg = cooperative_groups;

constexpr int THREADS = 256;
constexpr int NWARP = THREADS / 32;

// ---------------------------------------------------------------- elementary functions
// cos, sin and exp for the evaluation loop, written so that the integer work is a
// few ALU instructions beside the FP64 pipe.  The reductions are Cody-Waite with
// the constant split in two doubles; the polynomials interpolate cos(sqrt u),
// sin(sqrt u) / sqrt u on [0, (pi/2)^2] and exp on [-ln 2 / 2, ln 2 / 2] at Chebyshev
// nodes (60-digit arithmetic; 7.7e-17, 1.3e-17 and 1.2e-17 with the rounded
// coefficients).
constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer (low word)
// The coefficients live in constant memory, highest power first: an FP64 FMA reads
// its addend from there, while a literal costs two moves per use (72 of the 121
// instructions of an evaluation with literals were not FP64).
__constant__ double kCos[8] = {4.60894348170413739e-14, -1.14628987994669932e-11, 2.08765617238124609e-09,
                               -2.75573163887740038e-07, 2.48015872773908771e-05, -1.38888888887728516e-03,
                               4.16666666666638819e-02,  -4.99999999999999722e-01};
__constant__ double kSin[8] = {2.72155724195411150e-15, -7.64302491987768254e-13, 1.60589408171723864e-10,
                               -2.50521068893805669e-08, 2.75573192112169089e-06, -1.98412698412086028e-04,
                               8.33333333333318577e-03,  -1.66666666666666657e-01};
__constant__ double kExp[10] = {2.51100608048383455e-08, 2.76326698075302949e-07, 2.75572408558713503e-06,
                                2.48014854007818843e-05, 1.98412698901057061e-04, 1.38888889523909706e-03,
                                8.33333333331957860e-03, 4.16666666664878074e-02, 1.66666666666666796e-01,
                                5.00000000000001887e-01};
__constant__ double kRed[8] = {0.3183098861837907, 3.141592653589793,  1.2246467991473532e-16,  // 1 / pi, pi
                               1.4426950408889634, 0.6931471805599453, 2.3190468138462996e-17,  // 1 / ln 2, ln 2
                               kRound, 1.0};

// a exp(x) (cos ph, sin ph) by the library
__device__ __noinline__ double2 far_value(double a, double ph, double x) {
    double s, c;
    sincos(ph, &s, &c);
    const double e = exp(x);
    return make_double2(a * c * e, a * s * e);
}

// |cos| and |sin| up to the common sign (-1)^n of the reduced angle: returns n; c
// and (with SIN) s.  far is set for angles beyond 2^49 (and inf, NaN), whose value is
// not valid: the caller evaluates those with the library's functions, once for
// all of its evaluations in flight, so that their chains interleave.
template <bool SIN>
__device__ __forceinline__ int reduced_sincos(double x, double &c, double &s, bool &far) {
    double nd = fma(x, kRed[0], kRed[6]);
    int n = __double2loint(nd);
    nd -= kRed[6];
    double r = fma(-nd, kRed[1], x);
    r = fma(-nd, kRed[2], r);
    const double u = r * r;
    double p = kCos[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) p = fma(p, u, kCos[k]);
    c = fma(p, u, kRed[7]);
    if (SIN) {
        double q = kSin[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) q = fma(q, u, kSin[k]);
        s = fma(q * u, r, r);
    }
    far |= (unsigned)(__double2hiint(x) & 0x7fffffff) >= 0x43000000u;
    return n;
}

// exp(x) = p * s1 * s2 with s1, s2 powers of two (two factors: the product may be
// subnormal or zero); flip: its low bit is xored into the sign of s1.  x below -1400
// is taken as -1400: the product is zero either way, and in a large domain narrow
// beams are that far from most sensors.  far is set for x >= 1400, inf and NaN.
__device__ __forceinline__ void split_exp(double x, int flip, double &p, double &s1, double &s2, bool &far) {
    const int hi = __double2hiint(x);
    const bool off = (unsigned)(hi & 0x7fffffff) >= 0x4095e000u;  // |x| >= 1400
    const bool zero = off && (unsigned)hi < 0xfff00000u && hi < 0;
    far |= off && !zero;
    if (zero) x = -1400.0;
    double nd = fma(x, kRed[3], kRed[6]);
    int n = __double2loint(nd);
    nd -= kRed[6];
    double r = fma(-nd, kRed[4], x);
    r = fma(-nd, kRed[5], r);
    p = kExp[0];
#pragma unroll
    for (int k = 1; k < 10; ++k) p = fma(p, r, kExp[k]);
    p = fma(p, r, kRed[7]);
    p = fma(p, r, kRed[7]);
    const int n1 = n >> 1, n2 = n - n1;
    s1 = __hiloint2double(((n1 + 1023) << 20) ^ (flip << 31), 0);
    s2 = __hiloint2double((n2 + 1023) << 20, 0);
}

// ---------------------------------------------------------------- records
// Forward: amp = 2 |A|, ang = arg A.  Transpose: amp, ang = 2 Re A, 2 Im A.
template <int D>
struct alignas(16) Rec64 {
    double x[D];
    double wp[D];
    double qr[D * (D + 1) / 2];  // w/2 * Re M (off-diagonals doubled)
    double qi[D * (D + 1) / 2];  // w/2 * Im M (off-diagonals doubled)
    double amp, ang;
};

template <int D>
__device__ __forceinline__ void load_beam(const BeamArgs &B, int64_t j, double *x0, double *p0,
                                          cd *al, cd &a0, double &w) {
#pragma unroll
    for (int i = 0; i < D; ++i) {
        x0[i] = B.x0[j * D + i];
        p0[i] = B.p0[j * D + i];
        al[i] = cd{B.alpha[2 * (j * D + i)], B.alpha[2 * (j * D + i) + 1]};
    }
    a0 = cd{B.a0[2 * j], B.a0[2 * j + 1]};
    w = B.omega[j];
}

template <int D>
struct TrajView {  // msgb_rk4_trajectories rec64 layout
    int64_t nb, b_first;
    const double *rec64;
};

template <int D, bool POLAR>
__device__ __forceinline__ void set_amplitude(Rec64<D> &r, cd A) {
    if (POLAR) {
        r.amp = 2.0 * hypot(A.re, A.im);
        r.ang = safe_angle(A);
    } else {
        r.amp = 2.0 * A.re;
        r.ang = 2.0 * A.im;
    }
}

// Beam b in [0, 2n) (b >= n: mode -1) at time t, closed form.
template <int D, bool POLAR>
__device__ __forceinline__ void make_rec(const ProbArgs &P, const BeamArgs &B, int64_t b, double t,
                                         Rec64<D> &r) {
    const int64_t j = b < B.n ? b : b - B.n;
    const double c0 = b < B.n ? P.c : -P.c;
    double x0[D], p0[D], w;
    cd al[D], a0;
    load_beam<D>(B, j, x0, p0, al, a0, w);
    HomState<D> st;
    hom_state<D>(x0, p0, al, a0, c0, t, st);
#pragma unroll
    for (int i = 0; i < D; ++i) {
        r.x[i] = P.periodic[i] ? pymod(st.x[i], P.L[i]) : st.x[i];
        r.wp[i] = w * p0[i];
    }
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) {
            const int q = sym_index<D>(i, k);
            const double f = (i == k ? 0.5 : 1.0) * w;
            r.qr[q] = f * st.M[q].re;
            r.qi[q] = f * st.M[q].im;
        }
    set_amplitude<D, POLAR>(r, st.A);
}

// Beam bl of the chunk at save time k.
template <int D, bool POLAR>
__device__ __forceinline__ void make_rec_traj(const ProbArgs &P, const BeamArgs &B, const TrajView<D> &T, int64_t bl,
                                              int64_t k, Rec64<D> &r) {
    constexpr int NR = 2 * D + 2 * D * D + 2;
    const double *y = T.rec64 + (k * T.nb + bl) * NR;
    const int64_t b = T.b_first + bl;
    const int64_t j = b < B.n ? b : b - B.n;
    const double w = B.omega[j];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        r.x[i] = P.periodic[i] ? pymod(y[i], P.L[i]) : y[i];
        r.wp[i] = w * y[D + i];
    }
    const double *M = y + 2 * D;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int l = i; l < D; ++l) {
            const int q = sym_index<D>(i, l);
            const double mre = i == l ? M[2 * (i * D + i)] : M[2 * (i * D + l)] + M[2 * (l * D + i)];
            const double mim = i == l ? M[2 * (i * D + i) + 1] : M[2 * (i * D + l) + 1] + M[2 * (l * D + i) + 1];
            r.qr[q] = 0.5 * w * mre;
            r.qi[q] = 0.5 * w * mim;
        }
    const cd Au = cd{y[2 * D + 2 * D * D], y[2 * D + 2 * D * D + 1]};
    set_amplitude<D, POLAR>(r, cd{B.a0[2 * j], B.a0[2 * j + 1]} * Au);
}

template <int D>
__device__ __forceinline__ void zero_rec(Rec64<D> &r) {
    r.amp = r.ang = 0.0;  // contributes exactly zero
#pragma unroll
    for (int i = 0; i < D; ++i) r.x[i] = 0.0, r.wp[i] = 0.0;
#pragma unroll
    for (int q = 0; q < D * (D + 1) / 2; ++q) r.qr[q] = 0.0, r.qi[q] = 0.0;
}

// Phase (from ph0) and exponent of a record at sensor s.
template <int D, bool PERIODIC>
__device__ __forceinline__ void eval_terms(const Rec64<D> &r, const double *s, const ProbArgs &P, double ph0, double &ph,
                                           double &chi) {
    double Dl[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        double di = s[i] - r.x[i];
        if (PERIODIC && P.periodic[i]) di = di - P.L[i] * nearbyint(di / P.L[i]);
        Dl[i] = di;
    }
    double q = ph0;
    chi = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) q = fma(r.wp[i], Dl[i], q);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int k = i; k < D; ++k) {
            const int e = sym_index<D>(i, k);
            const double dd = Dl[i] * Dl[k];
            q = fma(r.qr[e], dd, q);
            chi = (i == 0 && k == 0) ? r.qi[e] * dd : fma(r.qi[e], dd, chi);
        }
    ph = q;
}

// Sum a cluster's partials v[0 .. n) of this thread into rank 0's, in rank order.
// buf: THREADS * n doubles of shared memory at the same offset in every CTA.
template <int N>
__device__ __forceinline__ bool cluster_sum(double *v, double *buf, int split) {
    if (split == 1) return true;
    cg::cluster_group cl = cg::this_cluster();
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) buf[k * THREADS + threadIdx.x] = v[k];
    cl.sync();
    const unsigned rank = cl.block_rank();
    if (rank == 0) {
        for (int r = 1; r < split; ++r) {
            const double *o = cl.map_shared_rank(buf, r);
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] += o[k * THREADS + threadIdx.x];
        }
    }
    cl.sync();  // the partials stay until they are read
    return rank == 0;
}

// ---------------------------------------------------------------- forward
// Tile of TT times x TS sensors, two sensors per lane so that a record is read
// from shared memory once for both.  TT = 16: a warp has two of the times and 64
// sensors; TT = 1: one time, 512 sensors (images, or wide sensor sets: no work
// for times that do not exist, and 8 x fewer records made; 65,536 image points at
// one time, 4,000 beams: 21.1 -> 1.0 ms).
template <int TT>
struct FwdTile {
    static constexpr int TS = TT == 16 ? 64 : 512;
    static constexpr int NT = TT == 16 ? 2 : 1;  // times per thread
    static constexpr int BC = THREADS / TT;      // beams per pass
    static_assert(TT == 16 || TT == 1, "tile shapes");
};

template <int D, bool TRAJ, int TT, bool PERIODIC>
__global__ void __launch_bounds__(THREADS, 2)
fwd64_kernel(ProbArgs P, BeamArgs B, TrajView<D> T, int split, double *out) {
    using F = FwdTile<TT>;
    constexpr int NT = F::NT, BC = F::BC, UB = NT == 1 ? 2 : 1;  // evaluations in flight: 4
    __shared__ Rec64<D> recs[THREADS];
    static_assert(sizeof(recs) >= sizeof(double) * THREADS * NT * 2, "cluster partials reuse the records");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t s0 = (int64_t)blockIdx.x * F::TS + (TT == 16 ? lane : tid);
    constexpr int SSTEP = TT == 16 ? 32 : THREADS;
    const int64_t t_base = (int64_t)blockIdx.y * TT;
    const int tw = TT == 16 ? warp * NT : 0;  // this thread's first time of the tile

    double s[2][D], acc[NT][2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < D; ++i) s[q][i] = s0 + q * SSTEP < P.ns ? P.sensors[(s0 + q * SSTEP) * D + i] : 0.0;
#pragma unroll
    for (int k = 0; k < NT; ++k) acc[k][0] = acc[k][1] = 0.0;

    int64_t b_lo = 0, b_hi = TRAJ ? T.nb : 2 * B.n;
    if (!TRAJ && B.modes == 1) b_hi = B.n;
    if (!TRAJ && B.modes == 2) b_lo = B.n;
    if (split > 1) {
        const int64_t len = ((b_hi - b_lo + split - 1) / split + BC - 1) / BC * BC;
        b_lo += len * blockIdx.z;
        b_hi = min(b_hi, b_lo + len);
    }
    for (int64_t b0 = b_lo; b0 < b_hi; b0 += BC) {
        {
            const int64_t b = b0 + tid / TT, t = t_base + tid % TT;
            if (b < b_hi && t < P.nt) {
                Rec64<D> r;
                if constexpr (TRAJ)
                    make_rec_traj<D, true>(P, B, T, b, t, r);
                else
                    make_rec<D, true>(P, B, b, P.ts[t], r);
                recs[tid] = r;
            } else {
                zero_rec<D>(recs[tid]);
            }
        }
        __syncthreads();
        const int nbl = (b_hi - b0) < BC ? (int)(b_hi - b0) : BC;
#pragma unroll UB
        for (int bl = 0; bl < nbl; ++bl) {
            double v[NT][2], w[NT][2], ph[NT][2], chi[NT][2];
            bool far = false;
#pragma unroll
            for (int k = 0; k < NT; ++k) {
                const Rec64<D> r = recs[bl * TT + tw + k];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double c, sn, p, s1;
                    eval_terms<D, PERIODIC>(r, s[q], P, r.ang, ph[k][q], chi[k][q]);
                    const int n = reduced_sincos<false>(ph[k][q], c, sn, far);
                    split_exp(-chi[k][q], n, p, s1, w[k][q], far);
                    v[k][q] = (r.amp * c) * p * s1;
                }
            }
            if (far) {
#pragma unroll
                for (int k = 0; k < NT; ++k)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        v[k][q] = far_value(recs[bl * TT + tw + k].amp, ph[k][q], -chi[k][q]).x;
                        w[k][q] = 1.0;
                    }
            }
#pragma unroll
            for (int k = 0; k < NT; ++k)
#pragma unroll
                for (int q = 0; q < 2; ++q) acc[k][q] = fma(v[k][q], w[k][q], acc[k][q]);
        }
        __syncthreads();
    }
    if (!cluster_sum<NT * 2>(&acc[0][0], reinterpret_cast<double *>(recs), split)) return;
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int64_t t = t_base + tw + k;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int64_t si = s0 + q * SSTEP;
            if (t < P.nt && si < P.ns) {
                if (TRAJ)
                    out[t * P.ns + si] += acc[k][q];
                else
                    out[t * P.ns + si] = acc[k][q];
            }
        }
    }
}

// ---------------------------------------------------------------- transpose
// CTA (x, z): coefficient (or trajectory beam) x, range z of its (mode, time)
// records.  256 records are made at once, one per thread; each warp takes 32 of
// them over all sensors.
template <int D, bool TRAJ, bool PERIODIC>
__global__ void __launch_bounds__(THREADS, 2)
adj64_kernel(ProbArgs P, BeamArgs B, TrajView<D> T, const double *__restrict__ data, int split, double *g) {
    __shared__ Rec64<D> recs[THREADS];
    __shared__ double red[2][NWARP];
    const int64_t j = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double acc_re = 0.0, acc_im = 0.0;
    // record q: mode q / nt, time q % nt
    int64_t q_lo = 0, q_hi = TRAJ ? P.nt : 2 * P.nt;
    if (!TRAJ && B.modes == 1) q_hi = P.nt;
    if (!TRAJ && B.modes == 2) q_lo = P.nt;
    if (split > 1) {
        const int64_t len = (q_hi - q_lo + split - 1) / split;
        q_lo += len * blockIdx.z;
        q_hi = min(q_hi, q_lo + len);
    }
    for (int64_t q0 = q_lo; q0 < q_hi; q0 += THREADS) {
        const int64_t q = q0 + tid;
        if (q < q_hi) {
            Rec64<D> r;
            if constexpr (TRAJ)
                make_rec_traj<D, false>(P, B, T, j, q, r);
            else
                make_rec<D, false>(P, B, q < P.nt ? j : B.n + j, P.ts[q < P.nt ? q : q - P.nt], r);
            recs[tid] = r;
        }
        __syncthreads();
        const int nr = (q_hi - q0) < THREADS ? (int)(q_hi - q0) : THREADS;
#pragma unroll 1
        for (int i = warp; i < nr; i += NWARP) {
            const Rec64<D> r = recs[i];
            const int64_t qi = q0 + i;
            const double *drow = data + (qi < P.nt ? qi : qi - P.nt) * P.ns;
            double sr = 0.0, si = 0.0;
            // two sensors in flight; the last trip's second may be absent (weight 0)
            // and the next trip's sensors and data are loaded ahead
            double np[2][D], nd[2];
            auto fetch = [&](int64_t s) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t sh = min(s + 32 * h, P.ns - 1);
#pragma unroll
                    for (int a = 0; a < D; ++a) np[h][a] = __ldg(P.sensors + sh * D + a);
                    nd[h] = __ldg(drow + sh);
                }
            };
            if (lane < P.ns) fetch(lane);
#pragma unroll 1
            for (int64_t s = lane; s < P.ns; s += 64) {
                double e[2], ph[2], chi[2], dv[2], c[2], sn[2], sp[2][D];
                bool far = false;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    dv[h] = nd[h];
#pragma unroll
                    for (int a = 0; a < D; ++a) sp[h][a] = np[h][a];
                }
                fetch(s + 64);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double p, s1, s2;
                    eval_terms<D, PERIODIC>(r, sp[h], P, 0.0, ph[h], chi[h]);
                    const int n = reduced_sincos<true>(ph[h], c[h], sn[h], far);
                    split_exp(-chi[h], n, p, s1, s2, far);
                    e[h] = dv[h] * p * s1 * s2;
                }
                if (far) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double2 z = far_value(dv[h], ph[h], -chi[h]);
                        c[h] = z.x;
                        sn[h] = z.y;
                        e[h] = 1.0;
                    }
                }
                sr = fma(e[0], c[0], sr);
                si = fma(-e[0], sn[0], si);
                if (s + 32 < P.ns) {
                    sr = fma(e[1], c[1], sr);
                    si = fma(-e[1], sn[1], si);
                }
            }
            // 2 conj(A) * (sr + i si)
            acc_re += r.amp * sr + r.ang * si;
            acc_im += r.amp * si - r.ang * sr;
        }
        __syncthreads();
    }
    // fixed-order reduction over the block, then over the cluster
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc_re += __shfl_down_sync(0xffffffffu, acc_re, o);
        acc_im += __shfl_down_sync(0xffffffffu, acc_im, o);
    }
    if (lane == 0) red[0][warp] = acc_re, red[1][warp] = acc_im;
    __syncthreads();
    double v[2] = {0.0, 0.0};
    if (tid == 0)
        for (int k = 0; k < NWARP; ++k) v[0] += red[0][k], v[1] += red[1][k];
    if (!cluster_sum<2>(v, reinterpret_cast<double *>(recs), split)) return;
    if (tid == 0) {
        g[2 * j] = v[0];
        g[2 * j + 1] = v[1];
    }
}

// ---------------------------------------------------------------- launches
// CTAs a launch should have: 4 per resident CTA (2 per SM of the 148; a constant, as the
// order of the sums follows from it); a cluster of at most 8
// shares what would be one CTA's work until there are as many.
constexpr int64_t kCtasWanted = 4 * 2 * 148;

int cluster_split(int64_t ctas, int64_t work, int64_t least) {
    int split = 1;
    while (split < 8 && ctas * split < kCtasWanted && work / (2 * split) >= least) split *= 2;
    return split;
}

template <typename K, typename... A>
int launch(const char *what, K kern, dim3 grid, int split, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = (unsigned)split;
    cfg.attrs = at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
    if (e != cudaSuccess) return fail(MSGB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return check_launch(what);
}

template <int D, bool TRAJ>
int run_fwd(const char *what, const msgb_problem *p, const msgb_beam_set *b, TrajView<D> T, double *out, cudaStream_t st) {
    const ProbArgs P = to_args(p);
    const BeamArgs B = to_args(b);
    bool periodic = false;
    for (int i = 0; i < D; ++i) periodic |= P.periodic[i] != 0;
    // the tile shape with less padding; at equal padding (within 10 %) the wide
    // one, which makes 8 x fewer records
    auto padded = [](int64_t n, int64_t t) { return (double)((n + t - 1) / t * t); };
    const double tall = padded(p->nt, 16) * padded(p->ns, 64), wide = (double)p->nt * padded(p->ns, 512);
    const bool use_wide = p->nt <= 65535 && wide <= 1.1 * tall;
    const int64_t beams = TRAJ ? T.nb : (B.modes == 0 ? 2 * B.n : B.n);
    const dim3 tiles = use_wide ? dim3((unsigned)((p->ns + 511) / 512), (unsigned)p->nt)
                                : dim3((unsigned)((p->ns + 63) / 64), (unsigned)((p->nt + 15) / 16));
    if (tiles.y > 65535u) return fail(MSGB_ERR_UNSUPPORTED, "%s: nt too large", what);
    // a range of beams no shorter than four passes
    const int split = cluster_split((int64_t)tiles.x * tiles.y, beams, use_wide ? 4 * 256 : 4 * 16);
    const dim3 grid(tiles.x, tiles.y, (unsigned)split);
    if (use_wide)
        return periodic ? launch(what, fwd64_kernel<D, TRAJ, 1, true>, grid, split, st, P, B, T, split, out)
                        : launch(what, fwd64_kernel<D, TRAJ, 1, false>, grid, split, st, P, B, T, split, out);
    return periodic ? launch(what, fwd64_kernel<D, TRAJ, 16, true>, grid, split, st, P, B, T, split, out)
                    : launch(what, fwd64_kernel<D, TRAJ, 16, false>, grid, split, st, P, B, T, split, out);
}

template <int D, bool TRAJ>
int run_adj(const char *what, const msgb_problem *p, const msgb_beam_set *b, TrajView<D> T, const double *data, double *g,
            cudaStream_t st) {
    const ProbArgs P = to_args(p);
    const BeamArgs B = to_args(b);
    bool periodic = false;
    for (int i = 0; i < D; ++i) periodic |= P.periodic[i] != 0;
    const int64_t ctas = TRAJ ? T.nb : B.n;
    const int split = cluster_split(ctas, TRAJ || B.modes ? P.nt : 2 * P.nt, THREADS / 4);
    const dim3 grid((unsigned)ctas, 1, (unsigned)split);
    return periodic ? launch(what, adj64_kernel<D, TRAJ, true>, grid, split, st, P, B, T, data, split, g)
                    : launch(what, adj64_kernel<D, TRAJ, false>, grid, split, st, P, B, T, data, split, g);
}

}  // namespace
}  // namespace msgb

using namespace msgb;

extern "C" int msgb_sum_fwd_f64(const msgb_problem *prob, const msgb_beam_set *beams, double *out,
                                msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!out) return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f64: out is NULL");
    if (prob->nt == 0 || prob->ns == 0) return MSGB_OK;
    const char *what = "msgb_sum_fwd_f64";
    cudaStream_t st = as_stream(stream);
    switch (prob->ndim) {
        case 1: return run_fwd<1, false>(what, prob, beams, TrajView<1>{}, out, st);
        case 2: return run_fwd<2, false>(what, prob, beams, TrajView<2>{}, out, st);
        default: return run_fwd<3, false>(what, prob, beams, TrajView<3>{}, out, st);
    }
}

extern "C" int msgb_adj_gather_f64(const msgb_problem *prob, const msgb_beam_set *beams,
                                   const double *data, double *g, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (!data || !g) return fail(MSGB_ERR_ARG, "msgb_adj_gather_f64: NULL data or g");
    if (beams->n == 0) return MSGB_OK;
    if (beams->n > 0x7fffffffLL) return fail(MSGB_ERR_UNSUPPORTED, "msgb_adj_gather_f64: too many beams");
    const char *what = "msgb_adj_gather_f64";
    cudaStream_t st = as_stream(stream);
    switch (prob->ndim) {
        case 1: return run_adj<1, false>(what, prob, beams, TrajView<1>{}, data, g, st);
        case 2: return run_adj<2, false>(what, prob, beams, TrajView<2>{}, data, g, st);
        default: return run_adj<3, false>(what, prob, beams, TrajView<3>{}, data, g, st);
    }
}

static int check_traj(const msgb_beam_set *beams, const msgb_trajectories *t, bool need64) {
    if (!t) return fail(MSGB_ERR_ARG, "trajectories are NULL");
    if (need64 && !t->rec64) return fail(MSGB_ERR_ARG, "FP64 trajectory records are NULL");
    if (t->nb < 0 || t->b_first < 0 || t->b_first + t->nb > 2 * beams->n)
        return fail(MSGB_ERR_ARG, "trajectory beam range outside [0, 2n)");
    return MSGB_OK;
}

extern "C" int msgb_sum_fwd_f64_traj(const msgb_problem *prob, const msgb_beam_set *beams,
                                     const msgb_trajectories *traj, double *out, msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (int e = check_traj(beams, traj, true)) return e;
    if (!out) return fail(MSGB_ERR_ARG, "msgb_sum_fwd_f64_traj: out is NULL");
    if (prob->nt == 0 || prob->ns == 0 || traj->nb == 0) return MSGB_OK;
    const char *what = "msgb_sum_fwd_f64_traj";
    cudaStream_t st = as_stream(stream);
    switch (prob->ndim) {
        case 1: return run_fwd<1, true>(what, prob, beams, TrajView<1>{traj->nb, traj->b_first, traj->rec64}, out, st);
        case 2: return run_fwd<2, true>(what, prob, beams, TrajView<2>{traj->nb, traj->b_first, traj->rec64}, out, st);
        default: return run_fwd<3, true>(what, prob, beams, TrajView<3>{traj->nb, traj->b_first, traj->rec64}, out, st);
    }
}

extern "C" int msgb_adj_gather_f64_traj(const msgb_problem *prob, const msgb_beam_set *beams,
                                        const msgb_trajectories *traj, const double *data, double *g,
                                        msgb_stream_t stream) {
    if (int e = validate_problem(prob)) return e;
    if (int e = validate_beams(prob, beams)) return e;
    if (int e = check_traj(beams, traj, true)) return e;
    if (!data || !g) return fail(MSGB_ERR_ARG, "msgb_adj_gather_f64_traj: NULL data or g");
    if (traj->nb == 0) return MSGB_OK;
    if (traj->nb > 0x7fffffffLL) return fail(MSGB_ERR_UNSUPPORTED, "too many beams in one chunk");
    const char *what = "msgb_adj_gather_f64_traj";
    cudaStream_t st = as_stream(stream);
    switch (prob->ndim) {
        case 1: return run_adj<1, true>(what, prob, beams, TrajView<1>{traj->nb, traj->b_first, traj->rec64}, data, g, st);
        case 2: return run_adj<2, true>(what, prob, beams, TrajView<2>{traj->nb, traj->b_first, traj->rec64}, data, g, st);
        default: return run_adj<3, true>(what, prob, beams, TrajView<3>{traj->nb, traj->b_first, traj->rec64}, data, g, st);
    }
}
