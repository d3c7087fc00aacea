// MSWPT tiling on the GPU: one global FFT (cuFFT, a library call) followed by one
// launch with a CTA per box, over all levels, that fuses the dual-filter division,
// the window multiply, the parity roll, the unitary box IFFT (register passes of
// radix 8, 4 and 2 in shared memory), the IVP half-wave factor, the conjugate
// half-mask and the top_n key.
//
// Restates beamax transforms.py:591-733 (MSWPT.forward/_compute_coeffs) and
// :735-850 (MSWPT.inverse); the Hermitian adjoint of the forward is the
// inverse's structure with the forward's roll convention and a final division
// by sum g^2 (see the derivation next to msgb_mswpt_synthesis).
//
// Index conventions (per axis, N even, S even):
//   shifted Fourier index k in [0, N) <-> frequency k - N/2 (fftshift order);
//   unshifted FFT index u = (k + N/2) mod N;
//   patch element j of the box centred at c covers k = (c + N/2 - S/2 + j) mod N;
//   roll by r then ifftshift moves patch element j to q = (j - S/2 + r) mod S.
#include <cufft.h>

#include <vector>

#include "common.cuh"

struct msgb_mswpt {
    int nd;
    int N[3];
    int aspect[3];
    int red;
    int levels;
    int nbox;
    int64_t total;
    int64_t prodN;
    int64_t half_prodN;  // complex elements of the D2Z output
    // host copies of per-level metadata
    std::vector<int> bl;          // box_lengths
    std::vector<int> bshape;      // levels x nd (half supports)
    std::vector<int64_t> ccum;    // levels + 1
    std::vector<int> bcum;        // levels + 1
    std::vector<int> lat_cnt, lat_first, lat_step;  // levels x nd
    std::vector<int64_t> lat_off;                   // levels
    std::vector<int64_t> goff;                      // levels
    std::vector<int64_t> cand_off;                  // levels x 3
    int max_patch;                                  // max prod S
    // device tables
    int32_t *d_centres = nullptr;
    int32_t *d_lattice = nullptr;
    double *d_gfilt = nullptr;
    double *d_ssq = nullptr;
    int64_t *d_ccum = nullptr;
    int32_t *d_bcum = nullptr;
    int32_t *d_bl = nullptr;
    int32_t *d_bshape = nullptr;
    int2 *d_cand = nullptr;  // synthesis gather: see GatherLevel
    double2 *d_tw = nullptr;  // exp(2 pi i m / tw_n), m < tw_n (the largest support)
    int tw_n = 1;
    cufftHandle plan_d2z = 0, plan_z2z = 0;
    size_t fft_work = 0;
};

namespace msgb {
namespace {

constexpr int THREADS = 256;

struct LevelArgs {
    int nd;
    int N[3];
    int S[3];        // support per axis (powers of two)
    int logS[3];
    int bhs[3];      // half support (box_shapes)
    int P;           // prod S
    int nbox;        // boxes at this level
    int box0;        // global id of the first box
    int blk0;        // first CTA of the level in a launch over all levels
    int64_t c0;      // coefficient offset of the level
    int64_t seg;     // coefficients in the level
    double inv_sqrtS;
    const double *g;  // window of the level (prod S)
};

constexpr int kMaxLevels = 8;
struct AllLevels {
    int levels;
    const double2 *tw;
    int tw_n;
    LevelArgs lv[kMaxLevels];
};

int ilog2(int n) {
    int k = 0;
    while ((1 << k) < n) ++k;
    return k;
}

// Every level that has boxes, for one launch with a CTA per box; returns the CTAs.
int all_levels(const msgb_mswpt *p, AllLevels &A) {
    int blocks = 0;
    A.levels = 0;
    A.tw = p->d_tw;
    A.tw_n = p->tw_n;
    // the largest boxes first: the small ones fill the last wave
    for (int l = p->levels - 1; l >= 0; --l) {
        LevelArgs a{};
        a.nd = p->nd;
        a.P = 1;
        for (int i = 0; i < 3; ++i) {
            a.N[i] = i < p->nd ? p->N[i] : 1;
            a.bhs[i] = i < p->nd ? p->bshape[l * p->nd + i] : 1;
            a.S[i] = i < p->nd ? 2 * a.bhs[i] : 1;
            a.logS[i] = ilog2(a.S[i]);
            a.P *= a.S[i];
        }
        a.nbox = p->bcum[l + 1] - p->bcum[l];
        if (a.nbox == 0) continue;
        a.box0 = p->bcum[l];
        a.c0 = p->ccum[l];
        a.seg = p->ccum[l + 1] - p->ccum[l];
        a.inv_sqrtS = 1.0 / sqrt((double)a.P);
        a.g = p->d_gfilt + p->goff[l];
        a.blk0 = blocks;
        blocks += a.nbox;
        A.lv[A.levels++] = a;
    }
    return blocks;
}

__device__ __forceinline__ int floordiv(int a, int b) {
    int q = a / b;
    if ((a % b != 0) && ((a < 0) != (b < 0))) --q;
    return q;
}
__device__ __forceinline__ int imod(int a, int b) {
    int r = a % b;
    return r < 0 ? r + b : r;
}

// ---- box FFT: a (S0, S1, S2) complex array in shared memory ------------------
// Elements are padded by one per eight, so that the strided accesses of a pass
// spread over the banks.
__device__ __forceinline__ int pad(int i) { return i + (i >> 3); }

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmulz(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * (sign i)
__device__ __forceinline__ double2 mul_i(double2 a, double sign) { return make_double2(-sign * a.y, sign * a.x); }

// DFT of R values in registers, outputs in natural order (v[k] = sum_j v[j] w^(jk)).
template <int R>
__device__ __forceinline__ void dft(double2 *v, double sign) {
    if (R == 2) {
        const double2 a = v[0], b = v[1 % R];
        v[0] = cadd(a, b);
        v[1 % R] = csub(a, b);
    } else if (R == 4) {
        const double2 a = cadd(v[0], v[2 % R]), b = csub(v[0], v[2 % R]);
        const double2 c = cadd(v[1 % R], v[3 % R]), d = mul_i(csub(v[1 % R], v[3 % R]), sign);
        v[0] = cadd(a, c);
        v[1 % R] = cadd(b, d);
        v[2 % R] = csub(a, c);
        v[3 % R] = csub(b, d);
    } else if (R == 8) {
        double2 e[4] = {v[0], v[2 % R], v[4 % R], v[6 % R]}, o[4] = {v[1 % R], v[3 % R], v[5 % R], v[7 % R]};
        dft<4>(e, sign);
        dft<4>(o, sign);
        const double h = 0.70710678118654752440;
        o[1] = cmulz(o[1], make_double2(h, sign * h));
        o[2] = mul_i(o[2], sign);
        o[3] = cmulz(o[3], make_double2(-h, sign * h));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = cadd(e[k], o[k]);
            v[(k + 4) % R] = csub(e[k], o[k]);
        }
    }
}

// One decimation-in-frequency pass of radix R over sub-length len of an axis of
// element stride 2^lst: outputs stay in place, multiplied by w_len^(k i).
template <int R>
__device__ __forceinline__ void fft_pass(double2 *x, int total, int loglen, int lst, double sign, const double2 *tw,
                                         int tw_n) {
    constexpr int LR = R == 8 ? 3 : (R == 4 ? 2 : 1);
    const int lsub = loglen - LR;  // log2(len / R)
    const int step = tw_n >> loglen;
    for (int t = threadIdx.x; t < total / R; t += blockDim.x) {
        const int lo = t & ((1 << lst) - 1), rest = t >> lst;
        const int i = rest & ((1 << lsub) - 1), blk = rest >> lsub;
        const int base = (((blk << loglen) + i) << lst) + lo;
        double2 v[R];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = x[pad(base + (j << (lsub + lst)))];
        dft<R>(v, sign);
#pragma unroll
        for (int k = 1; k < R; ++k) {
            if (i) {
                double2 w = __ldg(tw + (size_t)(k * i) * step);
                w.y *= sign;
                v[k] = cmulz(v[k], w);
            }
        }
#pragma unroll
        for (int j = 0; j < R; ++j) x[pad(base + (j << (lsub + lst)))] = v[j];
    }
}

// Where frequency f of an axis of length 2^logn is after fft_box (digit reversal:
// radix 8 first, then what is left).
__device__ __forceinline__ int fft_position(int f, int logn) {
    int p = 0, left = logn;
    while (left > 0) {
        const int lr = left >= 3 ? 3 : left;
        left -= lr;
        p |= (f & ((1 << lr) - 1)) << left;
        f >>= lr;
    }
    return p;
}

// DFT along every axis, sign +1 (inverse) or -1 (forward), no scaling; frequency
// (f0, f1, f2) ends at position (fft_position(f0), ...).  Starts with a barrier.
__device__ void fft_box(double2 *x, const LevelArgs &L, double sign, const double2 *tw, int tw_n) {
    int lst = L.logS[0] + L.logS[1] + L.logS[2];
    for (int ax = 0; ax < L.nd; ++ax) {
        lst -= L.logS[ax];
        for (int left = L.logS[ax]; left > 0;) {
            __syncthreads();
            if (left >= 3) {
                fft_pass<8>(x, L.P, left, lst, sign, tw, tw_n);
                left -= 3;
            } else if (left == 2) {
                fft_pass<4>(x, L.P, left, lst, sign, tw, tw_n);
                left = 0;
            } else {
                fft_pass<2>(x, L.P, left, lst, sign, tw, tw_n);
                left = 0;
            }
        }
    }
    __syncthreads();
}

// This CTA's level and its box within the level.
__device__ __forceinline__ int find_level(const AllLevels &A, int &box) {
    int l = 0;
    while (l + 1 < A.levels && (int)blockIdx.x >= A.lv[l + 1].blk0) ++l;
    box = blockIdx.x - A.lv[l].blk0;
    return l;
}

// element e of a box -> coordinates
__device__ __forceinline__ void unravel(int e, const LevelArgs &L, int *j) {
    j[2] = e & (L.S[2] - 1);
    j[1] = (e >> L.logS[2]) & (L.S[1] - 1);
    j[0] = e >> (L.logS[1] + L.logS[2]);
}

struct FwdArgs {
    const double2 *X;  // spectrum
    int half;          // X is a D2Z half spectrum
    int shifted;       // X is already in shifted order (Fourier input)
    double in_scale;   // 1/sqrt(prod N) for spatial input
    const double *ssq;
    const int32_t *centres;
    double scale;
    int half_mask;
    double2 *coeffs;
    double *keys;
};

// Shared memory of a box kernel: the padded patch, then per axis and support
// element two index tables.
size_t box_smem(const LevelArgs &L) {
    return sizeof(double2) * (size_t)(L.P + (L.P >> 3)) + 3 * sizeof(int) * (size_t)(L.S[0] + L.S[1] + L.S[2]);
}

// Bound: latency (loads, the barriers between the FFT's passes) and index instructions:
// issue active 50 %, FP64 pipe 12 %, 5.6 warps per scheduler; the bytes (16 read and 24
// written per coefficient) take a fifth of its time.  All index arithmetic with
// divisions is done once per axis and support element in tables.
// 4.2 million coefficients of 1024^2: 477 us with radix-2 passes, a launch per level
// and divisions per element, 114 now (25 at the HBM rate).
__global__ void __launch_bounds__(THREADS, 3) box_forward_kernel(AllLevels LV, FwdArgs A) {
    extern __shared__ double2 sm[];
    int lbox;
    const LevelArgs &L = LV.lv[find_level(LV, lbox)];
    double2 *patch = sm;
    int *tab = reinterpret_cast<int *>(sm + L.P + (L.P >> 3));
    const int ST = L.S[0] + L.S[1] + L.S[2];
    int *tk = tab, *tu = tab + ST, *tq = tab + 2 * ST;  // shifted index, unshifted index, patch coordinate
    const int box = L.box0 + lbox;
    const int off[3] = {0, L.S[0], L.S[0] + L.S[1]};
    for (int a = 0; a < 3; ++a) {
        const int c = a < L.nd ? A.centres[box * L.nd + a] : 0;
        // forward rolls: ((centre + N/2) + N/2) // bhs   (transforms.py:626,665-673)
        const int ri = floordiv(c + L.N[a] / 2 + L.N[a] / 2, L.bhs[a]);
        const int r = a < L.nd ? (1 - 2 * (ri & 1)) * (L.bhs[a] / 2) : 0;
        for (int j = threadIdx.x; j < L.S[a]; j += blockDim.x) {
            const int k = a < L.nd ? imod(c + L.N[a] / 2 - L.S[a] / 2 + j, L.N[a]) : 0;
            tk[off[a] + j] = k;
            tu[off[a] + j] = imod(k + L.N[a] / 2, L.N[a]);
            tq[off[a] + j] = imod(j - L.S[a] / 2 + r, L.S[a]);
        }
    }
    __syncthreads();
    const int last = L.nd - 1, hl = L.N[last] / 2 + 1;
    for (int e = threadIdx.x; e < L.P; e += blockDim.x) {
        int j[3], k[3], u[3], q[3];
        unravel(e, L, j);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            k[a] = tk[off[a] + j[a]];
            u[a] = tu[off[a] + j[a]];
            q[a] = tq[off[a] + j[a]];
        }
        int64_t kflat = 0;
        for (int a = 0; a < L.nd; ++a) kflat = kflat * L.N[a] + k[a];
        double2 v;
        if (A.shifted) {
            v = A.X[kflat];
        } else {
            // a D2Z half spectrum (last axis N/2 + 1) is completed by X[u] = conj(X[-u])
            const bool cj = A.half && u[last] >= hl;
            int64_t idx = 0;
            for (int a = 0; a < L.nd; ++a) {
                const int w = cj ? (u[a] ? L.N[a] - u[a] : 0) : u[a];
                idx = idx * (A.half && a == last ? hl : L.N[a]) + w;
            }
            v = __ldg(A.X + idx);
            if (cj) v.y = -v.y;
        }
        // unitary spectrum / sum g^2, then * g (transforms.py:731, :663)
        const double s = __ldg(A.ssq + kflat), gv = __ldg(L.g + e);
        patch[pad((((q[0] << L.logS[1]) + q[1]) << L.logS[2]) + q[2])] =
            make_double2(v.x * A.in_scale / s * gv, v.y * A.in_scale / s * gv);
    }
    fft_box(patch, L, 1.0, LV.tw, LV.tw_n);
    // the tables now hold the frequencies' positions
    for (int a = 0; a < 3; ++a)
        for (int j = threadIdx.x; j < L.S[a]; j += blockDim.x) tq[off[a] + j] = fft_position(j, L.logS[a]);
    __syncthreads();
    const int64_t base = L.c0 + (int64_t)lbox * L.P;
    for (int e = threadIdx.x; e < L.P; e += blockDim.x) {
        int j[3];
        unravel(e, L, j);
        const int p = (((tq[j[0]] << L.logS[1]) + tq[off[1] + j[1]]) << L.logS[2]) + tq[off[2] + j[2]];
        const int64_t loc = (int64_t)lbox * L.P + e;
        const double m = (!A.half_mask || loc < L.seg / 2) ? A.scale * L.inv_sqrtS : 0.0;
        const double2 v = patch[pad(p)];
        const double re = v.x * m, im = v.y * m;
        A.coeffs[base + e] = make_double2(re, im);
        if (A.keys) A.keys[base + e] = __dsqrt_rn(__dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im)));
    }
}

struct SynArgs {
    const double2 *coeffs;
    const int32_t *centres;
    int adjoint;       // forward roll convention
    double2 *contrib;  // per-box contributions, coefficient layout
};

// Per box: unitary FFT of the coefficient block, fftshift, unroll and window
// (transforms.py:826-837).
__global__ void __launch_bounds__(THREADS, 3) box_synth_kernel(AllLevels LV, SynArgs A) {
    extern __shared__ double2 sm[];
    int lbox;
    const LevelArgs &L = LV.lv[find_level(LV, lbox)];
    double2 *patch = sm;
    int *tq = reinterpret_cast<int *>(sm + L.P + (L.P >> 3));
    const int box = L.box0 + lbox;
    const int off[3] = {0, L.S[0], L.S[0] + L.S[1]};
    const int64_t base = L.c0 + (int64_t)lbox * L.P;
    for (int a = 0; a < 3; ++a) {
        const int c = a < L.nd ? A.centres[box * L.nd + a] : 0;
        const int shift = A.adjoint ? L.N[a] : L.N[a] / 2;
        const int ri = floordiv(c + shift, L.bhs[a]);
        const int r = a < L.nd ? (1 - 2 * (ri & 1)) * (L.bhs[a] / 2) : 0;
        for (int j = threadIdx.x; j < L.S[a]; j += blockDim.x)
            tq[off[a] + j] = fft_position(imod(j + r + L.S[a] / 2, L.S[a]), L.logS[a]);
    }
    for (int e = threadIdx.x; e < L.P; e += blockDim.x) patch[pad(e)] = __ldg(A.coeffs + base + e);
    fft_box(patch, L, -1.0, LV.tw, LV.tw_n);
    for (int e = threadIdx.x; e < L.P; e += blockDim.x) {
        int j[3];
        unravel(e, L, j);
        const int p = (((tq[j[0]] << L.logS[1]) + tq[off[1] + j[1]]) << L.logS[2]) + tq[off[2] + j[2]];
        const double2 v = patch[pad(p)];
        const double s = __ldg(L.g + e) * L.inv_sqrtS;
        A.contrib[base + e] = make_double2(v.x * s, v.y * s);
    }
}

// One axis of a level's candidate lists, a thread per shifted index k: box i covers k
// iff (k - (first + i step + N/2) + S/2) mod N < S.  In lattice order: first the boxes
// whose support starts at or below the bin, then those that reach it around the end of
// the axis.  (On the host, over all boxes per bin, a 1D plan of 32,768 points and 2,048
// boxes took 136 ms, 1.5 this way.)
__global__ void candidates_kernel(int N, int S, int step, int cnt, int first, int2 *out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    const int z = imod(k - N / 2 + S / 2 - first, N);
    int2 c[4] = {make_int2(-1, 0), make_int2(-1, 0), make_int2(-1, 0), make_int2(-1, 0)};
    int n = 0;
    // z - S < i step <= z
    int lo = max(0, floordiv(z - S, step) + 1), hi = min(floordiv(z, step), cnt - 1);
    for (int i = lo; i <= hi && n < 4; ++i) c[n++] = make_int2(i, z - i * step);
    // i step > max(z, z + N - S)
    lo = max(hi + 1, floordiv(max(z, z + N - S), step) + 1);
    for (int i = max(0, lo); i < cnt && n < 4; ++i) c[n++] = make_int2(i, z - i * step + N);
    for (int i = 0; i < 4; ++i) out[(int64_t)k * 4 + i] = c[i];
}

// Boxes covering a Fourier bin, per level and axis: cand + (cand_off[a] + k) * 4
// lists the at most 4 (lattice index, support element) pairs of shifted index k,
// closed by a pair (-1, 0); made with the plan (no divisions in the kernel).
struct GatherLevel {
    int cnt[3], S[3];
    int64_t cand_off[3];
    int64_t lat_off;
    int box0;
    int64_t c0;
    int P;
};

struct GatherArgs {
    int nd, levels;
    int N[3];
    GatherLevel lv[8];
    const int32_t *lattice;
    const int2 *cand;
    const double2 *contrib;
    const double *ssq;   // divide by sum g^2 (adjoint) when not NULL
    int fourier_out;     // write the shifted spectrum directly
    double out_scale;    // 1/sqrt(prod N)
    double2 *out;        // fourier_out: shifted order; else ifftshifted FFT input
};

// Deterministic synthesis gather: every Fourier bin sums the contributions of
// the boxes whose periodic support covers it, level by level in lattice order.
__global__ void __launch_bounds__(THREADS) synth_gather_kernel(GatherArgs A) {
    int64_t prodN = 1;
    for (int a = 0; a < A.nd; ++a) prodN *= A.N[a];
    const int64_t kf = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (kf >= prodN) return;
    int k[3] = {0, 0, 0};
    {
        int64_t rem = kf;
        for (int a = A.nd - 1; a >= 0; --a) {
            k[a] = (int)(rem % A.N[a]);
            rem /= A.N[a];
        }
    }
    double sr = 0.0, si = 0.0;
    for (int l = 0; l < A.levels; ++l) {
        const GatherLevel &G = A.lv[l];
        const int2 *c0 = A.cand + (G.cand_off[0] + k[0]) * 4;
        const int2 *c1 = A.cand + (G.cand_off[1] + k[1]) * 4, *c2 = A.cand + (G.cand_off[2] + k[2]) * 4;
#pragma unroll 1
        for (int i0 = 0; i0 < 4; ++i0) {
            const int2 q0 = __ldg(c0 + i0);
            if (q0.x < 0) break;
#pragma unroll 1
            for (int i1 = 0; i1 < 4; ++i1) {
                const int2 q1 = A.nd > 1 ? __ldg(c1 + i1) : make_int2(i1 ? -1 : 0, 0);
                if (q1.x < 0) break;
#pragma unroll 1
                for (int i2 = 0; i2 < 4; ++i2) {
                    const int2 q2 = A.nd > 2 ? __ldg(c2 + i2) : make_int2(i2 ? -1 : 0, 0);
                    if (q2.x < 0) break;
                    const int64_t li = ((int64_t)q0.x * G.cnt[1] + q1.x) * G.cnt[2] + q2.x;
                    const int box = __ldg(A.lattice + G.lat_off + li);
                    if (box < 0) continue;
                    const int e = (q0.y * G.S[1] + q1.y) * G.S[2] + q2.y;
                    const double2 v = __ldg(A.contrib + G.c0 + (int64_t)(box - G.box0) * G.P + e);
                    sr += v.x;
                    si += v.y;
                }
            }
        }
    }
    if (A.ssq) {
        const double s = A.ssq[kf];
        sr /= s;
        si /= s;
    }
    if (A.fourier_out) {
        A.out[kf] = make_double2(sr, si);
    } else {
        int64_t uf = 0;
        for (int a = 0; a < A.nd; ++a) uf = uf * A.N[a] + imod(k[a] + A.N[a] / 2, A.N[a]);
        A.out[uf] = make_double2(sr * A.out_scale, si * A.out_scale);
    }
}

__global__ void real_part_kernel(const double2 *in, int64_t n, double *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i].x;
}

__global__ void copy_complex_kernel(const double2 *in, int64_t n, double2 *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

struct WsLayout {
    size_t spec, contrib, fftwork, total;
};

WsLayout ws_layout(const msgb_mswpt *p) {
    WsLayout w{};
    size_t o = 0;
    w.spec = o;
    o = a256(o + sizeof(double2) * (size_t)p->prodN);
    w.contrib = o;
    o = a256(o + sizeof(double2) * (size_t)p->total);
    w.fftwork = o;
    o = a256(o + p->fft_work);
    w.total = o;
    return w;
}

int cufft_fail(const char *what, cufftResult r) { return fail(MSGB_ERR_CUDA, "%s: cuFFT error %d", what, (int)r); }

int smem_attr(const void *fn, size_t bytes) {
    if (bytes > 227 * 1024) return fail(MSGB_ERR_UNSUPPORTED, "box support too large for shared memory");
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(MSGB_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return MSGB_OK;
}

}  // namespace
}  // namespace msgb

using namespace msgb;

extern "C" int msgb_mswpt_create(const msgb_mswpt_desc *d, msgb_mswpt **out) {
    if (!d || !out) return fail(MSGB_ERR_ARG, "msgb_mswpt_create: NULL argument");
    *out = nullptr;
    if (d->ndim < 1 || d->ndim > 3) return fail(MSGB_ERR_ARG, "ndim must be 1, 2 or 3");
    if (d->num_levels < 1 || d->num_levels > 8) return fail(MSGB_ERR_UNSUPPORTED, "1..8 levels supported");
    if (d->redundancy != 1 && d->redundancy != 2) return fail(MSGB_ERR_ARG, "redundancy must be 1 or 2");
    auto *p = new msgb_mswpt();
    p->nd = d->ndim;
    p->red = d->redundancy;
    p->levels = d->num_levels;
    p->nbox = d->total_boxes;
    p->prodN = 1;
    for (int a = 0; a < 3; ++a) {
        p->N[a] = a < d->ndim ? d->N[a] : 1;
        p->aspect[a] = a < d->ndim ? d->aspect[a] : 1;
        if (a < d->ndim && (p->N[a] <= 0 || p->N[a] % 2)) {
            delete p;
            return fail(MSGB_ERR_ARG, "N must be positive and even");
        }
        p->prodN *= p->N[a];
    }
    p->half_prodN = p->prodN / p->N[p->nd - 1] * (p->N[p->nd - 1] / 2 + 1);
    const int L = d->num_levels, nd = d->ndim;
    p->bl.assign(d->box_length, d->box_length + L);
    p->bshape.assign(d->box_shape, d->box_shape + L * nd);
    p->ccum.assign(d->coeffs_cumsum, d->coeffs_cumsum + L + 1);
    p->bcum.assign(d->boxes_cumsum, d->boxes_cumsum + L + 1);
    p->lat_cnt.assign(d->lattice_counts, d->lattice_counts + L * nd);
    p->lat_first.assign(d->lattice_first, d->lattice_first + L * nd);
    p->lat_step.assign(d->lattice_step, d->lattice_step + L * nd);
    p->lat_off.assign(d->lattice_offset, d->lattice_offset + L);
    p->goff.assign(d->gfilt_offset, d->gfilt_offset + L);
    p->total = p->ccum[L];
    p->max_patch = 1;
    int64_t gsize = 0, latsize = 0;
    for (int l = 0; l < L; ++l) {
        int P = 1, lat = 1;
        for (int a = 0; a < nd; ++a) {
            const int S = 2 * p->bshape[l * nd + a];
            if (S & (S - 1)) {
                delete p;
                return fail(MSGB_ERR_UNSUPPORTED, "box supports must be powers of two (got %d)", S);
            }
            P *= S;
            lat *= p->lat_cnt[l * nd + a];
        }
        if (P > p->max_patch) p->max_patch = P;
        gsize = p->goff[l] + P > gsize ? p->goff[l] + P : gsize;
        latsize = p->lat_off[l] + lat > latsize ? p->lat_off[l] + lat : latsize;
    }
    cudaError_t e = cudaSuccess;
    auto up = [&](void **dst, const void *src, size_t bytes) {
        if (e != cudaSuccess) return;
        e = cudaMalloc(dst, bytes > 0 ? bytes : 1);
        if (e == cudaSuccess && bytes) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
    };
    up((void **)&p->d_centres, d->centres, sizeof(int32_t) * p->nbox * nd);
    up((void **)&p->d_lattice, d->lattice_box, sizeof(int32_t) * latsize);
    up((void **)&p->d_gfilt, d->gfilt, sizeof(double) * gsize);
    up((void **)&p->d_ssq, d->sum_gsquare, sizeof(double) * p->prodN);
    up((void **)&p->d_ccum, d->coeffs_cumsum, sizeof(int64_t) * (L + 1));
    up((void **)&p->d_bcum, d->boxes_cumsum, sizeof(int32_t) * (L + 1));
    up((void **)&p->d_bl, d->box_length, sizeof(int32_t) * L);
    up((void **)&p->d_bshape, d->box_shape, sizeof(int32_t) * L * nd);
    if (e != cudaSuccess) {
        msgb_mswpt_destroy(p);
        return fail(MSGB_ERR_CUDA, "msgb_mswpt_create: %s", cudaGetErrorString(e));
    }
    for (int l = 0; l < L; ++l)
        for (int a = 0; a < nd; ++a) p->tw_n = 2 * p->bshape[l * nd + a] > p->tw_n ? 2 * p->bshape[l * nd + a] : p->tw_n;
    std::vector<double> tw(2 * (size_t)p->tw_n);
    for (int m = 0; m < p->tw_n; ++m) {
        // from the first octant: exact at the multiples of a quarter turn
        const int q = (int)((8LL * m) / p->tw_n);  // octant
        double c, s;
        if ((4LL * m) % p->tw_n == 0) {
            const int k = (int)((4LL * m) / p->tw_n);
            c = k == 0 ? 1.0 : (k == 2 ? -1.0 : 0.0);
            s = k == 1 ? 1.0 : (k == 3 ? -1.0 : 0.0);
        } else {
            const double e = 2.0 * 3.14159265358979323846 / p->tw_n;  // angle from the nearest quarter turn
            const int k = (q + 1) / 2;                                // quarter turns
            const double b = e * (m - (double)k * p->tw_n / 4.0);
            const double cb = cos(b), sb = sin(b);
            c = k % 4 == 0 ? cb : (k % 4 == 1 ? -sb : (k % 4 == 2 ? -cb : sb));
            s = k % 4 == 0 ? sb : (k % 4 == 1 ? cb : (k % 4 == 2 ? -sb : -cb));
        }
        tw[2 * m] = c;
        tw[2 * m + 1] = s;
    }
    int64_t cand = 0;
    p->cand_off.assign((size_t)L * 3, 0);
    for (int l = 0; l < L; ++l)
        for (int a = 0; a < nd; ++a) {
            p->cand_off[l * 3 + a] = cand;
            cand += p->N[a];
        }
    if (e == cudaSuccess) e = cudaMalloc((void **)&p->d_cand, sizeof(int2) * 4 * (size_t)cand);
    for (int l = 0; l < L && e == cudaSuccess; ++l)
        for (int a = 0; a < nd; ++a)
            candidates_kernel<<<(p->N[a] + THREADS - 1) / THREADS, THREADS>>>(
                p->N[a], 2 * p->bshape[l * nd + a], p->lat_step[l * nd + a], p->lat_cnt[l * nd + a],
                p->lat_first[l * nd + a], p->d_cand + p->cand_off[l * 3 + a] * 4);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // ready for any stream
    up((void **)&p->d_tw, tw.data(), sizeof(double) * tw.size());
    if (e != cudaSuccess) {
        msgb_mswpt_destroy(p);
        return fail(MSGB_ERR_CUDA, "msgb_mswpt_create: %s", cudaGetErrorString(e));
    }
    int n[3] = {p->N[0], p->N[1], p->N[2]};
    size_t w1 = 0, w2 = 0;
    cufftResult r = cufftCreate(&p->plan_d2z);
    if (r == CUFFT_SUCCESS) r = cufftSetAutoAllocation(p->plan_d2z, 0);
    if (r == CUFFT_SUCCESS) r = cufftMakePlanMany(p->plan_d2z, nd, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_D2Z, 1, &w1);
    if (r == CUFFT_SUCCESS) r = cufftCreate(&p->plan_z2z);
    if (r == CUFFT_SUCCESS) r = cufftSetAutoAllocation(p->plan_z2z, 0);
    if (r == CUFFT_SUCCESS) r = cufftMakePlanMany(p->plan_z2z, nd, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_Z2Z, 1, &w2);
    if (r != CUFFT_SUCCESS) {
        msgb_mswpt_destroy(p);
        return cufft_fail("msgb_mswpt_create", r);
    }
    p->fft_work = w1 > w2 ? w1 : w2;
    *out = p;
    return MSGB_OK;
}

extern "C" int msgb_mswpt_destroy(msgb_mswpt *p) {
    if (!p) return MSGB_OK;
    cudaFree(p->d_centres);
    cudaFree(p->d_lattice);
    cudaFree(p->d_gfilt);
    cudaFree(p->d_ssq);
    cudaFree(p->d_ccum);
    cudaFree(p->d_bcum);
    cudaFree(p->d_bl);
    cudaFree(p->d_bshape);
    cudaFree(p->d_tw);
    cudaFree(p->d_cand);
    if (p->plan_d2z) cufftDestroy(p->plan_d2z);
    if (p->plan_z2z) cufftDestroy(p->plan_z2z);
    delete p;
    return MSGB_OK;
}

extern "C" int64_t msgb_mswpt_total_coeffs(const msgb_mswpt *p) { return p ? p->total : -1; }

extern "C" size_t msgb_mswpt_workspace_size(const msgb_mswpt *p) { return p ? ws_layout(p).total : 0; }

static int check_ws(const msgb_mswpt *p, void *ws, size_t bytes) {
    if (!ws || bytes < ws_layout(p).total)
        return fail(MSGB_ERR_WORKSPACE, "MSWPT workspace too small: need %zu, got %zu", ws_layout(p).total, bytes);
    if (((uintptr_t)ws & 255) != 0) return fail(MSGB_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    return MSGB_OK;
}

extern "C" int msgb_mswpt_forward(const msgb_mswpt *p, const double *in, int is_complex, int input_is_fourier,
                                  double scale, int apply_half_mask, double *coeffs, double *keys, void *workspace,
                                  size_t workspace_bytes, msgb_stream_t stream) {
    if (!p || !in || !coeffs) return fail(MSGB_ERR_ARG, "msgb_mswpt_forward: NULL argument");
    if (input_is_fourier && !is_complex) return fail(MSGB_ERR_ARG, "Fourier input must be complex");
    if (int e = check_ws(p, workspace, workspace_bytes)) return e;
    cudaStream_t st = as_stream(stream);
    const WsLayout w = ws_layout(p);
    char *ws = (char *)workspace;
    double2 *spec = (double2 *)(ws + w.spec);
    FwdArgs A{};
    A.half = 0;
    A.shifted = 0;
    A.in_scale = 1.0 / sqrt((double)p->prodN);
    if (input_is_fourier) {
        A.X = (const double2 *)in;
        A.shifted = 1;
        A.in_scale = 1.0;
    } else {
        cufftHandle h = is_complex ? p->plan_z2z : p->plan_d2z;
        cufftResult r = cufftSetStream(h, st);
        if (r == CUFFT_SUCCESS) r = cufftSetWorkArea(h, ws + w.fftwork);
        if (r == CUFFT_SUCCESS) {
            if (is_complex)
                r = cufftExecZ2Z(h, (cufftDoubleComplex *)in, (cufftDoubleComplex *)spec, CUFFT_FORWARD);
            else
                r = cufftExecD2Z(h, (cufftDoubleReal *)in, (cufftDoubleComplex *)spec);
        }
        if (r != CUFFT_SUCCESS) return cufft_fail("msgb_mswpt_forward", r);
        A.X = spec;
        A.half = is_complex ? 0 : 1;
    }
    A.ssq = p->d_ssq;
    A.centres = p->d_centres;
    A.scale = scale;
    A.half_mask = apply_half_mask;
    A.coeffs = (double2 *)coeffs;
    A.keys = keys;
    AllLevels LV;
    const int blocks = all_levels(p, LV);
    size_t smem = 0;
    for (int l = 0; l < LV.levels; ++l) smem = box_smem(LV.lv[l]) > smem ? box_smem(LV.lv[l]) : smem;
    if (int e = smem_attr((const void *)box_forward_kernel, smem)) return e;
    box_forward_kernel<<<blocks, THREADS, smem, st>>>(LV, A);
    return check_launch("msgb_mswpt_forward");
}

// Synthesis.  With W = (per box) unitary_ifft o roll(+r_fwd) o (g *) o extract
// o (/ sum g^2) o unitary_fft, the Hermitian adjoint is
//   W^H c = unitary_ifft( (1/sum g^2) * sum_boxes scatter( g * roll(unitary_fft(c_box), -r_fwd) ) ),
// which is MSWPT.inverse with the forward's roll convention and one extra
// division by sum g^2 (unitary_ifft^H = unitary_fft, roll^H = roll back,
// extract^H = periodic scatter-add; g and sum g^2 are real).
extern "C" int msgb_mswpt_synthesis(const msgb_mswpt *p, const double *coeffs, int mode, int real_output, double *out,
                                    void *workspace, size_t workspace_bytes, msgb_stream_t stream) {
    if (!p || !coeffs || !out) return fail(MSGB_ERR_ARG, "msgb_mswpt_synthesis: NULL argument");
    if (int e = check_ws(p, workspace, workspace_bytes)) return e;
    const int adjoint = mode & 1, fourier_out = (mode >> 1) & 1;
    cudaStream_t st = as_stream(stream);
    const WsLayout w = ws_layout(p);
    char *ws = (char *)workspace;
    double2 *spec = (double2 *)(ws + w.spec);
    double2 *contrib = (double2 *)(ws + w.contrib);
    SynArgs A{};
    A.coeffs = (const double2 *)coeffs;
    A.centres = p->d_centres;
    A.adjoint = adjoint;
    A.contrib = contrib;
    AllLevels LV;
    const int box_blocks = all_levels(p, LV);
    size_t smem = 0;
    for (int l = 0; l < LV.levels; ++l) smem = box_smem(LV.lv[l]) > smem ? box_smem(LV.lv[l]) : smem;
    if (int e = smem_attr((const void *)box_synth_kernel, smem)) return e;
    box_synth_kernel<<<box_blocks, THREADS, smem, st>>>(LV, A);
    GatherArgs G{};
    G.nd = p->nd;
    G.levels = p->levels;
    for (int a = 0; a < 3; ++a) G.N[a] = p->N[a];
    for (int l = 0; l < p->levels; ++l) {
        GatherLevel &gl = G.lv[l];
        gl.P = 1;
        for (int a = 0; a < 3; ++a) {
            const bool in = a < p->nd;
            gl.cnt[a] = in ? p->lat_cnt[l * p->nd + a] : 1;
            gl.cand_off[a] = in ? p->cand_off[l * 3 + a] : 0;
            gl.S[a] = in ? 2 * p->bshape[l * p->nd + a] : 1;
            gl.P *= gl.S[a];
        }
        gl.lat_off = p->lat_off[l];
        gl.box0 = p->bcum[l];
        gl.c0 = p->ccum[l];
    }
    G.lattice = p->d_lattice;
    G.cand = p->d_cand;
    G.contrib = contrib;
    G.ssq = adjoint ? p->d_ssq : nullptr;
    G.fourier_out = fourier_out;
    G.out_scale = 1.0 / sqrt((double)p->prodN);
    G.out = (fourier_out && !real_output) ? (double2 *)out : spec;
    const unsigned blocks = (unsigned)((p->prodN + THREADS - 1) / THREADS);
    synth_gather_kernel<<<blocks, THREADS, 0, st>>>(G);
    if (int e = check_launch("msgb_mswpt_synthesis gather")) return e;
    if (!fourier_out) {
        cufftHandle h = p->plan_z2z;
        cufftResult r = cufftSetStream(h, st);
        if (r == CUFFT_SUCCESS) r = cufftSetWorkArea(h, ws + w.fftwork);
        if (r == CUFFT_SUCCESS) r = cufftExecZ2Z(h, (cufftDoubleComplex *)spec, (cufftDoubleComplex *)spec, CUFFT_INVERSE);
        if (r != CUFFT_SUCCESS) return cufft_fail("msgb_mswpt_synthesis", r);
        if (real_output)
            real_part_kernel<<<blocks, THREADS, 0, st>>>(spec, p->prodN, out);
        else
            copy_complex_kernel<<<blocks, THREADS, 0, st>>>(spec, p->prodN, (double2 *)out);
    } else if (real_output) {
        real_part_kernel<<<blocks, THREADS, 0, st>>>(spec, p->prodN, out);
    }
    return check_launch("msgb_mswpt_synthesis");
}

namespace msgb {
struct PlanView {
    int nd, red, levels;
    int N[3], aspect[3];
    int64_t ccum[9];
    int bcum[9];
    int bl[8];
    int bshape[8][3];
    const int32_t *centres;
};

int plan_view(const msgb_mswpt *p, PlanView &v) {
    if (!p) return fail(MSGB_ERR_ARG, "NULL MSWPT plan");
    v.nd = p->nd;
    v.red = p->red;
    v.levels = p->levels;
    for (int a = 0; a < 3; ++a) {
        v.N[a] = p->N[a];
        v.aspect[a] = p->aspect[a];
    }
    for (int l = 0; l <= p->levels; ++l) {
        v.ccum[l] = p->ccum[l];
        v.bcum[l] = p->bcum[l];
    }
    for (int l = 0; l < p->levels; ++l) {
        v.bl[l] = p->bl[l];
        for (int a = 0; a < 3; ++a) v.bshape[l][a] = a < p->nd ? p->bshape[l * p->nd + a] : 1;
    }
    v.centres = p->d_centres;
    return MSGB_OK;
}
}  // namespace msgb
