// mfree.cu -- matrix-free projector / backprojector pairs (parallel beam and
// fan beam) and SIRT on them (include/fair_mf.h).
//
// Geometry of paralleltomo (system_generation.f90:309-492): ray (angle i,
// bin j) is the line with unit normal n_i = (cos th_i, sin th_i) at offset
// x0_j = j - (p-1)/2 (linspace(-(p-1)/2, (p-1)/2, p), unit bins), direction
// (-sin, cos). Pixel (ix, iy) (ix from the left, iy from the bottom, both
// 0..N-1) is the unit square centred at (ix + 1/2 - N/2, iy + 1/2 - N/2) and
// is column ix*N + (N-1-iy) of the matrix (JA = floor(xm)*N + (N - floor(ym))).
//
// The ray's length inside a unit square is a function of the signed distance
// d between the square's centre and the line (the chord of a unit square):
// with c = max(|cos|, |sin|), s = min(...):
//   L = 1/c                      for |d| <= (c - s)/2,
//   L = ((c + s)/2 - |d|)/(c s)  for (c - s)/2 < |d| < (c + s)/2,  else 0,
// which is the segment length the ray tracer measures between consecutive
// crossings; segments of 1e-10 or less are dropped, as there. An axis-aligned
// ray on a grid line (s = 0, |d| = 1/2) belongs to the pixel on the positive
// side, as the reference's floor-of-midpoint rule gives.
//
// d = ix*cos + iy*sin + K_i - j with K_i = (1/2 - N/2)(cos + sin) + (p-1)/2,
// evaluated in 64-bit fixed point with 46 fractional bits (N <= 8192 and
// p <= 16384 keep every term below 2^60): exact integer
// arithmetic, so every kernel computes bit-identical entries whatever the
// order it meets the (ray, pixel) pairs in. The projector walks the image
// along each ray's faster axis (per column when |sin| >= |cos|, else per row);
// at each step the only pixels within H2 of the ray are the two that bracket
// its crossing, which the walk tracks exactly with one 64-bit add per step
// (FP32: a warp walks 32 adjacent rays in step; FP64: a thread a ray). The
// backprojector evaluates, per pixel and angle, the two rays whose offsets
// bracket the pixel's (FP32: tiles of 32 x 32 pixels, their bins staged in
// shared memory; FP64: a thread per 4 pixels of a column). Both keep only pairs
// with L > 0, so they sum the same entries: an exact adjoint pair,
// deterministic, without atomics.
//
// Fan beam (fanlineartomo, system_generation.f90:79-307): ray (i, j) is the
// line through the rotated source P_i with direction u_ij = R(omega_j) u0_i,
// computed on the host exactly as the reference does (cos/sin of the bin
// angles, the same products and sums). Its unit normal n = (b, -a)/|u| and
// K_ij = n . ((1/2 - N/2, 1/2 - N/2) - P_i) give d = ix*n_x + iy*n_y + K_ij,
// the same fixed-point form, one record per ray. The projector walks each ray
// as above (and the rays that walk image rows read a transposed copy of x, so
// that a warp's rays gather adjacent addresses); the backprojector stages, per
// tile and angle, the rays whose bin angles the tile can see from the source
// (the reference's odd-p angles are not monotone in j: they are sorted once),
// and every pixel tests those within its own window with the exact distance.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "fair_internal.cuh"
#include "fair_mf.h"
#include "sirt_epi.cuh"

namespace fair {

namespace {

constexpr int kFix = 46;
constexpr double kOne = 70368744177664.0;  // 2^46

// The first 48 bytes hold what the FP32 backprojector reads per angle (three
// 16-byte loads), the next 32 what FP64 adds.
struct __align__(16) MfAngle {
    long long C, S;      // cos, sin in fixed point
    long long K, H2;     // K_i; (c + s)/2 in fixed point
    int H2s;             // H2 cut to 31 fractional bits (FP32 entries)
    float inv_c;         // 1/c
    float ramp;          // 2^-31 / s (0 on axis-aligned lines)
    int tie;             // s = 0: +1 / -1 = sign of d that keeps |d| = 1/2; 0 otherwise
    long long H1;        // (c - s)/2 in fixed point
    long long Hcut;      // |d| >= Hcut leaves a segment of at most 1e-10: dropped
    double inv_c64, scale_ramp64;
    float Cf, Sf, Kf;    // float copies for the walk's step range
    int by_column;       // 1: walk columns (|sin| >= |cos|)
};
static_assert(sizeof(MfAngle) == 96, "MfAngle layout");

// The fields of record p that a backprojector of entries T reads: the first
// 48 bytes (FP32), or 80 (FP64), by 16-byte loads.
template <typename T>
__device__ __forceinline__ MfAngle mf_load(const MfAngle *p) {
    const int4 *q = reinterpret_cast<const int4 *>(p);
    auto ll = [](int lo, int hi) { return (long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo); };
    MfAngle A;
    const int4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    A.C = ll(a.x, a.y);
    A.S = ll(a.z, a.w);
    A.K = ll(b.x, b.y);
    A.H2 = ll(b.z, b.w);
    A.H2s = c.x;
    A.inv_c = __int_as_float(c.y);
    A.ramp = __int_as_float(c.z);
    A.tie = c.w;
    if constexpr (sizeof(T) == 8) {
        const int4 d = __ldg(q + 3), e = __ldg(q + 4);
        A.H1 = ll(d.x, d.y);
        A.Hcut = ll(d.z, d.w);
        A.inv_c64 = __hiloint2double(e.y, e.x);
        A.scale_ramp64 = __hiloint2double(e.w, e.z);
    }
    return A;
}

template <typename T> struct Chord;
// The chord of a unit pixel at |d| = ad < 2^47 from the line: ramp() for s > 0,
// tied() for an axis-aligned line (s = 0), where tu = H2 when a ray on the
// pixel's edge, on this side of it, keeps the pixel (else -1).
//
// FP32 entries are (1/c) sat((H2 - u) / s), sat() the clamp to [0, 1], on the
// exact distance cut to 31 fractional bits: u = floor(d) for d >= 0 and
// -floor(d) - 1 (a one's complement: no negation, no carry) for d < 0, in units
// of 2^-31. H2 - u is exact in 32 bits, so an entry is one integer subtraction,
// one conversion and one saturated multiply-add (an axis-aligned ray has ramp 0
// and its entry, 0 or 1, as the addend); the cut of segments below 1e-10 is left
// to the FP64 entries. Every kernel evaluates the same expression on the same
// exact value, so they agree bit for bit.
template <> struct Chord<double> {
    static __device__ __forceinline__ double ramp(const MfAngle &A, long long ad) {
        const double w = ad <= A.H1 ? A.inv_c64 : (double)(A.H2 - ad) * A.scale_ramp64;
        return ad < A.Hcut ? w : 0.0;
    }
    static __device__ __forceinline__ double tied(const MfAngle &A, long long ad, long long tu) {
        return ad < A.H2 || ad == tu ? A.inv_c64 : 0.0;
    }
};

// ---- epilogues of the projector (per ray) and backprojector (per pixel) ---------
template <typename T> struct EpiStore {  // y = A x (or A' r)
    T *y;
    __device__ void operator()(int64_t i, T acc) const { y[i] = acc; }
};
struct EpiCimminoW {  // M = m * sum_j a_ij^2 (the sum arrives in acc)
    double *M;
    double m;
    __device__ void operator()(int64_t i, double acc) const { M[i] = m * acc; }
};

// One entry a_rq = w of a pass (valid: pixel q exists): MODE 0 adds w * v_q
// (v read only for w > 0, as a stored matrix reads only its entries), MODE 1
// adds w, MODE 2 w^2, MODE 3 counts w > 0.
template <typename VT, typename ACC, int MODE>
__device__ __forceinline__ void mf_add(ACC &acc, ACC w, bool valid, const VT *__restrict__ v,
                                       int64_t q) {
    if (MODE == 0) {
        const ACC vq = valid && w > (ACC)0 ? (ACC)__ldg(v + q) : (ACC)0;
        acc += w * vq;
    } else if (MODE == 1) {
        acc += valid ? w : (ACC)0;
    } else if (MODE == 2) {
        acc += valid ? w * w : (ACC)0;
    } else {
        acc += valid && w > (ACC)0 ? (ACC)1 : (ACC)0;
    }
}

// The steps of one ray (see k_mf_project): E = |d| at pixel ua, Qa - E at
// ua + 1; a step lowers E by Fw and moves ua down by one when E leaves
// [0, Qa). TIE: an axis-aligned ray (tied chords). Two steps per iteration,
// so that their gathers are in flight together.
template <typename XT, typename ACC, int MODE, bool TIE>
__device__ __forceinline__ ACC mf_walk(const MfAngle &A, long long E, int ua, long long Qa,
                                       long long Fw, const XT *__restrict__ xv, int qt, int su,
                                       int dqt, int N, int cnt, long long tua, long long tub) {
    ACC acc = 0;
    auto step = [&](ACC &wa, ACC &wb, int &qa, bool &va, bool &vb) {
        if constexpr (TIE) {
            wa = Chord<ACC>::tied(A, E, tua);
            wb = Chord<ACC>::tied(A, Qa - E, tub);
        } else {
            wa = Chord<ACC>::ramp(A, E);
            wb = Chord<ACC>::ramp(A, Qa - E);
        }
        qa = qt + ua * su;
        va = (unsigned)ua < (unsigned)N;
        vb = (unsigned)(ua + 1) < (unsigned)N;
        E -= Fw;
        if (E < 0) {
            --ua;
            E += Qa;
        }
        qt += dqt;
    };
    for (; cnt >= 2; cnt -= 2) {
        ACC w0, w1, w2, w3;
        int q0, q1;
        bool v0, v1, v2, v3;
        step(w0, w1, q0, v0, v1);
        step(w2, w3, q1, v2, v3);
        mf_add<XT, ACC, MODE>(acc, w0, v0, xv, q0);
        mf_add<XT, ACC, MODE>(acc, w1, v1, xv, q0 + su);
        mf_add<XT, ACC, MODE>(acc, w2, v2, xv, q1);
        mf_add<XT, ACC, MODE>(acc, w3, v3, xv, q1 + su);
    }
    if (cnt > 0) {
        ACC w0, w1;
        int q0;
        bool v0, v1;
        step(w0, w1, q0, v0, v1);
        mf_add<XT, ACC, MODE>(acc, w0, v0, xv, q0);
        mf_add<XT, ACC, MODE>(acc, w1, v1, xv, q0 + su);
    }
    return acc;
}

// Per ray r: MODE 0 sums a_rj * x_j, MODE 1 sums a_rj, MODE 2 sums a_rj^2,
// MODE 3 counts the pixels with a_rj > 0 (x unused for MODE 1-3).
// FAN: ang holds one record per ray (K its own offset), else one per angle
// (ray j of angle i at offset K - j).
//
// The ray walks its faster axis t (|F| <= |Q|): with g = sign(Q) d =
// t Fp + u Qa + Gk, the pixels u of step t with |d| <= H2 (< Qa) lie within
// one pixel of u* = -(t Fp + Gk)/Qa, so they are ua = floor(u*) and ua + 1,
// at |d| = -g(t, ua) in [0, Qa) and Qa - that. The walk keeps ua and that
// distance exactly: a step changes g by |Fp| (the walk runs in the direction
// that makes the change non-negative). Only steps whose candidates can lie
// in the image are walked (a float bound, widened).
//
// x is read as x[ix*N + N-1-iy] by the rays that walk columns (a warp's
// adjacent rays then gather adjacent pixels of one column) and as its
// transpose xt[(N-1-iy)*N + ix] by those that walk rows (adjacent pixels of
// one row).
template <typename XT, typename ACC, int MODE, bool FAN, class Epi>
__global__ void __launch_bounds__(128) k_mf_project(const MfAngle *__restrict__ ang, int nth,
                                                    int p, int N, const XT *__restrict__ x,
                                                    const XT *__restrict__ xt, Epi epi) {
    const int64_t m = (int64_t)nth * p;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m;
         r += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(r / p), j = (int)(r - (int64_t)i * p);
        const MfAngle &A = ang[FAN ? r : i];
        const long long K = FAN ? A.K : A.K - ((long long)j << kFix);
        const float Kf = FAN ? A.Kf : A.Kf - (float)j;
        const bool col = A.by_column != 0;
        const long long F = col ? A.C : A.S, Q = col ? A.S : A.C;
        const float Ff = col ? A.Cf : A.Sf, Qf = col ? A.Sf : A.Cf;
        const int sq = Q > 0 ? 1 : -1;
        const long long Qa = Q > 0 ? Q : -Q, Fp = sq * F, Gk = sq * K;
        const float Qaf = fabsf(Qf), Fpf = sq * Ff, Gkf = sq * Kf;
        // steps with u* in [-1, N): -N Qa < t Fp + Gk <= Qa (widened by 0.05)
        const float lo = -(float)N * Qaf - 0.05f - Gkf, hi = Qaf + 0.05f - Gkf;
        float ta = 0.f, tb = (float)(N - 1);
        if (Fpf > 0.f) {
            ta = fmaxf(ta, lo / Fpf);
            tb = fminf(tb, hi / Fpf);
        } else if (Fpf < 0.f) {
            ta = fmaxf(ta, hi / Fpf);
            tb = fminf(tb, lo / Fpf);
        } else if (!(lo < 0.f && hi >= 0.f)) {
            tb = -1.f;
        }
        const int t0 = max(0, (int)floorf(ta)), t1 = min(N - 1, (int)ceilf(tb));
        ACC acc = 0;
        if (t0 <= t1) {
            const int dir = Fp >= 0 ? 1 : -1;
            const long long Fw = Fp >= 0 ? Fp : -Fp;
            const int ts = dir > 0 ? t0 : t1;
            const long long G = (long long)ts * Fp + Gk;
            int ua = (int)floorf(-(float)G / (float)Qa);
            long long e = G + (long long)ua * Qa;
            while (e > 0) { --ua; e -= Qa; }
            while (e <= -Qa) { ++ua; e += Qa; }
            // pixel (t, u): element qt + u su of xv
            const XT *__restrict__ xv = col ? x : xt;
            const int su = col ? -1 : 1, dqt = col ? dir * N : -dir * N;
            const int qt = col ? ts * N + N - 1 : (N - 1 - ts) * N;
            if (A.tie != 0) {
                // d at ua is sign(Q) e <= 0, at ua + 1 sign(Q) (e + Qa) > 0
                const long long tua = A.tie == -sq ? A.H2 : -1, tub = A.tie == sq ? A.H2 : -1;
                acc = mf_walk<XT, ACC, MODE, true>(A, -e, ua, Qa, Fw, xv, qt, su, dqt, N,
                                                   t1 - t0 + 1, tua, tub);
            } else {
                acc = mf_walk<XT, ACC, MODE, false>(A, -e, ua, Qa, Fw, xv, qt, su, dqt, N,
                                                    t1 - t0 + 1, -1, -1);
            }
        }
        epi(r, acc);
    }
}

// xt = the transpose of x viewed as an N x N array (32 x 32 tiles through
// shared memory, both sides coalesced). *flag becomes 1 if x holds an Inf or NaN, for
// the projector behind it; the FP32 backprojectors take it back, so that an iteration,
// run or replayed from a graph, leaves nothing behind (a product of its own is
// followed by a copy of 0, mf_apply).
template <typename T>
__global__ void __launch_bounds__(256) k_mf_transpose(const T *__restrict__ x, T *__restrict__ xt,
                                                      int N, unsigned *flag) {
    __shared__ T tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        if (r < N && c < N) {
            const T v = x[(int64_t)r * N + c];
            tile[k][threadIdx.x] = v;
            if (sizeof(T) == 4 && !isfinite(v)) *flag = 1u;
        }
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int r = c0 + k, c = r0 + threadIdx.x;
        if (r < N && c < N) xt[(int64_t)r * N + c] = tile[threadIdx.x][k];
    }
}

// FP32 projector. A warp takes 32 adjacent rays of one angle and walks their
// image columns (or rows) in step, over the union of the rays' ranges, so that
// its lanes always gather neighbouring pixels. A ray's distance at its lower
// candidate, E in [0, Qa), is kept in units of 2^-63: the high word is the
// entry's u, and one 64-bit add forms H2 - u of the upper candidate (Cb + E).
// (sq = 1: the lower candidate lies at d = -E, and E - 1 is kept, whose high
// word is the one's complement rule's u; E = 0 is then the upper candidate of
// the pixel below, at d = 0.) Steps on which both candidates of all 32 rays
// lie in the image -- nearly all -- run without bounds checks, and without the
// test for entries 0 when x is finite (0 x adds nothing); the ends, and any x
// with Inf or NaN, take the checked step, which reads x only at positive
// entries, as a stored matrix does.
// Bound by integer issue. N = 1024, 720 angles, 1448 bins: 1.23 ms with every
// ray walking from its own start (47 instructions and 12 L1 wavefronts per warp
// step) -> 0.59 ms (25 and 3); fan beam N = 512, 720 angles: 0.33 -> 0.21 ms.
// Eight steps' loads in flight and 7 blocks per SM: 592 us, four 608 (8 blocks)
// and 643 (9); the checked steps one at a time cost another 110 us.
// Qa is 2^63 where a ray is that close to an axis without lying on it (|sin| or
// |cos| rounded to 1, an angle held in FP32 such as pi/2): E + Qa and Cb + E are
// sums modulo 2^64.
constexpr int kWalkUnroll = 8;  // interior steps whose loads are in flight together
struct Walk32 {
    long long E, Fw;          // E (see above); what a step takes off it
    unsigned long long Qa, Cb;  // Qa; the upper candidate's constant
    int H2s;
    float ramp, aa, ab;       // entry = sat((H2s - u) ramp + a)
    int ua;
};
template <bool COL>
__device__ __forceinline__ float mf_walk32(Walk32 w, bool on, const float *__restrict__ x, int qt, int dqt,
                                           int N, int steps, int k0, int k1) {
    constexpr int su = COL ? -1 : 1;
    float s0 = 0.f, s1 = 0.f;
    auto entries = [&](float &wa, float &wb) {
        wa = __saturatef(fmaf((float)(w.H2s - (int)(w.E >> 32)), w.ramp, w.aa));
        wb = __saturatef(fmaf((float)(int)((w.Cb + (unsigned long long)w.E) >> 32), w.ramp, w.ab));
    };
    auto advance = [&] {
        w.E -= w.Fw;
        if (w.E < 0) {
            w.E = (long long)((unsigned long long)w.E + w.Qa);
            --w.ua;
        }
        qt += dqt;
    };
    auto checked = [&](int n) {  // four steps' loads in flight together
#pragma unroll 1
        for (; n > 0; n -= 4) {
            float wa[4], wb[4], xa[4], xb[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                entries(wa[t], wb[t]);
                const int q = qt + w.ua * su;
                const bool h = on && t < n;
                xa[t] = h && (unsigned)w.ua < (unsigned)N && wa[t] > 0.f ? __ldg(x + q) : 0.f;
                xb[t] = h && (unsigned)(w.ua + 1) < (unsigned)N && wb[t] > 0.f ? __ldg(x + q + su) : 0.f;
                if (t < n) advance();
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                s0 = fmaf(wa[t], xa[t], s0);
                s1 = fmaf(wb[t], xb[t], s1);
            }
        }
    };
    checked(k0);
    unsigned q = 4u * (unsigned)(qt + w.ua * su);
    const unsigned dq = 4u * (unsigned)dqt;
    const char *xc = reinterpret_cast<const char *>(x);
#pragma unroll kWalkUnroll
    for (int n = k1 - k0; n > 0; --n) {
        float wa, wb;
        entries(wa, wb);
        const float *px = reinterpret_cast<const float *>(xc + q);
        s0 = fmaf(wa, __ldg(px), s0);
        s1 = fmaf(wb, __ldg(px + su), s1);
        w.E -= w.Fw;
        q += dq;
        if (w.E < 0) {
            w.E = (long long)((unsigned long long)w.E + w.Qa);
            q -= 4u * (unsigned)su;
        }
    }
    qt += (k1 - k0) * dqt;
    w.ua = (((int)q >> 2) - qt) * su;  // (q may be -4 here: one before the image)
    checked(steps - k1);
    return s0 + s1;
}

template <bool FAN, class Epi>
__global__ void __launch_bounds__(128, 7) k_mf_project32(const MfAngle *__restrict__ ang, int nth, int p,
                                                      int N, const float *__restrict__ x,
                                                      const float *__restrict__ xt,
                                                      const unsigned *__restrict__ flag, Epi epi) {
    const int lane = threadIdx.x & 31, wpa = (p + 31) / 32;
    const int64_t nw = (int64_t)nth * wpa;
    const bool guard = *flag != 0;
    for (int64_t g = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); g < nw;
         g += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int i = (int)(g / wpa), j = (int)(g - (int64_t)i * wpa) * 32 + lane;
        const bool ray = j < p;
        const int64_t r = (int64_t)i * p + (ray ? j : p - 1);
        const MfAngle &A = ang[FAN ? r : i];
        const long long K = FAN ? A.K : A.K - ((long long)j << kFix);
        const float Kf = FAN ? A.Kf : A.Kf - (float)j;
        const bool col = A.by_column != 0;
        const long long F = col ? A.C : A.S, Q = col ? A.S : A.C;
        const float Ff = col ? A.Cf : A.Sf, Qf = col ? A.Sf : A.Cf;
        const int sq = Q > 0 ? 1 : -1;
        const long long Qa = Q > 0 ? Q : -Q, Fp = sq * F, Gk = sq * K;
        const float Qaf = fabsf(Qf), Fpf = sq * Ff, Gkf = sq * Kf;
        // steps with u* in [-1, N): -N Qa < t Fp + Gk <= Qa (widened by 0.05)
        const float lo = -(float)N * Qaf - 0.05f - Gkf, hi = Qaf + 0.05f - Gkf;
        float ta = 0.f, tb = (float)(N - 1);
        if (Fpf > 0.f) {
            ta = fmaxf(ta, lo / Fpf);
            tb = fminf(tb, hi / Fpf);
        } else if (Fpf < 0.f) {
            ta = fmaxf(ta, hi / Fpf);
            tb = fminf(tb, lo / Fpf);
        } else if (!(lo < 0.f && hi >= 0.f)) {
            tb = -1.f;
        }
        const int t0 = max(0, (int)floorf(ta)), t1 = min(N - 1, (int)ceilf(tb));
        const bool live = ray && t0 <= t1;
        const bool up = Fp >= 0;
        const int kind = (col ? 2 : 0) + (up ? 1 : 0);  // one per parallel angle, up to four in a fan's warp
        float acc = 0.f;
        unsigned todo = __ballot_sync(0xffffffffu, live);
        while (todo) {
            const int kd = __shfl_sync(0xffffffffu, kind, __ffs(todo) - 1);
            const bool on = live && kind == kd;
            todo &= ~__ballot_sync(0xffffffffu, on);
            const int T0 = __reduce_min_sync(0xffffffffu, on ? t0 : N);
            const int T1 = __reduce_max_sync(0xffffffffu, on ? t1 : -1);
            const bool kup = (kd & 1) != 0, kcol = (kd & 2) != 0;
            const int ts = kup ? T0 : T1, dir = kup ? 1 : -1, steps = T1 - T0 + 1;
            Walk32 w{0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0};
            int k0 = 0, k1 = steps;
            if (on) {
                const long long G = (long long)ts * Fp + Gk, Fw = up ? Fp : -Fp;
                w.ua = (int)floorf(-(float)G / (float)Qa);
                long long e = G + (long long)w.ua * Qa;
                while (e > 0) { --w.ua; e -= Qa; }
                while (e <= -Qa) { ++w.ua; e += Qa; }
                w.E = -e;  // in [0, Qa)
                if (A.tie != 0) {  // Fw = 0: the same two entries on every step
                    const long long tua = A.tie == -sq ? A.H2 : -1, tub = A.tie == sq ? A.H2 : -1;
                    w.aa = w.E < A.H2 || w.E == tua ? 1.f : 0.f;
                    w.ab = Qa - w.E < A.H2 || Qa - w.E == tub ? 1.f : 0.f;
                    w.E = 0;
                } else {
                    w.Qa = (unsigned long long)Qa << 17;
                    w.Fw = Fw << 17;
                    w.E = (w.E << 17) - (sq > 0 ? 1 : 0);
                    if (w.E < 0) {
                        w.E = (long long)((unsigned long long)w.E + w.Qa);
                        --w.ua;
                    }
                    w.H2s = A.H2s;
                    w.ramp = A.ramp;
                    w.Cb = (((unsigned long long)(unsigned)A.H2s << 32) | 0xFFFFFFFFull) - w.Qa + 1ull;
                }
                // steps with both candidates inside for sure: -(G + k Fw)/Qa in [0.1, N - 2.1]
                const float Gf = (float)G, qf = (float)Qa, ff = (float)Fw, kmax = (float)steps;
                const float a = -((float)N - 2.1f) * qf - Gf, b = -0.1f * qf - Gf;
                float f0, f1;
                if (Fw > 0) {
                    f0 = ceilf(a / ff);
                    f1 = floorf(b / ff) + 1.f;
                } else {
                    f0 = a <= 0.f ? 0.f : kmax;
                    f1 = b >= 0.f ? kmax : 0.f;
                }
                k0 = (int)fminf(fmaxf(f0, 0.f), kmax);
                k1 = (int)fminf(fmaxf(f1, 0.f), kmax);
            }
            k0 = __reduce_max_sync(0xffffffffu, k0);
            k1 = __reduce_min_sync(0xffffffffu, k1);
            if (guard || k1 <= k0) k0 = k1 = 0;
            float v;
            // pixel (t, u): element qt + u su of x (columns) or xt (rows)
            if (kcol) v = mf_walk32<true>(w, on, x, ts * N + N - 1, dir * N, N, steps, k0, k1);
            else v = mf_walk32<false>(w, on, xt, (N - 1 - ts) * N, -dir * N, N, steps, k0, k1);
            if (on) acc = v * A.inv_c;
        }
        if (ray) epi(r, acc);
    }
}

// FP32 backprojector, parallel beam. A block takes a tile of 32 pixel rows (a
// warp's lanes) by 32 image columns (8 per warp) and walks its share of the
// angles in batches of kBpBatch, the next batch's loads in flight: the at most
// 46 bins of an angle that meet the tile are staged in shared memory as pairs
// (y_j, y_{j+1}) / c, so that a pixel reads its two rays' values with one load
// and no bounds check. A thread's distance D = jh + dl is kept as three words
// (jh relative to the tile's first bin, 32 bits of dl, the rest), stepped by
// cos from column to column with one three-word add: no shifts or masks but
// the one that cuts dl to 31 bits. A batch with an Inf or NaN in its staged
// values reads y itself, only where the entry is positive, as a stored
// matrix does.
// Bound by integer issue. N = 1024, 720 angles, 1448 bins: 0.92 ms with a
// thread per 4 pixels reading y from L1, 35 instructions per pixel and angle ->
// 0.46 ms, 19 of them (4 shares of the angles, their sums added by k_mf_finish).
constexpr int kBpBatch = 8;   // angles staged at once (half a warp each)
constexpr int kBpOcc = 7;     // resident blocks per SM (72 registers; 8 of 64: 4% slower)
constexpr int kBpBins = 48;   // bins of an angle that meet a tile: 31 (|cos| + |sin|) + 2 at most
struct __align__(16) BpAngle {
    unsigned c_lo, c_mid;     // cos as three words (the fraction's bits 46.. at the top of c_mid)
    int c_hi, H2s;
    int Hc;                   // H2s - (2^31 - 1): entry of the second ray from u of the first
    float ramp, a0, a1;       // entries sat((H2s - u) ramp + a0), sat((Hc + u) ramp + a1)
    long long S;
    int jlo;                  // first staged bin
    float inv_c;
    long long Dw[4];          // distance at the warps' first pixels, from bin jlo
};
template <class Epi>
__global__ void __launch_bounds__(128, kBpOcc) k_mf_backproject32(const MfAngle *__restrict__ ang, int nth, int p,
                                                             int N, const float *__restrict__ y, float *part,
                                                             unsigned *flag, Epi epi) {
    if (blockIdx.x + blockIdx.y + threadIdx.x == 0) *flag = 0;
    __shared__ BpAngle cs[2][kBpBatch];
    __shared__ float2 ys[2][kBpBatch][kBpBins];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nt = (N + 31) / 32, tx = blockIdx.x / nt, ty = blockIdx.x - tx * nt;
    const int nb = (nth + kBpBatch - 1) / kBpBatch;  // the share's angles: whole batches
    const int i0 = (int)((int64_t)nb * blockIdx.y / gridDim.y) * kBpBatch;
    const int i1 = min(nth, (int)((int64_t)nb * (blockIdx.y + 1) / gridDim.y) * kBpBatch);
    const int ix0 = tx * 32, iy0 = N - 1 - ty * 32;  // the tile's first pixel; lane l is iy0 - l
    const int sa = threadIdx.x >> 4, hl = threadIdx.x & 15;  // staging: angle of the batch, lane of 16
    float acc[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[b] = 0.f;
    MfAngle R;
    float yv[3];
    auto load_angle = [&](int ib) {  // this thread's angle of the batch from ib (none: weight 0)
        if (ib + sa < i1) R = mf_load<float>(ang + ib + sa);
        else R = MfAngle{};
    };
    auto put_angle = [&](int ib, int buf) {  // its constants to shared memory, its bins' loads
        const long long base = ix0 * R.C + iy0 * R.S + R.K;
        const long long mn = base + min(0LL, 31 * R.C) + min(0LL, -31 * R.S);
        const int jlo = (int)(mn >> kFix);
        const long long Dr = base - ((long long)jlo << kFix);
        BpAngle &B = cs[buf][sa];
        if (hl < 4) B.Dw[hl] = Dr + hl * 8 * R.C;
        if (hl == 0) {
            B.c_lo = (unsigned)R.C << 18;
            B.c_mid = (unsigned)(R.C >> 14);
            B.c_hi = (int)(R.C >> kFix);
            B.H2s = R.H2s;
            B.Hc = R.H2s - 0x7FFFFFFF;
            B.ramp = R.ramp;
            B.a0 = B.a1 = 0.f;
            if (R.tie != 0) {  // every pixel at the same fraction of a bin: entries 0 or 1
                const long long dl = R.K & ((1LL << kFix) - 1), dr = (1LL << kFix) - dl;
                B.a0 = dl < R.H2 || (R.tie == 1 && dl == R.H2) ? 1.f : 0.f;
                B.a1 = dr < R.H2 || (R.tie == -1 && dr == R.H2) ? 1.f : 0.f;
            }
            B.S = R.S;
            B.jlo = jlo;
            B.inv_c = R.inv_c;
        }
        const float *yi = y + (int64_t)(ib + sa) * p;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int j = jlo + hl + 16 * e;
            yv[e] = ib + sa < i1 && (unsigned)j < (unsigned)p ? __ldg(yi + j) : 0.f;
        }
    };
    auto put_bins = [&](float inv_c, int buf) {
        bool bad = false;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int k = hl + 16 * e;
            const float v = yv[e] * inv_c;
            bad |= !isfinite(v);
            ys[buf][sa][k].x = v;
            if (k > 0) ys[buf][sa][k - 1].y = v;
        }
        return bad;
    };
    load_angle(i0);
    put_angle(i0, 0);
    float inv_c = R.inv_c;
    load_angle(i0 + kBpBatch);
    bool bad = __syncthreads_or(put_bins(inv_c, 0));
    int buf = 0;
    for (int ib = i0; ib < i1; ib += kBpBatch) {
        const bool more = ib + kBpBatch < i1;
        if (more) {
            put_angle(ib + kBpBatch, buf ^ 1);
            inv_c = R.inv_c;
            load_angle(ib + 2 * kBpBatch);
        }
#pragma unroll 1
        for (int a = 0; a < kBpBatch; ++a) {
            const BpAngle &B = cs[buf][a];
            const unsigned c_lo = B.c_lo, c_mid = B.c_mid;
            const int c_hi = B.c_hi, H2s = B.H2s, Hc = B.Hc;
            const float ramp = B.ramp, a0 = B.a0, a1 = B.a1;
            const long long D = B.Dw[wid] - lane * B.S;
            unsigned lo = (unsigned)D << 18, mid = (unsigned)(D >> 14);
            int hi = (int)(D >> kFix);
            auto pixels = [&](auto guard) {
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const int u = (int)(mid >> 1);
                    const float w0 = __saturatef(fmaf((float)(H2s - u), ramp, a0));
                    const float w1 = __saturatef(fmaf((float)(Hc + u), ramp, a1));
                    if constexpr (decltype(guard)::value) {
                        const int j = B.jlo + hi;
                        const float *yi = y + (int64_t)(ib + a) * p;
                        if (w0 > 0.f && (unsigned)j < (unsigned)p) acc[b] += B.inv_c * w0 * __ldg(yi + j);
                        if (w1 > 0.f && (unsigned)(j + 1) < (unsigned)p) acc[b] += B.inv_c * w1 * __ldg(yi + j + 1);
                    } else {
                        const float2 v = ys[buf][a][hi];
                        acc[b] = fmaf(w0, v.x, acc[b]);
                        acc[b] = fmaf(w1, v.y, acc[b]);
                    }
                    asm("add.cc.u32 %0, %0, %3; addc.cc.u32 %1, %1, %4; addc.u32 %2, %2, %5;"
                        : "+r"(lo), "+r"(mid), "+r"(hi)
                        : "r"(c_lo), "r"(c_mid), "r"(c_hi));
                }
            };
            if (bad) {
                if (ib + a < i1) pixels(std::true_type{});
            } else {
                pixels(std::false_type{});
            }
        }
        bool nb = false;
        if (more) nb = put_bins(inv_c, buf ^ 1);
        bad = __syncthreads_or(nb);
        buf ^= 1;
    }
    const int k = ty * 32 + lane;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const int ix = ix0 + wid * 8 + b;
        if (ix >= N || k >= N) continue;
        const int64_t q = (int64_t)ix * N + k;
        if (gridDim.y > 1) part[(int64_t)blockIdx.y * N * N + q] = acc[b];
        else epi(q, acc[b]);
    }
}

// Sum over the rays through pixel q of a_rq * y_r, for every pixel; MODE 1
// sums a_rq (y unused). A thread takes PB vertically adjacent pixels of one
// image column (iy0, iy0 - 1, ...), which share the per-angle set-up. With
// D = ix C + iy S + K = jh 2^46 + dl (0 <= dl < 2^46), the rays j with
// |D - j 2^46| <= H2 (< 2^46) are jh (d = dl) and jh + 1 (d = dl - 2^46).
template <typename YT, typename ACC, int MODE, int PB, bool TIE>
__device__ __forceinline__ void bp_angle(const MfAngle &A, long long D, int p,
                                         const YT *__restrict__ yi, ACC (&acc)[PB]) {
    constexpr long long kMask = (1LL << kFix) - 1;
    const long long t0 = TIE && A.tie == 1 ? A.H2 : -1, t1 = TIE && A.tie == -1 ? A.H2 : -1;
#pragma unroll
    for (int b = 0; b < PB; ++b, D -= A.S) {
        const int jh = (int)(D >> kFix);
        const long long dl = D & kMask;
        ACC w0, w1;
        if constexpr (TIE) {
            w0 = Chord<ACC>::tied(A, dl, t0);
            w1 = Chord<ACC>::tied(A, (1LL << kFix) - dl, t1);
        } else {
            w0 = Chord<ACC>::ramp(A, dl);
            w1 = Chord<ACC>::ramp(A, (1LL << kFix) - dl);
        }
        mf_add<YT, ACC, MODE>(acc[b], w0, (unsigned)jh < (unsigned)p, yi, jh);
        mf_add<YT, ACC, MODE>(acc[b], w1, (unsigned)(jh + 1) < (unsigned)p, yi, jh + 1);
    }
}

// SPLIT: block row s sums its share of the angles into part (n values per
// share) and k_mf_finish adds the shares.
template <typename YT, typename ACC, int MODE, int PB, bool SPLIT, class Epi>
__global__ void __launch_bounds__(128) k_mf_backproject(const MfAngle *__restrict__ ang,
                                                        int nth, int p, int N,
                                                        const YT *__restrict__ y, ACC *part,
                                                        Epi epi) {
    const int groups = (N + PB - 1) / PB;  // pixel groups per image column
    const int64_t ngr = (int64_t)N * groups;
    const int i0 = SPLIT ? (int)((int64_t)nth * blockIdx.y / gridDim.y) : 0;
    const int i1 = SPLIT ? (int)((int64_t)nth * (blockIdx.y + 1) / gridDim.y) : nth;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ngr;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int ix = (int)(t / groups), k = (int)(t - (int64_t)ix * groups);
        const int iy0 = N - 1 - PB * k;  // pixel q = ix*N + PB*k + b is iy0 - b
        ACC acc[PB];
#pragma unroll
        for (int b = 0; b < PB; ++b) acc[b] = 0;
        for (int i = i0; i < i1; ++i) {
            const MfAngle A = mf_load<ACC>(ang + i);
            const YT *__restrict__ yi = y + (int64_t)i * p;
            const long long D = (long long)ix * A.C + (long long)iy0 * A.S + A.K;
            if (A.tie != 0) bp_angle<YT, ACC, MODE, PB, true>(A, D, p, yi, acc);
            else bp_angle<YT, ACC, MODE, PB, false>(A, D, p, yi, acc);
        }
        const int64_t q0 = (int64_t)ix * N + PB * k;
#pragma unroll
        for (int b = 0; b < PB; ++b) {
            if (iy0 - b < 0) continue;
            if (SPLIT) part[(int64_t)blockIdx.y * N * N + q0 + b] = acc[b];
            else epi(q0 + b, acc[b]);
        }
    }
}

// The shares of the angles added per pixel, in order, then the epilogue.
template <typename ACC, class Epi>
__global__ void __launch_bounds__(256) k_mf_finish(const ACC *__restrict__ part, int shares,
                                                   int64_t n, Epi epi) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        ACC acc = part[q];
        for (int s = 1; s < shares; ++s) acc += part[(int64_t)s * n + q];
        epi(q, acc);
    }
}

// Per angle of a fan: the source P and the unit direction u0 towards the
// origin (floats, for the candidate search only), and whether one of its rays
// is axis-aligned.
struct MfFanAngle {
    float px, py, ux, uy;
    int tie, pad[3];
};

// The sorted bin angles oms and, for a uniform grid of L cells over
// [oms[0], oms[p-1]], the first sorted index at or past each cell's start
// (tab[L] = p): the search for an angle starts one cell before the cell it
// falls in (the last cell past the grid), whose start lies below it, and
// steps forward.
struct MfBins {
    const float *oms;
    const int *omj;
    const int *tab;
    float om0, inv_cell;
    int L;
    // the sorted keys [ua, ub) that pixels of the image can reach, where those
    // are evenly spaced (ub > ua): key k is ukey + (k - ua) / uinv
    int ua, ub;
    float ukey, uinv;
    // the first k with oms[k] >= lo
    __device__ __forceinline__ int first(float lo, int p) const {
        const float t = (lo - om0) * inv_cell;
        const int k = t < 1.f ? 0 : (t >= (float)L ? L - 1 : (int)t - 1);
        int a = __ldg(tab + k);
        while (a < p && __ldg(oms + a) < lo) ++a;
        return a;
    }
    // the first k with oms[k] > hi
    __device__ __forceinline__ int past(float hi, int p) const {
        int a = first(hi, p);
        while (a < p && __ldg(oms + a) <= hi) ++a;
        return a;
    }
};

// Fan backprojector. A block takes a tile of 32 pixel rows (a warp's lanes) by
// 16 image columns (kFanPB per warp) and walks its share of the angles, two
// at a time: it stages the rays that can meet the tile -- their records,
// distances at the tile's origin and y -- in shared memory, the next angles'
// loads in flight while these are used, and every pixel meets its candidates
// there. (One thread per two pixels that read each candidate's 96-byte record
// from global memory was bound by those scattered, dependent loads.)
constexpr int kFanThreads = 128;        // 4 warps
constexpr int kFanPB = 4;               // image columns per warp
constexpr int kFanCap = kFanThreads / 2;  // most rays of an angle staged at once
constexpr int kFanPad = 4;              // records of weight 0 on either side of them
// A staged ray (48 or 80 bytes: the lanes' 16-byte reads of neighbouring
// records fall in different banks).
template <typename ACC> struct FanRay;
template <> struct __align__(16) FanRay<float> {
    longlong2 cs;          // C, -S
    int H2s;               // H2 at 31 bits
    float inv_c, ramp, y;
    long long d0, H2;      // the distance at the tile's origin pixel; H2
    __device__ __forceinline__ void put(const MfAngle &A, long long d, float v) {
        cs = longlong2{A.C, -A.S};
        H2s = A.H2s;
        inv_c = A.inv_c;
        ramp = A.ramp;
        y = v;
        d0 = d;
        H2 = A.H2;
    }
    __device__ __forceinline__ void none() {
        cs = longlong2{0, 0};
        H2s = 0;
        inv_c = 0.f;
        ramp = 0.f;
        y = 0.f;
        d0 = H2 = 0;
    }
    // acc += a_rq y_r at distance d: the same entry, from the same exact
    // distance, as the projector's. TIE: the ray may be axis-aligned (tie its
    // side), FAR: the pixel may be a pixel's width away or more.
    template <int MODE, bool TIE, bool FAR>
    __device__ __forceinline__ void add(long long d, int tie, float &acc) const {
        const long long ud = d ^ (d >> 63);
        float w = inv_c * __saturatef((float)(H2s - (int)(ud >> 15)) * ramp);
        if (TIE && tie != 0) {
            const long long ad = d < 0 ? -d : d;
            w = ad < H2 || (ad == H2 && tie == (d > 0 ? 1 : -1)) ? inv_c : 0.f;
        }
        if (FAR && (ud >> 46) != 0) w = 0.f;
        if (w > 0.f) acc += MODE == 0 ? w * y : w;
    }
};
template <> struct __align__(16) FanRay<double> {
    longlong2 cs;
    long long d0, H2;
    long long H1, Hcut;
    double inv_c, ramp;
    double y, pad;
    __device__ __forceinline__ void put(const MfAngle &A, long long d, double v) {
        cs = longlong2{A.C, -A.S};
        d0 = d;
        H2 = A.H2;
        H1 = A.H1;
        Hcut = A.Hcut;
        inv_c = A.inv_c64;
        ramp = A.scale_ramp64;
        y = v;
    }
    __device__ __forceinline__ void none() {
        cs = longlong2{0, 0};
        d0 = 0;
        Hcut = -1;
    }
    // below Hcut every entry is positive; an axis-aligned ray (Hcut = H1 = H2)
    // also keeps |d| = H2 on its positive side
    template <int MODE, bool TIE, bool FAR>
    __device__ __forceinline__ void add(long long d, int tie, double &acc) const {
        const long long ad = d < 0 ? -d : d;
        if (ad >= Hcut && !(TIE && tie != 0 && ad == Hcut && tie == (d > 0 ? 1 : -1))) return;
        const double w = ad <= H1 ? inv_c : (double)(H2 - ad) * ramp;
        acc += MODE == 0 ? w * y : w;
    }
};
template <typename ACC> struct FanRays {
    FanRay<ACC> ray[kFanCap + 2 * kFanPad];
    float key[kFanCap];
    int tie[kFanCap];
};

// d + l C for a small l >= 0.
__device__ __forceinline__ long long mad_small(long long d, unsigned l, long long C) {
    unsigned long long r = (unsigned long long)d + (unsigned long long)l * (unsigned)C;
    r += (unsigned long long)(l * (unsigned)((unsigned long long)C >> 32)) << 32;
    return (long long)r;
}

// TANK: the keys are tan(bin angle) (a source at least 1.42 N from the
// centre: every pixel lies within 30 degrees of the central ray, where tan is
// monotone); a pixel's window is the tangent of its angle window, t =
// tan(alpha) = cross/dot and tan(de) combined by the tangent addition formula
// -- no arctangent or arcsine. UNI (N >= 16): the keys the image can reach are
// evenly spaced, so a pixel's candidates are the indices in f -+ w: f from t,
// w from the half-width H2/|v| of a pixel square along its own direction, H2 =
// (|cos| + |sin|)/2 of v, bounded once per tile and angle. With at most
// kFanPad candidates every lane tests the same number (a ray that misses the
// pixel has entry 0), so the loop has no branch on the lane.
// N = 512, 720 angles, 728 bins, FP32: 3.12 ms (a thread per two pixels, records
// from global memory) -> 0.81 ms; bound by shared-memory reads (75% of the
// wavefront rate: 40 bytes per candidate) and issue (64%).
template <typename YT, typename ACC, int MODE, bool TANK, bool UNI, class Epi>
__global__ void __launch_bounds__(kFanThreads, 7) k_mf_backproject_fan(
        const MfAngle *__restrict__ rays, const MfFanAngle *__restrict__ fa, MfBins B, int nth,
        int p, int N, const YT *__restrict__ y, ACC *part, unsigned *flag, Epi epi) {
    if (sizeof(ACC) == 4 && blockIdx.x + blockIdx.y + threadIdx.x == 0) *flag = 0;
    constexpr int PB = kFanPB, CAP = kFanCap, PAD = kFanPad, NA = kFanThreads;
    __shared__ FanRays<ACC> W[2][2];
    __shared__ int2 win[NA];     // per angle: the sorted keys [x, y) that can meet the tile
    __shared__ float4 fs[NA];    // P, u0
    __shared__ float2 wt[NA];    // w (UNI), axis-aligned rays
    const int t = threadIdx.x, lane = t & 31, wc = (t >> 5) * PB;
    const int half_id = t / CAP, ts = t % CAP;  // this thread stages ray ts of piece half_id
    const int tiles_k = (N + 31) >> 5;
    const int k0 = (int)(blockIdx.x % tiles_k) * 32, ix0 = (int)(blockIdx.x / tiles_k) * 4 * PB;
    // pixel (ix0 + lx, iyT - lane) is element (ix0 + lx) N + k0 + lane
    const int iyT = N - 1 - k0;
    const float half = 0.5f * (float)N - 0.5f;
    const float cy = (float)(iyT - lane) - half, cx0 = (float)(ix0 + wc) - half;
    const int a0 = (int)((int64_t)nth * blockIdx.y / gridDim.y);
    const int a1 = (int)((int64_t)nth * (blockIdx.y + 1) / gridDim.y);
    ACC acc[PB];
#pragma unroll
    for (int c = 0; c < PB; ++c) acc[c] = 0;
    if (t < 4 * PAD) W[t / (2 * PAD)][t / PAD & 1].ray[t % PAD].none();  // the records before a window

    for (int i0 = a0; i0 < a1; i0 += NA) {
        const int na = min(NA, a1 - i0);
        if (t < na) {
            // the tile's centre and the radius that covers its pixels
            const int cols = min(4 * PB, N - ix0), rows = min(32, N - k0);
            const float tx = (float)ix0 + 0.5f * (float)(cols - 1) - half;
            const float ty = (float)iyT - 0.5f * (float)(rows - 1) - half;
            const float rho = 0.5f * sqrtf((float)((cols - 1) * (cols - 1) + (rows - 1) * (rows - 1))) + 0.75f;
            const MfFanAngle F = fa[i0 + t];
            const float vx = tx - F.px, vy = ty - F.py, vv = fmaf(vx, vx, vy * vy);
            const float cr = fmaf(F.ux, vy, -F.uy * vx), dt = fmaf(F.ux, vx, F.uy * vy);
            bool all = vv <= 1.05f * rho * rho;
            float lo = 0.f, hi = 0.f, w = 1e9f;
            if (TANK) {
                const float tt = cr / dt, tau = rho * rsqrtf(fmaxf(vv - rho * rho, 1e-6f)) * 1.001f + 1e-4f;
                all = all || dt <= 0.f || fabsf(tt) * tau > 0.9f;
                lo = (tt - tau) / (1.f + tt * tau);
                hi = (tt + tau) / (1.f - tt * tau);
            } else {
                const float al = atan2f(cr, dt), de = asinf(fminf(1.f, rho * rsqrtf(vv))) + 1e-3f;
                lo = al - de;
                hi = al + de;
                all = all || lo < -3.14f || hi > 3.14f;
            }
            int ka = 0, kb = p;
            if (!all) {
                ka = B.first(lo, p);
                kb = B.past(hi, p);
            }
            if (UNI) {
                ka = max(ka, B.ua);
                kb = min(kb, B.ub);
                if (!all) {
                    const float av = sqrtf(vv), rm = 1.f / (av - rho);  // 1/|v| of any pixel of the tile
                    const float h = fminf(0.7072f, 0.5f * (fabsf(vx) + fabsf(vy)) / av + rm * (0.71f * rho + 0.75f));
                    const float tm = fmaxf(fabsf(lo), fabsf(hi));
                    const float tau = h * rm * (1.f + 0.5f * rm * rm) + 8e-6f;  // >= tan(de) for |v| >= 2
                    if (rm > 0.f && tm * tau < 0.5f)
                        w = B.uinv * tau * (1.f + tm * tm) / (1.f - tm * tau) + 0.011f;
                }
            }
            fs[t] = make_float4(F.px, F.py, F.ux, F.uy);
            wt[t] = make_float2(w, F.tie != 0 ? 1.f : 0.f);
            win[t] = make_int2(ka, kb);
        }
        __syncthreads();
        // the windows in pieces of at most CAP rays: angle .x, first key .y;
        // .x = na past the last
        auto next = [&](int2 c, int by) {
            c.y += by;
            while (c.x < na && c.y >= win[c.x].y)
                if (++c.x < na) c.y = win[c.x].x;
            return c;
        };
        MfAngle R;
        YT yv = 0;
        float key = 0.f;
        int have = 0;  // 1: a ray of the piece; 2: past its end
        auto load = [&](int2 c) {  // this thread's ray of piece c
            have = c.x >= na ? 0 : (c.y + ts < win[c.x].y ? 1 : 2);
            if (have != 1) return;
            const int64_t r = (int64_t)(i0 + c.x) * p + __ldg(B.omj + c.y + ts);
            R = mf_load<ACC>(rays + r);
            if (MODE == 0) yv = __ldg(y + r);
            if (!UNI) key = __ldg(B.oms + c.y + ts);
        };
        auto store = [&](int b) {
            FanRays<ACC> &V = W[b][half_id];
            if (have == 1) {
                V.ray[PAD + ts].put(R, mad_small(mad_small(R.K, (unsigned)ix0, R.C), (unsigned)iyT, R.S), (ACC)yv);
                V.tie[ts] = R.tie;
                if (!UNI) V.key[ts] = key;
            } else if (have == 2) {
                V.ray[PAD + ts].none();
            }
            if (UNI && have != 0 && ts < PAD) V.ray[PAD + CAP + ts].none();
        };
        int buf = 0;
        int2 c0 = next(make_int2(0, win[0].x), 0), c1 = next(c0, CAP);
        load(half_id ? c1 : c0);
        store(buf);
        __syncthreads();
        while (c0.x < na) {
            const int2 n0 = next(c1, CAP), n1 = next(n0, CAP);
            load(half_id ? n1 : n0);
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
                const int2 cur = hh ? c1 : c0;
                if (cur.x >= na) break;
                const int len = min(CAP, win[cur.x].y - cur.y);
                const FanRays<ACC> &V = W[buf][hh];
                const float4 F = fs[cur.x];
                const float2 wf = wt[cur.x];
                const float vy = cy - F.y, vx0 = cx0 - F.x;
                float cr = fmaf(F.z, vy, -F.w * vx0), dt = fmaf(F.z, vx0, F.w * vy);
                const float w = wf.x, off = (float)(B.ua - cur.y);
                const int nc = (int)floorf(2.f * w) + 1;  // candidates of a pixel
                if (UNI && nc <= PAD && wf.y == 0.f) {
#pragma unroll
                    for (int c = 0; c < PB; ++c) {
                        const float f = fmaf(__fdividef(cr, dt) - B.ukey, B.uinv, off);
                        const int kl = min(max((int)ceilf(f - w), -PAD), len);
                        const FanRay<ACC> *r = V.ray + (PAD + kl);
#pragma unroll
                        for (int e = 0; e < PAD; ++e)
                            if (e < nc) {
                                const long long d = mad_small(mad_small(r[e].d0, (unsigned)(wc + c), r[e].cs.x),
                                                              (unsigned)lane, r[e].cs.y);
                                r[e].template add<MODE, false, true>(d, 0, acc[c]);
                            }
                        cr -= F.w;
                        dt += F.z;
                    }
                    continue;
                }
#pragma unroll
                for (int c = 0; c < PB; ++c) {
                    auto entry = [&](int k) {
                        const FanRay<ACC> &r = V.ray[PAD + k];
                        const long long d = mad_small(mad_small(r.d0, (unsigned)(wc + c), r.cs.x),
                                                      (unsigned)lane, r.cs.y);
                        r.template add<MODE, true, true>(d, V.tie[k], acc[c]);
                    };
                    const float tt = __fdividef(cr, dt);
                    if constexpr (UNI) {
                        const float f = fmaf(tt - B.ukey, B.uinv, off);
                        const int kl = max(0, (int)ceilf(f - w)), kh = min(len - 1, (int)floorf(f + w));
                        for (int k = kl; k <= kh; ++k) entry(k);
                    } else {
                        float lo, hi;
                        const float vx = vx0 + (float)c;
                        if constexpr (TANK) {
                            const float tau = 0.7072f * rsqrtf(fmaf(vx, vx, fmaf(vy, vy, -0.50014f))) + 2.5e-4f;
                            lo = __fdividef(tt - tau, fmaf(tt, tau, 1.f));
                            hi = __fdividef(tt + tau, fmaf(-tt, tau, 1.f));
                        } else {
                            const float al = atan2f(cr, dt);
                            const float de = asinf(fminf(1.f, 0.7072f * rsqrtf(fmaf(vx, vx, vy * vy)))) + 2e-4f;
                            lo = al - de;
                            hi = al + de;
                        }
                        // the first staged key >= lo: a guess by interpolation, then steps
                        const float f = V.key[0], l = V.key[len - 1];
                        int k = l > f ? (int)((lo - f) * __fdividef((float)(len - 1), l - f)) : 0;
                        k = max(0, min(len, k));
                        while (k > 0 && V.key[k - 1] >= lo) --k;
                        while (k < len && V.key[k] < lo) ++k;
                        for (; k < len && V.key[k] <= hi; ++k) entry(k);
                    }
                    cr -= F.w;
                    dt += F.z;
                }
            }
            buf ^= 1;
            store(buf);
            c0 = n0;
            c1 = n1;
            __syncthreads();
        }
    }
    const int k = k0 + lane;
#pragma unroll
    for (int c = 0; c < PB; ++c) {
        const int ix = ix0 + wc + c;
        if (ix >= N || k >= N) continue;
        const int64_t q = (int64_t)ix * N + k;
        if (gridDim.y > 1) part[(int64_t)blockIdx.y * N * N + q] = acc[c];
        else epi(q, acc[c]);
    }
}

constexpr int kMfPB = 4;  // pixels per backprojector thread (parallel beam)

int grid_for(int64_t items, int threads) {
    int64_t b = (items + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)sm_count() * 32));
}

}  // namespace
}  // namespace fair

struct fair_mf_s {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int prec = FAIR_PREC_F32;
    int N = 0, p = 0, nth = 0;
    int kind = 0;                      // 0: parallel beam, 1: fan beam
    fair::DevBuf ang;                  // MfAngle [nth] (parallel) or [nth*p] (fan: per ray)
    fair::DevBuf fang, oms, omj, omt;  // fan: MfFanAngle [nth], sorted bin angles, their bins,
                                       // first sorted index per cell of the angle grid
    float om0 = 0.f, om_inv = 0.f;     // the grid: start, 1 / cell width, cells
    int om_L = 1;
    bool tan_keys = false;             // oms holds tan(bin angle) (the backprojector's TANK)
    int uni_a = 0, uni_b = 0;          // evenly spaced reachable keys (MfBins), none: uni_b = 0
    float uni_key = 0.f, uni_inv = 0.f;
    fair::DevBuf part;                 // the backprojector's sums per share of the angles
    fair::DevBuf w_in, w_out;          // host-call staging (FP64)
    fair::DevBuf xt;                   // the projector's transposed copy of x
    fair::DevBuf nonfinite;            // whether x of the iteration under way holds an Inf or NaN
    fair::DevBuf v_a, v_b;             // reduced-precision staging
    // SIRT state
    bool ready = false, sart = false;
    double omg = 1.0, lb = 0.0, ub = 0.0;
    int bmode = 0;
    fair::DevBuf M_sart, M_cim, D;     // FP64 weights (computed on first use)
    bool have_sart = false, have_cim = false;
    fair::DevBuf x32, r, w_b, w_x;
    std::mutex mu;
};

namespace fair {
namespace {

int mf_grow_flag(fair_mf A) {
    if (A->nonfinite.p) return FAIR_OK;
    FAIR_TRY(A->nonfinite.grow(sizeof(unsigned)));
    FAIR_CUDA(cudaMemsetAsync(A->nonfinite.p, 0, sizeof(unsigned), A->stream));
    return FAIR_OK;
}

// Projector / backprojector launches of either geometry.
// The transposed copy of x that the projector reads (N^2 elements of the
// operator's precision), grown before a pass that reads x.
int mf_grow_xt(fair_mf A) {
    const size_t es = A->prec == FAIR_PREC_F64 ? sizeof(double) : sizeof(float);
    FAIR_TRY(mf_grow_flag(A));
    return A->xt.grow(es * (size_t)A->N * A->N);
}

template <typename XT, typename ACC, int MODE, class Epi>
void mf_project(fair_mf A, const XT *x, Epi epi, cudaStream_t s) {
    const int64_t m = (int64_t)A->nth * A->p;
    const int N = A->N;
    const MfAngle *ang = A->ang.as<MfAngle>();
    const XT *xt = nullptr;
    unsigned *nf = A->nonfinite.as<unsigned>();
    if (MODE == 0) {  // the rays that walk rows read the transpose (mf_grow_xt)
        const int nb = (N + 31) / 32;
        k_mf_transpose<XT><<<dim3(nb, nb), dim3(32, 8), 0, s>>>(x, A->xt.as<XT>(), N, nf);
        xt = A->xt.as<XT>();
    }
    if constexpr (std::is_same<ACC, float>::value) {
        static_assert(MODE == 0, "FP32 passes read x");
        const int g = grid_for((int64_t)A->nth * ((A->p + 31) / 32) * 32, 128);
        if (A->kind == 1)
            k_mf_project32<true><<<g, 128, 0, s>>>(ang, A->nth, A->p, N, x, xt, nf, epi);
        else
            k_mf_project32<false><<<g, 128, 0, s>>>(ang, A->nth, A->p, N, x, xt, nf, epi);
    } else if (A->kind == 1) {
        k_mf_project<XT, ACC, MODE, true><<<grid_for(m, 128), 128, 0, s>>>(ang, A->nth, A->p, N, x, xt, epi);
    } else {
        k_mf_project<XT, ACC, MODE, false><<<grid_for(m, 128), 128, 0, s>>>(ang, A->nth, A->p, N, x, xt, epi);
    }
}
// Blocks of the backprojector over the image, and the shares its angles are
// cut into so that a small image still fills the GPU: about 8 blocks of 4
// warps per SM, at least 8 angles each.
int64_t mf_bp_blocks(fair_mf A, bool f32) {
    const int64_t N = A->N;
    if (A->kind == 0 && f32) return ((N + 31) / 32) * ((N + 31) / 32);
    if (A->kind == 1) return ((N + 31) / 32) * ((N + 4 * kFanPB - 1) / (4 * kFanPB));
    return (N * ((N + kMfPB - 1) / kMfPB) + 127) / 128;
}
int mf_bp_shares(fair_mf A, bool f32) {
    const int64_t blocks = mf_bp_blocks(A, f32);
    if (A->kind == 0 && f32) {
        // k_mf_backproject32: 4 waves of blocks where a share keeps at least 12
        // batches of angles, 2 waves where it keeps 4, else one (the last wave's
        // idle SMs against the shares' first, unoverlapped loads and the pass that
        // adds them: N = 1024, 720 angles: 1, 2, 4 shares 518, 515, 477 us; N =
        // 512, 360 angles: 4, 9, 19 shares 89, 78, 89 us); whole batches each
        const int64_t nb = (A->nth + kBpBatch - 1) / kBpBatch;
        for (int waves = 4; waves >= 1; waves >>= 1) {
            const int64_t sh = std::min<int64_t>((int64_t)waves * kBpOcc * sm_count() / blocks, 32);
            if (sh <= 1) break;
            const int64_t keep = waves == 4 ? 12 : (waves == 2 ? 4 : 1);
            if (nb < sh * keep && waves > 1) continue;
            const int64_t per = (nb + sh - 1) / sh;  // batches per share
            return (int)((nb + per - 1) / per);
        }
        return 1;
    }
    const int64_t want = ((int64_t)sm_count() * 8) / blocks;
    return (int)std::max<int64_t>(1, std::min<int64_t>(want, std::min(A->nth / 8, 32)));
}
template <typename YT, typename ACC, int MODE, class Epi>
int mf_backproject(fair_mf A, const YT *y, Epi epi, cudaStream_t s) {
    const int64_t n = (int64_t)A->N * A->N;
    const MfAngle *ang = A->ang.as<MfAngle>();
    constexpr bool f32 = std::is_same<ACC, float>::value;
    const int shares = mf_bp_shares(A, f32);
    FAIR_TRY(mf_grow_flag(A));
    unsigned *flag = A->nonfinite.as<unsigned>();
    if (shares > 1) FAIR_TRY(A->part.grow(sizeof(ACC) * (size_t)shares * n));
    ACC *part = A->part.as<ACC>();
    if (A->kind == 1) {
        const MfBins B{A->oms.as<float>(), A->omj.as<int>(), A->omt.as<int>(), A->om0, A->om_inv, A->om_L,
                       A->uni_a, A->uni_b, A->uni_key, A->uni_inv};
        const dim3 g((unsigned)mf_bp_blocks(A, f32), shares);
        const MfFanAngle *fa = A->fang.as<MfFanAngle>();
        if (A->tan_keys && A->uni_b > A->uni_a)
            k_mf_backproject_fan<YT, ACC, MODE, true, true><<<g, kFanThreads, 0, s>>>(
                ang, fa, B, A->nth, A->p, A->N, y, part, flag, epi);
        else if (A->tan_keys)
            k_mf_backproject_fan<YT, ACC, MODE, true, false><<<g, kFanThreads, 0, s>>>(
                ang, fa, B, A->nth, A->p, A->N, y, part, flag, epi);
        else
            k_mf_backproject_fan<YT, ACC, MODE, false, false><<<g, kFanThreads, 0, s>>>(
                ang, fa, B, A->nth, A->p, A->N, y, part, flag, epi);
    } else if constexpr (f32) {
        const dim3 g((unsigned)mf_bp_blocks(A, f32), shares);
        k_mf_backproject32<<<g, 128, 0, s>>>(ang, A->nth, A->p, A->N, y, part, flag, epi);
    } else {
        const dim3 g((unsigned)std::min<int64_t>(mf_bp_blocks(A, f32), (int64_t)sm_count() * 32), shares);
        if (shares > 1)
            k_mf_backproject<YT, ACC, MODE, kMfPB, true><<<g, 128, 0, s>>>(ang, A->nth, A->p, A->N, y, part, epi);
        else
            k_mf_backproject<YT, ACC, MODE, kMfPB, false><<<g, 128, 0, s>>>(ang, A->nth, A->p, A->N, y, part, epi);
    }
    if (shares > 1) k_mf_finish<ACC><<<grid_for(n, 256), 256, 0, s>>>(part, shares, n, epi);
    return FAIR_OK;
}

int mf_weights(fair_mf A, bool sart, cudaStream_t s) {
    const int64_t m = (int64_t)A->nth * A->p, n = (int64_t)A->N * A->N;
    if (sart && !A->have_sart) {
        FAIR_TRY(A->M_sart.grow(sizeof(double) * (m + 1)));
        FAIR_TRY(A->D.grow(sizeof(double) * (n + 1)));
        EpiStore<double> e1{A->M_sart.as<double>()};
        mf_project<double, double, 1>(A, (const double *)nullptr, e1, s);
        EpiStore<double> e2{A->D.as<double>()};
        FAIR_TRY((mf_backproject<double, double, 1>(A, (const double *)nullptr, e2, s)));
        FAIR_CUDA(cudaGetLastError());
        FAIR_TRY(vec_reciprocal(A->M_sart.as<double>(), m, s));  // the epilogues multiply
        FAIR_TRY(vec_reciprocal(A->D.as<double>(), n, s));
        A->have_sart = true;
    }
    if (!sart && !A->have_cim) {
        FAIR_TRY(A->M_cim.grow(sizeof(double) * (m + 1)));
        EpiCimminoW e{A->M_cim.as<double>(), (double)m};
        mf_project<double, double, 2>(A, (const double *)nullptr, e, s);
        FAIR_CUDA(cudaGetLastError());
        FAIR_TRY(vec_reciprocal(A->M_cim.as<double>(), m, s));
        A->have_cim = true;
    }
    return FAIR_OK;
}

// One projector / backprojector pass of a SIRT iteration.
int mf_pass(fair_mf A, int pass, const double *d_b, double *d_x, cudaStream_t s) {
    const double *M = A->sart ? A->M_sart.as<double>() : A->M_cim.as<double>();
    const double *D = A->sart ? A->D.as<double>() : nullptr;
    if (A->prec == FAIR_PREC_F64) {
        if (pass == 1) {
            EpiResidF64 e{d_b, M, A->r.as<double>()};
            mf_project<double, double, 0>(A, (const double *)d_x, e, s);
        } else {
            EpiUpdateF64 e{D, d_x, A->omg, A->lb, A->ub, A->bmode};
            return mf_backproject<double, double, 0>(A, (const double *)A->r.as<double>(), e, s);
        }
    } else {
        if (pass == 1) {
            EpiResidLP e{d_b, M, A->r.as<float>(), 1.0};
            mf_project<float, float, 0>(A, (const float *)A->x32.as<float>(), e, s);
        } else {
            EpiUpdateLP e{D, d_x, A->x32.as<float>(), A->omg, A->lb, A->ub, A->bmode, 1.0};
            return mf_backproject<float, float, 0>(A, (const float *)A->r.as<float>(), e, s);
        }
    }
    return FAIR_OK;
}

}  // namespace
}  // namespace fair

#define MENTER(A)                                                  \
    do {                                                           \
        if (!(A)) { fair::set_detail("null operator"); return FAIR_ERR_NULL; } \
        FAIR_CUDA(cudaSetDevice((A)->device));                     \
    } while (0)

extern "C" {

}  // extern "C"

namespace fair {
namespace {

// The constants of the line with unit normal (C, S) and d = ix*C + iy*S + K
// for pixel (ix, iy): fixed-point terms, chord thresholds, walk axis, floats.
void mf_line(double C, double S, double K, MfAngle &a) {
    const double c = std::max(fabs(C), fabs(S)), s = std::min(fabs(C), fabs(S));
    a = MfAngle{};
    a.C = llround(C * kOne);
    a.S = llround(S * kOne);
    a.K = llround(K * kOne);
    a.H1 = llround(0.5 * (c - s) * kOne);
    a.H2 = llround(0.5 * (c + s) * kOne);
    a.Cf = (float)C;
    a.Sf = (float)S;
    a.Kf = (float)K;
    a.by_column = fabs(S) >= fabs(C) ? 1 : 0;
    a.inv_c = (float)(1.0 / c);
    a.inv_c64 = 1.0 / c;
    a.scale_ramp64 = s > 0 ? 1.0 / (kOne * c * s) : 0.0;
    a.tie = 0;
    if (a.S == 0) a.tie = C > 0 ? 1 : -1;        // vertical ray, normal (+-1, 0)
    else if (a.C == 0) a.tie = S > 0 ? 1 : -1;   // horizontal ray, normal (0, +-1)
    if (a.tie != 0) a.H1 = a.H2;                 // s = 0: no ramp
    // segments of 1e-10 or less are dropped, as the ray tracer does
    // (system_generation.f90:393-394)
    a.Hcut = a.tie != 0 ? a.H2 : a.H2 - (long long)floor(1e-10 * c * s * kOne);
    a.H2s = (int)(a.H2 >> 15);
    a.ramp = a.tie == 0 ? (float)(1.0 / (2147483648.0 * s)) : 0.f;
}

// A new operator handle with its own stream, or a status.
int mf_new(fair_mf *out, const fair_data *dat, int32_t prec, int kind) {
    if (!out || !dat || !dat->theta) return FAIR_ERR_NULL;
    *out = nullptr;
    if (prec != FAIR_PREC_F64 && prec != FAIR_PREC_F32) {
        set_detail("the matrix-free operator runs in FP64 or FP32");
        return FAIR_ERR_ARG;
    }
    const int N = dat->n, p = dat->p, nth = dat->nth;
    if (N < 1 || p < 2 || nth < 1) { set_detail("n >= 1, p >= 2, nth >= 1 required"); return FAIR_ERR_ARG; }
    if ((int64_t)nth * p > INT32_MAX || N > 8192 || p > 16384) {
        set_detail("the matrix-free operator needs n <= 8192, p <= 16384, nth*p < 2^31");
        return FAIR_ERR_ARG;
    }
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_detail(e != cudaSuccess ? cudaGetErrorString(e) : "no CUDA device");
        return FAIR_ERR_NOGPU;
    }
    fair_mf A = new (std::nothrow) fair_mf_s();
    if (!A) return FAIR_ERR_ALLOC;
    cudaGetDevice(&A->device);
    A->prec = prec;
    A->N = N;
    A->p = p;
    A->nth = nth;
    A->kind = kind;
    e = cudaStreamCreateWithFlags(&A->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete A;
        return cuda_fail(e, "cudaStreamCreate", __FILE__, __LINE__);
    }
    A->own_stream = true;
    *out = A;
    return FAIR_OK;
}

template <typename T>
int mf_upload(DevBuf &d, const std::vector<T> &v) {
    if (d.grow(sizeof(T) * std::max<size_t>(v.size(), 1)) != FAIR_OK) return FAIR_ERR_ALLOC;
    if (cudaMemcpy(d.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        return FAIR_ERR_ALLOC;
    }
    return FAIR_OK;
}

}  // namespace
}  // namespace fair

extern "C" {

int fair_mf_create_parallel(fair_mf *out, const fair_data *dat, int32_t prec) {
    FAIR_TRY(fair::mf_new(out, dat, prec, 0));
    fair_mf A = *out;
    const int N = dat->n, p = dat->p, nth = dat->nth;
    // per-angle constants (cos/sin from the host libm, as paralleltomo)
    std::vector<fair::MfAngle> t(nth);
    for (int i = 0; i < nth; ++i) {
        const double C = cos(dat->theta[i]), S = sin(dat->theta[i]);
        const double K = (0.5 - 0.5 * N) * (C + S) + 0.5 * (p - 1);
        fair::mf_line(C, S, K, t[i]);
    }
    if (fair::mf_upload(A->ang, t) != FAIR_OK) {
        fair_mf_destroy(A);
        *out = nullptr;
        return FAIR_ERR_ALLOC;
    }
    return FAIR_OK;
}

int fair_mf_create_fan(fair_mf *out, const fair_data *dat, int32_t geometry_fix, int32_t prec) {
    FAIR_TRY(fair::mf_new(out, dat, prec, 1));
    fair_mf A = *out;
    const int N = dat->n, p = dat->p, nth = dat->nth;
    const double pi = 3.141592653589793;  // 4*atan(1d0), system_generation.f90:4
    // the bin angles and the rotated source and central direction, as
    // fanlineartomo computes them (system_generation.f90:98-157)
    const double R = dat->r * N, dwn = dat->dw * N, sdn = dat->sd * N;
    const double dew = dwn / p;
    std::vector<double> omega(p), com(p), som(p);
    if (p % 2 == 1) {
        const int hh = (p - 1) / 2;
        for (int i = 1; i <= hh; ++i) {
            const double dep = i * dew;
            omega[hh - i] = atan(sdn / dep) - (geometry_fix ? .5 * pi : .5);  // :122
            omega[hh + i] = .5 * pi - atan(sdn / dep);
        }
        omega[hh] = 0.0;
    } else {
        const int hh = p / 2;
        for (int i = 1; i <= hh; ++i) {
            const double dep = (i - .5) * dew;
            omega[hh - i] = atan(sdn / dep) - .5 * pi;  // :129
            omega[hh + i - 1] = .5 * pi - atan(sdn / dep);
        }
    }
    for (int j = 0; j < p; ++j) {
        com[j] = cos(omega[j]);
        som[j] = sin(omega[j]);
    }
    std::vector<fair::MfAngle> rays((size_t)nth * p);
    std::vector<fair::MfFanAngle> fa(nth);
    for (int i = 0; i < nth; ++i) {
        const double c = cos(dat->theta[i]), s = sin(dat->theta[i]);
        const double x0th = c * 0.0 - s * R, y0th = s * 0.0 + c * R;
        const double ath = -x0th / R, bth = -y0th / R;
        fa[i] = fair::MfFanAngle{(float)x0th, (float)y0th, (float)ath, (float)bth, 0, {0, 0, 0}};
        for (int j = 0; j < p; ++j) {
            // the ray direction of the reference's tracer (:163-166)
            const double a = com[j] * ath - som[j] * bth;
            const double b = som[j] * ath + com[j] * bth;
            const double nu = sqrt(a * a + b * b);
            const double C = b / nu, S = -a / nu;  // unit normal
            const double K = C * (0.5 - 0.5 * N - x0th) + S * (0.5 - 0.5 * N - y0th);
            fair::mf_line(C, S, K, rays[(size_t)i * p + j]);
            if (rays[(size_t)i * p + j].tie != 0) fa[i].tie = 1;
        }
    }
    // the bin angles sorted (the odd-p angles of :122 are not monotone in j)
    std::vector<int> order(p);
    for (int j = 0; j < p; ++j) order[j] = j;
    std::stable_sort(order.begin(), order.end(),
                     [&](int u, int v) { return (float)omega[u] < (float)omega[v]; });
    // keys: tan of the bin angles when the source is at least 1.42 N from the
    // centre (every pixel within 30 degrees of the central ray) and every bin
    // angle below 1.5 rad, else the angles
    bool tk = R >= 1.42 * N;
    for (int j = 0; j < p; ++j) tk = tk && std::fabs(omega[j]) < 1.5;
    A->tan_keys = tk;
    std::vector<float> oms(p);
    for (int k = 0; k < p; ++k) oms[k] = (float)(tk ? std::tan(omega[order[k]]) : omega[order[k]]);
    // the sorted keys that a pixel of the image can reach, and whether they are
    // evenly spaced (a flat detector's tangents are; the odd-p angles of :122
    // lie past them)
    if (tk && N >= 16) {
        const double amax = asin(std::min(1.0, 0.7072 * (N + 2) / R)) + 2e-3;
        int ua = 0, ub = p;
        while (ua < p && atan((double)oms[ua]) < -amax) ++ua;
        while (ub > ua && atan((double)oms[ub - 1]) > amax) --ub;
        if (ub - ua >= 2) {
            const double step = ((double)oms[ub - 1] - (double)oms[ua]) / (ub - 1 - ua);
            bool even = step > 0;
            for (int k = ua; k < ub; ++k)
                even = even && std::fabs((double)oms[k] - ((double)oms[ua] + (k - ua) * step)) <= 2e-3 * step;
            if (even) {
                A->uni_a = ua;
                A->uni_b = ub;
                A->uni_key = oms[ua];
                A->uni_inv = (float)(1.0 / step);
            }
        }
    }
    // a grid of 4p cells over the sorted angles; tab[c] = first k with oms[k] >=
    // om0 + c / inv (the device starts one cell early and steps forward)
    const int L = 4 * p;
    const double span = (double)oms[p - 1] - (double)oms[0];
    A->om0 = oms[0];
    A->om_inv = span > 0 ? (float)(L / span) : 0.f;
    A->om_L = L;
    std::vector<int> tab(L + 1);
    for (int c = 0, k = 0; c <= L; ++c) {
        const double start = (double)oms[0] + (span > 0 ? c * span / L : 0.0);
        while (k < p && (double)oms[k] < start) ++k;
        tab[c] = c == L ? p : k;
    }
    if (fair::mf_upload(A->ang, rays) != FAIR_OK || fair::mf_upload(A->fang, fa) != FAIR_OK ||
        fair::mf_upload(A->oms, oms) != FAIR_OK || fair::mf_upload(A->omj, order) != FAIR_OK ||
        fair::mf_upload(A->omt, tab) != FAIR_OK) {
        fair_mf_destroy(A);
        *out = nullptr;
        return FAIR_ERR_ALLOC;
    }
    return FAIR_OK;
}

int fair_mf_destroy(fair_mf A) {
    if (!A) return FAIR_OK;
    cudaSetDevice(A->device);
    cudaStreamSynchronize(A->stream);
    for (fair::DevBuf *d : {&A->ang, &A->fang, &A->oms, &A->omj, &A->omt, &A->w_in, &A->w_out, &A->v_a,
                            &A->v_b, &A->M_sart, &A->M_cim, &A->D, &A->x32, &A->r, &A->w_b,
                            &A->w_x, &A->xt, &A->part, &A->nonfinite})
        d->release();
    if (A->own_stream) cudaStreamDestroy(A->stream);
    delete A;
    return FAIR_OK;
}

int fair_mf_set_stream(fair_mf A, void *cuda_stream) {
    MENTER(A);
    std::lock_guard<std::mutex> lk(A->mu);
    FAIR_CUDA(cudaStreamSynchronize(A->stream));
    if (A->own_stream) cudaStreamDestroy(A->stream);
    if (cuda_stream) {
        A->stream = (cudaStream_t)cuda_stream;
        A->own_stream = false;
    } else {
        FAIR_CUDA(cudaStreamCreateWithFlags(&A->stream, cudaStreamNonBlocking));
        A->own_stream = true;
    }
    return FAIR_OK;
}

int fair_mf_info(fair_mf A, int32_t *m, int32_t *n) {
    if (!A) return FAIR_ERR_NULL;
    if (m) *m = A->nth * A->p;
    if (n) *n = A->N * A->N;
    return FAIR_OK;
}

static int mf_apply(fair_mf A, bool back, const double *in, double *out) {
    MENTER(A);
    if (!in || !out) return FAIR_ERR_NULL;
    std::lock_guard<std::mutex> lk(A->mu);
    const int64_t m = (int64_t)A->nth * A->p, n = (int64_t)A->N * A->N;
    const int64_t nin = back ? m : n, nout = back ? n : m;
    cudaStream_t s = A->stream;
    FAIR_TRY(A->w_in.grow(sizeof(double) * (nin + 1)));
    FAIR_TRY(A->w_out.grow(sizeof(double) * (nout + 1)));
    if (!back) FAIR_TRY(fair::mf_grow_xt(A));
    FAIR_CUDA(cudaMemcpyAsync(A->w_in.p, in, sizeof(double) * nin, cudaMemcpyHostToDevice, s));
    if (A->prec == FAIR_PREC_F64) {
        fair::EpiStore<double> e{A->w_out.as<double>()};
        const double *vin = A->w_in.as<double>();
        if (back) FAIR_TRY((fair::mf_backproject<double, double, 0>(A, vin, e, s)));
        else fair::mf_project<double, double, 0>(A, vin, e, s);
        FAIR_CUDA(cudaGetLastError());
    } else {
        FAIR_TRY(A->v_a.grow(sizeof(float) * (nin + 1)));
        FAIR_TRY(A->v_b.grow(sizeof(float) * (nout + 1)));
        FAIR_TRY(fair::vec_to_f32(A->w_in.as<double>(), nin, A->v_a.as<float>(), s));
        fair::EpiStore<float> e{A->v_b.as<float>()};
        const float *vin = A->v_a.as<float>();
        if (back) FAIR_TRY((fair::mf_backproject<float, float, 0>(A, vin, e, s)));
        else fair::mf_project<float, float, 0>(A, vin, e, s);
        FAIR_CUDA(cudaGetLastError());
        if (!back) FAIR_CUDA(cudaMemsetAsync(A->nonfinite.p, 0, sizeof(unsigned), s));
        FAIR_TRY(fair::vec_to_f64(A->v_b.as<float>(), nout, A->w_out.as<double>(), s));
    }
    FAIR_CUDA(cudaMemcpyAsync(out, A->w_out.p, sizeof(double) * nout, cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    return FAIR_OK;
}

int fair_mf_nnz(fair_mf A, int64_t *nnz) {
    MENTER(A);
    if (!nnz) return FAIR_ERR_NULL;
    std::lock_guard<std::mutex> lk(A->mu);
    const int64_t m = (int64_t)A->nth * A->p;
    cudaStream_t s = A->stream;
    FAIR_TRY(A->w_out.grow(sizeof(double) * (m + 1)));
    fair::EpiStore<double> e{A->w_out.as<double>()};
    fair::mf_project<double, double, 3>(A, (const double *)nullptr, e, s);
    FAIR_CUDA(cudaGetLastError());
    std::vector<double> c(m);
    FAIR_CUDA(cudaMemcpyAsync(c.data(), A->w_out.p, sizeof(double) * m, cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    int64_t t = 0;
    for (double v : c) t += (int64_t)v;
    *nnz = t;
    return FAIR_OK;
}

int fair_mf_project(fair_mf A, const double *x, double *y) { return mf_apply(A, false, x, y); }
int fair_mf_backproject(fair_mf A, const double *y, double *x) { return mf_apply(A, true, y, x); }

int fair_mf_sirt_prepare(fair_mf A, const char *sirt_method, const fair_opts *options) {
    MENTER(A);
    if (!sirt_method) return FAIR_ERR_NULL;
    bool sart;
    if (!strcmp(sirt_method, "cimmino")) sart = false;
    else if (!strcmp(sirt_method, "sart")) sart = true;
    else { fair::set_detail("Not a recognised SIRT method."); return FAIR_ERR_METHOD; }
    std::lock_guard<std::mutex> lk(A->mu);
    fair_opts o;
    if (options) o = *options;
    else FAIR_TRY(fair_opts_initialise(&o));
    A->sart = sart;
    A->omg = o.relaxpar;
    A->lb = o.lbound;
    A->ub = o.ubound;
    A->bmode = (o.upb ? 1 : 0) | (o.lwrb ? 2 : 0);
    const int64_t m = (int64_t)A->nth * A->p, n = (int64_t)A->N * A->N;
    const bool red = A->prec != FAIR_PREC_F64;
    FAIR_TRY(A->r.grow((red ? sizeof(float) : sizeof(double)) * (m + 1)));
    if (red) FAIR_TRY(A->x32.grow(sizeof(float) * (n + 1)));
    FAIR_TRY(fair::mf_grow_xt(A));
    FAIR_TRY(fair::mf_weights(A, sart, A->stream));
    const int shares = fair::mf_bp_shares(A, red);
    if (shares > 1) FAIR_TRY(A->part.grow((red ? sizeof(float) : sizeof(double)) * (size_t)shares * n));
    FAIR_CUDA(cudaStreamSynchronize(A->stream));
    A->ready = true;
    return FAIR_OK;
}

static int mf_iterations(fair_mf A, const double *d_b, double *d_x, int32_t K, float *ms1,
                         float *ms2) {
    if (!A->ready) {
        fair::set_detail("call fair_mf_sirt_prepare first");
        return FAIR_ERR_STATE;
    }
    if (!d_b || !d_x) return FAIR_ERR_NULL;
    if (K < 0) { fair::set_detail("K >= 0 required"); return FAIR_ERR_ARG; }
    cudaStream_t s = A->stream;
    const int64_t n = (int64_t)A->N * A->N;
    if (A->prec != FAIR_PREC_F64) FAIR_TRY(fair::vec_to_f32(d_x, n, A->x32.as<float>(), s));
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    if (ms1)
        for (auto &e : ev) FAIR_CUDA(cudaEventCreate(&e));
    float t1 = 0.f, t2 = 0.f;
    int st = FAIR_OK;
    for (int it = 0; it < K; ++it) {
        if (ms1) cudaEventRecord(ev[0], s);
        st = fair::mf_pass(A, 1, d_b, d_x, s);
        if (ms1) cudaEventRecord(ev[1], s);
        if (st == FAIR_OK) st = fair::mf_pass(A, 2, d_b, d_x, s);
        if (st != FAIR_OK) break;
        if (ms1) {
            cudaEventRecord(ev[2], s);
            cudaError_t e = cudaEventSynchronize(ev[2]);
            if (e != cudaSuccess) { st = fair::cuda_fail(e, "matrix-free pass", __FILE__, __LINE__); break; }
            float a = 0.f, b = 0.f;
            cudaEventElapsedTime(&a, ev[0], ev[1]);
            cudaEventElapsedTime(&b, ev[1], ev[2]);
            t1 += a;
            t2 += b;
        }
    }
    if (ms1) {
        for (auto &e : ev) cudaEventDestroy(e);
        *ms1 = t1;
        *ms2 = t2;
    }
    if (st != FAIR_OK) return st;
    FAIR_CUDA(cudaGetLastError());
    return FAIR_OK;
}

int fair_mf_sirt_run_device(fair_mf A, const double *d_b, double *d_x, int32_t K) {
    MENTER(A);
    std::lock_guard<std::mutex> lk(A->mu);
    return mf_iterations(A, d_b, d_x, K, nullptr, nullptr);
}

int fair_mf_sirt_run_device_timed(fair_mf A, const double *d_b, double *d_x, int32_t K,
                                  float *ms_project, float *ms_backproject) {
    MENTER(A);
    if (!ms_project || !ms_backproject) return FAIR_ERR_NULL;
    std::lock_guard<std::mutex> lk(A->mu);
    return mf_iterations(A, d_b, d_x, K, ms_project, ms_backproject);
}

int fair_mf_sirt(fair_mf A, const char *sirt_method, const double *b, int32_t K,
                 const double *x0, const fair_opts *options, double *x) {
    MENTER(A);
    if (!b || !x) return FAIR_ERR_NULL;
    FAIR_TRY(fair_mf_sirt_prepare(A, sirt_method, options));
    std::lock_guard<std::mutex> lk(A->mu);
    const int64_t m = (int64_t)A->nth * A->p, n = (int64_t)A->N * A->N;
    cudaStream_t s = A->stream;
    FAIR_TRY(A->w_b.grow(sizeof(double) * (m + 1)));
    FAIR_TRY(A->w_x.grow(sizeof(double) * (n + 1)));
    FAIR_CUDA(cudaMemcpyAsync(A->w_b.p, b, sizeof(double) * m, cudaMemcpyHostToDevice, s));
    if (x0) FAIR_CUDA(cudaMemcpyAsync(A->w_x.p, x0, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    else FAIR_CUDA(cudaMemsetAsync(A->w_x.p, 0, sizeof(double) * n, s));
    FAIR_TRY(mf_iterations(A, A->w_b.as<double>(), A->w_x.as<double>(), K, nullptr, nullptr));
    FAIR_CUDA(cudaMemcpyAsync(x, A->w_x.p, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    return FAIR_OK;
}

}  // extern "C"
