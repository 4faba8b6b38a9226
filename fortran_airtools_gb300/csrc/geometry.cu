// geometry.cu -- ray-traced system matrix (paralleltomo / fanlineartomo) on
// the GPU, one thread per ray, two passes (count, scan, fill) like the
// reference (system_generation.f90:138-212 count, :214-302 fill).
//
// Per ray the reference computes the 2N+2 crossings with the grid lines,
// quicksorts them by the ray parameter t, keeps the points inside the square
// and emits one nonzero per pair of consecutive points further apart than
// 1e-10 (system_generation.f90:163-203, :357-397). Here the two crossing
// families are already monotone in t, so the fast path merges them instead of
// sorting: the in-box points of each family form one index interval (found by
// binary search on the monotone other coordinate), and the merge yields the
// same sequence as the sort whenever no two in-box keys are equal. A ray whose
// keys contain a NaN (a == 0 or b == 0 with the ray on a grid line, where the
// reference's quicksort no longer sorts) or an exact tie between the families
// (where the unstable sort picks the order) is sent to the exact path, which
// replays the reference's Hoare quicksort on that ray.
//
// Every product, sum and quotient on the ray uses explicit round-to-nearest
// intrinsics so that no multiply-add is fused: the results then match the
// reference's separately rounded operations bit for bit.
//
// This part runs 2 FP64 lanes per clock and SM, so the FP64 operations per
// nonzero set the time (about 50 in each pass of the merge above). Almost
// every ray stays clear of the grid's corners and lines, and on those the
// integer units do the rest (the plain path):
//  * the in-box crossings of both families are index intervals, so a ray's
//    count is their number less one. The count pass checks in fixed point
//    that every crossing of the ray's major axis is at least 2^-28 off the
//    other family's lines; a ray that is not (or has a or b = 0) is listed
//    and takes the merge (or exact) path in both passes;
//  * the fill merges by integer comparison of the keys' bits, takes the
//    columns from the cells' indices, and forms the quotient and the root with
//    one and three FP64 operations, rounded correctly by their exact integer
//    remainders: 13 FP64 operations per nonzero.
// N = 256, 360 angles, 362 bins (33.4M nonzeros): count 3.2 -> 0.04 ms, fill
// 3.8 -> 1.03 ms (FP64 pipe 83% busy), the listed rays 0.03 ms.
#include <algorithm>
#include <vector>

#include "exact_round.cuh"
#include "fair_internal.cuh"

namespace fair {

namespace {

struct GeomDev {
    int kind, N, nth, p;
    const double *grid;
    const double *cth, *sth, *bx0, *by0;
    const double *ax0th, *ay0th, *aath, *abth, *com, *som;
};

struct Ray {
    double a, b, x0th, y0th;
    bool excluded;
};

// system_generation.f90:348-353 (parallel) and :146-157 (fan).
__device__ __forceinline__ Ray ray_params(const GeomDev &G, int i, int j) {
    Ray r;
    if (G.kind == 0) {
        double ct = G.cth[i], st = G.sth[i], x0 = G.bx0[j], y0 = G.by0[j];
        r.x0th = __dsub_rn(__dmul_rn(ct, x0), __dmul_rn(st, y0));
        r.y0th = __dadd_rn(__dmul_rn(st, x0), __dmul_rn(ct, y0));
        r.a = -st;
        r.b = ct;
        const double h = 0.5 * G.N;
        // boundary rays excluded by :393-394 / :466-467
        r.excluded = (r.b == 0.0 && fabs(__dsub_rn(r.y0th, h)) < 1e-15) ||
                     (r.a == 0.0 && fabs(__dsub_rn(r.x0th, h)) < 1e-15);
    } else {
        r.x0th = G.ax0th[i];
        r.y0th = G.ay0th[i];
        double ath = G.aath[i], bth = G.abth[i], co = G.com[j], so = G.som[j];
        r.a = __dsub_rn(__dmul_rn(co, ath), __dmul_rn(so, bth));
        r.b = __dadd_rn(__dmul_rn(so, ath), __dmul_rn(co, bth));
        r.excluded = false;
    }
    return r;
}

// Crossing with the vertical grid line x = g[k]: tx, yx of :163-164 / :357-358.
__device__ __forceinline__ void eval_x(const double *g, const Ray &r, int k, double &t,
                                       double &px, double &py) {
    px = g[k];
    t = __ddiv_rn(__dsub_rn(px, r.x0th), r.a);
    py = __dadd_rn(__dmul_rn(r.b, t), r.y0th);
}
// Crossing with the horizontal grid line y = g[l]: ty, xy of :168-169 / :362-363.
__device__ __forceinline__ void eval_y(const double *g, const Ray &r, int l, double &t,
                                       double &px, double &py) {
    py = g[l];
    t = __ddiv_rn(__dsub_rn(py, r.y0th), r.b);
    px = __dadd_rn(__dmul_rn(r.a, t), r.x0th);
}

// Smallest k in [0, N] with pred(k) true (pred monotone false..true); N+1 if none.
template <class P>
__device__ __forceinline__ int first_true(int N, P pred) {
    int L = 0, R = N + 1;
    while (L < R) {
        int mid = (L + R) >> 1;
        if (pred(mid)) R = mid; else L = mid + 1;
    }
    return L;
}

struct CountSink {
    __device__ __forceinline__ void emit(int64_t, double, int) {}
};

struct WriteSink {
    int32_t *col;
    double *val;
    int64_t cap;     // nonzeros reserved for this row by the count pass
    int32_t ncols;
    int *err;
    __device__ __forceinline__ void emit(int64_t k, double d, int ja) {
        if (ja < 1 || ja > ncols) {  // "++ Something went wrong" (:293, :478)
            atomicOr(err, 1);
            return;
        }
        if (k < cap) {
            col[k] = ja - 1;
            val[k] = d;
        }
    }
};

// Segment between consecutive in-box points (:199-203 / :279-297).
template <class Sink>
__device__ __forceinline__ void segment(int N, double px0, double py0, double px1, double py1,
                                        int64_t &cnt, Sink &sink) {
    double dx = __dsub_rn(px0, px1), dy = __dsub_rn(py0, py1);
    double d = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    if (d > 1e-10) {
        double xm = __dmul_rn(0.5, __dadd_rn(__dadd_rn(px0, px1), (double)N));
        double ym = __dmul_rn(0.5, __dadd_rn(__dadd_rn(py0, py1), (double)N));
        int ja = (int)floor(xm) * N + (N - (int)floor(ym));
        sink.emit(cnt, d, ja);
        cnt++;
    }
}

// Fast path. Returns the nonzero count, or -1 when the ray needs the exact path.
template <class Sink>
__device__ int64_t trace_merge(const GeomDev &G, const Ray &r, Sink &sink) {
    if (r.excluded) return 0;
    const int N = G.N;
    const double *g = G.grid;
    const double lo = -0.5 * N, hi = 0.5 * N;

    // x-crossings: in-box interval [kx0, kx1] of k (py monotone in k)
    int kx0 = 0, kx1 = -1;
    if (r.a != 0.0) {
        double t, px, py0, pyN;
        eval_x(g, r, 0, t, px, py0);
        eval_x(g, r, N, t, px, pyN);
        auto py = [&](int k) { double tt, xx, yy; eval_x(g, r, k, tt, xx, yy); return yy; };
        if (py0 <= pyN) {
            kx0 = first_true(N, [&](int k) { return py(k) >= lo; });
            kx1 = first_true(N, [&](int k) { return py(k) > hi; }) - 1;
        } else {
            kx0 = first_true(N, [&](int k) { return py(k) <= hi; });
            kx1 = first_true(N, [&](int k) { return py(k) < lo; }) - 1;
        }
    } else {
        for (int k = 0; k <= N; ++k)
            if (g[k] == r.x0th) return -1;  // 0/0 = NaN key
    }
    // y-crossings: in-box interval [ly0, ly1] of l (px monotone in l)
    int ly0 = 0, ly1 = -1;
    if (r.b != 0.0) {
        double t, py, px0, pxN;
        eval_y(g, r, 0, t, px0, py);
        eval_y(g, r, N, t, pxN, py);
        auto px = [&](int l) { double tt, xx, yy; eval_y(g, r, l, tt, xx, yy); return xx; };
        if (px0 <= pxN) {
            ly0 = first_true(N, [&](int l) { return px(l) >= lo; });
            ly1 = first_true(N, [&](int l) { return px(l) > hi; }) - 1;
        } else {
            ly0 = first_true(N, [&](int l) { return px(l) <= hi; });
            ly1 = first_true(N, [&](int l) { return px(l) < lo; }) - 1;
        }
    } else {
        for (int l = 0; l <= N; ++l)
            if (g[l] == r.y0th) return -1;
    }

    int nx = kx1 >= kx0 ? kx1 - kx0 + 1 : 0;
    int ny = ly1 >= ly0 ? ly1 - ly0 + 1 : 0;
    // t increases with k when a > 0 and with l when b > 0
    int kx = r.a > 0.0 ? kx0 : kx1, sx = r.a > 0.0 ? 1 : -1;
    int ly = r.b > 0.0 ? ly0 : ly1, sy = r.b > 0.0 ? 1 : -1;
    double tX = 0, xX = 0, yX = 0, tY = 0, xY = 0, yY = 0;
    if (nx) eval_x(g, r, kx, tX, xX, yX);
    if (ny) eval_y(g, r, ly, tY, xY, yY);

    int64_t cnt = 0;
    bool have = false;
    double ppx = 0, ppy = 0;
    while (nx > 0 || ny > 0) {
        bool takeX;
        if (nx > 0 && ny > 0) {
            if (tX == tY) return -1;  // unstable-sort tie: exact path
            takeX = tX < tY;
        } else {
            takeX = nx > 0;
        }
        double px, py;
        if (takeX) {
            px = xX; py = yX;
            if (--nx) { kx += sx; eval_x(g, r, kx, tX, xX, yX); }
        } else {
            px = xY; py = yY;
            if (--ny) { ly += sy; eval_y(g, r, ly, tY, xY, yY); }
        }
        // in-box test of :188 / :382 (the grid coordinate is inside by construction)
        if (px >= lo && px <= hi && py >= lo && py <= hi) {
            if (have) segment(N, ppx, ppy, px, py, cnt, sink);
            ppx = px; ppy = py; have = true;
        }
    }
    return cnt;
}

// Exact path: the reference's quicksort (system_generation.f90:37-77) on the
// full key array of one ray, held in per-ray scratch.
struct RayScratch {
    double *t, *xxy, *yxy;
    int32_t *ind;
};

__device__ void quicksort_emul(double *a, int32_t *ind, int nt) {
    // The two recursive calls of :75-76 act on disjoint index ranges, so any
    // processing order gives the same result; the larger range is stacked.
    int stk_f[64], stk_l[64];
    int top = 0;
    stk_f[top] = 0; stk_l[top] = nt - 1; top++;
    while (top > 0) {
        --top;
        int f = stk_f[top], l = stk_l[top];
        while (f < l) {
            double x = a[(f + l) >> 1];  // 1-based (f+l)/2 maps to the same element
            int i = f, j = l;
            for (;;) {
                while (i < l && a[i] < x) i++;
                while (j > f && x < a[j]) j--;
                if (i >= j) break;
                double tt = a[i]; a[i] = a[j]; a[j] = tt;
                int32_t m = ind[i]; ind[i] = ind[j]; ind[j] = m;
                i++;
                j--;
            }
            int lf = f, ll = i - 1, rf = j + 1, rl = l;
            bool hasL = lf < ll, hasR = rf < rl;
            if (hasL && hasR) {
                if (ll - lf > rl - rf) {
                    if (top < 64) { stk_f[top] = lf; stk_l[top] = ll; top++; }
                    f = rf; l = rl;
                } else {
                    if (top < 64) { stk_f[top] = rf; stk_l[top] = rl; top++; }
                    f = lf; l = ll;
                }
            } else if (hasL) {
                f = lf; l = ll;
            } else if (hasR) {
                f = rf; l = rl;
            } else {
                break;
            }
        }
    }
}

template <class Sink>
__device__ int64_t trace_exact(const GeomDev &G, const Ray &r, RayScratch s, Sink &sink) {
    if (r.excluded) return 0;
    const int N = G.N, np = N + 1, nt = 2 * N + 2;
    const double *g = G.grid;
    for (int k = 0; k < np; ++k) {
        double tx, xx, yx, ty, xy, yy;
        eval_x(g, r, k, tx, xx, yx);
        eval_y(g, r, k, ty, xy, yy);
        s.t[k] = tx;       s.t[np + k] = ty;
        s.xxy[k] = xx;     s.xxy[np + k] = xy;
        s.yxy[k] = yx;     s.yxy[np + k] = yy;
        s.ind[k] = k;      s.ind[np + k] = np + k;
    }
    quicksort_emul(s.t, s.ind, nt);
    const double lo = -0.5 * N, hi = 0.5 * N;
    int64_t cnt = 0;
    bool have = false;
    double ppx = 0, ppy = 0;
    for (int k = 0; k < nt; ++k) {
        double px = s.xxy[s.ind[k]], py = s.yxy[s.ind[k]];
        if (px >= lo && px <= hi && py >= lo && py <= hi) {
            if (have) segment(N, ppx, ppy, px, py, cnt, sink);
            ppx = px; ppy = py; have = true;
        }
    }
    return cnt;
}

// ---- the plain path ----------------------------------------------------------
__device__ __forceinline__ long long key_of(double t) {  // order-preserving for numbers
    const long long b = __double_as_longlong(t);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// The cell of a segment by its midpoint (:200-203), a call as the rare operations
// of exact_round.cuh.
__device__ __noinline__ int mid_cell(double p0, double p1, int N) {
    return (int)floor(__dmul_rn(0.5, __dadd_rn(__dadd_rn(p0, p1), (double)N)));
}

// Crossings as eval_x / eval_y, the quotient by div_by.
__device__ __forceinline__ void cross(double line, double o0, double dir, double inv, double odir,
                                      double oo0, double &t, double &other) {
    t = div_by(__dsub_rn(line, o0), dir, inv);
    other = __dadd_rn(__dmul_rn(odir, t), oo0);
}

// The in-box interval [k0, k1] of one family: lines g[0..N], the other
// coordinate monotone in k and within [lo, hi] there.
struct Span {
    int k0, k1;
};
__device__ __forceinline__ Span in_box(const double *g, int N, double o0, double dir, double inv,
                                       double odir, double oo0, long long klo, long long khi) {
    auto at = [&](int k) {
        double t, o;
        cross(g[k], o0, dir, inv, odir, oo0, t, o);
        return key_of(o);
    };
    const bool up = at(0) <= at(N);
    // where the other coordinate meets lo / hi, from floats; the exact predicate decides
    const float f = (float)dir / (float)odir, z = (float)o0 + 0.5f * (float)N, w = (float)oo0;
    auto first = [&](float other, auto pred) {
        const float kf = ceilf(fmaf(other - w, f, z));
        const int k = kf >= 0.f && kf <= (float)(N + 1) ? (int)kf : (kf < 0.f ? 0 : N + 1);
        // k is the first true when pred(k) (or none left) and not pred(k - 1)
        for (int c = k - 1; c <= k + 1; ++c)
            if (c >= 0 && c <= N + 1 && (c > N || pred(c)) && (c == 0 || !pred(c - 1))) return c;
        return first_true(N, pred);
    };
    const float lo = -0.5f * (float)N, hi = 0.5f * (float)N;
    Span s;
    if (up) {
        s.k0 = first(lo, [&](int k) { return at(k) >= klo; });
        s.k1 = first(hi, [&](int k) { return at(k) > khi; }) - 1;
    } else {
        s.k0 = first(hi, [&](int k) { return at(k) <= khi; });
        s.k1 = first(lo, [&](int k) { return at(k) < klo; }) - 1;
    }
    return s;
}

// True when a crossing of the ray's major axis (direction component d, in-box
// lines s) comes within 2^-28 of a line of the other family: the other
// coordinate o(k) in fixed point with 46 fractional bits (its step rounded: off by
// at most N (2^-47 + 2^-52) + 2^-46, below 2^-30 up to N = 2^16), lines of the other
// family at its integers.
__device__ __forceinline__ bool near_line(const double *g, int N, double o0, double dir, double inv,
                                          double odir, double oo0, Span s) {
    if (s.k1 < s.k0) return false;
    double t, o;
    cross(g[s.k0], o0, dir, inv, odir, oo0, t, o);
    const double one = 70368744177664.0;  // 2^46
    long long Y = llrint((o + 0.5 * N) * one) + (1LL << 18);
    const long long S = llrint(odir * inv * one);
    unsigned bad = 0;
    for (int k = s.k0; k <= s.k1; ++k) {
        // bits 19..45 of Y all zero: within 2^18 units of an integer
        const unsigned lo = (unsigned)Y, hi = (unsigned)((unsigned long long)Y >> 32);
        bad |= ((lo >> 19) | (hi & 0x3fffu)) == 0u ? 1u : 0u;
        Y += S;
    }
    return bad != 0;
}

// Count pass: spans[r] = the in-box lines of both families; rays off the
// plain path are listed (their counts come from k_geom_count_list).
__global__ void __launch_bounds__(128) k_geom_spans(GeomDev G, int32_t *counts, int4 *spans,
                                                    int32_t *listed, int32_t *nlisted) {
    const int64_t m = (int64_t)G.nth * G.p;
    const int N = G.N;
    const long long klo = key_of(-0.5 * N), khi = key_of(0.5 * N);
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m;
         r += (int64_t)gridDim.x * blockDim.x) {
        const Ray ray = ray_params(G, (int)(r / G.p), (int)(r % G.p));
        int4 sp = make_int4(0, -1, 0, -1);
        int c = 0;
        if (!ray.excluded) {
            // NaN positions (p = 1) and infinite ones leave the comparisons false; a
            // direction component is 0 or large enough for finite parameters
            const double fa = fabs(ray.a), fb = fabs(ray.b);
            bool list = !((fa > 1e-30 || fa == 0.0) && (fb > 1e-30 || fb == 0.0) && fa + fb > 0.5 &&
                          fabs(ray.x0th) < 1e15 && fabs(ray.y0th) < 1e15);
            if (!list) {
                const double ia = __drcp_rn(ray.a), ib = __drcp_rn(ray.b);
                Span x{0, -1}, y{0, -1};
                if (fa > 0.0) x = in_box(G.grid, N, ray.x0th, ray.a, ia, ray.b, ray.y0th, klo, khi);
                if (fb > 0.0) y = in_box(G.grid, N, ray.y0th, ray.b, ib, ray.a, ray.x0th, klo, khi);
                // (an axis-aligned ray on a line of the other family, where the reference
                // divides 0 by 0, may lie on any of the N + 1: also outside the box's ends)
                list = fa >= fb ? near_line(G.grid, N, ray.x0th, ray.a, ia, ray.b, ray.y0th, x)
                                : near_line(G.grid, N, ray.y0th, ray.b, ib, ray.a, ray.x0th, y);
                const int nx = max(0, x.k1 - x.k0 + 1), ny = max(0, y.k1 - y.k0 + 1);
                c = max(0, nx + ny - 1);
                sp = make_int4(x.k0, x.k1, y.k0, y.k1);
            }
            if (list) {
                listed[atomicAdd(nlisted, 1)] = (int32_t)r;
                sp = make_int4(0, -1, 0, -2);  // not the plain path's
                c = 0;
            }
        }
        spans[r] = sp;
        counts[r] = c;
    }
}

// A listed ray by a block: the merge of trace_merge with every crossing
// evaluated at once, a point's place its own index plus the number of the
// other family's points before it. Returns the nonzero count, or -1 for the
// exact path. (One thread per listed ray took 0.8 ms for the few hundred rays
// that meet corners at 30 and 60 degrees; a block takes ~10 us.)
constexpr int kListThreads = 128;
template <class Sink>
__device__ int64_t trace_block(const GeomDev &G, const Ray &r, unsigned char *smem, Sink &sink) {
    const int N = G.N, t = threadIdx.x;
    const double *g = G.grid;
    double *T = reinterpret_cast<double *>(smem);       // tX [N+1], tY [N+1]
    double *O = T + 2 * (N + 1);                        // yX, xY
    int *place = reinterpret_cast<int *>(O + 2 * (N + 1));  // merged point -> point
    __shared__ int s_scan[kListThreads / 32];
    if (r.excluded) return 0;
    const double lo = -0.5 * N, hi = 0.5 * N;
    int k0[2] = {0, 0}, cnt[2] = {0, 0};
    const double dir[2] = {r.a, r.b}, org[2] = {r.x0th, r.y0th};
    const bool usual = fabs(r.a) > 1e-30 && fabs(r.b) > 1e-30 && fabs(r.x0th) < 1e15 && fabs(r.y0th) < 1e15;
    bool special = false;
    for (int f = 0; f < 2; ++f) {
        if (dir[f] == 0.0) {
            for (int k = t; k <= N; k += kListThreads) special |= g[k] == org[f];  // 0/0 = NaN key
            continue;
        }
        auto other = [&](int k) {
            double tt, px, py;
            if (f == 0) eval_x(g, r, k, tt, px, py); else eval_y(g, r, k, tt, px, py);
            return f == 0 ? py : px;
        };
        int a, b;
        if (usual) {
            const Span sp = in_box(g, N, org[f], dir[f], __drcp_rn(dir[f]), dir[1 - f], org[1 - f],
                                   key_of(lo), key_of(hi));
            a = sp.k0;
            b = sp.k1;
        } else if (other(0) <= other(N)) {
            a = first_true(N, [&](int k) { return other(k) >= lo; });
            b = first_true(N, [&](int k) { return other(k) > hi; }) - 1;
        } else {
            a = first_true(N, [&](int k) { return other(k) <= hi; });
            b = first_true(N, [&](int k) { return other(k) < lo; }) - 1;
        }
        k0[f] = dir[f] > 0.0 ? a : b;  // first in ray order
        cnt[f] = b >= a ? b - a + 1 : 0;
    }
    for (int f = 0; f < 2; ++f)
        for (int i = t; i < cnt[f]; i += kListThreads) {
            const int k = k0[f] + (dir[f] > 0.0 ? i : -i);
            double tt, px, py;
            if (f == 0) eval_x(g, r, k, tt, px, py); else eval_y(g, r, k, tt, px, py);
            T[f * (N + 1) + i] = tt;
            O[f * (N + 1) + i] = f == 0 ? py : px;
        }
    __syncthreads();
    for (int f = 0; f < 2; ++f) {
        const double *A = T + f * (N + 1), *B = T + (1 - f) * (N + 1);
        const int nb = cnt[1 - f];
        for (int i = t; i < cnt[f]; i += kListThreads) {
            const double v = A[i];
            int L = 0, R = nb;
            while (L < R) {
                const int mid = (L + R) >> 1;
                if (B[mid] < v) L = mid + 1; else R = mid;
            }
            special |= L < nb && B[L] == v;  // unstable-sort tie
            place[i + L] = f * (N + 1) + i;
        }
    }
    if (__syncthreads_or(special)) return -1;
    const int n = cnt[0] + cnt[1];
    auto point = [&](int q, double &px, double &py) {
        const int u = place[q], f = u > N, i = u - f * (N + 1);
        const double line = g[k0[f] + (dir[f] > 0.0 ? i : -i)];
        px = f ? O[u] : line;
        py = f ? line : O[u];
    };
    int64_t total = 0;
    for (int base = 0; base + 1 < n; base += kListThreads) {
        const int q = base + t;
        double x0 = 0, y0 = 0, x1 = 0, y1 = 0;
        bool keep = false;
        if (q + 1 < n) {
            point(q, x0, y0);
            point(q + 1, x1, y1);
            CountSink cs;
            int64_t c = 0;
            segment(N, x0, y0, x1, y1, c, cs);
            keep = c > 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if ((t & 31) == 0) s_scan[t >> 5] = __popc(m);
        __syncthreads();
        int64_t at = total + __popc(m & ((1u << (t & 31)) - 1u));
        for (int w = 0; w < kListThreads / 32; ++w) {
            if (w < t >> 5) at += s_scan[w];
            total += s_scan[w];
        }
        if (keep) segment(N, x0, y0, x1, y1, at, sink);
        __syncthreads();
    }
    return total;
}
size_t list_smem(int N) { return (size_t)(N + 1) * (4 * sizeof(double) + 2 * sizeof(int)); }
constexpr size_t kListSmem = 200 * 1024;  // N <= 5119; longer rays take the merge, one thread each

// The listed rays; those neither can order go on to the exact path.
__global__ void __launch_bounds__(kListThreads) k_geom_count_list(GeomDev G, const int32_t *listed,
                                                                  int32_t nlisted, int32_t *counts,
                                                                  int32_t *special, int32_t *nspecial,
                                                                  bool block) {
    extern __shared__ __align__(16) unsigned char list_smem_buf[];
    for (int q = blockIdx.x; q < nlisted; q += gridDim.x) {
        const int32_t r = listed[q];
        const Ray ray = ray_params(G, r / G.p, r % G.p);
        CountSink cs;
        int64_t c = 0;
        if (block) c = trace_block(G, ray, list_smem_buf, cs);
        else if (threadIdx.x == 0) c = trace_merge(G, ray, cs);
        if (threadIdx.x == 0) {
            if (c < 0) {
                special[atomicAdd(nspecial, 1)] = r;
                c = 0;
            }
            counts[r] = (int32_t)c;
        }
        __syncthreads();
    }
}

__global__ void k_geom_count_exact(GeomDev G, const int32_t *special, int32_t nsp,
                                   double *scr_d, int32_t *scr_i, int32_t *counts) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nsp) return;
    const int nt = 2 * G.N + 2;
    RayScratch s{scr_d + (size_t)q * 3 * nt, scr_d + (size_t)q * 3 * nt + nt,
                 scr_d + (size_t)q * 3 * nt + 2 * nt, scr_i + (size_t)q * nt};
    int32_t r = special[q];
    Ray ray = ray_params(G, r / G.p, r % G.p);
    CountSink cs;
    counts[r] = (int32_t)trace_exact(G, ray, s, cs);
}

// Fill pass of the plain path. A ray's crossings are cut into parts of
// kPart lines of its major axis, one lane per ray and part (a warp: the same
// part of 32 neighbouring rays), so that the warps' work is even; a part
// starts at a major crossing, whose place in the row is its own index plus
// the minor lines before it (the cell it lies in tells them).
constexpr int kPart = 64;
__global__ void __launch_bounds__(128) k_geom_fill(GeomDev G, const int4 *spans, const int64_t *rowptr,
                                                   int32_t *col, double *val, int parts, int *err) {
    const int64_t m = (int64_t)G.nth * G.p;
    const int N = G.N, lane = threadIdx.x & 31;
    const double *g = G.grid;
    const long long never = 0x7fffffffffffffffLL;
    const int64_t items = ((m + 31) >> 5) * parts;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < items;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t r = (w / parts) * 32 + lane;
        const int part = (int)(w % parts);
        if (r >= m) continue;
        const int4 sp = spans[r];
        if (sp.w == -2) continue;  // listed
        const Ray ray = ray_params(G, (int)(r / G.p), (int)(r % G.p));
        const bool xm = fabs(ray.a) >= fabs(ray.b);  // the major axis
        const double dm = xm ? ray.a : ray.b, dn = xm ? ray.b : ray.a;
        const double om = xm ? ray.x0th : ray.y0th, on = xm ? ray.y0th : ray.x0th;
        const int m0 = xm ? sp.x : sp.z, m1 = xm ? sp.y : sp.w, n0 = xm ? sp.z : sp.x, n1 = xm ? sp.w : sp.y;
        const int nm = max(0, m1 - m0 + 1), nn = max(0, n1 - n0 + 1);
        if (part > 0 ? part * kPart >= nm : nm + nn < 2) continue;
        const int stop = (part + 1) * kPart < nm ? (part + 1) * kPart : -1;  // major crossing it ends at
        const double im = __drcp_rn(dm), in = __drcp_rn(dn);
        // line numbers grow along the ray when its direction component is positive
        const int sm = dm > 0.0 ? 1 : -1, sn = dn > 0.0 ? 1 : -1;
        int q = part * kPart, c = 0;  // major and minor crossings passed
        int km = sm > 0 ? m0 + q : m1 - q, kn = sn > 0 ? n0 : n1;
        double tm = 0, om1 = 0, gm = 0, tn = 0, on1 = 0, gn = 0;
        long long Km = never, Kn = never;
        double pt = 0, pm = 0, pn = 0;
        int cm = -1, cn = -1;  // the cell behind the last crossing, -1: not known yet
        int64_t o = rowptr[r];
        const int64_t end = rowptr[r + 1];
        bool have = false;
        if (q < nm) {
            gm = g[km];
            cross(gm, om, dm, im, dn, on, tm, om1);
            Km = key_of(tm);
        }
        if (part > 0) {  // start at that crossing
            pt = tm; pm = gm; pn = om1;
            have = true;
            cm = sm > 0 ? km : km - 1;
            cn = (int)floor(__dadd_rn(om1, 0.5 * N));
            c = max(0, min(nn, sn > 0 ? cn - n0 + 1 : n1 - cn));
            kn += sn * c;
            o += q + c;
            ++q;
            km += sm;
            Km = never;
            if (q < nm) {
                gm = g[km];
                cross(gm, om, dm, im, dn, on, tm, om1);
                Km = key_of(tm);
            }
        }
        if (c < nn) {
            gn = g[kn];
            cross(gn, on, dn, in, dm, om, tn, on1);
            Kn = key_of(tn);
        }
        while (q < nm || c < nn) {
            const bool maj = Km < Kn;
            const double ct = maj ? tm : tn, vm = maj ? gm : on1, vn = maj ? om1 : gn;
            if (have) {
                const double d1 = __dsub_rn(pm, vm), d2 = __dsub_rn(pn, vn);
                const double v = __dadd_rn(__dmul_rn(d1, d1), __dmul_rn(d2, d2));
                const double s0 = __longlong_as_double(
                    __double_as_longlong(__dsub_rn(ct, pt)) & 0x7fffffffffffffffLL);
                const double d = sqrt_near(v, s0);
                if (cm < 0) cm = mid_cell(pm, vm, N);  // the first segment's
                if (cn < 0) cn = mid_cell(pn, vn, N);
                const int ix = xm ? cm : cn, iy = xm ? cn : cm;
                if ((unsigned)ix >= (unsigned)N || (unsigned)iy >= (unsigned)N) atomicOr(err, 1);
                else if (o < end) {
                    col[o] = ix * N + (N - 1 - iy);
                    val[o] = d;
                }
                ++o;
            }
            have = true;
            pt = ct; pm = vm; pn = vn;
            // the next crossing of the family just passed: selects around one
            // evaluation (in a branch per family a warp would evaluate both)
            if (maj && q == stop) break;
            int mj = maj ? 1 : 0;
            asm volatile("" : "+r"(mj));
            cm = mj ? (sm > 0 ? km : km - 1) : cm;
            cn = mj ? cn : (sn > 0 ? kn : kn - 1);
            km += mj ? sm : 0;
            kn += mj ? 0 : sn;
            q += mj;
            c += 1 - mj;
            const bool more = mj ? q < nm : c < nn;
            const double line = g[more ? (mj ? km : kn) : 0];
            double t1, o1;
            cross(line, mj ? om : on, mj ? dm : dn, mj ? im : in, mj ? dn : dm, mj ? on : om, t1, o1);
            const long long K1 = more ? key_of(t1) : never;
            tm = mj ? t1 : tm;
            om1 = mj ? o1 : om1;
            gm = mj ? line : gm;
            Km = mj ? K1 : Km;
            tn = mj ? tn : t1;
            on1 = mj ? on1 : o1;
            gn = mj ? gn : line;
            Kn = mj ? Kn : K1;
        }
        if (stop < 0 && o != end) atomicOr(err, 2);  // "Didn't hit all elements" (:304)
    }
}

// The listed rays' fill.
__global__ void __launch_bounds__(kListThreads) k_geom_fill_list(GeomDev G, const int32_t *listed,
                                                                 int32_t nlisted, const int64_t *rowptr,
                                                                 int32_t *col, double *val, int32_t ncols,
                                                                 int *err, bool block) {
    extern __shared__ __align__(16) unsigned char list_smem_buf[];
    for (int q = blockIdx.x; q < nlisted; q += gridDim.x) {
        const int32_t r = listed[q];
        const Ray ray = ray_params(G, r / G.p, r % G.p);
        const int64_t s0 = rowptr[r], cap = rowptr[r + 1] - s0;
        WriteSink ws{col + s0, val + s0, cap, ncols, err};
        int64_t c = -1;
        if (block) c = trace_block(G, ray, list_smem_buf, ws);
        else if (threadIdx.x == 0) c = trace_merge(G, ray, ws);
        if (threadIdx.x == 0 && c >= 0 && c != cap) atomicOr(err, 2);
        __syncthreads();
    }
}

__global__ void k_geom_fill_exact(GeomDev G, const int32_t *special, int32_t nsp, double *scr_d,
                                  int32_t *scr_i, const int64_t *rowptr, int32_t *col,
                                  double *val, int32_t ncols, int *err) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nsp) return;
    const int nt = 2 * G.N + 2;
    RayScratch s{scr_d + (size_t)q * 3 * nt, scr_d + (size_t)q * 3 * nt + nt,
                 scr_d + (size_t)q * 3 * nt + 2 * nt, scr_i + (size_t)q * nt};
    int32_t r = special[q];
    Ray ray = ray_params(G, r / G.p, r % G.p);
    int64_t s0 = rowptr[r], cap = rowptr[r + 1] - s0;
    WriteSink ws{col + s0, val + s0, cap, ncols, err};
    int64_t c = trace_exact(G, ray, s, ws);
    if (c != cap) atomicOr(err, 2);
}

GeomDev to_dev(const GeomTables &T) {
    GeomDev G;
    G.kind = T.kind; G.N = T.N; G.nth = T.nth; G.p = T.p;
    G.grid = T.grid.as<double>();
    G.cth = T.cth.as<double>(); G.sth = T.sth.as<double>();
    G.bx0 = T.bx0.as<double>(); G.by0 = T.by0.as<double>();
    G.ax0th = T.ax0th.as<double>(); G.ay0th = T.ay0th.as<double>();
    G.aath = T.aath.as<double>(); G.abth = T.abth.as<double>();
    G.com = T.com.as<double>(); G.som = T.som.as<double>();
    return G;
}

constexpr int kExactBatch = 2048;  // special rays traced per launch (scratch bound)

}  // namespace

namespace {
// The count pass (k_geom_spans, the listed rays through the merge, then the
// exact path for those whose keys need the quicksort replay): entries per ray
// into counts [m]; the spans, the lists and the exact path's scratch stay for
// the fill.
struct GeomCount {
    DevBuf counts, spans, listed, special, nsp, scr_d, scr_i;
    int32_t h_listed = 0, h_nsp = 0, batch = 0;
    int blocks = 1;
    static constexpr int threads = 128;
    // a block per listed ray, its crossings in shared memory where they fit
    bool in_blocks(int N) const { return list_smem(N) <= kListSmem; }
    int list_blocks() const { return h_listed < 4096 ? h_listed : 4096; }
    size_t smem(int N) const { return in_blocks(N) ? list_smem(N) : 0; }
    void release() {
        counts.release(); spans.release(); listed.release(); special.release(); nsp.release();
        scr_d.release(); scr_i.release();
    }
};

int geometry_count(const GeomTables &T, const GeomDev &G, GeomCount &C, cudaStream_t s) {
    const int64_t m = (int64_t)T.nth * T.p;
    FAIR_TRY(C.counts.grow(sizeof(int32_t) * (m > 0 ? m : 1)));
    FAIR_TRY(C.spans.grow(sizeof(int4) * (m > 0 ? m : 1)));
    FAIR_TRY(C.listed.grow(sizeof(int32_t) * (m > 0 ? m : 1)));
    FAIR_TRY(C.nsp.grow(2 * sizeof(int32_t)));
    FAIR_CUDA(cudaMemsetAsync(C.nsp.p, 0, 2 * sizeof(int32_t), s));
    int64_t blocks64 = (m + C.threads - 1) / C.threads;
    C.blocks = (int)(blocks64 < (int64_t)sm_count() * 64 ? (blocks64 > 0 ? blocks64 : 1)
                                                         : (int64_t)sm_count() * 64);
    k_geom_spans<<<C.blocks, C.threads, 0, s>>>(G, C.counts.as<int32_t>(), C.spans.as<int4>(),
                                                C.listed.as<int32_t>(), C.nsp.as<int32_t>());
    FAIR_CUDA(cudaGetLastError());
    FAIR_CUDA(cudaMemcpyAsync(&C.h_listed, C.nsp.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    if (C.h_listed > 0) {
        FAIR_TRY(C.special.grow(sizeof(int32_t) * (size_t)C.h_listed));
        FAIR_CUDA(cudaFuncSetAttribute(k_geom_count_list, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kListSmem));
        k_geom_count_list<<<C.list_blocks(), kListThreads, C.smem(T.N), s>>>(
            G, C.listed.as<int32_t>(), C.h_listed, C.counts.as<int32_t>(), C.special.as<int32_t>(),
            C.nsp.as<int32_t>() + 1, C.in_blocks(T.N));
        FAIR_CUDA(cudaGetLastError());
        FAIR_CUDA(cudaMemcpyAsync(&C.h_nsp, C.nsp.as<int32_t>() + 1, sizeof(int32_t),
                                  cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaStreamSynchronize(s));
    }
    // Scratch for the exact path: keys, two coordinate arrays, permutation.
    const int nt = 2 * T.N + 2;
    C.batch = C.h_nsp < kExactBatch ? C.h_nsp : kExactBatch;
    if (C.h_nsp > 0) {
        FAIR_TRY(C.scr_d.grow(sizeof(double) * 3 * (size_t)nt * C.batch));
        FAIR_TRY(C.scr_i.grow(sizeof(int32_t) * (size_t)nt * C.batch));
        for (int32_t q0 = 0; q0 < C.h_nsp; q0 += C.batch) {
            int32_t nq = C.h_nsp - q0 < C.batch ? C.h_nsp - q0 : C.batch;
            k_geom_count_exact<<<(nq + 63) / 64, 64, 0, s>>>(G, C.special.as<int32_t>() + q0, nq,
                                                            C.scr_d.as<double>(),
                                                            C.scr_i.as<int32_t>(),
                                                            C.counts.as<int32_t>());
            FAIR_CUDA(cudaGetLastError());
        }
    }
    return FAIR_OK;
}
}  // namespace

int geometry_nnz(const GeomTables &T, int64_t *nnz, cudaStream_t s) {
    const int64_t m = (int64_t)T.nth * T.p;
    GeomDev G = to_dev(T);
    GeomCount C;
    FAIR_TRY(geometry_count(T, G, C, s));
    DevBuf rp;
    FAIR_TRY(rp.grow(sizeof(int64_t) * (m + 1)));
    FAIR_TRY(scan_counts(C.counts.as<int32_t>(), m, rp.as<int64_t>(), s));
    FAIR_CUDA(cudaMemcpyAsync(nnz, rp.as<int64_t>() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    return FAIR_OK;
}

int build_geometry(const GeomTables &T, DevCSR &A, cudaStream_t s) {
    const int64_t m = (int64_t)T.nth * T.p;
    const int32_t ncols = T.N * T.N;
    GeomDev G = to_dev(T);
    A.release();
    A.m = (int32_t)m;
    A.n = ncols;
    A.stride_hint = T.N;   // pixel (x, y) is column x*N + (N - y)
    A.tstride_hint = T.p;  // ray (angle i, bin j) is row i*p + j

    GeomCount C;
    FAIR_TRY(geometry_count(T, G, C, s));
    DevBuf err;
    FAIR_TRY(err.grow(sizeof(int)));
    FAIR_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    DevBuf &counts = C.counts, &special = C.special, &scr_d = C.scr_d, &scr_i = C.scr_i;
    const int32_t h_nsp = C.h_nsp, batch = C.batch;

    FAIR_TRY(A.rowptr.grow(sizeof(int64_t) * (m + 1)));
    FAIR_TRY(scan_counts(counts.as<int32_t>(), m, A.rowptr.as<int64_t>(), s));
    int64_t nnz = 0;
    FAIR_CUDA(cudaMemcpyAsync(&nnz, A.rowptr.as<int64_t>() + m, sizeof(int64_t),
                              cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    A.nnz = nnz;
    FAIR_TRY(A.alloc_entries(nnz, s));

    const int parts = T.N / kPart + 1;  // of up to N + 1 major lines
    const int64_t items = (m + 31) / 32 * parts;
    k_geom_fill<<<(unsigned)std::min<int64_t>((items + 3) / 4, 1 << 20), 128, 0, s>>>(
        G, C.spans.as<int4>(), A.rowptr.as<int64_t>(), A.col.as<int32_t>(), A.v64.as<double>(), parts,
        err.as<int>());
    FAIR_CUDA(cudaGetLastError());
    if (C.h_listed > 0) {
        FAIR_CUDA(cudaFuncSetAttribute(k_geom_fill_list, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kListSmem));
        k_geom_fill_list<<<C.list_blocks(), kListThreads, C.smem(T.N), s>>>(
            G, C.listed.as<int32_t>(), C.h_listed, A.rowptr.as<int64_t>(), A.col.as<int32_t>(),
            A.v64.as<double>(), ncols, err.as<int>(), C.in_blocks(T.N));
        FAIR_CUDA(cudaGetLastError());
    }
    for (int32_t q0 = 0; q0 < h_nsp; q0 += batch) {
        int32_t nq = h_nsp - q0 < batch ? h_nsp - q0 : batch;
        k_geom_fill_exact<<<(nq + 63) / 64, 64, 0, s>>>(
            G, special.as<int32_t>() + q0, nq, scr_d.as<double>(), scr_i.as<int32_t>(),
            A.rowptr.as<int64_t>(), A.col.as<int32_t>(), A.v64.as<double>(), ncols, err.as<int>());
        FAIR_CUDA(cudaGetLastError());
    }
    int h_err = 0;
    FAIR_CUDA(cudaMemcpyAsync(&h_err, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    C.release();
    err.release();
    if (h_err) {
        set_detail(h_err & 1 ? "column index outside 1..N^2 while tracing a ray"
                             : "fill pass wrote a different count than the count pass");
        A.release();
        return FAIR_ERR_GEOMETRY;
    }
    FAIR_TRY(csr_max_row(A, s));
    return FAIR_OK;
}

}  // namespace fair
